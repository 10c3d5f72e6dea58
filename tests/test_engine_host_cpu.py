"""The engine's host side (lcb_engine.cu: buffers, re-plans, staging) on CPU.

lcb_engine.cu is compiled by g++ and linked with a stand-in for the CUDA runtime:
device memory is host memory, a copy or a clear happens at once (or is recorded,
during a capture), kernels do nothing but the last, which writes run r's flux of
datum d as 1000 r + d.  The stand-in counts allocations and can fail a call."""
import importlib
import shutil
import subprocess

import pytest

from conftest import ROOT

FAKE = r"""
#include <cuda_runtime.h>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <fstream>
#include <functional>
#include <map>
#include <string>
#include <vector>
#include "lcurve_b200.h"
#include "lcb_kernels.cuh"
#include "lcb_plan.h"
static std::map<std::string, long> calls;  // of the functions that allocate, free or copy
static std::string fail_call;              // this function fails from its `fail_at`-th call on
static long fail_at = 0;
static bool capturing = false;
using Ops = std::vector<std::function<void()>>;
static Ops* recorded = nullptr;
static int runs = 0;
static cudaError_t called(const char* f) {
    const long n = ++calls[f];
    return fail_call == f && n >= fail_at ? cudaErrorMemoryAllocation : cudaSuccess;
}
static void issue(std::function<void()> f) {
    if (capturing) recorded->push_back(std::move(f));
    else f();
}
extern "C" {
cudaError_t cudaMalloc(void** p, size_t n) { if (called("cudaMalloc")) return cudaErrorMemoryAllocation; *p = std::malloc(n); std::memset(*p, 0x5a, n); return cudaSuccess; }
cudaError_t cudaFree(void* p) { std::free(p); return called("cudaFree"); }
cudaError_t cudaMallocHost(void** p, size_t n) { if (called("cudaMallocHost")) return cudaErrorMemoryAllocation; *p = std::malloc(n); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { std::free(p); return called("cudaFreeHost"); }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { std::memcpy(d, s, n); return called("cudaMemcpy"); }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
    if (called("cudaMemcpyAsync")) return cudaErrorMemoryAllocation;
    issue([=] { std::memcpy(d, s, n); });
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) { issue([=] { std::memset(d, v, n); }); return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = (cudaEvent_t)1; return called("cudaEventCreate"); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = (cudaEvent_t)1; return called("cudaEventCreate"); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 0.f; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDeviceProperties(cudaDeviceProp* p, int) { std::memset(p, 0, sizeof *p); p->major = 10; p->multiProcessorCount = 148; return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "an error of the stand-in"; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void** p, const void* s) { *p = const_cast<void*>(s); return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t g) { delete (Ops*)g; return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t g, unsigned long long) { *e = (cudaGraphExec_t)g; return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t g, cudaStream_t) { for (auto& f : *(Ops*)g) f(); return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) { std::memset(a, 0, sizeof *a); return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { capturing = true; recorded = new Ops; return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) { capturing = false; *g = (cudaGraph_t)recorded; return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = (cudaStream_t)1; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
}
namespace lcb {
cudaError_t launch_phase(const PhaseArgs&, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_elements(const ElemArgs&, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_roche(const ElemArgs&, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_aux(const ElemArgs&, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_flux(const FluxArgs&, int, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_epilogue(const EpiArgs& a, cudaStream_t) {
    issue([=] {
        ++runs;
        for (int64_t m = 0; m < a.nmodels; ++m) {  // results show the model table that the run saw
            for (int k = 0; k < 12; ++k) a.results[m * 12 + k] = runs + a.models[m].t0;
            for (int64_t d = 0; d < a.models[m].ndatum; ++d) a.calc[a.models[m].datum_begin + d] = 1000.0 * runs + d;
        }
    });
    return cudaSuccess;
}
int flux_blocks_per_sm() { return 4; }
cudaError_t measure_fma_peak(int, int, cudaStream_t, double*) { return cudaSuccess; }
cudaError_t launch_ecl_export(const double2*, int64_t, int64_t, int64_t, double2*, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_ecl_import(const double2*, int64_t, double2*, unsigned*, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_stream(const double*, int, double*, int*, cudaStream_t) { return cudaErrorMemoryAllocation; }
cudaError_t launch_wait_probe(long long, int*, long long*, cudaStream_t) { return cudaSuccess; }
}
#define CHECK(cond)                                                                            \
    do {                                                                                       \
        if (!(cond)) { std::printf("line %d: %s (%s)\n", __LINE__, #cond, lcb_last_error()); return 1; } \
    } while (0)
static std::string read(const char* f) {
    std::ifstream s(f, std::ios::binary);
    return std::string((std::istreambuf_iterator<char>(s)), std::istreambuf_iterator<char>());
}
static std::vector<lcb_datum> times(int n) {
    std::vector<lcb_datum> v(n);
    for (int k = 0; k < n; ++k) { v[k] = lcb_datum{}; v[k].time = k / 500.0; v[k].ferr = 0.01; v[k].weight = 1.0; v[k].ndiv = 1; }
    return v;
}
static lcb_batch* batch(lcb_ctx* C, lcb_model* m, int models, int n) {
    std::vector<const lcb_model*> ms(models, m);
    std::vector<int64_t> off;
    for (int i = 0; i <= models; ++i) off.push_back((int64_t)i * n);
    const auto d = times(models * n);
    lcb_batch* B = nullptr;
    if (lcb_batch_create(C, ms.data(), models, d.data(), off.data(), &B) != LCB_OK) return nullptr;
    return B;
}
// the batch holds run r's chi-squared and fluxes
static bool holds(lcb_batch* B, int models, int n, double chi, int r) {
    std::vector<double> c(models), f((size_t)models * n);
    if (lcb_batch_results(B, c.data(), f.data(), nullptr) != LCB_OK) return false;
    for (int m = 0; m < models; ++m) {
        if (c[m] != chi) return false;
        for (int d = 0; d < n; ++d)
            if (f[(size_t)m * n + d] != 1000.0 * r + d) return false;
    }
    return true;
}
"""

# The last run's fluxes stay with the batch when a re-plan moves or regrows its tables.
RESULTS_AFTER_REPLAN = r"""
int main(int, char** argv) {
    lcb_ctx* C; lcb_model* m;
    CHECK(lcb_ctx_create(0, &C) == LCB_OK && lcb_model_parse(read(argv[1]).c_str(), &m) == LCB_OK);
    const int n = 700;
    lcb_batch* B = batch(C, m, 3, n);
    CHECK(B && lcb_batch_run(B, 0) == LCB_OK && holds(B, 3, n, 1, 1));
    for (int chunks : {8, 1, 0}) {
        CHECK(lcb_batch_set_tuning(B, chunks, 0, 0) == LCB_OK);
        CHECK(holds(B, 3, n, 1, 1));
    }
    CHECK(lcb_batch_run(B, 0) == LCB_OK && holds(B, 3, n, 2, 2));
    const char* name = "rdisc2";
    for (double outer : {0.2, 0.4, 0.1}) {  // more and fewer elements of the disc: the arena grows, tables move
        const double v[3] = {outer, outer, outer};
        CHECK(lcb_batch_set_params(B, &name, 1, v) == LCB_OK);
        CHECK(holds(B, 3, n, 2, 2));
    }
    CHECK(lcb_batch_run(B, 1) == LCB_OK && holds(B, 3, n, 3, 3));
    lcb_batch_destroy(B);
    lcb_ctx_destroy(C);
    std::printf("ok\n");
    return 0;
}
"""

# lcb_light_curve_noalloc on a fresh context allocates nothing, whatever the size of its results.
NOALLOC = r"""
int main(int, char** argv) {
    lcb_ctx* C; lcb_model* m;
    CHECK(lcb_ctx_create(0, &C) == LCB_OK && lcb_model_parse(read(argv[1]).c_str(), &m) == LCB_OK);
    int r = 0;
    for (int n : {500, 20000, 60000}) {
        const auto d = times(n);
        std::vector<double> f(n);
        lcb_result res;
        auto before = calls;
        CHECK(lcb_light_curve_noalloc(C, m, d.data(), n, 0, 1, f.data(), &res) == LCB_OK);
        for (const char* name : {"cudaMalloc", "cudaMallocHost", "cudaFree", "cudaFreeHost", "cudaEventCreate"})
            CHECK(calls[name] == before[name]);
        ++r;
        CHECK(res.chisq == r && f[0] == 1000.0 * r && f[n - 1] == 1000.0 * r + n - 1);
    }
    lcb_ctx_destroy(C);
    std::printf("ok\n");
    return 0;
}
"""

# lcb_light_curve_noalloc refuses a call for the scratch that its limit counts, and for nothing else:
# discs from inside the limit to beyond it, in steps of less than its slack.
NOALLOC_LIMIT = r"""
int main(int, char** argv) {
    lcb_ctx* C; lcb_model* m;
    CHECK(lcb_ctx_create(0, &C) == LCB_OK && lcb_model_parse(read(argv[1]).c_str(), &m) == LCB_OK);
    const auto d = times(10);
    double f[10];
    int taken = 0, refused = 0;
    for (int nrad = 180; nrad <= 380; ++nrad) {
        CHECK(lcb_model_set_comp(m, "nrad", std::to_string(nrad).c_str()) == LCB_OK);
        const int rc = lcb_light_curve_noalloc(C, m, d.data(), 10, 0, 0, f, nullptr);
        if (rc == LCB_OK) {
            CHECK(refused == 0);
            ++taken;
        } else {
            const std::string msg = lcb_last_error();
            CHECK(rc == LCB_ERR_INVALID && msg.find("need ") != std::string::npos);
            CHECK(std::atoll(msg.c_str() + msg.find("need ") + 5) > (long long)LCB_NOALLOC_ARENA_BYTES);
            ++refused;
        }
    }
    CHECK(taken > 5 && refused > 5);
    lcb_ctx_destroy(C);
    std::printf("ok\n");
    return 0;
}
"""

# New parameters whose upload fails: the batch runs on neither the old nor the new ones until it is set again.
FAILED_UPLOAD = r"""
int main(int, char** argv) {
    lcb_ctx* C; lcb_model* m;
    CHECK(lcb_ctx_create(0, &C) == LCB_OK && lcb_model_parse(read(argv[1]).c_str(), &m) == LCB_OK);
    const int n = 300;
    const char* name = "t0";
    for (const char* call : {"cudaMemcpyAsync", "cudaMallocHost"}) {
        runs = 0;
        lcb_batch* B = batch(C, m, 3, n);
        CHECK(B && lcb_batch_run(B, 0) == LCB_OK && holds(B, 3, n, 1, 1));
        const double v[3] = {0.25, 0.25, 0.25};
        lcb_ctx* other = C;
        if (std::string(call) == "cudaMallocHost") {  // staging to be allocated yet: a fresh context's batch
            lcb_batch_destroy(B);
            CHECK(lcb_ctx_create(0, &other) == LCB_OK);
            fail_call = call; fail_at = calls[call] + 1;
            CHECK(batch(other, m, 3, n) == nullptr);  // the creation itself reports it
            fail_call = "";
            B = batch(other, m, 3, n);
            CHECK(B && lcb_batch_run(B, 0) == LCB_OK);
        }
        fail_call = "cudaMemcpyAsync"; fail_at = calls["cudaMemcpyAsync"] + 1;
        CHECK(lcb_batch_set_params(B, &name, 1, v) == LCB_ERR_CUDA);
        fail_call = "";
        CHECK(lcb_batch_run(B, 0) == LCB_ERR_INVALID);
        CHECK(lcb_batch_set_params(B, &name, 1, v) == LCB_OK && lcb_batch_run(B, 0) == LCB_OK);
        CHECK(holds(B, 3, n, runs + 0.25, runs));
        lcb_batch_destroy(B);
        if (other != C) lcb_ctx_destroy(other);
    }
    lcb_ctx_destroy(C);
    std::printf("ok\n");
    return 0;
}
"""


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    """Runs a driver's main on a model text."""
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    W = importlib.import_module("lcurve-rs_b200.workloads")
    d = tmp_path_factory.mktemp("host")
    src = ROOT / "lcurve-rs_b200" / "csrc"
    flags = ["g++", "-O1", "-std=c++17", "-I/usr/local/cuda/include", f"-I{src}", f"-I{ROOT / 'include'}"]
    for s in ("lcb_engine.cu", "lcb_plan.cpp", "lcb_model.cpp"):
        subprocess.run(flags + ["-x", "c++", "-c", str(src / s), "-o", str(d / (s + ".o"))], check=True)

    def run(name, main, **model):
        (d / "m.dat").write_text(W.model_text(**model))
        (d / f"{name}.cpp").write_text(FAKE + main)
        subprocess.run(flags + [str(d / f"{name}.cpp"), *map(str, d.glob("*.o")), "-o", str(d / name), "-lpthread", "-ldl"],
                       check=True)
        r = subprocess.run([str(d / name), str(d / "m.dat")], capture_output=True, text=True, timeout=300)
        assert r.returncode == 0 and r.stdout == "ok\n", (r.returncode, r.stdout, r.stderr)

    return run


DISC = dict(r2=-1.0, nlat1f=20, nlat2f=30, nlat1c=10, nlat2c=15, add_disc=1, opaque=1, nrad=20)


def test_results_outlive_a_replan(host):
    host("replan", RESULTS_AFTER_REPLAN, **DISC)


def test_noalloc_allocates_nothing(host):
    host("noalloc", NOALLOC, **DISC)


def test_noalloc_refuses_by_its_limit_alone(host):
    host("limit", NOALLOC_LIMIT, **{**DISC, "roche1": 1, "r1": 0.3, "rdisc2": 0.35, "rdisc1": 0.1})


def test_parameters_whose_upload_failed_are_not_run(host):
    host("upload", FAILED_UPLOAD, **DISC)
