"""The planner (lcb_plan.cpp: plan_batch) at the limits of what it is given, on CPU:
a model it cannot plan fails alone, whatever the rest of the batch shares with it."""
import importlib
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

DRIVER = r"""
#include <sys/resource.h>
#include <cstdio>
#include <cstdlib>
#include <fstream>
#include <string>
#include <vector>
#include "lcb_plan.h"
using namespace lcb;
int main(int argc, char** argv) {  // model file, models, how many of them with a grid beyond the memory limit
    std::ifstream f(argv[1], std::ios::binary);
    std::string text((std::istreambuf_iterator<char>(f)), std::istreambuf_iterator<char>());
    const int n = std::atoi(argv[2]), big = std::atoi(argv[3]);
    std::vector<Model> ms(n, parse_model_text(text));
    for (int i = 0; i < n; ++i) {
        ms[i].nlat1f = 20 + i;  // a table of its own for every model
        if (i >= 1 && i <= big) ms[i].nlat1f = 400000000;
    }
    std::vector<const Model*> mp;
    for (auto& m : ms) mp.push_back(&m);
    lcb_datum d{};
    d.ferr = 1.0; d.weight = 1.0; d.ndiv = 1;
    std::vector<int64_t> st(n, 0), cnt(n, 1);
    rlimit r{4000000000ull, 4000000000ull};
    if (setrlimit(RLIMIT_AS, &r)) return 3;
    Plan P;
    plan_batch(mp.data(), n, &d, st.data(), cnt.data(), 148, P);
    for (int i = 0; i < n; ++i) std::printf("%d", P.model_ok[i]);
    std::printf("\n%s\n", P.model_err[1].c_str());
    return 0;
}
"""


@pytest.fixture(scope="module")
def build(tmp_path_factory):
    """Builds a driver against the planner; returns its path and a model file's."""
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    W = importlib.import_module("lcurve-rs_b200.workloads")
    d = tmp_path_factory.mktemp("plan")
    src = ROOT / "lcurve-rs_b200" / "csrc"
    flags = ["g++", "-O1", "-std=c++17", "-I/usr/local/cuda/include", f"-I{src}"]
    for s in ("lcb_plan.cpp", "lcb_model.cpp"):
        subprocess.run(flags + ["-c", str(src / s), "-o", str(d / (s + ".o"))], check=True)
    (d / "m.dat").write_text(W.model_text(nlat1f=20, nlat2f=30, nlat1c=10, nlat2c=15))

    def make(name, text):
        (d / f"{name}.cpp").write_text(text)
        subprocess.run(flags + [str(d / f"{name}.cpp"), *map(str, d.glob("*.o")), "-o", str(d / name), "-lpthread"],
                       check=True)
        return d / name, d / "m.dat"

    return make


@pytest.fixture(scope="module")
def grids(build):
    return build("grids", DRIVER)


# tables built by one thread (few models) and by several (many), one model or two with the same huge grid
@pytest.mark.parametrize("n,big", [(3, 1), (40, 1), (40, 2)])
def test_a_grid_beyond_memory_fails_its_models_alone(grids, n, big):
    r = subprocess.run([*map(str, grids), str(n), str(big)], capture_output=True, text=True, timeout=120,
                       env={**os.environ, "MALLOC_ARENA_MAX": "1"})
    assert r.returncode == 0, r.stderr
    ok, err = r.stdout.split("\n")[:2]
    assert ok == "1" + "0" * big + "1" * (n - 1 - big)
    assert "bad_alloc" in err


SUBS = r"""
#include <cstdio>
#include <fstream>
#include <string>
#include <vector>
#include "lcb_plan.h"
using namespace lcb;
int main(int, char** argv) {
    std::ifstream f(argv[1], std::ios::binary);
    std::string text((std::istreambuf_iterator<char>(f)), std::istreambuf_iterator<char>());
    const Model m = parse_model_text(text);
    const int ndiv[4][3] = {{2, 2, 2}, {0, 0, 0}, {0, 1, 0}, {-1, -1, -1}};
    int bad = 0;
    for (int which = 0; which < 5; ++which) {  // each alone, then all together
        std::vector<const Model*> mp;
        std::vector<lcb_datum> data;
        std::vector<int64_t> st, cnt;
        for (int i = 0; i < 4; ++i) {
            if (which < 4 && i != which) continue;
            mp.push_back(&m);
            st.push_back((int64_t)data.size());
            cnt.push_back(3);
            for (int k = 0; k < 3; ++k) {
                lcb_datum d{};
                d.time = 0.1 * k; d.ferr = 1.0; d.weight = 1.0; d.ndiv = ndiv[i][k];
                data.push_back(d);
            }
        }
        PlanTuning t;
        t.datum_tables = false;
        Plan P;
        plan_batch(mp.data(), (int64_t)mp.size(), data.data(), st.data(), cnt.data(), 148, P, t);
        for (const ModelDev& M : P.models)
            for (int64_t d = 0; d < M.ndatum; ++d) {
                // first_sub reads the table for this datum: it has to have the entry
                if (M.ndiv <= 0 && M.datum_begin + d >= (int64_t)P.datum_sub0.size()) { ++bad; continue; }
                const int64_t j = first_sub(M, P.datum_sub0.data(), d);
                if (j < M.sub_begin || j + std::max(data[M.data_begin + d].ndiv, 0) > M.sub_begin + M.nsub) ++bad;
            }
    }
    std::printf("%d\n", bad);
    return 0;
}
"""


def test_every_datum_has_a_first_sub_phase(build):
    """Exposures with no sub-division (the data parser takes ndiv <= 0) among or instead of others."""
    r = subprocess.run([*map(str, build("subs", SUBS))], capture_output=True, text=True, timeout=120)
    assert r.stdout == "0\n", (r.stdout, r.stderr)
