// lcb_engine.cu — context, device buffers, batch execution and the C ABI.
//
// A batch runs as one launch sequence on the context's stream:
//   memset(aux, status, counter) -> k_phase -> k_elements -> k_roche ->
//   k_roche_open -> k_roche_chop2 -> k_aux -> k_flux -> k_curve -> k_results
// For a resident batch (lcb_batch_*) the sequence is captured once in a CUDA
// graph and replayed; between runs only the model table and the tables
// derived from it are uploaded, and the graph is rebuilt only when the
// plan's shapes change.
#include <cuda_runtime.h>
#include <nvtx3/nvToolsExt.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <functional>
#include <memory>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/lcurve_b200.h"
#include "lcb_kernels.cuh"
#include "lcb_model.h"
#include "lcb_plan.h"
#include "lcb_stream.h"

using lcb::Error;

namespace {

thread_local std::string t_last_error;

int fail(int code, const std::string& msg) {
    t_last_error = msg;
    return code;
}

// NVTX range around one host-side stage (planning, uploads, launches, result
// copies): visible in Nsight Systems / ncu's NVTX filters; header-only, inert
// when no tool is attached.
struct Range {
    explicit Range(const char* name) { nvtxRangePushA(name); }
    ~Range() { nvtxRangePop(); }
    Range(const Range&) = delete;
    Range& operator=(const Range&) = delete;
};

#define CUDA_TRY(expr)                                                                              \
    do {                                                                                            \
        cudaError_t e_ = (expr);                                                                    \
        if (e_ != cudaSuccess) throw Error(LCB_ERR_CUDA, std::string(#expr) + ": " + cudaGetErrorString(e_)); \
    } while (0)

struct DevBuf {
    void* p = nullptr;
    size_t cap = 0;
    void ensure(size_t bytes) {
        if (((bytes + 255) & ~size_t(255)) <= cap && p) return;
        if (p) cudaFree(p);
        p = nullptr;
        cap = 0;
        const size_t want = (std::max<size_t>(bytes, 1) + 255) & ~size_t(255);  // push() copies whole 256 bytes
        CUDA_TRY(cudaMalloc(&p, want));
        cap = want;
    }
    void release() {
        if (p) cudaFree(p);
        p = nullptr;
        cap = 0;
    }
    template <class T>
    T* as() const { return static_cast<T*>(p); }
};

struct View {  // a part of another buffer
    void* p = nullptr;
    template <class T>
    T* as() const { return static_cast<T*>(p); }
};

// All device storage of one planned batch, parts of one allocation (carve), but for a resident batch's
// fluxes: they have a buffer of their own, whose size no re-plan changes, since lcb_batch_results may ask
// for the last run's after the tables have moved.
struct DeviceSet {
    DevBuf arena, fluxes;
    bool resident = false;
    // the plan's tables, uploaded as one piece
    View tables, models, segs, bands, rings, eblocks, rblocks, ablocks, units, dsub0;
    // what a run clears and what it returns, so that one memset and one copy do: [egrp | aux | counter |
    // status | ecount | results | calc], a resident batch's without calc
    View work, egrp, aux, counter, status, ecount, results, calc;
    View datum, rec, pos, p64, d64, ecl, spe, spphi, sptype, spw, slfac, partial, fcomp, svda, firsthit, episum, open;
    void release() {
        arena.release();
        fluxes.release();
    }
};

// Page-locked staging of host arrays: two slots used in turn, so that one fills while the other's copy
// runs.  A slot grows with the transfers that use it, up to kSlotMax.
struct Staging {
    static constexpr size_t kSlotMax = 8u << 20;
    struct Slot {
        char* p = nullptr;
        size_t cap = 0;
        cudaEvent_t done = nullptr;  // its last copy
        bool busy = false;
    } slot[2];
    int next = 0;
    // a slot of at least `bytes` (<= kSlotMax), its last copy finished
    Slot& take(size_t bytes) {
        Slot& s = slot[next];
        next ^= 1;
        if (!s.done) CUDA_TRY(cudaEventCreateWithFlags(&s.done, cudaEventDisableTiming));
        if (s.busy) CUDA_TRY(cudaEventSynchronize(s.done));
        s.busy = false;
        if (s.cap < bytes) {
            const size_t want = std::min(std::max<size_t>(2 * bytes, 64u << 10), kSlotMax);
            if (s.p) CUDA_TRY(cudaFreeHost(s.p));
            s.p = nullptr;
            s.cap = 0;
            CUDA_TRY(cudaMallocHost((void**)&s.p, want));
            s.cap = want;
        }
        return s;
    }
    void release() {
        for (Slot& s : slot) {
            if (s.done) {
                if (s.busy) cudaEventSynchronize(s.done);
                cudaEventDestroy(s.done);
            }
            if (s.p) cudaFreeHost(s.p);
            s = Slot();
        }
    }
};

}  // namespace

struct lcb_model {
    lcb::Model m;
};

constexpr int kStages = 6;  // phase, elements, roche, aux, flux, epilogue

struct lcb_ctx {
    int device = 0;
    int num_sms = 148;
    cudaStream_t stream = nullptr;
    bool own_stream = false;
    std::mutex mu;
    std::string last_error;
    DeviceSet scratch;  // buffers of transient (non-resident) calls
    lcb::Plan plan;     // plan of the last transient call (its buffers are reused)
    Staging up, down;              // host -> device and device -> host
    std::vector<char> fetched;     // the last fetched results
    int flux_bps = 0;              // k_flux blocks that fit an SM
    cudaStream_t copy = nullptr;   // large data uploads, beside the kernels that do not need them
    cudaEvent_t entered = nullptr, copied = nullptr;  // the call's start on `stream`; the copy stream's end
    cudaEvent_t ev[kStages + 1] = {};
    int64_t h2d = 0, d2h = 0;  // bytes moved by the current / last call
    int fblink_cap = lcb::kFblinkEvalCap;  // lcb_ctx_set_search_cap
    DevBuf probe;                          // lcb_wait_probe's status words
};

struct lcb_batch {
    lcb_ctx* ctx = nullptr;
    std::vector<lcb::Model> models;
    std::vector<lcb_datum> data;
    std::vector<int64_t> start, count;
    lcb::Plan plan;
    lcb::Plan spare;  // the plan before the last lcb_batch_set_params: its storage is planned into next
    lcb::PlanTuning tune;  // launch-shape choices (lcb_batch_set_tuning); zeros = heuristics
    DeviceSet dev;
    cudaGraphExec_t graph = nullptr;
    int graph_scale = -1;
    int graph_cap = -1;  // the search cap baked into the captured graph's kernel arguments
    std::vector<int64_t> graph_key;
    bool ran = false;
    bool broken = false;  // a re-plan failed part-way: buffers may not match the plan
    double stage_ms[kStages] = {0, 0, 0, 0, 0, 0};
    std::vector<double> h_results, h_calc;
    std::vector<int> h_status;
    unsigned long long ecount[5] = {0, 0, 0, 0, 0};
};

namespace {

// Words of the per-group eclipse slot masks (one per kEclGroup elements).
size_t ecl_groups(const lcb::Plan& P) { return (size_t)((P.nelem + lcb::kEclGroup - 1) / lcb::kEclGroup); }

// Entries of the split scan's first hits: every Roche thread of a small batch; of a large one as
// many as a list that is split can have (a fixed split takes them all).
size_t first_hits(const lcb_ctx* C, const lcb::Plan& P) {
    const size_t all = std::max<size_t>(P.rblocks.size() * lcb::kRocheBlock, 1);
    return P.split_fix > 1 ? all : std::min<size_t>(all, (size_t)lcb::split_target(C->num_sms) / 2 + lcb::kRocheBlock);
}

// Doubles of the epilogue's per-block sums: four per k_curve block, one per k_results block.
size_t epi_sums(const lcb::Plan& P) { return P.models.size() * (size_t)(4 * P.curve_blocks + P.result_blocks); }

size_t pad256(size_t b) { return (b + 255) & ~size_t(255); }

// Host pieces that follow one another in a device range (each padded to 256 bytes).
struct Piece {
    const void* src;
    size_t bytes;
};

// Copies pieces to dst through the page-locked slots; returns once the host memory has been read.
void push(lcb_ctx* C, cudaStream_t s, void* dst, const std::vector<Piece>& pieces) {
    size_t total = 0;
    for (const Piece& p : pieces) {
        total += pad256(p.bytes);
        C->h2d += (int64_t)p.bytes;
    }
    size_t k = 0, in = 0;  // piece, and how much of it is done
    for (size_t at = 0; at < total;) {
        const size_t len = std::min(total - at, Staging::kSlotMax);
        Staging::Slot& slot = C->up.take(len);
        for (size_t o = 0; o < len;) {
            const Piece& p = pieces[k];
            const size_t n = std::min(pad256(p.bytes) - in, len - o);
            if (in < p.bytes) lcb::host_copy(slot.p + o, (const char*)p.src + in, std::min(n, p.bytes - in));
            o += n;
            in += n;
            if (in == pad256(p.bytes)) {
                ++k;
                in = 0;
            }
        }
        CUDA_TRY(cudaMemcpyAsync((char*)dst + at, slot.p, len, cudaMemcpyHostToDevice, s));
        slot.busy = true;
        CUDA_TRY(cudaEventRecord(slot.done, s));
        at += len;
    }
}

// The plan's tables in upload order, and their device views.
std::vector<Piece> plan_tables(const lcb::Plan& P, DeviceSet& D, void* base) {
    std::vector<Piece> pieces;
    size_t off = 0;
    auto add = [&](View& v, const auto& t) {
        v.p = base ? (char*)base + off : nullptr;
        pieces.push_back({t.data(), t.size() * sizeof(t[0])});
        off += pad256(pieces.back().bytes);
    };
    add(D.models, P.models);
    add(D.segs, P.segs);
    add(D.bands, P.bands);
    add(D.rings, P.rings);
    add(D.eblocks, P.eblocks);
    add(D.rblocks, P.rblocks);
    add(D.ablocks, P.ablocks);
    add(D.units, P.units);
    add(D.dsub0, P.datum_sub0);
    return pieces;
}

// Sizes of the work buffer's parts, in its order.
std::vector<size_t> work_sizes(const lcb::Plan& P, const DeviceSet& D) {
    const size_t nm = P.models.size();
    return {ecl_groups(P) * sizeof(unsigned), nm * lcb::kNumAux * sizeof(double), sizeof(int) * 4, nm * sizeof(int),
            sizeof(unsigned long long) * 8, nm * 12 * sizeof(double), D.resident ? 0 : P.ndatum * sizeof(double)};
}
void work_views(const lcb::Plan& P, DeviceSet& D, void* base) {
    View* v[7] = {&D.egrp, &D.aux, &D.counter, &D.status, &D.ecount, &D.results, &D.calc};
    size_t off = 0, k = 0;
    for (size_t b : work_sizes(P, D)) {
        v[k++]->p = base ? (char*)base + off : nullptr;
        off += pad256(b);
    }
    if (D.resident) D.calc.p = D.fluxes.p;
}
size_t total_of(const std::vector<size_t>& v) {
    size_t t = 0;
    for (size_t b : v) t += pad256(b);
    return t;
}

// Lays out every buffer of a planned batch from `base` on (nullptr only measures).  Returns the bytes
// used; `counted`, if given, those that lcb_light_curve_noalloc's limit counts.
size_t carve(const lcb_ctx* C, const lcb::Plan& P, void* base, DeviceSet& D, size_t* counted = nullptr) {
    size_t off = 0;
    auto take = [&](View& v, size_t bytes) {
        v.p = base ? (char*)base + off : nullptr;
        off += pad256(bytes);
    };
    size_t tables = 0;
    for (const Piece& p : plan_tables(P, D, nullptr)) tables += pad256(p.bytes);
    take(D.tables, tables);
    plan_tables(P, D, D.tables.p);
    take(D.work, total_of(work_sizes(P, D)));
    work_views(P, D, D.work.p);
    take(D.datum, P.data_count * sizeof(lcb_datum));
    take(D.rec, P.nelem * sizeof(float4));
    take(D.pos, P.nelem * sizeof(float4));
    take(D.p64, P.nelem * sizeof(double4));
    take(D.d64, P.nelem * sizeof(double4));
    take(D.ecl, P.nelem * lcb::kMaxEcl * sizeof(double2));
    take(D.spe, P.nsub * sizeof(float4));
    take(D.spphi, P.nsub * sizeof(double));
    take(D.sptype, P.nsub * sizeof(int8_t));
    take(D.spw, P.nsub * sizeof(double));
    take(D.slfac, P.ndatum * sizeof(double));
    take(D.partial, P.npartial * sizeof(double));
    const size_t ncomp = P.any_iscale ? (size_t)P.ndatum * 5 : 1;
    take(D.fcomp, ncomp * sizeof(double));
    take(D.svda, ncomp * sizeof(double));
    // the above and four bytes per Roche thread of a split search
    if (counted) *counted = off + pad256((P.roche_split > 1 ? P.rblocks.size() * lcb::kRocheBlock : 1) * sizeof(int));
    take(D.firsthit, first_hits(C, P) * sizeof(int));
    take(D.open, std::max<size_t>(P.rblocks.size() * lcb::kRocheBlock, 1) * sizeof(unsigned));
    take(D.episum, epi_sums(P) * sizeof(double));
    return off;
}

// Device arrays and tables of a plan (not the data).
void upload_plan(lcb_ctx* C, DeviceSet& D, const lcb::Plan& P) {
    D.arena.ensure(carve(C, P, nullptr, D));
    carve(C, P, D.arena.p, D);
    push(C, C->stream, D.tables.p, plan_tables(P, D, D.tables.p));
}

// The data of a plan, on the context's stream; large ones on the copy stream, which `joined` (the
// caller, before the first kernel that reads them) makes the context's stream wait for.
constexpr size_t kCopyBeside = 1u << 20;
void upload_data(lcb_ctx* C, DeviceSet& D, const lcb::Plan& P, const lcb_datum* data, bool beside = false) {
    const lcb_datum* src = data + P.data_first;
    const size_t bytes = P.data_count * sizeof(lcb_datum);
    if (!bytes) return;
    const bool other = beside && bytes >= kCopyBeside;
    cudaStream_t s = C->stream;
    if (other) {
        if (!C->copy) CUDA_TRY(cudaStreamCreateWithFlags(&C->copy, cudaStreamNonBlocking));
        if (!C->copied) CUDA_TRY(cudaEventCreateWithFlags(&C->copied, cudaEventDisableTiming));
        s = C->copy;
        CUDA_TRY(cudaStreamWaitEvent(s, C->entered, 0));  // whatever an earlier call left on the stream is done
    }
    cudaPointerAttributes at{};
    if (bytes >= kCopyBeside && cudaPointerGetAttributes(&at, src) == cudaSuccess && at.type == cudaMemoryTypeHost) {
        CUDA_TRY(cudaMemcpyAsync(D.datum.p, src, bytes, cudaMemcpyHostToDevice, s));  // page-locked already
        C->h2d += (int64_t)bytes;
    } else {
        (void)cudaGetLastError();
        push(C, s, D.datum.p, {{src, bytes}});
    }
    if (other) {
        CUDA_TRY(cudaEventRecord(C->copied, s));
        CUDA_TRY(cudaStreamWaitEvent(C->stream, C->copied, 0));
    }
}

// Parts of the launch sequence: the element stage (grids, continuum, eclipses:
// k_elements, k_roche) and the rest (k_phase, k_aux, k_flux, k_curve, k_results).
constexpr int kStageElements = 1, kStageRest = 2, kStagesAll = 3;

// The device launch sequence of one batch evaluation.  nblk / nrblk (>= 0)
// launch only the first nblk element blocks and nrblk Roche blocks of the
// uploaded block lists (an element slab, lcb_model_elements).  `data` runs
// before the first kernel that reads the data (k_phase).
void enqueue_run(lcb_ctx* C, DeviceSet& D, const lcb::Plan& P, int scale, int rdata, bool timed,
                 int stages = kStagesAll, int64_t nblk = -1, int64_t nrblk = -1,
                 const std::function<void()>& data = nullptr) {
    cudaStream_t s = C->stream;
    const int64_t nm = (int64_t)P.models.size();
    if (nblk < 0) nblk = (int64_t)P.eblocks.size();
    if (nrblk < 0) nrblk = (int64_t)P.rblocks.size();
    const bool rest = stages & kStageRest, elem = stages & kStageElements;
    {   // used-slot words (element stage), sums, counters and status words
        void* from = elem ? D.egrp.p : D.aux.p;
        CUDA_TRY(cudaMemsetAsync(from, 0, (char*)D.results.p - (char*)from, s));
    }
    if (timed) CUDA_TRY(cudaEventRecord(C->ev[0], s));
    const lcb::Sizes sz{P.nelem, P.nsub, P.npartial, P.ndatum, (int64_t)P.bands.size(), (int64_t)P.rings.size(), P.data_count};
    lcb::ElemArgs ea{D.models.as<lcb::ModelDev>(), D.segs.as<lcb::SegDesc>(), D.eblocks.as<lcb::ElemBlock>(),
                     D.rblocks.as<lcb::ElemBlock>(), D.ablocks.as<lcb::ElemBlock>(), D.bands.as<lcb::Band>(),
                     D.rings.as<lcb::Ring>(), D.rec.as<float4>(), D.pos.as<float4>(), D.p64.as<double4>(),
                     D.d64.as<double4>(), D.ecl.as<double2>(), D.egrp.as<unsigned>(), D.aux.as<double>(),
                     D.status.as<int>(), nblk, nrblk, (int64_t)P.ablocks.size(),
                     D.ecount.as<unsigned long long>(), D.open.as<unsigned>(), D.counter.as<unsigned>() + 1,
                     D.firsthit.as<int>(), (unsigned)first_hits(C, P), P.split_fix, P.roche_split > 1, lcb::split_target(C->num_sms),
                     C->num_sms * 5, C->fblink_cap, sz};
    if (elem) CUDA_TRY(lcb::launch_elements(ea, s));
    if (timed) CUDA_TRY(cudaEventRecord(C->ev[1], s));
    if (elem) CUDA_TRY(lcb::launch_roche(ea, s));
    if (timed) CUDA_TRY(cudaEventRecord(C->ev[2], s));
    if (!rest) return;
    CUDA_TRY(lcb::launch_aux(ea, s));
    if (timed) CUDA_TRY(cudaEventRecord(C->ev[3], s));
    if (data) data();
    lcb::PhaseArgs pa{D.models.as<lcb::ModelDev>(), D.datum.as<lcb_datum>(), D.dsub0.as<int64_t>(), nm, P.most_data,
                      D.spe.as<float4>(), D.spphi.as<double>(), D.sptype.as<int8_t>(), D.spw.as<double>(),
                      D.slfac.as<double>()};
    CUDA_TRY(lcb::launch_phase(pa, s));
    if (timed) CUDA_TRY(cudaEventRecord(C->ev[4], s));
    lcb::FluxArgs fa{D.models.as<lcb::ModelDev>(), D.units.as<lcb::FluxUnit>(), (int64_t)P.units.size(),
                     P.flux_share, D.counter.as<int>(), D.rec.as<float4>(), D.pos.as<float4>(), D.ecl.as<double2>(),
                     D.egrp.as<unsigned>(), D.spe.as<float4>(), D.spphi.as<double>(), D.sptype.as<int8_t>(), D.partial.as<double>(),
                     D.status.as<int>(), sz};
    const int bps_max = C->flux_bps;
    const int bps = P.flux_blocks_per_sm > 0 ? std::min(P.flux_blocks_per_sm, bps_max) : bps_max;
    int64_t grid = (int64_t)C->num_sms * bps;
    grid = std::min<int64_t>(grid, std::max<int64_t>((int64_t)P.units.size(), 1));
    CUDA_TRY(lcb::launch_flux(fa, (int)grid, s));
    if (timed) CUDA_TRY(cudaEventRecord(C->ev[5], s));
    lcb::EpiArgs pe{D.models.as<lcb::ModelDev>(), D.datum.as<lcb_datum>(), D.dsub0.as<int64_t>(),
                    D.spphi.as<double>(), D.spw.as<double>(), D.slfac.as<double>(), D.partial.as<double>(),
                    D.aux.as<double>(), D.status.as<int>(), scale, rdata, D.calc.as<double>(),
                    D.results.as<double>(), D.fcomp.as<double>(), D.svda.as<double>(), D.episum.as<double>(),
                    D.episum.as<double>() + nm * 4 * P.curve_blocks, nm, P.curve_blocks, P.result_blocks, P.curve_share, sz,
                    D.status.as<int>()};
    CUDA_TRY(lcb::launch_epilogue(pe, s));
    if (timed) CUDA_TRY(cudaEventRecord(C->ev[6], s));
}
// the order of the timed stages above in the reported one (phase, elements, roche, aux, flux, epilogue)
constexpr int kStageOrder[kStages] = {1, 2, 3, 0, 4, 5};

void set_device(lcb_ctx* C) { CUDA_TRY(cudaSetDevice(C->device)); }

// Copies a device range into dst through the page-locked slots (synchronises).
void pull(lcb_ctx* C, void* dst, const void* src, size_t bytes) {
    struct { Staging::Slot* s; size_t at, len; } open[2] = {};
    int n = 0;
    auto drain = [&](int k) {
        CUDA_TRY(cudaEventSynchronize(open[k].s->done));
        open[k].s->busy = false;
        lcb::host_copy((char*)dst + open[k].at, open[k].s->p, open[k].len);
        open[k].s = nullptr;
    };
    for (size_t at = 0; at < bytes; n ^= 1) {
        if (open[n].s) drain(n);
        const size_t len = std::min(bytes - at, Staging::kSlotMax);
        Staging::Slot& s = C->down.take(len);
        CUDA_TRY(cudaMemcpyAsync(s.p, (const char*)src + at, len, cudaMemcpyDeviceToHost, C->stream));
        s.busy = true;
        CUDA_TRY(cudaEventRecord(s.done, C->stream));
        open[n] = {&s, at, len};
        at += len;
    }
    for (int k = 0; k < 2; ++k, n ^= 1)
        if (open[n].s) drain(n);
    C->d2h += (int64_t)bytes;
}

// The status words, search counters and results of a run, and with `calc` (not a resident batch's) its
// fluxes: one copy, through the page-locked slots or (staged = false: they may have to be allocated) straight
// into pageable memory.
void fetch_results(lcb_ctx* C, DeviceSet& D, const lcb::Plan& P, std::vector<double>& res, std::vector<double>* calc,
                   std::vector<int>* status, unsigned long long* ecount = nullptr, bool staged = true) {
    auto get = [&](void* dst, const void* src, size_t bytes) {
        if (staged) return pull(C, dst, src, bytes);
        CUDA_TRY(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, C->stream));
        CUDA_TRY(cudaStreamSynchronize(C->stream));
        C->d2h += (int64_t)bytes;
    };
    const int64_t nm = (int64_t)P.models.size();
    const char* base = (const char*)D.status.p;
    const size_t head = (const char*)D.results.p + pad256(nm * 12 * sizeof(double)) - base;
    const size_t tail = calc ? P.ndatum * sizeof(double) : 0;
    std::vector<char>& h = C->fetched;
    const bool one = head + tail <= Staging::kSlotMax;  // else the fluxes straight into their vector
    h.resize(head + (one ? tail : 0));
    get(h.data(), base, h.size());
    auto part = [&](const View& v) { return h.data() + ((const char*)v.p - base); };
    res.resize(nm * 12);
    std::memcpy(res.data(), part(D.results), nm * 12 * sizeof(double));
    if (status) {
        status->resize(nm);
        std::memcpy(status->data(), part(D.status), nm * sizeof(int));
    }
    if (ecount) std::memcpy(ecount, part(D.ecount), 5 * sizeof(unsigned long long));
    if (calc) {
        calc->resize(P.ndatum);
        if (one) std::memcpy(calc->data(), part(D.calc), tail);
        else get(calc->data(), D.calc.p, tail);
    }
    CUDA_TRY(cudaStreamSynchronize(C->stream));
}

// Device checks that fail a whole call (as opposed to one model's NaN): in the
// LCURVE_DEBUG_BOUNDS build an index out of range.
void check_device_status(int st) {
    if (st & lcb::kStatusBounds) throw Error(LCB_ERR_DEVICE_CHECK, "a device-side bounds check failed");
}

void fill_result(const double* r, lcb_result* out) {
    out->wdwarf = r[0]; out->chisq = r[1]; out->wnok = r[2]; out->logg1 = r[3]; out->logg2 = r[4];
    out->rv1 = r[5]; out->rv2 = r[6];
    for (int k = 0; k < 5; ++k) out->sfac[k] = r[7 + k];
}


// The engine's plans carry no per-datum tables where a model's data are sub-divided alike.
lcb::PlanTuning engine_tuning() {
    lcb::PlanTuning t;
    t.datum_tables = false;
    return t;
}

// A transient evaluation on the context's scratch buffers.
void run_transient(lcb_ctx* C, const lcb::Model* const* models, int64_t n, const lcb_datum* data,
                   const int64_t* start, const int64_t* count, int scale, int rdata, std::vector<double>& res,
                   std::vector<double>* calc, lcb::Plan& P, std::vector<int>& st) {
    {
        Range r("lcb plan");
        lcb::plan_batch(models, n, data, start, count, C->num_sms, P, engine_tuning());
    }
    {
        Range r("lcb upload");
        upload_plan(C, C->scratch, P);
        if (P.data_count * sizeof(lcb_datum) >= kCopyBeside) {
            if (!C->entered) CUDA_TRY(cudaEventCreateWithFlags(&C->entered, cudaEventDisableTiming));
            CUDA_TRY(cudaEventRecord(C->entered, C->stream));
        }
    }
    {
        Range r("lcb launch");  // the data follow while the kernels that do not need them run
        enqueue_run(C, C->scratch, P, scale, rdata, false, kStagesAll, -1, -1,
                    [&] { upload_data(C, C->scratch, P, data, true); });
    }
    {
        Range r("lcb results");
        fetch_results(C, C->scratch, P, res, calc, &st);
    }
    for (int64_t i = 0; i < n; ++i)
        check_device_status(st[i]);
}

template <class F>
int guarded(lcb_ctx* C, F&& f) {
    try {
        if (C) {
            std::lock_guard<std::mutex> g(C->mu);
            set_device(C);
            (void)cudaGetLastError();  // a stale non-sticky error must not be blamed on this call
            C->h2d = C->d2h = 0;
            f();
        } else {
            f();
        }
        return LCB_OK;
    } catch (const Error& e) {
        if (C) C->last_error = e.what();
        return fail(e.code, e.what());
    } catch (const std::bad_alloc&) {
        if (C) C->last_error = "out of host memory";
        return fail(LCB_ERR_INVALID, "out of host memory");
    } catch (const std::exception& e) {
        if (C) C->last_error = e.what();
        return fail(LCB_ERR_INVALID, e.what());
    }
}

}  // namespace

// ===========================================================================
// C ABI
// ===========================================================================
extern "C" {

const char* lcb_version(void) { return "lcurve-b200 0.1.0 (sm_100a)"; }
const char* lcb_last_error(void) { return t_last_error.c_str(); }

int lcb_device_count(int* count) {
    if (!count) return fail(LCB_ERR_INVALID, "null pointer");
    int n = 0;
    cudaError_t e = cudaGetDeviceCount(&n);
    if (e != cudaSuccess) { *count = 0; return fail(LCB_ERR_NO_DEVICE, cudaGetErrorString(e)); }
    *count = n;
    return LCB_OK;
}

int lcb_ctx_create(int device, lcb_ctx** out) {
    if (!out) return fail(LCB_ERR_INVALID, "null pointer");
    *out = nullptr;
    int n = 0;
    if (cudaGetDeviceCount(&n) != cudaSuccess || n <= 0) return fail(LCB_ERR_NO_DEVICE, "no CUDA device");
    if (device < 0 || device >= n) return fail(LCB_ERR_NO_DEVICE, "device id out of range");
    auto C = std::make_unique<lcb_ctx>();
    C->device = device;
    int rc = guarded(nullptr, [&] {
        CUDA_TRY(cudaSetDevice(device));
        cudaDeviceProp prop;
        CUDA_TRY(cudaGetDeviceProperties(&prop, device));
        if (prop.major < 10) throw Error(LCB_ERR_NO_DEVICE, "this library is built for sm_100a (B200)");
        C->num_sms = prop.multiProcessorCount;
        // fails here, not later, if the sm_100a image cannot load on this device
        C->flux_bps = lcb::flux_blocks_per_sm();
        if (C->flux_bps <= 0) throw Error(LCB_ERR_NO_DEVICE, "kernel image not loadable");
        CUDA_TRY(cudaStreamCreateWithFlags(&C->stream, cudaStreamNonBlocking));
        C->own_stream = true;
        for (auto& e : C->ev) CUDA_TRY(cudaEventCreate(&e));
    });
    if (rc != LCB_OK) return rc;
    *out = C.release();
    return LCB_OK;
}

void lcb_ctx_destroy(lcb_ctx* C) {
    if (!C) return;
    cudaSetDevice(C->device);
    if (C->stream) cudaStreamSynchronize(C->stream);
    if (C->copy) cudaStreamSynchronize(C->copy);
    C->scratch.release();
    C->probe.release();
    C->up.release();
    C->down.release();
    if (C->entered) cudaEventDestroy(C->entered);
    if (C->copied) cudaEventDestroy(C->copied);
    if (C->copy) cudaStreamDestroy(C->copy);
    for (auto& e : C->ev)
        if (e) cudaEventDestroy(e);
    if (C->own_stream && C->stream) cudaStreamDestroy(C->stream);
    delete C;
}

int lcb_ctx_set_stream(lcb_ctx* C, void* stream) {
    if (!C) return fail(LCB_ERR_INVALID, "null context");
    return guarded(C, [&] {
        if (C->own_stream && C->stream) {
            CUDA_TRY(cudaStreamSynchronize(C->stream));
            CUDA_TRY(cudaStreamDestroy(C->stream));
        }
        C->own_stream = stream == nullptr;
        if (stream) C->stream = (cudaStream_t)stream;
        else CUDA_TRY(cudaStreamCreateWithFlags(&C->stream, cudaStreamNonBlocking));
    });
}

const char* lcb_ctx_last_error(const lcb_ctx* C) { return C ? C->last_error.c_str() : "null context"; }

// ---- models -----------------------------------------------------------------
int lcb_model_load(const char* path, lcb_model** out) {
    if (!path || !out) return fail(LCB_ERR_INVALID, "null pointer");
    return guarded(nullptr, [&] { *out = new lcb_model{lcb::load_model_file(path)}; });
}
int lcb_model_parse(const char* text, lcb_model** out) {
    if (!text || !out) return fail(LCB_ERR_INVALID, "null pointer");
    return guarded(nullptr, [&] { *out = new lcb_model{lcb::parse_model_text(text)}; });
}
int lcb_model_clone(const lcb_model* m, lcb_model** out) {
    if (!m || !out) return fail(LCB_ERR_INVALID, "null pointer");
    return guarded(nullptr, [&] { *out = new lcb_model{m->m}; });
}
void lcb_model_destroy(lcb_model* m) { delete m; }

int lcb_model_set_param(lcb_model* m, const char* name, double value) {
    if (!m || !name) return fail(LCB_ERR_INVALID, "null pointer");
    int i = lcb::phys_index(name);
    if (i < 0) return fail(LCB_ERR_UNKNOWN_PARAM, std::string("unknown parameter: '") + name + "'");
    m->m.p[i].value = value;
    return LCB_OK;
}
int lcb_model_get_param(const lcb_model* m, const char* name, double* value) {
    if (!m || !name || !value) return fail(LCB_ERR_INVALID, "null pointer");
    int i = lcb::phys_index(name);
    if (i < 0) return fail(LCB_ERR_UNKNOWN_PARAM, std::string("unknown parameter: '") + name + "'");
    *value = m->m.p[i].value;
    return LCB_OK;
}
int lcb_model_get_pparam(const lcb_model* m, const char* name, double* value, double* range, double* dstep,
                         int* vary, int* defined) {
    if (!m || !name) return fail(LCB_ERR_INVALID, "null pointer");
    int i = lcb::phys_index(name);
    if (i < 0) return fail(LCB_ERR_UNKNOWN_PARAM, std::string("unknown parameter: '") + name + "'");
    const lcb::Pparam& p = m->m.p[i];
    if (value) *value = p.value;
    if (range) *range = p.range;
    if (dstep) *dstep = p.dstep;
    if (vary) *vary = p.vary;
    if (defined) *defined = p.defined;
    return LCB_OK;
}
int lcb_model_set_pparam(lcb_model* m, const char* name, const double* value, const double* range,
                         const double* dstep, const int* vary) {
    if (!m || !name) return fail(LCB_ERR_INVALID, "null pointer");
    int i = lcb::phys_index(name);
    if (i < 0) return fail(LCB_ERR_UNKNOWN_PARAM, std::string("unknown parameter: '") + name + "'");
    lcb::Pparam& p = m->m.p[i];
    if (value) p.value = *value;
    if (range) p.range = *range;
    if (dstep) p.dstep = *dstep;
    if (vary) p.vary = *vary != 0;
    return LCB_OK;
}
int lcb_model_set_comp(lcb_model* m, const char* name, const char* value) {
    if (!m || !name || !value) return fail(LCB_ERR_INVALID, "null pointer");
    return guarded(nullptr, [&] { lcb::set_comp_param(m->m, name, value); });
}
int lcb_model_get_comp(const lcb_model* m, const char* name, char* buf, int buflen) {
    if (!m || !name || !buf || buflen <= 0) return fail(LCB_ERR_INVALID, "null pointer");
    return guarded(nullptr, [&] {
        std::string s = lcb::get_comp_param(m->m, name);
        std::snprintf(buf, (size_t)buflen, "%s", s.c_str());
    });
}
const char* lcb_param_name(int i) { return lcb::phys_name(i); }

// ---- data -------------------------------------------------------------------
int lcb_read_data(const char* path, lcb_datum** out, int64_t* n) {
    if (!path || !out || !n) return fail(LCB_ERR_INVALID, "null pointer");
    return guarded(nullptr, [&] {
        std::vector<lcb_datum> d = lcb::read_data_file(path);
        lcb_datum* p = (lcb_datum*)std::malloc(std::max<size_t>(d.size(), 1) * sizeof(lcb_datum));
        if (!p) throw std::bad_alloc();
        if (!d.empty()) std::memcpy(p, d.data(), d.size() * sizeof(lcb_datum));
        *out = p;
        *n = (int64_t)d.size();
    });
}
void lcb_free_data(lcb_datum* d) { std::free(d); }

// ---- evaluation ---------------------------------------------------------------
int lcb_light_curve(lcb_ctx* C, const lcb_model* model, const lcb_datum* data, int64_t n, int scale, int rdata,
                    double* calc_out, lcb_result* res_out) {
    if (!C || !model || (!data && n > 0) || !calc_out) return fail(LCB_ERR_INVALID, "null pointer");
    if (n <= 0) return fail(LCB_ERR_EMPTY, "No data points");
    return guarded(C, [&] {
        const lcb::Model* mp = &model->m;
        int64_t st = 0, cnt = n;
        std::vector<double> res, calc;
        std::vector<int> status;
        lcb::Plan P;
        run_transient(C, &mp, 1, data, &st, &cnt, scale, rdata, res, &calc, P, status);
        if (!P.model_ok[0]) throw Error(LCB_ERR_MODEL, P.model_err[0]);
        if (status[0] & lcb::kStatusIterCap)
            throw Error(LCB_ERR_DEVICE_CHECK, "a device-side iteration cap tripped for this model");
        std::memcpy(calc_out, calc.data(), n * sizeof(double));
        if (res_out) fill_result(res.data(), res_out);
    });
}

int lcb_model_grid(lcb_ctx* C, const lcb_model* model, int which, int64_t* n, double* posn, double* dirn,
                   float* area, float* gravity, float* flux, double* ecl) {
    if (!C || !model || !n || which < 0 || which > 6) return fail(LCB_ERR_INVALID, "bad arguments");
    return guarded(C, [&] {
        const lcb::Model* mp = &model->m;
        lcb_datum d{};
        d.time = 0.0; d.expose = 0.0; d.ferr = 1.0; d.weight = 1.0; d.ndiv = 1;
        int64_t st = 0, cnt = 1;
        lcb::Plan P;
        lcb::plan_batch(&mp, 1, &d, &st, &cnt, C->num_sms, P, engine_tuning());
        if (!P.model_ok[0]) throw Error(LCB_ERR_MODEL, P.model_err[0]);
        const lcb::SegDesc* g = nullptr;
        for (const auto& sg : P.segs) {
            bool star = sg.kind == lcb::SEG_STAR1 || sg.kind == lcb::SEG_STAR2;
            int k = sg.kind == lcb::SEG_STAR1 ? 1 : 2;
            if (star && which <= 3) {
                bool fine = which <= 1;
                if ((which % 2 == 0 ? 1 : 2) != k) continue;
                if (sg.role == lcb::ROLE_BOTH || (sg.role == lcb::ROLE_FINE) == fine) { g = &sg; break; }
            } else if ((which == 4 && sg.kind == lcb::SEG_DISC) || (which == 5 && sg.kind == lcb::SEG_EDGE) ||
                       (which == 6 && sg.kind == lcb::SEG_SPOT)) {
                g = &sg;
                break;
            }
        }
        *n = g ? g->count : 0;
        if (!g || !posn) return;
        upload_plan(C, C->scratch, P);
        upload_data(C, C->scratch, P, &d);
        enqueue_run(C, C->scratch, P, 0, 0, false);
        CUDA_TRY(cudaStreamSynchronize(C->stream));
        std::vector<double4> p64(g->count), d64(g->count);
        std::vector<float4> rec(g->count);
        std::vector<double2> e(g->count * lcb::kMaxEcl);
        CUDA_TRY(cudaMemcpy(p64.data(), C->scratch.p64.as<double4>() + g->first, g->count * sizeof(double4),
                            cudaMemcpyDeviceToHost));
        CUDA_TRY(cudaMemcpy(d64.data(), C->scratch.d64.as<double4>() + g->first, g->count * sizeof(double4),
                            cudaMemcpyDeviceToHost));
        CUDA_TRY(cudaMemcpy(rec.data(), C->scratch.rec.as<float4>() + g->first, g->count * sizeof(float4),
                            cudaMemcpyDeviceToHost));
        for (int k = 0; k < lcb::kMaxEcl; ++k)  // slot-major on the device
            CUDA_TRY(cudaMemcpy(e.data() + k * g->count, C->scratch.ecl.as<double2>() + k * P.nelem + g->first,
                                g->count * sizeof(double2), cudaMemcpyDeviceToHost));
        for (int64_t i = 0; i < g->count; ++i) {
            posn[3 * i] = p64[i].x; posn[3 * i + 1] = p64[i].y; posn[3 * i + 2] = p64[i].z;
            if (dirn) { dirn[3 * i] = d64[i].x; dirn[3 * i + 1] = d64[i].y; dirn[3 * i + 2] = d64[i].z; }
            if (area) area[i] = (float)p64[i].w;
            if (gravity) gravity[i] = (float)d64[i].w;
            if (flux) flux[i] = rec[i].w;
            if (ecl)
                for (int k = 0; k < lcb::kMaxEcl; ++k) {
                    ecl[8 * i + 2 * k] = e[k * g->count + i].x;
                    ecl[8 * i + 2 * k + 1] = e[k * g->count + i].y;
                }
        }
    });
}

// Element records of one model exchanged across devices (a model split into element slabs):
// five device arrays in the engine's own element order; the eclipse slots element-major
// (kMaxEcl pairs per element), converted from and to the engine's slot-major array.
static const size_t kElemBytes[4] = {sizeof(float4), sizeof(float4), sizeof(double4), sizeof(double4)};

int lcb_model_elements(lcb_ctx* C, const lcb_model* model, int64_t first, int64_t count, void* rec_dev,
                       void* pos_dev, void* p64_dev, void* d64_dev, void* ecl_dev, int64_t* total) {
    if (!C || !model || !total || first < 0 || count < 0) return fail(LCB_ERR_INVALID, "bad arguments");
    return guarded(C, [&] {
        const lcb::Model* mp = &model->m;
        lcb_datum d{};
        d.ferr = 1.0; d.weight = 1.0; d.ndiv = 1;
        int64_t st = 0, cnt = 1;
        lcb::Plan& P = C->plan;
        lcb::plan_batch(&mp, 1, &d, &st, &cnt, C->num_sms, P, engine_tuning());
        if (!P.model_ok[0]) throw Error(LCB_ERR_MODEL, P.model_err[0]);
        *total = P.nelem;
        if (!rec_dev) return;
        if (!pos_dev || !p64_dev || !d64_dev || !ecl_dev) throw Error(LCB_ERR_INVALID, "null device array");
        if (first + count > P.nelem) throw Error(LCB_ERR_INVALID, "element range beyond the model's elements");
        if (count == 0) return;
        // the element blocks and Roche blocks that touch [first, first + count): every Roche
        // block lies inside an element block, so the slab's elements are all computed
        const int64_t last = first + count;
        auto touches = [&](const lcb::ElemBlock& b, int64_t width) {
            const int64_t e0 = P.segs[b.seg].first + b.offset;
            return e0 < last && e0 + width > first;
        };
        std::vector<lcb::ElemBlock> eb, rb;
        for (const auto& b : P.eblocks)
            if (touches(b, lcb::kElemThreads)) eb.push_back(b);
        for (const auto& b : P.rblocks)
            if (touches(b, lcb::kRocheBlock)) rb.push_back(b);
        upload_plan(C, C->scratch, P);
        DeviceSet& D = C->scratch;
        if (!eb.empty())
            CUDA_TRY(cudaMemcpyAsync(D.eblocks.p, eb.data(), eb.size() * sizeof(lcb::ElemBlock),
                                     cudaMemcpyHostToDevice, C->stream));
        if (!rb.empty())
            CUDA_TRY(cudaMemcpyAsync(D.rblocks.p, rb.data(), rb.size() * sizeof(lcb::ElemBlock),
                                     cudaMemcpyHostToDevice, C->stream));
        enqueue_run(C, D, P, 0, 0, false, kStageElements, (int64_t)eb.size(), (int64_t)rb.size());
        void* dst[4] = {rec_dev, pos_dev, p64_dev, d64_dev};
        const void* src[4] = {D.rec.p, D.pos.p, D.p64.p, D.d64.p};
        for (int k = 0; k < 4; ++k)
            CUDA_TRY(cudaMemcpyAsync(dst[k], (const char*)src[k] + first * kElemBytes[k], count * kElemBytes[k],
                                     cudaMemcpyDeviceToDevice, C->stream));
        CUDA_TRY(lcb::launch_ecl_export(D.ecl.as<double2>(), P.nelem, first, count, (double2*)ecl_dev, C->stream));
        int status = 0;
        CUDA_TRY(cudaMemcpyAsync(&status, D.status.p, sizeof(int), cudaMemcpyDeviceToHost, C->stream));
        CUDA_TRY(cudaStreamSynchronize(C->stream));
        check_device_status(status);
        if (status & lcb::kStatusIterCap)
            throw Error(LCB_ERR_DEVICE_CHECK, "a device-side iteration cap tripped for this model");
    });
}

int lcb_light_curve_elements(lcb_ctx* C, const lcb_model* model, const lcb_datum* data, int64_t n, int scale,
                             int rdata, const void* rec_dev, const void* pos_dev, const void* p64_dev,
                             const void* d64_dev, const void* ecl_dev, double* calc_out, lcb_result* res_out) {
    if (!C || !model || (!data && n > 0) || !calc_out || !rec_dev || !pos_dev || !p64_dev || !d64_dev || !ecl_dev)
        return fail(LCB_ERR_INVALID, "null pointer");
    if (n <= 0) return fail(LCB_ERR_EMPTY, "No data points");
    return guarded(C, [&] {
        const lcb::Model* mp = &model->m;
        int64_t st = 0, cnt = n;
        lcb::Plan& P = C->plan;
        lcb::plan_batch(&mp, 1, data, &st, &cnt, C->num_sms, P, engine_tuning());
        if (!P.model_ok[0]) throw Error(LCB_ERR_MODEL, P.model_err[0]);
        upload_plan(C, C->scratch, P);
        upload_data(C, C->scratch, P, data);
        DeviceSet& D = C->scratch;
        const void* src[4] = {rec_dev, pos_dev, p64_dev, d64_dev};
        void* dst[4] = {D.rec.p, D.pos.p, D.p64.p, D.d64.p};
        for (int k = 0; k < 4; ++k)
            if (P.nelem)
                CUDA_TRY(cudaMemcpyAsync(dst[k], src[k], P.nelem * kElemBytes[k], cudaMemcpyDeviceToDevice, C->stream));
        CUDA_TRY(cudaMemsetAsync(D.egrp.p, 0, ecl_groups(P) * sizeof(unsigned), C->stream));
        CUDA_TRY(lcb::launch_ecl_import((const double2*)ecl_dev, P.nelem, D.ecl.as<double2>(), D.egrp.as<unsigned>(),
                                        C->stream));
        enqueue_run(C, D, P, scale, rdata, false, kStageRest);
        std::vector<double> res, calc;
        std::vector<int> status;
        fetch_results(C, D, P, res, &calc, &status);
        check_device_status(status[0]);
        std::memcpy(calc_out, calc.data(), n * sizeof(double));
        if (res_out) fill_result(res.data(), res_out);
    });
}

int lcb_chisq_batch(lcb_ctx* C, const lcb_model* base, const lcb_datum* data, int64_t n, const char* const* names,
                    int ndim, const double* values, int64_t nsets, int scale, double* chisq_out) {
    if (!C || !base || !data || !names || !values || !chisq_out) return fail(LCB_ERR_INVALID, "null pointer");
    if (ndim <= 0 || nsets < 0) return fail(LCB_ERR_INVALID, "ndim must be > 0");
    if (n <= 0) return fail(LCB_ERR_EMPTY, "No data points");
    return guarded(C, [&] {
        std::vector<int> idx(ndim);
        for (int j = 0; j < ndim; ++j) idx[j] = lcb::phys_index(names[j]);  // unknown names are ignored
        std::vector<lcb::Model> ms(nsets, base->m);
        std::vector<const lcb::Model*> mp(nsets);
        for (int64_t i = 0; i < nsets; ++i) {
            for (int j = 0; j < ndim; ++j)
                if (idx[j] >= 0) ms[i].p[idx[j]].value = values[i * ndim + j];
            mp[i] = &ms[i];
        }
        if (nsets == 0) return;
        std::vector<int64_t> st(nsets, 0), cnt(nsets, n);
        std::vector<double> res;
        std::vector<int> status;
        lcb::Plan& P = C->plan;
        run_transient(C, mp.data(), nsets, data, st.data(), cnt.data(), scale, 1, res, nullptr, P, status);
        for (int64_t i = 0; i < nsets; ++i) chisq_out[i] = P.model_ok[i] ? res[i * 12 + 1] : NAN;
    });
}

int lcb_chisq_batch_ragged(lcb_ctx* C, const lcb_model* const* models, int64_t nmodels, const lcb_datum* data,
                           const int64_t* offsets, int scale, double* chisq_out, double* calc_out,
                           lcb_result* res_out) {
    if (!C || !models || !data || !offsets || !chisq_out) return fail(LCB_ERR_INVALID, "null pointer");
    if (nmodels <= 0) return fail(LCB_ERR_INVALID, "nmodels must be > 0");
    return guarded(C, [&] {
        std::vector<const lcb::Model*> mp(nmodels);
        std::vector<int64_t> st(nmodels), cnt(nmodels);
        for (int64_t i = 0; i < nmodels; ++i) {
            if (!models[i]) throw Error(LCB_ERR_INVALID, "null model");
            mp[i] = &models[i]->m;
            st[i] = offsets[i];
            cnt[i] = offsets[i + 1] - offsets[i];
            if (cnt[i] < 0) throw Error(LCB_ERR_INVALID, "offsets must be non-decreasing");
        }
        std::vector<double> res, calc;
        std::vector<int> status;
        lcb::Plan& P = C->plan;
        run_transient(C, mp.data(), nmodels, data, st.data(), cnt.data(), scale, 1, res, calc_out ? &calc : nullptr, P,
                      status);
        for (int64_t i = 0; i < nmodels; ++i) {
            chisq_out[i] = P.model_ok[i] ? res[i * 12 + 1] : NAN;
            if (res_out) {
                if (P.model_ok[i]) fill_result(&res[i * 12], &res_out[i]);
                else {
                    double nanv[12];
                    for (double& v : nanv) v = NAN;
                    fill_result(nanv, &res_out[i]);
                }
            }
        }
        if (calc_out)
            lcb::host_copy(calc_out + offsets[0], calc.data(), P.ndatum * sizeof(double));
    });
}

// ---- resident batch -------------------------------------------------------------
int lcb_batch_create(lcb_ctx* C, const lcb_model* const* models, int64_t nmodels, const lcb_datum* data,
                     const int64_t* offsets, lcb_batch** out) {
    if (!C || !models || !data || !offsets || !out) return fail(LCB_ERR_INVALID, "null pointer");
    if (nmodels <= 0) return fail(LCB_ERR_INVALID, "nmodels must be > 0");
    *out = nullptr;
    auto B = std::make_unique<lcb_batch>();
    B->ctx = C;
    int rc = guarded(C, [&] {
        int64_t total = offsets[nmodels] - offsets[0];
        if (total < 0) throw Error(LCB_ERR_INVALID, "offsets must be non-decreasing");
        B->data.assign(data + offsets[0], data + offsets[0] + total);
        for (int64_t i = 0; i < nmodels; ++i) {
            if (!models[i]) throw Error(LCB_ERR_INVALID, "null model");
            B->models.push_back(models[i]->m);
            B->start.push_back(offsets[i] - offsets[0]);
            B->count.push_back(offsets[i + 1] - offsets[i]);
            if (B->count.back() < 0) throw Error(LCB_ERR_INVALID, "offsets must be non-decreasing");
        }
        std::vector<const lcb::Model*> mp(nmodels);
        for (int64_t i = 0; i < nmodels; ++i) mp[i] = &B->models[i];
        B->tune = engine_tuning();
        B->dev.resident = true;
        B->dev.fluxes.ensure(total * sizeof(double));
        lcb::plan_batch(mp.data(), nmodels, B->data.data(), B->start.data(), B->count.data(), C->num_sms, B->plan,
                        B->tune);
        upload_plan(C, B->dev, B->plan);
        upload_data(C, B->dev, B->plan, B->data.data());
        CUDA_TRY(cudaStreamSynchronize(C->stream));
    });
    if (rc != LCB_OK) {
        B->dev.release();
        return rc;
    }
    *out = B.release();
    return LCB_OK;
}

void lcb_batch_destroy(lcb_batch* B) {
    if (!B) return;
    std::lock_guard<std::mutex> g(B->ctx->mu);
    cudaSetDevice(B->ctx->device);
    cudaStreamSynchronize(B->ctx->stream);
    if (B->graph) cudaGraphExecDestroy(B->graph);
    B->dev.release();
    delete B;
}

// Re-plans a resident batch after its models or its tuning changed: plans into the spare
// storage, uploads what changed, drops the captured graph when the shapes changed.
// If the uploads fail part-way (a buffer could not grow), the device buffers no longer
// match the plan: the batch is marked broken, its graph dropped and its shape key
// cleared, so no launch runs on it until a later re-plan uploads everything again.
static void replan_batch(lcb_batch* B, bool params_only) {
    lcb_ctx* C = B->ctx;
    const int64_t n = (int64_t)B->models.size();
    std::vector<const lcb::Model*> mp(n);
    for (int64_t i = 0; i < n; ++i) mp[i] = &B->models[i];
    Range r("lcb replan");
    // parameters that change no table (a sampler's, mostly) change the model table alone
    const bool models_only = params_only && !B->broken &&
                             lcb::replan_models(mp.data(), n, B->data.data(), B->start.data(), B->count.data(), B->plan);
    bool same = models_only;
    if (!models_only) {
        lcb::Plan& P = B->spare;
        lcb::plan_batch(mp.data(), n, B->data.data(), B->start.data(), B->count.data(), C->num_sms, P, B->tune);
        same = !B->broken && P.shape_key == B->plan.shape_key;
        std::swap(B->plan, P);
    }
    try {
        if (models_only) {
            push(C, C->stream, B->dev.models.p, {{B->plan.models.data(), n * sizeof(lcb::ModelDev)}});
            return;
        }
        upload_plan(C, B->dev, B->plan);
        if (!same) upload_data(C, B->dev, B->plan, B->data.data());
        if (!same && B->graph) {
            cudaGraphExecDestroy(B->graph);
            B->graph = nullptr;
        }
        // a new shape waits for its uploads here
        if (!same) CUDA_TRY(cudaStreamSynchronize(C->stream));
    } catch (...) {
        cudaStreamSynchronize(C->stream);
        if (B->graph) cudaGraphExecDestroy(B->graph);
        B->graph = nullptr;
        B->plan.shape_key.clear();
        B->broken = true;
        throw;
    }
    B->broken = false;
}

static void check_usable(const lcb_batch* B) {
    if (B->broken)
        throw Error(LCB_ERR_INVALID, "the batch's last re-plan failed (device memory); set its parameters or "
                                     "tuning again before running it");
}

int lcb_batch_set_tuning(lcb_batch* B, int flux_chunks, int roche_split, int flux_blocks_per_sm) {
    if (!B) return fail(LCB_ERR_INVALID, "null batch");
    if (flux_chunks < 0 || flux_chunks > 16 || roche_split < 0 || roche_split > 16 || flux_blocks_per_sm < 0)
        return fail(LCB_ERR_INVALID, "tuning out of range (flux_chunks, roche_split 0..16; blocks per SM >= 0)");
    lcb_ctx* C = B->ctx;
    return guarded(C, [&] {
        B->tune.flux_chunks = flux_chunks;
        B->tune.roche_split = roche_split;
        B->tune.flux_blocks_per_sm = flux_blocks_per_sm;
        replan_batch(B, false);
    });
}

int lcb_batch_get_tuning(const lcb_batch* B, int* out3) {
    if (!B || !out3) return fail(LCB_ERR_INVALID, "null pointer");
    return guarded(B->ctx, [&] {
        const lcb::Plan& P = B->plan;
        const int bps_max = B->ctx->flux_bps;
        out3[0] = P.flux_chunks;
        out3[1] = P.roche_split;
        out3[2] = P.flux_blocks_per_sm > 0 ? std::min(P.flux_blocks_per_sm, bps_max) : bps_max;
    });
}

int lcb_batch_set_params(lcb_batch* B, const char* const* names, int ndim, const double* values) {
    if (!B || !names || !values || ndim <= 0) return fail(LCB_ERR_INVALID, "bad arguments");
    lcb_ctx* C = B->ctx;
    return guarded(C, [&] {
        const int64_t n = (int64_t)B->models.size();
        for (int j = 0; j < ndim; ++j) {
            int k = lcb::phys_index(names[j]);
            if (k < 0) throw Error(LCB_ERR_UNKNOWN_PARAM, std::string("unknown parameter: '") + names[j] + "'");
            for (int64_t i = 0; i < n; ++i) B->models[i].p[k].value = values[i * ndim + j];
        }
        // planned into the previous call's storage (kept capacity: no allocation or first-touch
        // page faults when a resident batch is re-parameterised step after step); with unchanged
        // tables only the model table is uploaded
        replan_batch(B, true);
    });
}

int lcb_batch_run(lcb_batch* B, int scale) {
    if (!B) return fail(LCB_ERR_INVALID, "null batch");
    lcb_ctx* C = B->ctx;
    return guarded(C, [&] {
        check_usable(B);
        if (B->graph && (B->graph_scale != scale || B->graph_key != B->plan.shape_key || B->graph_cap != C->fblink_cap)) {
            cudaGraphExecDestroy(B->graph);
            B->graph = nullptr;
        }
        if (!B->graph) {
            cudaGraph_t g;
            CUDA_TRY(cudaStreamBeginCapture(C->stream, cudaStreamCaptureModeThreadLocal));
            try {
                enqueue_run(C, B->dev, B->plan, scale, 1, false);
            } catch (...) {
                cudaStreamEndCapture(C->stream, &g);
                throw;
            }
            CUDA_TRY(cudaStreamEndCapture(C->stream, &g));
            cudaError_t e = cudaGraphInstantiate(&B->graph, g, 0);
            cudaGraphDestroy(g);
            CUDA_TRY(e);
            B->graph_scale = scale;
            B->graph_key = B->plan.shape_key;
            B->graph_cap = C->fblink_cap;
        }
        Range r("lcb batch run");
        CUDA_TRY(cudaGraphLaunch(B->graph, C->stream));
        fetch_results(C, B->dev, B->plan, B->h_results, nullptr, &B->h_status, B->ecount);
        B->ran = true;
        for (int s : B->h_status)
            check_device_status(s);
    });
}

int lcb_batch_profile(lcb_batch* B, int scale) {
    if (!B) return fail(LCB_ERR_INVALID, "null batch");
    lcb_ctx* C = B->ctx;
    return guarded(C, [&] {
        check_usable(B);
        enqueue_run(C, B->dev, B->plan, scale, 1, true);
        fetch_results(C, B->dev, B->plan, B->h_results, nullptr, &B->h_status, B->ecount);
        for (int k = 0; k < kStages; ++k) {
            float ms = 0.f;
            CUDA_TRY(cudaEventElapsedTime(&ms, C->ev[k], C->ev[k + 1]));
            B->stage_ms[kStageOrder[k]] = ms;
        }
        B->ran = true;
        for (int s : B->h_status)
            check_device_status(s);
    });
}

int lcb_batch_results(lcb_batch* B, double* chisq_out, double* calc_out, lcb_result* res_out) {
    if (!B) return fail(LCB_ERR_INVALID, "null batch");
    if (!B->ran) return fail(LCB_ERR_INVALID, "lcb_batch_run has not been called");
    lcb_ctx* C = B->ctx;
    return guarded(C, [&] {
        check_usable(B);
        const lcb::Plan& P = B->plan;
        const int64_t n = (int64_t)P.models.size();
        for (int64_t i = 0; i < n; ++i) {
            if (chisq_out) chisq_out[i] = P.model_ok[i] ? B->h_results[i * 12 + 1] : NAN;
            if (res_out) {
                double nanv[12];
                for (double& v : nanv) v = NAN;
                fill_result(P.model_ok[i] ? &B->h_results[i * 12] : nanv, &res_out[i]);
            }
        }
        if (calc_out && P.ndatum) {
            CUDA_TRY(cudaMemcpy(calc_out, B->dev.calc.p, P.ndatum * sizeof(double), cudaMemcpyDeviceToHost));
        }
    });
}

int lcb_batch_stats(const lcb_batch* B, int64_t* out8) {
    if (!B || !out8) return fail(LCB_ERR_INVALID, "null pointer");
    const lcb::Plan& P = B->plan;
    int64_t v[8] = {(int64_t)P.models.size(), P.nelem, P.nsub, P.evals, (int64_t)P.units.size(), P.roche_elems,
                    (int64_t)B->ecount[0], (int64_t)B->ecount[1]};
    std::memcpy(out8, v, sizeof v);
    return LCB_OK;
}

int lcb_batch_search_counts(const lcb_batch* B, int64_t* out5) {
    if (!B || !out5) return fail(LCB_ERR_INVALID, "null pointer");
    for (int k = 0; k < 5; ++k) out5[k] = (int64_t)B->ecount[k];
    return LCB_OK;
}

int lcb_batch_stage_ms(const lcb_batch* B, double* out6) {
    if (!B || !out6) return fail(LCB_ERR_INVALID, "null pointer");
    for (int k = 0; k < kStages; ++k) out6[k] = B->stage_ms[k];
    return LCB_OK;
}

int lcb_ctx_transfer_bytes(const lcb_ctx* C, int64_t* h2d, int64_t* d2h) {
    if (!C || !h2d || !d2h) return fail(LCB_ERR_INVALID, "null pointer");
    *h2d = C->h2d;
    *d2h = C->d2h;
    return LCB_OK;
}

namespace {

// The planner's GPU path for many bright-spot streams (lcb_plan.h: StreamDeviceFn): one
// k_stream launch on the calling thread's default stream of the current device; false on
// any CUDA error (the planner then integrates on the host).
bool stream_on_device(const double* in, int n, double* out, int* status) {
    if (n <= 0) return true;
    char* buf = nullptr;
    const size_t bin = 3 * sizeof(double) * (size_t)n, bst = sizeof(int) * (size_t)n;
    cudaStream_t s = cudaStreamPerThread;
    bool ok = cudaMalloc(&buf, 2 * bin + bst) == cudaSuccess;
    ok = ok && cudaMemcpyAsync(buf, in, bin, cudaMemcpyHostToDevice, s) == cudaSuccess;
    ok = ok && lcb::launch_stream((const double*)buf, n, (double*)(buf + bin), (int*)(buf + 2 * bin), s) == cudaSuccess;
    ok = ok && cudaMemcpyAsync(out, buf + bin, bin, cudaMemcpyDeviceToHost, s) == cudaSuccess;
    ok = ok && cudaMemcpyAsync(status, buf + 2 * bin, bst, cudaMemcpyDeviceToHost, s) == cudaSuccess;
    ok = ok && cudaStreamSynchronize(s) == cudaSuccess;
    if (buf) cudaFree(buf);
    if (!ok) cudaGetLastError();  // clear a non-sticky error; the host path takes over
    return ok;
}

const bool g_stream_device_registered = (lcb::set_stream_device(&stream_on_device), true);

}  // namespace

int lcb_stream_points(lcb_ctx* C, const double* q, const double* radius, int64_t n, int on_device, double* out) {
    if (!C || (n > 0 && (!q || !radius || !out)) || n < 0 || n > (1 << 24)) return fail(LCB_ERR_INVALID, "bad arguments");
    return guarded(C, [&] {
        (void)g_stream_device_registered;
        std::vector<double> in(3 * n);
        std::vector<int> st(n, lcb::stream::kStreamOk);
        for (int64_t i = 0; i < n; ++i) {
            in[3 * i] = q[i];
            in[3 * i + 1] = lcb::host_xl1(q[i]);
            in[3 * i + 2] = radius[i];
        }
        if (on_device) {
            if (!stream_on_device(in.data(), (int)n, out, st.data()))
                throw Error(LCB_ERR_CUDA, "the gas-stream kernel failed");
        } else {
            for (int64_t i = 0; i < n; ++i)
                st[i] = lcb::stream::stream_to_radius_core(q[i], in[3 * i + 1], radius[i], out + 3 * i);
        }
        bool bad = false;
        for (int64_t i = 0; i < n; ++i)
            if (st[i] != lcb::stream::kStreamOk) {
                out[3 * i] = out[3 * i + 1] = out[3 * i + 2] = NAN;
                bad = true;
            }
        if (bad) throw Error(LCB_ERR_MODEL, "the gas stream did not reach a radius (NaN rows)");
    });
}

int lcb_model_work(const lcb_model* model, const lcb_datum* data, int64_t n, int64_t* out4) {
    if (!model || (!data && n > 0) || !out4 || n < 0) return fail(LCB_ERR_INVALID, "bad arguments");
    return guarded(nullptr, [&] {
        const lcb::Model* mp = &model->m;
        int64_t st = 0, cnt = n;
        lcb::Plan P;
        lcb::plan_batch(&mp, 1, data, &st, &cnt, 148, P, engine_tuning());
        const bool ok = !P.model_ok.empty() && P.model_ok[0];
        int64_t v[4] = {ok ? P.nelem : 0, ok ? P.roche_elems : 0, ok ? P.nsub : 0, ok ? P.evals : 0};
        std::memcpy(out4, v, sizeof v);
    });
}

int lcb_ctx_set_search_cap(lcb_ctx* C, int evals) {
    if (!C || evals < 0) return fail(LCB_ERR_INVALID, "bad arguments");
    return guarded(C, [&] { C->fblink_cap = evals > 0 ? evals : lcb::kFblinkEvalCap; });
}

int lcb_wait_probe(lcb_ctx* C, int64_t limit_cycles, int64_t* waited_cycles) {
    if (!C || limit_cycles <= 0 || limit_cycles > 4000000000LL) return fail(LCB_ERR_INVALID, "bad arguments");
    return guarded(C, [&] {
        C->probe.ensure(2 * sizeof(long long));
        int* status = C->probe.as<int>();
        long long* waited = C->probe.as<long long>() + 1;
        CUDA_TRY(cudaMemsetAsync(C->probe.p, 0, 2 * sizeof(long long), C->stream));
        CUDA_TRY(lcb::launch_wait_probe((long long)limit_cycles, status, waited, C->stream));
        long long h[2] = {0, 0};
        CUDA_TRY(cudaMemcpyAsync(h, C->probe.p, sizeof h, cudaMemcpyDeviceToHost, C->stream));
        CUDA_TRY(cudaStreamSynchronize(C->stream));
        if (waited_cycles) *waited_cycles = h[1];
        if ((int)(h[0] & 0xffffffff) & lcb::kStatusTmaTimeout)
            throw Error(LCB_ERR_DEVICE_CHECK, "a bounded device wait timed out");
    });
}

int lcb_measure_fma_peak(lcb_ctx* C, int which, double* tflops) {
    if (!C || !tflops || (which != 0 && which != 1)) return fail(LCB_ERR_INVALID, "bad arguments");
    return guarded(C, [&] { CUDA_TRY(lcb::measure_fma_peak(which, C->num_sms, C->stream, tflops)); });
}

}  // extern "C"

// ===========================================================================
// lcb_light_curve_noalloc: the light curve of one model with no device
// allocation.
//
// Some callers cannot call cudaMalloc: a process whose device memory is
// already claimed by another framework's pool allocator (JAX preallocating
// most of the GPU, a serving runtime with a fixed memory budget), a plugin
// host that forbids allocation inside its callbacks, or a timing-sensitive
// loop that cannot afford the device-wide synchronisation cudaMalloc and
// cudaFree may imply.  For them this entry point runs the same kernels as
// lcb_light_curve, but every device buffer (plan tables, element and
// sub-phase arrays, flux partials, results) is carved out of one statically
// allocated arena of LCB_NOALLOC_ARENA_BYTES.  Host staging uses ordinary
// pageable host memory.
//
// The arena is file-scope device memory: every device on which this
// library's device code is loaded holds it until the process exits.  In host
// code its name is only a host-side shadow; each call looks up the device
// address (cudaGetSymbolAddress, with the context's device current).
//
// Every call on a device shares the arena, which keeps the previous call's
// contents.  The accumulators that must start at zero (per-model sums, status
// words, the work-unit counter and search counters) are cleared by the launch
// sequence itself; every other region is written in full before it is read.
// Two calls whose GPU work overlapped would race on the arena, so calls on one
// device are serialised by a per-device lock, and each call waits for its GPU
// work (also on its error paths) before it returns.
// ===========================================================================
// The limit on a call's scratch counts the tables, element, sub-phase and result arrays.  The list of
// open elements (4 bytes per Roche thread: at most 8 per element of 160 or more) and the epilogue's
// sums (about one byte per datum of 76 or more) come on top, under a sixteenth of the rest; and where no
// split search was counted, the first hits of one on a short list (first_hits, 2.9 MiB on 148 SMs).
static constexpr size_t kNoallocHits = (size_t)(lcb::split_target(148) / 2 + lcb::kRocheBlock) * sizeof(int);
static constexpr size_t kNoallocArena =
    (size_t)LCB_NOALLOC_ARENA_BYTES + LCB_NOALLOC_ARENA_BYTES / 16 + kNoallocHits + (64u << 10);
static __device__ __align__(256) unsigned char g_noalloc_arena[kNoallocArena];

namespace {

constexpr int kNoallocMaxDevices = 64;
std::mutex g_noalloc_mu[kNoallocMaxDevices];   // one per device

// The arena's device address on the current device.  Looked up on every call
// (it is cheap next to the launch sequence), so a device or primary-context
// reset between calls, which reloads the module at a new address, cannot leave
// a stale pointer behind.  Caller holds g_noalloc_mu[device] and has made
// `device` current.
unsigned char* noalloc_arena() {
    void* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_arena);
    if (e != cudaSuccess || !p)
        throw Error(LCB_ERR_CUDA, std::string("cudaGetSymbolAddress(no-alloc arena): ") + cudaGetErrorString(e));
    return static_cast<unsigned char*>(p);
}

// Host -> arena copies of the plan's tables and the data (no allocation).
void noalloc_upload(lcb_ctx* C, DeviceSet& D, const lcb::Plan& P, const lcb_datum* data) {
    auto put = [&](void* dst, const void* src, size_t bytes) {
        if (bytes) CUDA_TRY(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, C->stream));
        C->h2d += (int64_t)bytes;
    };
    size_t off = 0;
    for (const Piece& p : plan_tables(P, D, D.tables.p)) {
        put((char*)D.tables.p + off, p.src, p.bytes);
        off += pad256(p.bytes);
    }
    put(D.datum.p, data + P.data_first, P.data_count * sizeof(lcb_datum));
}

}  // namespace

extern "C" int lcb_light_curve_noalloc(lcb_ctx* C, const lcb_model* model, const lcb_datum* data, int64_t n,
                                       int scale, int rdata, double* calc_out, lcb_result* res_out) {
    if (!C || !model || (!data && n > 0) || !calc_out) return fail(LCB_ERR_INVALID, "null pointer");
    if (n <= 0) return fail(LCB_ERR_EMPTY, "No data points");
    if (C->device < 0 || C->device >= kNoallocMaxDevices)
        return fail(LCB_ERR_INVALID, "lcb_light_curve_noalloc: device index beyond the supported 64");
    return guarded(C, [&] {
        const lcb::Model* mp = &model->m;
        int64_t st = 0, cnt = n;
        lcb::Plan P;  // with the table of first sub-phases, regular data or not: it is part of what the limit counts
        lcb::plan_batch(&mp, 1, data, &st, &cnt, C->num_sms, P);
        if (!P.model_ok[0]) throw Error(LCB_ERR_MODEL, P.model_err[0]);
        DeviceSet D;  // views into the static arena: its own is never allocated
        size_t need = 0;
        const size_t total = carve(C, P, nullptr, D, &need);
        const bool over = need > (size_t)LCB_NOALLOC_ARENA_BYTES;
        if (over || total > kNoallocArena)
            throw Error(LCB_ERR_INVALID, "lcb_light_curve_noalloc: this model and data need " +
                                             std::to_string(over ? need : total) +
                                             " bytes of device scratch, more than the fixed arena's " +
                                             std::to_string(over ? (size_t)LCB_NOALLOC_ARENA_BYTES : kNoallocArena) +
                                             "; use lcb_light_curve (or coarser grids / fewer points)");
        std::lock_guard<std::mutex> lock(g_noalloc_mu[C->device]);
        carve(C, P, noalloc_arena(), D);
        std::vector<double> res, calc;
        std::vector<int> status;
        try {
            noalloc_upload(C, D, P, data);
            enqueue_run(C, D, P, scale, rdata, false);
            fetch_results(C, D, P, res, &calc, &status, nullptr, false);  // ends with a stream synchronise
        } catch (...) {
            cudaStreamSynchronize(C->stream);  // no work may touch the arena after the lock is released
            throw;
        }
        check_device_status(status[0]);
        if (status[0] & lcb::kStatusIterCap)
            throw Error(LCB_ERR_DEVICE_CHECK, "a device-side iteration cap tripped for this model");
        std::memcpy(calc_out, calc.data(), n * sizeof(double));
        if (res_out) fill_result(res.data(), res_out);
    });
}
