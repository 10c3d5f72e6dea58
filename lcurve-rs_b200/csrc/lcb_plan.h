// lcb_plan.h — host planning of a batch: per-model constants and work decomposition.
#pragma once

#include <string>
#include <vector>

#include "lcb_internal.h"
#include "lcb_model.h"

namespace lcb {

// Launch-shape choices an autotuner may fix; 0 leaves each to the planner's heuristic.  Every
// value lies in the range the heuristic itself produces, so the kernels handle it as usual.
struct PlanTuning {
    int flux_chunks = 0;         // elements per flux work unit, in chunks of kFluxChunk (1..16)
    int roche_split = 0;         // threads per Roche-eclipsed element in the phase scan (1..16)
    int flux_blocks_per_sm = 0;  // persistent flux blocks per SM (1..occupancy limit)
    bool datum_tables = true;    // fill datum_model / datum_sub0 / datum_src for regular models too
};

struct Plan {
    std::vector<ModelDev> models;
    std::vector<SegDesc> segs;
    std::vector<Band> bands;
    std::vector<Ring> rings;
    std::vector<ElemBlock> eblocks;    // k_elements
    std::vector<ElemBlock> rblocks;    // k_roche
    std::vector<ElemBlock> ablocks;    // k_aux
    std::vector<FluxUnit> units;
    // per (model, datum), with PlanTuning::datum_tables, or datum_sub0 where some model is irregular:
    std::vector<int32_t> datum_model;   // model index
    std::vector<int64_t> datum_sub0;    // first global sub-phase
    std::vector<int64_t> datum_src;     // index into the caller's data array
    // the records to upload, the caller's [data_first, data_first + data_count): the range that the
    // models' data span (they may share records); the largest model's data
    int64_t data_first = 0, data_count = 0, most_data = 0;
    std::vector<std::vector<uint64_t>> keys;  // per model: what its tables and units depend on (replan_models)
    std::vector<int32_t> model_ok;      // 1 = planned, 0 = failed (NaN chisq)
    std::vector<std::string> model_err;
    int64_t nelem = 0, nsub = 0, ndatum = 0, npartial = 0;
    int64_t evals = 0, roche_elems = 0;
    // Signature of everything that fixes buffer sizes and launch shapes.
    std::vector<int64_t> shape_key;
    bool any_iscale = false;  // some model fits per-component scale factors (needs fcomp scratch)
    int roche_split = 1;      // threads per element of the general eclipse search, were every element left to it
    int split_fix = 0;        // PlanTuning::roche_split where it applies: fixed, whatever the list's length
    int flux_chunks = 1;      // elements per flux work unit / kFluxChunk
    int flux_blocks_per_sm = 0;  // persistent flux blocks per SM; 0 = the occupancy limit
    int flux_share = 1;          // 1: a block's four warps share a flux unit, 0: each warp has its own
    int curve_blocks = 1, result_blocks = 1;  // blocks per model of k_curve and (scaled) k_results
    int curve_share = 0;  // k_curve: 1 = a block's eight warps share one tile of data, 0 = a tile each

    // Empties the plan but keeps every buffer's capacity, so re-planning a
    // batch of the same size touches no fresh memory.
    void reset() {
        models.clear(); segs.clear(); bands.clear(); rings.clear(); eblocks.clear(); rblocks.clear();
        ablocks.clear(); units.clear(); datum_model.clear(); datum_sub0.clear(); datum_src.clear();
        model_ok.clear(); model_err.clear(); shape_key.clear();
        nelem = nsub = ndatum = npartial = evals = roche_elems = 0;
        data_first = data_count = most_data = 0;
        keys.clear();
        any_iscale = false;
        roche_split = 1;
        split_fix = 0;
        flux_chunks = 1;
        flux_blocks_per_sm = 0;
        curve_blocks = result_blocks = 1;
        curve_share = 0;
        flux_share = 1;
    }
};

// Plans models[0..n); model i is evaluated on data[start[i] .. start[i]+count[i])
// (ranges may overlap, e.g. one shared data set).  Models that are physically
// invalid are marked failed (model_ok = 0) instead of throwing.
void plan_batch(const Model* const* models, int64_t n, const lcb_datum* data, const int64_t* start,
                const int64_t* count, int num_sms, Plan& out, const PlanTuning& tune = PlanTuning{});

// New physical parameters for the models of a plan on the same data: fills in the model table alone and
// returns true when no table, block or unit of the plan depends on what changed; false: plan again (the
// plan is then unchanged).
bool replan_models(const Model* const* models, int64_t n, const lcb_datum* data, const int64_t* start,
                   const int64_t* count, Plan& P);

// Copies bytes on the host's threads (large copies only; a few MB and more).
void host_copy(void* dst, const void* src, size_t bytes);

// Scan threads of the split eclipse search that fill the GPU: sixteen waves of five 128-thread blocks.
constexpr int64_t split_target(int num_sms) { return (int64_t)(num_sms > 1 ? num_sms : 1) * 640 * 16; }

// Host FP64 helpers also used by tests of the planner.
double host_xl1(double q);
double host_xl11(double q, double spin);
double host_xl12(double q, double spin);
void host_stream_spot(double q, double radius, double out[3]);

// Gas-stream end points on a GPU for many (q, radius) pairs at once: in[3 i ..] = (q,
// L1 distance, radius), out[3 i ..] = the position, status[i] = a stream:: code.
// Returns false where no GPU path is available.  The engine registers one; the
// planner calls it for a batch with more new pairs than the host's threads
// integrate quickly (more than four per thread), and memoises the results.
using StreamDeviceFn = bool (*)(const double* in, int n, double* out, int* status);
void set_stream_device(StreamDeviceFn fn);
// The memo's value for (q, radius) if present; stores a result in it.
bool spot_memo_get(double q, double radius, double out[3]);
void spot_memo_put(double q, double radius, const double out[3]);
int64_t host_numface(int nlat);

}  // namespace lcb
