// Layer runs (run.cu): many small layers of a request in one launch.
#pragma once

#include "common.cuh"

namespace pmdd {
namespace dev {

constexpr int kRunBlocks = 8;            // blocks (one cluster) per request
constexpr int64_t kRunCap = int64_t(kRunBlocks) * 2048;  // points of a layer (run.cu: 2048 per block)

// What the host reads back per request.
struct RunOut {
    int32_t done;                        // layers finished (method 3: top-down)
    int32_t done_bu;                     // method 3: bottom-up
    int32_t final_size, pad;             // points of the last layer's first node
    int64_t final_off;                   // and where its slot starts
    int64_t cand_total, cand_peak;       // candidates over the layers, of the largest
    int64_t surv_total, surv_peak;       // points of the layers (method 1: but the first and the last)
    int64_t tile_surv, stair;            // as ExpandJob::tile_surv
    int64_t removed;                     // labels removed by state dominance
};

// One direction of a request: its arcs by destination, and its frontiers.
struct RunSide {
    const int32_t *item_arc_off;         // in-arc CSR top-down, out-arc CSR bottom-up (global ids)
    const int32_t *arc_nbr;
    const int32_t *arc_wrow;
    const void *pts;                     // frontier of layer `layer`
    const int64_t *off;
    const int32_t *size;
    const uint8_t *sorted;
    int32_t layer;
    int32_t pad;
    int64_t score;                       // method 3: the engine's side rule
    // the j-th layer from there is written to buffer set j & 1
    void *b_pts[2];                      // kRunCap points
    int64_t *b_off[2];                   // vcap nodes
    int32_t *b_size[2];
    uint8_t *b_sorted[2];
    CountJob *count;                     // the count of the layer after the last one finished:
                                         // its layer-dependent fields are filled in
};

// Method 1 runs a request top-down (td) from its layer until `last`; method 3 both sides, by
// the engine's side rule (top-down while its score <= the bottom-up one), for at most
// `steps` layers and until they are one layer apart.  Either stops before a layer that has
// an oversized destination or does not fit its blocks' regions.
struct RunJob {
    RunSide td, bu;
    const int32_t *weights;
    const int32_t *layer_off;
    int32_t last;
    int32_t terminal;                    // the DD's last layer
    int32_t steps;
    int32_t vcap;
    int32_t pair_max;
    int32_t sd_kind;                     // state dominance (statedom.cuh), 0: none
    const int32_t *sd_order;             // over all nodes, as the DD carries it
    const int32_t *sd_next;
    const uint64_t *sd_state;
    int32_t state_words;
    int32_t pad;
    uint8_t *keep;                       // kRunCap flags
    RunOut *out;
    uint32_t *err;
};

// method 1: run_layers_kernel; method 3 (meet): run_meet_kernel.
cudaError_t launch_layer_runs(int d, bool wide, bool lex, bool meet, const RunJob *jobs, int num_jobs,
                              cudaStream_t stream);

}  // namespace dev
}  // namespace pmdd
