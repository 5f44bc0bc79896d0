// Layer runs (run.cu): many small layers of a request in one launch.
#pragma once

#include "common.cuh"

namespace pmdd {
namespace dev {

constexpr int kRunBlocks = 8;            // blocks (one cluster) per request
constexpr int64_t kRunCap = int64_t(kRunBlocks) * 2048;  // points of a layer (run.cu: 2048 per block)

// What the host reads back per request.
struct RunOut {
    int32_t done;                        // layers finished
    int32_t final_size;                  // points of the last layer's first node
    int64_t final_off;                   // and where its slot starts
    int64_t cand_total, cand_peak;       // candidates over the layers, of the largest
    int64_t surv_total, surv_peak;       // points of the layers before the last (not the first)
    int64_t tile_surv, stair;            // as ExpandJob::tile_surv
    int64_t removed;                     // labels removed by state dominance
};

// Runs a request top-down from `layer` until `last`, or until a layer has an oversized
// destination or does not fit its blocks' regions.
struct RunJob {
    const int32_t *item_arc_off;         // in-arc CSR (global node ids)
    const int32_t *arc_nbr;
    const int32_t *arc_wrow;
    const int32_t *weights;
    const int32_t *layer_off;
    const void *pts;                     // frontier of layer `layer`
    const int64_t *off;
    const int32_t *size;
    const uint8_t *sorted;
    int32_t layer, last;
    int32_t terminal;                    // the DD's last layer
    // layer `layer + j` is written to buffer set j & 1
    void *b_pts[2];                      // kRunCap points
    int64_t *b_off[2];                   // vcap nodes
    int32_t *b_size[2];
    uint8_t *b_sorted[2];
    int32_t vcap;
    int32_t pair_max;
    int32_t sd_kind;                     // state dominance (statedom.cuh), 0: none
    const int32_t *sd_order;             // over all nodes, as the DD carries it
    const int32_t *sd_next;
    const uint64_t *sd_state;
    int32_t state_words;
    uint8_t *keep;                       // kRunCap flags
    RunOut *out;
    CountJob *count;                     // the count of the layer after the last one finished:
                                         // its layer-dependent fields are filled in
    uint32_t *err;
};

cudaError_t launch_layer_runs(int d, bool wide, bool lex, const RunJob *jobs, int num_jobs, cudaStream_t stream);

}  // namespace dev
}  // namespace pmdd
