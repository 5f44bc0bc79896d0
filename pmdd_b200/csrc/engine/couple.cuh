// Method-3 coupling and DD-preparation launchers (couple.cu).
#pragma once

#include <algorithm>

#include "common.cuh"

namespace pmdd {
namespace dev {

constexpr int kCoupleThreads = 256;

// Per-job device counters (int64 each), followed by the units before each cutset node
// (num_nodes + 1 of them).
enum CoupleCtr {
    kCtrF = 0,          // points of the running frontier at the front of U
    kCtrB = 1,          // survivors appended this round (may exceed room; clamped)
    kCtrResume = 2,     // first unit whose survivors did not fit (INT64_MAX: none)
    kCtrCursor = 3,     // next unit to hand out this round
    kCtrUnits = 4,      // units in all: per cutset node, its top-down frontier in groups of 8
    kCtrDone = 5,       // 1 once a product round finished every unit
    kCtrValidEnd = 6,   // U slots below this index hold written points (set on overflow)
    kCtrProducts = 7,   // sum over cutset nodes of |TD_v| * |BU_v| (statistics)
    kCtrCount = 8
};

struct CoupleJob {
    void *td_pts;       // the cutset's frontiers; each is put in a spatial order at the start
    const int64_t *td_off;
    const int32_t *td_size;
    void *bu_pts;
    const int64_t *bu_off;
    const int32_t *bu_size;
    int32_t num_nodes;
    int32_t pad0;
    void *U;            // running frontier followed by this round's survivors
    void *U_alt;        // receives the next running frontier (the buffers swap each round)
    int64_t ucap;       // points each of U / U_alt can hold
    void *sc_slab;      // scratch: 2 * ucap points (refilter slab; product rounds: the index of F)
    int32_t *sc_idx;    // refilter scratch: ucap ints (keys)
    int32_t *sc_sidx;   // refilter scratch: ucap ints (places)
    int64_t *ctr;       // kCtrCount counters, then num_nodes + 1 unit offsets
};

// Bytes of device memory a coupling job with capacity ucap needs besides the counters.
inline size_t couple_bytes(int64_t ucap, int d, size_t elem) {
    const size_t pts = (static_cast<size_t>(ucap) * d * elem + 255) / 256 * 256;
    const size_t idx = (static_cast<size_t>(ucap) * 4 + 255) / 256 * 256;
    return 4 * pts + 2 * idx;
}

// The bottom-up (outgoing-arc) CSR of a DD: arc order within a node unspecified.
struct CsrJob {
    const int32_t *in_off;
    const int32_t *arc_src;
    const int32_t *arc_w;
    int32_t num_nodes, num_arcs;
    int32_t *out_off;   // [num_nodes + 1]
    int32_t *cursor;    // [num_nodes] scratch
    int32_t *out_head;  // [num_arcs]
    int32_t *out_w;     // [num_arcs]
};
constexpr int kCsrLaunches = 4;
cudaError_t launch_build_out_csr(const CsrJob &job, cudaStream_t stream);
// Of many DDs at once (device array).
cudaError_t launch_build_out_csrs(const CsrJob *jobs, int count, int32_t max_nodes, int32_t max_arcs,
                                  cudaStream_t stream);

// One coupling round for `num_jobs` jobs of one (d, wide) group.  A seed round counts the
// units and products, orders the cutset's frontiers, and appends, per cutset node, the sums
// of the two frontiers' per-objective and sum maximisers; a product round streams the
// products against the running frontier.  Either way the maxima of running frontier +
// appended points (maxima.cuh) land in U_alt as the next running frontier.  `points`: most
// points a job's U can hold after the appends; *launches: kernels launched.
cudaError_t launch_couple_round(int d, bool wide, const CoupleJob *jobs, int num_jobs, int blocks_per_job,
                                bool seed, int64_t points, int64_t *launches, cudaStream_t stream);

}  // namespace dev
}  // namespace pmdd
