// Layer runs: one cluster of 8 blocks takes a request through as many small layers as it
// can in one launch.
//
// A small layer is bound by latency: a launch for its tiles and one for its counts cost
// about 23 us however few candidates there are (each dependent global load, block barrier
// and launch gap in a row), and every few layers a host round trip.  Here the layers
// follow one another inside the launch.  Destinations are split over the blocks by number;
// a block counts, expands and filters its own (lex_items.cuh / pair_items.cuh) into its own
// region of the layer's slots, so that the blocks meet once per layer, at the cluster's
// barrier, and there agree whether the layer stands.  A layer that holds an oversized
// destination or outgrows a block's region is left to the ordinary steps: the run ends
// before it, and the count job of that layer is completed for the count kernel that
// follows.  State dominance (statedom_node.cuh) takes two barriers more.
//
// What a layer waits for in turn is kept short: a block fetches the next layer's arcs into
// shared memory while it waits at the barrier, then gathers every arc's size, slot and
// order flag at once, and the blocks' words travel through distributed shared memory.
//
// Frontiers written by other blocks are read past the L1 cache (ld_live): the buffers
// alternate, so a line of the layer before last may still be there.
//
// One B200, a layer: about 10 us, a chain of dependent loads, block barriers and the
// cluster's, against 23 us for the two launches of a chained one.  KP d=3 n=20: 20 layers
// in 0.22 ms (call 0.74 -> 0.33 ms); a set packing d=3 n=100 whose layers all fit: 1.1 ms
// (call 3.0 -> 1.3 ms; 1.6 - 1.9 ms where layers in its middle outgrow the regions); n=91 with
// state dominance, which ordinary steps take one layer at a time: 2.2 ms (call 9.0 -> 2.7 -
// 3.2 ms; a node's loads out together, its partners' labels 32 at a time, and no compaction
// of nodes that lose no label are 0.5 ms of it).
#include "run.cuh"

#include <cooperative_groups.h>

#include <utility>

#include "lex_items.cuh"
#include "pair_items.cuh"
#include "statedom_node.cuh"

namespace pmdd {
namespace dev {

namespace {

constexpr int kRunThreads = 512;
static_assert(kRunCap == static_cast<int64_t>(kRunBlocks) * kRunRegion, "regions");

template <int D, typename T, bool LEX>
struct RunItems {
    using Smem = PairSmem<D, T>;
};
template <int D, typename T>
struct RunItems<D, T, true> {
    using Smem = LexSmem<T>;
};

// What a block tells the others of its request about a layer.
struct RunPub {
    int64_t cand;     // candidates of its destinations
    int64_t surv;     // points it kept
    int64_t removed;  // labels it removed from the layer before (state dominance)
    int64_t bad;      // 1: the layer cannot be run here
};

template <int D, typename T, bool LEX>
struct RunSmem {
    typename RunItems<D, T, LEX>::Smem items;
    RunStage st;
    ExpandJob J;
    StateDomJob sd;
    RunPub pub[2][kRunBlocks];
    int64_t warp_l[32], tot;
    unsigned long long tile[2];
    int32_t removed;
};

// A layer's share of one block: destinations [v0, v1) and their arcs [a0, a1).
struct RunShare {
    int32_t y0, nodes, v0, v1, a0, a1;
};

// The frontier a side expands from after `done` layers of the run.
struct RunFrom {
    const void *pts;
    const int64_t *off;
    const int32_t *size;
    const uint8_t *sorted;
};
__device__ __forceinline__ RunFrom run_from(const RunSide &d, int done) {
    if (done == 0) return {d.pts, d.off, d.size, d.sorted};
    const int b = done & 1;
    return {d.b_pts[b], d.b_off[b], d.b_size[b], d.b_sorted[b]};
}

// The block's share of layer y, expanded from layer x, with its arcs' neighbours and weight
// rows fetched (as many as fit).
__device__ __forceinline__ RunShare run_fetch(RunStage &st, const RunSide &d, const int32_t *layer_off, int x, int y,
                                              int rank) {
    RunShare h;
    const int32_t x0 = layer_off[x];
    h.y0 = layer_off[y];
    h.nodes = layer_off[y + 1] - h.y0;
    h.v0 = static_cast<int32_t>(static_cast<int64_t>(h.nodes) * rank / kRunBlocks);
    h.v1 = static_cast<int32_t>(static_cast<int64_t>(h.nodes) * (rank + 1) / kRunBlocks);
    h.a0 = d.item_arc_off[h.y0 + h.v0];
    h.a1 = d.item_arc_off[h.y0 + h.v1];
    for (int32_t k = threadIdx.x; k < min(h.a1 - h.a0, kRunRegion); k += kRunThreads) {
        st.nbr[k] = d.arc_nbr[h.a0 + k] - x0;
        st.w[k] = d.arc_wrow[h.a0 + k];
    }
    for (int32_t i = h.v0 + threadIdx.x; i <= h.v1; i += kRunThreads)
        asm volatile("prefetch.global.L1 [%0];" ::"l"(d.item_arc_off + h.y0 + i));
    return h;
}

// Candidate offsets of the block's arcs within its region, their parents' slots and order;
// returns the candidates.  After run_fetch and a barrier; ends with a barrier.
__device__ __forceinline__ int64_t run_gather(RunStage &st, const RunFrom &from, int32_t arcs, int64_t region,
                                              int64_t *warp_l, int64_t *tot) {
    constexpr int PER = kRunRegion / kRunThreads;
    int32_t c[PER];
    int64_t mine = 0;
#pragma unroll
    for (int r = 0; r < PER; ++r) {
        const int k = threadIdx.x * PER + r;
        c[r] = 0;
        if (k < arcs) {
            const int32_t nb = st.nbr[k];
            c[r] = ld_live<true>(from.size + nb);
            st.src[k] = ld_live64<true>(from.off + nb);
            st.sorted[k] = ld_live<true>(reinterpret_cast<const unsigned char *>(from.sorted) + nb);
        }
        mine += c[r];
    }
    int64_t at = region + block_exclusive_scan<int64_t, kRunThreads>(mine, warp_l, tot);
    const int64_t cand = *tot;
#pragma unroll
    for (int r = 0; r < PER; ++r) {
        const int k = threadIdx.x * PER + r;
        if (k < arcs) st.off[k] = at;
        at += c[r];
    }
    if (threadIdx.x == 0) st.off[arcs] = region + cand;
    __syncthreads();
    return cand;
}

// The expansion of a share into buffer set b (one thread calls it).
__device__ __forceinline__ void run_describe(ExpandJob &J, const RunJob &R, const RunSide &d, const RunShare &h,
                                             const void *prev_pts, RunStage &st, int b, unsigned long long *tile) {
    J.item_arc_off = d.item_arc_off;
    J.weights = R.weights;
    J.arc_cand_off = st.off;
    J.arc_base = h.a0;
    J.item_base = h.y0;
    J.num_items = h.nodes;
    J.prev_pts = prev_pts;
    J.out_pts = d.b_pts[b];
    J.out_off = d.b_off[b];
    J.out_size = d.b_size[b];
    J.out_sorted = d.b_sorted[b];
    J.err = R.err;
    J.tile_surv = tile;
    J.pair_max = R.pair_max;
    J.phase_clk = nullptr;
    tile[0] = tile[1] = 0;
    st.over = 0;
}

// Completes the count job of the layer y after layer x (y outside the DD: nothing to count).
__device__ __forceinline__ void run_count_job(CountJob &C, const RunSide &d, const int32_t *layer_off, int x, int y,
                                              bool more, const int32_t *x_size) {
    C.cur_base = layer_off[x];
    C.cur_nodes = more ? layer_off[x + 1] - layer_off[x] : 0;
    C.cur_size = x_size;
    C.item_base = more ? layer_off[y] : 0;
    C.num_items = more ? layer_off[y + 1] - layer_off[y] : 0;
    C.arc_base = more ? d.item_arc_off[layer_off[y]] : 0;
    C.num_arcs = more ? d.item_arc_off[layer_off[y + 1]] - C.arc_base : 0;
}

}  // namespace

template <int D, typename T, bool LEX>
__global__ void __cluster_dims__(kRunBlocks, 1, 1) __launch_bounds__(kRunThreads, 1)
    run_layers_kernel(const RunJob *__restrict__ jobs) {
    constexpr int NT = kRunThreads;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    RunSmem<D, T, LEX> &S = *reinterpret_cast<RunSmem<D, T, LEX> *>(smem_raw);
    RunStage &st = S.st;
    cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    const RunJob &R = jobs[blockIdx.x / kRunBlocks];
    const RunSide &d = R.td;
    const int rank = static_cast<int>(blockIdx.x % kRunBlocks);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t region = static_cast<int64_t>(rank) * kRunRegion;
    int done = 0;
    int64_t removed_total = 0, before_surv = 0;
    unsigned long long tile_surv = 0, stair = 0;
    int64_t cand_total = 0, cand_peak = 0, surv_total = 0, surv_peak = 0;
    if (tid == 0) S.removed = 0;
    RunShare h = run_fetch(st, d, R.layer_off, d.layer, d.layer + 1, rank);
    cluster.sync();  // every block has started: its shared memory may be written to
    for (int y = d.layer + 1; y <= R.last; ++y) {
        const int b = (done + 1) & 1;
        const RunFrom from = run_from(d, done);
        const int32_t arcs = h.a1 - h.a0;
        bool bad = h.nodes > R.vcap || arcs > kRunRegion;
        if (tid == 0) run_describe(S.J, R, d, h, from.pts, st, b, S.tile);
        __syncthreads();
        int64_t cand = 0;
        if (!bad) {
            cand = run_gather(st, from, arcs, region, S.warp_l, &S.tot);
            bad = cand > kRunRegion;
        }
        // --- expand and filter
        if (!bad) {
            if constexpr (LEX) lex_items<T, NT, true>(S.items, S.J, &st, h.v0, h.v1, []() {});
            else pair_items<D, T, NT, true>(S.items, S.J, &st, h.v0, h.v1, []() {});
            bad = st.over != 0;
        }
        if (tid < kRunBlocks) {  // tell every block of the cluster
            RunPub *to = cluster.map_shared_rank(&S.pub[b][rank], tid);
            to->cand = cand;
            to->surv = static_cast<int64_t>(S.tile[0]);
            to->removed = S.removed;
            to->bad = bad ? 1 : 0;
        }
        __syncwarp();
        auto token = cluster.barrier_arrive();
        const int32_t y0 = h.y0, nodes = h.nodes;
        if (y < R.last) h = run_fetch(st, d, R.layer_off, y, y + 1, rank);
        cluster.barrier_wait(std::move(token));
        // --- does the layer stand?
        int64_t all_cand = 0, all_surv = 0, all_removed = 0, any_bad = 0;
#pragma unroll
        for (int r = 0; r < kRunBlocks; ++r) {
            all_cand += S.pub[b][r].cand;
            all_surv += S.pub[b][r].surv;
            all_removed += S.pub[b][r].removed;
            any_bad |= S.pub[b][r].bad;
        }
        if (done > 0) removed_total += all_removed;
        if (any_bad) break;  // every block of the cluster alike
        if (done > 0) {  // the layer before is not the last
            surv_total += before_surv - all_removed;
            surv_peak = max(surv_peak, before_surv - all_removed);
        }
        before_surv = all_surv;
        cand_total += all_cand;
        cand_peak = max(cand_peak, all_cand);
        tile_surv += S.tile[0];
        stair += S.tile[1];
        ++done;
        __syncthreads();  // S.J, S.tile and S.removed are rewritten
        // --- state dominance: mark against the labels as they are, then compact
        if (tid == 0) S.removed = 0;
        if (R.sd_kind != 0 && nodes > 1) {
            if (tid == 0) {
                StateDomJob &sd = S.sd;
                sd.order = R.sd_order + y0;
                sd.next = R.sd_kind == 2 ? R.sd_next + 2 * static_cast<int64_t>(y0) : nullptr;
                sd.state = R.sd_state;
                sd.in_off = d.item_arc_off;
                sd.arc_src = d.arc_nbr;
                sd.arc_w = d.arc_wrow;
                sd.pts = d.b_pts[b];
                sd.off = d.b_off[b];
                sd.size = d.b_size[b];
                sd.keep = R.keep;
                sd.removed = nullptr;
                sd.node_base = y0;
                sd.num_nodes = nodes;
                sd.kind = R.sd_kind;
                sd.state_words = R.state_words;
            }
            __syncthreads();
            constexpr int kWarps = NT / 32;
            const int32_t p0 = rank * kWarps + warp;
            uint64_t drops = 0;  // of the warp's nodes, the ones that lose a label (its 64th on: unknown)
            int i = 0;
            for (int32_t p = p0; p < nodes; p += kRunBlocks * kWarps, ++i)
                if (sd_mark_node<D, T, true>(S.sd, p, lane) && i < 64) drops |= uint64_t(1) << i;
            cluster.sync();
            i = 0;
            for (int32_t p = p0; p < nodes; p += kRunBlocks * kWarps, ++i) {
                if (i < 64 && !(drops >> i & 1)) continue;
                const int32_t gone = sd_compact_node<D, T, true>(S.sd, S.sd.order[p], lane);
                if (lane == 0 && gone > 0) atomicAdd(&S.removed, gone);
            }
            cluster.sync();
        }
    }
    // --- results (zeroed by the host): the blocks' own counts, block 0's totals
    __syncthreads();
    RunOut &O = *R.out;
    if (tid == 0) {
        if (tile_surv) atomicAdd(reinterpret_cast<unsigned long long *>(&O.tile_surv), tile_surv);
        if (stair) atomicAdd(reinterpret_cast<unsigned long long *>(&O.stair), stair);
        // the last layer's removals were told to nobody when the run went to its end
        const int64_t rest = d.layer + done == R.last ? S.removed : 0;
        const int64_t all = rest + (rank == 0 ? removed_total : 0);
        if (all) atomicAdd(reinterpret_cast<unsigned long long *>(&O.removed), static_cast<unsigned long long>(all));
    }
    if (rank == 0 && tid == 0) {
        O.done = done;
        O.cand_total = cand_total;
        O.cand_peak = cand_peak;
        O.surv_total = surv_total;
        O.surv_peak = surv_peak;
        const int x = d.layer + done;
        const RunFrom last = run_from(d, done);
        O.final_size = ld_live<true>(last.size);
        O.final_off = ld_live64<true>(last.off);
        run_count_job(*d.count, d, R.layer_off, x, x + 1, x < R.terminal, last.size);
    }
}

// Method 3: both sides, by the engine's rule.  The rule needs a side's next count, so a layer
// meets twice: when it is written, and when the layer after it is counted (which also
// gathers that layer's arcs, kept unless the other side goes next).
template <int D, typename T, bool LEX>
__global__ void __cluster_dims__(kRunBlocks, 1, 1) __launch_bounds__(kRunThreads, 1)
    run_meet_kernel(const RunJob *__restrict__ jobs) {
    constexpr int NT = kRunThreads;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    RunSmem<D, T, LEX> &S = *reinterpret_cast<RunSmem<D, T, LEX> *>(smem_raw);
    RunStage &st = S.st;
    cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    const RunJob &R = jobs[blockIdx.x / kRunBlocks];
    const int rank = static_cast<int>(blockIdx.x % kRunBlocks);
    const int tid = threadIdx.x;
    const int64_t region = static_cast<int64_t>(rank) * kRunRegion;
    int layer[2] = {R.td.layer, R.bu.layer}, done[2] = {0, 0};
    int64_t score[2] = {R.td.score, R.bu.score};
    unsigned long long tile_surv = 0, stair = 0;
    int64_t cand_total = 0, cand_peak = 0, surv_total = 0, surv_peak = 0;
    int staged = -1;  // the side whose next layer's arcs are gathered
    int64_t cand = 0;
    bool bad = false;
    RunShare h{};
    cluster.sync();  // every block has started: its shared memory may be written to
    for (int step = 0; step < R.steps && layer[1] - layer[0] > 1; ++step) {
        const int side = score[0] <= score[1] ? 0 : 1;
        const RunSide &d = side == 0 ? R.td : R.bu;
        const int dir = side == 0 ? 1 : -1;
        const int b = (done[side] + 1) & 1;
        const RunFrom from = run_from(d, done[side]);
        if (staged != side) {
            h = run_fetch(st, d, R.layer_off, layer[side], layer[side] + dir, rank);
            bad = h.nodes > R.vcap || h.a1 - h.a0 > kRunRegion;
            __syncthreads();
            if (!bad) cand = run_gather(st, from, h.a1 - h.a0, region, S.warp_l, &S.tot);
            bad |= cand > kRunRegion;
        }
        if (tid == 0) run_describe(S.J, R, d, h, from.pts, st, b, S.tile);
        __syncthreads();
        if (!bad) {
            if constexpr (LEX) lex_items<T, NT, true>(S.items, S.J, &st, h.v0, h.v1, []() {});
            else pair_items<D, T, NT, true>(S.items, S.J, &st, h.v0, h.v1, []() {});
            bad = st.over != 0;
        }
        if (tid < kRunBlocks) {
            RunPub *to = cluster.map_shared_rank(&S.pub[0][rank], tid);
            to->cand = cand;
            to->surv = static_cast<int64_t>(S.tile[0]);
            to->bad = bad ? 1 : 0;
        }
        __syncwarp();
        auto token = cluster.barrier_arrive();
        const int next = layer[side] + 2 * dir;  // its next layer, if the sides stay apart
        const bool count = layer[1] - layer[0] > 2;
        if (count) h = run_fetch(st, d, R.layer_off, layer[side] + dir, next, rank);
        cluster.barrier_wait(std::move(token));
        int64_t all_cand = 0, all_surv = 0, any_bad = 0;
#pragma unroll
        for (int r = 0; r < kRunBlocks; ++r) {
            all_cand += S.pub[0][r].cand;
            all_surv += S.pub[0][r].surv;
            any_bad |= S.pub[0][r].bad;
        }
        if (any_bad) break;  // every block of the cluster alike
        cand_total += all_cand;
        cand_peak = max(cand_peak, all_cand);
        surv_total += all_surv;
        surv_peak = max(surv_peak, all_surv);
        tile_surv += S.tile[0];
        stair += S.tile[1];
        layer[side] += dir;
        ++done[side];
        if (!count) break;  // one layer apart
        // --- the next layer's count on this side: its score
        bad = h.nodes > R.vcap || h.a1 - h.a0 > kRunRegion;
        __syncthreads();
        cand = 0;
        if (!bad) cand = run_gather(st, run_from(d, done[side]), h.a1 - h.a0, region, S.warp_l, &S.tot);
        if (tid < kRunBlocks) {
            RunPub *to = cluster.map_shared_rank(&S.pub[1][rank], tid);
            to->cand = cand;
            to->bad = bad ? 1 : 0;
        }
        cluster.sync();
        int64_t total = 0;
        any_bad = 0;
#pragma unroll
        for (int r = 0; r < kRunBlocks; ++r) {
            total += S.pub[1][r].cand;
            any_bad |= S.pub[1][r].bad;
        }
        if (any_bad) break;
        bad = cand > kRunRegion;
        score[side] = side == 0 ? total : static_cast<int64_t>(1.5 * static_cast<double>(total));
        staged = side;
    }
    __syncthreads();
    RunOut &O = *R.out;
    if (tid == 0) {
        if (tile_surv) atomicAdd(reinterpret_cast<unsigned long long *>(&O.tile_surv), tile_surv);
        if (stair) atomicAdd(reinterpret_cast<unsigned long long *>(&O.stair), stair);
    }
    if (rank == 0 && tid == 0) {
        O.done = done[0];
        O.done_bu = done[1];
        O.cand_total = cand_total;
        O.cand_peak = cand_peak;
        O.surv_total = surv_total;
        O.surv_peak = surv_peak;
        run_count_job(*R.td.count, R.td, R.layer_off, layer[0], layer[0] + 1, true, run_from(R.td, done[0]).size);
        run_count_job(*R.bu.count, R.bu, R.layer_off, layer[1], layer[1] - 1, true, run_from(R.bu, done[1]).size);
    }
}

namespace {

template <int D, typename T, bool LEX>
cudaError_t launch_run_t(bool meet, const RunJob *jobs, int num_jobs, cudaStream_t stream) {
    const size_t smem = sizeof(RunSmem<D, T, LEX>);
    auto *kernel = meet ? run_meet_kernel<D, T, LEX> : run_layers_kernel<D, T, LEX>;
    const cudaError_t e = ensure_smem_limit(reinterpret_cast<const void *>(kernel), smem);
    if (e != cudaSuccess) return e;
    kernel<<<static_cast<unsigned>(num_jobs) * kRunBlocks, kRunThreads, smem, stream>>>(jobs);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_layer_runs(int d, bool wide, bool lex, bool meet, const RunJob *jobs, int num_jobs,
                              cudaStream_t stream) {
    if (num_jobs <= 0) return cudaSuccess;
    if (lex && d == 3)
        return wide ? launch_run_t<3, int64_t, true>(meet, jobs, num_jobs, stream)
                    : launch_run_t<3, int32_t, true>(meet, jobs, num_jobs, stream);
    if (wide) { PMDD_DISPATCH_D(d, (launch_run_t<DD, int64_t, false>(meet, jobs, num_jobs, stream))); }
    PMDD_DISPATCH_D(d, (launch_run_t<DD, int32_t, false>(meet, jobs, num_jobs, stream)));
}

}  // namespace dev
}  // namespace pmdd
