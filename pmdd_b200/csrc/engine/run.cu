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
// One B200, a layer: about 10 us, a chain of dependent loads, block barriers and the cluster's,
// against 23 us for the two launches of a chained one.  KP d=3 n=20: 21 layers in 0.21 ms (call 0.77 -> 0.37 ms); set packing d=3 n=100: 1.1
// ms (3.0 -> 1.27 ms); n=91 with state dominance, which ordinary steps take one layer at a
// time: 2.7 ms (8.9 -> 5.1 ms).
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
    int32_t x0, y0, nodes, v0, v1, a0, a1;
};

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
    const int rank = static_cast<int>(blockIdx.x % kRunBlocks);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t region = static_cast<int64_t>(rank) * kRunRegion;
    // the share of layer y, with its arcs' neighbours and weight rows fetched (as many as fit)
    auto fetch = [&](int y) -> RunShare {
        RunShare h;
        h.x0 = R.layer_off[y - 1];
        h.y0 = R.layer_off[y];
        h.nodes = R.layer_off[y + 1] - h.y0;
        h.v0 = static_cast<int32_t>(static_cast<int64_t>(h.nodes) * rank / kRunBlocks);
        h.v1 = static_cast<int32_t>(static_cast<int64_t>(h.nodes) * (rank + 1) / kRunBlocks);
        h.a0 = R.item_arc_off[h.y0 + h.v0];
        h.a1 = R.item_arc_off[h.y0 + h.v1];
        for (int32_t k = tid; k < min(h.a1 - h.a0, kRunRegion); k += NT) {
            st.nbr[k] = R.arc_nbr[h.a0 + k] - h.x0;
            st.w[k] = R.arc_wrow[h.a0 + k];
        }
        for (int32_t i = h.v0 + tid; i <= h.v1; i += NT)
            asm volatile("prefetch.global.L1 [%0];" ::"l"(R.item_arc_off + h.y0 + i));
        return h;
    };
    int done = 0;
    int64_t removed_total = 0, before_surv = 0;
    unsigned long long tile_surv = 0, stair = 0;
    int64_t cand_total = 0, cand_peak = 0, surv_total = 0, surv_peak = 0;
    if (tid == 0) S.removed = 0;
    RunShare h = fetch(R.layer + 1);
    cluster.sync();  // every block has started: its shared memory may be written to
    for (int y = R.layer + 1; y <= R.last; ++y) {
        const int b = (y - R.layer) & 1;
        const int64_t *x_off = done == 0 ? R.off : R.b_off[b ^ 1];
        const int32_t *x_size = done == 0 ? R.size : R.b_size[b ^ 1];
        const uint8_t *x_sorted = done == 0 ? R.sorted : R.b_sorted[b ^ 1];
        const int32_t arcs = h.a1 - h.a0;
        bool bad = h.nodes > R.vcap || arcs > kRunRegion;
        if (tid == 0) {
            S.tile[0] = S.tile[1] = 0;
            st.over = 0;
            ExpandJob &J = S.J;
            J.item_arc_off = R.item_arc_off;
            J.weights = R.weights;
            J.arc_cand_off = st.off;
            J.arc_base = h.a0;
            J.item_base = h.y0;
            J.num_items = h.nodes;
            J.prev_pts = done == 0 ? R.pts : R.b_pts[b ^ 1];
            J.out_pts = R.b_pts[b];
            J.out_off = R.b_off[b];
            J.out_size = R.b_size[b];
            J.out_sorted = R.b_sorted[b];
            J.err = R.err;
            J.tile_surv = S.tile;
            J.pair_max = R.pair_max;
            J.phase_clk = nullptr;
        }
        __syncthreads();
        // --- candidate offsets of this block's arcs, within its region
        int64_t cand = 0;
        if (!bad) {
            constexpr int PER = kRunRegion / NT;
            int32_t c[PER];
            int64_t mine = 0;
#pragma unroll
            for (int r = 0; r < PER; ++r) {
                const int k = tid * PER + r;
                c[r] = 0;
                if (k < arcs) {
                    const int32_t nb = st.nbr[k];
                    c[r] = ld_live<true>(x_size + nb);
                    st.src[k] = ld_live64<true>(x_off + nb);
                    st.sorted[k] = ld_live<true>(reinterpret_cast<const unsigned char *>(x_sorted) + nb);
                }
                mine += c[r];
            }
            int64_t at = region + block_exclusive_scan<int64_t, NT>(mine, S.warp_l, &S.tot);
            cand = S.tot;
#pragma unroll
            for (int r = 0; r < PER; ++r) {
                const int k = tid * PER + r;
                if (k < arcs) st.off[k] = at;
                at += c[r];
            }
            if (tid == 0) st.off[arcs] = region + cand;
            bad = cand > kRunRegion;
            __syncthreads();
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
        if (y < R.last) h = fetch(y + 1);
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
                sd.in_off = R.item_arc_off;
                sd.arc_src = R.arc_nbr;
                sd.arc_w = R.arc_wrow;
                sd.pts = R.b_pts[b];
                sd.off = R.b_off[b];
                sd.size = R.b_size[b];
                sd.keep = R.keep;
                sd.removed = nullptr;
                sd.node_base = y0;
                sd.num_nodes = nodes;
                sd.kind = R.sd_kind;
                sd.state_words = R.state_words;
            }
            __syncthreads();
            constexpr int kWarps = NT / 32;
            for (int32_t n = rank * kWarps + warp; n < nodes; n += kRunBlocks * kWarps)
                sd_mark_node<D, T, true>(S.sd, n, lane);
            cluster.sync();
            for (int32_t n = rank * kWarps + warp; n < nodes; n += kRunBlocks * kWarps) {
                const int32_t gone = sd_compact_node<D, T, true>(S.sd, n, lane);
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
        const int64_t rest = R.layer + done == R.last ? S.removed : 0;
        const int64_t all = rest + (rank == 0 ? removed_total : 0);
        if (all) atomicAdd(reinterpret_cast<unsigned long long *>(&O.removed), static_cast<unsigned long long>(all));
    }
    if (rank == 0 && tid == 0) {
        O.done = done;
        O.cand_total = cand_total;
        O.cand_peak = cand_peak;
        O.surv_total = surv_total;
        O.surv_peak = surv_peak;
        const int x = R.layer + done, b = done & 1;
        const int32_t *x_size = done == 0 ? R.size : R.b_size[b];
        O.final_size = ld_live<true>(x_size);
        O.final_off = ld_live64<true>(done == 0 ? R.off : R.b_off[b]);
        CountJob &C = *R.count;
        const bool more = x < R.terminal;  // a layer follows: its count
        const int32_t x0 = R.layer_off[x], y0 = R.layer_off[x + 1];
        C.cur_base = x0;
        C.cur_nodes = more ? y0 - x0 : 0;
        C.cur_size = x_size;
        C.arc_base = more ? R.item_arc_off[y0] : 0;
        C.num_arcs = more ? R.item_arc_off[R.layer_off[x + 2]] - C.arc_base : 0;
        C.item_base = y0;
        C.num_items = more ? R.layer_off[x + 2] - y0 : 0;
    }
}

namespace {

template <int D, typename T, bool LEX>
cudaError_t launch_run_t(const RunJob *jobs, int num_jobs, cudaStream_t stream) {
    const size_t smem = sizeof(RunSmem<D, T, LEX>);
    const cudaError_t e = ensure_smem_limit(reinterpret_cast<const void *>(run_layers_kernel<D, T, LEX>), smem);
    if (e != cudaSuccess) return e;
    run_layers_kernel<D, T, LEX><<<static_cast<unsigned>(num_jobs) * kRunBlocks, kRunThreads, smem, stream>>>(jobs);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_layer_runs(int d, bool wide, bool lex, const RunJob *jobs, int num_jobs, cudaStream_t stream) {
    if (num_jobs <= 0) return cudaSuccess;
    if (lex && d == 3)
        return wide ? launch_run_t<3, int64_t, true>(jobs, num_jobs, stream)
                    : launch_run_t<3, int32_t, true>(jobs, num_jobs, stream);
    if (wide) { PMDD_DISPATCH_D(d, (launch_run_t<DD, int64_t, false>(jobs, num_jobs, stream))); }
    PMDD_DISPATCH_D(d, (launch_run_t<DD, int32_t, false>(jobs, num_jobs, stream)));
}

}  // namespace dev
}  // namespace pmdd
