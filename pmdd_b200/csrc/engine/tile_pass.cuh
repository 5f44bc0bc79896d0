// One pass of a tile over some of its destinations, shared by the tile kernels (tile.cu,
// tile_lex.cu) and the layer-run kernel (run.cu): staging of destinations and arcs, the
// arc of each candidate, survivor masks to slot positions.
//
// RUN: the frontiers were written by other blocks of the same launch, so they are read past
// the L1 cache; what the arcs lead to was gathered beforehand (RunStage).
#pragma once

#include <climits>

#include "scan.cuh"

namespace pmdd {
namespace dev {

constexpr int kChunks = kTileCap / 32;
constexpr unsigned kWarpAll = 0xffffffffu;
constexpr int kSortRun = 32;

template <bool RUN, typename V>
__device__ __forceinline__ V ld_live(const V *p) {
    if constexpr (RUN) return __ldcg(p);
    else return *p;
}
// (int64_t and uint8_t have no overload of their own on every platform)
template <bool RUN>
__device__ __forceinline__ int64_t ld_live64(const int64_t *p) {
    if constexpr (RUN) return static_cast<int64_t>(__ldcg(reinterpret_cast<const long long *>(p)));
    else return *p;
}
template <bool RUN, typename T>
__device__ __forceinline__ T ld_point(const T *p) {
    if constexpr (sizeof(T) == 8) return static_cast<T>(ld_live64<RUN>(reinterpret_cast<const int64_t *>(p)));
    else return ld_live<RUN>(p);
}

// Destinations of a pass.
struct TileItems {
    uint16_t item_of[kTileCap];          // staged destination of each candidate
    uint32_t keep[kChunks];              // survivors of each 32 candidates
    int32_t kept_ex[kChunks];            // survivors before each 32
    int16_t item_s[kTileItemCap + 1];    // staged destination -> first candidate position
    int16_t item_arc0[kTileItemCap + 1]; // staged destination -> first staged arc
    int32_t item_a0g[kTileItemCap];      // staged destination -> first arc (global id)
    int64_t item_c0[kTileItemCap];       // staged destination -> job-local candidate start
    int64_t warp_l[32], tot_l;           // scans
    int32_t warp_i[32];
    int32_t tot_i, tot_a;
    int32_t next_chunk, n_stair, n_sort;
    int16_t sort_list[kTileCap / kSortRun];  // staged arcs whose runs are sorted first (lex_items.cuh)
};

// Their arcs.
constexpr int16_t kUnsorted = 0x4000;    // the run's parent frontier is in no order
struct TileArcs {
    int16_t tag[kTileCap];               // staged arc of each candidate
    int16_t arc_pos[kTileArcCap + 1];    // staged arc -> first candidate position
    int16_t arc_item[kTileArcCap];       // staged arc -> staged destination, | kUnsorted
    int32_t arc_w[kTileArcCap];          // staged arc -> weight row
    int32_t arc_nbr[kTileArcCap];        // staged arc -> job-local neighbour (RUN: RunStage index)
};

// Phase clock (J.phase_clk, a diagnostic): thread 0 adds the cycles its block spent in
// each phase of a pass (stage destinations, stage arcs, arc assignment, expand, merge,
// filter, scan and write) to the job's counters.
struct PhaseClock {
    unsigned long long *out;
    long long t;
    __device__ __forceinline__ void start() {
        if (out) t = clock64();
    }
    __device__ __forceinline__ void lap(int phase) {
        if (out) {
            const long long now = clock64();
            atomicAdd(out + phase, static_cast<unsigned long long>(now - t));
            t = now;
        }
    }
};

// Largest x over the threads before this one (-1 for thread 0); every thread calls it.
template <int THREADS>
__device__ __forceinline__ int32_t block_exclusive_max(int32_t x, int32_t *warp_buf) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int32_t inc = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int32_t y = __shfl_up_sync(kWarpAll, inc, o);
        if (lane >= o) inc = max(inc, y);
    }
    int32_t exc = __shfl_up_sync(kWarpAll, inc, 1);
    if (lane == 0) exc = -1;
    if (lane == 31) warp_buf[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        const int32_t w = lane < THREADS / 32 ? warp_buf[lane] : -1;
        int32_t winc = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int32_t y = __shfl_up_sync(kWarpAll, winc, o);
            if (lane >= o) winc = max(winc, y);
        }
        int32_t wexc = __shfl_up_sync(kWarpAll, winc, 1);
        if (lane == 0) wexc = -1;
        if (lane < THREADS / 32) warp_buf[lane] = wexc;
    }
    __syncthreads();
    const int32_t r = max(exc, warp_buf[warp]);
    __syncthreads();  // warp_buf may be reused right after
    return r;
}

// A run's arcs of one layer and block (run.cu): candidate offsets, and per arc its weight row
// and its neighbour's slot start and order flag.  J.arc_cand_off is `off`, J.arc_base the
// first arc.
constexpr int kRunRegion = 2048;         // arcs, and candidates, of a layer a block holds
struct RunStage {
    int64_t off[kRunRegion + 1];
    int64_t src[kRunRegion];
    int32_t nbr[kRunRegion];             // job-local neighbour
    int32_t w[kRunRegion];
    uint8_t sorted[kRunRegion];
    int32_t over;                        // an oversized destination was staged
};

// Stages destinations [ic, i1) of J as far as their candidates and arcs fit and returns how
// many (0: none, which well-formed plans rule out).  in_order: the pass writes frontiers
// in lexicographic order.  Every thread calls it; S.tot_i / S.tot_a receive the candidates
// and arcs.
template <int NT, bool RUN>
__device__ __forceinline__ int stage_items(TileItems &S, const ExpandJob &J, RunStage *st, int32_t ic, int32_t i1,
                                           bool in_order) {
    const int tid = threadIdx.x, lane = tid & 31;
    const int n_stage = min(kTileItemCap, i1 - ic);
    constexpr int PER = kTileItemCap / NT;
    static_assert(PER >= 1, "one destination per thread at least");
    int32_t cnt[PER], narc[PER];
    int32_t local = 0, local_a = 0;
#pragma unroll
    for (int r = 0; r < PER; ++r) {
        const int k = tid * PER + r;
        cnt[r] = 0;
        narc[r] = 0;
        if (k < n_stage) {
            const int32_t i = ic + k;
            const int32_t v = J.item_base + i;
            const int32_t a0 = J.item_arc_off[v], a1 = J.item_arc_off[v + 1];
            const int64_t s = J.arc_cand_off[a0 - J.arc_base];
            const int64_t c = J.arc_cand_off[a1 - J.arc_base] - s;
            J.out_off[i] = s;
            const bool resident = c > 0 && tile_resident(c, a1 - a0);
            if (RUN && c > 0 && !resident) st->over = 1;
            if (c == 0) J.out_size[i] = 0;
            if (J.out_sorted) J.out_sorted[i] = (c == 0 || (resident && in_order)) ? 1 : 0;
            S.item_c0[k] = s;
            S.item_a0g[k] = a0;
            if (resident) {
                cnt[r] = static_cast<int32_t>(c);
                narc[r] = a1 - a0;
            }
        }
        local += cnt[r];
        local_a += narc[r];
    }
    // candidates and arcs before this thread's destinations, in one scan
    const int64_t exl = block_exclusive_scan<int64_t, NT>((static_cast<int64_t>(local_a) << 32) | local, S.warp_l,
                                                          &S.tot_l);
    // the longest prefix of staged destinations whose candidates and arcs fit
    int fit = 0;
    int32_t end_s[PER], end_a[PER];  // where this thread's destinations end
    {
        int32_t run = static_cast<int32_t>(exl & 0xffffffff), runa = static_cast<int32_t>(exl >> 32);
#pragma unroll
        for (int r = 0; r < PER; ++r) {
            const int k = tid * PER + r;
            if (k < n_stage) {
                S.item_s[k] = static_cast<int16_t>(run);
                S.item_arc0[k] = static_cast<int16_t>(runa);
                if (runa + narc[r] <= kTileArcCap && run + cnt[r] <= kTileCap) fit = k + 1;
            }
            run += cnt[r];
            runa += narc[r];
            end_s[r] = run;
            end_a[r] = runa;
        }
    }
    fit = __reduce_max_sync(kWarpAll, fit);
    if (lane == 0) S.warp_i[tid >> 5] = fit;
    __syncthreads();
    int n_it = 0;
#pragma unroll
    for (int w = 0; w < NT / 32; ++w) n_it = max(n_it, S.warp_i[w]);
    if (n_it == 0) return 0;
    // end markers of this pass, from the thread that staged its last destination
#pragma unroll
    for (int r = 0; r < PER; ++r) {
        if (tid * PER + r == n_it - 1) {
            S.item_s[n_it] = static_cast<int16_t>(end_s[r]);
            S.item_arc0[n_it] = static_cast<int16_t>(end_a[r]);
            S.tot_i = end_s[r];
            S.tot_a = end_a[r];
        }
    }
    if (tid == 0) {
        S.next_chunk = 0;
        S.n_stair = 0;
        S.n_sort = 0;
    }
    __syncthreads();
    return n_it;
}

// Stages the arcs of the pass' n_it destinations (marking runs from unsorted parents) and
// clears the tags.  A barrier must follow.
template <int NT, bool RUN>
__device__ __forceinline__ void stage_arcs(TileItems &S, TileArcs &A, const ExpandJob &J, const RunStage *st, int n_it) {
    const int tid = threadIdx.x;
    const int32_t total = S.tot_i, total_a = S.tot_a;
    for (int x = tid; x < total_a; x += NT) {
        int lo = 0, hi = n_it - 1;  // destination owning staged arc x
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (S.item_arc0[mid] <= x) lo = mid;
            else hi = mid - 1;
        }
        const int k = lo;
        const int32_t a = S.item_a0g[k] + (x - S.item_arc0[k]);
        const int64_t c0 = J.arc_cand_off[a - J.arc_base];
        A.arc_pos[x] = static_cast<int16_t>(S.item_s[k] + (c0 - S.item_c0[k]));
        bool sorted;
        if constexpr (RUN) {
            A.arc_nbr[x] = a - J.arc_base;
            A.arc_w[x] = st->w[a - J.arc_base];
            sorted = st->sorted[a - J.arc_base] != 0;
        } else {
            const int32_t nb = J.arc_nbr[a] - J.prev_base;
            A.arc_nbr[x] = nb;
            A.arc_w[x] = J.arc_wrow[a];
            sorted = J.prev_sorted != nullptr && J.prev_sorted[nb] != 0;
        }
        A.arc_item[x] = static_cast<int16_t>(sorted ? k : k | kUnsorted);
    }
    if (tid == 0) A.arc_pos[total_a] = static_cast<int16_t>(total);
    for (int q = tid; q < total; q += NT) A.tag[q] = -1;
}

// Slot start of staged arc x's neighbour.
template <bool RUN>
__device__ __forceinline__ int64_t parent_slot(const TileArcs &A, const ExpandJob &J, const RunStage *st, int x) {
    if constexpr (RUN) return st->src[A.arc_nbr[x]];
    else return J.prev_off[A.arc_nbr[x]];
}

// Each candidate's arc: every non-empty run's first position is marked, then a block-wide
// running maximum carries the arc over its run.  Ends with a barrier.
template <int NT>
__device__ __forceinline__ void assign_arcs(TileItems &S, TileArcs &A) {
    const int tid = threadIdx.x;
    const int32_t total = S.tot_i, total_a = S.tot_a;
    for (int x = tid; x < total_a; x += NT)
        if (A.arc_pos[x + 1] > A.arc_pos[x]) A.tag[A.arc_pos[x]] = static_cast<int16_t>(x);
    __syncthreads();
    constexpr int QP = kTileCap / NT;
    int32_t run = -1, seen[QP];
#pragma unroll
    for (int r = 0; r < QP; ++r) {
        const int q = tid * QP + r;
        if (q < total) run = max(run, static_cast<int32_t>(A.tag[q]));
        seen[r] = run;
    }
    const int32_t before = block_exclusive_max<NT>(run, S.warp_i);
#pragma unroll
    for (int r = 0; r < QP; ++r) {
        const int q = tid * QP + r;
        if (q < total) A.tag[q] = static_cast<int16_t>(max(before, seen[r]));
    }
    __syncthreads();
}

// Survivors before each 32 candidates (the first warp calls it) and the tile statistics.
__device__ __forceinline__ void scan_kept(TileItems &S, const ExpandJob &J, int chunks) {
    static_assert(kChunks == 64, "two chunks per lane");
    const int lane = threadIdx.x & 31;
    const int a = 2 * lane < chunks ? __popc(S.keep[2 * lane]) : 0;
    const int b = 2 * lane + 1 < chunks ? __popc(S.keep[2 * lane + 1]) : 0;
    int inc = a + b;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(kWarpAll, inc, o);
        if (lane >= o) inc += y;
    }
    S.kept_ex[2 * lane] = inc - a - b;
    S.kept_ex[2 * lane + 1] = inc - b;
    if (lane == 31 && J.tile_surv != nullptr) {
        if (inc > 0) atomicAdd(J.tile_surv, static_cast<unsigned long long>(inc));
        if (S.n_stair > 0) atomicAdd(J.tile_surv + 1, static_cast<unsigned long long>(S.n_stair));
    }
}

// Survivors before candidate position q.
__device__ __forceinline__ int kept_before(const TileItems &S, int q) {
    if (q == 0) return 0;
    const int c = (q - 1) >> 5;
    return S.kept_ex[c] + __popc(S.keep[c] & (kWarpAll >> (31 - ((q - 1) & 31))));
}

// Slot position (points) of kept candidate q.
__device__ __forceinline__ int64_t slot_of(const TileItems &S, int q) {
    const int k = S.item_of[q];
    return S.item_c0[k] + (kept_before(S, q) - kept_before(S, S.item_s[k]));
}

template <int NT>
__device__ __forceinline__ void write_sizes(const TileItems &S, const ExpandJob &J, int32_t ic, int n_it) {
    for (int k = threadIdx.x; k < n_it; k += NT) {
        const int js = S.item_s[k], je = S.item_s[k + 1];
        if (je > js) J.out_size[ic + k] = kept_before(S, je) - kept_before(S, js);
    }
}

// A block's tiles from the launch's queue: the tile, its job and destinations.
struct TileDraw {
    int64_t tile[2];                     // this one, the next
    int32_t job[2], i0[2], i1[2];
};

// Draws a tile into slot `slot` (one warp calls it): its job is found 32 bases at a time.
__device__ __forceinline__ void draw_tile(TileDraw &S, int slot, const ExpandJob *jobs, const int64_t *tile_bases,
                                          int num_jobs, int64_t total_tiles, unsigned long long *queue) {
    const int lane = threadIdx.x & 31;
    int64_t t = 0;
    if (lane == 0) t = static_cast<int64_t>(atomicAdd(queue, 1ull));
    t = __shfl_sync(kWarpAll, t, 0);
    int j = 0;
    if (t < total_tiles) {
        int n = num_jobs;  // the last job in [j, j + n) whose first tile is <= t
        while (n > 1) {
            const int step = (n + 31) >> 5;
            const int at = j + lane * step;
            const unsigned m = __ballot_sync(kWarpAll, lane * step < n && __ldg(tile_bases + at) <= t);
            const int last = 31 - __clz(m | 1u);
            j += last * step;
            n = min(step, n - last * step);
        }
    }
    if (lane == 0) {
        S.tile[slot] = t;
        if (t < total_tiles) {
            const ExpandJob &J = jobs[j];
            const int64_t x = t - tile_bases[j];
            S.job[slot] = j;
            // a job sized on the device may have fewer tiles than the launch allows for
            S.i0[slot] = x < J.num_tiles ? J.tile_first[x] : 0;
            S.i1[slot] = x < J.num_tiles ? J.tile_first[x + 1] : 0;
        }
    }
}

// The tiles of a launch, drawn by its blocks: items(J, i0, i1, last) filters a tile's
// destinations and has one warp call last() while it finishes the final pass (returning
// whether it did).
template <class Items>
__device__ __forceinline__ void for_each_tile(TileDraw &S, const ExpandJob *jobs, const int64_t *tile_bases,
                                              int num_jobs, int64_t total_tiles, unsigned long long *queue,
                                              const int64_t *tiles_dev, Items items) {
    // jobs sized on the device (chain.cu) publish their tiles' total there
    if (tiles_dev != nullptr) total_tiles = min(total_tiles, *tiles_dev);
    int cur = 0;
    if (threadIdx.x < 32) draw_tile(S, 0, jobs, tile_bases, num_jobs, total_tiles, queue);
    __syncthreads();
    for (; S.tile[cur] < total_tiles; cur ^= 1) {
        const bool drawn = items(jobs[S.job[cur]], S.i0[cur], S.i1[cur], [&]() {
            draw_tile(S, cur ^ 1, jobs, tile_bases, num_jobs, total_tiles, queue);
        });
        if (!drawn) {  // an empty tile, or one given up
            if (threadIdx.x < 32) draw_tile(S, cur ^ 1, jobs, tile_bases, num_jobs, total_tiles, queue);
            __syncthreads();
        }
    }
}

}  // namespace dev
}  // namespace pmdd
