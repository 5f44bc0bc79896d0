// Fused expand + dominance filter for three objectives, in lexicographic order.
//
// Every node's frontier is kept in descending lexicographic order (objective 0, then 1,
// then 2).  Adding an arc's weight vector to every point of a frontier keeps that order,
// so the candidates of one arc ("a run") arrive sorted, and a destination's candidates
// are a few sorted runs.  In that order a point can only be dominated by a point before
// it, and since every point before q has objective 0 >= q's, q is dominated (or a later
// copy of an equal point) iff some earlier point has objectives 1 and 2 both >= q's: a
// two-dimensional question.
//
//   stage:   as the pairwise tile kernel (tile.cu): destinations and their arcs, with
//            each arc's parent flag "frontier sorted";
//   expand:  candidate = parent point + arc weight, in run order;
//   merge:   each candidate's position in its destination's lexicographic order is its
//            index in its run plus, per other run, a binary search for how many of that
//            run's points come before it (equal points: the lower run first); the points of
//            a run from an unsorted parent are counted one by one;
//   filter:  a warp per chunk of 32 consecutive merged positions, whatever destinations
//            they belong to.  First every candidate against the 32 of its chunk (bit masks
//            of the ones >= it in objective 1, and in both); a destination that goes on
//            past the chunk leaves its staircase there: the chunk's survivors of that
//            destination by objective 1 descending, with the running maximum of objective
//            2, so that one binary search answers the question for the whole chunk.  Then,
//            after a barrier, the survivors of a destination that began in an earlier chunk
//            ask the staircases of the chunks in between (destinations of at most
//            J.pair_max candidates: look at those points one by one);
//   write:   survivors go to the destination's slot in merged order, so the next
//            layer's runs are sorted again (out_sorted = 1).
//
// Every warp has the same work in the first half of the filter and one uniform loop in the
// second.  It replaced one staircase warp per 64-candidate segment, whose walks were serial
// chains of shuffles (51 % of the kernel's time, its warps 61 % busy): 1.68 G -> 0.93 G warp
// instructions on a captured launch of the 192-instance stream.  The kernel waits on
// barriers, shared-memory latency and dependent loads, not on a unit (issue slots 53 % busy,
// ALU 50 %): tile time of that stream's 684 M candidates 73.8 ms before, 49.7 ms with the
// chunk filter at 512 threads and 79 KB, 40.3 ms with four blocks of 256 threads per SM,
// the merge in place and the next tile fetched ahead, 38.3 ms with the sorts of kMergeRuns
// (one B200).
//
// The keep rule is the reference GPU filter's (src/pmdd/enum/gpu/dominance_utils.cuh:
// 10-23): q is dropped iff another candidate p of the destination has p >= q on every
// objective and (p != q or p comes first).  Of equal points the first in the merged order
// stays; which copy stays does not change the frontier.  Oversized destinations are
// left to big.cu, whose output is not in this order (out_sorted = 0): its runs are counted.
#pragma once

#include "tile_pass.cuh"

namespace pmdd {
namespace dev {

// 256 threads and 54 KB of shared memory (int32): four blocks share an SM, so that one
// block's barriers and dependent loads are covered by the others (64 registers, 20 bytes of
// them spilled).  int64 points take 95 KB: two blocks of 128 registers.
constexpr int kLexThreads = 256;
// Destinations of more than kMergeRuns runs are sorted in shared memory instead of merged
// (a search per other run: hundreds on the last layers of a knapsack), and so are runs of
// more than kSortRun points from unsorted parents; shorter ones are counted.  Tile time of
// the 192-instance stream 40.5 ms without, 39.3 with the sorted runs, 38.3 - 38.8 with
// whole destinations sorted above 8, 16 or 32 runs, 40.8 above 4.
constexpr int kMergeRuns = 16;

template <typename T>
struct LexSmem {
    alignas(16) T p0[kTileCap], p1[kTileCap], p2[kTileCap];  // candidates: run order, then merged order
    union {
        TileArcs a;                        // for the merge; its tags become merged positions
        struct {
            T s1[kTileCap], s2[kTileCap];  // chunk staircases: objective 1 descending, running
        } f;                               // maximum of objective 2
    };
    TileItems t;
    TileDraw draw;
};

template <typename T>
__device__ __forceinline__ T lowest() {
    return sizeof(T) == 4 ? static_cast<T>(INT32_MIN) : static_cast<T>(INT64_MIN);
}

// Bits j of the chunk's 32 positions at c0 with m1[c0 + j] >= q1 (*ge1, with WITH_GE1) and
// with both objectives >= (q1, q2) (returned).  Warp-uniform addresses, 16 bytes at a time.
template <typename T, bool WITH_GE1>
__device__ __forceinline__ unsigned chunk_masks(const T *m1, const T *m2, T q1, T q2, unsigned *ge1) {
    struct alignas(16) V {
        T v[16 / sizeof(T)];
    };
    constexpr int W = 16 / sizeof(T);
    unsigned both = 0, g1 = 0;
#pragma unroll
    for (int j = 0; j < 32; j += W) {
        const V a = *reinterpret_cast<const V *>(m1 + j);
        const V b = *reinterpret_cast<const V *>(m2 + j);
#pragma unroll
        for (int u = 0; u < W; ++u) {
            const bool g = a.v[u] >= q1;
            if (WITH_GE1 && g) g1 |= 1u << (j + u);
            if (g && b.v[u] >= q2) both |= 1u << (j + u);
        }
    }
    if (WITH_GE1) *ge1 = g1;
    return both;
}

// Has the staircase at s1 / s2 (32 entries) a point >= (q1, q2) in both?
template <typename T>
__device__ __forceinline__ bool stair_covers(const T *s1, const T *s2, T q1, T q2) {
    int at = 0;  // entries with objective 1 >= q1
#pragma unroll
    for (int step = 16; step > 0; step >>= 1)
        if (s1[at + step - 1] >= q1) at += step;
    if (s1[at] >= q1) ++at;  // at <= 31: the 32nd entry
    return at > 0 && s2[at - 1] >= q2;
}

__device__ __forceinline__ bool sorts_whole(const TileItems &I, int k) {
    return I.item_arc0[k + 1] - I.item_arc0[k] > kMergeRuns && I.item_s[k + 1] - I.item_s[k] > kSortRun;
}

// Sorts positions [lo, lo + n) of the candidates in descending lexicographic order (the whole
// block; Batcher's odd-even mergesort, whose comparators all point one way, so that n need
// not be a power of two).
template <typename T, int NT>
__device__ __forceinline__ void sort_run(LexSmem<T> &S, int lo, int n) {
    for (int p = 1; p < n; p <<= 1)
        for (int k = p; k >= 1; k >>= 1) {
            const int j0 = k & (p - 1);  // 0 in the first round of a merge, else k
            for (int t = threadIdx.x;; t += NT) {
                const int a = j0 + (((t & ~(k - 1)) << 1) | (t & (k - 1)));
                if (a + k >= n) break;
                if (((a ^ (a + k)) & ~(2 * p - 1)) != 0) continue;  // not in the same pair of blocks
                const int u = lo + a, v = u + k;
                const T u0 = S.p0[u], v0 = S.p0[v];
                if (u0 > v0) continue;
                const T u1 = S.p1[u], v1 = S.p1[v], u2 = S.p2[u], v2 = S.p2[v];
                if (u0 == v0 && (u1 > v1 || (u1 == v1 && u2 >= v2))) continue;
                S.p0[u] = v0;
                S.p0[v] = u0;
                S.p1[u] = v1;
                S.p1[v] = u1;
                S.p2[u] = v2;
                S.p2[v] = u2;
            }
            __syncthreads();
        }
}

// Filters destinations [i0, i1) of J; see above.  Every thread of a block of NT calls it;
// `st` with RUN.
template <typename T, int NT, bool RUN, class Last>
__device__ __forceinline__ bool lex_items(LexSmem<T> &S, const ExpandJob &J, RunStage *st, int32_t i0, int32_t i1,
                                          Last last) {
    TileItems &I = S.t;
    TileArcs &A = S.a;
    const int tid = threadIdx.x, lane = tid & 31;
    const unsigned lt_mask = (1u << lane) - 1u;
    const T *prev = static_cast<const T *>(J.prev_pts);
    T *outp = static_cast<T *>(J.out_pts);
    const int pair_max = J.pair_max;
    PhaseClock clk{tid == 0 ? J.phase_clk : nullptr, 0};
    clk.start();
    bool called = false;
    for (int32_t ic = i0; ic < i1;) {
        const int n_it = stage_items<NT, RUN>(I, J, st, ic, i1, true);
        if (n_it == 0) {
            if (tid == 0) atomicOr(J.err, kErrBounds);
            return false;
        }
        const int32_t total = I.tot_i;
        clk.lap(0);
        stage_arcs<NT, RUN>(I, A, J, st, n_it);
        __syncthreads();
        clk.lap(1);
        assign_arcs<NT>(I, A);
        clk.lap(2);
        // --- expand: candidate = parent point + arc weight (run order)
        for (int q = tid; q < total; q += NT) {
            const int x = A.tag[q];
            const T *src = prev + (parent_slot<RUN>(A, J, st, x) + (q - A.arc_pos[x])) * 3;
            const int32_t *w = J.weights + static_cast<int64_t>(A.arc_w[x]) * 3;
            S.p0[q] = ld_point<RUN>(src) + static_cast<T>(w[0]);
            S.p1[q] = ld_point<RUN>(src + 1) + static_cast<T>(w[1]);
            S.p2[q] = ld_point<RUN>(src + 2) + static_cast<T>(w[2]);
            I.item_of[q] = static_cast<uint16_t>(A.arc_item[x] & ~kUnsorted);
        }
        // --- sort destinations of many runs, and the longer runs of unsorted parents
        for (int k = tid; k < n_it; k += NT)
            if (sorts_whole(I, k)) I.sort_list[atomicAdd(&I.n_sort, 1)] = static_cast<int16_t>(~k);
        for (int x = tid; x < I.tot_a; x += NT)
            if ((A.arc_item[x] & kUnsorted) && A.arc_pos[x + 1] - A.arc_pos[x] > kSortRun &&
                !sorts_whole(I, A.arc_item[x] & ~kUnsorted))
                I.sort_list[atomicAdd(&I.n_sort, 1)] = static_cast<int16_t>(x);
        __syncthreads();
        for (int i = 0; i < I.n_sort; ++i) {
            const int x = I.sort_list[i];
            if (x < 0) {
                sort_run<T, NT>(S, I.item_s[~x], I.item_s[~x + 1] - I.item_s[~x]);
            } else {
                if (tid == 0) A.arc_item[x] &= ~kUnsorted;
                sort_run<T, NT>(S, A.arc_pos[x], A.arc_pos[x + 1] - A.arc_pos[x]);
            }
        }
        clk.lap(3);
        // --- merge: each candidate's position in its destination's lexicographic order
        for (int q = tid; q < total; q += NT) {
            const int k = I.item_of[q];
            const int x = A.tag[q];
            const int js = I.item_s[k], je = I.item_s[k + 1];
            const T q0 = S.p0[q], q1 = S.p1[q], q2 = S.p2[q];
            // is position j's point before this one (equal points: if `tie`)?
            auto before = [&](int j, bool tie) -> bool {
                const T c0 = S.p0[j];
                if (c0 != q0) return c0 > q0;
                const T c1 = S.p1[j], c2 = S.p2[j];
                if (c1 != q1) return c1 > q1;
                if (c2 != q2) return c2 > q2;
                return tie;
            };
            int rank = 0;
            const int y0 = I.item_arc0[k], y1 = I.item_arc0[k + 1];
            const bool whole = sorts_whole(I, k);
            if (whole) rank = q - js;  // in order already
            for (int y = whole ? y1 : y0; y < y1; ++y) {
                const int lo = A.arc_pos[y], hi = (y + 1 < y1) ? A.arc_pos[y + 1] : je;
                if (A.arc_item[y] & kUnsorted) {  // a run in no order: count
                    for (int j = lo; j < hi; ++j) rank += before(j, j < q) ? 1 : 0;
                } else if (y == x) {
                    rank += q - lo;
                } else {
                    // points of run y before me: larger, or equal in a lower run; a prefix
                    int a = lo, b = hi;
                    while (a < b) {
                        const int mid = (a + b) >> 1;
                        if (before(mid, y < x)) a = mid + 1;
                        else b = mid;
                    }
                    rank += a - lo;
                }
            }
            A.tag[q] = static_cast<int16_t>(js + rank);
        }
        {  // in place: every thread picks its candidates up before any is put down
            constexpr int QP = kTileCap / NT;
            T v0[QP], v1[QP], v2[QP];
            int16_t to[QP];
#pragma unroll
            for (int r = 0; r < QP; ++r) {
                const int q = tid + r * NT;
                to[r] = -1;
                if (q < total) {
                    to[r] = A.tag[q];
                    v0[r] = S.p0[q];
                    v1[r] = S.p1[q];
                    v2[r] = S.p2[q];
                }
            }
            __syncthreads();
#pragma unroll
            for (int r = 0; r < QP; ++r)
                if (to[r] >= 0) {
                    S.p0[to[r]] = v0[r];
                    S.p1[to[r]] = v1[r];
                    S.p2[to[r]] = v2[r];
                }
        }
        __syncthreads();
        clk.lap(4);
        const int chunks = (total + 31) >> 5;
        // --- filter inside the chunks, and the staircases of destinations that go on
        for (int c = tid >> 5; c < chunks; c += NT / 32) {
            const int c0 = c << 5, q = c0 + lane;
            const bool valid = q < total;
            const T q1 = S.p1[q], q2 = S.p2[q];
            const int k = I.item_of[valid ? q : c0];
            const int js = I.item_s[k];
            // the chunk's candidates of the same destination before this one
            const unsigned mine = js > c0 ? ~((1u << (js - c0)) - 1u) : kWarpAll;
            const int kl = __shfl_sync(kWarpAll, k, 31);
            if (c0 + 32 >= total || I.item_s[kl + 1] <= c0 + 32) {
                const unsigned both = chunk_masks<T, false>(S.p1 + c0, S.p2 + c0, q1, q2, nullptr);
                const unsigned kept = __ballot_sync(kWarpAll, valid && (both & mine & lt_mask) == 0);
                if (lane == 0) I.keep[c] = kept;
            } else {
                unsigned ge1;
                const unsigned both = chunk_masks<T, true>(S.p1 + c0, S.p2 + c0, q1, q2, &ge1);
                const unsigned kept = __ballot_sync(kWarpAll, (both & mine & lt_mask) == 0);
                const unsigned members = kept & __ballot_sync(kWarpAll, k == kl);
                const unsigned equal = __match_any_sync(kWarpAll, q1);
                T *s1 = S.f.s1 + c0, *s2 = S.f.s2 + c0;
                if ((members >> lane) & 1u) {
                    const int at = __popc(members & ge1 & (~equal | lt_mask));
                    s1[at] = q1;
                    s2[at] = q2;
                }
                if (lane >= __popc(members)) {
                    s1[lane] = lowest<T>();
                    s2[lane] = lowest<T>();
                }
                __syncwarp();
                T mx = s2[lane];
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const T y = __shfl_up_sync(kWarpAll, mx, o);
                    if (lane >= o) mx = max(mx, y);
                }
                s2[lane] = mx;
                if (lane == 0) I.keep[c] = kept;
            }
        }
        __syncthreads();
        // --- filter against the earlier chunks of the destination that reaches into the
        // chunk (at most one), the longest loops first
        while (true) {
            int c = 0;
            if (lane == 0) c = chunks - 1 - atomicAdd(&I.next_chunk, 1);
            c = __shfl_sync(kWarpAll, c, 0);
            if (c <= 0) break;
            const int c0 = c << 5;
            const int k = I.item_of[c0];
            const int js = I.item_s[k], je = I.item_s[k + 1];
            if (js >= c0) continue;
            const int q = c0 + lane;
            const T q1 = S.p1[q], q2 = S.p2[q];
            const unsigned kept = I.keep[c];
            bool dom = q >= je || ((kept >> lane) & 1u) == 0;
            const unsigned others = je - c0 >= 32 ? 0u : kept & ~((1u << (je - c0)) - 1u);
            if (je - js <= pair_max) {
                for (int j = js; j < c0; ++j) dom |= (S.p1[j] >= q1) & (S.p2[j] >= q2);
            } else {
                for (int t = js >> 5; t < c && !__all_sync(kWarpAll, dom); ++t)
                    dom |= stair_covers<T>(S.f.s1 + (t << 5), S.f.s2 + (t << 5), q1, q2);
            }
            const unsigned left = __ballot_sync(kWarpAll, !dom);
            if (lane == 0) I.keep[c] = left | others;
        }
        // candidates of destinations above the pairwise limit (statistics)
        if (J.tile_surv != nullptr)
            for (int k = tid; k < n_it; k += NT) {
                const int c = I.item_s[k + 1] - I.item_s[k];
                if (c > pair_max) atomicAdd(&I.n_stair, c);
            }
        __syncthreads();
        clk.lap(5);
        // --- survivors before each chunk (one warp); another one draws the next tile
        if (tid < 32) scan_kept(I, J, chunks);
        if (ic + n_it >= i1) {
            called = true;
            if (tid >= 32 && tid < 64) last();
        }
        __syncthreads();
        // --- write survivors into each destination's slot, in merged order
        for (int q = tid; q < total; q += NT) {
            if (((I.keep[q >> 5] >> (q & 31)) & 1u) == 0) continue;
            T *o_ = outp + slot_of(I, q) * 3;
            o_[0] = S.p0[q];
            o_[1] = S.p1[q];
            o_[2] = S.p2[q];
        }
        write_sizes<NT>(I, J, ic, n_it);
        __syncthreads();
        clk.lap(6);
        ic += n_it;
    }
    return called;
}

}  // namespace dev
}  // namespace pmdd
