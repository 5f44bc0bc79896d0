// Fused expand + dominance filter over candidate tiles, pairwise: every objective count but
// three.
//
// A tile owns every destination assigned to it by tile_plan_kernel (those whose
// candidate range starts inside the tile's window of J.tile_window <= kTileWindow
// candidates);
// destinations with at most kSmallMax candidates are handled here entirely in shared
// memory, larger ones only get their slot offset (the oversized path in big.cu filters
// them).  A tile therefore holds < kTileCap points.
//
//   stage:   the tile's destinations and their arcs (candidate offsets, parent slot
//            starts, weight rows) are read once into shared memory;
//   expand:  candidate = parent frontier point + arc weight vector; consecutive
//            candidates of an arc are consecutive parent points, so loads coalesce and
//            each candidate costs one independent global load;
//   filter:  each warp takes 32 candidates and sweeps the candidates of their
//            destinations with warp-uniform shared-memory broadcast reads, four at a time:
//            only when one of the four is >= a candidate is the keep rule applied (rare:
//            the candidate itself, or its dominator, after which it asks no more).  A warp
//            whose 32 lie in one arc's run skips that run (shifts of one non-dominated,
//            duplicate-free parent frontier never dominate each other), and a warp leaves
//            as soon as all 32 are decided;
//   write:   survivors go to the destination's slot in the next layer's frontier.
//
// Dominance rule (the reference GPU filter's dominates_or_tie_before,
// src/pmdd/enum/gpu/dominance_utils.cuh:10-23, and the weak-dominance insert of
// src/pmdd/enum/pareto_frontier.hpp:237-303): candidate q is dropped iff another
// candidate p of the same destination has p >= q on every objective and (p != q or p
// comes first).
//
// Bound by integer compares (half the issue rate).  Against a block of 512 threads whose 128
// registers let one run per SM, with an equality test beside every compare: tile time of
// KP d=4 n=60 12.9 -> 7.5 ms (37.5 M candidates), of its method 3 3.8 -> 2.9 ms, of TSP d=5
// n=13 1.9 -> 1.2 ms, of KP d=7 n=25 0.55 -> 0.36 ms (one B200).
#pragma once

#include "tile_pass.cuh"

namespace pmdd {
namespace dev {

// Points of 16 bytes make 61 KB a block: three blocks of 256 threads share an SM; points of 32
// bytes 93 KB, two blocks of 512; larger ones (int64, five objectives and more) 125-157 KB, one.
// The launch bounds ask for four or two, which holds every instance at 64 registers (int64
// points of five objectives and more spill 4-22 bytes, int32 ones of eight 8).
template <int D, typename T>
constexpr int pair_threads() {
    return sizeof(PackedPt<D, T>) <= 16 ? 256 : 512;
}

template <int D, typename T>
struct PairSmem {
    PackedPt<D, T> pts[kTileCap + 4];    // read four at a time
    TileArcs a;
    TileItems t;
    TileDraw draw;
};

// Filters destinations [i0, i1) of J; see above.  Every thread of a block of NT calls it;
// `st` with RUN.
template <int D, typename T, int NT, bool RUN, class Last>
__device__ __forceinline__ bool pair_items(PairSmem<D, T> &S, const ExpandJob &J, RunStage *st, int32_t i0, int32_t i1,
                                           Last last) {
    constexpr T kMost = sizeof(T) == 4 ? static_cast<T>(INT32_MAX) : static_cast<T>(INT64_MAX);
    TileItems &I = S.t;
    TileArcs &A = S.a;
    const int tid = threadIdx.x, lane = tid & 31;
    const T *prev = static_cast<const T *>(J.prev_pts);
    T *outp = static_cast<T *>(J.out_pts);
    bool called = false;
    for (int32_t ic = i0; ic < i1;) {
        const int n_it = stage_items<NT, RUN>(I, J, st, ic, i1, false);
        if (n_it == 0) {
            if (tid == 0) atomicOr(J.err, kErrBounds);
            return false;
        }
        const int32_t total = I.tot_i;
        stage_arcs<NT, RUN>(I, A, J, st, n_it);
        __syncthreads();
        assign_arcs<NT>(I, A);
        // --- expand: candidate = parent point + arc weight
        for (int q = tid; q < total; q += NT) {
            const int x = A.tag[q];
            const T *src = prev + (parent_slot<RUN>(A, J, st, x) + (q - A.arc_pos[x])) * D;
            const int32_t *w = J.weights + static_cast<int64_t>(A.arc_w[x]) * D;
            PackedPt<D, T> pt;
#pragma unroll
            for (int o = 0; o < PackedPt<D, T>::kPad; ++o)
                pt.v[o] = o < D ? ld_point<RUN>(src + (o < D ? o : 0)) + static_cast<T>(w[o < D ? o : 0]) : T(0);
            S.pts[q] = pt;
            I.item_of[q] = static_cast<uint16_t>(A.arc_item[x] & ~kUnsorted);
        }
        __syncthreads();
        // --- filter
        const int chunks = (total + 31) >> 5;
        while (true) {
            int c = 0;
            if (lane == 0) c = atomicAdd(&I.next_chunk, 1);
            c = __shfl_sync(kWarpAll, c, 0);
            if (c >= chunks) break;
            const int c0 = c << 5, q = c0 + lane;
            const bool valid = q < total;
            bool dom = !valid;
            const int k = I.item_of[valid ? q : c0];
            const int js = I.item_s[k], je = I.item_s[k + 1];
            T p[D];
            {
                const PackedPt<D, T> me = S.pts[valid ? q : c0];
#pragma unroll
                for (int o = 0; o < D; ++o) p[o] = valid ? me.v[o] : kMost;
            }
            // the keep rule against points [j, j + 4) within [a, b); a decided lane asks no more
            auto settle = [&](int j, int a, int b) {
#pragma unroll 1
                for (int u = 0; u < 4; ++u) {
                    const PackedPt<D, T> x = S.pts[j + u];
                    const int at = j + u;
                    if (at >= a && at < b && at != q && ge_all<D, T>(x, p) && (at < q || !eq_all<D, T>(x, p))) dom = true;
                }
                if (dom) {
#pragma unroll
                    for (int o = 0; o < D; ++o) p[o] = kMost;
                }
            };
            // sweeps [a, b): one destination, or (mixed) each lane within its own
            auto sweep = [&](int a, int b, bool mixed) -> bool {
                int it = 0;
                for (int j = a; j < b; j += 4) {
                    bool any = false;
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        bool ge = ge_all<D, T>(S.pts[j + u], p);
                        if (mixed) ge = ge && static_cast<unsigned>(j + u - js) < static_cast<unsigned>(je - js);
                        any |= ge;
                    }
                    if (any) settle(j, mixed ? max(a, js) : a, mixed ? min(b, je) : b);
                    if ((++it & 7) == 0 && __all_sync(kWarpAll, dom)) return true;
                }
                return __all_sync(kWarpAll, dom);
            };
            const int kf = __shfl_sync(kWarpAll, k, 0);
            const int kl = I.item_of[min(c0 + 31, total - 1)];
            if (kf == kl) {
                // all in one arc's run: the points before it, then those after it
                const int x0 = A.tag[c0], x1 = A.tag[min(c0 + 31, total - 1)];
                int lo = je, hi = je;
                if (x0 == x1) {
                    lo = A.arc_pos[x0];
                    hi = x0 + 1 < I.item_arc0[k + 1] ? A.arc_pos[x0 + 1] : je;
                }
                if (!sweep(js, lo, false)) sweep(hi, je, false);
            } else {
                sweep(I.item_s[kf], I.item_s[kl + 1], true);
            }
            const unsigned kept = __ballot_sync(kWarpAll, !dom);
            if (lane == 0) I.keep[c] = kept;
        }
        __syncthreads();
        // --- survivors before each chunk (one warp); another one draws the next tile
        if (tid < 32) scan_kept(I, J, chunks);
        if (ic + n_it >= i1) {
            called = true;
            if (tid >= 32 && tid < 64) last();
        }
        __syncthreads();
        // --- write survivors into each destination's slot
        for (int q = tid; q < total; q += NT) {
            if (((I.keep[q >> 5] >> (q & 31)) & 1u) == 0) continue;
            T *o_ = outp + slot_of(I, q) * D;
            const PackedPt<D, T> me = S.pts[q];
#pragma unroll
            for (int o = 0; o < D; ++o) o_[o] = me.v[o];
        }
        write_sizes<NT>(I, J, ic, n_it);
        __syncthreads();
        ic += n_it;
    }
    return called;
}

}  // namespace dev
}  // namespace pmdd
