// State dominance of one node (statedom.cuh), by one warp: its labels marked against its
// partners', then its slot compacted.  Used by the state-dominance kernels (statedom.cu) and
// the layer-run kernel (run.cu), where RUN reads what other blocks wrote past the L1 cache.
#pragma once

#include "statedom.cuh"
#include "tile_pass.cuh"

namespace pmdd {
namespace dev {

// Arc index of a node's only incoming arc, or -1.
__device__ __forceinline__ int32_t single_in_arc(const StateDomJob &J, int32_t local) {
    const int32_t v = J.node_base + local;
    const int32_t a = J.in_off[v];
    return J.in_off[v + 1] - a == 1 ? a : -1;
}

// Lowest vertex of a set-packing state, or -1 for the empty state.
__device__ __forceinline__ int first_vertex(const uint64_t *s, int W) {
    for (int w = 0; w < W; ++w)
        if (s[w] != 0) return w * 64 + __ffsll(static_cast<long long>(s[w])) - 1;
    return -1;
}

// Keep flags of the labels of the node at position `pos` of the layer's order; whether any
// of them goes.  What a node needs is asked for at once, then waited for: one warp has one
// node in a small layer, and its loads in a row are the time.
template <int D, typename T, bool RUN>
__device__ __forceinline__ bool sd_mark_node(const StateDomJob &J, int32_t pos, int lane) {
    const int32_t n1 = J.order[pos];
    const int32_t s1 = ld_live<RUN>(J.size + n1);
    const int64_t o1 = ld_live64<RUN>(J.off + n1);
    const int32_t b1 = J.in_off[J.node_base + n1], e1 = J.in_off[J.node_base + n1 + 1];
    const int W = J.state_words;
    const uint64_t *st1 = J.state + static_cast<int64_t>(J.node_base + n1) * W;
    int32_t qb = 0, qe = 0;
    uint64_t w0 = 0;
    if (J.kind == 2) {
        qb = J.next[2 * pos];
        qe = J.next[2 * pos + 1];
        w0 = st1[0];
    }
    if (s1 == 0) return false;
    // siblings under one single parent (through different arc types) are not compared
    const int32_t a1 = e1 - b1 == 1 ? b1 : -1;
    auto skipped = [&](int32_t n2) -> bool {
        if (n2 < 0 || a1 < 0) return false;
        const int32_t a2 = single_in_arc(J, n2);
        return a2 >= 0 && J.arc_src[a1] == J.arc_src[a2] && ((J.arc_w[a1] != 0) != (J.arc_w[a2] != 0));
    };
    int32_t part0 = -1, part1 = -1;
    if (J.kind == 2) {
        // first node of the partner bucket with the same lowest vertex, not a
        // single-parent sibling, whose state contains n1's
        const int ff1 = w0 != 0 ? __ffsll(static_cast<long long>(w0)) - 1 : first_vertex(st1, W);
        for (int32_t p = qb; p < qe && part0 < 0; p += 32) {
            const int32_t q = p + lane;
            bool ok = false;
            if (q < qe) {
                const int32_t n2 = J.order[q];
                const uint64_t *st2 = J.state + static_cast<int64_t>(J.node_base + n2) * W;
                ok = (w0 & ~st2[0]) == 0;
                for (int w = 1; w < W; ++w) ok &= (st1[w] & ~st2[w]) == 0;
                // few contain the state: the rest of the test is theirs alone
                ok = ok && first_vertex(st2, W) == ff1 && !skipped(n2);
            }
            const unsigned m = __ballot_sync(kWarpAll, ok);
            if (m != 0) part0 = J.order[p + __ffs(m) - 1];
        }
    } else {
        // the next two positions of the order whose node holds labels
        int found = 0;
        for (int32_t p = pos + 1; p < J.num_nodes && found < 2; p += 32) {
            const int32_t q = p + lane;
            const bool act = q < J.num_nodes && ld_live<RUN>(J.size + J.order[q]) > 0;
            unsigned m = __ballot_sync(kWarpAll, act);
            while (m != 0 && found < 2) {
                const int b = __ffs(m) - 1;
                m &= m - 1;
                const int32_t node = J.order[p + b];
                if (found == 0) part0 = node;
                else part1 = node;
                ++found;
            }
        }
        if (skipped(part0)) part0 = -1;
        if (skipped(part1)) part1 = -1;
    }
    const T *P = static_cast<const T *>(J.pts);
    bool drops = false;
    for (int32_t kb = 0; kb < s1; kb += 32) {
        const int32_t k = kb + lane;
        const bool valid = k < s1;
        T x[D];
#pragma unroll
        for (int o = 0; o < D; ++o) x[o] = valid ? ld_point<RUN>(P + (o1 + k) * D + o) : T(0);
        bool dom = !valid;
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            const int32_t n2 = c == 0 ? part0 : part1;
            if (n2 < 0) continue;
            const int64_t o2 = ld_live64<RUN>(J.off + n2);
            const int32_t s2 = ld_live<RUN>(J.size + n2);
            for (int32_t tb = 0; tb < s2; tb += 32) {
                if (__all_sync(kWarpAll, dom)) break;
                T y[D];
#pragma unroll
                for (int o = 0; o < D; ++o) y[o] = tb + lane < s2 ? ld_point<RUN>(P + (o2 + tb + lane) * D + o) : T(0);
                const int n = min(s2 - tb, 32);
                for (int t = 0; t < n; ++t) {
                    bool ge = true;
#pragma unroll
                    for (int o = 0; o < D; ++o) ge &= (__shfl_sync(kWarpAll, y[o], t) >= x[o]);
                    dom |= ge;
                }
            }
        }
        if (valid) J.keep[o1 + k] = dom ? 0 : 1;
        drops |= __any_sync(kWarpAll, valid && dom);
    }
    return drops;
}

// Packs the kept labels of node n to the front of its slot; returns how many went.
template <int D, typename T, bool RUN>
__device__ __forceinline__ int32_t sd_compact_node(const StateDomJob &J, int32_t n, int lane) {
    const int32_t s = ld_live<RUN>(J.size + n);
    if (s == 0) return 0;
    T *P = static_cast<T *>(J.pts);
    const int64_t o = ld_live64<RUN>(J.off + n);
    int32_t kept = 0;
    for (int32_t kb = 0; kb < s; kb += 32) {
        const int32_t k = kb + lane;
        const bool keep = k < s && ld_live<RUN>(reinterpret_cast<const unsigned char *>(J.keep) + o + k) != 0;
        const unsigned m = __ballot_sync(kWarpAll, keep);
        const int32_t dst = kept + __popc(m & ((1u << lane) - 1u));
        const bool moves = keep && dst != k;
        T x[D];
#pragma unroll
        for (int q = 0; q < D; ++q) x[q] = moves ? ld_point<RUN>(P + (o + k) * D + q) : T(0);
        __syncwarp();  // every lane has loaded before any stores
        if (moves) {
#pragma unroll
            for (int q = 0; q < D; ++q) P[(o + dst) * D + q] = x[q];
        }
        kept += __popc(m);
        __syncwarp();
    }
    if (lane == 0 && kept != s) J.size[n] = kept;
    return s - kept;
}

}  // namespace dev
}  // namespace pmdd
