// Maxima of many point sets ("segments") at once, each spread over every SM: the filter
// of the oversized destinations (big.cu) and of standalone point sets (pareto.cu).
//
// What bounds a skyline of n points is the number of pairs compared.  On the oversized
// destinations of 4- and 5-objective diagrams 30-40 % of the candidates are maxima, so a
// pairwise sweep cannot exit early and costs the square of what it is given.  Here the
// rows that a few pivots leave are put in an order in which neighbours lie close in every
// objective, and a warp of 32 neighbouring rows skips every group of 8 rows whose
// componentwise maximum (its corner) no row of the warp lies under:
//
//   stats:    block per segment.  An even sample of up to 4096 points gives, per
//             objective, a 256-bin table from value to rank (so that the order adapts to
//             the distribution), and the pivots: the maxima of about 64 points of largest
//             objective sum;
//   prefilter: thread per point.  Points under a pivot are dropped, the pivots themselves
//             stay.  The others get a key, the interleaved leading bits
//             of their objectives' ranks read as a Gray code (so that neighbouring keys are
//             neighbouring cells: 17-24 % fewer pairs than the plain interleaving), of
//             log2(n / 16) bits, and their place within the key's bucket from one atomic;
//   scan:     block per segment: bucket counts to bucket starts;
//   scatter:  thread per point: the remaining rows into key order, padded for vector loads;
//   corner:   thread per group of 8 rows: the group's componentwise maximum;
//   mark:     warp per 32 rows: lanes test 32 corners at a time against the warp's
//             componentwise minimum, then the corners left against each row, and only the
//             groups left after that are compared row by row.  Survivors are appended to
//             the segment's output (order unspecified).
//
// A pivot only drops what it dominates or equals, and whatever dominates a remaining point
// is itself remaining or dominated by a remaining one, so the marked rows are exact for
// any pivots.
// Key, group size and pivot count come from a CPU model over the destinations of
// 3-, 4-, 5- and 7-objective knapsack and TSP diagrams: pairs compared per destination,
// against n * 4*sqrt(n) pivot tests plus all pairs of the remaining rows, fall 6.7-fold
// (TSP d=5 n=13), 4.3-fold (knapsack d=4 n=60), 6-fold (d=3 n=55); groups of 16 and 32
// compare 15 % and 40 % more, 32 or 128 pivots within 10 % of 64.  Integer compares run at
// half the issue rate: the mark kernel keeps the ALU pipe 64 % busy (ncu, TSP d=5 n=13);
// 4 blocks per SM instead of the 3 its registers allow are level (TSP d=5 5 % faster, KP
// d=4 2 % and KP d=7 13 % slower), 5 and 6 spill and are 7-60 % slower.
#pragma once

#include <climits>

#include "scan.cuh"

namespace pmdd {
namespace dev {

// A sorted row: padded to 16-byte multiples from three objectives on.
template <int D, typename T>
struct alignas(D == 1 ? sizeof(T) : D * sizeof(T) == 8 ? 8 : 16) SortedPt {
    static constexpr int kPad = D == 1 ? 1 : D == 2 ? 2 : PackedPt<D, T>::kPad;
    T v[kPad];
};

constexpr int kMaxPivots = 64;
constexpr int kMaxGroup = 8;          // rows per corner
constexpr int kMaxSample = 4096;
constexpr int kMaxStatThreads = 1024;
constexpr int kMaxThreads = 256;      // points per chunk (prefilter, scatter, mark)
constexpr int kMaxBins = 256;

// Per-segment head, in the segment's slab.
template <int D, typename T>
struct SegHead {
    uint32_t rows;                    // points the pivots left
    int32_t npiv;
    T mn[D];
    uint32_t range[D];                // sampled range, shifted right by shift
    uint32_t scale[D];                // bin = (x - mn >> shift) * scale >> 16
    int32_t shift[D];
    uint32_t piv_idx[kMaxPivots];
    alignas(4) uint8_t lut[D][kMaxBins];  // bin -> rank, 8 bits
    SortedPt<D, T> piv[kMaxPivots];
};

// One segment.  The slab holds rows | corners | bucket counts | head and takes at most
// 2 * n * D * sizeof(T) bytes for n > 1024 (seg_slab_bytes).
template <typename T>
struct Seg {
    const T *pts;                     // n points, D values each
    int64_t n;                        // < 2^32
    unsigned char *slab;
    uint32_t *key;                    // [n]
    uint32_t *place;                  // [n] place within the key's bucket
    T *out;                           // survivors, D values each
    int32_t *out_size;                // their number (nullptr with ordered output)
};

template <int D, typename T>
struct SegView {
    SortedPt<D, T> *rows;             // room for n rounded up to a group
    T *corner;                        // [D][groups]
    uint32_t *hist;                   // bucket counts, then bucket starts
    SegHead<D, T> *head;
    int64_t groups;                   // corner stride
    int32_t bits;
    size_t end;                       // slab bytes used
};

// Bits of the key: about 16 points (7 remaining ones) per bucket, at most the ranks' 8
// bits per objective.
template <int D>
__host__ __device__ inline int seg_bits(int64_t n) {
    int b = 0;
    while (b < 20 && b < 8 * D && (int64_t(32) << b) <= n) ++b;
    return b;
}

template <int D, typename T>
__host__ __device__ inline SegView<D, T> seg_view(unsigned char *slab, int64_t n) {
    SegView<D, T> v;
    uintptr_t p = reinterpret_cast<uintptr_t>(slab);
    auto up = [](uintptr_t x, uintptr_t a) { return (x + a - 1) / a * a; };
    p = up(p, 16);
    v.rows = reinterpret_cast<SortedPt<D, T> *>(p);
    v.groups = (n + kMaxGroup - 1) / kMaxGroup;
    p += sizeof(SortedPt<D, T>) * static_cast<size_t>(v.groups) * kMaxGroup;
    p = up(p, 16);
    v.corner = reinterpret_cast<T *>(p);
    p += sizeof(T) * D * static_cast<size_t>(v.groups);
    p = up(p, 4);
    v.hist = reinterpret_cast<uint32_t *>(p);
    v.bits = seg_bits<D>(n);
    p += sizeof(uint32_t) << v.bits;
    p = up(p, 16);
    v.head = reinterpret_cast<SegHead<D, T> *>(p);
    p += sizeof(SegHead<D, T>);
    v.end = static_cast<size_t>(p - reinterpret_cast<uintptr_t>(slab));
    return v;
}

// Slab bytes of n points whatever the slab's alignment.
template <int D, typename T>
__host__ __device__ inline size_t seg_slab_bytes(int64_t n) {
    return seg_view<D, T>(reinterpret_cast<unsigned char *>(static_cast<uintptr_t>(1024 + 1)), n).end;
}

template <typename T>
__device__ __forceinline__ T warp_min_of(T x) {
    if constexpr (sizeof(T) == 4) {
        return __reduce_min_sync(0xffffffffu, x);
    } else {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x = min(x, static_cast<T>(__shfl_xor_sync(0xffffffffu, static_cast<long long>(x), o)));
        return x;
    }
}

template <typename T>
__device__ __forceinline__ T type_max() {
    return sizeof(T) == 4 ? static_cast<T>(INT32_MAX) : static_cast<T>(INT64_MAX);
}
template <typename T>
__device__ __forceinline__ T type_min() {
    return sizeof(T) == 4 ? static_cast<T>(INT32_MIN) : static_cast<T>(INT64_MIN);
}

__device__ __forceinline__ void atomic_min_t(int32_t *p, int32_t x) { atomicMin(p, x); }
__device__ __forceinline__ void atomic_max_t(int32_t *p, int32_t x) { atomicMax(p, x); }
__device__ __forceinline__ void atomic_min_t(int64_t *p, int64_t x) {
    atomicMin(reinterpret_cast<long long *>(p), static_cast<long long>(x));
}
__device__ __forceinline__ void atomic_max_t(int64_t *p, int64_t x) {
    atomicMax(reinterpret_cast<long long *>(p), static_cast<long long>(x));
}

// x - mn without overflow, for x >= mn
template <typename T>
__device__ __forceinline__ uint64_t above(T x, T mn) {
    return sizeof(T) == 4 ? static_cast<uint64_t>(static_cast<uint32_t>(x) - static_cast<uint32_t>(mn))
                          : static_cast<uint64_t>(x) - static_cast<uint64_t>(mn);
}

template <typename T>
__device__ __forceinline__ int bin_of(T x, T mn, uint32_t range, uint32_t scale, int shift) {
    if (x <= mn) return 0;
    const uint64_t u = above<T>(x, mn) >> shift;
    return static_cast<int>((static_cast<uint64_t>(u < range ? u : range) * scale) >> 16);
}

template <int D, typename T, class Src>
__global__ void __launch_bounds__(kMaxStatThreads) maxima_stats_kernel(Src src) {
    constexpr int PER = kMaxSample / kMaxStatThreads;
    constexpr int SB = 1024;  // bins of the objective sum
    __shared__ T s_mn[D], s_mx[D];
    __shared__ unsigned long long s_smax, s_smin;  // sums, offset to unsigned order
    __shared__ int32_t s_hist[D * kMaxBins];
    __shared__ int32_t s_sum[SB];
    __shared__ int32_t s_from, s_npiv;
    __shared__ T s_piv[kMaxPivots][D];
    __shared__ uint32_t s_idx[kMaxPivots];
    __shared__ uint8_t s_drop[kMaxPivots];
    const int h = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (h >= src.count()) return;
    Seg<T> g;
    src.template seg<D>(h, &g);
    const SegView<D, T> v = seg_view<D, T>(g.slab, g.n);
    const int m = g.n < kMaxSample ? static_cast<int>(g.n) : kMaxSample;
    if (m <= 0) return;  // an empty segment (ordered output only): no chunks either
    if (tid < D) {
        s_mn[tid] = g.pts[tid];
        s_mx[tid] = g.pts[tid];
    }
    if (tid == 0) {
        s_smax = 0;
        s_smin = ~0ull;
        s_npiv = 0;
        if (g.out_size) *g.out_size = 0;
    }
    for (int k = tid; k < D * kMaxBins; k += kMaxStatThreads) s_hist[k] = 0;
    for (int k = tid; k < SB; k += kMaxStatThreads) s_sum[k] = 0;
    for (int64_t k = tid; k < (int64_t(1) << v.bits); k += kMaxStatThreads) v.hist[k] = 0;
    __syncthreads();
    // the sample, held in registers; an objective sum that wraps (int64) only changes the
    // choice of pivots
    T p[PER][D];
    unsigned long long sum[PER];
    uint32_t idx[PER];
    constexpr unsigned long long kBias = 1ull << 63;
#pragma unroll
    for (int r = 0; r < PER; ++r) {
        const int k = tid + r * kMaxStatThreads;
        sum[r] = 0;
        idx[r] = 0;
        if (k < m) {
            const int64_t i = static_cast<int64_t>(k) * g.n / m;
            idx[r] = static_cast<uint32_t>(i);
            unsigned long long s = 0;
#pragma unroll
            for (int o = 0; o < D; ++o) {
                p[r][o] = g.pts[i * D + o];
                s += static_cast<unsigned long long>(static_cast<long long>(p[r][o]));
            }
            sum[r] = s + kBias;
        } else {
#pragma unroll
            for (int o = 0; o < D; ++o) p[r][o] = g.pts[o];  // point 0: leaves the ranges as they are
        }
    }
#pragma unroll
    for (int o = 0; o < D; ++o) {
        T a = p[0][o], b = p[0][o];
#pragma unroll
        for (int r = 1; r < PER; ++r) {
            a = min(a, p[r][o]);
            b = max(b, p[r][o]);
        }
        for (int s = 16; s > 0; s >>= 1) {
            a = min(a, __shfl_xor_sync(0xffffffffu, a, s));
            b = max(b, __shfl_xor_sync(0xffffffffu, b, s));
        }
        if (lane == 0) {
            atomic_min_t(&s_mn[o], a);
            atomic_max_t(&s_mx[o], b);
        }
    }
    {
        unsigned long long a = ~0ull, b = 0;
#pragma unroll
        for (int r = 0; r < PER; ++r)
            if (tid + r * kMaxStatThreads < m) {
                a = min(a, sum[r]);
                b = max(b, sum[r]);
            }
        for (int s = 16; s > 0; s >>= 1) {
            a = min(a, __shfl_xor_sync(0xffffffffu, a, s));
            b = max(b, __shfl_xor_sync(0xffffffffu, b, s));
        }
        if (lane == 0) {
            atomicMin(&s_smin, a);
            atomicMax(&s_smax, b);
        }
    }
    __syncthreads();
    // bins: the range shifted into 16 bits, then scaled to 256
    if (tid < D) {
        const uint64_t rng = above<T>(s_mx[tid], s_mn[tid]);
        int sh = 0;
        while ((rng >> sh) > 0xffffull) ++sh;
        const uint32_t r16 = static_cast<uint32_t>(rng >> sh);
        v.head->mn[tid] = s_mn[tid];
        v.head->shift[tid] = sh;
        v.head->range[tid] = r16;
        v.head->scale[tid] = (static_cast<uint32_t>(kMaxBins) << 16) / (r16 + 1);
    }
    __syncthreads();
    const unsigned long long smin = s_smin, smax = s_smax;
    const unsigned long long swidth = (smax - smin) / SB + 1;
#pragma unroll
    for (int r = 0; r < PER; ++r) {
        if (tid + r * kMaxStatThreads < m) {
#pragma unroll
            for (int o = 0; o < D; ++o)
                atomicAdd(&s_hist[o * kMaxBins + bin_of<T>(p[r][o], v.head->mn[o], v.head->range[o], v.head->scale[o],
                                                           v.head->shift[o])],
                          1);
            atomicAdd(&s_sum[static_cast<int>((smax - sum[r]) / swidth)], 1);  // bin 0: largest sums
        }
    }
    __syncthreads();
    // bin -> rank: the share of the sample below the middle of the bin (warp per objective)
    for (int o = warp; o < D; o += kMaxStatThreads / 32) {
        int32_t c[kMaxBins / 32], run = 0;
#pragma unroll
        for (int k = 0; k < kMaxBins / 32; ++k) {
            c[k] = s_hist[o * kMaxBins + lane * (kMaxBins / 32) + k];
            run += c[k];
        }
        int32_t inc = run;
        for (int s = 1; s < 32; s <<= 1) {
            const int32_t y = __shfl_up_sync(0xffffffffu, inc, s);
            if (lane >= s) inc += y;
        }
        int32_t at = inc - run;
#pragma unroll
        for (int k = 0; k < kMaxBins / 32; ++k) {
            const int32_t q = static_cast<int32_t>((static_cast<int64_t>(2 * at + c[k]) * 128) / m);
            v.head->lut[o][lane * (kMaxBins / 32) + k] = static_cast<uint8_t>(q > 255 ? 255 : q);
            at += c[k];
        }
    }
    // the fewest top bins that hold kMaxPivots sampled points (the last warp)
    if (warp == kMaxStatThreads / 32 - 1) {
        int32_t c = 0;
        for (int k = 0; k < SB / 32; ++k) c += s_sum[lane * (SB / 32) + k];
        int32_t inc = c;
        for (int s = 1; s < 32; s <<= 1) {
            const int32_t y = __shfl_up_sync(0xffffffffu, inc, s);
            if (lane >= s) inc += y;
        }
        const unsigned hit = __ballot_sync(0xffffffffu, inc >= kMaxPivots);
        const int first = hit ? __ffs(hit) - 1 : 31;
        if (lane == first) {
            int32_t run = inc - c;
            int k = 0;
            for (; k < SB / 32 - 1; ++k) {
                run += s_sum[lane * (SB / 32) + k];
                if (run >= kMaxPivots) break;
            }
            s_from = lane * (SB / 32) + k;
        }
    }
    __syncthreads();
    const int from = s_from;
#pragma unroll
    for (int r = 0; r < PER; ++r) {
        if (tid + r * kMaxStatThreads < m && static_cast<int>((smax - sum[r]) / swidth) <= from) {
            const int at = atomicAdd(&s_npiv, 1);
            if (at < kMaxPivots) {
#pragma unroll
                for (int o = 0; o < D; ++o) s_piv[at][o] = p[r][o];
                s_idx[at] = idx[r];
            }
        }
    }
    __syncthreads();
    // the pivots' own maxima (of equal ones the first point), in point order
    const int np = s_npiv < kMaxPivots ? s_npiv : kMaxPivots;
    if (tid < np) {
        bool dom = false;
        for (int j = 0; j < np; ++j) {
            bool ge = true, eq = true;
#pragma unroll
            for (int o = 0; o < D; ++o) {
                ge &= s_piv[j][o] >= s_piv[tid][o];
                eq &= s_piv[j][o] == s_piv[tid][o];
            }
            dom |= ge && (!eq || s_idx[j] < s_idx[tid]);
        }
        s_drop[tid] = dom ? 1 : 0;
    }
    __syncthreads();
    if (tid < np && !s_drop[tid]) {
        int at = 0;
        for (int j = 0; j < np; ++j) at += (!s_drop[j] && s_idx[j] < s_idx[tid]) ? 1 : 0;
        SortedPt<D, T> q;
#pragma unroll
        for (int o = 0; o < SortedPt<D, T>::kPad; ++o) q.v[o] = o < D ? s_piv[tid][o < D ? o : 0] : T(0);
        v.head->piv[at] = q;
        v.head->piv_idx[at] = s_idx[tid];
    }
    if (tid == 0) {
        int kept = 0;
        for (int j = 0; j < np; ++j) kept += s_drop[j] ? 0 : 1;
        v.head->npiv = kept;
    }
}

template <int D, typename T, class Src>
__global__ void __launch_bounds__(kMaxThreads) maxima_prefilter_kernel(Src src) {
    __shared__ SortedPt<D, T> s_piv[kMaxPivots];
    __shared__ uint32_t s_idx[kMaxPivots];
    __shared__ alignas(4) uint8_t s_lut[D][kMaxBins];  // copied a word at a time
    int h;
    int64_t base;
    if (!src.chunk(blockIdx.x, &h, &base)) return;
    Seg<T> g;
    src.template seg<D>(h, &g);
    const SegView<D, T> v = seg_view<D, T>(g.slab, g.n);
    const int npiv = v.head->npiv;
    const int tid = threadIdx.x;
    if (tid < npiv) {
        s_piv[tid] = v.head->piv[tid];
        s_idx[tid] = v.head->piv_idx[tid];
    }
    for (int k = tid; k < D * kMaxBins / 4; k += kMaxThreads)
        reinterpret_cast<uint32_t *>(&s_lut[0][0])[k] = reinterpret_cast<const uint32_t *>(&v.head->lut[0][0])[k];
    __syncthreads();
    const int64_t i = base + tid;
    const bool valid = i < g.n;
    T p[D];
#pragma unroll
    for (int o = 0; o < D; ++o) p[o] = valid ? g.pts[i * D + o] : T(0);
    bool dom = !valid;
    for (int j = 0; j < npiv; ++j) {
        const SortedPt<D, T> c = s_piv[j];
        bool ge = true;
#pragma unroll
        for (int o = 0; o < D; ++o) ge &= c.v[o] >= p[o];
        dom |= ge;
        if ((j & 7) == 7 && __all_sync(0xffffffffu, dom)) break;
    }
    // a pivot is under itself only (they are their own maxima): it stays, and of the points
    // equal to it, it alone
    if (dom && valid) {
        int lo = 0, hi = npiv;  // pivots before i
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (s_idx[mid] < static_cast<uint32_t>(i)) lo = mid + 1;
            else hi = mid;
        }
        if (lo < npiv && s_idx[lo] == static_cast<uint32_t>(i)) dom = false;
    }
    if (!valid) return;
    uint32_t key = 0xffffffffu;
    if (!dom) {
        uint32_t rank[D];
#pragma unroll
        for (int o = 0; o < D; ++o)
            rank[o] = s_lut[o][bin_of<T>(p[o], v.head->mn[o], v.head->range[o], v.head->scale[o], v.head->shift[o])];
        key = 0;
        int left = v.bits;
        for (int b = 7; b >= 0 && left > 0; --b) {
#pragma unroll
            for (int o = 0; o < D; ++o)
                if (left > 0) {
                    key = (key << 1) | ((rank[o] >> b) & 1u);
                    --left;
                }
        }
        for (int b = 1; b < v.bits; b <<= 1) key ^= key >> b;  // position along the Gray-code curve
        key = (1u << v.bits) - 1u - key;  // the largest points first
        g.place[i] = atomicAdd(v.hist + key, 1u);
    }
    g.key[i] = key;
}

template <int D, typename T, class Src>
__global__ void __launch_bounds__(kMaxStatThreads) maxima_scan_kernel(Src src) {
    __shared__ uint32_t warp_buf[32];
    __shared__ uint32_t s_total;
    const int h = blockIdx.x;
    if (h >= src.count()) return;
    Seg<T> g;
    src.template seg<D>(h, &g);
    if (g.n <= 0) return;
    const SegView<D, T> v = seg_view<D, T>(g.slab, g.n);
    const int64_t nb = int64_t(1) << v.bits;
    uint32_t carry = 0;
    for (int64_t b0 = 0; b0 < nb; b0 += kMaxStatThreads) {
        const int64_t b = b0 + threadIdx.x;
        const uint32_t c = b < nb ? v.hist[b] : 0u;
        const uint32_t ex = block_exclusive_scan<uint32_t, kMaxStatThreads>(c, warp_buf, &s_total);
        if (b < nb) v.hist[b] = carry + ex;
        carry += s_total;
    }
    if (threadIdx.x == 0) v.head->rows = carry;
}

template <int D, typename T, class Src>
__global__ void __launch_bounds__(kMaxThreads) maxima_scatter_kernel(Src src) {
    int h;
    int64_t base;
    if (!src.chunk(blockIdx.x, &h, &base)) return;
    Seg<T> g;
    src.template seg<D>(h, &g);
    const int64_t i = base + threadIdx.x;
    if (i >= g.n) return;
    const uint32_t key = g.key[i];
    if (key == 0xffffffffu) return;
    const SegView<D, T> v = seg_view<D, T>(g.slab, g.n);
    SortedPt<D, T> q;
#pragma unroll
    for (int o = 0; o < SortedPt<D, T>::kPad; ++o) q.v[o] = o < D ? g.pts[i * D + (o < D ? o : 0)] : T(0);
    v.rows[static_cast<int64_t>(v.hist[key]) + g.place[i]] = q;
}

// Thread per group (a chunk covers 32 groups: one warp's worth of threads each).
template <int D, typename T, class Src>
__global__ void __launch_bounds__(kMaxThreads) maxima_corner_kernel(Src src) {
    const int64_t b = static_cast<int64_t>(blockIdx.x) * (kMaxThreads / 32) + (threadIdx.x >> 5);
    int h;
    int64_t base;
    if (!src.chunk(b, &h, &base)) return;
    Seg<T> g;
    src.template seg<D>(h, &g);
    const SegView<D, T> v = seg_view<D, T>(g.slab, g.n);
    const int64_t r = v.head->rows;
    const int64_t t = base / kMaxGroup + (threadIdx.x & 31);
    const int64_t j0 = t * kMaxGroup;
    if (j0 >= r) return;
    T mx[D];
#pragma unroll
    for (int o = 0; o < D; ++o) mx[o] = type_min<T>();
#pragma unroll
    for (int u = 0; u < kMaxGroup; ++u) {
        if (j0 + u < r) {
            const SortedPt<D, T> q = v.rows[j0 + u];
#pragma unroll
            for (int o = 0; o < D; ++o) mx[o] = max(mx[o], q.v[o]);
        } else {  // the last group's unused rows: below everything, and past the row count
            SortedPt<D, T> q;
#pragma unroll
            for (int o = 0; o < SortedPt<D, T>::kPad; ++o) q.v[o] = type_min<T>();
            v.rows[j0 + u] = q;
        }
    }
#pragma unroll
    for (int o = 0; o < D; ++o) v.corner[o * v.groups + t] = mx[o];
}

template <int D, typename T, bool ORDERED, class Src>
__global__ void __launch_bounds__(kMaxThreads) maxima_mark_kernel(Src src) {
    constexpr unsigned kAll = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    int h;
    int64_t base;
    if (!src.chunk(blockIdx.x, &h, &base)) return;
    Seg<T> g;
    src.template seg<D>(h, &g);
    const SegView<D, T> v = seg_view<D, T>(g.slab, g.n);
    const int64_t r = v.head->rows;
    const int64_t w0 = base + (threadIdx.x & ~31);
    if (w0 >= r) return;  // the warp's 32 rows
    const int64_t i = w0 + lane;
    const int64_t groups = (r + kMaxGroup - 1) / kMaxGroup;
    T p[D], lo[D];
    bool dom = i >= r;
    {
        const SortedPt<D, T> q = v.rows[dom ? w0 : i];
#pragma unroll
        for (int o = 0; o < D; ++o) p[o] = dom ? type_max<T>() : q.v[o];
    }
#pragma unroll
    for (int o = 0; o < D; ++o) lo[o] = warp_min_of<T>(p[o]);
    unsigned dead = __ballot_sync(kAll, dom);
    for (int64_t t0 = 0; t0 < groups; t0 += 32) {
        const int64_t t = t0 + lane;
        T c[D];
        bool pass = t < groups;
#pragma unroll
        for (int o = 0; o < D; ++o) {
            c[o] = pass ? v.corner[o * v.groups + t] : type_min<T>();
            pass = pass && c[o] >= lo[o];
        }
        unsigned todo = __ballot_sync(kAll, pass);
        while (todo) {
            const int k = __ffs(todo) - 1;
            todo &= todo - 1;
            bool under = true;
#pragma unroll
            for (int o = 0; o < D; ++o) under &= __shfl_sync(kAll, c[o], k) >= p[o];
            if (!__any_sync(kAll, under)) continue;
            const int64_t j0 = (t0 + k) * kMaxGroup;
            const SortedPt<D, T> *q = v.rows + j0;
            bool any = false;
#pragma unroll
            for (int u = 0; u < kMaxGroup; ++u) {
                const SortedPt<D, T> x = q[u];
                bool ge = true;
#pragma unroll
                for (int o = 0; o < D; ++o) ge &= x.v[o] >= p[o];
                any |= ge;
            }
            if (any) {  // rare: the row itself, or a dominator; decide by the keep rule
                for (int u = 0; u < kMaxGroup; ++u) {
                    const SortedPt<D, T> x = q[u];
                    const int64_t j = j0 + u;
                    bool ge = true, eq = true;
#pragma unroll
                    for (int o = 0; o < D; ++o) {
                        ge &= x.v[o] >= p[o];
                        eq &= x.v[o] == p[o];
                    }
                    dom |= ge && j < r && (!eq || j < i);
                }
                if (dom) {  // decided: from here on under no corner and below no row
#pragma unroll
                    for (int o = 0; o < D; ++o) p[o] = type_max<T>();
                }
            }
            __syncwarp();
        }
        const unsigned now = __ballot_sync(kAll, dom);
        if (now != dead) {
            if (now == kAll) {
                if (ORDERED && lane == 0) g.place[w0 >> 5] = 0;
                return;
            }
            dead = now;
#pragma unroll
            for (int o = 0; o < D; ++o) lo[o] = warp_min_of<T>(p[o]);
        }
    }
    if (ORDERED) {  // maxima_order_kernel and maxima_write_kernel follow
        if (lane == 0) g.place[w0 >> 5] = ~dead;
        return;
    }
    int32_t at = 0;
    if (lane == 0) at = atomicAdd(g.out_size, __popc(~dead));
    at = __shfl_sync(kAll, at, 0);
    if (!dom) {
        T *out = g.out + (static_cast<int64_t>(at) + __popc(~dead & ((1u << lane) - 1u))) * D;
#pragma unroll
        for (int o = 0; o < D; ++o) out[o] = p[o];
    }
}

// Ordered output, block per segment: survivors before each 32 rows (into key), and their
// number to src.finish.
template <int D, typename T, class Src>
__global__ void __launch_bounds__(kMaxStatThreads) maxima_order_kernel(Src src) {
    __shared__ int64_t warp_buf[32];
    __shared__ int64_t s_total;
    const int h = blockIdx.x;
    if (h >= src.count()) return;
    Seg<T> g;
    src.template seg<D>(h, &g);
    int64_t carry = 0;
    if (g.n > 0) {
        const int64_t warps = (static_cast<int64_t>(seg_view<D, T>(g.slab, g.n).head->rows) + 31) / 32;
        for (int64_t w0 = 0; w0 < warps; w0 += kMaxStatThreads) {
            const int64_t w = w0 + threadIdx.x;
            const int64_t c = w < warps ? __popc(g.place[w]) : 0;
            const int64_t ex = block_exclusive_scan<int64_t, kMaxStatThreads>(c, warp_buf, &s_total);
            if (w < warps) g.key[w] = static_cast<uint32_t>(carry + ex);
            carry += s_total;
        }
    }
    if (threadIdx.x == 0) src.finish(h, carry);
}

// Ordered output: the survivors in row order.
template <int D, typename T, class Src>
__global__ void __launch_bounds__(kMaxThreads) maxima_write_kernel(Src src) {
    int h;
    int64_t base;
    if (!src.chunk(blockIdx.x, &h, &base)) return;
    Seg<T> g;
    src.template seg<D>(h, &g);
    const SegView<D, T> v = seg_view<D, T>(g.slab, g.n);
    const int64_t i = base + threadIdx.x;
    if (i >= v.head->rows) return;
    const unsigned keep = g.place[i >> 5], lane = threadIdx.x & 31;
    if (((keep >> lane) & 1u) == 0) return;
    const SortedPt<D, T> q = v.rows[i];
    T *out = g.out + (static_cast<int64_t>(g.key[i >> 5]) + __popc(keep & ((1u << lane) - 1u))) * D;
#pragma unroll
    for (int o = 0; o < D; ++o) out[o] = q.v[o];
}

// `segs`: upper bound on the segments, `chunks`: on their 256-point chunks.
// ORDERED: survivors in the rows' order, their number to src.finish(segment, number).
template <int D, typename T, bool ORDERED = false, class Src>
cudaError_t launch_maxima(const Src &src, int segs, int64_t chunks, cudaStream_t stream) {
    const unsigned c = static_cast<unsigned>(chunks);
    maxima_stats_kernel<D, T, Src><<<segs, kMaxStatThreads, 0, stream>>>(src);
    maxima_prefilter_kernel<D, T, Src><<<c, kMaxThreads, 0, stream>>>(src);
    maxima_scan_kernel<D, T, Src><<<segs, kMaxStatThreads, 0, stream>>>(src);
    maxima_scatter_kernel<D, T, Src><<<c, kMaxThreads, 0, stream>>>(src);
    maxima_corner_kernel<D, T, Src><<<(c + kMaxThreads / 32 - 1) / (kMaxThreads / 32), kMaxThreads, 0, stream>>>(src);
    maxima_mark_kernel<D, T, ORDERED, Src><<<c, kMaxThreads, 0, stream>>>(src);  // kMaximaLaunches kernels
    if constexpr (ORDERED) {
        maxima_order_kernel<D, T, Src><<<segs, kMaxStatThreads, 0, stream>>>(src);
        maxima_write_kernel<D, T, Src><<<c, kMaxThreads, 0, stream>>>(src);
    }
    return cudaGetLastError();
}

}  // namespace dev
}  // namespace pmdd
