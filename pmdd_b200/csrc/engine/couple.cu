// sm_100a kernels for method 3 (dynamic layer cutset) and DD preparation:
//  - out-arc CSR (transpose of the in-arc CSR) for the bottom-up direction;
//  - the cutset join  F = ND( U_v { t + b : t in TD_v, b in BU_v } )  of
//    src/pmdd/enum/gpu/couple.cu:340-498 / src/pmdd/enum/cpu/enum.cpp:333-398, done in
//    rounds without ever materialising all products.  A seed round builds a first
//    running frontier F from a few extreme products per cutset node; a product round
//    streams the products against F and appends the survivors behind it; after either, the
//    maxima of F + the appended points (maxima.cuh, in spatial order) are the next F.  A
//    round that fills U is cut short at the first unit that did not fit.
//
// What bounds the join is how many points of F a product is compared with before it is
// found to be dominated (nearly all are).  So products are not taken one by one: both
// frontiers of a cutset node are put in a spatial order once, a warp takes 8 top-down
// points (a unit) against 32 groups of 8 bottom-up points at a time, and first asks whether
// the upper corner of each 8 x 8 block of products -- the sum of the two groups'
// componentwise maxima -- lies under F; only the blocks left are asked product by product.
// Each question goes first to 64 points spread over F, then to the groups of 8 rows of F
// whose corner no lane can rule out (as in maxima.cuh).  Before, every product swept F in
// sum order 32 products at a time, and the refilter compared every survivor with those of
// no smaller sum.  The join of KP d=4 n=60 on one B200, before -> now: 13.1 -> 2.7 ms (3.8 k
// frontier points), 58 -> 5.4 ms (5.4 k), 198 -> 11 ms (10.8 k); of TSP d=3 n=13 1.7 -> 0.5 ms.
#include "couple.cuh"
#include "kernels.cuh"
#include "maxima.cuh"

namespace pmdd {
namespace dev {

// ------------------------------------------------------------ out-arc CSR
// Of one DD (`one`, jobs nullptr) or of every DD of a set (grid.y), in four launches: zeroed
// counts, out-degrees, their scan (a block per DD), scatter.
__global__ void __launch_bounds__(256) csr_zero_kernel(const CsrJob *__restrict__ jobs, CsrJob one) {
    const CsrJob &J = jobs ? jobs[blockIdx.y] : one;
    for (int32_t v = blockIdx.x * 256 + threadIdx.x; v <= J.num_nodes; v += gridDim.x * 256) J.out_off[v] = 0;
}

__global__ void __launch_bounds__(256) out_degree_kernel(const CsrJob *__restrict__ jobs, CsrJob one) {
    const CsrJob &J = jobs ? jobs[blockIdx.y] : one;
    for (int32_t a = blockIdx.x * 256 + threadIdx.x; a < J.num_arcs; a += gridDim.x * 256)
        atomicAdd(&J.out_off[J.arc_src[a] + 1], 1);
}

// Inclusive scan of out_off[1..n] in place (one block per DD), 16 counts per thread at a
// time: a single DD's scan is a serial chain of block scans, and 1024 counts per link took
// 0.28 ms for 316 k nodes, 16384 take 0.03 ms.
constexpr int kCsrPer = 16;
__global__ void __launch_bounds__(1024) csr_scan_kernel(const CsrJob *__restrict__ jobs, CsrJob one) {
    const CsrJob &J = jobs ? jobs[blockIdx.x] : one;
    __shared__ int32_t warp_buf[32];
    __shared__ int32_t total;
    int32_t carry = 0;
    for (int64_t base = 0; base < J.num_nodes; base += 1024 * kCsrPer) {
        const int64_t i0 = base + static_cast<int64_t>(threadIdx.x) * kCsrPer;
        int32_t x[kCsrPer], sum = 0;
#pragma unroll
        for (int r = 0; r < kCsrPer; ++r) {
            x[r] = i0 + r < J.num_nodes ? J.out_off[i0 + r + 1] : 0;
            sum += x[r];
        }
        int32_t run = carry + block_exclusive_scan<int32_t, 1024>(sum, warp_buf, &total);
        carry += total;
#pragma unroll
        for (int r = 0; r < kCsrPer; ++r) {
            if (i0 + r < J.num_nodes) {
                J.cursor[i0 + r] = run;  // start of the node's out-arcs
                J.out_off[i0 + r + 1] = run + x[r];
            }
            run += x[r];
        }
    }
}

__global__ void __launch_bounds__(256) out_scatter_kernel(const CsrJob *__restrict__ jobs, CsrJob one) {
    const CsrJob &J = jobs ? jobs[blockIdx.y] : one;
    for (int32_t v = blockIdx.x * 256 + threadIdx.x; v < J.num_nodes; v += gridDim.x * 256) {
        for (int32_t a = J.in_off[v]; a < J.in_off[v + 1]; ++a) {
            const int32_t pos = atomicAdd(&J.cursor[J.arc_src[a]], 1);
            J.out_head[pos] = v;
            J.out_w[pos] = J.arc_w[a];
        }
    }
}

static cudaError_t launch_csr(const CsrJob *jobs, const CsrJob &one, int count, int32_t max_nodes, int32_t max_arcs,
                              cudaStream_t stream) {
    if (count <= 0) return cudaSuccess;
    const int cap = std::max(1, 148 * 8 / std::min(count, 64));  // 8 blocks per SM over the set
    const dim3 gn(std::min(cap, max_nodes / 256 + 1), count), ga(std::min(cap, max_arcs / 256 + 1), count);
    csr_zero_kernel<<<gn, 256, 0, stream>>>(jobs, one);
    out_degree_kernel<<<ga, 256, 0, stream>>>(jobs, one);
    csr_scan_kernel<<<count, 1024, 0, stream>>>(jobs, one);
    out_scatter_kernel<<<gn, 256, 0, stream>>>(jobs, one);
    return cudaGetLastError();
}

cudaError_t launch_build_out_csr(const CsrJob &job, cudaStream_t stream) {
    return launch_csr(nullptr, job, 1, job.num_nodes, job.num_arcs, stream);
}

cudaError_t launch_build_out_csrs(const CsrJob *jobs, int count, int32_t max_nodes, int32_t max_arcs,
                                  cudaStream_t stream) {
    for (int at = 0; at < count; at += 32768) {  // grid.y
        const cudaError_t e = launch_csr(jobs + at, CsrJob{}, std::min(count - at, 32768), max_nodes, max_arcs, stream);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

// ------------------------------------------------------------------ coupling
constexpr int kUnit = 8;  // top-down points of a unit, bottom-up points of a group

// Units before each cutset node and the products in all (one block per job).
__global__ void __launch_bounds__(1024) couple_units_kernel(const CoupleJob *__restrict__ jobs) {
    __shared__ int64_t warp_buf[32];
    __shared__ int64_t s_total;
    const CoupleJob &J = jobs[blockIdx.x];
    int64_t *units = J.ctr + kCtrCount;
    int64_t carry = 0, products = 0;
    for (int32_t b0 = 0; b0 < J.num_nodes; b0 += 1024) {
        const int32_t v = b0 + threadIdx.x;
        const int64_t nt = v < J.num_nodes ? J.td_size[v] : 0, nb = v < J.num_nodes ? J.bu_size[v] : 0;
        const int64_t u = nb > 0 ? (nt + kUnit - 1) / kUnit : 0;
        products += nt * nb;
        const int64_t ex = block_exclusive_scan<int64_t, 1024>(u, warp_buf, &s_total);
        if (v < J.num_nodes) units[v] = carry + ex;
        carry += s_total;
    }
    (void)block_exclusive_scan<int64_t, 1024>(products, warp_buf, &s_total);
    if (threadIdx.x == 0) {
        units[J.num_nodes] = carry;
        J.ctr[kCtrUnits] = carry;
        J.ctr[kCtrProducts] = s_total;
    }
}

// Block per cutset node of one side: the node's points, kSortMax at a time, sorted along a
// Gray-code curve through their value range (32-bit keys).  The order only decides how
// tight the groups' corners are.
constexpr int kSortMax = 1024;
constexpr int kSortThreads = 256;

template <int D, typename T>
__global__ void __launch_bounds__(kSortThreads) couple_order_kernel(const CoupleJob *__restrict__ jobs, int bu) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T *pts = reinterpret_cast<T *>(smem_raw);  // [kSortMax * D]
    __shared__ unsigned long long key[kSortMax];
    __shared__ T s_mn[D], s_mx[D];
    const CoupleJob &J = jobs[blockIdx.y];
    T *base = static_cast<T *>(bu ? J.bu_pts : J.td_pts);
    const int64_t *off = bu ? J.bu_off : J.td_off;
    const int32_t *size = bu ? J.bu_size : J.td_size;
    constexpr int kBits = 32 / D < 8 ? 32 / D : 8;  // of each objective
    const int tid = threadIdx.x;
    for (int32_t v = blockIdx.x; v < J.num_nodes; v += gridDim.x) {
        const int32_t total = size[v];
        if (total <= kUnit) continue;
        for (int32_t c0 = 0; c0 < total; c0 += kSortMax) {
            const int n = min(kSortMax, total - c0);
            T *P = base + (off[v] + c0) * D;
            int m = 1;
            while (m < n) m <<= 1;
            for (int i = tid; i < n * D; i += kSortThreads) pts[i] = P[i];
            if (tid < D) {
                s_mn[tid] = type_max<T>();
                s_mx[tid] = type_min<T>();
            }
            __syncthreads();
#pragma unroll
            for (int o = 0; o < D; ++o) {
                T a = type_max<T>(), b = type_min<T>();
                for (int i = tid; i < n; i += kSortThreads) {
                    a = min(a, pts[i * D + o]);
                    b = max(b, pts[i * D + o]);
                }
                for (int s = 16; s > 0; s >>= 1) {
                    a = min(a, __shfl_xor_sync(0xffffffffu, a, s));
                    b = max(b, __shfl_xor_sync(0xffffffffu, b, s));
                }
                if ((tid & 31) == 0) {
                    atomic_min_t(&s_mn[o], a);
                    atomic_max_t(&s_mx[o], b);
                }
            }
            __syncthreads();
            for (int i = tid; i < m; i += kSortThreads) {
                uint32_t k = 0xffffffffu;
                if (i < n) {
                    uint32_t code[D];
#pragma unroll
                    for (int o = 0; o < D; ++o) {
                        const uint64_t rng = above<T>(s_mx[o], s_mn[o]);
                        uint64_t u = above<T>(pts[i * D + o], s_mn[o]), r = rng;
                        const int sh = 64 - __clzll(static_cast<long long>(r | 1ull)) - 40;
                        if (sh > 0) {  // keep the product below in 64 bits
                            u >>= sh;
                            r >>= sh;
                        }
                        code[o] = static_cast<uint32_t>((u << kBits) / (r + 1));
                    }
                    k = 0;
#pragma unroll
                    for (int b = kBits - 1; b >= 0; --b)
#pragma unroll
                        for (int o = 0; o < D; ++o) k = (k << 1) | ((code[o] >> b) & 1u);
#pragma unroll
                    for (int b = 1; b < 32; b <<= 1) k ^= k >> b;
                }
                key[i] = (static_cast<unsigned long long>(k) << 32) | static_cast<unsigned>(i);
            }
            __syncthreads();
            for (int k = 2; k <= m; k <<= 1)  // bitonic sort, ascending; unused keys end last
                for (int j = k >> 1; j > 0; j >>= 1) {
                    for (int i = tid; i < m; i += kSortThreads) {
                        const int p = i ^ j;
                        if (p > i) {
                            const unsigned long long a = key[i], b = key[p];
                            if (((i & k) == 0) == (a > b)) {
                                key[i] = b;
                                key[p] = a;
                            }
                        }
                    }
                    __syncthreads();
                }
            for (int i = tid; i < n; i += kSortThreads) {
                const int from = static_cast<int>(key[i] & 0xffffffffu);
#pragma unroll
                for (int o = 0; o < D; ++o) P[static_cast<int64_t>(i) * D + o] = pts[from * D + o];
            }
            __syncthreads();
        }
    }
}

// Appends points behind F; warp-aggregated.  Returns false (and records the unit at which
// the round must resume) when U is full.
template <int D, typename T>
__device__ __forceinline__ bool append_points(const CoupleJob &J, T *U, int64_t fn, bool keep, const T (&p)[D],
                                              int64_t unit, int lane) {
    const unsigned m = __ballot_sync(0xffffffffu, keep);
    if (m == 0) return true;
    unsigned long long base = 0;
    if (lane == 0)
        base = atomicAdd(reinterpret_cast<unsigned long long *>(&J.ctr[kCtrB]), static_cast<unsigned long long>(__popc(m)));
    base = __shfl_sync(0xffffffffu, base, 0);
    const int64_t pos0 = fn + static_cast<int64_t>(base);
    if (pos0 + __popc(m) > J.ucap) {
        // every later append lands further out, so [F, pos0) is complete
        if (lane == 0) {
            atomicMin(reinterpret_cast<unsigned long long *>(&J.ctr[kCtrResume]), static_cast<unsigned long long>(unit));
            atomicMin(reinterpret_cast<unsigned long long *>(&J.ctr[kCtrValidEnd]),
                      static_cast<unsigned long long>(pos0));
        }
        return false;
    }
    if (keep) {
        const int64_t pos = pos0 + __popc(m & ((1u << lane) - 1u));
#pragma unroll
        for (int o = 0; o < D; ++o) U[pos * D + o] = p[o];
    }
    return true;
}

// Seed round: per cutset node, the products of the two frontiers' maximisers of each
// objective and of the objective sum (warp per node).
template <int D, typename T>
__global__ void __launch_bounds__(kCoupleThreads) couple_seed_kernel(const CoupleJob *__restrict__ jobs) {
    const CoupleJob &J = jobs[blockIdx.y];
    T *U = static_cast<T *>(J.U);
    const T *td = static_cast<const T *>(J.td_pts);
    const T *bu = static_cast<const T *>(J.bu_pts);
    const int lane = threadIdx.x & 31;
    const int warps = gridDim.x * (kCoupleThreads / 32);
    for (int32_t v = blockIdx.x * (kCoupleThreads / 32) + (threadIdx.x >> 5); v < J.num_nodes; v += warps) {
        const int32_t nt = J.td_size[v], nb = J.bu_size[v];
        if (nt == 0 || nb == 0) continue;
        const T *tdv = td + J.td_off[v] * D;
        const T *buv = bu + J.bu_off[v] * D;
        // argmax per objective (0..D-1) and of the sum (D), per side
        int64_t bt[D + 1], bb[D + 1];
        int32_t it[D + 1], ib[D + 1];
#pragma unroll
        for (int k = 0; k <= D; ++k) {
            bt[k] = bb[k] = INT64_MIN;
            it[k] = ib[k] = 0;
        }
        for (int32_t i = lane; i < nt; i += 32) {
            int64_t s = 0;
#pragma unroll
            for (int o = 0; o < D; ++o) {
                const int64_t x = tdv[static_cast<int64_t>(i) * D + o];
                s += x;
                if (x > bt[o]) { bt[o] = x; it[o] = i; }
            }
            if (s > bt[D]) { bt[D] = s; it[D] = i; }
        }
        for (int32_t i = lane; i < nb; i += 32) {
            int64_t s = 0;
#pragma unroll
            for (int o = 0; o < D; ++o) {
                const int64_t x = buv[static_cast<int64_t>(i) * D + o];
                s += x;
                if (x > bb[o]) { bb[o] = x; ib[o] = i; }
            }
            if (s > bb[D]) { bb[D] = s; ib[D] = i; }
        }
#pragma unroll
        for (int k = 0; k <= D; ++k) {
            for (int sft = 16; sft > 0; sft >>= 1) {
                const int64_t ot = __shfl_xor_sync(0xffffffffu, bt[k], sft);
                const int32_t oi = __shfl_xor_sync(0xffffffffu, it[k], sft);
                if (ot > bt[k] || (ot == bt[k] && oi < it[k])) { bt[k] = ot; it[k] = oi; }
                const int64_t ob = __shfl_xor_sync(0xffffffffu, bb[k], sft);
                const int32_t oj = __shfl_xor_sync(0xffffffffu, ib[k], sft);
                if (ob > bb[k] || (ob == bb[k] && oj < ib[k])) { bb[k] = ob; ib[k] = oj; }
            }
        }
        // lane k < D+1 emits product k
        T p[D];
        bool keep = false;
#pragma unroll
        for (int k = 0; k <= D; ++k) {
            if (lane == k) {
#pragma unroll
                for (int o = 0; o < D; ++o)
                    p[o] = tdv[static_cast<int64_t>(it[k]) * D + o] + buv[static_cast<int64_t>(ib[k]) * D + o];
                keep = true;
            }
        }
        if (!keep) {
#pragma unroll
            for (int o = 0; o < D; ++o) p[o] = T(0);
        }
        if (!append_points<D, T>(J, U, 0, keep, p, v, lane)) break;
    }
}

// The running frontier as the product rounds read it: padded rows, the corner of each group
// of 8 rows, and up to 64 pivots -- the row of largest objective sum in each 64th of F,
// which is in spatial order.  Laid out by seg_view in the job's slab.
template <int D, typename T>
__global__ void __launch_bounds__(256) couple_index_kernel(const CoupleJob *__restrict__ jobs) {
    const CoupleJob &J = jobs[blockIdx.y];
    const T *U = static_cast<const T *>(J.U);
    const int64_t fn = J.ctr[kCtrF];
    const SegView<D, T> v = seg_view<D, T>(static_cast<unsigned char *>(J.sc_slab), fn);
    for (int64_t t = static_cast<int64_t>(blockIdx.x) * 256 + threadIdx.x; t < v.groups;
         t += static_cast<int64_t>(gridDim.x) * 256) {
        T mx[D];
#pragma unroll
        for (int o = 0; o < D; ++o) mx[o] = type_min<T>();
        for (int u = 0; u < kMaxGroup; ++u) {
            const int64_t j = t * kMaxGroup + u;
            const int64_t from = j < fn ? j : fn - 1;  // past the end: the last row again
            SortedPt<D, T> q;
#pragma unroll
            for (int o = 0; o < SortedPt<D, T>::kPad; ++o) q.v[o] = o < D ? U[from * D + (o < D ? o : 0)] : T(0);
#pragma unroll
            for (int o = 0; o < D; ++o) mx[o] = max(mx[o], q.v[o]);
            v.rows[j] = q;
        }
#pragma unroll
        for (int o = 0; o < D; ++o) v.corner[o * v.groups + t] = mx[o];
    }
    // pivots: warp per 64th of F
    const int lane = threadIdx.x & 31;
    const int64_t parts = fn < kMaxPivots ? fn : kMaxPivots;
    if (blockIdx.x == 0 && threadIdx.x == 0) v.head->npiv = static_cast<int32_t>(parts);
    for (int64_t k = static_cast<int64_t>(blockIdx.x) * 8 + (threadIdx.x >> 5); k < parts;
         k += static_cast<int64_t>(gridDim.x) * 8) {
        unsigned long long best = 0;
        int64_t at = k * fn / parts;
        for (int64_t j = k * fn / parts + lane; j < (k + 1) * fn / parts; j += 32) {
            const unsigned long long s = static_cast<unsigned long long>(point_sum<D, T>(U + j * D)) + (1ull << 63);
            if (s >= best) {
                best = s;
                at = j;
            }
        }
        for (int s = 16; s > 0; s >>= 1) {
            const unsigned long long ob = __shfl_xor_sync(0xffffffffu, best, s);
            const int64_t oa = __shfl_xor_sync(0xffffffffu, at, s);
            if (ob > best || (ob == best && oa < at)) {
                best = ob;
                at = oa;
            }
        }
        if (lane == 0) {
            SortedPt<D, T> q;
#pragma unroll
            for (int o = 0; o < SortedPt<D, T>::kPad; ++o) q.v[o] = o < D ? U[at * D + (o < D ? o : 0)] : T(0);
            v.head->piv[k] = q;
        }
    }
}

// Which lanes' points lie under F (a point of F >= on every objective)?  Lanes with `dom`
// set do not ask.  All lanes of the warp call it; p is used up.
template <int D, typename T>
__device__ __forceinline__ bool under_frontier(const SortedPt<D, T> *piv, int npiv, const SegView<D, T> &v, T (&p)[D],
                                               bool dom, int lane) {
    constexpr unsigned kAll = 0xffffffffu;
    for (int j = 0; j < npiv; ++j) {
        const SortedPt<D, T> c = piv[j];
        bool ge = true;
#pragma unroll
        for (int o = 0; o < D; ++o) ge &= c.v[o] >= p[o];
        dom |= ge;
        if ((j & 7) == 7 && __all_sync(kAll, dom)) return true;
    }
    unsigned dead = __ballot_sync(kAll, dom);
    if (dead == kAll) return true;
    T lo[D];
#pragma unroll
    for (int o = 0; o < D; ++o) {
        if (dom) p[o] = type_max<T>();  // decided: under no corner and below no row
        lo[o] = warp_min_of<T>(p[o]);
    }
    for (int64_t t0 = 0; t0 < v.groups; t0 += 32) {
        const int64_t t = t0 + lane;
        T c[D];
        bool pass = t < v.groups;
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
            const SortedPt<D, T> *q = v.rows + (t0 + k) * kMaxGroup;
            bool any = false;
#pragma unroll
            for (int u = 0; u < kMaxGroup; ++u) {
                const SortedPt<D, T> x = q[u];
                bool ge = true;
#pragma unroll
                for (int o = 0; o < D; ++o) ge &= x.v[o] >= p[o];
                any |= ge;
            }
            if (any) {
                dom = true;
#pragma unroll
                for (int o = 0; o < D; ++o) p[o] = type_max<T>();
            }
        }
        const unsigned now = __ballot_sync(kAll, dom);
        if (now != dead) {
            if (now == kAll) return true;
            dead = now;
#pragma unroll
            for (int o = 0; o < D; ++o) lo[o] = warp_min_of<T>(p[o]);
        }
    }
    return dom;
}

template <int D, typename T>
__global__ void __launch_bounds__(kCoupleThreads) couple_prune_kernel(const CoupleJob *__restrict__ jobs) {
    constexpr unsigned kAll = 0xffffffffu;
    __shared__ SortedPt<D, T> piv[kMaxPivots];
    const CoupleJob &J = jobs[blockIdx.y];
    T *U = static_cast<T *>(J.U);
    const int64_t fn = J.ctr[kCtrF];
    const SegView<D, T> v = seg_view<D, T>(static_cast<unsigned char *>(J.sc_slab), fn);
    const int npiv = v.head->npiv;
    if (threadIdx.x < npiv) piv[threadIdx.x] = v.head->piv[threadIdx.x];
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const int64_t num_units = J.ctr[kCtrUnits];
    const int64_t *units = J.ctr + kCtrCount;
    volatile const int64_t *resume_flag = J.ctr + kCtrResume;
    while (true) {
        int64_t unit = 0;
        if (lane == 0) {
            // once some unit overflowed U, the rest of the round is redone next round
            if (*resume_flag < num_units) unit = num_units;
            else unit = static_cast<int64_t>(atomicAdd(reinterpret_cast<unsigned long long *>(&J.ctr[kCtrCursor]), 1ULL));
        }
        unit = __shfl_sync(kAll, unit, 0);
        if (unit >= num_units) break;
        int lo = 0, hi = J.num_nodes - 1;  // the last node with units[node] <= unit
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (units[mid] <= unit) lo = mid;
            else hi = mid - 1;
        }
        const int node = lo;
        const int32_t t_at = static_cast<int32_t>(unit - units[node]) * kUnit;
        const int nt = min(kUnit, J.td_size[node] - t_at), nb = J.bu_size[node];
        const T *td = static_cast<const T *>(J.td_pts) + (J.td_off[node] + t_at) * D;
        const T *bu = static_cast<const T *>(J.bu_pts) + J.bu_off[node] * D;
        T tc[D];  // the unit's corner
#pragma unroll
        for (int o = 0; o < D; ++o) {
            tc[o] = td[o];
            for (int x = 1; x < nt; ++x) tc[o] = max(tc[o], td[x * D + o]);
        }
        bool full = false;
        for (int g0 = 0; g0 < nb && !full; g0 += 32 * kUnit) {
            // blocks of products under F by their upper corner (lane: a group of 8 bottom-up
            // points); a unit with one group goes straight to the products
            const int b_at = g0 + lane * kUnit;
            unsigned blocks = __ballot_sync(kAll, b_at < nb);
            if (nb > kUnit) {
                T c[D];
#pragma unroll
                for (int o = 0; o < D; ++o) c[o] = type_max<T>();
                if (b_at < nb) {
#pragma unroll
                    for (int o = 0; o < D; ++o) c[o] = bu[static_cast<int64_t>(b_at) * D + o];
                    for (int x = 1; x < min(kUnit, nb - b_at); ++x)
#pragma unroll
                        for (int o = 0; o < D; ++o) c[o] = max(c[o], bu[static_cast<int64_t>(b_at + x) * D + o]);
#pragma unroll
                    for (int o = 0; o < D; ++o) c[o] += tc[o];
                }
                blocks = ~__ballot_sync(kAll, under_frontier<D, T>(piv, npiv, v, c, b_at >= nb, lane));
            }
            while (blocks && !full) {
                const int g = __ffs(blocks) - 1;
                blocks &= blocks - 1;
                const int b = g0 + g * kUnit + (lane & 7);
                for (int t0 = 0; t0 < nt; t0 += 4) {  // 4 top-down points x 8 bottom-up points
                    const int t = t0 + (lane >> 3);
                    const bool valid = t < nt && b < nb;
                    T p[D], q[D];
#pragma unroll
                    for (int o = 0; o < D; ++o) {
                        p[o] = valid ? td[t * D + o] + bu[static_cast<int64_t>(b) * D + o] : type_max<T>();
                        q[o] = p[o];
                    }
                    const bool dom = under_frontier<D, T>(piv, npiv, v, q, !valid, lane);
                    if (!append_points<D, T>(J, U, fn, !dom, p, unit, lane)) {
                        full = true;
                        break;
                    }
                }
            }
        }
        if (full) break;
    }
}

// F + the points appended behind it, as the segments of maxima.cuh (job h).
template <typename T>
struct CoupleSrc {
    const CoupleJob *jobs;
    int num_jobs;
    int64_t chunks_per_job;
    int seed;
    __device__ __forceinline__ int64_t extent(const CoupleJob &J) const {
        int64_t m = J.ctr[kCtrF] + J.ctr[kCtrB];
        if (m > J.ctr[kCtrValidEnd]) m = J.ctr[kCtrValidEnd];
        return m < J.ucap ? m : J.ucap;
    }
    __device__ __forceinline__ int count() const { return num_jobs; }
    __device__ __forceinline__ bool chunk(int64_t b, int *h, int64_t *base) const {
        const int64_t j = b / chunks_per_job;
        if (j >= num_jobs) return false;
        *h = static_cast<int>(j);
        *base = (b - j * chunks_per_job) * kMaxThreads;
        return *base < extent(jobs[j]);
    }
    template <int D>
    __device__ __forceinline__ void seg(int h, Seg<T> *g) const {
        const CoupleJob &J = jobs[h];
        g->pts = static_cast<const T *>(J.U);
        g->n = extent(J);
        g->slab = static_cast<unsigned char *>(J.sc_slab);
        g->key = reinterpret_cast<uint32_t *>(J.sc_idx);
        g->place = reinterpret_cast<uint32_t *>(J.sc_sidx);
        g->out = static_cast<T *>(J.U_alt);
        g->out_size = nullptr;
    }
    __device__ __forceinline__ void finish(int, int64_t) const {}
};

// The round's bookkeeping, after the survivors were written (the extents depend on the
// counters until then): survivors from the last rows' offset and mask.
template <int D, typename T>
__global__ void couple_finish_kernel(CoupleSrc<T> src) {
    const int h = blockIdx.x;
    const CoupleJob &J = src.jobs[h];
    Seg<T> g;
    src.template seg<D>(h, &g);
    int64_t kept = 0;
    if (g.n > 0) {
        const int64_t rows = seg_view<D, T>(g.slab, g.n).head->rows;
        if (rows > 0) {
            const int64_t w = (rows - 1) / 32;
            kept = static_cast<int64_t>(g.key[w]) + __popc(g.place[w]);
        }
    }
    const int64_t resume = J.ctr[kCtrResume];
    const int64_t units = J.ctr[kCtrUnits];
    J.ctr[kCtrF] = kept;
    J.ctr[kCtrB] = 0;
    if (src.seed) {
        J.ctr[kCtrCursor] = 0;
        J.ctr[kCtrDone] = 0;
    } else {
        J.ctr[kCtrCursor] = resume < units ? resume : units;
        J.ctr[kCtrDone] = resume >= units ? 1 : 0;
    }
    J.ctr[kCtrResume] = INT64_MAX;
    J.ctr[kCtrValidEnd] = J.ucap;
}

template <int D, typename T>
static cudaError_t launch_couple_round_t(const CoupleJob *jobs, int num_jobs, int blocks_per_job, bool seed,
                                        int64_t points, int64_t *launches, cudaStream_t stream) {
    const dim3 grid(blocks_per_job, num_jobs);
    if (seed) {
        const size_t smem = sizeof(T) * D * kSortMax;
        const cudaError_t e = ensure_smem_limit(reinterpret_cast<const void *>(couple_order_kernel<D, T>), smem);
        if (e != cudaSuccess) return e;
        couple_units_kernel<<<num_jobs, 1024, 0, stream>>>(jobs);
        for (int bu = 0; bu < 2; ++bu) couple_order_kernel<D, T><<<grid, kSortThreads, smem, stream>>>(jobs, bu);
        couple_seed_kernel<D, T><<<grid, kCoupleThreads, 0, stream>>>(jobs);
        *launches += 4;
    } else {
        couple_index_kernel<D, T><<<grid, 256, 0, stream>>>(jobs);
        couple_prune_kernel<D, T><<<grid, kCoupleThreads, 0, stream>>>(jobs);
        *launches += 2;
    }
    const CoupleSrc<T> src{jobs, num_jobs, (points + kMaxThreads - 1) / kMaxThreads, seed ? 1 : 0};
    const cudaError_t e = launch_maxima<D, T, true>(src, num_jobs, src.chunks_per_job * num_jobs, stream);
    if (e != cudaSuccess) return e;
    couple_finish_kernel<D, T><<<num_jobs, 1, 0, stream>>>(src);
    *launches += kMaximaLaunches + 3;
    return cudaGetLastError();
}

cudaError_t launch_couple_round(int d, bool wide, const CoupleJob *jobs, int num_jobs, int blocks_per_job, bool seed,
                                int64_t points, int64_t *launches, cudaStream_t stream) {
    if (num_jobs <= 0) return cudaSuccess;
    if (wide) {
        PMDD_DISPATCH_D(d, (launch_couple_round_t<DD, int64_t>(jobs, num_jobs, blocks_per_job, seed, points, launches,
                                                               stream)));
    }
    PMDD_DISPATCH_D(d, (launch_couple_round_t<DD, int32_t>(jobs, num_jobs, blocks_per_job, seed, points, launches,
                                                           stream)));
}

}  // namespace dev
}  // namespace pmdd
