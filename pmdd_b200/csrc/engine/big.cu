// Oversized destinations (those tile_resident() rejects).  Their candidates are
// materialised in scratch, then filtered; everything works on one scratch pass at a time
// (see ExpandJob::big_window).
//
//   big_expand_kernel: thread per candidate over the pass's flat candidate space, so a
//       destination of n candidates gets ~n threads whatever the other sizes are;
//   big_sfs_kernel:    destinations below ExpandJob::big_mark_min candidates: one block
//       each runs the sort-filter-skyline of sfs.cuh, which compares each point only
//       with the maxima found so far; many such destinations keep the GPU busy side by
//       side;
//   big_plan_kernel and maxima.cuh: destinations of big_mark_min candidates and more, each
//       spread over every SM.  The plan lists them with their 256-candidate chunks; a
//       few pivots drop what they dominate, the rest is put in a spatially coherent order
//       and compared group by group, skipping groups whose corner dominates nothing.
//
// The GPU-wide pass wins from the smallest oversized destinations up (on the batched
// knapsack / set-packing stream as on single 5-objective TSPs), so by default it takes
// every destination above kSmallMax candidates; SFS blocks keep those that leave the tiles
// for their arc count, and whatever a fixed or tuned crossover assigns them.
//
// The pass replaced one that tested every candidate against 4*sqrt(n) pivots and then
// compared all pairs of the rest (one B200, oversized path per enumeration, before -> now):
// TSP d=5 n=13 38.7 -> 9.6 ms (23.7 M candidates), KP d=4 n=60 18.8 -> 6.0 ms (17.7 M),
// KP d=7 n=25 1.14 -> 0.56 ms, the 192-instance stream 31.4 -> 11.2 ms, where it also took
// over the three-objective destinations with sorted runs, which one staircase warp each
// walked in lexicographic order (against 2 ms more in the tiles, whose runs from these
// parents arrive unsorted).
#include "big_common.cuh"
#include "kernels.cuh"
#include "maxima.cuh"
#include "sfs.cuh"

#include <algorithm>

namespace pmdd {
namespace dev {

namespace {

using namespace big;

constexpr int kFlatThreads = 256;
constexpr int kPlanThreads = 1024;

// The destinations that take the mark path in one pass: destination h is seg[h], its
// candidates form chunks [chunk_base[h], chunk_base[h + 1]) of kMaxThreads.
struct MarkPlan {
    int32_t count;
    int32_t pad;
    int64_t total;   // chunks
};

struct MarkSeg {
    int32_t job, item;
    int64_t soff, c0, n;   // as BigItem
};

struct PlanArrays {
    MarkSeg *seg;          // [cap]
    int64_t *chunk_base;   // [cap + 1]
};

__host__ __device__ __forceinline__ size_t plan_round(size_t b) { return (b + 255) & ~static_cast<size_t>(255); }

__device__ __forceinline__ PlanArrays plan_arrays(const MarkPlan *plan, int cap) {
    char *p = reinterpret_cast<char *>(const_cast<MarkPlan *>(plan)) + 256;
    PlanArrays A;
    A.seg = reinterpret_cast<MarkSeg *>(p);
    A.chunk_base = reinterpret_cast<int64_t *>(p + plan_round(static_cast<size_t>(cap) * sizeof(MarkSeg)));
    return A;
}

// The plan's destinations as the segments of maxima.cuh.
template <typename T>
struct BigSrc {
    const ExpandJob *jobs;
    const MarkPlan *plan;
    int cap;
    __device__ __forceinline__ int count() const { return plan->count; }
    __device__ __forceinline__ bool chunk(int64_t b, int *h, int64_t *base) const {
        if (b >= plan->total) return false;  // the grid is an upper bound
        const int64_t *cb = plan_arrays(plan, cap).chunk_base;
        int lo = 0, hi = plan->count - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (cb[mid] <= b) lo = mid;
            else hi = mid - 1;
        }
        *h = lo;
        *base = (b - cb[lo]) * kMaxThreads;
        return true;
    }
    template <int D>
    __device__ __forceinline__ void seg(int h, Seg<T> *g) const {
        const MarkSeg M = plan_arrays(plan, cap).seg[h];
        const ExpandJob &J = jobs[M.job];
        g->pts = static_cast<const T *>(J.big_pts) + M.soff * D;
        g->n = M.n;
        g->slab = big_slab<D, T>(J, M.soff);
        g->key = reinterpret_cast<uint32_t *>(J.big_idx) + M.soff;
        g->place = reinterpret_cast<uint32_t *>(J.big_surv_idx) + M.soff;
        g->out = static_cast<T *>(J.out_pts) + M.c0 * D;
        g->out_size = J.out_size + M.item;
    }
};

}  // namespace

size_t big_plan_bytes(int cap) {
    const size_t c = static_cast<size_t>(cap);
    return 256 + plan_round(c * sizeof(MarkSeg)) + plan_round((c + 1) * 8);
}

// Materialise the oversized candidates of one pass (AoS, D values each).
template <int D, typename T>
__global__ void __launch_bounds__(kFlatThreads) big_expand_kernel(const ExpandJob *__restrict__ jobs,
                                                                  const int64_t *__restrict__ job_bases, int num_jobs,
                                                                  int64_t total, int64_t pass) {
    for (int64_t g = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; g < total;
         g += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        BigCand c;
        if (!big_cand(jobs, job_bases, num_jobs, g, pass, &c)) continue;
        const ExpandJob &J = jobs[c.job];
        int64_t rs, re;
        const int32_t a = run_of(J, c.B, c.i, &rs, &re);
        const int32_t u = J.arc_nbr[a] - J.prev_base;
        const T *src = static_cast<const T *>(J.prev_pts) + (J.prev_off[u] + (c.i - rs)) * D;
        const int32_t *w = J.weights + static_cast<int64_t>(J.arc_wrow[a]) * D;
        T *dst = static_cast<T *>(J.big_pts) + (c.B.soff + c.i) * D;
#pragma unroll
        for (int o = 0; o < D; ++o) dst[o] = src[o] + static_cast<T>(w[o]);
    }
}

// One block: the mark-path destinations of this pass (at most `cap`) and their chunks.
__global__ void __launch_bounds__(kPlanThreads) big_plan_kernel(const ExpandJob *__restrict__ jobs,
                                                                const BigWork *__restrict__ work, int num_work,
                                                                int64_t pass, MarkPlan *plan, int cap) {
    __shared__ int64_t warp_buf[32];
    __shared__ int64_t s_total;
    const PlanArrays A = plan_arrays(plan, cap);
    int64_t chunks = 0, count = 0;
    for (int b0 = 0; b0 < num_work; b0 += kPlanThreads) {
        const int w = b0 + threadIdx.x;
        int64_t nch = 0;
        BigItem B;
        if (w < num_work) {
            const ExpandJob &J = jobs[work[w].job];
            if (big_item(J, work[w], pass, &B) && B.n >= J.big_mark_min) nch = (B.n + kMaxThreads - 1) / kMaxThreads;
        }
        const int64_t sel = nch > 0 ? 1 : 0;
        const int64_t pos = count + block_exclusive_scan<int64_t, kPlanThreads>(sel, warp_buf, &s_total);
        const int64_t nsel = s_total;
        const int64_t cb = chunks + block_exclusive_scan<int64_t, kPlanThreads>(nch, warp_buf, &s_total);
        const int64_t nchunks = s_total;
        if (sel && pos < cap) {
            A.seg[pos] = MarkSeg{work[w].job, B.item, B.soff, B.c0, B.n};
            A.chunk_base[pos] = cb;
        }
        count += nsel;
        chunks += nchunks;
    }
    if (threadIdx.x == 0) {
        if (count > cap) {  // cap is an upper bound by construction; never drop work silently
            atomicOr(jobs[0].err, kErrBounds);
            count = cap;
            chunks = 0;
        }
        plan->total = chunks;
        A.chunk_base[count] = chunks;
        plan->count = static_cast<int32_t>(count);
    }
}

// Destinations below big_mark_min candidates: one block each.
template <int D, typename T>
__global__ void __launch_bounds__(SfsSmallCfg<D, T>::kThreads) big_sfs_kernel(const ExpandJob *__restrict__ jobs,
                                                                         const BigWork *__restrict__ work,
                                                                         const int32_t *__restrict__ order,
                                                                         int64_t pass) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const BigWork W = work[order ? order[blockIdx.x] : blockIdx.x];
    const ExpandJob &J = jobs[W.job];
    BigItem B;
    if (!big_item(J, W, pass, &B) || B.n >= J.big_mark_min) return;
    SfsScratch<T> s;
    s.P2 = reinterpret_cast<T *>(big_slab<D, T>(J, B.soff));
    s.I2 = J.big_idx + B.soff;
    s.SV = s.P2 + B.n * D;
    s.SVI = J.big_surv_idx + B.soff;
    const int32_t kept = sfs_block<D, T, SfsSmallCfg<D, T>>(smem_raw, static_cast<const T *>(J.big_pts) + B.soff * D,
                                                            B.n, s, static_cast<T *>(J.out_pts) + B.c0 * D);
    if (threadIdx.x == 0) J.out_size[B.item] = kept;
}

// SFS blocks largest destination first: one block sorts the pass's work list by
// candidate count, descending (ties in list order; destinations outside the pass or for
// the mark path count as empty), so that the longest blocks start first and the tail of
// the launch is short.  num_work <= kBigOrderMax.
__global__ void __launch_bounds__(1024) big_order_kernel(const ExpandJob *__restrict__ jobs,
                                                         const BigWork *__restrict__ work, int num_work, int64_t pass,
                                                         int32_t *__restrict__ order) {
    __shared__ unsigned long long key[kBigOrderMax];
    int m = 1;
    while (m < num_work) m <<= 1;
    constexpr unsigned long long kMaxN = (1ULL << 40) - 1;
    for (int i = threadIdx.x; i < m; i += blockDim.x) {
        unsigned long long k = ~0ULL;
        if (i < num_work) {
            const BigWork W = work[i];
            const ExpandJob &J = jobs[W.job];
            BigItem B;
            unsigned long long n = 0;
            if (big_item(J, W, pass, &B) && B.n < J.big_mark_min)
                n = B.n > static_cast<int64_t>(kMaxN) ? kMaxN : static_cast<unsigned long long>(B.n);
            k = ((kMaxN - n) << 12) | static_cast<unsigned long long>(i);
        }
        key[i] = k;
    }
    __syncthreads();
    for (int k = 2; k <= m; k <<= 1)
        for (int j = k >> 1; j > 0; j >>= 1) {
            for (int i = threadIdx.x; i < m; i += blockDim.x) {
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
    for (int i = threadIdx.x; i < num_work; i += blockDim.x) order[i] = static_cast<int32_t>(key[i] & 4095ULL);
}

template <int D, typename T>
static cudaError_t launch_big_t(const BigLaunch &L, cudaStream_t stream) {
    if (L.num_work <= 0 || L.total <= 0) return cudaSuccess;
    using Cfg = SfsSmallCfg<D, T>;
    {
        const cudaError_t e = ensure_smem_limit(reinterpret_cast<const void *>(big_sfs_kernel<D, T>), Cfg::kSmem);
        if (e != cudaSuccess) return e;
    }
    {
        const int64_t want = (L.total + kFlatThreads - 1) / kFlatThreads;
        const unsigned grid = static_cast<unsigned>(std::max<int64_t>(1, std::min<int64_t>(want, int64_t(L.sms) * 32)));
        big_expand_kernel<D, T><<<grid, kFlatThreads, 0, stream>>>(L.jobs, L.job_bases, L.num_jobs, L.total, L.pass);
    }
    if (L.with_sfs) {
        const int32_t *order = nullptr;
        if (L.order && L.num_work <= kBigOrderMax) {
            big_order_kernel<<<1, 1024, 0, stream>>>(L.jobs, L.work, L.num_work, L.pass, L.order);
            order = L.order;
        }
        big_sfs_kernel<D, T><<<L.num_work, Cfg::kThreads, Cfg::kSmem, stream>>>(L.jobs, L.work, order, L.pass);
    }
    if (L.mark_cap > 0) {
        MarkPlan *plan = static_cast<MarkPlan *>(L.plan);
        big_plan_kernel<<<1, kPlanThreads, 0, stream>>>(L.jobs, L.work, L.num_work, L.pass, plan, L.mark_cap);
        // chunks: at most one per 256 candidates of the pass plus one per listed destination
        const int64_t chunks = (L.total + kMaxThreads - 1) / kMaxThreads + L.mark_cap;
        const cudaError_t e = launch_maxima<D, T>(BigSrc<T>{L.jobs, plan, L.mark_cap}, L.mark_cap, chunks, stream);
        if (e != cudaSuccess) return e;
    }
    return cudaGetLastError();
}

cudaError_t launch_big(int d, bool wide, const BigLaunch &L, cudaStream_t stream) {
    if (wide) { PMDD_DISPATCH_D(d, (launch_big_t<DD, int64_t>(L, stream))); }
    PMDD_DISPATCH_D(d, (launch_big_t<DD, int32_t>(L, stream)));
}

}  // namespace dev
}  // namespace pmdd
