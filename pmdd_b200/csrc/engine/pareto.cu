// Standalone Pareto filter of one int32 point set: the maxima under componentwise >=,
// one copy of each (ParetoFrontier::merge semantics, src/pmdd/enum/pareto_frontier.hpp:
// 237-303).  Sets of at most kParetoBlockMax points take the block-wide sort-filter-skyline
// sweep of sfs.cuh (one launch), larger ones the GPU-wide pass of maxima.cuh as its one
// segment: a host call on 32768 points of 4 objectives takes 0.15 ms instead of 11 ms with the
// one block, on 131072 of 5 objectives 0.7 ms instead of 1.05 s.
#include "kernels.cuh"
#include "maxima.cuh"
#include "pareto.cuh"
#include "sfs.cuh"

#include <algorithm>

namespace pmdd {
namespace dev {

namespace {

// Below, one block's single launch wins over the six of the GPU-wide pass, whose fixed cost is
// about 20 us: a call on 300 points takes 78-93 us by the block, on 600 points 165-203 us,
// on 1025 points by the GPU-wide pass 84-112 us (d = 2 .. 7, host call included).  The block's
// time goes with the maxima, which nothing tells beforehand: where a handful of points lies
// above nearly all others it stays ahead up to some 8000 points (50-120 us against 70-140 us),
// where most points are maxima it takes 0.4 ms for 1025 and 4-6 ms for 4097.
constexpr int64_t kParetoBlockMax = 320;

struct OneSrc {
    Seg<int32_t> s;
    __device__ __forceinline__ int count() const { return 1; }
    __device__ __forceinline__ bool chunk(int64_t b, int *h, int64_t *base) const {
        *h = 0;
        *base = b * kMaxThreads;
        return *base < s.n;
    }
    template <int D>
    __device__ __forceinline__ void seg(int, Seg<int32_t> *g) const {
        *g = s;
    }
};

}  // namespace

template <int D>
__global__ void __launch_bounds__(SfsCfg<D, int32_t>::kThreads)
    pareto_filter_kernel(const int32_t *__restrict__ in, int64_t n, SfsScratch<int32_t> s, int32_t *__restrict__ out,
                         int64_t *__restrict__ out_n) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int32_t k = sfs_block<D, int32_t>(smem_raw, in, n, s, out);
    if (threadIdx.x == 0) *out_n = k;
}

template <int D>
static size_t slab_bytes(int64_t n) {
    return seg_slab_bytes<D, int32_t>(n);
}

static size_t slab_bytes_of(int d, int64_t n) {
    switch (d) {
    case 1: return slab_bytes<1>(n);
    case 2: return slab_bytes<2>(n);
    case 3: return slab_bytes<3>(n);
    case 4: return slab_bytes<4>(n);
    case 5: return slab_bytes<5>(n);
    case 6: return slab_bytes<6>(n);
    case 7: return slab_bytes<7>(n);
    default: return slab_bytes<8>(n);
    }
}

size_t pareto_scratch_bytes(int d, int64_t n) {
    const size_t pts = (static_cast<size_t>(n) * d * sizeof(int32_t) + 255) / 256 * 256;
    const size_t idx = (static_cast<size_t>(n) * sizeof(int32_t) + 255) / 256 * 256;
    // the GPU-wide pass' slab is the larger of the two for small sets only (its head)
    const size_t slab = n > kParetoBlockMax ? (slab_bytes_of(d, n) + 255) / 256 * 256 : 0;
    return 2 * idx + std::max(2 * pts, slab);
}

SfsScratch<int32_t> pareto_scratch_layout(void *scratch, int d, int64_t n) {
    const size_t pts = (static_cast<size_t>(n) * d * sizeof(int32_t) + 255) / 256 * 256;
    const size_t idx = (static_cast<size_t>(n) * sizeof(int32_t) + 255) / 256 * 256;
    char *m = static_cast<char *>(scratch);
    SfsScratch<int32_t> s;
    s.P2 = reinterpret_cast<int32_t *>(m);
    s.SV = reinterpret_cast<int32_t *>(m + pts);
    s.I2 = reinterpret_cast<int32_t *>(m + 2 * pts);
    s.SVI = reinterpret_cast<int32_t *>(m + 2 * pts + idx);
    return s;
}

template <int D>
static cudaError_t launch_pareto_t(const int32_t *in, int64_t n, void *scratch, int32_t *out, int64_t *out_n,
                                   cudaStream_t stream) {
    if (n > kParetoBlockMax) {
        const size_t idx = (static_cast<size_t>(n) * sizeof(int32_t) + 255) / 256 * 256;
        unsigned char *m = static_cast<unsigned char *>(scratch);
        // keys | places | slab; the count is a 64-bit word whose low half the survivors are
        // added to
        cudaError_t e = cudaMemsetAsync(out_n, 0, sizeof(int64_t), stream);
        if (e != cudaSuccess) return e;
        OneSrc src{{in, n, m + 2 * idx, reinterpret_cast<uint32_t *>(m), reinterpret_cast<uint32_t *>(m + idx), out,
                    reinterpret_cast<int32_t *>(out_n)}};
        return launch_maxima<D, int32_t>(src, 1, (n + kMaxThreads - 1) / kMaxThreads, stream);
    }
    using Cfg = SfsCfg<D, int32_t>;
    {
        const cudaError_t e = ensure_smem_limit(reinterpret_cast<const void *>(pareto_filter_kernel<D>), Cfg::kSmem);
        if (e != cudaSuccess) return e;
    }
    pareto_filter_kernel<D><<<1, Cfg::kThreads, Cfg::kSmem, stream>>>(in, n, pareto_scratch_layout(scratch, D, n),
                                                                       out, out_n);
    return cudaGetLastError();
}

int pareto_launches(int64_t n) { return n > kParetoBlockMax ? kMaximaLaunches : 1; }

cudaError_t launch_pareto_filter(int d, const int32_t *in, int64_t n, void *scratch, int32_t *out, int64_t *out_n,
                                 cudaStream_t stream) {
    PMDD_DISPATCH_D(d, (launch_pareto_t<DD>(in, n, scratch, out, out_n, stream)));
}

}  // namespace dev
}  // namespace pmdd
