// The tile plan, and the pairwise tile kernel: tiles from the launch's queue, filtered by
// pair_items.cuh.
#include "kernels.cuh"
#include "pair_items.cuh"

#include <algorithm>

namespace pmdd {
namespace dev {

// ------------------------------------------------------------------ tile plan
__global__ void tile_plan_kernel(const ExpandJob *__restrict__ jobs, const int64_t *__restrict__ item_bases,
                                 int num_jobs, int64_t total_items) {
    for (int64_t g = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; g < total_items;
         g += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const int j = find_base(item_bases, num_jobs, g);
        const ExpandJob &J = jobs[j];
        const int32_t i = static_cast<int32_t>(g - item_bases[j]);
        const int64_t T = J.num_tiles;
        if (T == 0) continue;  // a chained expansion that stopped (chain.cu)
        auto tile_of = [&](int32_t k) -> int64_t {
            const int64_t s = item_start(J.item_arc_off, J.arc_cand_off, J.item_base, J.arc_base, k);
            const int64_t t = s / J.tile_window;
            return t < T - 1 ? t : T - 1;
        };
        const int64_t ti = tile_of(i);
        const int64_t tp = i == 0 ? -1 : tile_of(i - 1);
        for (int64_t t = tp + 1; t <= ti; ++t) J.tile_first[t] = i;
        if (i == J.num_items - 1)
            for (int64_t t = ti + 1; t <= T; ++t) J.tile_first[t] = J.num_items;
    }
}

cudaError_t launch_tile_plan(const ExpandJob *jobs, const int64_t *item_bases, int num_jobs, int64_t total_items,
                             cudaStream_t stream) {
    if (num_jobs <= 0 || total_items <= 0) return cudaSuccess;
    const int64_t g = std::min<int64_t>((total_items + 255) / 256, 148 * 16);
    tile_plan_kernel<<<static_cast<unsigned>(g), 256, 0, stream>>>(jobs, item_bases, num_jobs, total_items);
    return cudaGetLastError();
}

// ------------------------------------------------------------------ the tiles
template <int D, typename T>
__global__ void __launch_bounds__(pair_threads<D, T>(), 1024 / pair_threads<D, T>())
    expand_tile_kernel(const ExpandJob *__restrict__ jobs, const int64_t *__restrict__ tile_bases, int num_jobs,
                       int64_t total_tiles, unsigned long long *queue, const int64_t *tiles_dev) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    PairSmem<D, T> &S = *reinterpret_cast<PairSmem<D, T> *>(smem_raw);
    for_each_tile(S.draw, jobs, tile_bases, num_jobs, total_tiles, queue, tiles_dev,
                  [&](const ExpandJob &J, int32_t i0, int32_t i1, auto last) {
                      return pair_items<D, T, pair_threads<D, T>(), false>(S, J, nullptr, i0, i1, last);
                  });
}

template <int D, typename T>
static cudaError_t launch_expand_tiles_t(const ExpandJob *jobs, const int64_t *tile_bases, int num_jobs,
                                         int64_t total_tiles, int grid, unsigned long long *queue,
                                         const int64_t *tiles_dev, cudaStream_t stream) {
    const size_t smem = sizeof(PairSmem<D, T>);
    {
        const cudaError_t e = ensure_smem_limit(reinterpret_cast<const void *>(expand_tile_kernel<D, T>), smem);
        if (e != cudaSuccess) return e;
    }
    if (total_tiles <= 0) return cudaSuccess;
    const int64_t g = std::min<int64_t>(total_tiles, grid);
    expand_tile_kernel<D, T><<<static_cast<unsigned>(g), pair_threads<D, T>(), smem, stream>>>(
        jobs, tile_bases, num_jobs, total_tiles, queue, tiles_dev);
    return cudaGetLastError();
}

cudaError_t launch_expand_tiles(int d, bool wide, const ExpandJob *jobs, const int64_t *tile_bases, int num_jobs,
                                int64_t total_tiles, int grid, unsigned long long *queue, const int64_t *tiles_dev,
                                cudaStream_t stream) {
    if (wide) {
        PMDD_DISPATCH_D(d, (launch_expand_tiles_t<DD, int64_t>(jobs, tile_bases, num_jobs, total_tiles, grid, queue,
                                                               tiles_dev, stream)));
    }
    PMDD_DISPATCH_D(d, (launch_expand_tiles_t<DD, int32_t>(jobs, tile_bases, num_jobs, total_tiles, grid, queue,
                                                           tiles_dev, stream)));
}

}  // namespace dev
}  // namespace pmdd
