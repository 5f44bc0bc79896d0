// The three-objective tile kernel: tiles from the launch's queue, filtered in lexicographic
// order (lex_items.cuh).
#include "kernels.cuh"
#include "lex_items.cuh"

#include <algorithm>

namespace pmdd {
namespace dev {

template <typename T>
__global__ void __launch_bounds__(kLexThreads, sizeof(T) == 4 ? 4 : 2)
    expand_tile_lex_kernel(const ExpandJob *__restrict__ jobs, const int64_t *__restrict__ tile_bases, int num_jobs,
                           int64_t total_tiles, unsigned long long *queue, const int64_t *tiles_dev) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    LexSmem<T> &S = *reinterpret_cast<LexSmem<T> *>(smem_raw);
    for_each_tile(S.draw, jobs, tile_bases, num_jobs, total_tiles, queue, tiles_dev,
                  [&](const ExpandJob &J, int32_t i0, int32_t i1, auto last) {
                      return lex_items<T, kLexThreads, false>(S, J, nullptr, i0, i1, last);
                  });
}

namespace {

template <typename T>
cudaError_t launch_lex_t(const ExpandJob *jobs, const int64_t *tile_bases, int num_jobs, int64_t total_tiles, int grid,
                         unsigned long long *queue, const int64_t *tiles_dev, cudaStream_t stream) {
    const size_t smem = sizeof(LexSmem<T>);
    const cudaError_t e = ensure_smem_limit(reinterpret_cast<const void *>(expand_tile_lex_kernel<T>), smem);
    if (e != cudaSuccess) return e;
    if (total_tiles <= 0) return cudaSuccess;
    const int64_t g = std::min<int64_t>(total_tiles, grid);
    expand_tile_lex_kernel<T><<<static_cast<unsigned>(g), kLexThreads, smem, stream>>>(
        jobs, tile_bases, num_jobs, total_tiles, queue, tiles_dev);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_expand_tiles_lex(bool wide, const ExpandJob *jobs, const int64_t *tile_bases, int num_jobs,
                                    int64_t total_tiles, int grid, unsigned long long *queue,
                                    const int64_t *tiles_dev, cudaStream_t stream) {
    if (wide) return launch_lex_t<int64_t>(jobs, tile_bases, num_jobs, total_tiles, grid, queue, tiles_dev, stream);
    return launch_lex_t<int32_t>(jobs, tile_bases, num_jobs, total_tiles, grid, queue, tiles_dev, stream);
}

}  // namespace dev
}  // namespace pmdd
