// State dominance (knapsack and set packing): one warp per node of every job's layer, in
// two launches (mark against the labels as they were, then compact each node's slot in
// place).
#include <algorithm>

#include "statedom_node.cuh"

namespace pmdd {
namespace dev {

namespace {

constexpr int kSdThreads = 256;

__device__ __forceinline__ int find_job(const int64_t *node_bases, int num_jobs, int64_t w) {
    int lo = 0, hi = num_jobs - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (node_bases[mid] <= w) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

template <int D, typename T>
__global__ void __launch_bounds__(kSdThreads) sd_mark_kernel(const StateDomJob *jobs, const int64_t *node_bases,
                                                             int num_jobs, int64_t total) {
    const int lane = threadIdx.x & 31;
    const int64_t warps = static_cast<int64_t>(gridDim.x) * (kSdThreads / 32);
    for (int64_t w = static_cast<int64_t>(blockIdx.x) * (kSdThreads / 32) + (threadIdx.x >> 5); w < total;
         w += warps) {
        const int j = find_job(node_bases, num_jobs, w);
        sd_mark_node<D, T, false>(jobs[j], static_cast<int32_t>(w - node_bases[j]), lane);
    }
}

template <int D, typename T>
__global__ void __launch_bounds__(kSdThreads) sd_compact_kernel(const StateDomJob *jobs, const int64_t *node_bases,
                                                                int num_jobs, int64_t total) {
    const int lane = threadIdx.x & 31;
    const int64_t warps = static_cast<int64_t>(gridDim.x) * (kSdThreads / 32);
    for (int64_t w = static_cast<int64_t>(blockIdx.x) * (kSdThreads / 32) + (threadIdx.x >> 5); w < total;
         w += warps) {
        const int j = find_job(node_bases, num_jobs, w);
        const StateDomJob &J = jobs[j];
        const int32_t removed = sd_compact_node<D, T, false>(J, static_cast<int32_t>(w - node_bases[j]), lane);
        if (lane == 0 && removed > 0)
            atomicAdd(reinterpret_cast<unsigned long long *>(J.removed), static_cast<unsigned long long>(removed));
    }
}

template <int D, typename T>
cudaError_t launch_sd_t(const StateDomJob *jobs, const int64_t *node_bases, int num_jobs, int64_t total, int sms,
                        cudaStream_t stream) {
    if (num_jobs <= 0 || total <= 0) return cudaSuccess;
    const int64_t want = (total + kSdThreads / 32 - 1) / (kSdThreads / 32);
    const int grid = static_cast<int>(std::max<int64_t>(1, std::min<int64_t>(want, static_cast<int64_t>(sms) * 16)));
    sd_mark_kernel<D, T><<<grid, kSdThreads, 0, stream>>>(jobs, node_bases, num_jobs, total);
    sd_compact_kernel<D, T><<<grid, kSdThreads, 0, stream>>>(jobs, node_bases, num_jobs, total);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_state_dominance(int d, bool wide, const StateDomJob *jobs, const int64_t *node_bases, int num_jobs,
                                   int64_t total_nodes, int sms, cudaStream_t stream) {
    if (wide) { PMDD_DISPATCH_D(d, (launch_sd_t<DD, int64_t>(jobs, node_bases, num_jobs, total_nodes, sms, stream))); }
    PMDD_DISPATCH_D(d, (launch_sd_t<DD, int32_t>(jobs, node_bases, num_jobs, total_nodes, sms, stream)));
}

}  // namespace dev
}  // namespace pmdd
