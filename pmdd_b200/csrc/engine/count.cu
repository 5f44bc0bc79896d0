// Next-layer counting: per-arc candidate offsets (exclusive scan of the neighbour's
// frontier size), destination sizes, the list of oversized destinations with their
// scratch offsets, and the current layer's survivor total.  One block per job.
//
// A block alone is bound by the latency of its loads, barriers and shared atomics in a row,
// so an arc row takes 8 of each thread's arcs at once (their loads together, three barriers
// for 8192 arcs; a last or only row of at most 1024 arcs keeps the shorter scan of one), a
// destination row 4, the largest destination is kept in a register and reduced once instead
// of a 64-bit shared atomic per destination, and a chain's tile plan, whose candidates are
// below 2^22, divides in 32 bits.  One B200, before -> now: counts and tile plans of KP d=4
// n=60 1.36 -> 0.88 ms (call 31.2 -> 30.1 ms, method 3 18.9 -> 18.0 ms), TSP d=3 n=13 by
// method 3 1.43 -> 1.36 ms.
//
// In a chained layer (chain.cu) the block also sizes its request's next chained
// expansion from these counts -- candidates and tiles, or a stop at an oversized
// destination, a full buffer or the request's last chained layer -- and writes that
// expansion's tile plan (each tile's first destination, as tile_plan_kernel does); the
// last block of the launch to finish then writes the first tile of every request, so
// the next layer's tile kernel follows with no other launch in between.
#include "kernels.cuh"
#include "scan.cuh"

namespace pmdd {
namespace dev {

namespace {

constexpr int kRows = 8;      // arc rows of a thread at a time
constexpr int kItemRows = 4;  // destination rows
static_assert(kCountThreads == 1024, "32 warps a row");

// Next chained expansion of the block's request (every thread of the block calls it).
__device__ void chain_next(const CountJob &J, bool skip, int64_t *warp_buf, int64_t *s_total) {
    __shared__ int64_t s_tiles;
    __shared__ int s_last;
    ExpandJob &N = *J.next;
    const int tid = threadIdx.x;
    if (tid == 0) {
        int64_t tiles = 0;
        bool stop = skip || J.next_layer > J.last;
        if (!stop) {
            const CountResult r = *J.result;  // written by this block's thread 0
            stop = r.num_big > 0 || r.total > J.cap || !chain_side_goes_on(r.total, J.other_score, J.bu != 0);
            if (!stop) {
                tiles = r.total > 0 ? (r.total + N.tile_window - 1) / N.tile_window : 1;
                N.total_cand = r.total;
                N.num_tiles = tiles;
            }
        }
        if (stop) {
            N.total_cand = 0;
            N.num_tiles = 0;
            if (*J.stop == 0) {
                *J.stop = 1;
                *J.stopped_at = J.next_layer;
            }
        }
        s_tiles = tiles;
    }
    __syncthreads();
    const int64_t T = s_tiles;
    if (T > 0) {  // tile plan: destination i belongs to tile min(start_i / window, T - 1)
        const uint32_t window = static_cast<uint32_t>(N.tile_window);  // starts are <= J.cap <= 2^22
        auto tile_of = [&](int32_t k) -> int64_t {
            const uint32_t start =
                static_cast<uint32_t>(item_start(N.item_arc_off, J.arc_cand_off, N.item_base, N.arc_base, k));
            const int64_t t = start / window;
            return t < T - 1 ? t : T - 1;
        };
        for (int32_t i = tid; i < N.num_items; i += kCountThreads) {
            const int64_t ti = tile_of(i);
            const int64_t tp = i == 0 ? -1 : tile_of(i - 1);
            for (int64_t t = tp + 1; t <= ti; ++t) N.tile_first[t] = i;
            if (i == N.num_items - 1)
                for (int64_t t = ti + 1; t <= T; ++t) N.tile_first[t] = N.num_items;
        }
    }
    // the last block to finish writes every request's first tile
    if (tid == 0) {
        J.next_tiles[J.slot] = T;
        __threadfence();
        s_last = atomicAdd(J.done, 1u) == static_cast<unsigned>(J.chain_n - 1) ? 1 : 0;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    for (int base = 0; base < J.chain_n; base += kCountThreads) {  // chain_n <= kChainThreads
        const int k = base + tid;
        const int64_t x = k < J.chain_n ? __ldcg(J.next_tiles + k) : 0;
        const int64_t ex = block_exclusive_scan<int64_t, kCountThreads>(x, warp_buf, s_total);
        if (k < J.chain_n) J.next_bases[k] = ex;
    }
    if (tid == 0) *J.next_total = *s_total;
}

// The counts of one job (every thread of the block calls it).
__device__ void count_body(const CountJob &J, int64_t *warp_buf) {
    __shared__ int64_t s_total;
    __shared__ int64_t s_row[kRows * 32];
    __shared__ int64_t s_max[32];
    __shared__ int s_nbig;
    __shared__ int s_maxarcs;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) {
        s_nbig = 0;
        s_maxarcs = 0;
    }
    int64_t carry = 0;
    int base = 0;
    for (; J.num_arcs - base > kCountThreads; base += kRows * kCountThreads) {
        int32_t nbr[kRows], c[kRows];
        int64_t inc[kRows];
#pragma unroll
        for (int r = 0; r < kRows; ++r) {
            const int a = base + r * kCountThreads + tid;
            nbr[r] = a < J.num_arcs ? J.arc_nbr[J.arc_base + a] : -1;
        }
#pragma unroll
        for (int r = 0; r < kRows; ++r) inc[r] = c[r] = nbr[r] >= 0 ? J.cur_size[nbr[r] - J.cur_base] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
#pragma unroll
            for (int r = 0; r < kRows; ++r) {
                const int64_t y = __shfl_up_sync(0xffffffffu, inc[r], o);
                if (lane >= o) inc[r] += y;
            }
        }
        if (lane == 31) {
#pragma unroll
            for (int r = 0; r < kRows; ++r) s_row[r * 32 + warp] = inc[r];
        }
        __syncthreads();
        if (warp == 0) {  // the rows' warps in order, kRows of them a lane
            int64_t x[kRows], sum = 0;
#pragma unroll
            for (int k = 0; k < kRows; ++k) {
                x[k] = s_row[lane * kRows + k];
                sum += x[k];
            }
            int64_t winc = sum;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int64_t y = __shfl_up_sync(0xffffffffu, winc, o);
                if (lane >= o) winc += y;
            }
            int64_t run = winc - sum;
#pragma unroll
            for (int k = 0; k < kRows; ++k) {
                s_row[lane * kRows + k] = run;
                run += x[k];
            }
            if (lane == 31) s_total = winc;
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < kRows; ++r) {
            const int a = base + r * kCountThreads + tid;
            if (a < J.num_arcs) J.arc_cand_off[a] = carry + s_row[r * 32 + warp] + inc[r] - c[r];
        }
        carry += s_total;
        __syncthreads();  // s_row and s_total are rewritten
    }
    if (base < J.num_arcs) {
        const int a = base + tid;
        int64_t c = 0;
        if (a < J.num_arcs) c = J.cur_size[J.arc_nbr[J.arc_base + a] - J.cur_base];
        const int64_t ex = block_exclusive_scan<int64_t, kCountThreads>(c, warp_buf, &s_total);
        if (a < J.num_arcs) J.arc_cand_off[a] = carry + ex;
        carry += s_total;
    }
    if (tid == 0) J.arc_cand_off[J.num_arcs] = carry;
    const int64_t total = carry;
    __syncthreads();
    int64_t cmax = 0;
    for (int i0 = tid; i0 < J.num_items; i0 += kItemRows * kCountThreads) {
        int32_t b[kItemRows], e[kItemRows];
        int64_t c[kItemRows];
#pragma unroll
        for (int r = 0; r < kItemRows; ++r) {
            const int i = i0 + r * kCountThreads;
            b[r] = e[r] = J.arc_base;
            if (i < J.num_items) {
                b[r] = J.item_arc_off[J.item_base + i];
                e[r] = J.item_arc_off[J.item_base + i + 1];
            }
        }
#pragma unroll
        for (int r = 0; r < kItemRows; ++r)
            c[r] = J.arc_cand_off[e[r] - J.arc_base] - J.arc_cand_off[b[r] - J.arc_base];
#pragma unroll
        for (int r = 0; r < kItemRows; ++r) {
            cmax = max(cmax, c[r]);
            if (c[r] > 0 && !tile_resident(c[r], e[r] - b[r])) {
                atomicMax(&s_maxarcs, e[r] - b[r]);
                const int k = atomicAdd(&s_nbig, 1);
                J.big_list[2 * k] = i0 + r * kCountThreads;
                J.big_list[2 * k + 1] = c[r];
            }
        }
    }
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) cmax = max(cmax, static_cast<int64_t>(__shfl_xor_sync(0xffffffffu, cmax, s)));
    if (lane == 0) s_max[warp] = cmax;
    __syncthreads();
    // scratch offsets of the oversized destinations (exclusive scan of their sizes)
    const int nbig = s_nbig;
    carry = 0;
    for (int at = 0; at < nbig; at += kCountThreads) {
        const int k = at + tid;
        const int64_t c = k < nbig ? J.big_list[2 * k + 1] : 0;
        const int64_t ex = block_exclusive_scan<int64_t, kCountThreads>(c, warp_buf, &s_total);
        if (k < nbig) J.big_list[2 * k + 1] = carry + ex;
        carry += s_total;
    }
    // survivors of the current layer
    int64_t cur = 0;
    for (int i = tid; i < J.cur_nodes; i += kCountThreads) cur += J.cur_size[i];
    for (int s = 16; s > 0; s >>= 1) cur += __shfl_xor_sync(0xffffffffu, cur, s);
    if (lane == 0) warp_buf[warp] = cur;
    __syncthreads();
    if (tid == 0) {
        int64_t cur_total = 0, item = 0;
        for (int w = 0; w < kCountThreads / 32; ++w) {
            cur_total += warp_buf[w];
            item = max(item, s_max[w]);
        }
        J.result->total = total;
        J.result->max_item = item;
        J.result->big_total = carry;
        J.result->cur_total = cur_total;
        J.result->num_big = nbig;
        J.result->max_big_arcs = s_maxarcs;
    }
}

}  // namespace

__global__ void __launch_bounds__(kCountThreads) count_scan_kernel(const CountJob *jobs) {
    const CountJob J = jobs[blockIdx.x];
    // a chained request whose expansion before did not run has nothing to count
    const bool skip = J.stop != nullptr && *J.stop != 0;
    __shared__ int64_t warp_buf[32];
    __shared__ int64_t s_sum;
    if (!skip) count_body(J, warp_buf);
    if (J.next != nullptr) {
        __syncthreads();
        chain_next(J, skip, warp_buf, &s_sum);
    }
}

cudaError_t launch_count_scan(const CountJob *jobs, int num_jobs, cudaStream_t stream) {
    if (num_jobs <= 0) return cudaSuccess;
    count_scan_kernel<<<num_jobs, kCountThreads, 0, stream>>>(jobs);
    return cudaGetLastError();
}

}  // namespace dev
}  // namespace pmdd
