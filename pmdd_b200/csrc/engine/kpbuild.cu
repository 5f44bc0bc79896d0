// Exact knapsack BDDs built on the device: see kpbuild.cuh for the construction.
#include <algorithm>
#include <climits>

#include "kpbuild.cuh"
#include "scan.cuh"

namespace pmdd {
namespace dev {

namespace {

constexpr int NT = kKpThreads;

// In-place exclusive scan of a[0..m) by the whole block; returns the total (all threads).
__device__ int32_t block_scan_array(int32_t *a, int64_t m, int32_t *warp_buf, int32_t *total) {
    const int64_t chunk = (m + NT - 1) / NT;
    const int64_t b = threadIdx.x * chunk, e = min(m, b + chunk);
    int32_t sum = 0;
    for (int64_t i = b; i < e; ++i) sum += a[i];
    int32_t run = block_exclusive_scan<int32_t, NT>(sum, warp_buf, total);
    for (int64_t i = b; i < e; ++i) {
        const int32_t x = a[i];
        a[i] = run;
        run += x;
    }
    __syncthreads();
    return *total;
}

}  // namespace

__global__ void __launch_bounds__(NT) kp_reduce_kernel(const KpBuildJob *jobs) {
    const KpBuildJob &J = jobs[blockIdx.x];
    __shared__ int32_t warp_buf[32];
    __shared__ int32_t total;
    __shared__ int32_t s_count;
    const int n = J.n, tid = threadIdx.x;
    const int64_t S = static_cast<int64_t>(J.cap) + 1;
    int32_t *key = J.tmp;              // [S]
    int32_t *flag = J.tmp + S;         // [2S]
    int32_t *remap_a = J.tmp + 3 * S;  // [S]
    int32_t *remap_b = J.tmp + 4 * S;  // [S]
    int32_t *st = J.tmp + 5 * S;       // [S] reachable states of a layer, ascending
    int32_t *r0j = J.tmp + 6 * S;      // [S]
    int32_t *r1j = J.tmp + 7 * S;      // [S]
    int32_t *head = J.tmp + 8 * S;     // [S]
    int32_t *minold = J.tmp + 9 * S;   // [S]

    // ---- top-down: reachable states and their first-seen numbering
    for (int64_t s = tid; s < S; s += NT) J.idx[s] = s == 0 ? 0 : -1;
    if (tid == 0) {
        J.width[0] = 1;
        J.width[n] = 1;
        *J.err = 0;
    }
    int32_t W = 1;
    for (int l = 0; l + 1 < n; ++l) {
        const int32_t *cur = J.idx + l * S;
        int32_t *nxt = J.idx + (l + 1) * S;
        const int32_t wl = J.w[l];
        for (int64_t f = tid; f < 2 * static_cast<int64_t>(W); f += NT) flag[f] = 0;
        __syncthreads();
        for (int64_t s = tid; s < S; s += NT) {
            int32_t k = INT_MAX;
            const int32_t a = cur[s];
            if (a >= 0) k = 2 * a;
            if (s >= wl) {
                const int32_t b = cur[s - wl];
                if (b >= 0) k = min(k, 2 * b + 1);
            }
            key[s] = k;
            if (k != INT_MAX) flag[k] = 1;
        }
        __syncthreads();
        W = block_scan_array(flag, 2 * static_cast<int64_t>(W), warp_buf, &total);
        for (int64_t s = tid; s < S; s += NT) nxt[s] = key[s] == INT_MAX ? -1 : flag[key[s]];
        if (tid == 0) J.width[l + 1] = W;
        __syncthreads();
    }

    // ---- bottom-up reduction
    int32_t *remap_next = remap_a, *remap_cur = remap_b;
    if (tid == 0) {
        remap_next[0] = 0;  // the terminal
        J.classes[n] = 1;
        J.arcs_into[0] = 0;
    }
    __syncthreads();
    for (int l = n - 1; l >= 0; --l) {
        const int32_t *cur = J.idx + l * S;
        const int32_t *nxt = l + 1 < n ? J.idx + (l + 1) * S : nullptr;
        const int32_t wl = J.w[l];
        const int32_t Wl = J.width[l];
        // a. reachable states in ascending order
        for (int64_t s = tid; s < S; s += NT) flag[s] = cur[s] >= 0 ? 1 : 0;
        __syncthreads();
        const int32_t cnt = block_scan_array(flag, S, warp_buf, &total);
        if (cnt != Wl && tid == 0) *J.err = 1;
        for (int64_t s = tid; s < S; s += NT)
            if (cur[s] >= 0 && flag[s] < Wl) st[flag[s]] = static_cast<int32_t>(s);
        __syncthreads();
        const int32_t Wc = min(cnt, Wl);
        // b. child classes of every state
        for (int32_t j = tid; j < Wc; j += NT) {
            const int32_t s = st[j];
            // both children of a reachable state are reachable (checked, never indexed at -1)
            int32_t c0old = nxt ? nxt[s] : 0, c1old = -1;
            if (static_cast<int64_t>(s) + wl <= J.cap) c1old = nxt ? nxt[s + wl] : 0;
            if (c0old < 0 || (c1old < 0 && static_cast<int64_t>(s) + wl <= J.cap)) {
                *J.err = 1;
                c0old = max(c0old, 0);
                c1old = static_cast<int64_t>(s) + wl <= J.cap ? max(c1old, 0) : -1;
            }
            r0j[j] = remap_next[c0old];
            r1j[j] = c1old >= 0 ? remap_next[c1old] : -1;
        }
        __syncthreads();
        // c. runs of equal (0-child, 1-child): one class each
        for (int32_t j = tid; j < Wc; j += NT) head[j] = (j == 0 || r0j[j] != r0j[j - 1] || r1j[j] != r1j[j - 1]) ? 1 : 0;
        __syncthreads();
        const int32_t K = block_scan_array(head, Wc, warp_buf, &total);
        int32_t *cnew = J.cls_new + l * S, *c0 = J.cls_c0 + l * S, *c1 = J.cls_c1 + l * S;
        for (int32_t c = tid; c < K; c += NT) minold[c] = INT_MAX;
        __syncthreads();
        // class of j = exclusive count of heads up to and including j, minus one
        for (int32_t j = tid; j < Wc; j += NT) {
            const bool h = j == 0 || r0j[j] != r0j[j - 1] || r1j[j] != r1j[j - 1];
            const int32_t c = head[j] + (h ? 0 : -1);
            atomicMin(&minold[c], cur[st[j]]);
            if (h) {
                c0[c] = r0j[j];
                c1[c] = r1j[j];
            }
        }
        __syncthreads();
        // d. number the classes by their first occurrence (smallest old index)
        for (int32_t x = tid; x < Wl; x += NT) flag[x] = 0;
        __syncthreads();
        for (int32_t c = tid; c < K; c += NT)
            if (minold[c] >= 0 && minold[c] < Wl) flag[minold[c]] = 1;
        __syncthreads();
        block_scan_array(flag, Wl, warp_buf, &total);
        for (int32_t c = tid; c < K; c += NT) cnew[c] = minold[c] >= 0 && minold[c] < Wl ? flag[minold[c]] : 0;
        __syncthreads();
        for (int32_t j = tid; j < Wc; j += NT) {
            const bool h = j == 0 || r0j[j] != r0j[j - 1] || r1j[j] != r1j[j - 1];
            const int32_t c = head[j] + (h ? 0 : -1);
            const int32_t old = cur[st[j]];
            if (old >= 0 && old < S) remap_cur[old] = cnew[c];
        }
        if (tid == 0) s_count = 0;
        __syncthreads();
        int32_t ones = 0;
        for (int32_t c = tid; c < K; c += NT) ones += c1[c] >= 0 ? 1 : 0;
        atomicAdd(&s_count, ones);
        __syncthreads();
        if (tid == 0) {
            J.classes[l] = K;
            J.arcs_into[l + 1] = K + s_count;
        }
        int32_t *t = remap_next;
        remap_next = remap_cur;
        remap_cur = t;
        __syncthreads();
    }
}

// Block (l, k): the arcs of instance k from layer l into layer l + 1; block (0, k) also the
// layer offsets, the weight table and the root.  Layers do not depend on one another, and
// a run of more than kLongRun parents is sorted by the whole block: one thread's insertion
// of a layer's longest run (hundreds of parents, its square in dependent global accesses)
// took 20 of the 37 ms that 64 instances of 20..60 items spent in construction kernels.
constexpr int kLongRun = 12;
constexpr int kLongStage = 2048;

__global__ void __launch_bounds__(NT) kp_flatten_kernel(const KpBuildJob *jobs) {
    const KpBuildJob &J = jobs[blockIdx.y];
    __shared__ int32_t warp_buf[32];
    __shared__ int32_t total, s_long, s_arc_base, s_lo, s_nodes;
    __shared__ int32_t stage[kLongStage];
    const int n = J.n, d = J.nobjs, tid = threadIdx.x, l = blockIdx.x;
    if (l >= n) return;
    const int64_t S = static_cast<int64_t>(J.cap) + 1;
    if (tid < 32) {  // nodes before layer l, in all, and arcs into the layers up to l
        int32_t lo = 0, nodes = 0, arcs = 0;
        for (int q = tid; q <= n; q += 32) {
            const int32_t k = J.classes[q];
            nodes += k;
            if (q < l) lo += k;
            if (q <= l) arcs += J.arcs_into[q];
        }
        for (int o = 16; o > 0; o >>= 1) {
            lo += __shfl_xor_sync(0xffffffffu, lo, o);
            nodes += __shfl_xor_sync(0xffffffffu, nodes, o);
            arcs += __shfl_xor_sync(0xffffffffu, arcs, o);
        }
        if (tid == 0) {
            s_lo = lo;
            s_nodes = nodes;
            s_arc_base = arcs;
            s_long = 0;
        }
    }
    __syncthreads();
    const int32_t lo = s_lo, N = s_nodes;
    if (tid == 0) J.layer_offsets[l] = lo;
    if (l == 0) {
        for (int r = tid; r <= n; r += NT)
            for (int o = 0; o < d; ++o) J.weights[r * d + o] = r == 0 ? 0 : J.profit[o * n + (r - 1)];
        if (tid == 0) {
            J.layer_offsets[n] = N - 1;  // the terminal
            J.layer_offsets[n + 1] = N;
            J.in_arc_offsets[0] = 0;
            J.in_arc_offsets[1] = 0;  // the root has no incoming arcs
            J.sd_order[N - 1] = 0;
        }
    }
    const int32_t Kp = J.classes[l], Kc = J.classes[l + 1];
    const int32_t base = lo + Kp;
    int32_t *s1 = J.first1 + base - 1, *e1 = J.last1 + base - 1, *s0 = J.first0 + base - 1, *e0 = J.last0 + base - 1;
    int32_t *deg = J.degree + base - 1;
    int32_t *longs = J.idx + l * S;  // children with a long run (the states are done with)
    const int32_t *cnew = J.cls_new + l * S, *c0 = J.cls_c0 + l * S, *c1 = J.cls_c1 + l * S;
    for (int32_t v = tid; v < Kc; v += NT) {
        s1[v] = -1;
        e1[v] = -1;
        s0[v] = -1;
        e0[v] = -1;
    }
    __syncthreads();
    // the parents of a child through one arc type are a run of classes in state order
    for (int32_t p = tid; p < Kp; p += NT) {
        const int32_t v1 = c1[p], v0 = c0[p];
        if (v1 >= 0 && v1 < Kc) {
            if (p == 0 || c1[p - 1] != v1) s1[v1] = p;
            if (p == Kp - 1 || c1[p + 1] != v1) e1[v1] = p;
        }
        if (v0 >= 0 && v0 < Kc) {
            if (p == 0 || c0[p - 1] != v0) s0[v0] = p;
            if (p == Kp - 1 || c0[p + 1] != v0) e0[v0] = p;
        }
        J.sd_order[lo + (Kp - 1 - p)] = cnew[p];
    }
    __syncthreads();
    for (int32_t v = tid; v < Kc; v += NT)
        deg[v] = (s1[v] >= 0 ? e1[v] - s1[v] + 1 : 0) + (s0[v] >= 0 ? e0[v] - s0[v] + 1 : 0);
    __syncthreads();
    block_scan_array(deg, Kc, warp_buf, &total);
    for (int32_t v = tid; v < Kc; v += NT) {
        int32_t a = s_arc_base + deg[v];
        bool any_long = false;
#pragma unroll 1
        for (int t = 1; t >= 0; --t) {
            const int32_t sb = t ? s1[v] : s0[v], se = t ? e1[v] : e0[v];
            if (sb < 0) continue;
            const int32_t a0 = a;
            if (se - sb >= kLongRun) {  // for the whole block
                any_long = true;
                a += se - sb + 1;
                continue;
            }
            for (int32_t p = sb; p <= se; ++p) {
                const int32_t u = cnew[p];
                // insertion into [a0, a) kept ascending by parent id
                int32_t q = a;
                while (q > a0 && J.arc_src[q - 1] > lo + u) {
                    J.arc_src[q] = J.arc_src[q - 1];
                    --q;
                }
                J.arc_src[q] = lo + u;
                J.arc_weight[a] = t ? 1 + l : 0;
                ++a;
            }
        }
        J.in_arc_offsets[base + v + 1] = a;
        if (any_long) longs[atomicAdd(&s_long, 1)] = v;
    }
    __syncthreads();
    // long runs: each parent's place is the number of smaller ids in the run
    const int32_t num_long = s_long;
    for (int32_t i = 0; i < num_long; ++i) {
        const int32_t v = longs[i];
        int32_t a = s_arc_base + deg[v];
#pragma unroll 1
        for (int t = 1; t >= 0; --t) {
            const int32_t sb = t ? s1[v] : s0[v], se = t ? e1[v] : e0[v];
            if (sb < 0) continue;
            const int32_t len = se - sb + 1;
            if (len > kLongRun) {
                for (int32_t p0 = 0; p0 < len; p0 += NT) {
                    const int32_t p = p0 + tid;
                    const int32_t u = p < len ? cnew[sb + p] : 0;
                    int32_t place = 0;
                    for (int32_t q0 = 0; q0 < len; q0 += kLongStage) {
                        const int32_t m = min(kLongStage, len - q0);
                        __syncthreads();
                        for (int32_t q = tid; q < m; q += NT) stage[q] = cnew[sb + q0 + q];
                        __syncthreads();
                        if (p < len)
                            for (int32_t q = 0; q < m; ++q) place += stage[q] < u ? 1 : 0;
                    }
                    if (p < len) {
                        J.arc_src[a + place] = lo + u;
                        J.arc_weight[a + place] = t ? 1 + l : 0;
                    }
                }
            }
            a += len;
        }
    }
}

__global__ void __launch_bounds__(NT) kp_minw_kernel(const KpBuildJob *jobs) {
    const KpBuildJob &J = jobs[blockIdx.x];
    const int n = J.n, tid = threadIdx.x;
    const int64_t S = static_cast<int64_t>(J.cap) + 1;
    const int32_t *lo = J.layer_offsets;
    if (tid == 0) J.min_weight[0] = 0;
    __syncthreads();
    for (int l = 0; l < n; ++l) {
        const int32_t wl = J.w[l];
        for (int32_t v = lo[l + 1] + tid; v < lo[l + 2]; v += NT) {
            int32_t mw = INT_MAX;
            for (int32_t a = J.in_arc_offsets[v]; a < J.in_arc_offsets[v + 1]; ++a)
                mw = min(mw, J.min_weight[J.arc_src[a]] + (J.arc_weight[a] != 0 ? wl : 0));
            J.min_weight[v] = mw == INT_MAX ? 0 : mw;
        }
        __syncthreads();
    }
    // min_weight order per layer (descending, ties by id): the reverse state order of the
    // classes, since a class's min_weight is its smallest reachable state
    for (int l = 0; l < n; ++l) {
        const int32_t K = J.classes[l];
        const int32_t *cnew = J.cls_new + l * S;
        for (int32_t p = tid; p + 1 < K; p += NT)
            if (J.min_weight[lo[l] + cnew[p]] >= J.min_weight[lo[l] + cnew[p + 1]]) atomicMax(J.err, 2);
    }
}

cudaError_t launch_kp_reduce(const KpBuildJob *jobs, int count, cudaStream_t stream) {
    if (count <= 0) return cudaSuccess;
    kp_reduce_kernel<<<count, NT, 0, stream>>>(jobs);
    return cudaGetLastError();
}

cudaError_t launch_kp_flatten(const KpBuildJob *jobs, int count, int max_layers, cudaStream_t stream) {
    if (count <= 0) return cudaSuccess;
    for (int at = 0; at < count; at += 32768)  // grid.y
        kp_flatten_kernel<<<dim3(max_layers, std::min(count - at, 32768)), NT, 0, stream>>>(jobs + at);
    kp_minw_kernel<<<count, NT, 0, stream>>>(jobs);
    return cudaGetLastError();
}

}  // namespace dev
}  // namespace pmdd
