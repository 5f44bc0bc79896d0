// Fused expand + dominance filter for three objectives, in lexicographic order.
//
// Every node's frontier is kept in descending lexicographic order (objective 0, then 1,
// then 2).  Adding an arc's weight vector to every point of a frontier keeps that order,
// so the candidates of one arc ("a run") arrive sorted, and a destination's candidates
// are a few sorted runs.  In that order a point can only be dominated by a point before
// it, and since every point before q has objective 0 >= q's, q is dominated (or a later
// copy of an equal point) iff some earlier point has objectives 1 and 2 both >= q's: a
// two-dimensional question.
//
//   stage:   as the pairwise tile kernel (tile.cu): destinations and their arcs, with
//            each arc's parent flag "frontier sorted";
//   expand:  candidate = parent point + arc weight, in run order;
//   merge:   each candidate's position in its destination's lexicographic order is its
//            index in its run plus, per other run, a binary search for how many of that
//            run's points come before it (equal points: the lower run first); a
//            destination with a run from an unsorted parent counts the points before it
//            instead;
//   filter:  a warp per chunk of 32 consecutive merged positions, whatever destinations
//            they belong to.  First every candidate against the 32 of its chunk (bit masks
//            of the ones >= it in objective 1, and in both); a destination that goes on
//            past the chunk leaves its staircase there: the chunk's survivors of that
//            destination by objective 1 descending, with the running maximum of objective
//            2, so that one binary search answers the question for the whole chunk.  Then,
//            after a barrier, the survivors of a destination that began in an earlier chunk
//            ask the staircases of the chunks in between (destinations of at most
//            J.pair_max candidates: look at those points one by one);
//   write:   survivors go to the destination's slot in merged order, so the next
//            layer's runs are sorted again (out_sorted = 1).
//
// Every warp has the same work in the first half of the filter and one uniform loop in the
// second.  It replaced one staircase warp per 64-candidate segment, whose walks were serial
// chains of shuffles (51 % of the kernel's time, its warps 61 % busy): 1.68 G -> 0.93 G warp
// instructions on a captured launch of the 192-instance stream.  The kernel waits on
// barriers, shared-memory latency and dependent loads, not on a unit (issue slots 56 % busy,
// ALU 51 %): tile time of that stream's 684 M candidates 73.8 ms before, 49.7 ms with the
// chunk filter at 512 threads and 79 KB, 40.3 ms with four blocks of 256 threads per SM,
// the merge in place and the next tile fetched ahead (one B200).
//
// The keep rule is the reference GPU filter's (src/pmdd/enum/gpu/dominance_utils.cuh:
// 10-23): q is dropped iff another candidate p of the destination has p >= q on every
// objective and (p != q or p comes first).  Of equal points the first in the merged order
// stays; which copy stays does not change the frontier.  Oversized destinations are
// left to big.cu, whose output is not in this order (out_sorted = 0): their children
// merge by counting.
#include "kernels.cuh"
#include "scan.cuh"

#include <algorithm>
#include <climits>

namespace pmdd {
namespace dev {

namespace {

// 256 threads and 55 KB of shared memory (int32): four blocks share an SM, so that one
// block's barriers and dependent loads are covered by the others.
constexpr int kLT = 256;
constexpr int kLexWarps = kLT / 32;
constexpr int kChunks = kTileCap / 32;
constexpr unsigned kFull = 0xffffffffu;

// What the merge needs and the filter does not.
struct LexStage {
    int16_t tag[kTileCap];               // staged arc of each candidate, then its merged position
    int16_t arc_pos[kTileArcCap + 1];    // staged arc -> first candidate position
    int16_t arc_item[kTileArcCap];       // staged arc -> staged destination
    int32_t arc_w[kTileArcCap];          // staged arc -> weight row
    int32_t arc_nbr[kTileArcCap];        // staged arc -> job-local neighbour
};

template <typename T>
struct LexSmem {
    alignas(16) T p0[kTileCap], p1[kTileCap], p2[kTileCap];  // candidates: run order, then merged order
    union {
        LexStage a;
        struct {
            T s1[kTileCap], s2[kTileCap];  // chunk staircases: objective 1 descending, running
        } f;                               // maximum of objective 2
    };
    uint16_t item_of[kTileCap];          // staged destination of each candidate (either order)
    uint32_t keep[kChunks];              // survivors of each chunk of merged positions
    int32_t kept_ex[kChunks];            // survivors before each chunk
    int16_t item_s[kTileItemCap + 1];    // staged destination -> first candidate position
    int16_t item_arc0[kTileItemCap + 1]; // staged destination -> first staged arc
    int32_t item_a0g[kTileItemCap];      // staged destination -> first arc (global id)
    int64_t item_c0[kTileItemCap];       // staged destination -> job-local candidate start
    uint8_t item_count[kTileItemCap];    // 1: merge by counting
    int64_t warp_l[32], tot_l;           // scans
    int32_t warp_i[32];
    int32_t tot_i, tot_a;
    int32_t next_chunk, n_stair;
    int64_t tile[2];                     // tiles taken from the launch's queue: this one, the next
    int32_t job[2], i0[2], i1[2];        // their jobs and destinations
};

// Phase clock (J.phase_clk, a diagnostic): thread 0 adds the cycles its block spent in
// each phase of a pass (stage destinations, stage arcs, arc assignment, expand, merge,
// filter, scan and write) to the job's counters.
struct PhaseClock {
    unsigned long long *out;
    long long t;
    __device__ __forceinline__ void start() {
        if (out) t = clock64();
    }
    __device__ __forceinline__ void lap(int phase) {
        if (out) {
            const long long now = clock64();
            atomicAdd(out + phase, static_cast<unsigned long long>(now - t));
            t = now;
        }
    }
};

// Largest x over the threads before this one (-1 for thread 0); every thread calls it.
template <int THREADS>
__device__ __forceinline__ int32_t block_exclusive_max(int32_t x, int32_t *warp_buf) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int32_t inc = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int32_t y = __shfl_up_sync(kFull, inc, o);
        if (lane >= o) inc = max(inc, y);
    }
    int32_t exc = __shfl_up_sync(kFull, inc, 1);
    if (lane == 0) exc = -1;
    if (lane == 31) warp_buf[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        const int32_t w = lane < THREADS / 32 ? warp_buf[lane] : -1;
        int32_t winc = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int32_t y = __shfl_up_sync(kFull, winc, o);
            if (lane >= o) winc = max(winc, y);
        }
        int32_t wexc = __shfl_up_sync(kFull, winc, 1);
        if (lane == 0) wexc = -1;
        if (lane < THREADS / 32) warp_buf[lane] = wexc;
    }
    __syncthreads();
    const int32_t r = max(exc, warp_buf[warp]);
    __syncthreads();  // warp_buf may be reused right after
    return r;
}

template <typename T>
__device__ __forceinline__ T lowest() {
    return sizeof(T) == 4 ? static_cast<T>(INT32_MIN) : static_cast<T>(INT64_MIN);
}

// Bits j of the chunk's 32 positions at c0 with m1[c0 + j] >= q1 (*ge1, with WITH_GE1) and
// with both objectives >= (q1, q2) (returned).  Warp-uniform addresses, 16 bytes at a time.
template <typename T, bool WITH_GE1>
__device__ __forceinline__ unsigned chunk_masks(const T *m1, const T *m2, T q1, T q2, unsigned *ge1) {
    struct alignas(16) V {
        T v[16 / sizeof(T)];
    };
    constexpr int W = 16 / sizeof(T);
    unsigned both = 0, g1 = 0;
#pragma unroll
    for (int j = 0; j < 32; j += W) {
        const V a = *reinterpret_cast<const V *>(m1 + j);
        const V b = *reinterpret_cast<const V *>(m2 + j);
#pragma unroll
        for (int u = 0; u < W; ++u) {
            const bool g = a.v[u] >= q1;
            if (WITH_GE1 && g) g1 |= 1u << (j + u);
            if (g && b.v[u] >= q2) both |= 1u << (j + u);
        }
    }
    if (WITH_GE1) *ge1 = g1;
    return both;
}

// Has the staircase at s1 / s2 (32 entries) a point >= (q1, q2) in both?
template <typename T>
__device__ __forceinline__ bool stair_covers(const T *s1, const T *s2, T q1, T q2) {
    int at = 0;  // entries with objective 1 >= q1
#pragma unroll
    for (int step = 16; step > 0; step >>= 1)
        if (s1[at + step - 1] >= q1) at += step;
    if (s1[at] >= q1) ++at;  // at <= 31: the 32nd entry
    return at > 0 && s2[at - 1] >= q2;
}

}  // namespace

template <typename T>
__global__ void __launch_bounds__(kLT) expand_tile_lex_kernel(const ExpandJob *__restrict__ jobs,
                                                              const int64_t *__restrict__ tile_bases, int num_jobs,
                                                              int64_t total_tiles, unsigned long long *queue,
                                                              const int64_t *tiles_dev) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    LexSmem<T> &S = *reinterpret_cast<LexSmem<T> *>(smem_raw);
    const int tid = threadIdx.x, lane = tid & 31;
    const unsigned lt_mask = (1u << lane) - 1u;
    // jobs sized on the device (chain.cu) publish their tiles' total there
    if (tiles_dev != nullptr) total_tiles = min(total_tiles, *tiles_dev);
    // Tiles are handed out by an atomic counter over all the launch's jobs, so a block
    // that drew cheap tiles takes more.  One warp fetches the tile after the current one
    // while the others finish it: its job (32 bases at a time) and destinations.
    auto fetch = [&](int slot) {
        int64_t t = 0;
        if (lane == 0) t = static_cast<int64_t>(atomicAdd(queue, 1ull));
        t = __shfl_sync(kFull, t, 0);
        int j = 0;
        if (t < total_tiles) {
            int n = num_jobs;  // the last job in [j, j + n) whose first tile is <= t
            while (n > 1) {
                const int step = (n + 31) >> 5;
                const int at = j + lane * step;
                const unsigned m = __ballot_sync(kFull, lane * step < n && __ldg(tile_bases + at) <= t);
                const int last = 31 - __clz(m | 1u);
                j += last * step;
                n = min(step, n - last * step);
            }
        }
        if (lane == 0) {
            S.tile[slot] = t;
            if (t < total_tiles) {
                const ExpandJob &J = jobs[j];
                const int64_t x = t - tile_bases[j];
                S.job[slot] = j;
                // a job sized on the device may have fewer tiles than the launch allows for
                S.i0[slot] = x < J.num_tiles ? J.tile_first[x] : 0;
                S.i1[slot] = x < J.num_tiles ? J.tile_first[x + 1] : 0;
            }
        }
    };
    int cur = 0;
    if (tid < 32) fetch(0);
    __syncthreads();
    for (; S.tile[cur] < total_tiles; cur ^= 1) {
        const ExpandJob &J = jobs[S.job[cur]];
        const int32_t i0 = S.i0[cur], i1 = S.i1[cur];
        const T *__restrict__ prev = static_cast<const T *>(J.prev_pts);
        T *__restrict__ outp = static_cast<T *>(J.out_pts);
        const int pair_max = J.pair_max;
        PhaseClock clk{tid == 0 ? J.phase_clk : nullptr, 0};
        clk.start();
        int32_t ic = i0;
        bool done = false;  // the last pass has fetched the next tile
        while (ic < i1) {
            const int n_stage = min(kTileItemCap, i1 - ic);
            // --- stage destinations: candidate starts and sizes, arc ranges
            constexpr int PER = kTileItemCap / kLT;
            static_assert(PER >= 1, "one destination per thread at least");
            int32_t cnt[PER], narc[PER];
            int32_t local = 0, local_a = 0;
#pragma unroll
            for (int r = 0; r < PER; ++r) {
                const int k = tid * PER + r;
                cnt[r] = 0;
                narc[r] = 0;
                if (k < n_stage) {
                    const int32_t i = ic + k;
                    const int32_t v = J.item_base + i;
                    const int32_t a0 = J.item_arc_off[v], a1 = J.item_arc_off[v + 1];
                    const int64_t s = J.arc_cand_off[a0 - J.arc_base];
                    const int64_t c = J.arc_cand_off[a1 - J.arc_base] - s;
                    J.out_off[i] = s;
                    const bool resident = c > 0 && tile_resident(c, a1 - a0);
                    if (c == 0) J.out_size[i] = 0;
                    if (J.out_sorted) J.out_sorted[i] = (c == 0 || resident) ? 1 : 0;
                    S.item_c0[k] = s;
                    S.item_a0g[k] = a0;
                    S.item_count[k] = 0;
                    if (resident) {
                        cnt[r] = static_cast<int32_t>(c);
                        narc[r] = a1 - a0;
                    }
                }
                local += cnt[r];
                local_a += narc[r];
            }
            // candidates and arcs before this thread's destinations, in one scan
            const int64_t exl = block_exclusive_scan<int64_t, kLT>(
                (static_cast<int64_t>(local_a) << 32) | local, S.warp_l, &S.tot_l);
            // this pass takes the longest prefix of staged destinations whose arcs fit
            int fit = 0;
            int32_t end_s[PER], end_a[PER];  // where this thread's destinations end
            {
                int32_t run = static_cast<int32_t>(exl & 0xffffffff), runa = static_cast<int32_t>(exl >> 32);
#pragma unroll
                for (int r = 0; r < PER; ++r) {
                    const int k = tid * PER + r;
                    if (k < n_stage) {
                        S.item_s[k] = static_cast<int16_t>(run);
                        S.item_arc0[k] = static_cast<int16_t>(runa);
                        if (runa + narc[r] <= kTileArcCap) fit = k + 1;
                    }
                    run += cnt[r];
                    runa += narc[r];
                    end_s[r] = run;
                    end_a[r] = runa;
                }
            }
            fit = __reduce_max_sync(kFull, fit);
            if (lane == 0) S.warp_i[tid >> 5] = fit;
            __syncthreads();
            int n_it = 0;  // >= 1: one destination has at most kTileArcCap / 2 arcs
#pragma unroll
            for (int w = 0; w < kLexWarps; ++w) n_it = max(n_it, S.warp_i[w]);
            if (n_it == 0) {           // impossible for well-formed plans; skip defensively
                if (tid == 0) atomicOr(J.err, kErrBounds);
                break;
            }
            // end markers of this pass, from the thread that staged its last destination
#pragma unroll
            for (int r = 0; r < PER; ++r) {
                if (tid * PER + r == n_it - 1) {
                    S.item_s[n_it] = static_cast<int16_t>(end_s[r]);
                    S.item_arc0[n_it] = static_cast<int16_t>(end_a[r]);
                    S.tot_i = end_s[r];
                    S.tot_a = end_a[r];
                }
            }
            if (tid == 0) {
                S.next_chunk = 0;
                S.n_stair = 0;
            }
            __syncthreads();
            const int32_t total = S.tot_i, total_a = S.tot_a;
            if (total > kTileCap || total_a > kTileArcCap) {  // impossible for well-formed offsets
                if (tid == 0) atomicOr(J.err, kErrBounds);
                break;
            }
            clk.lap(0);
            // --- stage the arcs of the small destinations (and whether each parent is sorted)
            for (int x = tid; x < total_a; x += kLT) {
                int lo = 0, hi = n_it - 1;  // destination owning staged arc x
                while (lo < hi) {
                    const int mid = (lo + hi + 1) >> 1;
                    if (S.item_arc0[mid] <= x) lo = mid;
                    else hi = mid - 1;
                }
                const int k = lo;
                const int32_t a = S.item_a0g[k] + (x - S.item_arc0[k]);
                const int64_t c0 = J.arc_cand_off[a - J.arc_base];
                const int32_t nb = J.arc_nbr[a] - J.prev_base;
                S.a.arc_pos[x] = static_cast<int16_t>(S.item_s[k] + (c0 - S.item_c0[k]));
                S.a.arc_nbr[x] = nb;
                S.a.arc_w[x] = J.arc_wrow[a];
                S.a.arc_item[x] = static_cast<int16_t>(k);
                if (J.prev_sorted == nullptr || J.prev_sorted[nb] == 0) S.item_count[k] = 1;
            }
            if (tid == 0) S.a.arc_pos[total_a] = static_cast<int16_t>(total);
            for (int q = tid; q < total; q += kLT) S.a.tag[q] = -1;
            __syncthreads();
            clk.lap(1);
            // --- each candidate's arc: mark every non-empty run's first position, then a
            // block-wide running maximum carries the arc over its run
            for (int x = tid; x < total_a; x += kLT)
                if (S.a.arc_pos[x + 1] > S.a.arc_pos[x]) S.a.tag[S.a.arc_pos[x]] = static_cast<int16_t>(x);
            __syncthreads();
            {
                constexpr int QP = kTileCap / kLT;
                int32_t run = -1, seen[QP];
#pragma unroll
                for (int r = 0; r < QP; ++r) {
                    const int q = tid * QP + r;
                    if (q < total) run = max(run, static_cast<int32_t>(S.a.tag[q]));
                    seen[r] = run;
                }
                const int32_t before = block_exclusive_max<kLT>(run, S.warp_i);
#pragma unroll
                for (int r = 0; r < QP; ++r) {
                    const int q = tid * QP + r;
                    if (q < total) S.a.tag[q] = static_cast<int16_t>(max(before, seen[r]));
                }
            }
            __syncthreads();
            clk.lap(2);
            // --- expand: candidate = parent point + arc weight (run order)
            for (int q = tid; q < total; q += kLT) {
                const int x = S.a.tag[q];
                const T *src = prev + (J.prev_off[S.a.arc_nbr[x]] + (q - S.a.arc_pos[x])) * 3;
                const int32_t *w = J.weights + static_cast<int64_t>(S.a.arc_w[x]) * 3;
                S.p0[q] = src[0] + static_cast<T>(w[0]);
                S.p1[q] = src[1] + static_cast<T>(w[1]);
                S.p2[q] = src[2] + static_cast<T>(w[2]);
                S.item_of[q] = static_cast<uint16_t>(S.a.arc_item[x]);
            }
            __syncthreads();
            clk.lap(3);
            // --- merge: each candidate's position in its destination's lexicographic order
            for (int q = tid; q < total; q += kLT) {
                const int k = S.item_of[q];
                const int x = S.a.tag[q];
                const int js = S.item_s[k], je = S.item_s[k + 1];
                const T q0 = S.p0[q], q1 = S.p1[q], q2 = S.p2[q];
                // is position j's point before this one (equal points: if `tie`)?
                auto before = [&](int j, bool tie) -> bool {
                    const T c0 = S.p0[j];
                    if (c0 != q0) return c0 > q0;
                    const T c1 = S.p1[j], c2 = S.p2[j];
                    if (c1 != q1) return c1 > q1;
                    if (c2 != q2) return c2 > q2;
                    return tie;
                };
                int rank = 0;
                if (S.item_count[k] == 0) {
                    rank = q - S.a.arc_pos[x];
                    const int y0 = S.item_arc0[k], y1 = S.item_arc0[k + 1];
                    for (int y = y0; y < y1; ++y) {
                        if (y == x) continue;
                        const int lo = S.a.arc_pos[y], hi = (y + 1 < y1) ? S.a.arc_pos[y + 1] : je;
                        // points of run y before me: larger, or equal in a lower run; a prefix
                        int a = lo, b = hi;
                        while (a < b) {
                            const int mid = (a + b) >> 1;
                            if (before(mid, y < x)) a = mid + 1;
                            else b = mid;
                        }
                        rank += a - lo;
                    }
                } else {
                    for (int j = js; j < je; ++j) rank += before(j, j < q) ? 1 : 0;
                }
                S.a.tag[q] = static_cast<int16_t>(js + rank);
            }
            {  // in place: every thread picks its candidates up before any is put down
                constexpr int QP = kTileCap / kLT;
                T v0[QP], v1[QP], v2[QP];
                int16_t to[QP];
#pragma unroll
                for (int r = 0; r < QP; ++r) {
                    const int q = tid + r * kLT;
                    to[r] = -1;
                    if (q < total) {
                        to[r] = S.a.tag[q];
                        v0[r] = S.p0[q];
                        v1[r] = S.p1[q];
                        v2[r] = S.p2[q];
                    }
                }
                __syncthreads();
#pragma unroll
                for (int r = 0; r < QP; ++r)
                    if (to[r] >= 0) {
                        S.p0[to[r]] = v0[r];
                        S.p1[to[r]] = v1[r];
                        S.p2[to[r]] = v2[r];
                    }
            }
            __syncthreads();
            clk.lap(4);
            const int chunks = (total + 31) >> 5;
            // --- filter inside the chunks, and the staircases of destinations that go on
            for (int c = tid >> 5; c < chunks; c += kLexWarps) {
                const int c0 = c << 5, q = c0 + lane;
                const bool valid = q < total;
                const T q1 = S.p1[q], q2 = S.p2[q];
                const int k = S.item_of[valid ? q : c0];
                const int js = S.item_s[k];
                // the chunk's candidates of the same destination before this one
                const unsigned mine = js > c0 ? ~((1u << (js - c0)) - 1u) : kFull;
                const int kl = __shfl_sync(kFull, k, 31);
                if (c0 + 32 >= total || S.item_s[kl + 1] <= c0 + 32) {
                    const unsigned both = chunk_masks<T, false>(S.p1 + c0, S.p2 + c0, q1, q2, nullptr);
                    const unsigned kept = __ballot_sync(kFull, valid && (both & mine & lt_mask) == 0);
                    if (lane == 0) S.keep[c] = kept;
                } else {
                    unsigned ge1;
                    const unsigned both = chunk_masks<T, true>(S.p1 + c0, S.p2 + c0, q1, q2, &ge1);
                    const unsigned kept = __ballot_sync(kFull, (both & mine & lt_mask) == 0);
                    const unsigned members = kept & __ballot_sync(kFull, k == kl);
                    const unsigned equal = __match_any_sync(kFull, q1);
                    T *s1 = S.f.s1 + c0, *s2 = S.f.s2 + c0;
                    if ((members >> lane) & 1u) {
                        const int at = __popc(members & ge1 & (~equal | lt_mask));
                        s1[at] = q1;
                        s2[at] = q2;
                    }
                    if (lane >= __popc(members)) {
                        s1[lane] = lowest<T>();
                        s2[lane] = lowest<T>();
                    }
                    __syncwarp();
                    T mx = s2[lane];
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const T y = __shfl_up_sync(kFull, mx, o);
                        if (lane >= o) mx = max(mx, y);
                    }
                    s2[lane] = mx;
                    if (lane == 0) S.keep[c] = kept;
                }
            }
            __syncthreads();
            // --- filter against the earlier chunks of the destination that reaches into the
            // chunk (at most one), the longest loops first
            while (true) {
                int c = 0;
                if (lane == 0) c = chunks - 1 - atomicAdd(&S.next_chunk, 1);
                c = __shfl_sync(kFull, c, 0);
                if (c <= 0) break;
                const int c0 = c << 5;
                const int k = S.item_of[c0];
                const int js = S.item_s[k], je = S.item_s[k + 1];
                if (js >= c0) continue;
                const int q = c0 + lane;
                const T q1 = S.p1[q], q2 = S.p2[q];
                const unsigned kept = S.keep[c];
                bool dom = q >= je || ((kept >> lane) & 1u) == 0;
                const unsigned others = je - c0 >= 32 ? 0u : kept & ~((1u << (je - c0)) - 1u);
                if (je - js <= pair_max) {
                    for (int j = js; j < c0; ++j) dom |= (S.p1[j] >= q1) & (S.p2[j] >= q2);
                } else {
                    for (int t = js >> 5; t < c && !__all_sync(kFull, dom); ++t)
                        dom |= stair_covers<T>(S.f.s1 + (t << 5), S.f.s2 + (t << 5), q1, q2);
                }
                const unsigned left = __ballot_sync(kFull, !dom);
                if (lane == 0) S.keep[c] = left | others;
            }
            // candidates of destinations above the pairwise limit (statistics)
            if (J.tile_surv != nullptr)
                for (int k = tid; k < n_it; k += kLT) {
                    const int c = S.item_s[k + 1] - S.item_s[k];
                    if (c > pair_max) atomicAdd(&S.n_stair, c);
                }
            __syncthreads();
            clk.lap(5);
            // --- survivors before each chunk (one warp); another fetches the next tile
            if (tid >= 32 && tid < 64 && ic + n_it >= i1) fetch(cur ^ 1);
            if (tid < 32) {
                static_assert(kChunks == 64, "two chunks per lane");
                const int a = 2 * lane < chunks ? __popc(S.keep[2 * lane]) : 0;
                const int b = 2 * lane + 1 < chunks ? __popc(S.keep[2 * lane + 1]) : 0;
                int inc = a + b;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int y = __shfl_up_sync(kFull, inc, o);
                    if (lane >= o) inc += y;
                }
                S.kept_ex[2 * lane] = inc - a - b;
                S.kept_ex[2 * lane + 1] = inc - b;
                if (lane == 31 && J.tile_surv != nullptr) {
                    if (inc > 0) atomicAdd(J.tile_surv, static_cast<unsigned long long>(inc));
                    if (S.n_stair > 0) atomicAdd(J.tile_surv + 1, static_cast<unsigned long long>(S.n_stair));
                }
            }
            __syncthreads();
            // survivors before merged position q
            auto kept_before = [&](int q) -> int {
                if (q == 0) return 0;
                const int c = (q - 1) >> 5;
                return S.kept_ex[c] + __popc(S.keep[c] & (kFull >> (31 - ((q - 1) & 31))));
            };
            // --- write survivors into each destination's slot, in merged order
            for (int q = tid; q < total; q += kLT) {
                if (((S.keep[q >> 5] >> (q & 31)) & 1u) == 0) continue;
                const int k = S.item_of[q];
                T *o_ = outp + (S.item_c0[k] + (kept_before(q) - kept_before(S.item_s[k]))) * 3;
                o_[0] = S.p0[q];
                o_[1] = S.p1[q];
                o_[2] = S.p2[q];
            }
            for (int k = tid; k < n_it; k += kLT) {
                const int js = S.item_s[k], je = S.item_s[k + 1];
                if (je > js) J.out_size[ic + k] = kept_before(je) - kept_before(js);
            }
            __syncthreads();
            clk.lap(6);
            ic += n_it;
            done = ic >= i1;
        }
        if (!done) {  // an empty tile, or one given up
            if (tid < 32) fetch(cur ^ 1);
            __syncthreads();
        }
    }
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
    expand_tile_lex_kernel<T><<<static_cast<unsigned>(g), kLT, smem, stream>>>(jobs, tile_bases, num_jobs,
                                                                              total_tiles, queue, tiles_dev);
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
