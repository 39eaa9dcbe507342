// Graph construction: LightGraph::buildGraph (src/LightGraph.h:287-318).
//
// The reference loops i = 0..N-1, j = 0..N-1 and connects i < j when
// |p_i - p_j|^2 < r^2 (FP64 on float-valued points) unless either endpoint
// already has max_connect edges. The decision for row i depends only on the
// edge counts left by rows < i, and inside one row every partner j is
// independent, so:
//   1. k_candidates (parallel over rows): the ascending list of j > i with
//      |p_i - p_j|^2 < r^2. The test runs in FP32; only pairs inside a
//      2^-17 relative band of r^2 (where FP32 rounding could disagree with the
//      reference's FP64) are re-tested with FP64 arithmetic.
//   2. k_greedy (one CTA per graph, rows in order): a warp takes the first
//      (max_connect - cnt[i]) candidates whose partner count is below the cap;
//   or, for graphs of many points with few partners each (sweep_form):
//   2. k_lower (parallel over rows): the same for j < i;
//   3. k_pair_sweep (a warp per point) decides the pairs many at a time, in no
//      set order but with the outcome of the set one, and k_pair_finish (one
//      CTA per graph) writes the edges in order.
#include <algorithm>
#include <mutex>
#include <utility>
#include <vector>

#include "lg_kernels.h"

namespace lg {

__device__ __forceinline__ bool pair_close(const float* pi, const float* pj, float r2, float lo,
                                           float hi) {
    const float dx = pi[0] - pj[0], dy = pi[1] - pj[1], dz = pi[2] - pj[2];
    const float d2 = __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
    if (d2 < lo) return true;
    if (d2 > hi) return false;
    // near the radius: evaluate exactly as the reference does, in FP64
    // without contraction (Vec3::lengthSqr, x*x + y*y + z*z left to right)
    const double ex = __dsub_rn((double)pi[0], (double)pj[0]);
    const double ey = __dsub_rn((double)pi[1], (double)pj[1]);
    const double ez = __dsub_rn((double)pi[2], (double)pj[2]);
    const double e2 = __dadd_rn(__dadd_rn(__dmul_rn(ex, ex), __dmul_rn(ey, ey)), __dmul_rn(ez, ez));
    return e2 < (double)r2;
}

// A graph's sum of candidate counts from here on: some list does not hold all
// of its row's partners, which rules the sweep form out. (Set by a maximum, not
// added: the counts of all other rows together stay below 2^23, so it is neither
// reached by them nor carried past 2^31.)
constexpr int32_t kListsOverflow = 1 << 30;
static_assert(65535 * kCandCap < (1 << 23), "the largest graph with full lists");

// One warp per row; rows of all graphs in one launch.
__global__ void __launch_bounds__(256) k_candidates(const float* __restrict__ pts,
                                                    const GraphInfo* __restrict__ graphs,
                                                    const int32_t* __restrict__ pt_graph,
                                                    int64_t n_points, uint16_t* __restrict__ cand,
                                                    int32_t* __restrict__ cand_cnt, int32_t* __restrict__ sums) {
    const int64_t row = (int64_t)blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32;
    const int lane = threadIdx.x & 31;
    if (row >= n_points) return;
    const GraphInfo g = graphs[pt_graph[row]];
    const int i = (int)(row - g.pt_off);
    const float* P = pts + 3 * g.pt_off;
    const float pi[3] = {P[3 * i], P[3 * i + 1], P[3 * i + 2]};
    const float lo = g.r2 * (1.f - 7.62939453125e-06f), hi = g.r2 * (1.f + 7.62939453125e-06f);
    int cnt = 0;
    uint16_t* out = cand + row * kCandCap;
    for (int j0 = i + 1; j0 < g.n; j0 += 32) {
        const int j = j0 + lane;
        bool close = false;
        if (j < g.n) {
            const float pj[3] = {P[3 * j], P[3 * j + 1], P[3 * j + 2]};
            close = pair_close(pi, pj, g.r2, lo, hi);
        }
        const unsigned m = __ballot_sync(0xffffffffu, close);
        const int pos = cnt + __popc(m & ((1u << lane) - 1u));
        if (close && pos < kCandCap) out[pos] = (uint16_t)j;
        cnt += __popc(m);
    }
    if (lane == 0) {
        cand_cnt[row] = cnt;
        if (sums) {
            if (cnt > kCandCap) atomicMax(sums + pt_graph[row], kListsOverflow);
            else atomicAdd(sums + pt_graph[row], cnt);
        }
    }
}

// Whether a graph of n points whose candidate counts add up to sum is decided
// by sweeps. Row by row the edges take ~0.124 us a point; sweeps take a chain
// of pairs that wait for one another, about as long as the neighbourhood of
// twice the radius (8 partner counts), at ~0.7 us each, and ~20 us to start:
// 4096 points with 22 partners 0.51 against 0.13 ms; 3531 points with 160
// partners 0.44 against 1.3 ms.
__device__ __forceinline__ bool sweep_form(int n, int32_t sum) {
    return sum < kListsOverflow && (int64_t)n * (n - 160) > 45 * 2 * (int64_t)sum;
}

// One CTA per graph. Candidate rows are staged into shared memory in chunks
// of 64 rows, double buffered: warp 0 resolves the rows of one chunk in order
// while warps 1-7 stage the next.
constexpr int kGreedyChunk = 64;
static_assert((kCandCap * sizeof(uint16_t)) % sizeof(uint4) == 0, "candidate rows are copied as 16-byte words");

// A chunk's candidate rows are one contiguous block of rows * kCandCap
// entries whose start, (pt_off + r0) * 192 bytes into the array, is 16-byte
// aligned: it is copied as 16-byte words, every load independent of the
// others (entries past a row's count are copied too and never read).
__device__ __forceinline__ void greedy_stage(const GraphInfo& g, const uint16_t* __restrict__ cand,
                                             const int32_t* __restrict__ cand_cnt, int r0, int rows, uint16_t* cs,
                                             int32_t* cc, int t, int nt) {
    constexpr int kWordsPerRow = kCandCap * (int)sizeof(uint16_t) / (int)sizeof(uint4);
    const uint4* __restrict__ src = reinterpret_cast<const uint4*>(cand + (g.pt_off + r0) * kCandCap);
    uint4* dst = reinterpret_cast<uint4*>(cs);
    const int words = rows * kWordsPerRow;
#pragma unroll 4
    for (int k = t; k < words; k += nt) dst[k] = __ldg(src + k);
    for (int k = t; k < rows; k += nt) cc[k] = cand_cnt[g.pt_off + r0 + k];
}

__global__ void __launch_bounds__(256) k_greedy(const float* __restrict__ pts,
                                                const GraphInfo* __restrict__ graphs,
                                                const uint16_t* __restrict__ cand,
                                                const int32_t* __restrict__ cand_cnt,
                                                int max_connect, int2* __restrict__ edges,
                                                int32_t* __restrict__ edge_cnt, const int32_t* __restrict__ sums) {
    extern __shared__ __align__(16) uint8_t smem[];
    const GraphInfo g = graphs[blockIdx.x];
    const int n = g.n;
    if (sums && sweep_form(n, sums[blockIdx.x])) return;
    uint16_t* cs2 = reinterpret_cast<uint16_t*>(smem);                       // 2 x chunk x cap
    int32_t* cc2 = reinterpret_cast<int32_t*>(cs2 + 2 * kGreedyChunk * kCandCap);  // 2 x chunk
    uint8_t* cnt = reinterpret_cast<uint8_t*>(cc2 + 2 * kGreedyChunk);        // n
    for (int k = threadIdx.x; k < n; k += blockDim.x) cnt[k] = 0;
    if (n > 0) greedy_stage(g, cand, cand_cnt, 0, min(kGreedyChunk, n), cs2, cc2, threadIdx.x, blockDim.x);
    const int lane = threadIdx.x & 31;
    const float* P = pts + 3 * g.pt_off;
    const float lo = g.r2 * (1.f - 7.62939453125e-06f), hi = g.r2 * (1.f + 7.62939453125e-06f);
    int ecount = 0;  // valid in warp 0
    int2* E = edges + g.e_off;
    for (int r0 = 0, buf = 0; r0 < n; r0 += kGreedyChunk, buf ^= 1) {
        const int rows = min(kGreedyChunk, n - r0);
        __syncthreads();  // chunk r0 staged; the other buffer is free
        const uint16_t* cs = cs2 + buf * kGreedyChunk * kCandCap;
        const int32_t* cc = cc2 + buf * kGreedyChunk;
        if (threadIdx.x >= 32) {
            const int r1 = r0 + kGreedyChunk;
            if (r1 < n)
                greedy_stage(g, cand, cand_cnt, r1, min(kGreedyChunk, n - r1), cs2 + (buf ^ 1) * kGreedyChunk * kCandCap,
                             cc2 + (buf ^ 1) * kGreedyChunk, threadIdx.x - 32, blockDim.x - 32);
        } else {
            // A row's candidates do not depend on the edge counts: its count and
            // first 64 are loaded during the row before, and both batches are
            // decided without a branch, so that the chain of a row is the loads
            // of the counts, two ballots and the update (1024 points with 90
            // partners: 213 -> 127 us; 32 graphs of 257 to 3805: 724 -> 436 us).
            const unsigned below = (1u << lane) - 1u;
            int next_total = cc[0], next_a = cs[lane], next_b = cs[32 + lane];
            for (int r = 0; r < rows; ++r) {
                const int i = r0 + r;
                const int total = next_total, ja = next_a, jb = next_b;
                const int rn = min(r + 1, rows - 1);
                next_total = cc[rn];
                next_a = cs[rn * kCandCap + lane];
                next_b = cs[rn * kCandCap + 32 + lane];
                const int stored = min(total, kCandCap);
                const int ci = cnt[i];
                const int ca = lane < stored ? (int)cnt[ja] : max_connect;
                const int cb = 32 + lane < stored ? (int)cnt[jb] : max_connect;
                int need = max(max_connect - ci, 0);
                const unsigned ma = __ballot_sync(0xffffffffu, ca < max_connect);
                const unsigned mb = __ballot_sync(0xffffffffu, cb < max_connect);
                const int ra = __popc(ma & below), rb = __popc(ma) + __popc(mb & below);
                if (ca < max_connect && ra < need) {
                    cnt[ja] = (uint8_t)(ca + 1);
                    E[ecount + ra] = make_int2(i, ja);
                }
                if (cb < max_connect && rb < need) {
                    cnt[jb] = (uint8_t)(cb + 1);
                    E[ecount + rb] = make_int2(i, jb);
                }
                const int got = min(__popc(ma) + __popc(mb), need);
                need -= got;
                ecount += got;
                __syncwarp();
                if (need == 0 || stored <= 64) continue;
                static_assert(kCandCap == 96, "one more batch");
                {
                    const int j = 64 + lane < stored ? cs[r * kCandCap + 64 + lane] : 0;
                    const int c = 64 + lane < stored ? (int)cnt[j] : max_connect;
                    const unsigned m = __ballot_sync(0xffffffffu, c < max_connect);
                    const int rank = __popc(m & below);
                    if (c < max_connect && rank < need) {
                        cnt[j] = (uint8_t)(c + 1);
                        E[ecount + rank] = make_int2(i, j);
                    }
                    const int acc = min(__popc(m), need);
                    need -= acc;
                    ecount += acc;
                    __syncwarp();
                }
                if (need > 0 && total > kCandCap) {
                    // more partners than stored: continue the scan past the last stored one
                    const int jstart = cs[r * kCandCap + kCandCap - 1] + 1;
                    const float pi[3] = {P[3 * i], P[3 * i + 1], P[3 * i + 2]};
                    for (int j0 = jstart; j0 < n && need > 0; j0 += 128) {
                        // four batches: their loads and tests are independent
                        bool elig[4];
#pragma unroll
                        for (int b = 0; b < 4; ++b) {
                            const int j = j0 + 32 * b + lane;
                            elig[b] = false;
                            if (j < n) {
                                const float pj[3] = {P[3 * j], P[3 * j + 1], P[3 * j + 2]};
                                elig[b] = pair_close(pi, pj, g.r2, lo, hi) && (int)cnt[j] < max_connect;
                            }
                        }
#pragma unroll
                        for (int b = 0; b < 4; ++b) {
                            const int j = j0 + 32 * b + lane;
                            const unsigned m = __ballot_sync(0xffffffffu, elig[b]);
                            const int rank = __popc(m & below);
                            if (elig[b] && rank < need) {
                                cnt[j] = cnt[j] + 1;
                                E[ecount + rank] = make_int2(i, j);
                            }
                            const int acc = min(__popc(m), need);
                            need -= acc;
                            ecount += acc;
                        }
                        __syncwarp();
                    }
                }
                // cnt[i] is not written back: later rows read only the
                // counts of partners j > their own row, never row i's
            }
        }
    }
    if (threadIdx.x == 0) edge_cnt[blockIdx.x] = ecount;
}

// Sweeps. A point's partners in ascending order are its pairs in the order they
// are taken. With A a point's connected pairs and U its undecided ones so
// far, a pair is below the cap at that point for certain when fewer than
// max_connect of A and U come before it, and above it for certain when
// max_connect of A do. The first holds for the partners before the
// (max_connect + 1)-th of A and U, the second for those past the max_connect-th
// of A: two partner numbers a point (its limit), which is all that its
// partners need of it. A pair is dropped once either end is certainly above,
// and connected once both are certainly below; the first undecided pair in the
// order is always one of the two, so some can always be decided, and what is
// certain stays so, whichever of a point's limits a partner happens to read:
// no barriers, no order. A warp holds a point: its partners' numbers, a lane
// for every 32nd, and their state stay in registers while it reads the
// partners' limits again and again. Bound by latency: a read through L2 for
// each pair of the longest chain that wait for one another.
constexpr int kListWords = kCandCap / 32;
constexpr int kWords = 2 * kListWords;  // the partners below, then those above
constexpr uint32_t kNoLimit = 0xFFFFu;
// Sweeps without a change after which a warp leaves the rest to k_pair_finish
// (the launch has no more warps than fit the GPU, but other work may hold some
// back).
constexpr int kStalled = 1024;

__device__ __forceinline__ uint32_t ld_limit(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_limit(uint32_t* p, uint32_t v) {
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// The partners below each point (k_candidates' counterpart), its first limit
// and an empty state.
__global__ void __launch_bounds__(256) k_lower(const float* __restrict__ pts, const GraphInfo* __restrict__ graphs,
                                               const int32_t* __restrict__ pt_graph, int64_t n_points, int max_connect,
                                               const uint16_t* __restrict__ cand, const int32_t* __restrict__ cand_cnt,
                                               int32_t* __restrict__ sums, PairScratch ps) {
    const int64_t row = (int64_t)blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32;
    const int lane = threadIdx.x & 31;
    if (row >= n_points) return;
    const int gi = pt_graph[row];
    const GraphInfo g = graphs[gi];
    if (!sweep_form(g.n, sums[gi])) return;
    const int i = (int)(row - g.pt_off);
    const float* P = pts + 3 * g.pt_off;
    const float pi[3] = {P[3 * i], P[3 * i + 1], P[3 * i + 2]};
    const float lo = g.r2 * (1.f - 7.62939453125e-06f), hi = g.r2 * (1.f + 7.62939453125e-06f);
    int cnt = 0;
    uint16_t* out = ps.lower + row * kCandCap;
    uint32_t cap_th = kNoLimit;  // the max_connect-th partner (from 0)
    for (int j0 = 0; j0 < i; j0 += 32) {
        const int j = j0 + lane;
        bool close = false;
        if (j < i) {
            const float pj[3] = {P[3 * j], P[3 * j + 1], P[3 * j + 2]};
            close = pair_close(pi, pj, g.r2, lo, hi);
        }
        const unsigned m = __ballot_sync(0xffffffffu, close);
        const int pos = cnt + __popc(m & ((1u << lane) - 1u));
        if (close && pos < kCandCap) out[pos] = (uint16_t)j;
        const unsigned at = __ballot_sync(0xffffffffu, close && pos == max_connect);
        if (at) cap_th = (uint32_t)(j0 + __ffs(at) - 1);
        cnt += __popc(m);
    }
    if (lane == 0) {
        ps.lower_cnt[row] = cnt;
        if (cnt > kCandCap) ps.left[gi] = 1 << 30;  // row by row after all
        if (cap_th == kNoLimit && max_connect - cnt < cand_cnt[row])
            cap_th = cand[row * kCandCap + max(max_connect - cnt, 0)];
        st_limit(ps.limits + row, cap_th | (kNoLimit << 16));
    }
}

// One point in a warp's registers: partner (list w / kListWords, place 32 (w %
// kListWords) + lane) is u[w], undecided and connected in bit w of und and con.
struct PairPoint {
    uint32_t u[kWords];
    uint32_t und, con, limit;
    unsigned used;  // bit w: some lane has a partner there
};

__device__ __forceinline__ void pair_load(PairPoint& x, const uint16_t* lower, int n_lower, const uint16_t* upper,
                                          int n_upper, int lane) {
    x.und = x.con = 0u;
    x.used = 0u;
#pragma unroll
    for (int w = 0; w < kWords; ++w) {
        const int k = 32 * (w % kListWords), n = w < kListWords ? n_lower : n_upper;
        const bool on = k + lane < n;
        x.u[w] = on ? (w < kListWords ? lower : upper)[k + lane] : 0u;
        x.und |= (on ? 1u : 0u) << w;
        x.used |= (k < n ? 1u : 0u) << w;
    }
}

// The limit of a point from its state: below in the low half, above in the
// high half.
__device__ __forceinline__ uint32_t pair_limit(const PairPoint& x, int max_connect, uint32_t lt) {
    uint32_t below = kNoLimit, above = kNoLimit;
    int n_au = 0, n_a = 0;
#pragma unroll
    for (int w = 0; w < kWords; ++w) {
        if (!((x.used >> w) & 1u)) continue;
        const bool a = (x.con >> w) & 1u, au = a || ((x.und >> w) & 1u);
        const unsigned ma = __ballot_sync(0xffffffffu, a), mau = __ballot_sync(0xffffffffu, au);
        const unsigned mb = __ballot_sync(0xffffffffu, au && n_au + __popc(mau & lt) == max_connect);
        const unsigned mt = __ballot_sync(0xffffffffu, a && n_a + __popc(ma & lt) == max_connect - 1);
        if (mb) below = __shfl_sync(0xffffffffu, x.u[w], __ffs(mb) - 1);
        if (mt) above = __shfl_sync(0xffffffffu, x.u[w], __ffs(mt) - 1);
        n_au += __popc(mau);
        n_a += __popc(ma);
    }
    return below | (above << 16);
}

// Decides what the partners' limits allow; returns whether anything changed
// (the new limit then published). Only the pairs that this point would
// connect now are asked for, at most max_connect of them: the rest can wait
// until they are among those, or past the point's own limit.
__device__ __forceinline__ bool pair_decide(PairPoint& x, int v, int max_connect, uint32_t lt, uint32_t* limits) {
    uint32_t l[kWords];
#pragma unroll
    for (int w = 0; w < kWords; ++w)
        l[w] = ((x.und >> w) & 1u) && x.u[w] < (x.limit & 0xFFFFu) ? ld_limit(limits + x.u[w]) : kNoLimit << 16;
    const uint32_t was = x.und;
#pragma unroll
    for (int w = 0; w < kWords; ++w) {
        if (!((x.und >> w) & 1u)) continue;
        // (above first: a partner that has dropped the pair no longer counts
        // it in its `below`)
        if (x.u[w] > (x.limit >> 16) || (uint32_t)v > (l[w] >> 16)) {
            x.und &= ~(1u << w);
        } else if (x.u[w] < (x.limit & 0xFFFFu) && (uint32_t)v < (l[w] & 0xFFFFu)) {
            x.und &= ~(1u << w);
            x.con |= 1u << w;
        }
    }
    if (!__any_sync(0xffffffffu, was != x.und)) return false;
    const uint32_t n = pair_limit(x, max_connect, lt);
    if (n != x.limit) {
        x.limit = n;
        if ((threadIdx.x & 31) == 0) st_limit(limits + v, n);
    }
    return true;
}

// A point's state in memory: the words of its connected partners, those of its
// undecided ones, and the number of connected partners past it.
__device__ __forceinline__ void pair_store(const PairPoint& x, uint32_t* st, int lane) {
    int later = 0;
#pragma unroll
    for (int w = 0; w < kWords; ++w) {
        const unsigned a = __ballot_sync(0xffffffffu, (x.con >> w) & 1u), u = __ballot_sync(0xffffffffu, (x.und >> w) & 1u);
        if (lane == w) st[w] = a;
        if (lane == kWords + w) st[kWords + w] = u;
        if (w >= kListWords) later += __popc(a);
    }
    if (lane == 2 * kWords) st[2 * kWords] = (uint32_t)later;
}

__global__ void __launch_bounds__(256) k_pair_sweep(const GraphInfo* __restrict__ graphs,
                                                    const int32_t* __restrict__ pt_graph, int64_t n_points,
                                                    const uint16_t* __restrict__ cand, const int32_t* __restrict__ cand_cnt,
                                                    int max_connect, const int32_t* __restrict__ sums, PairScratch ps) {
    const int64_t row = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (row >= n_points) return;
    const int gi = pt_graph[row];
    const GraphInfo g = graphs[gi];
    if (!sweep_form(g.n, sums[gi]) || ps.left[gi] >= (1 << 30)) return;
    const int v = (int)(row - g.pt_off);
    const uint32_t lt = (1u << lane) - 1u;
    uint32_t* limits = ps.limits + g.pt_off;
    PairPoint x;
    pair_load(x, ps.lower + row * kCandCap, ps.lower_cnt[row], cand + row * kCandCap, cand_cnt[row], lane);
    x.limit = ld_limit(limits + v);
    for (int idle = 0; idle < kStalled && __any_sync(0xffffffffu, x.und != 0u);)
        idle = pair_decide(x, v, max_connect, lt, limits) ? 0 : idle + 1;
    pair_store(x, ps.states + row * kPairStateWords, lane);
    if (__any_sync(0xffffffffu, x.und != 0u) && lane == 0) atomicAdd(ps.left + gi, 1);
}

constexpr int kFinishThreads = 1024;
static_assert(2 * kWords + 1 <= kPairStateWords && 2 * kWords < 32, "a state is written by one warp");

// One CTA per graph: passes over the points that the sweeps left undecided, if
// any, then the edges (i, j), i < j, in order. A graph whose lists overflow is
// left to k_greedy (sums[graph] says so). So is one in which a pass decides
// nothing, which complete lists rule out: there are no more passes than pairs,
// whatever the lists hold.
__global__ void __launch_bounds__(kFinishThreads) k_pair_finish(const GraphInfo* __restrict__ graphs,
                                                                const uint16_t* __restrict__ cand,
                                                                const int32_t* __restrict__ cand_cnt, int max_connect,
                                                                int32_t* __restrict__ sums, PairScratch ps,
                                                                int2* __restrict__ edges, int32_t* __restrict__ edge_cnt) {
    __shared__ int warp_sum[32];
    const GraphInfo g = graphs[blockIdx.x];
    const int n = g.n, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int32_t left = ps.left[blockIdx.x];
    if (!sweep_form(n, sums[blockIdx.x])) return;
    if (left >= (1 << 30)) {
        __syncthreads();
        if (threadIdx.x == 0) sums[blockIdx.x] = kListsOverflow;
        return;
    }
    uint32_t* states = ps.states + g.pt_off * kPairStateWords;
    if (left) {
        const uint32_t lt = (1u << lane) - 1u;
        for (;;) {
            bool open = false, decided = false;
            for (int v = warp; v < n; v += kFinishThreads / 32) {
                uint32_t* st = states + (size_t)v * kPairStateWords;
                if (!__any_sync(0xffffffffu, lane < kWords && st[kWords + lane] != 0u)) continue;
                const int64_t row = g.pt_off + v;
                PairPoint x;
                pair_load(x, ps.lower + row * kCandCap, ps.lower_cnt[row], cand + row * kCandCap, cand_cnt[row], lane);
                x.und = 0u;
#pragma unroll
                for (int w = 0; w < kWords; ++w) {
                    x.con |= ((st[w] >> lane) & 1u) << w;
                    x.und |= ((st[kWords + w] >> lane) & 1u) << w;
                }
                x.limit = ld_limit(ps.limits + row);
                __syncwarp();
                if (pair_decide(x, v, max_connect, lt, ps.limits + g.pt_off)) {
                    pair_store(x, st, lane);
                    decided = true;
                }
                open |= __any_sync(0xffffffffu, x.und != 0u);
            }
            if (!__syncthreads_or(open)) break;
            if (!__syncthreads_or(decided)) {
                if (threadIdx.x == 0) sums[blockIdx.x] = kListsOverflow;
                return;
            }
        }
    }
    int2* E = edges + g.e_off;
    int base = 0;
    for (int r0 = 0; r0 < n; r0 += kFinishThreads) {
        const int v = r0 + threadIdx.x;
        const uint32_t* st = states + (size_t)v * kPairStateWords;
        const int mine = v < n ? (int)st[2 * kWords] : 0;
        int at = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, at, o);
            if (lane >= o) at += y;
        }
        __syncthreads();  // the last round's sums have been read
        if (lane == 31) warp_sum[warp] = at;
        __syncthreads();
        int all = 0;
        for (int k = 0; k < 32; ++k) {
            if (k < warp) at += warp_sum[k];
            all += warp_sum[k];
        }
        at += base - mine;
        base += all;
        if (mine > 0) {
            const uint16_t* row = cand + (g.pt_off + v) * kCandCap;
#pragma unroll
            for (int w = 0; w < kListWords; ++w)
                for (uint32_t m = st[kListWords + w]; m; m &= m - 1u)
                    E[at++] = make_int2(v, row[32 * w + __ffs(m) - 1]);
        }
    }
    if (threadIdx.x == 0) edge_cnt[blockIdx.x] = base;
}

__global__ void k_adjacency(const GraphInfo* __restrict__ graphs, const int2* __restrict__ edges,
                            const int32_t* __restrict__ edge_cnt, uint8_t* __restrict__ adj,
                            const int64_t* __restrict__ adj_off) {
    const GraphInfo g = graphs[blockIdx.y];
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= edge_cnt[blockIdx.y]) return;
    const int2 ij = edges[g.e_off + e];
    uint8_t* A = adj + adj_off[blockIdx.y];
    A[(int64_t)ij.x * g.n + ij.y] = 1;
    A[(int64_t)ij.y * g.n + ij.x] = 1;
}

__global__ void k_fill(float* p, int64_t n, float v) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t k = i; k < n; k += stride) p[k] = v;
}

cudaError_t raise_smem_limit(const void* func) {
    // the limit belongs to the current device's context: one entry per
    // (device, kernel)
    static std::mutex mu;
    static std::vector<std::pair<int, const void*>> done;
    int dev = 0, optin = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> lk(mu);
    if (std::find(done.begin(), done.end(), std::make_pair(dev, func)) != done.end()) return cudaSuccess;
    e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    cudaFuncAttributes fa{};
    if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, func);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(func, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - (int)fa.sharedSizeBytes);
    if (e == cudaSuccess) done.push_back(std::make_pair(dev, func));
    return e;
}

size_t pair_scratch_bytes(int64_t n_points, int n_graphs) {
    return (size_t)n_points * (sizeof(uint16_t) * kCandCap + sizeof(int32_t) * (2 + kPairStateWords)) +
           2 * sizeof(int32_t) * (size_t)n_graphs;
}

PairScratch pair_scratch(void* p, int64_t n_points) {
    PairScratch ps;
    ps.lower = reinterpret_cast<uint16_t*>(p);  // kCandCap places are 48 words
    ps.lower_cnt = reinterpret_cast<int32_t*>(ps.lower + n_points * kCandCap);
    ps.limits = reinterpret_cast<uint32_t*>(ps.lower_cnt + n_points);
    ps.states = ps.limits + n_points;
    ps.left = reinterpret_cast<int32_t*>(ps.states + n_points * kPairStateWords);
    return ps;
}

// Sweeps want all points' warps on the GPU at once (4 CTAs of 8 an SM), and
// pay from some hundred points on; many graphs side by side are as fast row by
// row (48 of 750 points: 0.16 ms either way).
bool edge_sweeps(int max_n, int64_t n_points, int max_connect, int sms) {
    return max_connect > 0 && max_n >= 512 && n_points <= 32 * (int64_t)sms;
}

cudaError_t launch_edges(const float* pts, const GraphInfo* graphs, const int32_t* pt_graph, int n_graphs, int max_n,
                         int64_t n_points, int max_connect, uint16_t* cand, int32_t* cand_cnt, const PairScratch& ps,
                         int2* edges, int32_t* edge_cnt, int sms, cudaStream_t st) {
    if (n_graphs == 0) return cudaSuccess;
    cudaError_t e = raise_smem_limit(reinterpret_cast<const void*>(k_greedy));
    if (e != cudaSuccess) return e;
    const bool sweeps = edge_sweeps(max_n, n_points, max_connect, sms);
    int32_t* sums = nullptr;
    if (sweeps) {
        sums = ps.left + n_graphs;
        if ((e = cudaMemsetAsync(ps.left, 0, 2 * sizeof(int32_t) * n_graphs, st)) != cudaSuccess) return e;
    }
    const unsigned blocks = (unsigned)((n_points + 7) / 8);
    if (n_points > 0) {
        k_candidates<<<blocks, 256, 0, st>>>(pts, graphs, pt_graph, n_points, cand, cand_cnt, sums);
        ++g_launch_counter;
    }
    if (sweeps) {
        k_lower<<<blocks, 256, 0, st>>>(pts, graphs, pt_graph, n_points, max_connect, cand, cand_cnt, sums, ps);
        k_pair_sweep<<<blocks, 256, 0, st>>>(graphs, pt_graph, n_points, cand, cand_cnt, max_connect, sums, ps);
        k_pair_finish<<<n_graphs, kFinishThreads, 0, st>>>(graphs, cand, cand_cnt, max_connect, sums, ps, edges, edge_cnt);
        g_launch_counter += 3;
    }
    const size_t smem = 2 * kGreedyChunk * kCandCap * sizeof(uint16_t) + 2 * kGreedyChunk * sizeof(int32_t) +
                        (size_t)max_n;
    k_greedy<<<n_graphs, 256, smem, st>>>(pts, graphs, cand, cand_cnt, max_connect, edges, edge_cnt, sums);
    ++g_launch_counter;
    return cudaGetLastError();
}

cudaError_t launch_adjacency(const GraphInfo* graphs, int n_graphs, int max_edges,
                             const int2* edges, const int32_t* edge_cnt, uint8_t* adj,
                             const int64_t* adj_off, cudaStream_t st) {
    if (n_graphs == 0 || max_edges == 0) return cudaSuccess;
    dim3 grid((max_edges + 127) / 128, n_graphs);
    k_adjacency<<<grid, 128, 0, st>>>(graphs, edges, edge_cnt, adj, adj_off);
    ++g_launch_counter;
    return cudaGetLastError();
}

cudaError_t launch_fill(float* p, int64_t n, float v, cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    int64_t blocks = (n + 255) / 256;
    if (blocks > 152 * 16) blocks = 152 * 16;
    k_fill<<<(unsigned)blocks, 256, 0, st>>>(p, n, v);
    ++g_launch_counter;
    return cudaGetLastError();
}

}  // namespace lg
