// All-pairs shortest paths of LightGraph's own graphs (LightGraph::floydAlgo,
// src/LightGraph.h:512-542), from their edges instead of the dense matrix.
//
// A LightGraph has at most max_connect edges a vertex, so a solve from the
// edges does far fewer sums than Floyd-Warshall's n^3: a vertex is relaxed
// over its ~11 edges some 10 to 15 times per source. One CTA takes K sources
// that lie close together (vertices are numbered along a Morton curve first)
// and keeps their distances to every vertex in shared memory, K consecutive
// words a vertex. In passes:
//   1. vertices whose distances fell, and lie below a bound that grows with
//      the passes, mark their neighbours;
//   2. the marked vertices become a list;
//   3. each takes the minimum over its edges of the neighbour's distances plus
//      the edge, a lane for four sources.
// Updates are in place and in no set order; the distances they end at are the
// same in any, since a distance only ever falls and its least is the least
// over all paths.
//
// The passes add in FP32, rounded up: a distance never falls short of the one it
// came from, so the edges by which the distances came form trees (an edge of
// depth 0 counts as the least number above it). What each edge of a path was
// rounded by, an exact difference, is then summed down the trees in 64-bit
// integers, and the sum of distance and correction is rounded to FP32 once. What
// is left of the rounding is in the choice between paths that nearly tie, by
// less than Floyd-Warshall's own sums as long as a graph's depths lie within a
// factor of 2^20 of one another (Ctx::depths_near). Against FP64, 4096 random points,
// density uniform / over a range of 10^4: root mean square 2.5e-8 / 2.6e-8, largest
// 6.0e-8 / 2.2e-7; Floyd-Warshall 4.4e-8 / 4.7e-8 and 2.3e-7 / 2.5e-7. The same in
// thin volumes as in thick ones, and finite wherever there is a path. Of paths of
// the same rounded length the one through the lowest place is taken.
//
// LightGraph's edges are symmetric and non-negative, and few; dense or
// directed matrices are solved by k_fw.cu.
//
// Bound by shared-memory loads, 16 bytes for four sums in rows of 4 K bytes that
// meet in the same banks 1.5 (K = 16) to ~2.6 times (K = 4), and by the barriers
// of the passes where a graph is small; summing the corrections takes a
// fifth of the time. March, preparation and mirror included, against march, fill
// and the symmetric Floyd-Warshall: 200 points 0.072 against 0.130 ms, 1024 points
// 0.17 against 0.39 ms, 2500 points 0.71 against 0.99 ms, 4096 points 1.70 against
// 2.55 ms, 8900 points 9.6 against 24.4 ms, 24 graphs of 2500 points 10.9 against
// 15.2 ms. (Distances as integers of one unit of optical depth for all graphs, with
// corrections of 18 bits: 4096 points 1.65 ms, 24 of 2500 10.3 ms; but the unit was
// coarser than FP32 in thin volumes, where paths were off by up to 1%.)
#include <algorithm>

#include "lg_kernels.h"

namespace lg {

namespace {

constexpr int kPrepThreads = 1024;
constexpr int kCells = 4096;           // Morton cells of the vertex order, 16 a side

// Bits 0..3 of v at every third bit.
__device__ __forceinline__ uint32_t spread_bits4(uint32_t v) {
    v = (v | (v << 4)) & 0x0C3u;
    return (v | (v << 2)) & 0x249u;
}

constexpr uint32_t kFar = 0x7F800000u;  // the bits of inf: no path

// A word per vertex and source: the place that the vertex's path leads through,
// and the correction from there.
constexpr int kSumBits = 50;
constexpr unsigned long long kSumMask = (1ull << kSumBits) - 1;
__device__ __forceinline__ unsigned long long path_word(uint32_t place, long long sum) {
    return ((unsigned long long)place << kSumBits) | ((unsigned long long)sum & kSumMask);
}

// One CTA per graph: numbers the vertices along a Morton curve over their
// bounding box (perm: place -> vertex, rank: vertex -> place; by vertex inside
// a cell) and lays the edges out in pairs, edge pair p of place v at
// ell[p * n + v] as {neighbour's place, depth, neighbour's place, depth};
// unused halves repeat the first edge. The depth is the bits of a float, the
// least one for an edge of depth 0. step: a fifth of the mean depth. The order
// of a vertex's edges is left to chance and does not reach the distances.
__global__ void __launch_bounds__(kPrepThreads) k_path_prep(const float* __restrict__ pts,
                                                            const GraphInfo* __restrict__ graphs,
                                                            const int2* __restrict__ edges,
                                                            const int32_t* __restrict__ edge_cnt,
                                                            const float* __restrict__ W, int stride,
                                                            uint16_t* __restrict__ perm, uint16_t* __restrict__ rank,
                                                            int4* __restrict__ ell, float* __restrict__ step) {
    extern __shared__ __align__(16) int prep_shared[];  // cell offsets, then a degree, a place and a cell member per vertex
    __shared__ float red[6][32];
    __shared__ int warp_sum[32];
    __shared__ float total;
    __shared__ int finite;
    const GraphInfo g = graphs[blockIdx.x];
    const int n = g.n, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (n == 0) return;
    int* cell = prep_shared;
    int* deg = cell + kCells;
    uint16_t* place = reinterpret_cast<uint16_t*>(deg + n);
    uint16_t* member = place + n;
    const float* P = pts + 3 * g.pt_off;
    float lo[3] = {kInf, kInf, kInf}, hi[3] = {-kInf, -kInf, -kInf};
    for (int i = tid; i < n; i += kPrepThreads) {
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            lo[a] = fminf(lo[a], P[3 * i + a]);
            hi[a] = fmaxf(hi[a], P[3 * i + a]);
        }
        deg[i] = 0;
    }
    for (int i = tid; i < kCells; i += kPrepThreads) cell[i] = 0;
    if (tid == 0) {
        total = 0.f;
        finite = 0;
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            lo[a] = fminf(lo[a], __shfl_xor_sync(0xffffffffu, lo[a], o));
            hi[a] = fmaxf(hi[a], __shfl_xor_sync(0xffffffffu, hi[a], o));
        }
        if (lane == 0) {
            red[a][warp] = lo[a];
            red[3 + a][warp] = hi[a];
        }
    }
    __syncthreads();
    float ext = 0.f;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        for (int k = 0; k < 32; ++k) {
            lo[a] = fminf(lo[a], red[a][k]);
            hi[a] = fmaxf(hi[a], red[3 + a][k]);
        }
        ext = fmaxf(ext, hi[a] - lo[a]);
    }
    const float scale = ext > 0.f ? 16.f / ext : 0.f;
    auto cell_of = [&](int i) {
        uint32_t c = 0;
#pragma unroll
        for (int a = 0; a < 3; ++a) c |= spread_bits4((uint32_t)min(max((int)((P[3 * i + a] - lo[a]) * scale), 0), 15)) << a;
        return c;
    };
    for (int i = tid; i < n; i += kPrepThreads) atomicAdd(cell + cell_of(i), 1);
    __syncthreads();
    // exclusive scan of the cells, four a thread
    int4 c4 = reinterpret_cast<int4*>(cell)[tid];
    const int mine = c4.x + c4.y + c4.z + c4.w;
    int at = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, at, o);
        if (lane >= o) at += y;
    }
    if (lane == 31) warp_sum[warp] = at;
    __syncthreads();
    for (int k = 0; k < warp; ++k) at += warp_sum[k];
    at -= mine;
    reinterpret_cast<int4*>(cell)[tid] = make_int4(at, at + c4.x, at + c4.x + c4.y, at + c4.x + c4.y + c4.z);
    __syncthreads();
    for (int i = tid; i < n; i += kPrepThreads) member[atomicAdd(cell + cell_of(i), 1)] = (uint16_t)i;
    __syncthreads();
    for (int i = tid; i < n; i += kPrepThreads) {
        const int c = cell_of(i);  // cell[] holds the cells' ends by now
        const int begin = c > 0 ? cell[c - 1] : 0, end = cell[c];
        int k = begin;
        for (int m = begin; m < end; ++m) k += member[m] < i;
        place[i] = (uint16_t)k;
        perm[g.pt_off + k] = (uint16_t)i;
        rank[g.pt_off + i] = (uint16_t)k;
    }
    __syncthreads();
    int2* row = reinterpret_cast<int2*>(ell) + g.pt_off * stride;
    const int ne = edge_cnt[blockIdx.x];
    float sum = 0.f;
    int cnt = 0;
    for (int e0 = tid; e0 < ne; e0 += 4 * kPrepThreads) {
        float ws[4];
        int2 es[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {  // loads of four edges in flight
            const int e = e0 + k * kPrepThreads;
            ws[k] = e < ne ? W[g.e_off + e] : kInf;
            es[k] = e < ne ? edges[g.e_off + e] : make_int2(0, 0);
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (!(ws[k] < kInf)) continue;  // dropped
            const int d = max(__float_as_int(ws[k]), 1);
            const int a = place[es[k].x], b = place[es[k].y];
            const int ka = atomicAdd(deg + a, 1), kb = atomicAdd(deg + b, 1);
            row[((int64_t)(ka >> 1) * n + a) * 2 + (ka & 1)] = make_int2(b, d);
            row[((int64_t)(kb >> 1) * n + b) * 2 + (kb & 1)] = make_int2(a, d);
            sum += ws[k];
            ++cnt;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    cnt = __reduce_add_sync(0xffffffffu, cnt);
    if (lane == 0 && cnt > 0) {
        atomicAdd(&total, sum);
        atomicAdd(&finite, cnt);
    }
    __syncthreads();
    for (int i = tid; i < n; i += kPrepThreads) {
        const int2 any = deg[i] > 0 ? row[(int64_t)i * 2] : make_int2(i, 1);
        for (int k = deg[i]; k < stride; ++k) row[((int64_t)(k >> 1) * n + i) * 2 + (k & 1)] = any;
    }
    // (the sum's last bits, and so the passes, are left to chance too)
    if (tid == 0) step[blockIdx.x] = finite > 0 ? total / (5.f * (float)finite) : 0.f;
}

// Shared memory of a k_paths CTA for n vertices: the distances, then pending
// values, marks and two lists (9 bytes a vertex), or in their place four bits a
// distance and a word per vertex.
__host__ __device__ constexpr size_t path_smem(int n, int K) {
    const size_t n16 = ((size_t)n + 15) / 16 * 16;
    return (size_t)n * 4 * K + n16 * (K / 2 + 8);
}

// Distances are the bits of floats from 0 to inf, which compare as integers.
__device__ __forceinline__ uint32_t add_up(uint32_t x, int w) {
    return __float_as_uint(__fadd_ru(__uint_as_float(x), __int_as_float(w)));
}

// Room for the warp's c values each in a list of *count: where the lane's begin.
__device__ __forceinline__ int claim(int* count, int c, int lane) {
    int at = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, at, o);
        if (lane >= o) at += y;
    }
    int base = 0;
    if (lane == 31) base = atomicAdd(count, at);
    return at + __shfl_sync(0xffffffffu, base, 31) - c;
}

// Four sources' distances of place v, column q, over its edges in kPairs
// pairs (all loaded up front; 0: `half` pairs, three at a time).
template <int Q, int kPairs>
__device__ __forceinline__ uint4 relax(const uint4* d, const int4* __restrict__ edge, int n, int half, int v, int q,
                                       uint4 m) {
    auto pair = [&](int4 r) {
        const uint4 x = d[r.x * Q + q], y = d[r.z * Q + q];
        m.x = __vimin3_u32(m.x, add_up(x.x, r.y), add_up(y.x, r.w));
        m.y = __vimin3_u32(m.y, add_up(x.y, r.y), add_up(y.y, r.w));
        m.z = __vimin3_u32(m.z, add_up(x.z, r.y), add_up(y.z, r.w));
        m.w = __vimin3_u32(m.w, add_up(x.w, r.y), add_up(y.w, r.w));
    };
    if constexpr (kPairs > 0) {
        int4 r[kPairs];
#pragma unroll
        for (int k = 0; k < kPairs; ++k) r[k] = __ldg(edge + (int64_t)k * n + v);
#pragma unroll
        for (int k = 0; k < kPairs; ++k) pair(r[k]);
    } else {
#pragma unroll 3
        for (int k = 0; k < half; ++k) pair(__ldg(edge + (int64_t)k * n + v));
    }
    return m;
}

// Group blockIdx.x of K = 4 Q sources of graph blockIdx.y, if that graph has
// more than n_min and at most n_max vertices; half: edge pairs a vertex (kPairs
// of them unless that is 0).
template <int Q, int kPairs>
__global__ void __launch_bounds__(1024) k_paths(const GraphInfo* __restrict__ graphs, const uint16_t* __restrict__ perm,
                                                const uint16_t* __restrict__ rank, const int4* __restrict__ ell,
                                                const float* __restrict__ steps, int half, int n_min, int n_max,
                                                float* __restrict__ S) {
    constexpr int K = 4 * Q;
    extern __shared__ __align__(16) uint8_t path_shared[];
    __shared__ int count[2], going[2];
    __shared__ uint32_t low[2], top;
    const GraphInfo g = graphs[blockIdx.y];
    const int n = g.n, tid = threadIdx.x, nt = blockDim.x, lane = tid & 31;
    const int s0 = blockIdx.x * K;
    if (s0 >= n || n <= n_min || n > n_max) return;
    constexpr uint32_t far = kFar;
    const int n16 = (n + 15) / 16;
    uint4* d = reinterpret_cast<uint4*>(path_shared);
    uint32_t* pending = reinterpret_cast<uint32_t*>(d + (size_t)Q * n);  // least distance not passed on yet
    uint8_t* mark = reinterpret_cast<uint8_t*>(pending + 16 * n16);
    uint16_t* list = reinterpret_cast<uint16_t*>(mark + 16 * n16);
    uint16_t* go = list + 16 * n16;
    const int4* edge = ell + g.pt_off * half;
    const int ns = min(K, n - s0);
    const float step = steps[blockIdx.y];
    for (int i = tid; i < Q * n; i += nt) d[i] = make_uint4(far, far, far, far);
    for (int i = tid; i < 16 * n16; i += nt) pending[i] = i >= s0 && i < s0 + ns ? 0u : far;
    for (int i = tid; i < n16; i += nt) reinterpret_cast<uint4*>(mark)[i] = make_uint4(0, 0, 0, 0);
    if (tid < 2) {
        count[tid] = 0;
        going[tid] = 0;
        low[tid] = far;
        top = 0u;
    }
    __syncthreads();
    if (tid < ns) reinterpret_cast<uint32_t*>(d)[(s0 + tid) * K + tid] = 0u;
    uint32_t bound = min(__float_as_uint(step), far - 1u);
    const bool small = n <= 4 * nt;
    for (int par = 0;; par ^= 1) {
        // 1. the vertices whose distances fell to the bound or below, and the
        // least of the others'
        uint32_t least = far;
        for (int i0 = 0; i0 < 4 * n16; i0 += nt) {
            const int i = i0 + tid;
            uint4 p = make_uint4(far, far, far, far);
            if (i < 4 * n16) p = reinterpret_cast<const uint4*>(pending)[i];
            const uint32_t ps[4] = {p.x, p.y, p.z, p.w};
            int c = 0;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                c += ps[k] <= bound;
                least = min(least, ps[k] <= bound ? far : ps[k]);
            }
            if (!__any_sync(0xffffffffu, c > 0)) continue;
            int at = claim(&going[par], c, lane);
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (ps[k] <= bound) {
                    pending[4 * i + k] = far;
                    go[at++] = (uint16_t)(4 * i + k);
                }
        }
        least = __reduce_min_sync(0xffffffffu, least);
        if (lane == 0 && least < far) atomicMin(&low[par], least);
        __syncthreads();
        // 2. their neighbours are marked,
        const int marks = going[par];
        for (int i = tid; i < marks; i += nt) {
            const int u = go[i];
            auto set = [&](int4 r) {
                mark[r.x] = 1;
                mark[r.z] = 1;
            };
            if constexpr (kPairs > 0) {
                int4 r[kPairs];
#pragma unroll
                for (int k = 0; k < kPairs; ++k) r[k] = __ldg(edge + (int64_t)k * n + u);
#pragma unroll
                for (int k = 0; k < kPairs; ++k) set(r[k]);
            } else {
#pragma unroll 3
                for (int k = 0; k < half; ++k) set(__ldg(edge + (int64_t)k * n + u));
            }
        }
        __syncthreads();
        // and the marked vertices become a list, four marks a thread
        for (int i0 = 0; marks > 0 && i0 < 4 * n16; i0 += nt) {
            const int i = i0 + tid;
            uint32_t w = 0;
            if (i < 4 * n16) {
                w = reinterpret_cast<const uint32_t*>(mark)[i];
                if (w) reinterpret_cast<uint32_t*>(mark)[i] = 0;
            }
            if (!__any_sync(0xffffffffu, w != 0)) continue;
            int at = claim(&count[par], __popc(w), lane);
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (w & (1u << (8 * k))) list[at++] = (uint16_t)(4 * i + k);
        }
        __syncthreads();
        const int items = count[par] * Q;
        const uint32_t waiting = low[par];
        if (items == 0 && waiting == far) break;
        if (tid == 0) {
            count[par ^ 1] = 0;
            going[par ^ 1] = 0;
            low[par ^ 1] = far;
        }
        // 3. the list's distances
        for (int i = tid; i < items; i += nt) {
            const int v = list[i / Q], q = i % Q;
            const uint4 a = d[v * Q + q];
            const uint4 m = relax<Q, kPairs>(d, edge, n, half, v, q, a);
            const uint32_t f = min(min(m.x < a.x ? m.x : far, m.y < a.y ? m.y : far),
                                   min(m.z < a.z ? m.z : far, m.w < a.w ? m.w : far));
            if (f < far) {
                d[v * Q + q] = m;
                atomicMin(pending + v, f);
            }
        }
        // In a small graph the bound grows faster where a pass leaves threads idle
        // (200 points: 0.070 -> 0.055 ms, of them chains of few neighbours 0.19 ->
        // 0.07 ms; 4096 points: 2.23 -> 2.36 ms, so not in a large one). It stays
        // below far, the mark of vertices with nothing pending.
        const float by = small && items > 0 ? (float)min(max(nt / items, 1), 4) : 1.f;
        bound = items == 0 ? waiting : min(__float_as_uint(fmaf(by, step, __uint_as_float(bound))), far - 1u);
        __syncthreads();
    }
    // The edge by which each distance came: of those that give it, the one to
    // the lowest place. Four bits each; d tells where there is none.
    uint16_t* by = reinterpret_cast<uint16_t*>(d + (size_t)Q * n);
    uint32_t most = 0;
    for (int i = tid; i < Q * n; i += nt) {
        const int v = i / Q, q = i % Q;
        const uint4 m = d[i];
        uint32_t best[4] = {~0u, ~0u, ~0u, ~0u};  // place, edge
        auto tie = [&](uint32_t u, int w, uint32_t slot) {
            const uint4 x = d[u * Q + q];
            const uint32_t key = (u << 4) | slot;
            if (add_up(x.x, w) == m.x) best[0] = min(best[0], key);
            if (add_up(x.y, w) == m.y) best[1] = min(best[1], key);
            if (add_up(x.z, w) == m.z) best[2] = min(best[2], key);
            if (add_up(x.w, w) == m.w) best[3] = min(best[3], key);
        };
#pragma unroll 3
        for (int k = 0; k < half; ++k) {
            const int4 r = __ldg(edge + (int64_t)k * n + v);
            tie(r.x, r.y, 2 * k);
            tie(r.z, r.w, 2 * k + 1);
        }
        by[i] = (uint16_t)((best[0] & 15u) | ((best[1] & 15u) << 4) | ((best[2] & 15u) << 8) | ((best[3] & 15u) << 12));
        const uint32_t ms[4] = {m.x, m.y, m.z, m.w};
#pragma unroll
        for (int c = 0; c < 4; ++c) most = max(most, ms[c] < far ? ms[c] : 0u);
    }
    most = __reduce_max_sync(0xffffffffu, most);
    if (lane == 0) atomicMax(&top, most);
    __syncthreads();
    // Source by source: each vertex's word starts as its edge's and takes over
    // the word of the place it names until that is the source. Words only move
    // towards the source and their sums are exact, so another's may be read at
    // any stage (8 bytes are read and written at once). Then the source's row of
    // the matrix, columns in vertex order; the padding is inf.
    volatile unsigned long long* word =
        reinterpret_cast<volatile unsigned long long*>(by + ((size_t)Q * n + 3) / 4 * 4);
    const uint16_t* rk = rank + g.pt_off;
    const int2* lone = reinterpret_cast<const int2*>(edge);
    const uint32_t* dist = reinterpret_cast<const uint32_t*>(d);
    // Rounding up adds less than a unit in the last place of the CTA's largest
    // distance to an edge (one such unit where the depth is 0): 2^(49 - log2 n)
    // fractions to that unit. A power of two in two factors, since it can exceed a float's.
    const int fine = 23 - ((int)(top >> 23) - 127) + kSumBits - 1 - (32 - __clz(n - 1));
    auto power = [](int e) { return __int_as_float((e + 127) << 23); };
    const int fine0 = min(fine, 100);
    const float up0 = power(fine0), up1 = power(fine - fine0), down0 = power(-fine0), down1 = power(fine0 - fine);
    float* M = S + g.s_off;
    for (int k = 0; k < ns; ++k) {
        const int root = s0 + k;
        for (int v0 = tid; v0 < n; v0 += 4 * nt) {
            unsigned long long w[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const int v = v0 + c * nt;
                w[c] = path_word(root, 0);
                if (v >= n || v == root || dist[v * K + k] >= far) continue;
                const uint32_t slot = (by[v * Q + k / 4] >> (4 * (k & 3))) & 15u;
                const int2 r = __ldg(lone + ((int64_t)(slot >> 1) * n + v) * 2 + (slot & 1u));
                // (dist[r.x] + depth) - dist[v], exact but for bits far below the fractions
                const float x = __uint_as_float(dist[r.x * K + k]), y = r.y == 1 ? 0.f : __int_as_float(r.y);
                const float s = __fadd_rn(x, y), b = __fsub_rn(s, x);
                const float err = __fadd_rn(__fsub_rn(x, __fsub_rn(s, b)), __fsub_rn(y, b));
                const float lost = __fadd_rn(err, __fsub_rn(s, __uint_as_float(dist[v * K + k])));
                w[c] = path_word((uint32_t)r.x, __float2ll_rn(lost * up0 * up1));
            }
#pragma unroll
            for (int c = 0; c < 4; ++c)
                if (v0 + c * nt < n) word[v0 + c * nt] = w[c];
        }
        __syncthreads();
        for (bool more = true; more;) {  // all of a thread's vertices a step at a time: log2(path) steps
            more = false;
            for (int v0 = tid; v0 < n; v0 += 4 * nt) {
                unsigned long long w[4], u[4];
#pragma unroll
                for (int c = 0; c < 4; ++c) w[c] = v0 + c * nt < n ? word[v0 + c * nt] : path_word(root, 0);
#pragma unroll
                for (int c = 0; c < 4; ++c) u[c] = word[w[c] >> kSumBits];
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    if ((int)(w[c] >> kSumBits) == root) continue;
                    word[v0 + c * nt] = (u[c] & ~kSumMask) | ((w[c] + u[c]) & kSumMask);
                    more |= (int)(u[c] >> kSumBits) != root;
                }
            }
        }
        __syncthreads();
        float* row = M + (int64_t)perm[g.pt_off + root] * g.ld;
        for (int j = tid; j < g.ld; j += nt) {
            float out = kInf;
            if (j < n) {
                const int v = rk[j];
                const uint32_t m = dist[v * K + k];
                const long long sum = (long long)(word[v] << (64 - kSumBits)) >> (64 - kSumBits);
                // (a path of n edges of depth 0 counts fewer than 2^14 least numbers)
                if (m < 1u << 14) out = 0.f;
                else if (m < far) out = __fadd_rn(__uint_as_float(m), __ll2float_rn(sum) * down0 * down1);
            }
            row[j] = out;
        }
        __syncthreads();
    }
    if (s0 + K >= n)  // the last group also pads the rows
        for (int64_t i = (int64_t)n * g.ld + tid; i < (int64_t)g.ld * g.ld; i += nt) M[i] = kInf;
}

// The two directions of a path may take other edges among equals and round
// otherwise: every entry below the diagonal becomes the one above it (64 x 64
// blocks through shared memory, so both sides are coalesced).
__global__ void __launch_bounds__(256) k_path_mirror(const GraphInfo* __restrict__ graphs, float* __restrict__ S) {
    __shared__ float tile[64][65];
    const GraphInfo g = graphs[blockIdx.y];
    const int nb = (g.n + 63) / 64;
    float* M = S + g.s_off;
    for (int t = blockIdx.x; t < nb * nb; t += gridDim.x) {
        const int bi = t / nb, bj = t % nb;
        if (bi > bj) continue;
        for (int e = threadIdx.x; e < 64 * 64; e += 256) tile[e >> 6][e & 63] = M[(int64_t)(bi * 64 + (e >> 6)) * g.ld + bj * 64 + (e & 63)];
        __syncthreads();
        for (int e = threadIdx.x; e < 64 * 64; e += 256) {
            const int r = bj * 64 + (e >> 6), c = bi * 64 + (e & 63);
            if (c < r && r < g.n && c < g.n) M[(int64_t)r * g.ld + c] = tile[e & 63][e >> 6];
        }
        __syncthreads();
    }
}

// The depth of every edge from its entry of the matrices.
__global__ void k_edge_depths(const GraphInfo* __restrict__ graphs, const int2* __restrict__ edges,
                              const int32_t* __restrict__ edge_cnt, const float* __restrict__ S, float* __restrict__ W) {
    const GraphInfo g = graphs[blockIdx.y];
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= edge_cnt[blockIdx.y]) return;
    const int2 ij = edges[g.e_off + e];
    W[g.e_off + e] = S[g.s_off + (int64_t)ij.x * g.ld + ij.y];
}

}  // namespace

int path_stride(int max_connect) { return std::max(2, (max_connect + 1) / 2 * 2); }

cudaError_t launch_paths(const float* pts, const GraphInfo* graphs, int n_graphs, int min_n, int max_n, int64_t n_points,
                         int max_connect, const int2* edges, const int32_t* edge_cnt, const float* W,
                         const PathScratch& ps, float* S, int sms, cudaStream_t st) {
    if (n_graphs == 0 || max_n == 0) return cudaSuccess;
    const int stride = path_stride(max_connect), half = stride / 2;
    cudaError_t e = raise_smem_limit(reinterpret_cast<const void*>(k_path_prep));
    if (e != cudaSuccess) return e;
    k_path_prep<<<n_graphs, kPrepThreads, sizeof(int) * (kCells + (size_t)max_n) + 2 * sizeof(uint16_t) * (size_t)max_n, st>>>(
        pts, graphs, edges, edge_cnt, W, stride, ps.perm, ps.rank, ps.ell, ps.step);
    ++g_launch_counter;
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    // Sources per CTA: few while that makes CTAs for idle SMs (1024 points: K =
    // 4, 8, 16 in 0.22,
    // 0.22, 0.30 ms; 2000 points: 0.64, 0.57, 0.51 ms), then many, for wide rows
    // (24 graphs of 2500 points: 12.4, 9.8, 8.4 ms), but not 16 where they just
    // miss being one wave (2500 points, 157 CTAs: 1.10, 0.95, 1.03 ms). Threads:
    // 512 where only one or two CTAs fit an SM.
    int Q = 4;
    const int64_t groups = (n_points + 15) / 16;
    if (n_points <= 11 * (int64_t)sms) Q = 1;
    else if (groups > sms && groups < 2 * (int64_t)sms) Q = 2;
    constexpr int n_max4 = 2896, n_max2 = 5280, kSmall = 1700;
    constexpr size_t most = 227 * 1024 - 64;  // less the static words
    static_assert(kPathMaxPoints <= 1 << 14, "places in the words");
    static_assert(path_smem(n_max4, 16) <= most && path_smem(n_max2, 8) <= most && path_smem(kPathMaxPoints, 4) <= most);
    auto run = [&](auto pairs6, auto pairs, int K, int n_min, int n_max) {
        n_max = std::min(n_max, max_n);
        if (e != cudaSuccess || n_max <= n_min || n_max < min_n) return;
        auto kernel = half == 6 ? pairs6 : pairs;
        if ((e = raise_smem_limit(reinterpret_cast<const void*>(kernel))) != cudaSuccess) return;
        kernel<<<dim3((n_max + K - 1) / K, n_graphs), n_max > kSmall ? 512 : 256, path_smem(n_max, K), st>>>(
            graphs, ps.perm, ps.rank, ps.ell, ps.step, half, n_min, n_max, S);
        ++g_launch_counter;
        e = cudaGetLastError();
    };
    // the largest graphs first
    run(k_paths<1, 6>, k_paths<1, 0>, 4, Q == 1 ? kSmall : n_max2, kPathMaxPoints);
    if (Q == 4) {
        run(k_paths<2, 6>, k_paths<2, 0>, 8, n_max4, n_max2);
        run(k_paths<4, 6>, k_paths<4, 0>, 16, kSmall, n_max4);
        run(k_paths<4, 6>, k_paths<4, 0>, 16, 0, kSmall);
    } else if (Q == 2) {
        run(k_paths<2, 6>, k_paths<2, 0>, 8, kSmall, n_max2);
        run(k_paths<2, 6>, k_paths<2, 0>, 8, 0, kSmall);
    } else {
        run(k_paths<1, 6>, k_paths<1, 0>, 4, 0, kSmall);
    }
    if (e != cudaSuccess) return e;
    const int nb = (max_n + 63) / 64;
    k_path_mirror<<<dim3(std::min(nb * nb, 4096), n_graphs), 256, 0, st>>>(graphs, S);
    ++g_launch_counter;
    return cudaGetLastError();
}

cudaError_t launch_edge_depths(const GraphInfo* graphs, int n_graphs, int max_edges, const int2* edges,
                               const int32_t* edge_cnt, const float* S, float* W, cudaStream_t st) {
    if (n_graphs == 0 || max_edges == 0) return cudaSuccess;
    k_edge_depths<<<dim3((max_edges + 255) / 256, n_graphs), 256, 0, st>>>(graphs, edges, edge_cnt, S, W);
    ++g_launch_counter;
    return cudaGetLastError();
}

}  // namespace lg
