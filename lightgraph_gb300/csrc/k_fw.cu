// Blocked min-plus Floyd-Warshall: LightGraph::floydAlgo (src/LightGraph.h:512-542).
//
// The reference runs a max-times FW on RGB transmittance T (FP64):
//   T_ij = maxComponent(T_ij, T_ik * T_kj), skipping zero T_ik / T_kj.
// Every channel is T_c = exp(-a_c * S) for one scalar optical depth S (see
// k_march.cu), so the per-channel max-times recurrences are all the same
// min-plus recurrence on S (zero T <-> S = +inf):
//   S_ij = min(S_ij, S_ik + S_kj).
// This file solves that recurrence in FP32 with the 3-phase blocked schedule,
// k-blocks of 64:
//   diagonal    : the 64 x 64 diagonal block is closed in shared memory
//                 (blocked FW on 16 x 16 sub-blocks, close_diag_blocked);
//   panels      : the k-block row and column panels, one min-plus product
//                 each against the closed diagonal block;
//   update tiles: every other element, S_ij = min(S_ij, min_k A_ik + B_kj),
//                 a min-plus product on the CUDA cores. Each thread owns an
//                 8x8 register tile and consumes k in pairs:
//                   s = add.rn.f32x2({A_ik, A_ik+1}, {B_kj, B_k+1,j})
//                   C_ij = min.f32(C_ij, s.x, s.y)        (3-input min)
//                 i.e. 4 FP32 ops in 2 instructions. Each op still takes an
//                 FP32 lane cycle, so min-plus tops out near half of the
//                 FMA-counted FP32 peak (k_fw_inner_loop measures it).
// It is not a dense contraction, so tensor cores do not apply.
// All values must be >= 0 (or +inf); then row and column k do not change in
// round k, which makes each round's updates independent of their order.
//
// Three drivers share the tile code:
//   fw_solve             : one matrix of any kind, two launches per round
//                          (k_fw_panels, k_fw_update);
//   fw_solve_batched     : many matrices of any kind and different sizes in
//                          ONE persistent launch (k_fw_persistent);
//   fw_solve_batched_sym : the same for symmetric matrices (LightGraph's),
//                          computing only the blocks on and above the
//                          diagonal (k_fw_persistent_sym, then k_fw_mirror).
// In the persistent launches CTAs claim work items from a queue; an item waits
// (bounded) on the version counters of the 64 x 64 blocks it reads, whose
// writers always come earlier in the queue, so the schedule cannot deadlock
// whatever the residency (fw_queue_replay checks every queue on the host).
#include <algorithm>
#include <functional>
#include <queue>
#include <vector>

#include "lg_kernels.h"

namespace lg {

constexpr int kKB = 64;      // k-block
constexpr int kTile = 128;   // update tile (rows and cols)
constexpr int kApad = 2;     // float2 padding per k-pair row of the A stage
constexpr int kPanelSlots = 3;  // column-panel slots of the symmetric solve (round r uses r % 3)

__device__ __forceinline__ float min3f(float a, float b, float c) {
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// Loads of the matrix. The persistent kernel reads data other CTAs wrote
// during the same launch, so it reads through L2 (ld.global.cg), never a
// possibly stale L1 line.
template <bool kL2>
__device__ __forceinline__ float ldm(const float* p) {
    if (kL2) return __ldcg(p);
    return *p;
}
template <bool kL2>
__device__ __forceinline__ float2 ldm2(const float* p) {
    if (kL2) return __ldcg(reinterpret_cast<const float2*>(p));
    return *reinterpret_cast<const float2*>(p);
}
template <bool kL2>
__device__ __forceinline__ float4 ldm4(const float* p) {
    if (kL2) return __ldcg(reinterpret_cast<const float4*>(p));
    return *reinterpret_cast<const float4*>(p);
}

template <bool kL2>
__device__ __forceinline__ float ld_or_inf(const float* d, int n, int ld, int i, int j) {
    return (i < n && j < n) ? ldm<kL2>(d + (int64_t)i * ld + j) : kInf;
}

constexpr int kPS = kKB + 2;  // row stride of the panel stage (even: k-pairs are 8-byte loads)

struct PanelSmem {
    float Dg[kKB][kPS];
    float T[kKB][kPS];
};

__device__ __forceinline__ int outside16(int o, int S0) { return o < S0 ? o : o + 16; }

// Closes the 64 x 64 diagonal tile D (shared memory, 256 threads) by blocked
// FW with 16 x 16 sub-blocks s = 0..3:
//   1. warp 0 closes sub-block (s, s) in registers: 16 steps, lane (i, half)
//      holds 8 elements of row i and fetches row k and column k by warp
//      shuffles (they do not change in step k because D_kk >= 0);
//   2. the sub-block's row and column panels become min(P, Dss* (x) P) and
//      min(P, P (x) Dss*) (computed from the old panels, written after a
//      barrier);
//   3. the other 48 x 48 elements take min(D, column panel (x) row panel) in
//      place (neither panel changes in this phase).
// 16 barriers in all instead of one per step. The products take k in pairs,
// one add.rn.f32x2 and one 3-input min per two k.
__device__ __forceinline__ void close_diag_blocked(float (*D)[kPS]) {
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int p = tid >> 4, q = tid & 15;
    for (int S0 = 0; S0 < kKB; S0 += 16) {
        if (warp == 0) {
            const int i = lane >> 1, j0 = (lane & 1) * 8;
            float v[8];
#pragma unroll
            for (int jj = 0; jj < 8; ++jj) v[jj] = D[S0 + i][S0 + j0 + jj];
#pragma unroll
            for (int k = 0; k < 16; ++k) {
                const float dik = __shfl_sync(0xffffffffu, v[k & 7], 2 * i + (k >> 3));
                float dkj[8];
#pragma unroll
                for (int jj = 0; jj < 8; ++jj) dkj[jj] = __shfl_sync(0xffffffffu, v[jj], 2 * k + (lane & 1));
#pragma unroll
                for (int jj = 0; jj < 8; ++jj) v[jj] = fminf(v[jj], dik + dkj[jj]);
            }
#pragma unroll
            for (int jj = 0; jj < 8; ++jj) D[S0 + i][S0 + j0 + jj] = v[jj];
        }
        __syncthreads();
        // 2. row panel elements (S0 + p, out(q + 16m)), column panel elements
        //    (out(p + 16m), S0 + q)
        float rp[3], cp[3];
#pragma unroll
        for (int m = 0; m < 3; ++m) {
            rp[m] = D[S0 + p][outside16(q + 16 * m, S0)];
            cp[m] = D[outside16(p + 16 * m, S0)][S0 + q];
        }
#pragma unroll
        for (int kp = 0; kp < 8; ++kp) {
            const int k = S0 + 2 * kp;
            const float2 dp = *reinterpret_cast<const float2*>(&D[S0 + p][k]);
            const float2 dq = make_float2(D[k][S0 + q], D[k + 1][S0 + q]);
#pragma unroll
            for (int m = 0; m < 3; ++m) {
                const int j = outside16(q + 16 * m, S0), i = outside16(p + 16 * m, S0);
                const float2 sr = __fadd2_rn(dp, make_float2(D[k][j], D[k + 1][j]));
                rp[m] = min3f(rp[m], sr.x, sr.y);
                const float2 sc = __fadd2_rn(*reinterpret_cast<const float2*>(&D[i][k]), dq);
                cp[m] = min3f(cp[m], sc.x, sc.y);
            }
        }
        __syncthreads();
#pragma unroll
        for (int m = 0; m < 3; ++m) {
            D[S0 + p][outside16(q + 16 * m, S0)] = rp[m];
            D[outside16(p + 16 * m, S0)][S0 + q] = cp[m];
        }
        __syncthreads();
        // 3. elements (out(p + 16m), out(q + 16m'))
        float acc[3][3];
#pragma unroll
        for (int m = 0; m < 3; ++m)
#pragma unroll
            for (int mm = 0; mm < 3; ++mm) acc[m][mm] = D[outside16(p + 16 * m, S0)][outside16(q + 16 * mm, S0)];
#pragma unroll
        for (int kp = 0; kp < 8; ++kp) {
            const int k = S0 + 2 * kp;
            float2 a[3], b[3];
#pragma unroll
            for (int m = 0; m < 3; ++m) {
                a[m] = *reinterpret_cast<const float2*>(&D[outside16(p + 16 * m, S0)][k]);
                const int j = outside16(q + 16 * m, S0);
                b[m] = make_float2(D[k][j], D[k + 1][j]);
            }
#pragma unroll
            for (int m = 0; m < 3; ++m)
#pragma unroll
                for (int mm = 0; mm < 3; ++mm) {
                    const float2 sm2 = __fadd2_rn(a[m], b[mm]);
                    acc[m][mm] = min3f(acc[m][mm], sm2.x, sm2.y);
                }
        }
#pragma unroll
        for (int m = 0; m < 3; ++m)
#pragma unroll
            for (int mm = 0; mm < 3; ++mm) D[outside16(p + 16 * m, S0)][outside16(q + 16 * mm, S0)] = acc[m][mm];
        __syncthreads();
    }
}

// One min-plus product of a panel tile against the closed diagonal tile Dg*
// (thread (ty, tx) owns the 4 x 4 elements (ty + 16r, tx + 16c)):
//   row panel    : acc = min(T, Dg* (x) T)
//   column panel : acc = min(T, T (x) Dg*)
// Every path that leaves the k-block for the last time at k' costs
// Dg*[k][k'] + T[k'][j], so one product replaces the 64 sequential panel
// steps. k is taken in pairs (add.rn.f32x2 + 3-input min); the minimum of the
// same sums is exact whatever the grouping.
__device__ __forceinline__ void panel_product(const PanelSmem& sm, bool row_panel, int ty, int tx,
                                              float (&acc)[4][4]) {
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[r][c] = sm.T[ty + 16 * r][tx + 16 * c];
    const float (*L)[kPS] = row_panel ? sm.Dg : sm.T;  // left factor (rows)
    const float (*R)[kPS] = row_panel ? sm.T : sm.Dg;  // right factor (columns)
#pragma unroll 4
    for (int kp = 0; kp < kKB / 2; ++kp) {
        float2 a[4], bb[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) a[r] = *reinterpret_cast<const float2*>(&L[ty + 16 * r][2 * kp]);
#pragma unroll
        for (int c = 0; c < 4; ++c) bb[c] = make_float2(R[2 * kp][tx + 16 * c], R[2 * kp + 1][tx + 16 * c]);
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const float2 sv = __fadd2_rn(a[r], bb[c]);
                acc[r][c] = min3f(acc[r][c], sv.x, sv.y);
            }
    }
}

// Panel tile b of round kb: 0 = diagonal, 1..nt-1 = row panel, nt..2nt-2 =
// column panel (the diagonal's index skipped). 256 threads, each owning the
// 4x4 elements (ty + 16r, tx + 16c) of the panel product. The diagonal tile
// is closed in shared memory (close_diag_blocked) unless closed_diag says
// it is already closed in d (the persistent schedule closes it once, in its
// own item).
template <bool kL2>
__device__ __forceinline__ void fw_panel_tile(float* __restrict__ d, int n, int ld, int nt, int kb, int b, PanelSmem& sm,
                                              bool closed_diag = false) {
    const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
    const int K0 = kb * kKB;
    int kind = 0, other = kb;  // 0 diag, 1 row tile (K0, other), 2 col tile (other, K0)
    if (b > 0) {
        int q = b - 1;
        kind = 1;
        if (q >= nt - 1) { kind = 2; q -= nt - 1; }
        other = q < kb ? q : q + 1;
    }
    const int O0 = other * kKB;
    // 16 bytes a load: 11 us a launch of k_fw_panels at n = 1021, 17.6 with 4 bytes
    const int R0 = kind == 2 ? O0 : K0, C0 = kind == 2 ? K0 : O0;  // the panel tile's corner
    if (max(K0, O0) + kKB <= n) {
        float4 dg[4], pt[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int r = (tid >> 4) + 16 * q, c = (tid & 15) * 4;
            dg[q] = ldm4<kL2>(d + (int64_t)(K0 + r) * ld + K0 + c);
            if (kind != 0) pt[q] = ldm4<kL2>(d + (int64_t)(R0 + r) * ld + C0 + c);
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int r = (tid >> 4) + 16 * q, c = (tid & 15) * 4;
            float2* to = reinterpret_cast<float2*>(&sm.Dg[r][c]);
            to[0] = make_float2(dg[q].x, dg[q].y);
            to[1] = make_float2(dg[q].z, dg[q].w);
            if (kind != 0) {
                to = reinterpret_cast<float2*>(&sm.T[r][c]);
                to[0] = make_float2(pt[q].x, pt[q].y);
                to[1] = make_float2(pt[q].z, pt[q].w);
            }
        }
    } else {
        for (int e = tid; e < kKB * kKB; e += 256) {
            const int r = e >> 6, c = e & 63;
            sm.Dg[r][c] = ld_or_inf<kL2>(d, n, ld, K0 + r, K0 + c);
            if (kind != 0) sm.T[r][c] = ld_or_inf<kL2>(d, n, ld, R0 + r, C0 + c);
        }
    }
    __syncthreads();
    if (kind == 0 || !closed_diag) close_diag_blocked(sm.Dg);
    if (kind == 0) {
        for (int e = tid; e < kKB * kKB; e += 256) {
            const int r = e >> 6, c = e & 63;
            if (K0 + r < n && K0 + c < n) d[(int64_t)(K0 + r) * ld + K0 + c] = sm.Dg[r][c];
        }
        return;
    }
    float acc[4][4];
    panel_product(sm, kind == 1, ty, tx, acc);
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int i = ty + 16 * r, j = tx + 16 * c;
            const int gi = kind == 1 ? K0 + i : O0 + i;
            const int gj = kind == 1 ? O0 + j : K0 + j;
            if (gi < n && gj < n) d[(int64_t)gi * ld + gj] = acc[r][c];
        }
}

// Update tile (ti, tj) of round kb, 128 x kCols. 256 threads = 8 warps (4 x 2),
// each warp 32 x kCols / 2, each thread 8 x kCols / 16 (rows/cols interleaved so
// the shared-memory fragment loads are conflict-free 128-bit reads).
template <bool kL2, int kCols = kTile>
__device__ __forceinline__ void fw_update_tile(float* __restrict__ d, int n, int ld, int kb, int ti, int tj,
                                               float2* __restrict__ As, float2* __restrict__ Bs) {
    constexpr int kP = kCols / 32;  // column pairs a thread
    const int I0 = ti * kTile, J0 = tj * kCols, K0 = kb * kKB;
    const int tid = threadIdx.x;
    const bool full = (I0 + kTile <= n) && (J0 + kCols <= n) && (K0 + kKB <= n);

    // stage A = S[I0:I0+128, K0:K0+64] as k-pairs: As[kp][i] = {S[i][2kp], S[i][2kp+1]}
    {
        const int i = tid & 127, h = tid >> 7;
        const int gi = I0 + i;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int kp = h * 16 + 2 * q;
            const int gk = K0 + 2 * kp;
            float4 v;
            if (full) {
                v = ldm4<kL2>(d + (int64_t)gi * ld + gk);
            } else {
                v.x = ld_or_inf<kL2>(d, n, ld, gi, gk);
                v.y = ld_or_inf<kL2>(d, n, ld, gi, gk + 1);
                v.z = ld_or_inf<kL2>(d, n, ld, gi, gk + 2);
                v.w = ld_or_inf<kL2>(d, n, ld, gi, gk + 3);
            }
            As[kp * (kTile + kApad) + i] = make_float2(v.x, v.y);
            As[(kp + 1) * (kTile + kApad) + i] = make_float2(v.z, v.w);
        }
    }
    // stage B = S[K0:K0+64, J0:J0+kCols] as k-pairs: Bs[kp][j] = {S[2kp][j], S[2kp+1][j]}
    {
        constexpr int kQ = kCols / 4;  // threads a row
        const int j4 = tid % kQ;
#pragma unroll
        for (int q = 0; q < 32 * kQ / 256; ++q) {
            const int kp = tid / kQ + 256 / kQ * q;
            const int gk = K0 + 2 * kp, gj = J0 + 4 * j4;
            float4 r0, r1;
            if (full) {
                r0 = ldm4<kL2>(d + (int64_t)gk * ld + gj);
                r1 = ldm4<kL2>(d + (int64_t)(gk + 1) * ld + gj);
            } else {
                r0.x = ld_or_inf<kL2>(d, n, ld, gk, gj); r0.y = ld_or_inf<kL2>(d, n, ld, gk, gj + 1);
                r0.z = ld_or_inf<kL2>(d, n, ld, gk, gj + 2); r0.w = ld_or_inf<kL2>(d, n, ld, gk, gj + 3);
                r1.x = ld_or_inf<kL2>(d, n, ld, gk + 1, gj); r1.y = ld_or_inf<kL2>(d, n, ld, gk + 1, gj + 1);
                r1.z = ld_or_inf<kL2>(d, n, ld, gk + 1, gj + 2); r1.w = ld_or_inf<kL2>(d, n, ld, gk + 1, gj + 3);
            }
            float4* dst = reinterpret_cast<float4*>(Bs + kp * kCols + 4 * j4);
            dst[0] = make_float4(r0.x, r1.x, r0.y, r1.y);
            dst[1] = make_float4(r0.z, r1.z, r0.w, r1.w);
        }
    }

    const int warp = tid >> 5, lane = tid & 31;
    const int wy = warp >> 1, wx = warp & 1, ty = lane >> 3, tx = lane & 7;
    const int rbase = wy * 32 + ty * 2;  // rows rbase + 8q + {0,1}
    const int cbase = wx * (kCols / 2) + tx * 2;  // cols cbase + 16p + {0,1}

    // a warp whose rows or columns are the k-block's has nothing to do
    const int wr = I0 + wy * 32, wc = J0 + wx * (kCols / 2);
    const bool own = wr < n && wc < n && (wr >> 6) != kb && (wc >> 6) != kb;
    float acc[8][2 * kP];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            const int gi = I0 + rbase + 8 * q + s;
#pragma unroll
            for (int p = 0; p < kP; ++p) {
                const int gj = J0 + cbase + 16 * p;
                float2 v;
                if (!own) {
                    v = make_float2(kInf, kInf);
                } else if (full) {
                    v = ldm2<kL2>(d + (int64_t)gi * ld + gj);
                } else {
                    v.x = ld_or_inf<kL2>(d, n, ld, gi, gj);
                    v.y = ld_or_inf<kL2>(d, n, ld, gi, gj + 1);
                }
                acc[2 * q + s][2 * p] = v.x;
                acc[2 * q + s][2 * p + 1] = v.y;
            }
        }
    }
    __syncthreads();
    if (!own) return;

#pragma unroll 1
    for (int kp = 0; kp < 32; ++kp) {
        float2 a[8], b[2 * kP];
        const float4* ap = reinterpret_cast<const float4*>(As + kp * (kTile + kApad) + rbase);
        const float4* bp = reinterpret_cast<const float4*>(Bs + kp * kCols + cbase);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const float4 va = ap[4 * q];   // rows rbase + 8q, +1
            a[2 * q] = make_float2(va.x, va.y);
            a[2 * q + 1] = make_float2(va.z, va.w);
        }
#pragma unroll
        for (int q = 0; q < kP; ++q) {
            const float4 vb = bp[8 * q];   // cols cbase + 16q, +1
            b[2 * q] = make_float2(vb.x, vb.y);
            b[2 * q + 1] = make_float2(vb.z, vb.w);
        }
#pragma unroll
        for (int r = 0; r < 8; ++r) {
#pragma unroll
            for (int c = 0; c < 2 * kP; ++c) {
                const float2 s = __fadd2_rn(a[r], b[c]);
                acc[r][c] = min3f(acc[r][c], s.x, s.y);
            }
        }
    }

#pragma unroll
    for (int q = 0; q < 4; ++q) {
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            const int gi = I0 + rbase + 8 * q + s;
            if (gi >= n) continue;
#pragma unroll
            for (int p = 0; p < kP; ++p) {
                const int gj = J0 + cbase + 16 * p;
                float* dst = d + (int64_t)gi * ld + gj;
                if (gj + 1 < n) {
                    *reinterpret_cast<float2*>(dst) = make_float2(acc[2 * q + s][2 * p], acc[2 * q + s][2 * p + 1]);
                } else if (gj < n) {
                    dst[0] = acc[2 * q + s][2 * p];
                }
            }
        }
    }
}

constexpr size_t kUpdateSmem = sizeof(float2) * 32 * (kTile + kApad) + sizeof(float2) * 32 * kTile;
static_assert(sizeof(PanelSmem) <= kUpdateSmem, "panel tiles reuse the update stage");

__global__ void __launch_bounds__(256) k_fw_panels(float* __restrict__ d, int n, int ld, int kb, int nt) {
    __shared__ PanelSmem sm;
    fw_panel_tile<false>(d, n, ld, nt, kb, blockIdx.x, sm);
}

template <int kCols>
__global__ void __launch_bounds__(256, 2) k_fw_update(float* __restrict__ d, int n, int ld, int kb) {
    extern __shared__ float4 fw_smem[];
    float2* As = reinterpret_cast<float2*>(fw_smem);
    float2* Bs = As + 32 * (kTile + kApad);
    fw_update_tile<false, kCols>(d, n, ld, kb, blockIdx.y, blockIdx.x, As, Bs);
}

cudaError_t fw_solve(float* d, int n, int ld, int padded, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    int sms = 0, dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) e = raise_smem_limit(reinterpret_cast<const void*>(k_fw_update<kTile>));
    if (e == cudaSuccess) e = raise_smem_limit(reinterpret_cast<const void*>(k_fw_update<kTile / 2>));
    if (e != cudaSuccess) return e;
    const int nt = (n + kKB - 1) / kKB;
    const int nu = (n + kTile - 1) / kTile;
    // Tiles of 64 columns as long as each gets an SM of its own (n = 1021: 143
    // against 233 us in 16 rounds, 64 tiles of 128 x 128 leave 88 SMs idle; n =
    // 1300: 296 against 305, n = 2048: 844 against 747).
    const bool narrow = nt * nu <= sms;
    for (int kb = 0; kb < nt; ++kb) {
        k_fw_panels<<<2 * nt - 1, 256, 0, st>>>(d, padded, ld, kb, nt);
        ++g_launch_counter;
        if (nt > 1) {
            if (narrow) k_fw_update<kTile / 2><<<dim3(nt, nu), 256, kUpdateSmem, st>>>(d, padded, ld, kb);
            else k_fw_update<kTile><<<dim3(nu, nu), 256, kUpdateSmem, st>>>(d, padded, ld, kb);
            ++g_launch_counter;
        }
    }
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// persistent batched solve
// ---------------------------------------------------------------------------

// Each CTA claims items until the queue is empty. An item is
// {graph, round, kind (0 panel, 1 update), tile}. Every 64 x 64 block of a
// graph has a version counter: the number of rounds whose writes to it are
// done (round r writes each block once, by its panel tile when the block is
// in row or column block r, else by the update tile holding it). An item of
// round r waits for exactly the blocks it reads:
//   panel  (r, X)    : X at version >= r, and block (r, r) at version >= r
//                      for the diagonal item (which closes it) or >= r + 1
//                      for the row and column items (which read it closed);
//   update (r, tile) : its A and B panel blocks (column / row block r) at
//                      version >= r + 1 and its own blocks outside row and
//                      column block r at version >= r; a tile holding row or
//                      column block r - 1 also waits for every update tile of
//                      round r - 1 (per-round counters after the versions),
//                      which read those blocks as operands and must not see
//                      them rewritten.
// The queue is ordered with a one-round look-ahead: the update tiles of round
// r that hold row or column block r + 1 come first, then the panel tiles of
// round r + 1, then the rest of round r's update tiles. Every item's
// dependencies come earlier in the queue, so the holder of the earliest
// unfinished item can always proceed: the schedule cannot deadlock whatever
// the residency, and panels overlap the bulk of the previous round's update.
// Waits spin at most kSpinLimit polls (with nanosleep) and then raise
// err[0] = 1; every CTA checks err[0] before each item, so a stalled queue
// ends the launch instead of hanging the GPU.
constexpr uint32_t kSpinLimit = 1u << 24;  // x ~100-200 ns sleeps: seconds

__device__ __forceinline__ uint32_t ld_acquire(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// Bounded wait for *v >= target, at most `limit` polls; false (and err set)
// when it gives up.
__device__ __forceinline__ bool wait_version_limit(const uint32_t* v, uint32_t target, uint32_t* err,
                                                   uint32_t limit) {
    uint32_t spins = 0;
    while (ld_acquire(v) < target) {
        if (++spins > limit || ld_acquire(err) != 0) {
            atomicExch(err, 1u);
            return false;
        }
        __nanosleep(100);
    }
    return true;
}

__device__ __forceinline__ bool wait_version(const uint32_t* v, uint32_t target, uint32_t* err) {
    return wait_version_limit(v, target, err, kSpinLimit);
}

// The persistent solves' bounded wait on its own: one thread waits for
// words[0] >= 1, which nothing sets, for at most `limit` polls and then
// raises words[1] as the solves raise their error word; words[2] = 1 when
// the wait gave up, 2 when it returned.
__global__ void k_wait_probe(uint32_t* words, uint32_t limit) {
    if (threadIdx.x != 0) return;
    const bool ok = wait_version_limit(words, 1u, words + 1, limit);
    words[2] = ok ? 2u : 1u;
}

cudaError_t wait_probe(uint32_t* words, uint32_t limit, cudaStream_t st) {
    k_wait_probe<<<1, 32, 0, st>>>(words, limit);
    ++g_launch_counter;
    return cudaGetLastError();
}

__global__ void __launch_bounds__(256, 2) k_fw_persistent(float* __restrict__ base, const FwGraph* __restrict__ gs,
                                                          const int4* __restrict__ items, int n_items,
                                                          uint32_t* __restrict__ sync) {
    // sync layout: [0] queue head, [1] error flag, then per graph g the nt^2
    // block versions at sync + 2 + gs[g].vofs (row-major blocks)
    extern __shared__ float4 fw_smem[];
    float2* As = reinterpret_cast<float2*>(fw_smem);
    float2* Bs = As + 32 * (kTile + kApad);
    PanelSmem& psm = *reinterpret_cast<PanelSmem*>(fw_smem);
    __shared__ int s_item;
    __shared__ int s_abort;
    uint32_t* head = sync;
    uint32_t* err = sync + 1;
    for (;;) {
        if (threadIdx.x == 0) {
            s_item = (int)atomicAdd(head, 1u);
            s_abort = ld_acquire(err) != 0;
        }
        __syncthreads();
        const int it = s_item;
        if (it >= n_items || s_abort) break;
        const int4 w = items[it];
        const FwGraph g = gs[w.x];
        uint32_t* ver = sync + 2 + g.vofs;
        const int r = w.y, nt = g.nt;
        if (threadIdx.x == 0) {
            bool ok = true;
            if (w.z == 0) {
                int bi = r, bj = r;  // the block this panel tile writes
                if (w.w > 0) {
                    int q = w.w - 1;
                    const bool col = q >= nt - 1;
                    if (col) q -= nt - 1;
                    const int other = q < r ? q : q + 1;
                    bi = col ? other : r;
                    bj = col ? r : other;
                }
                // the diagonal item waits for its block's round r - 1; row
                // and column panels for the diagonal closed in round r
                ok = wait_version(ver + r * nt + r, (uint32_t)r + (w.w > 0 ? 1u : 0u), err) &&
                     wait_version(ver + bi * nt + bj, (uint32_t)r, err);
            } else {
                const int ti = w.w / g.nu, tj = w.w % g.nu;
                // a tile that rewrites row or column block r - 1 waits until
                // every update tile of round r - 1 (which read those blocks
                // as operands) is done
                if (r >= 1 && (2 * ti == r - 1 || 2 * ti + 1 == r - 1 || 2 * tj == r - 1 || 2 * tj + 1 == r - 1))
                    ok = wait_version(ver + nt * nt + (r - 1), (uint32_t)(g.nu * g.nu), err);
                for (int a = 0; a < 2 && ok; ++a) {
                    const int bi = 2 * ti + a, bj = 2 * tj + a;
                    if (bi < nt) ok = wait_version(ver + bi * nt + r, (uint32_t)r + 1u, err);
                    if (ok && bj < nt) ok = wait_version(ver + r * nt + bj, (uint32_t)r + 1u, err);
                }
                for (int a = 0; a < 2 && ok; ++a)
                    for (int c = 0; c < 2 && ok; ++c) {
                        const int bi = 2 * ti + a, bj = 2 * tj + c;
                        if (bi < nt && bj < nt && bi != r && bj != r)
                            ok = wait_version(ver + bi * nt + bj, (uint32_t)r, err);
                    }
            }
            if (!ok) s_abort = 1;
        }
        __syncthreads();
        if (s_abort) break;
        float* d = base + g.off;
        if (w.z == 0) {
            fw_panel_tile<true>(d, g.n, g.ld, nt, r, w.w, psm, /*closed_diag=*/true);
        } else {
            fw_update_tile<true>(d, g.n, g.ld, r, w.w / g.nu, w.w % g.nu, As, Bs);
        }
        __threadfence();
        __syncthreads();
        if (threadIdx.x == 0) {
            if (w.z == 0) {
                int bi = r, bj = r;
                if (w.w > 0) {
                    int q = w.w - 1;
                    const bool col = q >= nt - 1;
                    if (col) q -= nt - 1;
                    const int other = q < r ? q : q + 1;
                    bi = col ? other : r;
                    bj = col ? r : other;
                }
                atomicAdd(ver + bi * nt + bj, 1u);
            } else {
                const int ti = w.w / g.nu, tj = w.w % g.nu;
                for (int a = 0; a < 2; ++a)
                    for (int c = 0; c < 2; ++c) {
                        const int bi = 2 * ti + a, bj = 2 * tj + c;
                        if (bi < nt && bj < nt && bi != r && bj != r) atomicAdd(ver + bi * nt + bj, 1u);
                    }
                atomicAdd(ver + nt * nt + r, 1u);  // finished update tiles of round r
            }
        }
    }
}

size_t fw_batched_items(const FwGraph* graphs, int n_graphs, int4* items, bool sym) {
    int max_nt = 0;
    for (int g = 0; g < n_graphs; ++g) max_nt = std::max(max_nt, graphs[g].nt);
    size_t k = 0;
    auto emit = [&](int g, int r, int kind, int t) {
        if (items) items[k] = make_int4(g, r, kind, t);
        ++k;
    };
    // the general solve has a diagonal, row and column panel tiles per round;
    // the symmetric one the diagonal and the column panel only
    // (the symmetric solve closes the diagonal blocks of rounds >= 1 in the
    // strip item that finishes them)
    auto panels = [&](int r) {
        for (int g = 0; g < n_graphs; ++g)
            if (r < graphs[g].nt)
                for (int b = sym && r > 0 ? 1 : 0; b < (sym ? graphs[g].nt : 2 * graphs[g].nt - 1); ++b)
                    emit(g, r, 0, b);
    };
    // prio: the update tiles of round r holding row or column block r + ahead
    auto updates = [&](int r, bool prio, int ahead) {
        for (int g = 0; g < n_graphs; ++g) {
            const FwGraph& G = graphs[g];
            if (r >= G.nt || G.nt < 2) continue;
            const int tn = (r + ahead) / 2;
            for (int t = 0; t < G.nu * G.nu; ++t) {
                const int ti = t / G.nu, tj = t % G.nu;
                if (sym && ti > tj) continue;
                const bool p = r + ahead < G.nt && (ti == tn || tj == tn);
                if (p == prio) emit(g, r, 1, t);
            }
        }
    };
    // symmetric solve: the strip blocks of round r (row / column block r + 1,
    // the diagonal block first) as their own items
    auto strips = [&](int r) {
        for (int g = 0; g < n_graphs; ++g) {
            const int nt = graphs[g].nt;
            if (r + 1 >= nt) continue;
            emit(g, r, 2, r + 1);
            for (int X = 0; X < nt; ++X)
                if (X != r && X != r + 1) emit(g, r, 2, X);
        }
    };
    panels(0);
    for (int r = 0; r < max_nt; ++r) {
        if (sym) {
            // strip blocks, then the next round's panels, then the tiles that
            // hold the next round's strip blocks, then the rest
            strips(r);
            panels(r + 1);
            updates(r, true, 2);
            updates(r, false, 2);
        } else {
            updates(r, true, 1);
            panels(r + 1);
            updates(r, false, 1);
        }
    }
    return k;
}

// List-scheduled order of the symmetric queue. The persistent kernel hands
// items out in queue order; an item claimed before its dependencies are done
// holds its CTA idle, and one claimed long after they are done delays
// everything that waits on it. This reorders the queue by simulating
// `workers` CTAs on the item dependency graph (durations in units of one
// update tile, the ratios measured on GB300 at 2 CTAs per SM): a free CTA
// takes the ready item with the longest remaining dependency chain (ties: the
// structural order), and the simulated claim order becomes the queue. Every item is taken after its dependencies in the
// simulation, so the order stays a dependency order (deadlock-free, checked by
// fw_queue_replay).
void fw_order_sym(const FwGraph* graphs, int n_graphs, int4* items, size_t n_items, int workers) {
    if (n_items == 0 || workers < 1) return;
    const int N = (int)n_items;
    // item lookup: (graph, round, kind, index) -> position in the input
    std::vector<int64_t> pan_off(n_graphs), str_off(n_graphs), upd_off(n_graphs), v_off(n_graphs);
    int64_t tot = 0;
    for (int g = 0; g < n_graphs; ++g) {
        const int nt = graphs[g].nt, nu = graphs[g].nu;
        pan_off[g] = tot; tot += (int64_t)nt * nt;               // [r][b]
        str_off[g] = tot; tot += (int64_t)nt * nt;               // [r][X]
        upd_off[g] = tot; tot += (int64_t)nt * nu * nu;          // [r][t]
    }
    std::vector<int> pos(tot, -1);
    for (int i = 0; i < N; ++i) {
        const int4 w = items[i];
        const FwGraph& G = graphs[w.x];
        int64_t k;
        if (w.z == 0) k = pan_off[w.x] + (int64_t)w.y * G.nt + w.w;
        else if (w.z == 2) k = str_off[w.x] + (int64_t)w.y * G.nt + w.w;
        else k = upd_off[w.x] + ((int64_t)w.y * G.nu * G.nu + w.w);
        pos[k] = i;
    }
    // virtual nodes V(g, q): every update tile and strip item of round q done
    // (the panel slot reuse of round q + 3); numbered after the items
    int64_t nv = 0;
    for (int g = 0; g < n_graphs; ++g) { v_off[g] = N + nv; nv += graphs[g].nt; }
    const int M = N + (int)nv;
    auto panel = [&](int g, int r, int X) {  // the item writing block (X, r) in round r
        if (X == r && r > 0) return pos[str_off[g] + (int64_t)(r - 1) * graphs[g].nt + r];  // fused closure
        const int b = X == r ? 0 : (X < r ? X : X - 1) + 1;
        return pos[pan_off[g] + (int64_t)r * graphs[g].nt + b];
    };
    auto writer = [&](int g, int q, int a, int b) {  // the item writing block (a, b), a <= b, in round q
        const FwGraph& G = graphs[g];
        if (a == q || b == q) return panel(g, q, a == q ? b : a);
        if (a == q + 1 || b == q + 1) return pos[str_off[g] + (int64_t)q * G.nt + (a == q + 1 ? b : a)];
        return pos[upd_off[g] + ((int64_t)q * G.nu * G.nu + (a / 2) * G.nu + b / 2)];
    };
    std::vector<std::vector<int>> succ(M);
    std::vector<int> indeg(M, 0);
    std::vector<float> dur(M, 0.f);
    auto edge = [&](int from, int to) {
        if (from < 0) return;
        succ[from].push_back(to);
        ++indeg[to];
    };
    for (int i = 0; i < N; ++i) {
        const int4 w = items[i];
        const int g = w.x, r = w.y, nt = graphs[g].nt, nu = graphs[g].nu;
        std::vector<int> deps;
        if (w.z == 0) {
            const int X = w.w == 0 ? r : ((w.w - 1) < r ? (w.w - 1) : w.w);
            dur[i] = w.w == 0 ? 0.85f : 0.6f;
            if (w.w > 0) deps.push_back(panel(g, r, r));
            if (r >= 1) deps.push_back(writer(g, r - 1, std::min(X, r), std::max(X, r)));
            if (r >= kPanelSlots) deps.push_back((int)v_off[g] + r - kPanelSlots);
        } else if (w.z == 2) {
            const int X = w.w;
            dur[i] = X == r + 1 ? 0.8f : 0.33f;
            if (X == r + 1 && r + 1 >= kPanelSlots) deps.push_back((int)v_off[g] + r + 1 - kPanelSlots);
            deps.push_back(panel(g, r, X));
            deps.push_back(panel(g, r, r + 1));
            if (r >= 1) deps.push_back(writer(g, r - 1, std::min(X, r + 1), std::max(X, r + 1)));
            edge(i, (int)v_off[g] + r);
        } else {
            const int ti = w.w / nu, tj = w.w % nu;
            dur[i] = 1.f;
            for (int k = 0; k < 4; ++k) deps.push_back(panel(g, r, 2 * (k < 2 ? ti : tj) + (k & 1)));
            for (int a = 0; a < 2; ++a)
                for (int c = 0; c < 2; ++c) {
                    const int bi = 2 * ti + a, bj = 2 * tj + c;
                    if (r >= 1 && bi <= bj && bi != r && bj != r && bi != r + 1 && bj != r + 1)
                        deps.push_back(writer(g, r - 1, bi, bj));
                }
            edge(i, (int)v_off[g] + r);
        }
        (void)nt;
        std::sort(deps.begin(), deps.end());
        deps.erase(std::unique(deps.begin(), deps.end()), deps.end());
        for (int d : deps) edge(d, i);
    }
    // longest remaining chain (bottom level) by a reverse topological pass
    std::vector<int> topo;
    topo.reserve(M);
    {
        std::vector<int> deg = indeg;
        for (int i = 0; i < M; ++i)
            if (deg[i] == 0) topo.push_back(i);
        for (size_t h = 0; h < topo.size(); ++h)
            for (int t : succ[topo[h]])
                if (--deg[t] == 0) topo.push_back(t);
        if ((int)topo.size() != M) return;  // not a DAG: keep the structural order
    }
    std::vector<float> bl(M, 0.f);
    for (int h = M - 1; h >= 0; --h) {
        const int x = topo[h];
        float m = 0.f;
        for (int t : succ[x]) m = std::max(m, bl[t]);
        bl[x] = dur[x] + m;
    }
    // simulation: workers take the ready item with the largest bottom level
    auto cmp_ready = [&](int a, int b) { return bl[a] != bl[b] ? bl[a] < bl[b] : a > b; };
    std::priority_queue<int, std::vector<int>, decltype(cmp_ready)> ready(cmp_ready);
    using Ev = std::pair<float, int>;  // (completion time, node)
    std::priority_queue<Ev, std::vector<Ev>, std::greater<Ev>> events;
    std::priority_queue<float, std::vector<float>, std::greater<float>> free_at;
    for (int k = 0; k < workers; ++k) free_at.push(0.f);
    std::vector<int> deg = indeg;
    std::vector<int4> out;
    out.reserve(N);
    auto complete = [&](int x, float t, auto&& self) -> void {
        for (int s2 : succ[x])
            if (--deg[s2] == 0) {
                if (s2 >= N) self(s2, t, self);  // virtual nodes complete at once
                else ready.push(s2);
            }
    };
    for (int i = 0; i < M; ++i)
        if (deg[i] == 0) {
            if (i >= N) complete(i, 0.f, complete);
            else ready.push(i);
        }
    while ((int)out.size() < N) {
        float t = free_at.top();
        free_at.pop();
        while (!events.empty() && events.top().first <= t) {
            const Ev e = events.top();
            events.pop();
            complete(e.second, e.first, complete);
        }
        while (ready.empty()) {
            if (events.empty()) return;  // cannot happen for a DAG; keep the structural order
            const Ev e = events.top();
            events.pop();
            t = std::max(t, e.first);
            complete(e.second, e.first, complete);
        }
        const int x = ready.top();
        ready.pop();
        out.push_back(items[x]);
        events.push({t + dur[x], x});
        free_at.push(t + dur[x]);
    }
    std::copy(out.begin(), out.end(), items);
}

// Host replay of a queue with the waits and version updates of
// k_fw_persistent (sym = false) or k_fw_persistent_sym (sym = true), one item
// at a time in queue order. Returns 0 when every wait of every item is
// already met at its turn (so the persistent launch cannot deadlock, whatever
// the residency), every block is written exactly once per round, and every
// block ends at version nt; otherwise the 1-based index of the first item
// that breaks one of these.
size_t fw_queue_replay(const FwGraph* graphs, int n_graphs, const int4* items, size_t n_items, bool sym) {
    std::vector<std::vector<uint32_t>> ver(n_graphs), done(n_graphs);
    for (int g = 0; g < n_graphs; ++g) {
        ver[g].assign((size_t)graphs[g].nt * graphs[g].nt, 0u);
        done[g].assign(graphs[g].nt, 0u);
    }
    auto up = [](int a, int b, int nt) { return a < b ? a * nt + b : b * nt + a; };
    for (size_t it = 0; it < n_items; ++it) {
        const int4 w = items[it];
        const FwGraph& G = graphs[w.x];
        const int r = w.y, nt = G.nt;
        std::vector<uint32_t>& v = ver[w.x];
        bool ok = true;
        std::vector<int> writes;
        auto need = [&](int idx, uint32_t target) { ok = ok && v[idx] >= target; };
        if (!sym) {
            if (w.z == 0) {
                int bi = r, bj = r;
                if (w.w > 0) {
                    int q = w.w - 1;
                    const bool col = q >= nt - 1;
                    if (col) q -= nt - 1;
                    const int other = q < r ? q : q + 1;
                    bi = col ? other : r;
                    bj = col ? r : other;
                }
                need(r * nt + r, (uint32_t)r + (w.w > 0 ? 1u : 0u));
                need(bi * nt + bj, (uint32_t)r);
                writes.push_back(bi * nt + bj);
            } else {
                const int ti = w.w / G.nu, tj = w.w % G.nu;
                if (r >= 1 && (2 * ti == r - 1 || 2 * ti + 1 == r - 1 || 2 * tj == r - 1 || 2 * tj + 1 == r - 1))
                    ok = ok && done[w.x][r - 1] >= (uint32_t)(G.nu * G.nu);
                ++done[w.x][r];
                for (int a = 0; a < 2; ++a) {
                    const int bi = 2 * ti + a, bj = 2 * tj + a;
                    if (bi < nt) need(bi * nt + r, (uint32_t)r + 1u);
                    if (bj < nt) need(r * nt + bj, (uint32_t)r + 1u);
                }
                for (int a = 0; a < 2; ++a)
                    for (int c = 0; c < 2; ++c) {
                        const int bi = 2 * ti + a, bj = 2 * tj + c;
                        if (bi < nt && bj < nt && bi != r && bj != r) {
                            need(bi * nt + bj, (uint32_t)r);
                            writes.push_back(bi * nt + bj);
                        }
                    }
            }
        } else {
            const uint32_t n_upd = (uint32_t)(G.nu * (G.nu + 1) / 2 + G.nt - 1);
            if (w.z == 0) {
                int X = r;
                if (w.w > 0) {
                    const int q = w.w - 1;
                    X = q < r ? q : q + 1;
                }
                if (r >= kPanelSlots) ok = ok && done[w.x][r - kPanelSlots] >= n_upd;
                need(r * nt + r, (uint32_t)r + (w.w > 0 ? 1u : 0u));
                if (w.w > 0) need(up(X, r, nt), (uint32_t)r);
                writes.push_back(up(X, r, nt));
            } else if (w.z == 2) {
                const int X = w.w;
                if (X == r + 1 && r + 1 >= kPanelSlots) ok = ok && done[w.x][r + 1 - kPanelSlots] >= n_upd;
                need(up(X, r, nt), (uint32_t)r + 1u);
                need(up(r + 1, r, nt), (uint32_t)r + 1u);
                need(up(X, r + 1, nt), (uint32_t)r);
                writes.push_back(up(X, r + 1, nt));
                if (X == r + 1) {  // and round r + 1's closure of the same block
                    if (v[up(X, r + 1, nt)] != (uint32_t)r) ok = false;
                    ++v[up(X, r + 1, nt)];
                    writes.pop_back();
                    if (v[up(X, r + 1, nt)] != (uint32_t)r + 1u) ok = false;
                    ++v[up(X, r + 1, nt)];
                }
                ++done[w.x][r];
            } else {
                const int ti = w.w / G.nu, tj = w.w % G.nu;
                if (ti > tj) ok = false;
                for (int k = 0; k < 4; ++k) need(up(2 * (k < 2 ? ti : tj) + (k & 1), r, nt), (uint32_t)r + 1u);
                for (int a = 0; a < 2; ++a)
                    for (int c = 0; c < 2; ++c) {
                        const int bi = 2 * ti + a, bj = 2 * tj + c;
                        if (bi <= bj && bi != r && bj != r && bi != r + 1 && bj != r + 1) {
                            need(bi * nt + bj, (uint32_t)r);
                            writes.push_back(bi * nt + bj);
                        }
                    }
                ++done[w.x][r];
            }
        }
        for (int b : writes) {
            if (v[b] != (uint32_t)r) ok = false;  // exactly one write per block and round
            ++v[b];
        }
        if (!ok) return it + 1;
    }
    for (int g = 0; g < n_graphs; ++g) {
        const int nt = graphs[g].nt;
        for (int a = 0; a < nt; ++a)
            for (int b = 0; b < nt; ++b)
                if ((!sym || a <= b) && ver[g][(size_t)a * nt + b] != (uint32_t)nt) return n_items + 1;
    }
    return 0;
}

size_t fw_sync_words(const FwGraph* graphs, int n_graphs) {
    size_t w = 2;
    for (int g = 0; g < n_graphs; ++g) w += (size_t)graphs[g].nt * graphs[g].nt + graphs[g].nt;
    return w;
}

cudaError_t fw_solve_batched(float* base, const FwGraph* graphs, const int4* items, int n_items, uint32_t* sync,
                             size_t sync_words, int ctas, cudaStream_t st) {
    cudaError_t e = raise_smem_limit(reinterpret_cast<const void*>(k_fw_persistent));
    if (e != cudaSuccess) return e;
    e = cudaMemsetAsync(sync, 0, sizeof(uint32_t) * sync_words, st);
    if (e != cudaSuccess) return e;
    if (n_items == 0) return cudaSuccess;
    k_fw_persistent<<<ctas, 256, kUpdateSmem, st>>>(base, graphs, items, n_items, sync);
    ++g_launch_counter;
    return cudaGetLastError();
}

int fw_persistent_ctas_per_sm() {
    int blocks = 0;
    if (raise_smem_limit(reinterpret_cast<const void*>(k_fw_persistent)) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, k_fw_persistent, 256, kUpdateSmem) != cudaSuccess)
        return 1;
    return std::max(blocks, 1);
}

// ---------------------------------------------------------------------------
// symmetric persistent solve
// ---------------------------------------------------------------------------
// LightGraph's path matrices are symmetric (every edge is stored both ways,
// src/LightGraph.h:405-406), and the recurrence keeps them exactly symmetric
// in FP32: S_ik + S_kj and S_jk + S_ki are the same IEEE sum, so S_ij and S_ji
// see bit-identical candidates in every round. This solve therefore keeps only
// the 64 x 64 blocks on and above the diagonal up to date (block (a, b) with
// a > b is read as the transpose of block (b, a)) and mirrors them below the
// diagonal at the end: half the update tiles of the general solve, with
// results identical to it.
//
// Round r:
//   diagonal item : closes block (r, r);
//   panel item X  : block (X, r) = min(T, T (x) Dg*) with T = S[X-block][r-block]
//                   (stored as block (r, X) transposed when X > r);
//   strip item X  : block (X, r + 1), the blocks round r + 1's diagonal and
//                   panel items read, updated on their own right after the
//                   panels (64 x 64 items instead of whole update tiles on
//                   the round-to-round critical path);
//   update tile   : (ti <= tj), C = S[I][J] on and above the diagonal outside
//                   row / column blocks r and r + 1,
//                   C = min(C, A (x) B) with A = S[I][r-block] and, by symmetry,
//                   B = S[r-block][J] = (S[J][r-block])^T.
// Both operands are rows of the round's column panel S[*][r-block]. The panel
// items write that panel, in the k-pair form the update tiles consume, to one
// of three slots (round r uses slot r % 3):
//   slot[ti][kp][i] = {S[128 ti + i][64 r + 2 kp], S[128 ti + i][64 r + 2 kp + 1]}
// so an update tile stages each operand with one contiguous 32 KB copy and
// never reads the column blocks that round r + 1 rewrites. A panel item of
// round r reuses slot r % 3 only after all update tiles and strip items of
// round r - 3 are done (per-round counters after the block versions).
// Queue order per round: strips(r), panels(r + 1), the update tiles of round
// r holding row / column block r + 2 (the next strips' blocks), the rest.


size_t fw_panel_words(const FwGraph& g) { return (size_t)kPanelSlots * g.nu * 32 * kTile; }

__device__ __forceinline__ int up_block(int a, int b, int nt) { return a < b ? a * nt + b : b * nt + a; }

// TMA bulk copies (cp.async.bulk, global -> shared) completed on an mbarrier:
// the update tiles of the symmetric solve's TMA schedule stage their two
// panel-slot operands this way. One mbarrier per CTA; each update item arms it
// with its byte count (one arrival) and every thread waits for the phase.
__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(bar)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n\t}" ::"r"(
                     smem_addr(bar)),
                 "r"(bytes)
                 : "memory");
}

// Copy `bytes` (a multiple of 16; both addresses 16-byte aligned) from global
// src to shared dst; completion counts against bar's transaction bytes. The
// proxy fence orders the generic-proxy writes this thread has seen (panel
// slots published by other CTAs) before the async-proxy read.
__device__ __forceinline__ void tma_copy_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("fence.proxy.async.global;" ::: "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_addr(dst)),
                 "l"(src), "r"(bytes), "r"(smem_addr(bar))
                 : "memory");
}

__device__ __forceinline__ bool mbar_try(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, 20000;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// Bounded wait for phase `parity` of bar (try_wait suspends the thread until
// the phase completes or about 20 us pass). If it gives up it raises err (the
// whole launch then stops at its next item) and waits once more, again
// bounded, so that no copy is left writing this CTA's shared memory.
__device__ __forceinline__ void mbar_wait(uint64_t* bar, uint32_t parity, uint32_t* err) {
    uint32_t spins = 0;
    while (!mbar_try(bar, parity)) {
        if (++spins == (1u << 16)) atomicExch(err, 1u);
        if (spins >= (1u << 17)) return;
    }
}

// Generic-proxy shared-memory writes of this thread before a later TMA write
// of the same bytes (an item's shared memory is the next item's TMA target).
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// Closes diagonal block kb held in sm.T, writes it back to d and its rows to
// the round's panel slot Pr.
__device__ __noinline__ void close_publish_diag(float* __restrict__ d, int ld, int kb, float2* __restrict__ Pr,
                                                PanelSmem& sm) {
    const int tid = threadIdx.x, K0 = kb * kKB;
    close_diag_blocked(sm.T);
    for (int e = tid; e < kKB * kKB; e += 256) {
        const int r = e >> 6, c = e & 63;
        d[(int64_t)(K0 + r) * ld + K0 + c] = sm.T[r][c];
    }
    float2* dst = Pr + (size_t)(kb >> 1) * 32 * kTile + (kb & 1) * kKB;
    for (int e = tid; e < 32 * kKB; e += 256) {
        const int kp = e >> 6, i = e & 63;
        dst[kp * kTile + i] = *reinterpret_cast<const float2*>(&sm.T[i][2 * kp]);
    }
}

// Diagonal (b = 0, round 0 only: later diagonal blocks are closed by the
// strip item that finishes them) or column panel item b >= 1 of round kb
// (block X = the b-th block other than kb). 256 threads; the result goes back
// to its block above the diagonal and into the round's panel slot Pr.
__device__ __noinline__ void fw_panel_tile_sym(float* __restrict__ d, int ld, int kb, int b,
                                                  float2* __restrict__ Pr, PanelSmem& sm) {
    const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
    const int K0 = kb * kKB;
    int X = kb;
    if (b > 0) {
        const int q = b - 1;
        X = q < kb ? q : q + 1;
    }
    const int X0 = X * kKB;
    if (b == 0) {
        for (int e = tid; e < kKB * kKB; e += 256) {
            const int r = e >> 6, c = e & 63;
            sm.T[r][c] = __ldcg(d + (int64_t)(K0 + r) * ld + K0 + c);
        }
        __syncthreads();
        close_publish_diag(d, ld, kb, Pr, sm);
        return;
    } else {
        // every load in flight before the first store (48 graphs of 750 points: 1.15
        // -> 1.09 ms, one of 750: 0.33 -> 0.30 ms)
        const int r0 = tid >> 6, c0 = tid & 63, r4 = tid >> 4, c4 = (tid & 15) * 4;
        const float* from = X < kb ? d + (int64_t)X0 * ld + K0 : d + (int64_t)K0 * ld + X0;
        float pt[16];
        float4 dg[4];
#pragma unroll
        for (int q = 0; q < 16; ++q) pt[q] = __ldcg(from + (int64_t)(r0 + 4 * q) * ld + c0);
#pragma unroll
        for (int q = 0; q < 4; ++q) dg[q] = ldm4<true>(d + (int64_t)(K0 + r4 + 16 * q) * ld + K0 + c4);
#pragma unroll
        for (int q = 0; q < 16; ++q) {
            if (X < kb) sm.T[r0 + 4 * q][c0] = pt[q];
            else sm.T[c0][r0 + 4 * q] = pt[q];
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            float2* to = reinterpret_cast<float2*>(&sm.Dg[r4 + 16 * q][c4]);
            to[0] = make_float2(dg[q].x, dg[q].y);
            to[1] = make_float2(dg[q].z, dg[q].w);
        }
        __syncthreads();
        float acc[4][4];
        panel_product(sm, false, ty, tx, acc);
        __syncthreads();
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int c = 0; c < 4; ++c) sm.T[ty + 16 * r][tx + 16 * c] = acc[r][c];
        __syncthreads();
    }
    // the block above the diagonal (transposed when X > kb)
    for (int e = tid; e < kKB * kKB; e += 256) {
        const int r = e >> 6, c = e & 63;
        if (X <= kb) d[(int64_t)(X0 + r) * ld + K0 + c] = sm.T[r][c];
        else d[(int64_t)(K0 + r) * ld + X0 + c] = sm.T[c][r];
    }
    // the rows of block X in the panel slot
    float2* dst = Pr + (size_t)(X >> 1) * 32 * kTile + (X & 1) * kKB;
    for (int e = tid; e < 32 * kKB; e += 256) {
        const int kp = e >> 6, i = e & 63;
        dst[kp * kTile + i] = *reinterpret_cast<const float2*>(&sm.T[i][2 * kp]);
    }
}

// Strip block (a, b), a <= b, of round kb: one of the 64 x 64 blocks in row
// or column block kb + 1, which round kb + 1's diagonal and panel items read.
// It runs as its own item right after round kb's panels, so that the next
// round does not wait for whole update tiles:
//   C = min(C, A (x) B^T), A / B = the panel-slot rows of block a / b.
// The diagonal strip block (kb + 1, kb + 1) is then closed at once as round
// kb + 1's diagonal item (close_publish_diag, into that round's slot Pnext).
// 256 threads, each owning the 4 x 4 elements (ty + 16r, tx + 16c), k in
// pairs (add.rn.f32x2 + 3-input min) as in the update tiles.
__device__ __forceinline__ void fw_strip_tile_sym(float* __restrict__ d, int ld, int a, int b,
                                                  const float2* __restrict__ Pr, float2* __restrict__ Pnext,
                                                  float2* __restrict__ As, float2* __restrict__ Bs,
                                                  PanelSmem& sm) {
    const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
    const float4* pa = reinterpret_cast<const float4*>(Pr + (size_t)(a >> 1) * 32 * kTile + (a & 1) * kKB);
    const float4* pb = reinterpret_cast<const float4*>(Pr + (size_t)(b >> 1) * 32 * kTile + (b & 1) * kKB);
    // As[kp][i] = {S[64a + i][k], S[64a + i][k + 1]}: 32 k-pairs x 32 float4
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        const int e = tid + 256 * m, kp = e >> 5, i2 = e & 31;
        reinterpret_cast<float4*>(As)[e] = __ldcg(pa + kp * (kTile / 2) + i2);
        reinterpret_cast<float4*>(Bs)[e] = __ldcg(pb + kp * (kTile / 2) + i2);
    }
    float acc[4][4];
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[r][c] = __ldcg(d + (int64_t)(a * kKB + ty + 16 * r) * ld + b * kKB + tx + 16 * c);
    __syncthreads();
#pragma unroll 4
    for (int kp = 0; kp < 32; ++kp) {
        float2 av[4], bv[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) av[r] = As[kp * kKB + ty + 16 * r];
#pragma unroll
        for (int c = 0; c < 4; ++c) bv[c] = Bs[kp * kKB + tx + 16 * c];
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const float2 sv = __fadd2_rn(av[r], bv[c]);
                acc[r][c] = min3f(acc[r][c], sv.x, sv.y);
            }
    }
    if (a == b) {
        // the diagonal block a = kb + 1 is final for round kb: close it for
        // round a right here (its diagonal item) into the next slot Pnext
        __syncthreads();
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int c = 0; c < 4; ++c) sm.T[ty + 16 * r][tx + 16 * c] = acc[r][c];
        __syncthreads();
        close_publish_diag(d, ld, a, Pnext, sm);
        return;
    }
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) d[(int64_t)(a * kKB + ty + 16 * r) * ld + b * kKB + tx + 16 * c] = acc[r][c];
}

// Update tile (ti, tj), ti <= tj, of round kb: the inner loop of
// fw_update_tile with both operands copied from the panel slot Pr. Blocks
// that other items of the round own (row / column block kb: panel items;
// row / column block kb + 1: strip items) and, in a diagonal tile, the block
// below the diagonal are left out; each is two warps' work (48
// graphs of 750 points: 1.33 -> 1.15 ms, one of 4096: 2.70 -> 2.58 ms).
template <bool kTma>
__device__ __forceinline__ void fw_update_tile_sym(float* __restrict__ d, int ld, int kb, int ti, int tj,
                                                   const float2* __restrict__ Pr, float2* __restrict__ As,
                                                   float2* __restrict__ Bs, uint64_t* bar, uint32_t parity,
                                                   uint32_t* err) {
    const int I0 = ti * kTile, J0 = tj * kTile;
    const int tid = threadIdx.x;
    if (kTma) {
        // both operands are contiguous 32 KB runs of the panel slot: one TMA
        // copy each (lanes 0 and 1 of warp 0), in flight while the tile loads
        if (tid < 32) {
            if (tid == 0) mbar_expect_tx(bar, 2 * 32 * kTile * (uint32_t)sizeof(float2));
            __syncwarp();
            if (tid < 2)
                tma_copy_g2s(tid == 0 ? As : Bs, Pr + (size_t)(tid == 0 ? ti : tj) * 32 * kTile,
                             32 * kTile * (uint32_t)sizeof(float2), bar);
        }
    } else {
        // through registers: every thread moves 8 + 8 float4
        const float4* pa = reinterpret_cast<const float4*>(Pr + (size_t)ti * 32 * kTile);
        const float4* pb = reinterpret_cast<const float4*>(Pr + (size_t)tj * 32 * kTile);
        float4* sa = reinterpret_cast<float4*>(As);
        float4* sb = reinterpret_cast<float4*>(Bs);
        float4 va[8], vb[8];
#pragma unroll
        for (int m = 0; m < 8; ++m) va[m] = __ldcg(pa + tid + 256 * m);
#pragma unroll
        for (int m = 0; m < 8; ++m) vb[m] = __ldcg(pb + tid + 256 * m);
#pragma unroll
        for (int m = 0; m < 8; ++m) sa[tid + 256 * m] = va[m];
#pragma unroll
        for (int m = 0; m < 8; ++m) sb[tid + 256 * m] = vb[m];
    }
    const int warp = tid >> 5, lane = tid & 31;
    const int wy = warp >> 1, wx = warp & 1, ty = lane >> 3, tx = lane & 7;
    const int rbase = wy * 32 + ty * 2;  // rows rbase + 8q + {0,1}
    const int cbase = wx * 64 + tx * 2;  // cols cbase + 16p + {0,1}
    const int bi = 2 * ti + (wy >> 1), bj = 2 * tj + wx;  // the warp's block
    const bool own = bi <= bj && bi != kb && bj != kb && bi != kb + 1 && bj != kb + 1;
    float acc[8][8];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            const int gi = I0 + rbase + 8 * q + s;
#pragma unroll
            for (int p = 0; p < 4; ++p) {
                const int gj = J0 + cbase + 16 * p;
                float2 v = make_float2(kInf, kInf);
                if (own) v = __ldcg(reinterpret_cast<const float2*>(d + (int64_t)gi * ld + gj));
                acc[2 * q + s][2 * p] = v.x;
                acc[2 * q + s][2 * p + 1] = v.y;
            }
        }
    }
    if (kTma) mbar_wait(bar, parity, err);
    else __syncthreads();
    if (!own) return;

#pragma unroll 1
    for (int kp = 0; kp < 32; ++kp) {
        float2 a[8], b[8];
        const float4* ap = reinterpret_cast<const float4*>(As + kp * kTile + rbase);
        const float4* bp = reinterpret_cast<const float4*>(Bs + kp * kTile + cbase);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const float4 va = ap[4 * q];   // rows rbase + 8q, +1
            a[2 * q] = make_float2(va.x, va.y);
            a[2 * q + 1] = make_float2(va.z, va.w);
            const float4 vb = bp[8 * q];   // cols cbase + 16q, +1
            b[2 * q] = make_float2(vb.x, vb.y);
            b[2 * q + 1] = make_float2(vb.z, vb.w);
        }
#pragma unroll
        for (int r = 0; r < 8; ++r) {
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                const float2 s = __fadd2_rn(a[r], b[c]);
                acc[r][c] = min3f(acc[r][c], s.x, s.y);
            }
        }
    }

    // store the blocks this tile owns
#pragma unroll
    for (int q = 0; q < 4; ++q) {
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            const int gi = I0 + rbase + 8 * q + s;
#pragma unroll
            for (int p = 0; p < 4; ++p) {
                const int gj = J0 + cbase + 16 * p;
                *reinterpret_cast<float2*>(d + (int64_t)gi * ld + gj) =
                    make_float2(acc[2 * q + s][2 * p], acc[2 * q + s][2 * p + 1]);
            }
        }
    }
}

constexpr size_t kUpdateSymSmem = sizeof(float2) * 2 * 32 * kTile;
static_assert(sizeof(PanelSmem) <= kUpdateSymSmem, "panel items reuse the update stage");

// The persistent loop of the symmetric solve: the queue, the bounded waits
// and the error flag work as in k_fw_persistent. Waits of an item of round r:
//   diagonal      : block (r, r) at version >= r;
//   panel X       : block (r, r) at >= r + 1 (closed) and block (X, r) at >= r;
//   strip X       : the column-panel blocks (X, r) and (r + 1, r) at >= r + 1,
//                   its block (X, r + 1) at >= r;
//   update tile   : the column-panel blocks of its four block rows / columns
//                   at >= r + 1, the blocks it owns at >= r;
//   panel items of round r >= 3 also wait for every update tile and strip
//   item of round r - 3 (the last readers of their panel slot).
// Every dependency is an item earlier in the queue, so it cannot deadlock.
// One queue item of the symmetric solve, decoded (by thread 0, before the
// item for its waits and again after it for its version updates, so that
// nothing of it stays live in registers across the tile).
struct SymItem {
    uint32_t* ver;   // the graph's block versions
    uint32_t* done;  // the graph's finished update tiles per round
    int r, nt, kind, b, X, ti, tj;  // kind 0 panel (b, block X), 1 update tile (ti, tj), 2 strip block X
    uint32_t n_upd;
};

__device__ __forceinline__ SymItem decode_sym(const int4* items, const FwGraph* gs, uint32_t* sync, int it) {
    const int4 w = items[it];
    const FwGraph g = gs[w.x];
    SymItem m;
    m.ver = sync + 2 + g.vofs;
    m.done = m.ver + g.nt * g.nt;
    m.r = w.y;
    m.nt = g.nt;
    m.kind = w.z;
    m.b = w.w;
    m.X = m.r;
    if (w.z == 0 && w.w > 0) {
        const int q = w.w - 1;
        m.X = q < m.r ? q : q + 1;
    }
    if (w.z == 2) m.X = w.w;
    m.ti = w.w / g.nu;
    m.tj = w.w % g.nu;
    // update tiles and strip blocks of a round that has strip blocks (every
    // round a panel item waits for: r - 3 with r < nt)
    m.n_upd = (uint32_t)(g.nu * (g.nu + 1) / 2 + g.nt - 1);
    return m;
}

template <bool kTma>
__global__ void __launch_bounds__(256, 2) k_fw_persistent_sym(float* __restrict__ base, const FwGraph* __restrict__ gs,
                                                              const int4* __restrict__ items, int n_items,
                                                              uint32_t* __restrict__ sync, float2* __restrict__ panels) {
    extern __shared__ float4 fw_smem[];
    float2* As = reinterpret_cast<float2*>(fw_smem);
    float2* Bs = As + 32 * kTile;
    PanelSmem& psm = *reinterpret_cast<PanelSmem*>(fw_smem);
    __shared__ int s_item;
    __shared__ int s_abort;
    __shared__ __align__(8) uint64_t s_bar;  // the TMA copies of update items (kTma)
    uint32_t* head = sync;
    uint32_t* err = sync + 1;
    uint32_t tma_phase = 0;  // update items so far: s_bar's phase (uniform over the CTA)
    if (kTma && threadIdx.x == 0) mbar_init(&s_bar);
    for (;;) {
        if (threadIdx.x == 0) {
            const int it = (int)atomicAdd(head, 1u);
            s_item = it;
            s_abort = ld_acquire(err) != 0;
            if (it < n_items && !s_abort) {
                const SymItem m = decode_sym(items, gs, sync, it);
                const int r = m.r, nt = m.nt;
                bool ok = true;
                if (m.kind == 0) {
                    if (r >= kPanelSlots) ok = wait_version(m.done + (r - kPanelSlots), m.n_upd, err);
                    ok = ok && wait_version(m.ver + r * nt + r, (uint32_t)r + (m.b > 0 ? 1u : 0u), err);
                    if (ok && m.b > 0) ok = wait_version(m.ver + up_block(m.X, r, nt), (uint32_t)r, err);
                } else if (m.kind == 2) {
                    // the diagonal strip also opens round r + 1's panel slot
                    if (m.X == r + 1 && r + 1 >= kPanelSlots)
                        ok = wait_version(m.done + (r + 1 - kPanelSlots), m.n_upd, err);
                    ok = ok && wait_version(m.ver + up_block(m.X, r, nt), (uint32_t)r + 1u, err) &&
                         wait_version(m.ver + up_block(r + 1, r, nt), (uint32_t)r + 1u, err) &&
                         wait_version(m.ver + up_block(m.X, r + 1, nt), (uint32_t)r, err);
                } else {
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const int ob = 2 * (k < 2 ? m.ti : m.tj) + (k & 1);  // operand block rows
                        ok = ok && wait_version(m.ver + up_block(ob, r, nt), (uint32_t)r + 1u, err);
                    }
                    for (int a = 0; a < 2 && ok; ++a)
                        for (int c = 0; c < 2 && ok; ++c) {
                            const int bi = 2 * m.ti + a, bj = 2 * m.tj + c;
                            if (bi <= bj && bi != r && bj != r && bi != r + 1 && bj != r + 1)
                                ok = wait_version(m.ver + bi * nt + bj, (uint32_t)r, err);
                        }
                }
                if (!ok) s_abort = 1;
            }
        }
        __syncthreads();
        const int it = s_item;
        if (it >= n_items || s_abort) break;
        const int4 w = items[it];
        const FwGraph g = gs[w.x];
        float* d = base + g.off;
        float2* Pr = panels + g.pofs + (size_t)(w.y % kPanelSlots) * g.nu * 32 * kTile;
        if (w.z == 0) {
            fw_panel_tile_sym(d, g.ld, w.y, w.w, Pr, psm);
        } else if (w.z == 2) {
            float2* Pnext = panels + g.pofs + (size_t)((w.y + 1) % kPanelSlots) * g.nu * 32 * kTile;
            fw_strip_tile_sym(d, g.ld, min(w.w, w.y + 1), max(w.w, w.y + 1), Pr, Pnext, As, Bs, psm);
        } else {
            fw_update_tile_sym<kTma>(d, g.ld, w.y, w.w / g.nu, w.w % g.nu, Pr, As, Bs, &s_bar, tma_phase & 1u,
                                     err);
            if (kTma) ++tma_phase;
        }
        // this item's shared-memory writes come before the next TMA write
        if (kTma) fence_async_smem();
        __threadfence();
        __syncthreads();
        if (threadIdx.x == 0) {
            const SymItem m = decode_sym(items, gs, sync, it);
            const int r = m.r, nt = m.nt;
            if (m.kind == 0) {
                atomicAdd(m.ver + up_block(m.X, r, nt), 1u);
            } else if (m.kind == 2) {
                // the diagonal strip block also got its round r + 1 closure
                atomicAdd(m.ver + up_block(m.X, r + 1, nt), m.X == r + 1 ? 2u : 1u);
                atomicAdd(m.done + r, 1u);
            } else {
                for (int a = 0; a < 2; ++a)
                    for (int c = 0; c < 2; ++c) {
                        const int bi = 2 * m.ti + a, bj = 2 * m.tj + c;
                        if (bi <= bj && bi != r && bj != r && bi != r + 1 && bj != r + 1)
                            atomicAdd(m.ver + bi * nt + bj, 1u);
                    }
                atomicAdd(m.done + r, 1u);
            }
        }
    }
}

// Copies every block above the diagonal to its mirror below it (one 64 x 64
// block per CTA and step, through shared memory so both sides are coalesced).
__global__ void __launch_bounds__(256) k_fw_mirror(float* __restrict__ base, const FwGraph* __restrict__ gs) {
    __shared__ float tile[kKB][kKB + 1];
    const FwGraph g = gs[blockIdx.y];
    const int nt = g.nt;
    float* d = base + g.off;
    for (int t = blockIdx.x; t < nt * nt; t += gridDim.x) {
        const int bi = t / nt, bj = t % nt;
        if (bi >= bj) continue;
        for (int e = threadIdx.x; e < kKB * kKB; e += 256) {
            const int r = e >> 6, c = e & 63;
            tile[r][c] = d[(int64_t)(bi * kKB + r) * g.ld + bj * kKB + c];
        }
        __syncthreads();
        for (int e = threadIdx.x; e < kKB * kKB; e += 256) {
            const int r = e >> 6, c = e & 63;
            d[(int64_t)(bj * kKB + r) * g.ld + bi * kKB + c] = tile[c][r];
        }
        __syncthreads();
    }
}

cudaError_t fw_solve_batched_sym(float* base, const FwGraph* graphs, int n_graphs, int max_nt, const int4* items,
                                 int n_items, uint32_t* sync, size_t sync_words, float2* panels, int ctas, bool tma,
                                 cudaStream_t st) {
    cudaError_t e = raise_smem_limit(reinterpret_cast<const void*>(k_fw_persistent_sym<false>));
    if (e == cudaSuccess) e = raise_smem_limit(reinterpret_cast<const void*>(k_fw_persistent_sym<true>));
    if (e != cudaSuccess) return e;
    e = cudaMemsetAsync(sync, 0, sizeof(uint32_t) * sync_words, st);
    if (e != cudaSuccess) return e;
    if (n_items == 0) return cudaSuccess;
    if (tma)
        k_fw_persistent_sym<true><<<ctas, 256, kUpdateSymSmem, st>>>(base, graphs, items, n_items, sync, panels);
    else
        k_fw_persistent_sym<false><<<ctas, 256, kUpdateSymSmem, st>>>(base, graphs, items, n_items, sync, panels);
    ++g_launch_counter;
    if (max_nt > 1) {
        k_fw_mirror<<<dim3(std::min(max_nt * max_nt, 4096), n_graphs), 256, 0, st>>>(base, graphs);
        ++g_launch_counter;
    }
    return cudaGetLastError();
}

int fw_persistent_sym_ctas_per_sm() {
    int blocks = 0;
    int blocks_tma = 0;
    if (raise_smem_limit(reinterpret_cast<const void*>(k_fw_persistent_sym<false>)) != cudaSuccess ||
        raise_smem_limit(reinterpret_cast<const void*>(k_fw_persistent_sym<true>)) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, k_fw_persistent_sym<false>, 256, kUpdateSymSmem) !=
            cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks_tma, k_fw_persistent_sym<true>, 256, kUpdateSymSmem) !=
            cudaSuccess)
        return 1;
    return std::max(std::min(blocks, blocks_tma), 1);
}

// ---------------------------------------------------------------------------
// inner-loop ceiling
// ---------------------------------------------------------------------------
// The update tiles' inner loop alone: the same 8 x 8 register tile, the same
// conflict-free fragment loads and the same add.rn.f32x2 + 3-input min per two
// k, on operands that stay in shared memory (no staging, no dependency waits,
// no stores), at 2 CTAs per SM. Its rate is the ceiling of min-plus on the
// CUDA cores: each update needs one add and one min, and on GB300 each of
// them takes an FP32 lane cycle whether it is packed (add.rn.f32x2, 3-input
// min) or not, so the ceiling sits near half of the FMA-counted FP32 peak.
__global__ void __launch_bounds__(256, 2) k_fw_inner_loop(float* __restrict__ out, int reps) {
    extern __shared__ float4 fw_smem[];
    float2* As = reinterpret_cast<float2*>(fw_smem);
    float2* Bs = As + 32 * kTile;
    const int tid = threadIdx.x;
    // operand patterns whose minima differ from element to element (small
    // integers and halves: every sum and the tile sums are exact in FP32),
    // so that the results check the arithmetic
    for (int e = tid; e < 32 * kTile; e += 256) {
        As[e] = make_float2((float)((e * 37) % 101), (float)((e * 53) % 97) + 0.25f);
        Bs[e] = make_float2((float)((e * 29) % 89) + 0.5f, (float)((e * 61) % 83));
    }
    __syncthreads();
    const int warp = tid >> 5, lane = tid & 31;
    const int rbase = (warp >> 1) * 32 + (lane >> 3) * 2, cbase = (warp & 1) * 64 + (lane & 7) * 2;
    float acc[8][8];
#pragma unroll
    for (int r = 0; r < 8; ++r)
#pragma unroll
        for (int c = 0; c < 8; ++c) acc[r][c] = 1e30f + (float)(r + c + tid);
    for (int rep = 0; rep < reps; ++rep) {
#pragma unroll 1
        for (int kp = 0; kp < 32; ++kp) {
            float2 a[8], b[8];
            const float4* ap = reinterpret_cast<const float4*>(As + kp * kTile + rbase);
            const float4* bp = reinterpret_cast<const float4*>(Bs + kp * kTile + cbase);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float4 va = ap[4 * q];
                a[2 * q] = make_float2(va.x, va.y);
                a[2 * q + 1] = make_float2(va.z, va.w);
                const float4 vb = bp[8 * q];
                b[2 * q] = make_float2(vb.x, vb.y);
                b[2 * q + 1] = make_float2(vb.z, vb.w);
            }
#pragma unroll
            for (int r = 0; r < 8; ++r)
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    const float2 sv = __fadd2_rn(a[r], b[c]);
                    acc[r][c] = min3f(acc[r][c], sv.x, sv.y);
                }
        }
    }
    float sum = 0.f;
#pragma unroll
    for (int r = 0; r < 8; ++r)
#pragma unroll
        for (int c = 0; c < 8; ++c) sum += acc[r][c];
    out[blockIdx.x * 256 + tid] = sum;
}

cudaError_t fw_inner_loop_rate(float* scratch, int sms, double* tflops, cudaStream_t st) {
    const size_t smem = sizeof(float2) * 2 * 32 * kTile;
    cudaError_t e = cudaFuncSetAttribute(k_fw_inner_loop, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    const int grid = 2 * sms, reps = 200;
    cudaEvent_t e0, e1;
    if ((e = cudaEventCreate(&e0)) != cudaSuccess) return e;
    if ((e = cudaEventCreate(&e1)) != cudaSuccess) { cudaEventDestroy(e0); return e; }
    k_fw_inner_loop<<<grid, 256, smem, st>>>(scratch, reps);  // warm-up
    ++g_launch_counter;
    cudaEventRecord(e0, st);
    const int iters = 5;
    for (int k = 0; k < iters; ++k) {
        k_fw_inner_loop<<<grid, 256, smem, st>>>(scratch, reps);
        ++g_launch_counter;
    }
    cudaEventRecord(e1, st);
    e = cudaEventSynchronize(e1);
    float ms = 0.f;
    if (e == cudaSuccess) e = cudaEventElapsedTime(&ms, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (e != cudaSuccess) return e;
    // per thread and k-pair: 64 elements x 2 updates, each one add and one min
    const double ops = (double)grid * 256 * reps * 32 * 64 * 2 * 2 * iters;
    *tflops = ops / (ms * 1e-3) / 1e12;
    return cudaGetLastError();
}

__global__ void k_set_diag(float* __restrict__ S, const GraphInfo* __restrict__ graphs) {
    const GraphInfo g = graphs[blockIdx.y];
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < g.n) S[g.s_off + (int64_t)i * g.ld + i] = 0.f;
}

cudaError_t launch_set_diag(float* S, const GraphInfo* graphs, int n_graphs, int max_n,
                            cudaStream_t st) {
    if (n_graphs == 0 || max_n == 0) return cudaSuccess;
    k_set_diag<<<dim3((max_n + 255) / 256, n_graphs), 256, 0, st>>>(S, graphs);
    ++g_launch_counter;
    return cudaGetLastError();
}

}  // namespace lg
