// Dart throwing of the LightGraph points: LightGraph::scatterPoints
// (src/LightGraph.h:206-274), the caller-side step that feeds buildGraph.
//
// The reference throws, per iteration, up to scatterCount candidates in
// sequence: three draws of the iteration's mt19937 give a position in the
// active-voxel bbox; every scatterCount / nEstimates candidates the squared
// minimum distance is rescaled by pcSize / expectedSize (the expected sizes
// are computed on the host with the C library's pow, as the reference does);
// a candidate whose trilinear density is below the cutoff is skipped, one
// closer than the minimum distance to an accepted point is rejected, and the
// loop stops once more than targetSize points are accepted.
//
// Here one CTA, or a cluster, runs one iteration and reproduces that sequence
// exactly. A CTA takes the candidates a chunk at a time (3328 or 1664 of them),
// in ranges: a range is a chunk, or a part of one where a radius update falls
// inside it, so that the radius is one number in each range:
//   1. warps take groups of 64 candidates from a counter: position in FP32 index
//      space, one cell record, density test. A candidate whose density or
//      cell the FP32 error leaves undecided is tested again with an index
//      position of two floats, and if need be with the reference's arithmetic
//      (FP64 position, double weights, a float result per interpolation step).
//      Those that pass are tested against two accepted points: the ones that
//      last rejected candidates of the same hint cell (19 in 20 end here).
//      Meanwhile eight warps first make the next chunk's MT19937 words;
//   2. a warp per remaining candidate forms its position exactly as the
//      reference rounds it (position_exact) and tests it against the accepted
//      points in the cells of a kDartGrid^3 grid within the radius, a lane per
//      cell. A radius change needs no rebuilding: the cells hold positions
//      alone, and a hint is an accepted point wherever it is;
//   3. warp 0 walks the survivors in candidate order, testing each against
//      the points accepted in the same range, and accepts.
// Distances are compared in FP32 and re-tested in FP64 (the reference's
// arithmetic) when within 2^-18 of the squared radius, so the accepted set
// is the reference's. The accepted points live in shared memory.
//
// What bounds it: latency, the steps of a range one after the other with a
// barrier between (an iteration's ranges are a chain). Chunks of 208
// candidates (one state block) with every listed candidate tested against all
// accepted points by a warp and FP64 positions for every candidate took
// 44.6 ms for 48 iterations of 1M candidates (256^3 cumulus); this form takes
// 4.8 ms, and 500 iterations 16.4 ms instead of 76. Where there are SMs to
// spare a cluster runs an iteration (k_dart_cluster): words and density tests
// go ahead on the other CTAs, and the first one's hint tests beside the walk: 3.7 ms.
#include <algorithm>
#include <cmath>

#include "lg_kernels.h"
#include "lg_mt.h"

namespace lg {

namespace {

constexpr int kDartTwisters = 256;  // >= 227 threads that make the next words (the last eight warps)
constexpr int kDartGrid = 16;  // cells per axis over the points' bbox
constexpr int kDartHint = 20;  // hint cells per axis
constexpr uint16_t kNoPoint = 0xFFFFu;

// BoxSampler::sample restated as the reference evaluates it: float voxel
// values, double weights, each interpolation rounded to float (z, then y,
// then x). p is the index-space position.
__device__ __noinline__ float sample_exact(const DevGrid& g, double px, double py, double pz) {
    const double fx = floor(px), fy = floor(py), fz = floor(pz);
    const double u = px - fx, w = py - fy, t = pz - fz;
    float v[8];
    const int ix = (int)fx, iy = (int)fy, iz = (int)fz;
    if (g.dtype == 0) {
        // FP32 records hold the polynomial: each corner is the first entry
        // (the voxel itself) of its own cell's record
#pragma unroll
        for (int c = 0; c < 8; ++c) v[c] = voxel(g, ix + (c & 1), iy + ((c >> 1) & 1), iz + (c >> 2));
    } else {
        const uint32_t rec = cell_record(g, ix, iy, iz);
        if (g.dtype == 1) ld_cell<1>(g.data, rec, v);
        else ld_cell<2>(g.data, rec, v);
    }
    auto lerp = [](float a, float b, double wt) {
        const double tmp = __dmul_rn((double)__fsub_rn(b, a), wt);
        return __fadd_rn(a, __double2float_rn(tmp));
    };
    // v[a + 2b + 4c] = voxel (x + a, y + b, z + c)
    const float x0 = lerp(lerp(v[0], v[4], t), lerp(v[2], v[6], t), w);
    const float x1 = lerp(lerp(v[1], v[5], t), lerp(v[3], v[7], t), w);
    return lerp(x0, x1, u);
}

// The slow paths stay out of line: the kernel's steps are run in turn by every
// warp, so its code should fit the instruction cache.
__device__ __noinline__ float position_fp64(double bbmin, float x) {
    return __double2float_rn(__dadd_rn((double)x, bbmin));
}

// The candidate's coordinate as the reference rounds it,
// float(double(x) + bbmin) with x = float(u * size), for axis a. bbmin is
// hi + lo to within 2^-48 of itself; x + hi = s + e exactly (two-sum), and
// where s + (e + lo) rounds the same way after moving e + lo by more than
// every rounding left out, that is the answer. Otherwise FP64 decides (its
// additions and conversions run at 1/64 of the FP32 rate, which made them
// most of the time when every candidate used them).
__device__ __forceinline__ float position_exact(const DartParams& prm, int a, float x) {
    const float hi = prm.bb_hi[a];
    const float s = __fadd_rn(x, hi);
    const float bb = __fsub_rn(s, x);
    const float e = __fadd_rn(__fsub_rn(x, __fsub_rn(s, bb)), __fsub_rn(hi, bb));
    const float t = __fadd_rn(e, prm.bb_lo[a]);
    const float m = __fmaf_rn(fabsf(t), 2.384185791015625e-7f, prm.bb_err[a]);  // 2^-22
    const float r0 = __fadd_rn(s, __fsub_rn(t, m)), r1 = __fadd_rn(s, __fadd_rn(t, m));
    if (r0 == r1) return r0;
    return position_fp64(prm.bbmin[a], x);
}

// Position offsets from bbmin of the candidate whose three words are at w.
__device__ __forceinline__ void candidate_offsets(const DartParams& prm, const uint32_t* w, float x[3]) {
#pragma unroll
    for (int a = 0; a < 3; ++a) x[a] = __fmul_rn(mt_canonical_float(mt_temper(w[a])), prm.bbsize[a]);
}

// Its exact position.
__device__ __forceinline__ void candidate_position(const DartParams& prm, const uint32_t* w, float p[3]) {
    candidate_offsets(prm, w, p);
#pragma unroll
    for (int a = 0; a < 3; ++a) p[a] = position_exact(prm, a, p[a]);
}

// The cell record and weights under a candidate in FP32: index = x / h +
// (bbmin - wo) / h, off by at most prm.index_err voxels.
struct DartCell {
    float u, w, t;
    uint32_t rec;
};
__device__ __forceinline__ DartCell candidate_cell(const DevGrid& g, const DartParams& prm, const float x[3]) {
    const float ix = fmaf(x[0], prm.inv_h_f, prm.index0[0]), iy = fmaf(x[1], prm.inv_h_f, prm.index0[1]),
                iz = fmaf(x[2], prm.inv_h_f, prm.index0[2]);
    const float fx = floorf(ix), fy = floorf(iy), fz = floorf(iz);
    return {ix - fx, iy - fy, iz - fz, cell_record(g, (int)fx, (int)fy, (int)fz)};
}

__device__ __noinline__ float density_exact(const DevGrid& g, const DartParams& prm, float x, float y, float z) {
    const double px = ((double)position_fp64(prm.bbmin[0], x) - prm.wo[0]) / prm.h;
    const double py = ((double)position_fp64(prm.bbmin[1], y) - prm.wo[1]) / prm.h;
    const double pz = ((double)position_fp64(prm.bbmin[2], z) - prm.wo[2]) / prm.h;
    return sample_exact(g, px, py, pz);
}

// The density test in FP32: 0 fails, 1 passes, 2 undecided -- the value lies
// within its error bound of the cutoff or the position within twice its error
// of a cell face (where the exact position may sit in the neighbouring cell).
// Inside one cell the trilinear sample moves by at most 3 * (max tap - min
// tap) per voxel of position error index_err; the seven FP32 interpolations
// add under 2^-19 of the largest tap. For an FP32 record (the polynomial k0 +
// ...) S = sum of |k| over the non-constant terms stands in for the taps'
// spread: every partial derivative is at most S and every tap lies within S of
// k0, so |k0| + S bounds every tap; the coefficients' FP32 differences
// (54 * 2^-24 of the largest tap), their four evaluation steps and the exact
// sample's own roundings stay under 4e-6 of |k0| + S, and the bound takes twice
// that.
template <int DT>
__device__ __forceinline__ int density_test(const DartCell& c, const float v[8], float index_err, float cutoff) {
    float val, spread, mag, rel = 2e-6f;
    if (DT == 0) {
        rel = 8e-6f;
        val = trilinear_coefs(v, c.u, c.w, c.t);
        float sum = 0.f;
#pragma unroll
        for (int k = 1; k < 8; ++k) sum += fabsf(v[k]);
        spread = sum * (1.f + 1e-6f);
        mag = fabsf(v[0]) + spread;
    } else {
        float lo = v[0], hi = v[0];
#pragma unroll
        for (int k = 1; k < 8; ++k) { lo = fminf(lo, v[k]); hi = fmaxf(hi, v[k]); }
        auto lerp = [](float a, float b, float wt) { return fmaf(b - a, wt, a); };
        const float x0 = lerp(lerp(v[0], v[4], c.t), lerp(v[2], v[6], c.t), c.w);
        const float x1 = lerp(lerp(v[1], v[5], c.t), lerp(v[3], v[7], c.t), c.w);
        val = lerp(x0, x1, c.u);
        spread = hi - lo;
        mag = fmaxf(fabsf(hi), fabsf(lo));
    }
    const float e2 = 2.f * index_err;
    if (fminf(fminf(c.u, c.w), c.t) < e2 || fmaxf(fmaxf(c.u, c.w), c.t) > 1.f - e2) return 2;
    const float bound = 3.f * spread * index_err + mag * rel + 1e-30f;
    return val < cutoff - bound ? 0 : val > cutoff + bound ? 1 : 2;
}

// The same with the index position (p - wo) / h of the exact p carried as a
// sum of two floats, off by at most prm.index_err2 voxels: about one candidate
// in 700 comes here for lying near a cell face, one in a million is left for
// FP64, whose dependent steps at 1/64 of the FP32 rate made a whole range
// wait (48 iterations of 1M candidates: 7.7 ms with FP64 alone, 5.6 ms so).
template <int DT>
__device__ bool density_again(const DevGrid& g, const DartParams& prm, float x, float y, float z) {
    const float o[3] = {x, y, z};
    float f[3], w[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float p = position_exact(prm, a, o[a]);
        // p - wo = s + t (two-difference, then wo's second float)
        const float s = __fsub_rn(p, prm.wo_hi[a]);
        const float bb = __fsub_rn(p, s);
        const float e = __fadd_rn(__fsub_rn(p, __fadd_rn(s, bb)), __fsub_rn(bb, prm.wo_hi[a]));
        const float t = __fsub_rn(e, prm.wo_lo[a]);
        // times 1 / h = inv_h_f + inv_h_lo
        const float q = __fmul_rn(s, prm.inv_h_f);
        const float r = __fmaf_rn(t, prm.inv_h_f, __fmaf_rn(s, prm.inv_h_lo, __fmaf_rn(s, prm.inv_h_f, -q)));
        f[a] = floorf(q);
        w[a] = __fadd_rn(__fsub_rn(q, f[a]), r);  // outside [0, 1): undecided
    }
    const DartCell c = {w[0], w[1], w[2], cell_record(g, (int)f[0], (int)f[1], (int)f[2])};
    float v[8];
    ld_cell<DT>(g.data, c.rec, v);
    const int d = density_test<DT>(c, v, prm.index_err2, prm.cutoff);
    return d == 2 ? !(density_exact(g, prm, x, y, z) < prm.cutoff) : d == 1;
}

template <int DT>
__device__ __forceinline__ bool density_passes(const DevGrid& g, const DartParams& prm, const DartCell& c,
                                               const float v[8], const float x[3]) {
    const int d = density_test<DT>(c, v, prm.index_err, prm.cutoff);
    return d == 2 ? density_again<DT>(g, prm, x[0], x[1], x[2]) : d == 1;
}

// |a - b|^2 < m2 as the reference decides it (double arithmetic on float
// coordinates), with an FP32 fast path outside a 2^-18 relative band.
__device__ __noinline__ bool closer_fp64(float ax, float ay, float az, const float* b, float m2) {
    const double ex = __dsub_rn((double)ax, (double)b[0]);
    const double ey = __dsub_rn((double)ay, (double)b[1]);
    const double ez = __dsub_rn((double)az, (double)b[2]);
    const double e2 = __dadd_rn(__dadd_rn(__dmul_rn(ex, ex), __dmul_rn(ey, ey)), __dmul_rn(ez, ez));
    return e2 < (double)m2;
}
__device__ __forceinline__ bool closer(const float* a, const float* b, float m2) {
    const float dx = a[0] - b[0], dy = a[1] - b[1], dz = a[2] - b[2];
    const float d2 = dx * dx + dy * dy + dz * dz;
    if (d2 < m2 * (1.f - 3.814697265625e-6f)) return true;
    if (d2 > m2 * (1.f + 3.814697265625e-6f)) return false;
    return closer_fp64(a[0], a[1], a[2], b, m2);
}

// The next chunk's words nxt[0..kBlocks * 624) after this chunk's cur, a state
// block of 624 at a time. Word i of a block is made of the words 624, 623 and
// 227 before it, so thread t < 227 makes the words t, t + 227 and t + 454 (the
// last by 170 threads) from the block before and its own; only word 623 needs
// another, the block's first, and makes it for itself. The kDartTwisters
// threads that call it meet at barrier 1 after each block.
template <int kBlocks>
__device__ __forceinline__ void mt_next_chunk(const uint32_t* cur, uint32_t* nxt, int t) {
    const uint32_t* prev = cur + (kBlocks - 1) * kMtN;
#pragma unroll 1
    for (int k = 0; k < kBlocks; ++k) {
        uint32_t* out = nxt + k * kMtN;
        if (t < kMtN - kMtM) {
            const bool third = t < kMtN - 2 * (kMtN - kMtM);
            const uint32_t a0 = prev[t], b0 = prev[t + 1], c0 = prev[t + kMtM];
            const uint32_t a1 = prev[t + 227], b1 = prev[t + 228];
            uint32_t a2 = 0u, b2 = 0u;
            if (third) {
                a2 = prev[t + 454];
                b2 = t + 455 < kMtN ? prev[t + 455] : mt_twist_word(prev[0], prev[1], prev[kMtM]);
            }
            uint32_t x = mt_twist_word(a0, b0, c0);
            out[t] = x;
            x = mt_twist_word(a1, b1, x);
            out[t + 227] = x;
            if (third) out[t + 454] = mt_twist_word(a2, b2, x);
        }
        prev = out;
        __syncwarp();  // a warp has to arrive as a whole
        asm volatile("bar.sync 1, %0;" ::"n"(kDartTwisters) : "memory");
    }
}

// Cell coordinate along axis a, clamped to the grid; monotonic in x (every
// step rounds monotonically), so the points within r of x lie in the cells
// from that of x - r to that of x + r.
__device__ __forceinline__ int dart_cell(const DartParams& prm, int a, float x, float inv, int n) {
    return min(max((int)((x - prm.bb_hi[a]) * inv), 0), n - 1);
}
__device__ __forceinline__ int hint_cell(const DartParams& prm, const float p[3]) {
    return (dart_cell(prm, 2, p[2], prm.hint_inv[2], kDartHint) * kDartHint +
            dart_cell(prm, 1, p[1], prm.hint_inv[1], kDartHint)) *
               kDartHint +
           dart_cell(prm, 0, p[0], prm.hint_inv[0], kDartHint);
}

// The reference's radius update: minDist^2 *= pcSize / expectedSize, in
// double, rounded back to float.
__device__ __noinline__ void radius_update(float& m2, int pc, uint32_t expected) {
    const double ratio = (double)pc / (double)expected;
    m2 = __double2float_rn(__dmul_rn((double)m2, ratio));
}

// Whether one of the two points of the candidate's hint cell is certainly
// closer; x: its offsets from bbmin.
__device__ __forceinline__ bool hinted(const ushort2* hint, const float* acc, const DartParams& prm, const float x[3],
                                       float hint_m2) {
    const float p[3] = {x[0] + prm.bb_hi[0], x[1] + prm.bb_hi[1], x[2] + prm.bb_hi[2]};
    const ushort2 h = hint[hint_cell(prm, p)];
    auto near = [&](int q) {
        const float dx = p[0] - acc[3 * q], dy = p[1] - acc[3 * q + 1], dz = p[2] - acc[3 * q + 2];
        return dx * dx + dy * dy + dz * dz < hint_m2;
    };
    return (h.x != kNoPoint && near(h.x)) || (h.y != kNoPoint && near(h.y));
}

// Two warps may do this to one cell at once: whichever entries remain, each
// is an accepted point.
__device__ __forceinline__ void add_hint(ushort2& h, int q) { h = make_ushort2((unsigned short)q, h.x); }

// What an iteration keeps in shared memory from range to range, chunks of
// kCandidates. hard_limit x 3 floats (the accepted points) and hard_limit uint16
// (the next point of the same cell) stand behind the structure that holds it.
template <int kCandidates>
struct DartTables {
    static constexpr int kCand = kCandidates;
    static constexpr int kSurv = (kCand + 1023) / 1024 * 32;
    static_assert(kCand % 64 == 0, "groups of 64 are claimed");
    uint32_t surv[kSurv];  // survivors, a bit per candidate of the chunk
    uint16_t head[kDartGrid * kDartGrid * kDartGrid];
    ushort2 hint[kDartHint * kDartHint * kDartHint];  // the last two points found, the latest in x
    int pc, done;
    float m2, last;
};

// A CTA that runs an iteration by itself: kBlocks MT19937 state blocks a chunk.
template <int kBlocks>
struct DartShared : DartTables<kBlocks * kMtN / 3> {
    static constexpr int kWords = kBlocks * kMtN;
    uint32_t words[2][kWords];
    uint16_t queue[kWords / 3];  // candidates left by the hint test, in any order
    int claim, queued;
};

// The iteration's empty tables, by threads t of nt.
template <class Tables>
__device__ __forceinline__ void clear_tables(Tables& sh, const DartParams& prm, int t, int nt) {
    if (t == 0) {
        sh.pc = 0;
        sh.done = 0;
        sh.m2 = prm.min_dist_sq0;
        sh.last = prm.min_dist_sq0;
    }
#pragma unroll 1
    for (int k = t; k < kDartGrid * kDartGrid * kDartGrid; k += nt) sh.head[k] = kNoPoint;
#pragma unroll 1
    for (int k = t; k < kDartHint * kDartHint * kDartHint; k += nt) sh.hint[k] = make_ushort2(kNoPoint, kNoPoint);
    for (int k = t; k < Tables::kSurv; k += nt) sh.surv[k] = 0u;
}

// The seeded state of iteration it, one thread.
__device__ __forceinline__ void mt_seed(uint32_t* st, uint32_t seed) {
    uint32_t x = seed;
    st[0] = x;
#pragma unroll 1
    for (int k = 1; k < kMtN; ++k) {
        x = mt_init_word(x, (uint32_t)k);
        st[k] = x;
    }
}

// The radius that hint tests use: they take x + bbmin in plain FP32, off by
// less than cell_slack / 4 per axis, which moves a squared distance near m2 by
// less than root * cell_slack: below hint_m2 the exact test says the same, and
// whoever is not below it is left for the exact one.
__device__ __forceinline__ float hint_radius_sq(const DartParams& prm, float m2, float root) {
    return m2 * (1.f - 7.62939453125e-6f) - 2.f * prm.cell_slack * root;
}

// 1. Offsets and density tests of the candidates ja and ja + 32 of a chunk's
// words, as far as they lie in [j0, j1): both record loads are in flight
// together.
template <int DT>
__device__ __forceinline__ void density_tests(const DevGrid& g, const DartParams& prm, const uint32_t* words, int ja,
                                              int j0, int j1, float xa[3], float xb[3], bool& pa, bool& pb) {
    float va[8], vb[8];
    const int jb = ja + 32;
    candidate_offsets(prm, words + 3 * ja, xa);
    const DartCell ca = candidate_cell(g, prm, xa);
    ld_cell<DT>(g.data, ca.rec, va);
    candidate_offsets(prm, words + 3 * jb, xb);
    const DartCell cb = candidate_cell(g, prm, xb);
    ld_cell<DT>(g.data, cb.rec, vb);
    pa = ja >= j0 && ja < j1 && density_passes<DT>(g, prm, ca, va, xa);
    pb = jb >= j0 && jb < j1 && density_passes<DT>(g, prm, cb, vb, xb);
}

// 2. The accepted points near each of the nq candidates left by the hint test;
// lane k of a warp holds the position of its k-th. position(j, p): the exact
// position of the chunk's candidate j; r covers the radius and the rounding of
// x -+ r; p0: accepted points.
template <int kThreads, class Tables, class Position>
__device__ __forceinline__ void test_near(Tables& sh, const float* acc, const uint16_t* link, const DartParams& prm,
                                          const uint16_t* queue, int nq, const Position& position, int p0, float m2,
                                          float r) {
    constexpr int kWarps = kThreads / 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll 1
    for (int e0 = 0; e0 < nq; e0 += kThreads) {
        const int e = e0 + warp + kWarps * lane;
        int jj = 0;
        float p[3] = {0.f, 0.f, 0.f};
        if (e < nq) {
            jj = queue[e];
            position(jj, p);
        }
        const int mine = __popc(__ballot_sync(0xffffffffu, e < nq));
#pragma unroll 1
        for (int k = 0; k < mine; ++k) {
            const float q[3] = {__shfl_sync(0xffffffffu, p[0], k), __shfl_sync(0xffffffffu, p[1], k),
                                __shfl_sync(0xffffffffu, p[2], k)};
            const int jk = __shfl_sync(0xffffffffu, jj, k);
            int lo[3], hi[3];
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                lo[a] = dart_cell(prm, a, q[a] - r, prm.cell_inv[a], kDartGrid);
                hi[a] = dart_cell(prm, a, q[a] + r, prm.cell_inv[a], kDartGrid);
            }
            const int cells = (hi[0] - lo[0] + 1) * (hi[1] - lo[1] + 1) * (hi[2] - lo[2] + 1);
            unsigned hits = 0u;
            int near = 0;
            if (cells >= p0) {  // few points yet: all of them
#pragma unroll 1
                for (int i0 = 0; i0 < p0 && !hits; i0 += 32) {
                    near = i0 + lane;
                    hits = __ballot_sync(0xffffffffu, near < p0 && closer(q, acc + 3 * near, m2));
                }
            } else {
                // 4 x 4 x 2 cells at a time, a lane each
                const int lx = lane & 3, ly = (lane >> 2) & 3, lz = lane >> 4;
#pragma unroll 1
                for (int z = lo[2]; z <= hi[2] && !hits; z += 2)
#pragma unroll 1
                    for (int y = lo[1]; y <= hi[1] && !hits; y += 4)
#pragma unroll 1
                        for (int x = lo[0]; x <= hi[0] && !hits; x += 4) {
                            bool h = false;
                            if (x + lx <= hi[0] && y + ly <= hi[1] && z + lz <= hi[2]) {
                                near = sh.head[((z + lz) * kDartGrid + y + ly) * kDartGrid + x + lx];
                                while (near != kNoPoint && !(h = closer(q, acc + 3 * near, m2))) near = link[near];
                            }
                            hits = __ballot_sync(0xffffffffu, h);
                        }
            }
            if (hits) {
                if (lane == __ffs(hits) - 1) add_hint(sh.hint[hint_cell(prm, q)], near);
            } else if (lane == 0) {
                atomicOr(&sh.surv[jk >> 5], 1u << (jk & 31));
            }
        }
    }
}

// 3. The walk by one warp over the survivors in candidate order.
template <class Tables, class Position>
__device__ __forceinline__ void walk(Tables& sh, float* acc, uint16_t* link, const DartParams& prm,
                                     const Position& position, int p0, float m2) {
    const int lane = threadIdx.x & 31;
    int pc = p0;
    bool done = false;
    float last = sh.last;
#pragma unroll 1
    for (int half = 0; half < Tables::kSurv && !done; half += 32) {
        const uint32_t mine = sh.surv[half + lane];
        sh.surv[half + lane] = 0u;
        unsigned some = __ballot_sync(0xffffffffu, mine != 0u);
        while (some && !done) {
            const int k = __ffs(some) - 1;
            some &= some - 1;
            uint32_t bits = __shfl_sync(0xffffffffu, mine, k);
            float p[3] = {0.f, 0.f, 0.f};
            if ((bits >> lane) & 1u) position(32 * (half + k) + lane, p);
            while (bits && !done) {
                const int b = __ffs(bits) - 1;
                bits &= bits - 1;
                const float q[3] = {__shfl_sync(0xffffffffu, p[0], b), __shfl_sync(0xffffffffu, p[1], b),
                                    __shfl_sync(0xffffffffu, p[2], b)};
                bool h = false;
                for (int i0 = p0; i0 < pc && !h; i0 += 32)
                    h = __any_sync(0xffffffffu, i0 + lane < pc && closer(q, acc + 3 * (i0 + lane), m2));
                if (h) continue;
                if (lane == 0) {
                    acc[3 * pc] = q[0];
                    acc[3 * pc + 1] = q[1];
                    acc[3 * pc + 2] = q[2];
                    const int c = (dart_cell(prm, 2, q[2], prm.cell_inv[2], kDartGrid) * kDartGrid +
                                   dart_cell(prm, 1, q[1], prm.cell_inv[1], kDartGrid)) *
                                      kDartGrid +
                                  dart_cell(prm, 0, q[0], prm.cell_inv[0], kDartGrid);
                    link[pc] = sh.head[c];
                    sh.head[c] = (uint16_t)pc;
                    // hint tests of the next range may run meanwhile
                    __threadfence_block();
                    add_hint(sh.hint[hint_cell(prm, q)], pc);
                }
                __syncwarp();
                ++pc;
                last = m2;
                // the reference stops at the next candidate once
                // more than target points are accepted
                done = pc > (int)prm.target || pc >= (int)prm.hard_limit;
            }
        }
    }
    if (lane == 0) {
        sh.pc = pc;
        sh.last = last;
        sh.done = done;
    }
}

template <int DT, int kThreads, int kBlocks>
__global__ void __launch_bounds__(kThreads, 1024 / kThreads) k_dart(DevGrid g, DartParams prm, const uint32_t* __restrict__ expected,
                                                                    float* __restrict__ out_pts,
                                                                    int32_t* __restrict__ out_count,
                                                                    float* __restrict__ out_last_m2) {
    static_assert(kThreads > kDartTwisters && kThreads <= 1024, "the last warps make the next words");
    using Shared = DartShared<kBlocks>;
    extern __shared__ __align__(16) uint8_t dart_smem[];
    Shared& sh = *reinterpret_cast<Shared*>(dart_smem);
    float* acc = reinterpret_cast<float*>(dart_smem + sizeof(Shared));
    uint16_t* link = reinterpret_cast<uint16_t*>(acc + 3 * prm.hard_limit);

    const int it = prm.first_iter + (int)blockIdx.x;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) {
        // the seeded state stands before the first chunk
        mt_seed(sh.words[1] + Shared::kWords - kMtN, prm.seed_base + (uint32_t)it);
        sh.claim = 0;
        sh.queued = 0;
    } else {
        clear_tables(sh, prm, tid - 1, kThreads - 1);
    }
    __syncthreads();
    const int twister = tid - (kThreads - kDartTwisters);
    if (twister >= 0) mt_next_chunk<kBlocks>(sh.words[1], sh.words[0], twister);
    // candidate n updates the radius before its tests when (n + 1) % batch == 0:
    // the next such n, and which update it is
    uint64_t boundary = prm.batch - 1u;
    uint32_t update = 0;
    if (tid == 0 && boundary == 0u) radius_update(sh.m2, 0, expected[0]);
    __syncthreads();
    uint64_t chunk = 0, n0 = 0;  // first candidates of the chunk and of the range
    int buf = 0;
    while (n0 < prm.scatter_count) {
        if (n0 == boundary) {  // its update was made where the last range ended
            boundary += prm.batch;
            ++update;
        }
        const uint32_t* cur = sh.words[buf];
        const uint64_t chunk_end = min(chunk + (uint64_t)Shared::kCand, (uint64_t)prm.scatter_count);
        const uint64_t n1 = min(chunk_end, boundary);
        const int j0 = (int)(n0 - chunk), j1 = (int)(n1 - chunk);
        const int p0 = sh.pc;
        const float m2 = sh.m2;
        // r covers sqrt(m2) and the rounding of x -+ r
        const float root = sqrtf(m2), r = fmaf(root, 1.00001f, prm.cell_slack);
        // 1. the next chunk's words; density and hint tests
        if (twister >= 0 && j0 == 0 && chunk_end < prm.scatter_count)
            mt_next_chunk<kBlocks>(cur, sh.words[buf ^ 1], twister);
        const float hint_m2 = hint_radius_sq(prm, m2, root);
        for (;;) {
            int j = 0;
            if (lane == 0) j = atomicAdd(&sh.claim, 64);
            j = __shfl_sync(0xffffffffu, j, 0) + (j0 & ~63);
            if (j >= j1) break;
            float xa[3], xb[3];
            bool pa, pb;
            const int ja = j + lane, jb = ja + 32;
            density_tests<DT>(g, prm, cur, ja, j0, j1, xa, xb, pa, pb);
            const bool la = pa && !hinted(sh.hint, acc, prm, xa, hint_m2), lb = pb && !hinted(sh.hint, acc, prm, xb, hint_m2);
            const unsigned ma = __ballot_sync(0xffffffffu, la), mb = __ballot_sync(0xffffffffu, lb);
            if ((ma | mb) == 0u) continue;
            const unsigned below = (1u << lane) - 1u;
            int at = 0;
            if (lane == 0) at = atomicAdd(&sh.queued, __popc(ma) + __popc(mb));
            at = __shfl_sync(0xffffffffu, at, 0);
            if (la) sh.queue[at + __popc(ma & below)] = (uint16_t)ja;
            if (lb) sh.queue[at + __popc(ma) + __popc(mb & below)] = (uint16_t)jb;
        }
        __syncthreads();
        // 2.
        const auto position = [&](int j, float p[3]) { candidate_position(prm, cur + 3 * j, p); };
        test_near<kThreads>(sh, acc, link, prm, sh.queue, sh.queued, position, p0, m2, r);
        __syncthreads();
        // 3.
        if (warp == 0) {
            walk(sh, acc, link, prm, position, p0, m2);
            if (lane == 0) {
                sh.claim = 0;
                sh.queued = 0;
                if (n1 == boundary && n1 < prm.scatter_count) radius_update(sh.m2, sh.pc, expected[update]);
            }
        }
        __syncthreads();
        if (sh.done) break;
        n0 = n1;
        if (n1 == chunk_end) {
            chunk = n1;
            buf ^= 1;
        }
    }
    const int pc = sh.pc;
    float* dst = out_pts + (size_t)blockIdx.x * prm.hard_limit * 3;
    for (int k = tid; k < 3 * pc; k += kThreads) dst[k] = acc[k];
    if (tid == 0) {
        out_count[blockIdx.x] = pc;
        out_last_m2[blockIdx.x] = sh.last;
    }
}

// ---------------------------------------------------------------------------
// An iteration on a cluster: its first CTA takes the ranges in turn, the others
// make the words and the density tests of the chunks ahead, which need nothing
// of what was accepted.
// ---------------------------------------------------------------------------

constexpr int kDartChunk = 16 * kMtN / 3;  // candidates a chunk
constexpr int kDartSlots = 3;              // chunks between the helpers and the first CTA

// First CTA. A slot holds the offsets of the candidates that passed and a bit
// for each; ready: the number of the chunk in it, plus one.
struct DartFirst : DartTables<kDartChunk> {
    float x[kDartSlots][3][kDartChunk];
    uint32_t bits[kDartSlots][kDartChunk / 32];
    uint32_t ready[kDartSlots];
    int queued[2];
    uint16_t queue[2][kDartChunk];
};
// Helpers. used: chunks that the first CTA is done with.
struct DartHelper {
    uint32_t words[3][16 * kMtN];
    uint32_t used, stop;
    int claim[2];
};

__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
// p's address in the shared memory of another CTA of the cluster.
__device__ __forceinline__ uint32_t remote(const void* p, uint32_t rank) {
    uint32_t a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
    return a;
}
__device__ __forceinline__ void remote_store(uint32_t at, uint32_t v) {
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(at), "r"(v) : "memory");
}
// Everything this thread wrote or saw written comes before v for whoever
// acquires v.
__device__ __forceinline__ void remote_release(uint32_t at, uint32_t v) {
    asm volatile("fence.acq_rel.cluster;\n\tst.release.cluster.shared::cluster.u32 [%0], %1;" ::"r"(at), "r"(v) : "memory");
}
__device__ __forceinline__ uint32_t acquire(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.acquire.cluster.shared::cta.u32 %0, [%1];"
                 : "=r"(v)
                 : "r"((uint32_t)__cvta_generic_to_shared(p))
                 : "memory");
    return v;
}
// The warp waits until *p has reached v, or until *stop is set; false then or
// after `polls` looks.
__device__ __forceinline__ bool wait_for(const uint32_t* p, uint32_t v, const uint32_t* stop, uint32_t polls) {
    int ok = 0;
    if ((threadIdx.x & 31) == 0)
        for (uint32_t k = 0; k < polls && !(stop && acquire(stop)); ++k)
            if (acquire(p) >= v) {
                ok = 1;
                break;
            }
    ok = __shfl_sync(0xffffffffu, ok, 0);
    __syncwarp();
    return ok != 0;
}

// Helper h of n: chunks h, h + n, ... of the words, three buffers of them since
// the words after a chunk are made while it is tested, n chunks at a time.
template <int DT>
__device__ __forceinline__ void dart_helper(const DevGrid& g, const DartParams& prm, uint8_t* smem, int it, int h, int n) {
    DartHelper& sh = *reinterpret_cast<DartHelper*>(smem);
    DartFirst& first = *reinterpret_cast<DartFirst*>(smem);  // its addresses, in the first CTA
    const int tid = threadIdx.x, lane = tid & 31, twister = tid - (1024 - kDartTwisters);
    if (tid == 0) {
        mt_seed(sh.words[2] + 15 * kMtN, prm.seed_base + (uint32_t)it);
        sh.used = 0;
        sh.stop = 0;
        sh.claim[0] = sh.claim[1] = 0;
    }
    cluster_sync();
    int buf = 2;
    if (twister >= 0)
        for (int k = 0; k <= h; ++k) mt_next_chunk<16>(sh.words[(buf + k) % 3], sh.words[(buf + k + 1) % 3], twister);
    buf = (buf + h + 1) % 3;
    __syncthreads();
    const uint32_t chunks = (uint32_t)(((uint64_t)prm.scatter_count + kDartChunk - 1) / kDartChunk);
    int par = 0;
    for (uint32_t c = (uint32_t)h; c < chunks; c += n, par ^= 1) {
        const uint32_t* cur = sh.words[buf];
        const int len = (int)min((uint32_t)kDartChunk, prm.scatter_count - c * kDartChunk);
        if (twister >= 0 && c + n < chunks)
            for (int k = 0; k < n; ++k) mt_next_chunk<16>(sh.words[(buf + k) % 3], sh.words[(buf + k + 1) % 3], twister);
        const int slot = c % kDartSlots;
        const bool free = c < kDartSlots || wait_for(&sh.used, c + 1 - kDartSlots, &sh.stop, prm.polls);
        while (free) {
            int j = 0;
            if (lane == 0) j = atomicAdd(&sh.claim[par], 64);
            j = __shfl_sync(0xffffffffu, j, 0);
            if (j >= len) break;
            float xa[3], xb[3];
            bool pa, pb;
            density_tests<DT>(g, prm, cur, j + lane, 0, len, xa, xb, pa, pb);
            const unsigned ma = __ballot_sync(0xffffffffu, pa), mb = __ballot_sync(0xffffffffu, pb);
            if (lane < 2) remote_store(remote(&first.bits[slot][(j >> 5) + lane], 0), lane ? mb : ma);
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                const uint32_t at = remote(&first.x[slot][a][j + lane], 0);
                if (pa) remote_store(at, __float_as_uint(xa[a]));
                if (pb) remote_store(at + 32 * sizeof(float), __float_as_uint(xb[a]));
            }
        }
        asm volatile("fence.acq_rel.cluster;" ::: "memory");
        // all warps leave in the same round: the barrier itself carries the word,
        // since a flag could be set for the next round while some still read it
        if (__syncthreads_or(!free)) break;
        if (tid == 0) {
            sh.claim[par] = 0;  // used again in the chunk after next
            remote_release(remote(&first.ready[slot], 0), c + 1);
        }
        buf = (buf + n) % 3;
    }
}

template <int DT>
__global__ void __launch_bounds__(1024, 1) k_dart_cluster(DevGrid g, DartParams prm, int ctas,
                                                          const uint32_t* __restrict__ expected,
                                                          float* __restrict__ out_pts, int32_t* __restrict__ out_count,
                                                          float* __restrict__ out_last_m2) {
    extern __shared__ __align__(16) uint8_t dart_smem[];
    const int iter = (int)blockIdx.x / ctas, it = prm.first_iter + iter;
    const int rank = (int)cluster_rank();
    if (rank > 0) {
        dart_helper<DT>(g, prm, dart_smem, it, rank - 1, ctas - 1);
        cluster_sync();  // the first CTA may still write used and stop
        return;
    }
    DartFirst& sh = *reinterpret_cast<DartFirst*>(dart_smem);
    DartHelper& helper = *reinterpret_cast<DartHelper*>(dart_smem);  // its addresses, in the helpers
    float* acc = reinterpret_cast<float*>(dart_smem + sizeof(DartFirst));
    uint16_t* link = reinterpret_cast<uint16_t*>(acc + 3 * prm.hard_limit);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    clear_tables(sh, prm, tid, 1024);
    if (tid < kDartSlots) sh.ready[tid] = 0;
    if (tid < 2) sh.queued[tid] = 0;
    bool failed = false;  // a helper did not answer; the same in every thread
    uint64_t boundary = prm.batch - 1u;
    uint32_t update = 0;
    if (tid == 0 && boundary == 0u) radius_update(sh.m2, 0, expected[0]);
    cluster_sync();
    // the hint tests of candidates [j0, j1) of the slot with chunk c, by the
    // warps w of nw: those left go to the queue; false if the chunk did not come
    auto hint_tests = [&](uint32_t c, int j0, int j1, float hint_m2, int queue, int w, int nw) {
        const int slot = c % kDartSlots;
        if (!wait_for(&sh.ready[slot], c + 1, nullptr, prm.polls)) return false;
        for (int k = (j0 >> 5) + w; 32 * k < j1; k += nw) {
            const int j = 32 * k + lane;
            const bool in = ((sh.bits[slot][k] >> lane) & 1u) && j >= j0 && j < j1;
            float x[3] = {0.f, 0.f, 0.f};
            if (in) {
#pragma unroll
                for (int a = 0; a < 3; ++a) x[a] = sh.x[slot][a][j];
            }
            const bool left = in && !hinted(sh.hint, acc, prm, x, hint_m2);
            const unsigned m = __ballot_sync(0xffffffffu, left);
            if (m == 0u) continue;
            int at = 0;
            if (lane == 0) at = atomicAdd(&sh.queued[queue], __popc(m));
            at = __shfl_sync(0xffffffffu, at, 0);
            if (left) sh.queue[queue][at + __popc(m & ((1u << lane) - 1u))] = (uint16_t)j;
        }
        return true;
    };
    uint64_t n0 = 0;
    uint32_t c = 0;
    int queue = 0;
    bool tested = false;  // the range's hint tests ran during the last one's walk
    while (n0 < prm.scatter_count) {
        if (n0 == boundary) {  // its update was made where the last range ended
            boundary += prm.batch;
            ++update;
        }
        const uint64_t chunk = (uint64_t)c * kDartChunk;
        const uint64_t chunk_end = min(chunk + kDartChunk, (uint64_t)prm.scatter_count);
        const uint64_t n1 = min(chunk_end, boundary);
        const int p0 = sh.pc;
        const float m2 = sh.m2;
        const float root = sqrtf(m2), r = fmaf(root, 1.00001f, prm.cell_slack);
        const float hint_m2 = hint_radius_sq(prm, m2, root);
        if (!tested) {
            failed = __syncthreads_or(!hint_tests(c, (int)(n0 - chunk), (int)(n1 - chunk), hint_m2, queue, warp, 32));
            if (failed) break;
        }
        const auto position = [&](int j, float p[3]) {
#pragma unroll
            for (int a = 0; a < 3; ++a) p[a] = position_exact(prm, a, sh.x[c % kDartSlots][a][j]);
        };
        test_near<1024>(sh, acc, link, prm, sh.queue[queue], sh.queued[queue], position, p0, m2, r);
        __syncthreads();
        // the walk, and beside it the next range's hint tests if they use the
        // same radius: a hint seen early or late is an accepted point
        const bool more = n1 < prm.scatter_count;
        tested = more && n1 != boundary;
        bool came = true;
        if (warp == 0) {
            walk(sh, acc, link, prm, position, p0, m2);
            if (lane == 0) {
                sh.queued[queue] = 0;
                if (n1 == boundary && more) radius_update(sh.m2, sh.pc, expected[update]);
            }
        } else if (tested) {
            const uint64_t next_end = min(min(n1 + kDartChunk, (uint64_t)prm.scatter_count), boundary);
            came = hint_tests(c + 1, 0, (int)(next_end - n1), hint_m2, queue ^ 1, warp - 1, 31);
        }
        failed = __syncthreads_or(!came);
        if (failed || sh.done) break;
        if (tested) queue ^= 1;
        n0 = n1;
        if (n1 == chunk_end) {
            ++c;
            if (tid > 0 && tid < ctas) remote_release(remote(&helper.used, tid), c);
        }
    }
    if (tid > 0 && tid < ctas) remote_release(remote(&helper.stop, tid), 1u);
    const int pc = sh.pc;
    float* dst = out_pts + (size_t)iter * prm.hard_limit * 3;
    for (int k = tid; k < 3 * pc; k += 1024) dst[k] = acc[k];
    if (tid == 0) {
        out_count[iter] = failed ? -1 : pc;
        out_last_m2[iter] = sh.last;
    }
    cluster_sync();  // helpers may still write slots
}

size_t points_smem(const DartParams& prm) { return (3 * sizeof(float) + sizeof(uint16_t)) * (size_t)prm.hard_limit; }

template <int DT, int kThreads, int kBlocks>
cudaError_t launch_dart_t(const DevGrid& g, const DartParams& prm, int n_iter, const uint32_t* expected, float* out_pts,
                          int32_t* out_count, float* out_last_m2, cudaStream_t st) {
    const size_t smem = sizeof(DartShared<kBlocks>) + points_smem(prm);
    const cudaError_t e = raise_smem_limit(reinterpret_cast<const void*>(k_dart<DT, kThreads, kBlocks>));
    if (e != cudaSuccess) return e;
    k_dart<DT, kThreads, kBlocks><<<n_iter, kThreads, smem, st>>>(g, prm, expected, out_pts, out_count, out_last_m2);
    ++g_launch_counter;
    return cudaGetLastError();
}

template <int DT>
cudaError_t launch_dart_cluster(const DevGrid& g, const DartParams& prm, int n_iter, const uint32_t* expected,
                                float* out_pts, int32_t* out_count, float* out_last_m2, cudaStream_t st, bool& done) {
    const auto kernel = k_dart_cluster<DT>;
    done = false;
    const size_t smem = std::max(sizeof(DartFirst) + points_smem(prm), sizeof(DartHelper));
    if (smem > 227 * 1024) return cudaSuccess;
    cudaError_t e = raise_smem_limit(reinterpret_cast<const void*>(kernel));
    if (e != cudaSuccess) return e;
    for (int ctas = 3; ctas > 1; --ctas) {
        cudaLaunchAttribute attr = {};
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = ctas;
        attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(n_iter * ctas);
        cfg.blockDim = dim3(1024);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = st;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
        int most = 0;
        if ((e = cudaOccupancyMaxActiveClusters(&most, kernel, &cfg)) != cudaSuccess) return e;
        if (n_iter > most) continue;
        done = true;
        e = cudaLaunchKernelEx(&cfg, kernel, g, prm, ctas, expected, out_pts, out_count, out_last_m2);
        ++g_launch_counter;
        return e == cudaSuccess ? cudaGetLastError() : e;
    }
    return cudaSuccess;
}

}  // namespace

cudaError_t launch_dart(const DevGrid& g, DartParams prm, int n_iter, const uint32_t* expected, float* out_pts,
                        int32_t* out_count, float* out_last_m2, cudaStream_t st) {
    if (n_iter <= 0) return cudaSuccess;
    float extent = 0.f;
    for (int a = 0; a < 3; ++a) {
        prm.bb_hi[a] = (float)prm.bbmin[a];
        prm.bb_lo[a] = (float)(prm.bbmin[a] - (double)prm.bb_hi[a]);
        // what position_exact leaves out besides the rounding of e + lo: the
        // part of bbmin below hi + lo and the double sum's own rounding
        prm.bb_err[a] = (float)((std::fabs(prm.bbmin[a]) + (double)prm.bbsize[a]) * 1.4210854715202004e-14);  // 2^-46
        prm.wo_hi[a] = (float)prm.wo[a];
        prm.wo_lo[a] = (float)(prm.wo[a] - (double)prm.wo_hi[a]);
        prm.cell_inv[a] = (float)kDartGrid / prm.bbsize[a];
        prm.hint_inv[a] = (float)kDartHint / prm.bbsize[a];
        extent = std::max(extent, std::fabs(prm.bb_hi[a]) + prm.bbsize[a]);
    }
    prm.inv_h_lo = (float)(1.0 / prm.h - (double)prm.inv_h_f);
    prm.cell_slack = extent * 1e-6f;
    // Clusters of three CTAs, or two, as long as all run at once (24 iterations:
    // 4.6 -> 3.0 ms, 48: 4.8 -> 3.7 ms). As long as every iteration gets an SM of its own, the chain of its ranges
    // is what takes the time: 1024 threads and chunks of 3328 candidates shorten
    // it; past that, two CTAs of 512 threads with chunks of 1664 on an SM fill
    // each other's waits.
    int sms = 0, dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    auto go = [&](auto launch) { return launch(g, prm, n_iter, expected, out_pts, out_count, out_last_m2, st); };
    if (n_iter <= sms / 2) {
        bool done = false;
        auto clustered = [&](auto launch) {
            return launch(g, prm, n_iter, expected, out_pts, out_count, out_last_m2, st, done);
        };
        e = g.dtype == 1   ? clustered(launch_dart_cluster<1>)
            : g.dtype == 2 ? clustered(launch_dart_cluster<2>)
                           : clustered(launch_dart_cluster<0>);
        if (e != cudaSuccess || done) return e;
    }
    if (n_iter <= sms)
        return g.dtype == 1   ? go(launch_dart_t<1, 1024, 16>)
               : g.dtype == 2 ? go(launch_dart_t<2, 1024, 16>)
                              : go(launch_dart_t<0, 1024, 16>);
    return g.dtype == 1   ? go(launch_dart_t<1, 512, 8>)
           : g.dtype == 2 ? go(launch_dart_t<2, 512, 8>)
                          : go(launch_dart_t<0, 512, 8>);
}

}  // namespace lg
