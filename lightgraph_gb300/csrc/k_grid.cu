// Grid upload into the device brick layout, and the environment-map CDFs.
//
// Grids: a dense box of voxels (what a FloatGrid's active region looks like
// once copied to a dense array) is re-tiled into 8^3 bricks with one brick of
// zero padding on every side; every cell of the bricks stores the eight
// values of its trilinear footprint as one record, in FP32, FP16 or BF16.
// The leaf bitmap marks the bricks that are leaves of the VDB tree: given
// explicitly, or "any voxel non-zero" (a dense grid converted to a VDB keeps
// exactly those).
//
// Environment map: EnvLight's constructor (src/Light.h:150-177) weights each
// texel's luminance by sin(theta) and builds a Distribution2D
// (src/Sampling.h:128-167): per-row Distribution1D CDFs and a marginal CDF
// over the rows' integrals (src/Sampling.h:76-93). The prefix sums run in
// FP64 on the device (the reference uses FP32) and are stored as FP32.
#include <climits>

#include "lg_kernels.h"

namespace lg {

// Raises a bound that another block may have raised already.
__device__ __forceinline__ void lower_to(int* p, int v) {
    if (v < *reinterpret_cast<volatile int*>(p)) atomicMin(p, v);
}
__device__ __forceinline__ void raise_to(int* p, int v) {
    if (v > *reinterpret_cast<volatile int*>(p)) atomicMax(p, v);
}

// One CTA per brick of the box, padding included, two cells a thread: the
// brick's 9^3 voxels of the dense staging array (0 outside it) go to shared
// memory, every cell's eight of them become its record, and the brick's bits
// of the two bitmaps (cleared beforehand) and the two bounding boxes follow
// from the same voxels:
//   leafbits : the brick is a leaf (its leaf_mask entry, or without a mask any
//              voxel non-zero);
//   occbits  : some voxel of the brick is non-zero;
//   bbox     : {min x, y, z, max x, y, z} of the leaf bricks' coordinates, then
//              of the non-zero voxels in the array's own coordinates, preset to
//              +/-INT_MAX.
// Bound by the records written, 32 or 16 bytes a cell, and with 16 by the
// latency of a brick's steps: 512^3 in FP32 1.02 ms (4.7 GB: 4.6 TB/s), 192^3 61
// us. A kernel each for records, leaves and voxels read the array eight times,
// once and once: 1.06 + 0.13 + 2.38 ms and 66 + 56 + 146 us.
template <int DT>
__global__ void __launch_bounds__(256) k_pack_volume(const float* __restrict__ dense, int dx, int dy, int dz, int ox,
                                                     int oy, int oz, const uint8_t* __restrict__ leaf_mask, DevGrid g,
                                                     void* __restrict__ bricks, uint32_t* __restrict__ leafbits,
                                                     uint32_t* __restrict__ occbits, int* __restrict__ bbox) {
    __shared__ float tile[9 * 9 * 9];
    __shared__ uint32_t seen[8];
    const uint32_t b = blockIdx.x;
    const int tid = threadIdx.x;
    const int bx = (int)(b % (uint32_t)g.nb[0]), by = (int)((b / (uint32_t)g.nb[0]) % (uint32_t)g.nb[1]),
              bz = (int)(b / ((uint32_t)g.nb[0] * (uint32_t)g.nb[1]));
    const int x0 = (g.blo[0] + bx) * 8 - ox, y0 = (g.blo[1] + by) * 8 - oy, z0 = (g.blo[2] + bz) * 8 - oz;
    for (int i = tid; i < 9 * 9 * 9; i += 256) {
        const int x = x0 + i % 9, y = y0 + (i / 9) % 9, z = z0 + i / 81;
        tile[i] = ((unsigned)x < (unsigned)dx && (unsigned)y < (unsigned)dy && (unsigned)z < (unsigned)dz)
                      ? dense[((int64_t)z * dy + y) * dx + x]
                      : 0.f;
    }
    __syncthreads();
    uint32_t m = 0u;  // bits of the x, y and z places that hold a non-zero voxel
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int l = tid + 256 * h, x = l & 7, y = (l >> 3) & 7, z = l >> 6;
        float v[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) v[c] = tile[(z + (c >> 2)) * 81 + (y + ((c >> 1) & 1)) * 9 + x + (c & 1)];
        if (v[0] != 0.f) m |= (1u << x) | (1u << (8 + y)) | (1u << (16 + z));
        const int64_t t = (int64_t)b * 512 + l;
        if (DT == 0) {
            // FP32 records hold the cell's trilinear polynomial (cell_coefs)
            float c[8];
            cell_coefs(v, c);
            asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(
                             reinterpret_cast<float*>(bricks) + 8 * t),
                         "f"(c[0]), "f"(c[1]), "f"(c[2]), "f"(c[3]), "f"(c[4]), "f"(c[5]), "f"(c[6]), "f"(c[7])
                         : "memory");
        } else {
            uint32_t w[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                if (DT == 1) {
                    const __half2 q = __floats2half2_rn(v[2 * i], v[2 * i + 1]);
                    w[i] = *reinterpret_cast<const uint32_t*>(&q);
                } else {
                    const __nv_bfloat162 q = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
                    w[i] = *reinterpret_cast<const uint32_t*>(&q);
                }
            }
            reinterpret_cast<uint4*>(bricks)[t] = make_uint4(w[0], w[1], w[2], w[3]);
        }
    }
    m = __reduce_or_sync(0xffffffffu, m);
    if ((tid & 31) == 0) seen[tid >> 5] = m;
    __syncthreads();
    if (tid != 0) return;
#pragma unroll
    for (int w = 1; w < 8; ++w) m |= seen[w];
    const int cx = g.blo[0] + bx, cy = g.blo[1] + by, cz = g.blo[2] + bz;
    bool leaf = m != 0u;
    if (leaf_mask) {
        // leaf coordinates relative to the dense box (origin is leaf aligned)
        const int lx = cx - (ox >> 3), ly = cy - (oy >> 3), lz = cz - (oz >> 3);
        const int lnx = (dx + 7) >> 3, lny = (dy + 7) >> 3, lnz = (dz + 7) >> 3;
        leaf = (unsigned)lx < (unsigned)lnx && (unsigned)ly < (unsigned)lny && (unsigned)lz < (unsigned)lnz &&
               leaf_mask[((int64_t)lz * lny + ly) * lnx + lx] != 0;
    }
    const uint32_t lin = ((uint32_t)(bz + 1) * (uint32_t)g.lby + (uint32_t)(by + 1)) * (uint32_t)g.lbx + (uint32_t)(bx + 1);
    if (leaf) {
        atomicOr(leafbits + (lin >> 5), 1u << (lin & 31u));
        lower_to(bbox + 0, cx);
        lower_to(bbox + 1, cy);
        lower_to(bbox + 2, cz);
        raise_to(bbox + 3, cx);
        raise_to(bbox + 4, cy);
        raise_to(bbox + 5, cz);
    }
    if (m) {
        atomicOr(occbits + (lin >> 5), 1u << (lin & 31u));
        const uint32_t ax[3] = {m & 0xFFu, (m >> 8) & 0xFFu, (m >> 16) & 0xFFu};
        const int at[3] = {x0, y0, z0};
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            lower_to(bbox + 6 + a, at[a] + __ffs(ax[a]) - 1);
            raise_to(bbox + 9 + a, at[a] + 31 - __clz(ax[a]));
        }
    }
}

cudaError_t launch_pack_volume(const float* dense, const int dims[3], const int origin[3], const uint8_t* leaf_mask,
                               const DevGrid& g, void* bricks, uint32_t* leafbits, uint32_t* occbits, int* bbox,
                               cudaStream_t st) {
    const unsigned nbt = (unsigned)g.nb[0] * (unsigned)g.nb[1] * (unsigned)g.nb[2];  // < 2^23 (the upload's limit)
    auto kernel = g.dtype == 1 ? k_pack_volume<1> : g.dtype == 2 ? k_pack_volume<2> : k_pack_volume<0>;
    kernel<<<nbt, 256, 0, st>>>(dense, dims[0], dims[1], dims[2], origin[0], origin[1], origin[2], leaf_mask, g, bricks,
                                leafbits, occbits, bbox);
    ++g_launch_counter;
    return cudaGetLastError();
}

// --- environment map -------------------------------------------------------

__device__ void dist1d_build(const float* f, int n, float* cdf_out, float* int_out) {
    double acc = 0.0;
    cdf_out[0] = 0.f;
    // unnormalised prefix of f/n, then divide by the total (src/Sampling.h:83-92)
    for (int i = 1; i <= n; ++i) acc += (double)f[i - 1] / (double)n;
    const double total = acc;
    if (total == 0.0) {
        for (int i = 1; i <= n; ++i) cdf_out[i] = (float)((double)i / (double)n);
    } else {
        double run = 0.0;
        for (int i = 1; i <= n; ++i) {
            run += (double)f[i - 1] / (double)n;
            cdf_out[i] = (float)(run / total);
        }
    }
    *int_out = (float)total;
}

// One thread per row: the sin(theta)-weighted luminance and the row's CDF.
__global__ void k_env_rows(const float* __restrict__ rgb, int w, int h, float* __restrict__ cond_func,
                           float* __restrict__ cond_cdf, float* __restrict__ cond_int) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= h) return;
    const float sin_theta = (float)sin(3.14159265358979323846 * (double)((float)r / (float)(h - 1)));
    float* f = cond_func + (int64_t)r * w;
    for (int c = 0; c < w; ++c) {
        const float* p = rgb + ((int64_t)r * w + c) * 3;
        const float y = (float)(0.2126 * (double)p[0] + 0.7152 * (double)p[1] + 0.0722 * (double)p[2]);
        f[c] = y * sin_theta;
    }
    dist1d_build(f, w, cond_cdf + (int64_t)r * (w + 1), cond_int + r);
}

__global__ void k_env_marginal(const float* __restrict__ cond_int, int h, float* __restrict__ marg_func,
                               float* __restrict__ marg_cdf, float* __restrict__ marg_int) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    for (int r = 0; r < h; ++r) marg_func[r] = cond_int[r];
    dist1d_build(marg_func, h, marg_cdf, marg_int);
}

// Guide table entry g of each of `rows` CDFs of n + 1 values (row stride
// n + 1): the first index with cdf > g / kEnvGuide, by binary search.
__global__ void k_env_guide(const float* __restrict__ cdf, int n, int rows, int* __restrict__ guide) {
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= (int64_t)rows * (kEnvGuide + 1)) return;
    const int r = (int)(e / (kEnvGuide + 1)), g = (int)(e % (kEnvGuide + 1));
    const float x = (float)g / (float)kEnvGuide;  // exact
    const float* c = cdf + (int64_t)r * (n + 1);
    int first = 0, len = n + 1;
    while (len > 0) {
        const int half = len >> 1, middle = first + half;
        if (c[middle] <= x) { first = middle + 1; len -= half + 1; }
        else len = half;
    }
    guide[e] = first;
}

cudaError_t launch_env_cdf(const float* rgb, int w, int h, float* cond_func, float* cond_cdf,
                           float* cond_int, float* marg_func, float* marg_cdf, float* marg_int,
                           int* cond_guide, int* marg_guide, cudaStream_t st) {
    k_env_rows<<<(h + 63) / 64, 64, 0, st>>>(rgb, w, h, cond_func, cond_cdf, cond_int);
    k_env_marginal<<<1, 32, 0, st>>>(cond_int, h, marg_func, marg_cdf, marg_int);
    const int64_t ne = (int64_t)h * (kEnvGuide + 1);
    k_env_guide<<<(unsigned)((ne + 255) / 256), 256, 0, st>>>(cond_cdf, w, h, cond_guide);
    k_env_guide<<<(kEnvGuide + 1 + 255) / 256, 256, 0, st>>>(marg_cdf, h, 1, marg_guide);
    g_launch_counter += 4;
    return cudaGetLastError();
}

}  // namespace lg
