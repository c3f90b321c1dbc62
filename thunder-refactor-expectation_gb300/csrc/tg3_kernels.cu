// tg3_kernels.cu -- the plain (FP32) E-step and insertion kernels for sm_103a.
//
// Data layout in HBM (all particle-major):
//   projection volume  : 64-byte corner blocks (see k_volume_blocks), all
//                        eight corners of a trilinear sample in one half
//                        cache line, read by two lanes with one 256-bit load
//                        each, placed in 32^3-voxel cubes (brick_index);
//   projections P      : [row][Kp] floats, a complex row padded with zeros to
//                        Kp floats (Kp a multiple of 64);
//   shifted data A''   : [particle][translation][Kp] floats, the complex
//                        sigRcp * ctf * X * exp(+2 pi i k.t / N);
//   log-likelihoods D  : [particle][rotation][translation] floats, without the
//                        per-particle constant sum sigRcp |X|^2;
//   insertion volume   : float4 [vdim][vdim][nx] of (F.re, F.im, T, 0), one
//                        16-byte atomic per voxel update.
#include <algorithm>

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math_constants.h>
#include <stdint.h>

#include "tg3_internal.cuh"

namespace tg3 {

namespace {

// Store one complex value at element pair p of row `row` (pitch ldo
// elements): as two floats, or -- when splitLo != 0 -- as the bf16 pair
// hi = bf16(v) in the plane at `out` and lo = bf16(v - hi) in the plane
// splitLo elements further on.
__device__ __forceinline__ void store_pair(float* out, long long splitLo, size_t row, int ldo,
                                           int p, float a, float b)
{
    if (splitLo == 0) {
        reinterpret_cast<float2*>(out + row * ldo)[p] = make_float2(a, b);
        return;
    }
    __nv_bfloat16* hi = reinterpret_cast<__nv_bfloat16*>(out);
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    const float2 hf = __bfloat1622float2(h);
    const __nv_bfloat162 l = __floats2bfloat162_rn(a - hf.x, b - hf.y);
    reinterpret_cast<__nv_bfloat162*>(hi + row * ldo)[p] = h;
    reinterpret_cast<__nv_bfloat162*>(hi + splitLo + row * ldo)[p] = l;
}

// Lane-pair form of store_pair: both lanes of a pair hold (a, b); lane half
// h stores its share -- the real (h = 0) or imaginary (h = 1) float, or the
// hi (h = 0) or lo (h = 1) bf16 pair -- so a warp's stores are contiguous.
__device__ __forceinline__ void store_pair_half(float* out, long long splitLo, size_t row, int ldo,
                                                int p, int h, float a, float b)
{
    if (splitLo == 0) {
        out[row * ldo + 2 * (size_t)p + h] = h ? b : a;
        return;
    }
    __nv_bfloat16* hi = reinterpret_cast<__nv_bfloat16*>(out);
    __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    if (h) {
        const float2 hf = __bfloat1622float2(v);
        v = __floats2bfloat162_rn(a - hf.x, b - hf.y);
    }
    reinterpret_cast<__nv_bfloat162*>(hi + (h ? splitLo : 0) + row * ldo)[p] = v;
}

__device__ __forceinline__ float warp_sum(float v)
{
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ double warp_sum_d(double v)
{
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ float warp_max(float v)
{
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// Block-wide sum (double) through shared scratch of >= 32 doubles.
__device__ double block_sum_d(double v, double* scratch)
{
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int nw = (blockDim.x + 31) >> 5;
    v = warp_sum_d(v);
    __syncthreads();
    if (lane == 0) scratch[wid] = v;
    __syncthreads();
    double r = 0;
    if (wid == 0) {
        r = lane < nw ? scratch[lane] : 0.0;
        r = warp_sum_d(r);
        if (lane == 0) scratch[0] = r;
    }
    __syncthreads();
    r = scratch[0];
    __syncthreads();
    return r;
}

// Quaternion -> row-major rotation matrix, R = I + 2 w A + 2 A^2
// (rotate3D, src/Geometry/Euler.cpp:181-189).
__device__ __forceinline__ void quat_to_mat(const double* q, double* m)
{
    const double A[3][3] = {{0, -q[3], q[2]}, {q[3], 0, -q[1]}, {-q[2], q[1], 0}};
    for (int i = 0; i < 3; i++)
        for (int j = 0; j < 3; j++) {
            double aa = (2 * A[i][0]) * A[0][j] + (2 * A[i][1]) * A[1][j]
                      + (2 * A[i][2]) * A[2][j];
            m[3 * i + j] = ((i == j ? 1.0 : 0.0) + (2 * q[0]) * A[i][j]) + aa;
        }
}

// ------------------------------------------------------------------------
__global__ void k_rotmat(const double* __restrict__ quat, int n, double* __restrict__ mat)
{
    int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n) return;
    double q[4] = {quat[4 * r], quat[4 * r + 1], quat[4 * r + 2], quat[4 * r + 3]};
    quat_to_mat(q, mat + 9 * (size_t)r);
}

// Phase-shift bank S[t][p] = exp(-2 pi i (iCol tx + iRow ty) / N)
// (translate, src/Image/ImageFunctions.cpp:233-252).
__global__ void k_translate(const double* __restrict__ trans, int nT, int idim,
                            const int* __restrict__ iCol, const int* __restrict__ iRow,
                            int K, float2* __restrict__ out, int ldo2)
{
    const int t = blockIdx.y;
    const float tx = (float)trans[2 * t], ty = (float)trans[2 * t + 1];
    const float invN = 1.0f / (float)idim;
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < ldo2; p += gridDim.x * blockDim.x) {
        float2 v = make_float2(0.f, 0.f);
        if (p < K) {
            float f = ((float)iCol[p] * tx + (float)iRow[p] * ty) * invN;
            float s, c;
            sincospif(2.0f * f, &s, &c);
            v = make_float2(c, -s);
        }
        out[(size_t)t * ldo2 + p] = v;
    }
}

// CTF at the selected pixels (CTF(RFLOAT*, ...), src/CTF.cpp:98-145).
__global__ void k_ctf(const float* __restrict__ attr, int nImg, float px, int idim,
                      const int* __restrict__ iCol, const int* __restrict__ iRow,
                      int K, float* __restrict__ out)
{
    const int l = blockIdx.x;
    const float* a = attr + 7 * (size_t)l;
    const float V = a[0], dU = a[1], dV = a[2], th = a[3], Cs = a[4], A = a[5], ps = a[6];
    const float lambda = 12.2643247f / sqrtf(V * (1 + V * 0.978466e-6f));
    const float w1 = sqrtf(1 - A * A), w2 = A;
    const float K1 = CUDART_PI_F * lambda;
    const float K2 = (CUDART_PI_F / 2) * Cs * lambda * lambda * lambda;
    const float inv = 1.0f / (px * (float)idim);
    for (int p = threadIdx.x; p < K; p += blockDim.x) {
        float u = hypotf((float)iCol[p] * inv, (float)iRow[p] * inv);
        float ang = atan2f((float)iRow[p], (float)iCol[p]) - th;
        float dfc = -(dU + dV + (dU - dV) * cosf(2 * ang)) / 2;
        float u2 = u * u;
        float ki = K1 * dfc * u2 + K2 * u2 * u2 - ps;
        out[(size_t)l * K + p] = -w1 * sinf(ki) + w2 * cosf(ki);
    }
}

// Placement of the corner block of voxel (z, y, x), z and y counted from the
// lowest coordinate -vdim / 2 (so that a sample's index needs no wrap): the
// volume is cut into cubes of 32^3 voxels (32768 blocks = 2 MB, one large page
// each, cubes in z, y, x order), voxels x-fastest within a cube.  A projection's
// samples within one pixel band then touch a few hundred pages instead of one
// page per z plane of the band, which in the plain [z][y][x] order left the
// gather translation-bound.
__device__ __forceinline__ size_t brick_index(int x, int y, int z, int nxc, int nyc)
{
    const size_t cube = ((size_t)(z >> 5) * nyc + (y >> 5)) * nxc + (x >> 5);
    return cube * 32768 + ((z & 31) * 32 + (y & 31)) * 32 + (x & 31);
}


// Corner-block content: the 64-byte element of voxel (z, y, x) holds, for
// slab z then slab z + 1, V[.][y][x], V[.][y][x+1], V[.][y+1][x],
// V[.][y+1][x+1] (rows and slabs taken modulo vdim, the wrap of
// Volume::iFTHalf; x + 1 past the stored half reads zero).  A trilinear
// sample then reads one aligned half cache line.
__global__ void k_volume_blocks(const float2* __restrict__ vol, int vdim,
                                float4* __restrict__ blocks)
{
    const int nx = vdim / 2 + 1;
    const int nxc = cubes_x(vdim), nyc = cubes_yz(vdim);
    const size_t n = (size_t)vdim * vdim * nx;
    const float2 zero = make_float2(0.f, 0.f);
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
         i += (size_t)gridDim.x * blockDim.x) {
        const int x = (int)(i % nx);
        const int y = (int)((i / nx) % vdim);
        const int z = (int)(i / ((size_t)nx * vdim));
        const int half = vdim / 2;
        const size_t d = brick_index(x, y < half ? y + half : y - half,
                                     z < half ? z + half : z - half, nxc, nyc);
        const int y1 = y + 1 == vdim ? 0 : y + 1;
#pragma unroll
        for (int k = 0; k < 2; k++) {
            const int zz = k == 0 ? z : (z + 1 == vdim ? 0 : z + 1);
            const size_t i0 = ((size_t)zz * vdim + y) * nx + x;
            const size_t i1 = ((size_t)zz * vdim + y1) * nx + x;
            const float2 a = vol[i0], b = (x + 1 < nx) ? vol[i0 + 1] : zero;
            const float2 c = vol[i1], dd = (x + 1 < nx) ? vol[i1 + 1] : zero;
            blocks[4 * d + 2 * k] = make_float4(a.x, a.y, b.x, b.y);
            blocks[4 * d + 2 * k + 1] = make_float4(c.x, c.y, dd.x, dd.y);
        }
    }
}

// ------------------------------------------------------------------------
// Fourier-slice extraction: P[row][p] = trilinear(V, R_row (iCol pf, iRow pf,
// 0)), Friedel-mirrored when x < 0 (Projector::project,
// src/Projector.cpp:356-374; Volume::getByInterpolationFT,
// src/Image/Volume.cpp:308-332).
//
// Work order.  A CTA takes one pixel chunk (kProjChunk consecutive pixels) of
// one particle for a group of kProjG of its rotations, and consecutive CTAs
// take the rotation groups of the same chunk.  The CTAs resident at any time
// therefore sweep one narrow band of pixels through all of a particle's
// rotations: the volume blocks that band touches (a few MB) stay in L2 while
// every rotation that reuses them runs, instead of the particle's whole
// footprint (about 160 MB at box 256) streaming from HBM once per reuse.
//
// A lane pair serves one pixel: lane half h reads slab z0 + h of the pixel's
// 64-byte corner block (one 256-bit load) and the two partial sums meet
// through one shuffle.  Each pair carries kProjU pixels of the chunk, whose
// indices and norm weights are loaded once for all the CTA's rotations.
//
// With nrmPart != null, nrmPart[row * nChunks + chunk] receives the chunk's
// share of sum_p sigRcp ctf^2 |P|^2 (k_norm_reduce sums the chunks).
__global__ void __launch_bounds__(256, 4)
k_project(float4* const* __restrict__ volTable, const int* __restrict__ cls,
          const float4* __restrict__ vol0, int vdim, int pf, const float* __restrict__ mf,
          int rowsPerParticle, int nGroups, int nChunks, const int* __restrict__ iCol,
          const int* __restrict__ iRow, int K, float* __restrict__ out, int ldo,
          const float* __restrict__ sigRcp, const float* __restrict__ ctf,
          float* __restrict__ nrmPart, int* __restrict__ flag, long long splitLo)
{
    __shared__ float m[kProjG][9];
    __shared__ float red[kProjG][8];
    const int g = blockIdx.x % nGroups;
    const int chunk = (blockIdx.x / nGroups) % nChunks;
    const int l = blockIdx.x / (nGroups * nChunks);
    const int r0 = g * kProjG;
    const int nRot = min(kProjG, rowsPerParticle - r0);
    const size_t row0 = (size_t)l * rowsPerParticle + r0;
    // brick_index split into per-axis terms: tx[x] + ty[y + vdim/2] +
    // tz[z + vdim/2], the y and z tables absorbing the wrap of negative rows
    extern __shared__ int tab[];
    const int half = vdim / 2;
    int* tx = tab;
    int* ty = tab + vdim / 2 + 1;
    int* tz = ty + vdim;
    fill_brick_tables(vdim, tx, ty, tz);
    if (threadIdx.x < 9 * nRot) m[threadIdx.x / 9][threadIdx.x % 9] = mf[9 * row0 + threadIdx.x];
    __syncthreads();
    const int nOut = ldo / 2;
    const int h = threadIdx.x & 1;
    const int npairs = blockDim.x >> 1;
    const int pBase = chunk * kProjChunk + (threadIdx.x >> 5) * 16 + ((threadIdx.x & 31) >> 1);
    const float4* __restrict__ vol = vol0;
    if (volTable) {
        const int k = cls ? cls[l] : 0;
        vol = (k >= 0 && k < kMaxClasses) ? volTable[k] : nullptr;
        if (!vol) {
            // unknown class: record it, leave the rows' chunk zero and skip sampling
            if (threadIdx.x == 0 && flag) atomicOr(flag, 8);
            for (int i = 0; i < nRot; i++)
#pragma unroll
                for (int u = 0; u < kProjU; u++) {
                    const int p = pBase + u * npairs;
                    if (p < nOut) store_pair_half(out, splitLo, row0 + i, ldo, p, h, 0.f, 0.f);
                }
            if (nrmPart && threadIdx.x < nRot) nrmPart[(row0 + threadIdx.x) * nChunks + chunk] = 0.f;
            return;
        }
    }
    const float fpf = (float)pf;
    const float* sg = sigRcp ? sigRcp + (size_t)l * K : nullptr;
    const float* cf = ctf ? ctf + (size_t)l * K : nullptr;
    // the chunk's pixels: coordinates and norm weights, shared by all rotations
    float pa[kProjU], pb[kProjU], w2[kProjU];
#pragma unroll
    for (int u = 0; u < kProjU; u++) {
        const int p = pBase + u * npairs;
        const int q = p < K ? p : 0;
        pa[u] = (float)iCol[q] * fpf;
        pb[u] = (float)iRow[q] * fpf;
        w2[u] = (nrmPart && p < K) ? sg[q] * cf[q] * cf[q] : 0.f;
    }
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll 1
    for (int i = 0; i < nRot; i++) {   // nRot is uniform across the CTA
        const float* mm = m[i];
        float acc = 0.f;
        float fw[kProjU][3];
        bool cj[kProjU];
        const float4* e[kProjU];
#pragma unroll
        for (int u = 0; u < kProjU; u++) {
            float x = mm[0] * pa[u] + mm[1] * pb[u];
            float y = mm[3] * pa[u] + mm[4] * pb[u];
            float z = mm[6] * pa[u] + mm[7] * pb[u];
            cj[u] = x < 0.f;
            if (cj[u]) { x = -x; y = -y; z = -z; }
            const float xf = floorf(x), yf = floorf(y), zf = floorf(z);
            const int x0 = (int)xf, y0 = (int)yf, z0 = (int)zf;
            fw[u][0] = x - xf;
            fw[u][1] = y - yf;
            fw[u][2] = z - zf;
            const unsigned blk = (unsigned)(tx[x0] + ty[y0 + half] + tz[z0 + half]);
            e[u] = vol + 4 * (size_t)blk + 2 * h;
        }
        float4 c[kProjU][2];
#pragma unroll
        for (int u = 0; u < kProjU; u++)
            asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                : "=f"(c[u][0].x), "=f"(c[u][0].y), "=f"(c[u][0].z), "=f"(c[u][0].w),
                  "=f"(c[u][1].x), "=f"(c[u][1].y), "=f"(c[u][1].z), "=f"(c[u][1].w)
                : "l"(e[u]));
#pragma unroll
        for (int u = 0; u < kProjU; u++) {
            const float fx = fw[u][0], fy = fw[u][1], fz = fw[u][2];
            const float wz = h ? fz : 1.f - fz;
            const float wx0 = 1.f - fx, wx1 = fx;
            const float wy0 = (1.f - fy) * wz, wy1 = fy * wz;
            float re = c[u][0].x * (wx0 * wy0) + c[u][0].z * (wx1 * wy0);
            float im = c[u][0].y * (wx0 * wy0) + c[u][0].w * (wx1 * wy0);
            re += c[u][1].x * (wx0 * wy1) + c[u][1].z * (wx1 * wy1);
            im += c[u][1].y * (wx0 * wy1) + c[u][1].w * (wx1 * wy1);
            re += __shfl_xor_sync(0xffffffffu, re, 1);
            im += __shfl_xor_sync(0xffffffffu, im, 1);
            const int p = pBase + u * npairs;
            if (p < nOut) {
                if (p < K) {
                    if (cj[u]) im = -im;
                    store_pair_half(out, splitLo, row0 + i, ldo, p, h, re, im);
                    if (h == 0) acc = fmaf(w2[u], re * re + im * im, acc);
                } else {
                    store_pair_half(out, splitLo, row0 + i, ldo, p, h, 0.f, 0.f);
                }
            }
        }
        // the warp's share of this rotation's norm, in a fixed order
        if (nrmPart) {
            acc = warp_sum(acc);
            if (lane == 0) red[i][wid] = acc;
        }
    }
    if (nrmPart) {
        __syncthreads();
        if (threadIdx.x < nRot) {
            float s = 0.f;
            for (int w = 0; w < (int)(blockDim.x >> 5); w++) s += red[threadIdx.x][w];
            nrmPart[(row0 + threadIdx.x) * nChunks + chunk] = s;
        }
    }
}

// The same extraction with one lane per pixel (form 1).  A lane reads both
// slabs of its pixel's corner block (two 256-bit loads) and forms the sample
// alone, so the coordinates, the block address and the fractions are
// computed once per sample instead of once per lane of a pair, and no
// shuffle joins the halves.  The slab sums are formed in the pair form's
// order (slab z0's four corners, slab z0 + 1's, then their sum).  Pixels:
// p = chunk kProjChunk + u blockDim + threadIdx, u < kProjChunk / blockDim.
// A warp's 32 pixels are consecutive, so its hi and lo (or FP32) stores are
// 128-byte (256-byte) runs.
// kArith forms the block index from the coordinates with integer
// arithmetic instead of the per-axis shared-memory tables: lanes of a warp
// look up scattered table entries, and those lookups share the L1 data pipe
// with the corner-block loads.
constexpr int kLaneU = kProjChunk / 256;
template <bool kArith>
__global__ void __launch_bounds__(256, 4)
k_project_lane(float4* const* __restrict__ volTable, const int* __restrict__ cls,
               const float4* __restrict__ vol0, int vdim, int pf, const float* __restrict__ mf,
               int rowsPerParticle, int nGroups, int nChunks, const int* __restrict__ iCol,
               const int* __restrict__ iRow, int K, float* __restrict__ out, int ldo,
               const float* __restrict__ sigRcp, const float* __restrict__ ctf,
               float* __restrict__ nrmPart, int* __restrict__ flag, long long splitLo)
{
    __shared__ float m[kProjG][9];
    __shared__ float red[kProjG][8];
    const int g = blockIdx.x % nGroups;
    const int chunk = (blockIdx.x / nGroups) % nChunks;
    const int l = blockIdx.x / (nGroups * nChunks);
    const int r0 = g * kProjG;
    const int nRot = min(kProjG, rowsPerParticle - r0);
    const size_t row0 = (size_t)l * rowsPerParticle + r0;
    extern __shared__ int tab[];
    const int half = vdim / 2;
    const int nxc = cubes_x(vdim), nyc = cubes_yz(vdim);
    int* tx = tab;
    int* ty = tab + vdim / 2 + 1;
    int* tz = ty + vdim;
    if (!kArith) fill_brick_tables(vdim, tx, ty, tz);
    if (threadIdx.x < 9 * nRot) m[threadIdx.x / 9][threadIdx.x % 9] = mf[9 * row0 + threadIdx.x];
    __syncthreads();
    const int nOut = ldo / 2;
    const int pBase = chunk * kProjChunk + threadIdx.x;
    __nv_bfloat162* hiPlane = reinterpret_cast<__nv_bfloat162*>(out);
    __nv_bfloat162* loPlane = reinterpret_cast<__nv_bfloat162*>(
        reinterpret_cast<__nv_bfloat16*>(out) + splitLo);
    auto store = [&](size_t row, int p, float re, float im) {
        if (splitLo == 0) {
            reinterpret_cast<float2*>(out + row * ldo)[p] = make_float2(re, im);
        } else {
            const __nv_bfloat162 v = __floats2bfloat162_rn(re, im);
            const float2 hf = __bfloat1622float2(v);
            hiPlane[row * nOut + p] = v;
            loPlane[row * nOut + p] = __floats2bfloat162_rn(re - hf.x, im - hf.y);
        }
    };
    const float4* __restrict__ vol = vol0;
    if (volTable) {
        const int k = cls ? cls[l] : 0;
        vol = (k >= 0 && k < kMaxClasses) ? volTable[k] : nullptr;
        if (!vol) {
            // unknown class: record it, leave the rows' chunk zero and skip sampling
            if (threadIdx.x == 0 && flag) atomicOr(flag, 8);
            for (int i = 0; i < nRot; i++)
#pragma unroll
                for (int u = 0; u < kLaneU; u++) {
                    const int p = pBase + u * 256;
                    if (p < nOut) store(row0 + i, p, 0.f, 0.f);
                }
            if (nrmPart && threadIdx.x < nRot) nrmPart[(row0 + threadIdx.x) * nChunks + chunk] = 0.f;
            return;
        }
    }
    const float fpf = (float)pf;
    const float* sg = sigRcp ? sigRcp + (size_t)l * K : nullptr;
    const float* cf = ctf ? ctf + (size_t)l * K : nullptr;
    float pa[kLaneU], pb[kLaneU], w2[kLaneU];
#pragma unroll
    for (int u = 0; u < kLaneU; u++) {
        const int p = pBase + u * 256;
        const int q = p < K ? p : 0;
        pa[u] = (float)iCol[q] * fpf;
        pb[u] = (float)iRow[q] * fpf;
        w2[u] = (nrmPart && p < K) ? sg[q] * cf[q] * cf[q] : 0.f;
    }
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll 1
    for (int i = 0; i < nRot; i++) {   // nRot is uniform across the CTA
        const float* mm = m[i];
        float acc = 0.f;
        float fw[kLaneU][3];
        bool cj[kLaneU];
        const float4* e[kLaneU];
#pragma unroll
        for (int u = 0; u < kLaneU; u++) {
            float x = mm[0] * pa[u] + mm[1] * pb[u];
            float y = mm[3] * pa[u] + mm[4] * pb[u];
            float z = mm[6] * pa[u] + mm[7] * pb[u];
            cj[u] = x < 0.f;
            if (cj[u]) { x = -x; y = -y; z = -z; }
            const float xf = floorf(x), yf = floorf(y), zf = floorf(z);
            const int x0 = (int)xf, y0 = (int)yf, z0 = (int)zf;
            fw[u][0] = x - xf;
            fw[u][1] = y - yf;
            fw[u][2] = z - zf;
            unsigned blk;
            if (kArith) {
                const int yy = y0 + half, zz = z0 + half;
                blk = (unsigned)((((zz >> 5) * nyc + (yy >> 5)) * nxc + (x0 >> 5)) * 32768
                                 + ((zz & 31) * 32 + (yy & 31)) * 32 + (x0 & 31));
            } else {
                blk = (unsigned)(tx[x0] + ty[y0 + half] + tz[z0 + half]);
            }
            e[u] = vol + 4 * (size_t)blk;
        }
        float4 c[kLaneU][4];
#pragma unroll
        for (int u = 0; u < kLaneU; u++)
#pragma unroll
            for (int k = 0; k < 2; k++)
                asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                    : "=f"(c[u][2 * k].x), "=f"(c[u][2 * k].y), "=f"(c[u][2 * k].z),
                      "=f"(c[u][2 * k].w), "=f"(c[u][2 * k + 1].x), "=f"(c[u][2 * k + 1].y),
                      "=f"(c[u][2 * k + 1].z), "=f"(c[u][2 * k + 1].w)
                    : "l"(e[u] + 2 * k));
#pragma unroll
        for (int u = 0; u < kLaneU; u++) {
            const float fx = fw[u][0], fy = fw[u][1], fz = fw[u][2];
            const float wx0 = 1.f - fx, wx1 = fx;
            float sr[2], si[2];
#pragma unroll
            for (int k = 0; k < 2; k++) {
                const float wz = k ? fz : 1.f - fz;
                const float wy0 = (1.f - fy) * wz, wy1 = fy * wz;
                const float4 a = c[u][2 * k], b = c[u][2 * k + 1];
                float re = a.x * (wx0 * wy0) + a.z * (wx1 * wy0);
                float im = a.y * (wx0 * wy0) + a.w * (wx1 * wy0);
                re += b.x * (wx0 * wy1) + b.z * (wx1 * wy1);
                im += b.y * (wx0 * wy1) + b.w * (wx1 * wy1);
                sr[k] = re;
                si[k] = im;
            }
            float re = sr[0] + sr[1];
            float im = si[0] + si[1];
            const int p = pBase + u * 256;
            if (p < nOut) {
                if (p < K) {
                    if (cj[u]) im = -im;
                    store(row0 + i, p, re, im);
                    acc = fmaf(w2[u], re * re + im * im, acc);
                } else {
                    store(row0 + i, p, 0.f, 0.f);
                }
            }
        }
        if (nrmPart) {
            acc = warp_sum(acc);
            if (lane == 0) red[i][wid] = acc;
        }
    }
    if (nrmPart) {
        __syncthreads();
        if (threadIdx.x < nRot) {
            float s = 0.f;
            for (int w = 0; w < (int)(blockDim.x >> 5); w++) s += red[threadIdx.x][w];
            nrmPart[(row0 + threadIdx.x) * nChunks + chunk] = s;
        }
    }
}

// Two FP32 values in a 64-bit register, and the two-wide operations on them.
__device__ __forceinline__ uint64_t pack2(float x, float y)
{
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}

__device__ __forceinline__ float2 unpack2(uint64_t v)
{
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b)
{
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t mad2(uint64_t a, uint64_t b, uint64_t c)
{
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b)
{
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t sub2(uint64_t a, uint64_t b)
{
    return mad2(b, pack2(-1.f, -1.f), a);
}
__device__ __forceinline__ uint64_t add2_down(uint64_t a, uint64_t b)
{
    uint64_t r;
    asm("add.rm.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

// Block indexes and fractions of two samples, without tables and conversions:
// the floor comes out of an addition rounded down (x + 1.5 2^23 has the integer
// part of x in its low bits), the index (brick_index) out of shifted copies of
// those bits, x = a + 32 b -> a + 32768 b and so on, with all offsets in one
// constant.  A coordinate outside the volume (not a number) is held to the
// blocks there are.
struct BrickIndex {
    unsigned yc, zc, offset, last;
    float yMagic;
    __device__ __forceinline__ explicit BrickIndex(int vdim)
    {
        const unsigned nxc = cubes_x(vdim), nyc = cubes_yz(vdim), bias = 0x4b400000u;
        yc = nxc * 32768u - 1024u;
        zc = nxc * nyc * 32768u - 32768u;
        yMagic = 12582912.f + (float)(vdim / 2);
        last = nxc * nyc * nyc * 32768u - 1u;
        offset = 0u - (bias + 32736u * (bias >> 5)) - (32u * bias + yc * (bias >> 5)) -
                 (1024u * bias + zc * (bias >> 5));
    }
    __device__ __forceinline__ void operator()(const uint64_t (&v)[3], uint64_t (&f)[3],
                                               unsigned (&b)[2]) const
    {
        const float magic[3] = {12582912.f, yMagic, yMagic};
        unsigned n[3][2];
#pragma unroll
        for (int k = 0; k < 3; k++) {
            const uint64_t t = add2_down(v[k], pack2(magic[k], magic[k]));
            f[k] = sub2(v[k], add2(t, pack2(-magic[k], -magic[k])));
            n[k][0] = (unsigned)t;
            n[k][1] = (unsigned)(t >> 32);
        }
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const unsigned x = n[0][i], y = n[1][i], z = n[2][i];
            b[i] = min(offset + x + 32736u * (x >> 5) + 32u * y + yc * (y >> 5) + 1024u * z +
                           zc * (z >> 5),
                       last);
        }
    }
};

// Lane pairs that share loads (forms 3 and 4).  The pair's two loads read pixel
// A's block (the even lane slab z0, the odd lane slab z0 + 1) and then pixel B's,
// so every load instruction takes whole 64-byte blocks, one L1 wavefront per
// pixel as in the lane-pair form.  Each lane forms its slab's share of both
// pixels; the even lane keeps A and the odd one B, the other share arriving by
// shuffle (slab z0's share plus slab z0 + 1's, the pair form's sum).
// Coordinates, fractions and weights of A and B are formed together, two-wide.
// In form 4 (kArith) both lanes form them for both pixels; in form 3 a lane
// finds its own pixel's block by table and fractions, and the pair swaps them.
// Form 4 is bound by the L1's data stage and the issue slots about alike: 47
// wavefronts per 32 samples, 39 of them the blocks (80 % of its cycles), 176
// instructions (72 %).  So the matrix comes as two loads, the norms' lane sums go
// through shared memory for all rotations at once, and the index needs neither
// tables nor conversions nor exchange.  64 particles x 1,000 x 9,930: 3.73 ms;
// with four shuffles for the exchange 3.82; with five more a norm, six matrix
// loads, and conversions, wraps and 8^3 bricks in the index 4.00.
template <bool kArith, int G>
__global__ void __launch_bounds__(256, 4)
k_project_xchg(float4* const* __restrict__ volTable, const int* __restrict__ cls,
               const float4* __restrict__ vol0, int vdim, int pf, const float* __restrict__ mf,
               int rowsPerParticle, int nGroups, int nChunks, const int* __restrict__ iCol,
               const int* __restrict__ iRow, int K, float* __restrict__ out, int ldo,
               const float* __restrict__ sigRcp, const float* __restrict__ ctf,
               float* __restrict__ nrmPart, int* __restrict__ flag, long long splitLo)
{
    __shared__ __align__(16) float m[G][8];      // rows 0 - 2, columns 0 and 1
    __shared__ float red[G][8];
    // a warp's norm terms of every rotation, LPR lanes of it a rotation at the end
    constexpr int LPR = 32 / G, kPitch = 32 + LPR;
    __shared__ float part[8][G * kPitch];
    const int g = blockIdx.x % nGroups;
    const int chunk = (blockIdx.x / nGroups) % nChunks;
    const int l = blockIdx.x / (nGroups * nChunks);
    const int r0 = g * G;
    const int nRot = min(G, rowsPerParticle - r0);
    const size_t row0 = (size_t)l * rowsPerParticle + r0;
    extern __shared__ int tab[];
    const int half = vdim / 2;
    int* tx = tab;
    int* ty = tab + vdim / 2 + 1;
    int* tz = ty + vdim;
    if (!kArith) fill_brick_tables(vdim, tx, ty, tz);
    if (threadIdx.x < 6 * nRot) {
        const int i = threadIdx.x / 6, e = threadIdx.x % 6;
        m[i][e] = mf[9 * (row0 + i) + e / 2 * 3 + e % 2];
    }
    const BrickIndex bi(vdim);
    __syncthreads();
    const int nOut = ldo / 2;
    const int h = threadIdx.x & 1;
    const int pBase = chunk * kProjChunk + threadIdx.x;
    __nv_bfloat162* hiPlane = reinterpret_cast<__nv_bfloat162*>(out);
    __nv_bfloat162* loPlane = reinterpret_cast<__nv_bfloat162*>(
        reinterpret_cast<__nv_bfloat16*>(out) + splitLo);
    auto store = [&](size_t row, int p, float re, float im) {
        if (splitLo == 0) {
            reinterpret_cast<float2*>(out + row * ldo)[p] = make_float2(re, im);
        } else {
            const __nv_bfloat162 v = __floats2bfloat162_rn(re, im);
            const float2 hf = __bfloat1622float2(v);
            hiPlane[row * nOut + p] = v;
            loPlane[row * nOut + p] = __floats2bfloat162_rn(re - hf.x, im - hf.y);
        }
    };
    const float4* __restrict__ vol = vol0;
    if (volTable) {
        const int k = cls ? cls[l] : 0;
        vol = (k >= 0 && k < kMaxClasses) ? volTable[k] : nullptr;
        if (!vol) {
            // unknown class: record it, leave the rows' chunk zero and skip sampling
            if (threadIdx.x == 0 && flag) atomicOr(flag, 8);
            for (int i = 0; i < nRot; i++)
#pragma unroll
                for (int u = 0; u < kLaneU; u++) {
                    const int p = pBase + u * 256;
                    if (p < nOut) store(row0 + i, p, 0.f, 0.f);
                }
            if (nrmPart && threadIdx.x < nRot) nrmPart[(row0 + threadIdx.x) * nChunks + chunk] = 0.f;
            return;
        }
    }
    const float fpf = (float)pf;
    const float* sg = sigRcp ? sigRcp + (size_t)l * K : nullptr;
    const float* cf = ctf ? ctf + (size_t)l * K : nullptr;
    // own pixels' weights; the coordinates of the pair's pixels A and B (of the own
    // one, twice, with the table)
    uint64_t pa[kLaneU], pb[kLaneU];
    float w2[kLaneU];
#pragma unroll
    for (int u = 0; u < kLaneU; u++) {
        const int p = pBase + u * 256;
        const int q = p < K ? p : 0;
        const float a = (float)iCol[q] * fpf, b = (float)iRow[q] * fpf;
        const float a1 = __shfl_xor_sync(0xffffffffu, a, 1), b1 = __shfl_xor_sync(0xffffffffu, b, 1);
        pa[u] = !kArith ? pack2(a, a) : h ? pack2(a1, a) : pack2(a, a1);
        pb[u] = !kArith ? pack2(b, b) : h ? pack2(b1, b) : pack2(b, b1);
        w2[u] = (nrmPart && p < K) ? sg[q] * cf[q] * cf[q] : 0.f;
    }
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll 1
    for (int i = 0; i < nRot; i++) {   // nRot is uniform across the CTA
        const float4 m01 = *reinterpret_cast<const float4*>(m[i]);
        const float2 m2 = *reinterpret_cast<const float2*>(m[i] + 4);
        float acc = 0.f;
        uint64_t f[kLaneU][3];                // fractions of A and B
        unsigned blk[kLaneU][2];              // block index of A and B
        bool cj[kLaneU];
#pragma unroll
        for (int u = 0; u < kLaneU; u++) {
            uint64_t v[3] = {mad2(pack2(m01.x, m01.x), pa[u], mul2(pack2(m01.y, m01.y), pb[u])),
                             mad2(pack2(m01.z, m01.z), pa[u], mul2(pack2(m01.w, m01.w), pb[u])),
                             mad2(pack2(m2.x, m2.x), pa[u], mul2(pack2(m2.y, m2.y), pb[u]))};
            const float2 x = unpack2(v[0]);
            cj[u] = (kArith && h ? x.y : x.x) < 0.f;
            const uint64_t sign = pack2(x.x < 0.f ? -1.f : 1.f, x.y < 0.f ? -1.f : 1.f);
#pragma unroll
            for (int k = 0; k < 3; k++) v[k] = mul2(v[k], sign);
            if (kArith) {
                bi(v, f[u], blk[u]);
            } else {
                float o[3];
                int n[3];
#pragma unroll
                for (int k = 0; k < 3; k++) {
                    const float c = unpack2(v[k]).x, fl = floorf(c);
                    o[k] = c - fl;
                    n[k] = (int)fl;
                }
                const unsigned own = (unsigned)(tx[n[0]] + ty[n[1] + half] + tz[n[2] + half]);
                const unsigned other = __shfl_xor_sync(0xffffffffu, own, 1);
                blk[u][0] = h ? other : own;
                blk[u][1] = h ? own : other;
#pragma unroll
                for (int k = 0; k < 3; k++) {
                    const float p = __shfl_xor_sync(0xffffffffu, o[k], 1);
                    f[u][k] = h ? pack2(p, o[k]) : pack2(o[k], p);
                }
            }
        }
        // slab h of pixel A (the even lane's) then of pixel B (the odd lane's)
        float4 c[kLaneU][4];
#pragma unroll
        for (int u = 0; u < kLaneU; u++)
#pragma unroll
            for (int k = 0; k < 2; k++) {
                const float4* e = vol + 4 * (size_t)blk[u][k] + 2 * h;
                asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                    : "=f"(c[u][2 * k].x), "=f"(c[u][2 * k].y), "=f"(c[u][2 * k].z),
                      "=f"(c[u][2 * k].w), "=f"(c[u][2 * k + 1].x), "=f"(c[u][2 * k + 1].y),
                      "=f"(c[u][2 * k + 1].z), "=f"(c[u][2 * k + 1].w)
                    : "l"(e));
            }
#pragma unroll
        for (int u = 0; u < kLaneU; u++) {
            const uint64_t one = pack2(1.f, 1.f);
            const uint64_t wx0 = sub2(one, f[u][0]), wx1 = f[u][0];
            const uint64_t wz = h ? f[u][2] : sub2(one, f[u][2]);
            const uint64_t wy0 = mul2(sub2(one, f[u][1]), wz), wy1 = mul2(f[u][1], wz);
            const uint64_t w00 = mul2(wx0, wy0), w10 = mul2(wx1, wy0), w01 = mul2(wx0, wy1),
                           w11 = mul2(wx1, wy1);
            float sr[2], si[2];
#pragma unroll
            for (int k = 0; k < 2; k++) {
                const float2 p = unpack2(w00), q = unpack2(w10), r = unpack2(w01), t = unpack2(w11);
                const float v00 = k ? p.y : p.x, v10 = k ? q.y : q.x, v01 = k ? r.y : r.x,
                            v11 = k ? t.y : t.x;
                const float4 a = c[u][2 * k], b = c[u][2 * k + 1];
                float re = a.x * v00 + a.z * v10;
                float im = a.y * v00 + a.w * v10;
                re += b.x * v01 + b.z * v11;
                im += b.y * v01 + b.w * v11;
                sr[k] = re;
                si[k] = im;
            }
            // lane 0 keeps A (k = 0) and sends its share of B; lane 1 keeps B
            const float keepR = h ? sr[1] : sr[0], keepI = h ? si[1] : si[0];
            const float sendR = h ? sr[0] : sr[1], sendI = h ? si[0] : si[1];
            float re = keepR + __shfl_xor_sync(0xffffffffu, sendR, 1);
            float im = keepI + __shfl_xor_sync(0xffffffffu, sendI, 1);
            const int p = pBase + u * 256;
            if (p < nOut) {
                if (p < K) {
                    if (cj[u]) im = -im;
                    store(row0 + i, p, re, im);
                    acc = fmaf(w2[u], re * re + im * im, acc);
                } else {
                    store(row0 + i, p, 0.f, 0.f);
                }
            }
        }
        part[wid][i * kPitch + lane] = acc;
    }
    if (nrmPart) {
        // the sums over the lanes of all rotations together, in warp_sum's order
        // (lanes 16 apart, then 8, ...): LPR lanes a rotation
        __syncwarp();
        const int j = lane / LPR;
        float v[G];
#pragma unroll
        for (int k = 0; k < G; k++) v[k] = part[wid][j * kPitch + lane % LPR + LPR * k];
#pragma unroll
        for (int w = G / 2; w; w >>= 1)
#pragma unroll
            for (int k = 0; k < w; k++) v[k] += v[k + w];
#pragma unroll
        for (int o = LPR / 2; o; o >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
        if (lane % LPR == 0) red[j][wid] = v[0];
        __syncthreads();
        if (threadIdx.x < nRot) {
            float s = 0.f;
            for (int w = 0; w < (int)(blockDim.x >> 5); w++) s += red[threadIdx.x][w];
            nrmPart[(row0 + threadIdx.x) * nChunks + chunk] = s;
        }
    }
}

// FP32 rotation matrix of each projected row, from its quaternion
// (quat_to_mat in FP64, then rounded) or from an FP64 matrix.
__global__ void k_rot_f32(const double* __restrict__ quat, const double* __restrict__ mat,
                          int rows, float* __restrict__ mf)
{
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < rows; r += gridDim.x * blockDim.x) {
        double md[9];
        if (quat) {
            double q[4] = {quat[4 * (size_t)r], quat[4 * (size_t)r + 1], quat[4 * (size_t)r + 2],
                           quat[4 * (size_t)r + 3]};
            quat_to_mat(q, md);
        } else {
            for (int i = 0; i < 9; i++) md[i] = mat[9 * (size_t)r + i];
        }
        for (int i = 0; i < 9; i++) mf[9 * (size_t)r + i] = (float)md[i];
    }
}

// nrm[row] = sum over the row's pixel chunks of nrmPart, in chunk order.
__global__ void k_norm_reduce(const float* __restrict__ nrmPart, int rows, int nChunks,
                              float* __restrict__ nrm)
{
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < rows; r += gridDim.x * blockDim.x) {
        double s = 0.0;
        for (int c = 0; c < nChunks; c++) s += (double)nrmPart[(size_t)r * nChunks + c];
        nrm[r] = (float)s;
    }
}

// Shifted, weighted data A''[l][d][t][p] = sigRcp ctf_d X exp(+2 pi i (iCol tx
// + iRow ty) / N), the conjugate of sigRcp ctf_d conj(X) S_t, so that
// Re sum_p sigRcp ctf_d conj(X) S_t P = sum over the 2K floats of A'' . P.
// nD CTFs per particle (ctf [nP][nD][K]; one without a defocus search).
// CTA: (particle l, CTF d) x SHIFT_T translations; a thread loads its
// pixels' data, sigRcp and CTF once and writes them for every translation.
constexpr int SHIFT_T = 8;

__global__ void k_shift_bank(const float2* __restrict__ dat, const float* __restrict__ ctf,
                             const float* __restrict__ sigRcp,
                             const double* __restrict__ trans, const float2* __restrict__ bank,
                             int nT, int nD, int idim,
                             const int* __restrict__ iCol, const int* __restrict__ iRow,
                             int K, float* __restrict__ out, int ldo, long long splitLo,
                             int useTab, int tPer)
{
    // per-particle translations with useTab: the phase e^{2 pi i (iCol tx + iRow ty) / N}
    // is the product of a column factor and a row factor, tabulated once per
    // CTA for its translations (tabX [SHIFT_T][h + 1] over iCol = 0 .. h, tabY
    // [SHIFT_T][2h + 1] over iRow = -h .. h), so a pixel costs two shared
    // loads and a complex product instead of a sine and a cosine
    extern __shared__ float2 tabX[];
    const int ld = blockIdx.x;            // l nD + d
    const int l = ld / nD;
    // tPer (<= SHIFT_T) translations per CTA, spread evenly over the groups
    const int t0 = blockIdx.y * tPer;
    const int t1 = min(nT, t0 + tPer);
    const float invN = 1.0f / (float)idim;
    const int h = idim / 2, nc = h + 1, nr = 2 * h + 1;
    float2* tabY = tabX + SHIFT_T * nc;
    if (useTab && !bank) {
        for (int e = threadIdx.x; e < (t1 - t0) * (nc + nr); e += blockDim.x) {
            const int tt = e / (nc + nr), j = e % (nc + nr);
            const size_t lt = (size_t)l * nT + t0 + tt;
            float sn, cs;
            if (j < nc) {
                sincospif(2.0f * ((float)j * (float)trans[2 * lt]) * invN, &sn, &cs);
                tabX[tt * nc + j] = make_float2(cs, sn);
            } else {
                const int r = j - nc - h;
                sincospif(2.0f * ((float)r * (float)trans[2 * lt + 1]) * invN, &sn, &cs);
                tabY[tt * nr + (j - nc)] = make_float2(cs, sn);
            }
        }
        __syncthreads();
    }
    for (int p = threadIdx.x; p < ldo / 2; p += blockDim.x) {
        float sc = 0.f;
        float2 X = make_float2(0.f, 0.f);
        float fc = 0.f, fr = 0.f;
        int ic = 0, ir = 0;
        bool tabOk = false;
        if (p < K) {
            const size_t i = (size_t)l * K + p;
            sc = sigRcp[i] * ctf[(size_t)ld * K + p];
            X = dat[i];
            if (!bank) {
                ic = iCol[p];
                ir = iRow[p];
                fc = (float)ic;
                fr = (float)ir;
                tabOk = useTab && ic >= 0 && ic <= h && ir >= -h && ir <= h;
            }
        }
        for (int t = t0; t < t1; t++) {
            const size_t row = (size_t)ld * nT + t;     // (l nD + d) nT + t
            float2 v = make_float2(0.f, 0.f);
            if (p < K) {
                float s, c;
                if (bank) {
                    // shared phase bank S[t][p] = (cos, -sin): use conj(S)
                    const float2 S = bank[(size_t)t * K + p];
                    c = S.x;
                    s = -S.y;
                } else if (tabOk) {
                    const float2 ex = tabX[(t - t0) * nc + ic], ey = tabY[(t - t0) * nr + ir + h];
                    c = ex.x * ey.x - ex.y * ey.y;
                    s = ex.y * ey.x + ex.x * ey.y;
                } else {
                    const size_t lt = (size_t)l * nT + t;
                    const float tx = (float)trans[2 * lt], ty = (float)trans[2 * lt + 1];
                    float f = (fc * tx + fr * ty) * invN;
                    sincospif(2.0f * f, &s, &c);
                }
                v = make_float2(sc * (X.x * c - X.y * s), sc * (X.x * s + X.y * c));
            }
            store_pair(out, splitLo, row, ldo, p, v.x, v.y);
        }
    }
}

// Defocus search: the norm sum_p sigRcp ctf_d^2 |P|^2 of every projected row
// for each of the particle's nD CTFs, nrm[r][l][d] (the layout the weights
// kernel reads per (row, block)).  CTA: (particle, 8 rows), a warp per row,
// |P|^2 from the FP32 row or from the split planes (hi + lo).
constexpr int kMaxDefocus = 16;

__global__ void __launch_bounds__(256)
k_norm_defocus(const float* __restrict__ P, long long splitLo, int nP, int nR, int nD, int K,
               int Kp, const float* __restrict__ sigRcp, const float* __restrict__ ctf,
               float* __restrict__ nrm)
{
    const int l = blockIdx.x;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int r = blockIdx.y * 8 + warp;
    if (r >= nR) return;
    const size_t row = (size_t)l * nR + r;
    float acc[kMaxDefocus];
#pragma unroll
    for (int d = 0; d < kMaxDefocus; d++) acc[d] = 0.f;
    const __nv_bfloat162* hi = reinterpret_cast<const __nv_bfloat162*>(P);
    for (int p = lane; p < K; p += 32) {
        float re, im;
        if (splitLo == 0) {
            const float2 v = reinterpret_cast<const float2*>(P + row * Kp)[p];
            re = v.x;
            im = v.y;
        } else {
            const float2 h = __bfloat1622float2(hi[(row * Kp) / 2 + p]);
            const float2 o = __bfloat1622float2(hi[(splitLo + row * Kp) / 2 + p]);
            re = h.x + o.x;
            im = h.y + o.y;
        }
        const float a2 = sigRcp[(size_t)l * K + p] * (re * re + im * im);
#pragma unroll
        for (int d = 0; d < kMaxDefocus; d++) {
            if (d < nD) {
                const float c = ctf[((size_t)l * nD + d) * K + p];
                acc[d] = fmaf(a2, c * c, acc[d]);
            }
        }
    }
#pragma unroll
    for (int d = 0; d < kMaxDefocus; d++) {
        if (d >= nD) break;
        float v = acc[d];
        for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0) nrm[((size_t)r * nP + l) * nD + d] = v;
    }
}

// CTF of one particle for each defocus factor d (kernel_CalCTFL of the
// reference GPU path; the CTF of Optimiser::updateSP, src/Optimiser.cpp:
// 1196-1214): ki = k1 defO[p] d f[p]^2 + k2 f[p]^4 - phaseShift,
// ctf = -sqrt(1 - conT^2) sin ki + conT cos ki, in FP64; ctf [nD][K].
__global__ void k_ctf_defocus(const float* __restrict__ defO, const float* __restrict__ freQ,
                              const double* __restrict__ dpara, int K, double k1, double k2,
                              double phaseShift, double conT, float* __restrict__ ctf)
{
    const int d = blockIdx.y;
    const double w1 = sqrt(1.0 - conT * conT);
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < K; p += gridDim.x * blockDim.x) {
        const double f2 = (double)freQ[p] * freQ[p];
        const double ki = k1 * defO[p] * dpara[d] * f2 + k2 * f2 * f2 - phaseShift;
        ctf[(size_t)d * K + p] = (float)(-w1 * sin(ki) + conT * cos(ki));
    }
}

// 2-D projection (2-D classification): the bilinear sample of a class's
// half transform img [vdim][vdim/2 + 1] at the in-plane rotation (c, s) of
// every pixel (iCol pf, iRow pf): x = i c - j s, y = i s + j c (the
// reference's kernel_Project2D, gpu/src/Kernel.cu:786-819, reading as
// Image::getByInterpolationFT, src/Image/Image.cpp:345-368: x < 0 at (-x, -y)
// conjugated, rows wrapped).  Rows out [nR][ldo] as k_project writes them
// (FP32 pairs, or split planes when splitLo != 0), zero beyond K.
__global__ void k_project2d(const float2* __restrict__ img, int vdim, int pf,
                            const double* __restrict__ rot, const int* __restrict__ iCol,
                            const int* __restrict__ iRow, int K, float* __restrict__ out,
                            int ldo, long long splitLo)
{
    const int r = blockIdx.y;
    const float c = (float)rot[2 * (size_t)r], s = (float)rot[2 * (size_t)r + 1];
    const int nx = vdim / 2 + 1;
    const float fpf = (float)pf;
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < ldo / 2;
         p += gridDim.x * blockDim.x) {
        float re = 0.f, im = 0.f;
        if (p < K) {
            const float i = (float)iCol[p] * fpf, j = (float)iRow[p] * fpf;
            float x = i * c - j * s, y = i * s + j * c;
            const bool conj = x < 0.f;
            if (conj) {
                x = -x;
                y = -y;
            }
            const float xf = floorf(x), yf = floorf(y);
            const int x0 = (int)xf, y0 = (int)yf;
            const float fx = x - xf, fy = y - yf;
#pragma unroll
            for (int b = 0; b < 2; b++) {
                int yy = y0 + b;
                yy = yy < 0 ? yy + vdim : yy;
                const float wy = b ? fy : 1.f - fy;
                const float2 v0 = __ldg(img + (size_t)yy * nx + x0);
                const float2 v1 = __ldg(img + (size_t)yy * nx + x0 + 1);
                re += wy * ((1.f - fx) * v0.x + fx * v1.x);
                im += wy * ((1.f - fx) * v0.y + fx * v1.y);
            }
            if (conj) im = -im;
        }
        store_pair(out, splitLo, r, ldo, p, re, im);
    }
}

// 2-D insertion (2-D classification; Reconstructor::insertP's 2-D form,
// Image::addFT(value, iCol, iRow), src/Image/Image.cpp:370-386; the
// reference's kernel_InsertF2D / T2D / O2D, gpu/src/Kernel.cu:2276-2470):
// draw d (image d / drawsPerImage, class nC[d], in-plane rotation nR[d] =
// (c, s), shift nT[d]) adds w ctf X shifted by -(t - offS) and w ctf^2
// bilinearly at (c a - s b, s a + c b), (a, b) = (iCol pf, iRow pf), into its
// class's (F.re, F.im, T, 0) accumulator [vdim][vdim/2 + 1] (x < 0: at
// (-x, -y), conjugated); O2D[class] gets -R (t - offS), counter[class] + 1.
// CTA (share of the pixels, draw).
__global__ void __launch_bounds__(256)
k_insert2d(float4* __restrict__ acc, int vdim, const float2* __restrict__ dat,
           const float* __restrict__ ctf, int ctfPerDraw, const float* __restrict__ wgt,
           const double* __restrict__ offS, const int* __restrict__ nC,
           const double* __restrict__ nR, const double* __restrict__ nT,
           const int* __restrict__ iCol, const int* __restrict__ iRow, int K, int pf, int idim,
           int d0, int drawsPerImage, double* __restrict__ O2D, int* __restrict__ counter)
{
    const int d = d0 + blockIdx.y;
    const int l = d / drawsPerImage;
    const int k = nC[d];
    const double cd = nR[2 * (size_t)d], sd = nR[2 * (size_t)d + 1];
    const double dx = nT[2 * (size_t)d] - offS[2 * (size_t)l];
    const double dy = nT[2 * (size_t)d + 1] - offS[2 * (size_t)l + 1];
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        if (O2D) {
            atomicAdd(O2D + 2 * k, -(cd * dx - sd * dy));
            atomicAdd(O2D + 2 * k + 1, -(sd * dx + cd * dy));
        }
        if (counter) atomicAdd(counter + k, 1);
    }
    const int nx = vdim / 2 + 1;
    float4* a4 = acc + (size_t)k * vdim * nx;
    const float c = (float)cd, s = (float)sd, tx = (float)dx, ty = (float)dy, w = wgt[l];
    const float invN = 1.0f / (float)idim, fpf = (float)pf;
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < K; p += gridDim.x * blockDim.x) {
        const float2 X = dat[(size_t)l * K + p];
        const float cv = ctf[(ctfPerDraw ? (size_t)d : (size_t)l) * K + p];
        float sn, co;
        sincospif(2.0f * (((float)iCol[p] * tx + (float)iRow[p] * ty) * invN), &sn, &co);
        const float cw = cv * w;
        float vr = (X.x * co - X.y * sn) * cw, vi = (X.x * sn + X.y * co) * cw;
        const float vt = cv * cv * w;
        const float a = (float)iCol[p] * fpf, b = (float)iRow[p] * fpf;
        float x = c * a - s * b, y = s * a + c * b;
        if (x < 0.f) {
            x = -x;
            y = -y;
            vi = -vi;
        }
        const float xf = floorf(x), yf = floorf(y);
        const int x0 = (int)xf, y0 = (int)yf;
        const float fx = x - xf, fy = y - yf;
#pragma unroll
        for (int j = 0; j < 2; j++) {
            int yy = y0 + j;
            yy = yy < 0 ? yy + vdim : yy;
            const float wy = j ? fy : 1.f - fy;
#pragma unroll
            for (int i = 0; i < 2; i++) {
                const float ww = (i ? fx : 1.f - fx) * wy;
                atomicAdd(a4 + (size_t)yy * nx + x0 + i, make_float4(vr * ww, vi * ww, vt * ww, 0.f));
            }
        }
    }
}

// CTF attributes of every insertion draw with the defocus search: the
// image's attributes with defocusU, V scaled by the draw's factor nD (the
// defocus kernel_CalculateCTF uses, gpu/src/Kernel.cu:2132-2198).
__global__ void k_draw_attr(const float* __restrict__ attr, const double* __restrict__ nD,
                            int nDraws, int drawsPerImage, float* __restrict__ out)
{
    const int d = blockIdx.x * blockDim.x + threadIdx.x;
    if (d >= nDraws) return;
    const float* a = attr + 7 * (size_t)(d / drawsPerImage);
    float* o = out + 7 * (size_t)d;
    for (int k = 0; k < 7; k++) o[k] = a[k];
    o[1] = (float)((double)a[1] * nD[d]);
    o[2] = (float)((double)a[2] * nD[d]);
}

// dst[(row nRep + k) len + j] = src[row len + j] (per-block copies of a
// particle's priors for the weights kernel's (particle, defocus) blocks)
__global__ void k_repeat_rows(const double* __restrict__ src, int rows, int len, int nRep,
                              double* __restrict__ dst)
{
    const size_t n = (size_t)rows * nRep * len;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
         i += (size_t)gridDim.x * blockDim.x) {
        const size_t j = i % len, rk = i / len;
        dst[i] = src ? src[(rk / nRep) * len + j] : 1.0;
    }
}

// Merge of a particle's nD (particle, defocus) blocks, each relative to its
// own maximum, into the particle's weights relative to the overall maximum
// (the running baseline of Optimiser::updateSP, src/Optimiser.cpp:1326-1347,
// with its defocus axis): wD[d] = e_d wC_d, wC = sum_d pD[d] e_d wC_d,
// wR / wT = sum_d pD[d] e_d wR_d / wT_d, e_d = exp(base_d - base).
__global__ void k_merge_defocus(int nD, int nR, int nT, const double* __restrict__ wCb,
                                const double* __restrict__ wRb, const double* __restrict__ wTb,
                                const double* __restrict__ baseb, const double* __restrict__ pwD,
                                double* __restrict__ wC, double* __restrict__ wR,
                                double* __restrict__ wT, double* __restrict__ wD,
                                double* __restrict__ base)
{
    __shared__ double e[kMaxDefocus], pd[kMaxDefocus];
    const int l = blockIdx.x;
    if (threadIdx.x == 0) {
        double m = baseb[(size_t)l * nD];
        for (int d = 1; d < nD; d++) m = fmax(m, baseb[(size_t)l * nD + d]);
        double c = 0.0;
        for (int d = 0; d < nD; d++) {
            e[d] = exp(baseb[(size_t)l * nD + d] - m);
            pd[d] = pwD[(size_t)l * nD + d];
            wD[(size_t)l * nD + d] = e[d] * wCb[(size_t)l * nD + d];
            c += pd[d] * wD[(size_t)l * nD + d];
        }
        wC[l] = c;
        base[l] = m;
    }
    __syncthreads();
    for (int r = threadIdx.x; r < nR; r += blockDim.x) {
        double s = 0.0;
        for (int d = 0; d < nD; d++) s += pd[d] * e[d] * wRb[((size_t)l * nD + d) * nR + r];
        wR[(size_t)l * nR + r] = s;
    }
    for (int t = threadIdx.x; t < nT; t += blockDim.x) {
        double s = 0.0;
        for (int d = 0; d < nD; d++) s += pd[d] * e[d] * wTb[((size_t)l * nD + d) * nT + t];
        wT[(size_t)l * nT + t] = s;
    }
}

__global__ void k_x0(const float2* __restrict__ dat, const float* __restrict__ sigRcp,
                     int K, double* __restrict__ x0)
{
    __shared__ double red[32];
    const int l = blockIdx.x;
    double acc = 0;
    for (int p = threadIdx.x; p < K; p += blockDim.x) {
        // FP32 terms, FP64 sum: one double add a pixel (the GPU's FP64
        // rate is a small fraction of its FP32 rate)
        const float2 X = dat[(size_t)l * K + p];
        acc += (double)(sigRcp[(size_t)l * K + p] * fmaf(X.x, X.x, X.y * X.y));
    }
    double s = block_sum_d(acc, red);
    if (threadIdx.x == 0) x0[l] = s;
}

// ------------------------------------------------------------------------
// Batched FP32 "NT" GEMM on the CUDA cores: C[b][i][j] = alpha sum_k
// A[b][i][k] B[b][j][k] (+ nrm[b][i]).  128 threads as 8 x 16, TM x TN
// outputs a thread (tile 8 TM x 16 TN), K in tiles of BK through two shared
// buffers.  Every output is one chain of fused multiply-adds over ascending
// k, whatever the tile.  Kd must be a multiple of BK and lda/ldb multiples of 4
// (rows zero-padded).
//
// Bound by the FP32 pipe: the products go in pairs of rows (fma.rn.f32x2,
// one issue for two multiply-adds), which leaves issue slots for the shared
// loads.  The column operand of a pair is one value twice, a register move.
// A shared load costs a cycle for every 128 bytes that it returns, so a warp
// spends TM + TN cycles of the shared port on TM TN / 4 cycles of the FP32
// pipes: 16 x 8 outputs a thread keep that at three quarters, 8 x 8 at one.
// Measured against 128 x 128 tiles of 256 threads with single multiply-adds:
// 6,912 x 16,317 x 768 in 2.8 instead of 4.2 ms (62 TFLOP/s, cuBLAS SGEMM 70),
// 32 particles of 1,000 x 100 x 19,904 in 3.0 instead of 4.7 ms, one of
// 100 x 9 x 768 in 8 instead of 13 us.
// The staged tiles are transposed, [k][row], with row XOR f(k): f spreads the
// BK / 4 float4 columns that a warp stores together over the banks (no
// conflict at any BK) and moves whole float4 groups, so the reads stay vectors.
__device__ __forceinline__ void fma2(uint64_t& d, uint64_t a, uint64_t b)
{
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}

template <int TM, int TN>
__global__ void __launch_bounds__(128, TM == 16 ? 2 : TM == 8 ? 3 : 4)
k_gemm_nt_fp32(const float* __restrict__ A, long long sA, int lda,
               const float* __restrict__ B, long long sB, int ldb,
               int M, int N, int Kd, float* __restrict__ C, long long sC, int ldc,
               const float* __restrict__ nrm, long long sN, float alpha, int cGroup,
               long long cGroupStride)
{
    constexpr int BM = 8 * TM, BN = 16 * TN;
    constexpr int BK = TM == 2 ? 32 : 128 / TM;   // 8, 16, 32, 32
    constexpr int NA = BM * BK / 512;             // A float4 a thread and tile
    // K tiles in flight from global memory (registers allowing)
    constexpr int D = TM >= 8 || TN <= 4 ? 2 : 1;
    constexpr int QK = BK / 4;                    // float4 columns of a tile
    constexpr int PB = (BN + 31) / 32 * 32;       // column pitch of the staged B
    constexpr int NB = (BN * QK + 127) / 128;     // B float4 a thread and tile
    __shared__ __align__(16) float As[2][BK][(BM + 31) / 32 * 32];
    __shared__ __align__(16) float Bs[2][BK][PB];
    const int b = blockIdx.z;
    const int i0 = blockIdx.y * BM, j0 = blockIdx.x * BN;
    A += b * sA;
    B += b * sB;
    C += b * sC;
    const int tid = threadIdx.x;
    const int tx = tid & 15, ty = tid >> 4;
    // rows past the end read the last one: their outputs are not stored
    const float4* pa[NA];
    const float4* pb[NB];
#pragma unroll
    for (int h = 0; h < NA; h++) {
        const int e = tid + 128 * h;
        pa[h] = reinterpret_cast<const float4*>(A + (size_t)min(i0 + e / QK, M - 1) * lda) + e % QK;
    }
#pragma unroll
    for (int h = 0; h < NB; h++) {
        const int e = tid + 128 * h;
        pb[h] = reinterpret_cast<const float4*>(B + (size_t)min(j0 + e / QK, N - 1) * ldb) + e % QK;
    }
    float4 ra[D][NA], rb[D][NB];
    auto load = [&](int d) {
#pragma unroll
        for (int h = 0; h < NA; h++) {
            ra[d][h] = __ldg(pa[h]);
            pa[h] += QK;
        }
#pragma unroll
        for (int h = 0; h < NB; h++) {
            rb[d][h] = __ldg(pb[h]);
            pb[h] += QK;
        }
    };
    // f(k) = (k / 4) (32 / QK): the rows a warp stores together are 32 / QK
    auto store = [&](int buf, int d) {
#pragma unroll
        for (int h = 0; h < NA; h++) {
            const int e = tid + 128 * h, q = e % QK, r = (e / QK) ^ (q * (32 / QK));
            As[buf][4 * q + 0][r] = ra[d][h].x;
            As[buf][4 * q + 1][r] = ra[d][h].y;
            As[buf][4 * q + 2][r] = ra[d][h].z;
            As[buf][4 * q + 3][r] = ra[d][h].w;
        }
#pragma unroll
        for (int h = 0; h < NB; h++) {
            const int e = tid + 128 * h, q = e % QK, r = (e / QK) ^ (q * (32 / QK));
            if (BN * QK % 128 == 0 || e < BN * QK) {
                Bs[buf][4 * q + 0][r] = rb[d][h].x;
                Bs[buf][4 * q + 1][r] = rb[d][h].y;
                Bs[buf][4 * q + 2][r] = rb[d][h].z;
                Bs[buf][4 * q + 3][r] = rb[d][h].w;
            }
        }
    };
    uint64_t acc[TM / 2][TN];
#pragma unroll
    for (int i = 0; i < TM / 2; i++)
#pragma unroll
        for (int j = 0; j < TN; j++) acc[i][j] = 0ull;
    const int nk = Kd / BK;
#pragma unroll
    for (int d = 0; d < D; d++)
        if (d < nk) load(d);
    auto tile = [&](int buf) {
#pragma unroll
        for (int kk = 0; kk < BK; kk++) {
            const int f = (kk >> 2) * (32 / QK);
            uint64_t a[TM / 2];
            if (TM >= 4) {
#pragma unroll
                for (int i = 0; i < TM / 4; i++) {
                    const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(
                        &As[buf][kk][32 * i + ((ty * 4) ^ f)]);
                    a[2 * i] = v.x;
                    a[2 * i + 1] = v.y;
                }
            } else {
                a[0] = *reinterpret_cast<const uint64_t*>(&As[buf][kk][(ty * 2) ^ f]);
            }
#pragma unroll
            for (int j = 0; j < TN; j += 2) {
                if (j + 1 < TN) {
                    const float2 v = *reinterpret_cast<const float2*>(
                        &Bs[buf][kk][16 * j + ((2 * tx) ^ f)]);
                    const uint64_t b0 = pack2(v.x, v.x), b1 = pack2(v.y, v.y);
#pragma unroll
                    for (int i = 0; i < TM / 2; i++) {
                        fma2(acc[i][j], a[i], b0);
                        fma2(acc[i][j + 1], a[i], b1);
                    }
                } else {
                    const float v = Bs[buf][kk][16 * j + (tx ^ f)];
                    const uint64_t b0 = pack2(v, v);
#pragma unroll
                    for (int i = 0; i < TM / 2; i++) fma2(acc[i][j], a[i], b0);
                }
            }
        }
    };
    int buf = 0;
    for (int kt = 0; kt < nk; kt += D) {
#pragma unroll
        for (int d = 0; d < D; d++) {
            if (kt + d >= nk) break;
            store(buf, d);
            __syncthreads();
            if (kt + d + D < nk) load(d);
            tile(buf);
            buf ^= 1;
        }
    }
    // epilogue
#pragma unroll
    for (int j = 0; j < TN; j++) {
        const int gj = j0 + ((j | 1) < TN ? 16 * (j & ~1) + 2 * tx + (j & 1) : 16 * j + tx);
        if (gj >= N) continue;
        size_t col = gj;
        if (cGroup > 0) {
            const int l = gj / cGroup;
            col = (size_t)l * cGroupStride + (gj - l * cGroup);
        }
#pragma unroll
        for (int i = 0; i < TM / 2; i++) {
            const float2 v = unpack2(acc[i][j]);
            const int gi = i0 + (TM >= 4 ? 32 * (i >> 1) + ty * 4 + 2 * (i & 1) : ty * 2);
            if (gi < M)
                C[(size_t)gi * ldc + col] = fmaf(alpha, v.x, nrm ? nrm[b * sN + gi] : 0.f);
            if (gi + 1 < M)
                C[(size_t)(gi + 1) * ldc + col] = fmaf(alpha, v.y, nrm ? nrm[b * sN + gi + 1] : 0.f);
        }
    }
}

// ------------------------------------------------------------------------
// Marginal weights of one hypothesis block (a particle, or an image of the
// global scan): base = max D, s = exp(D - base),
//   wR[r] = sum_t s pwC pwT[t], wT[t] = sum_r s pwC pwR[r],
//   wC = sum s pwR[r] pwT[t]
// (the running-baseline accumulation of Optimiser::updateSP,
// src/Optimiser.cpp:1326-1347, evaluated in two passes).  D of block (b, g)
// is D[b sD + r ldc + g nT + t].  One CTA of 512 threads per block; a warp
// takes whole rotation rows (lanes over translations, coalesced), sums wR[r]
// with shuffles, and keeps its share of wT in registers (TS slots of 32
// translations; TS == 0: shared-memory atomics for long rows).  FP32
// accumulation, as in the reference GPU path; totals are combined in FP64.
// Callers with many small blocks (the multi-class scan) may launch fewer
// warps, so that the per-warp fixed work -- reductions, loop set-up -- is
// spread over more rows; the warp count sets the order of the wT sums.
constexpr int WEIGHTS_THREADS = 512;

template <int TS>
__global__ void __launch_bounds__(WEIGHTS_THREADS)
k_weights(const float* __restrict__ D, long long sD, int ldc, int nR, int nT, int G,
          const float* __restrict__ nrmG, int nrmRS, const double* __restrict__ x0,
          const double* __restrict__ pwR, long long sR,
          const double* __restrict__ pwT, long long sT, const double* __restrict__ pwC,
          double* __restrict__ wC, double* __restrict__ wR, double* __restrict__ wT,
          double* __restrict__ base, float* __restrict__ dvp, int nc, const int* __restrict__ best)
{
    extern __shared__ float wsm[];
    float* wTs = wsm;                // [nT]
    float* pTs = wTs + nT;           // [nT]
    float* wTw = pTs + nT;           // [warps][nT] when TS > 0: per-warp sums, added in order
    __shared__ float redf[32];
    __shared__ double red[32];
    // nc > 1: the rows of item blk / nc are cut into nc chunks, one per CTA;
    // wC, wT, base are then per chunk (relative to the chunk's maximum) and
    // k_merge_chunks folds them; wR and dvp rows go straight to the item's
    const int blk = blockIdx.x;
    const int item = blk / nc, chunk = blk % nc;
    const int rpb = (nR + nc - 1) / nc;
    const int r0c = min(nR, chunk * rpb);
    const int nRc = min(nR, r0c + rpb) - r0c;
    const int b = item / G, g = item % G;
    const float* Db = D + b * sD + (size_t)g * nT + (size_t)r0c * ldc;
    const double* pr = pwR + item * sR + r0c;
    const double* pt = pwT + item * sT;
    const double pc = pwC ? pwC[item] : 1.0;
    const float* nrmB = nrmG ? nrmG + (size_t)r0c * nrmRS : nullptr;
    const int nRall = nR;
    nR = nRc;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int t = threadIdx.x; t < nT; t += blockDim.x) {
        wTs[t] = 0.f;
        pTs[t] = (float)pt[t];
    }
    // pass 1: maximum (four rows per warp in flight), unless the GEMM that wrote
    // D found it
    float mx = -CUDART_INF_F;
    for (int r0 = wid; r0 < nR && !best; r0 += 4 * nw) {
        float v[4][TS > 0 ? TS : 1];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int r = r0 + q * nw;
            const float ad = (r < nR && nrmB) ? nrmB[(size_t)r * nrmRS + item] : 0.f;
            const float* row = Db + (size_t)(r < nR ? r : 0) * ldc;
#pragma unroll
            for (int j = 0; j < (TS > 0 ? TS : 1); j++) {
                const int t = lane + 32 * j;
                v[q][j] = (r < nR && t < nT && TS > 0) ? row[t] + ad : -CUDART_INF_F;
            }
            if (TS == 0 && r < nR)
                for (int t = lane; t < nT; t += 32) mx = fmaxf(mx, row[t] + ad);
        }
#pragma unroll
        for (int q = 0; q < 4; q++)
#pragma unroll
            for (int j = 0; j < (TS > 0 ? TS : 1); j++) mx = fmaxf(mx, v[q][j]);
    }
    mx = warp_max(mx);
    if (lane == 0) redf[wid] = mx;
    __syncthreads();
    if (wid == 0) {
        float v = lane < nw ? redf[lane] : -CUDART_INF_F;
        v = warp_max(v);
        if (lane == 0) redf[0] = v;
    }
    __syncthreads();
    const float M = best ? key_float(best[blk]) : redf[0];
    const double x0b = x0 ? x0[item] : 0.0;
    // pass 2: marginals
    float tacc[TS > 0 ? TS : 1], ptv[TS > 0 ? TS : 1];
#pragma unroll
    for (int j = 0; j < (TS > 0 ? TS : 1); j++) {
        tacc[j] = 0.f;
        const int t = lane + 32 * j;
        ptv[j] = (TS > 0 && t < nT) ? pTs[t] : 0.f;
    }
    float cacc = 0.f;
    // Four rows per warp in flight: their loads precede their arithmetic, and
    // their sums over the lanes share the steps of one reduction.  What a row
    // has in FP64 (its prior, its sum) is converted for 32 rows of the warp at
    // once, a lane each: the SM's two FP64 lanes take 16 cycles a warp
    // instruction.  Rows past the end are read as the last one with a prior of 0,
    // translations past the end as the last with a prior of 0: they add zeros.
    // 2,000 blocks of 6,912 x 49: 0.93 ms (with the FP64 pipe 75 % busy and 83
    // instructions a row: 1.38 ms).
    const bool b4 = lane & 16, b3 = lane & 8;
    const float* col[TS > 0 ? TS : 1];
#pragma unroll
    for (int j = 0; j < (TS > 0 ? TS : 1); j++) col[j] = Db + min(lane + 32 * j, nT - 1);
    const size_t step = (size_t)nw * ldc;
    for (int rb = wid; rb < nR; rb += 32 * nw) {
        const int rl = rb + lane * nw;               // the lane's row of the 32
        const float prv = rl < nR ? (float)pr[rl] : 0.f;
        const float adv = nrmB ? nrmB[(size_t)min(rl, nR - 1) * nrmRS + item] : 0.f;
        float sums = 0.f;
        for (int g = 0; g < 8; g++) {
            const int r0 = rb + 4 * g * nw;
            if (r0 >= nR) break;
            float dv[4][TS > 0 ? TS : 1], prr[4], racc[4];
            const bool whole = r0 + 3 * nw < nR;
            size_t off = (size_t)r0 * ldc;
#pragma unroll
            for (int q = 0; q < 4; q++) {
                prr[q] = __shfl_sync(0xffffffffu, prv, 4 * g + q);
                racc[q] = 0.f;
                if (!whole) off = (size_t)min(r0 + q * nw, nR - 1) * ldc;
                if (TS > 0) {
#pragma unroll
                    for (int j = 0; j < (TS > 0 ? TS : 1); j++) dv[q][j] = col[j][off];
                }
                off += step;
            }
            if (nrmB) {
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const float ad = __shfl_sync(0xffffffffu, adv, 4 * g + q);
#pragma unroll
                    for (int j = 0; j < (TS > 0 ? TS : 1); j++) dv[q][j] = TS > 0 ? dv[q][j] + ad : ad;
                }
            } else if (TS == 0) {
#pragma unroll
                for (int q = 0; q < 4; q++) dv[q][0] = 0.f;
            }
            if (dvp && TS > 0) {
#pragma unroll
                for (int q = 0; q < 4; q++)
#pragma unroll
                    for (int j = 0; j < (TS > 0 ? TS : 1); j++)
                        if (r0 + q * nw < nR && lane + 32 * j < nT)
                            dvp[((size_t)item * nRall + r0c + r0 + q * nw) * nT + lane + 32 * j] =
                                (float)(x0b + (double)dv[q][j]);
            }
#pragma unroll
            for (int q = 0; q < 4; q++) {
                if (TS > 0) {
#pragma unroll
                    for (int j = 0; j < (TS > 0 ? TS : 1); j++) {
                        const float sv = __expf(dv[q][j] - M);
                        racc[q] = fmaf(sv, ptv[j], racc[q]);
                        tacc[j] = fmaf(sv, prr[q], tacc[j]);
                    }
                } else if (r0 + q * nw < nR) {
                    const float* row = Db + (size_t)(r0 + q * nw) * ldc;
                    for (int t = lane; t < nT; t += 32) {
                        const float d = row[t] + dv[q][0];
                        const float sv = __expf(d - M);
                        racc[q] = fmaf(sv, pTs[t], racc[q]);
                        atomicAdd(wTs + t, sv * prr[q]);
                        if (dvp)
                            dvp[((size_t)item * nRall + r0c + r0 + q * nw) * nT + t] =
                                (float)(x0b + (double)d);
                    }
                }
            }
            // the four butterfly sums (the same additions as one after another):
            // a lane keeps two rows after the first step, one after the second;
            // lanes 8 q .. 8 q + 7 end with row q's
            float s0 = (b4 ? racc[2] : racc[0]) + __shfl_xor_sync(0xffffffffu, b4 ? racc[0] : racc[2], 16);
            float s1 = (b4 ? racc[3] : racc[1]) + __shfl_xor_sync(0xffffffffu, b4 ? racc[1] : racc[3], 16);
            float sr = (b3 ? s1 : s0) + __shfl_xor_sync(0xffffffffu, b3 ? s0 : s1, 8);
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) sr += __shfl_xor_sync(0xffffffffu, sr, o);
            // a row past the end has a prior of 0, but its sum may be infinite
            if (!whole && r0 + (lane >> 3) * nw >= nR) sr = 0.f;
#pragma unroll
            for (int q = 0; q < 4; q++)      // sum_t s pT[t] pR[r], once per row
                cacc = fmaf(__shfl_sync(0xffffffffu, sr, 8 * q), prr[q], cacc);
            const float mine = __shfl_sync(0xffffffffu, sr, 8 * (lane & 3));
            if (lane >> 2 == g) sums = mine;
        }
        if (rl < nR) wR[(size_t)item * nRall + r0c + rl] = (double)sums * pc;
    }
    if (TS > 0) {
#pragma unroll
        for (int j = 0; j < (TS > 0 ? TS : 1); j++) {
            const int t = lane + 32 * j;
            if (t < nT) wTw[wid * nT + t] = tacc[j];
        }
    }
    __syncthreads();
    for (int t = threadIdx.x; t < nT; t += blockDim.x) {
        float v = wTs[t];
        if (TS > 0) {
            // the warps' sums in warp order: the same bits on every run
            v = 0.f;
            for (int w = 0; w < nw; w++) v += wTw[w * nT + t];
        }
        wT[(size_t)blk * nT + t] = (double)v * pc;
    }
    // every lane holds the same cacc per warp: count lane 0's only
    const double c = block_sum_d(lane == 0 ? (double)cacc : 0.0, red);
    if (threadIdx.x == 0) {
        wC[blk] = c;
        base[blk] = x0b + (double)M;
    }
}

// Fold the weights of class kIdx into the reference's running per-image
// layout: wC [img][nK], wR [img][nK][nR], wT [img][nK][nT] relative to baseL
// (kernel_setBaseLine / kernel_UpdateW of the reference GPU path, with the
// CPU scan's rescale rule, src/Optimiser.cpp:835-898).
// The class's inputs of image l are wCn[l s], wRn[l s nR + r], wTn[l s nT + t],
// basen[l s], s = inStride (1: one class's arrays; nK: a class's column of
// per-(image, class) arrays).
__global__ void k_merge_class(int nK, int kIdx, int nR, int nT,
                              const double* __restrict__ wCn, const double* __restrict__ wRn,
                              const double* __restrict__ wTn, const double* __restrict__ basen,
                              float* __restrict__ wC, float* __restrict__ wR,
                              float* __restrict__ wT, float* __restrict__ baseL, int inStride)
{
    const int l = blockIdx.x;
    const size_t li = (size_t)l * inStride;
    const double bn = basen[li];
    double scaleOld = 0.0, scaleNew = 1.0, newBase = bn;
    if (kIdx > 0) {
        const double bo = baseL[l];
        if (bn > bo) { scaleOld = exp(bo - bn); newBase = bn; }
        else { scaleOld = 1.0; scaleNew = exp(bn - bo); newBase = bo; }
    }
    __syncthreads();
    for (int k = 0; k < nK; k++) {
        const bool cur = (k == kIdx);
        if (!cur && (kIdx == 0 || k > kIdx)) {
            // classes not yet scored: zero on the first class only
            if (kIdx == 0) {
                if (threadIdx.x == 0) wC[(size_t)l * nK + k] = 0.f;
                for (int r = threadIdx.x; r < nR; r += blockDim.x) wR[((size_t)l * nK + k) * nR + r] = 0.f;
                for (int t = threadIdx.x; t < nT; t += blockDim.x) wT[((size_t)l * nK + k) * nT + t] = 0.f;
            }
            continue;
        }
        if (cur) {
            if (threadIdx.x == 0) wC[(size_t)l * nK + k] = (float)(wCn[li] * scaleNew);
            for (int r = threadIdx.x; r < nR; r += blockDim.x)
                wR[((size_t)l * nK + k) * nR + r] = (float)(wRn[li * nR + r] * scaleNew);
            for (int t = threadIdx.x; t < nT; t += blockDim.x)
                wT[((size_t)l * nK + k) * nT + t] = (float)(wTn[li * nT + t] * scaleNew);
        } else if (scaleOld != 1.0) {
            if (threadIdx.x == 0) wC[(size_t)l * nK + k] = (float)(wC[(size_t)l * nK + k] * scaleOld);
            for (int r = threadIdx.x; r < nR; r += blockDim.x)
                wR[((size_t)l * nK + k) * nR + r] = (float)(wR[((size_t)l * nK + k) * nR + r] * scaleOld);
            for (int t = threadIdx.x; t < nT; t += blockDim.x)
                wT[((size_t)l * nK + k) * nT + t] = (float)(wT[((size_t)l * nK + k) * nT + t] * scaleOld);
        }
    }
    if (threadIdx.x == 0) baseL[l] = (float)newBase;
}

// ------------------------------------------------------------------------
// Narrowing + systematic resampling of one axis of one particle per CTA
// (Particle::keepHalfHeightPeak, src/Particle.cpp:1935-1973;
//  Particle::shuffle, :2173-2270; Particle::resample(n, pt), :1275-1463;
//  Particle::normW, :813-820; Particle::setPeakFactor(PAR_R) 3D, :1886-1896).
// Sums and the cumulative sum round as the reference's sequential double
// additions do, term after term (block_seq_sum); the draws use a binary
// search, which finds the same first index with cdf >= u_j as the reference's
// forward scan.  The rank of the peak factor is found by bits of an
// order-preserving integer key, 64 counts over the set instead of n
// comparisons an entry.

// Sequential rounding in parallel.  While s stays in one binade it is m U with
// an integer m < 2^53 and a fixed U, and RN(s + w) = (m + w / U rounded to an
// integer, ties to the even sum) U: a step that adds one of two integers, by
// the parity of m.  Such steps compose (SeqStep), so a block finds every
// partial sum of a window by a scan; the first term that takes m to 2^53 is
// added in FP64, and the next window starts from there in the new binade.  A
// chain of n dependent FP64 additions (about 75 cycles each on this GPU)
// becomes some log2(n) scans.  The whole resampling of 32 sets, with the rank:
// 8,000 terms in 0.31 instead of 4.5 ms, 1,000 in 78 instead of 209 us, 400 in
// 56 instead of 79 us; at 256 (kSeqSerial) the two are level.
struct SeqStep {
    unsigned long long d0, d1;   // what is added to an even / odd m
};
constexpr unsigned long long kSeqTop = 1ull << 53;   // m at the end of the binade
constexpr int kSeqWindow = 1024;                     // terms of a scan: their sum fits 64 bits
constexpr int kSeqSerial = 256;                      // sets summed term by term

// the step of adding w (finite, not negative) in the binade of exponent e
__device__ __forceinline__ SeqStep seq_step(double w, int e)
{
    const unsigned long long b = (unsigned long long)__double_as_longlong(w);
    const int eb = (int)(b >> 52);
    const unsigned long long mw = (b & ((1ull << 52) - 1)) | (eb ? 1ull << 52 : 0ull);
    const int d = e - (eb ? eb : 1);
    if (d < 0) return {mw ? kSeqTop : 0ull, mw ? kSeqTop : 0ull};
    if (d > 53) return {0ull, 0ull};
    const unsigned long long q = mw >> d, rem = mw - (q << d);
    if (2 * rem == (1ull << d)) {              // a tie (d > 0)
        const unsigned long long o = q & 1ull;
        return {q + o, q + 1ull - o};
    }
    const unsigned long long r = q + (2 * rem > (1ull << d) ? 1ull : 0ull);
    return {r, r};
}

__device__ __forceinline__ SeqStep seq_join(SeqStep a, SeqStep b)
{
    return {a.d0 + (a.d0 & 1ull ? b.d1 : b.d0), a.d1 + (a.d1 & 1ull ? b.d0 : b.d1)};
}

__device__ __forceinline__ double seq_value(unsigned long long m, int e)
{
    return __longlong_as_double((long long)(((unsigned long long)(e - 1) << 52) + m));
}

// s + w[0] + w[1] + ... in order (one thread); the loads of the next eight
// terms are under the additions of these
template <bool kAll>
__device__ double serial_sum(double s, const double* __restrict__ w, double* __restrict__ c, int n)
{
    double a[8], b[8];
#pragma unroll
    for (int k = 0; k < 8; k++) a[k] = k < n ? w[k] : 0.0;
    int i = 0;
    for (; i + 8 <= n; i += 8) {
#pragma unroll
        for (int k = 0; k < 8; k++) b[k] = i + 8 + k < n ? w[i + 8 + k] : 0.0;
#pragma unroll
        for (int k = 0; k < 8; k++) {
            s = __dadd_rn(s, a[k]);
            if (kAll) c[i + k] = s;
            a[k] = b[k];
        }
    }
#pragma unroll
    for (int k = 0; k < 8; k++)
        if (i + k < n) {
            s = __dadd_rn(s, a[k]);
            if (kAll) c[i + k] = s;
        }
    return s;
}

// All 256 threads: ((w[0] + w[1]) + w[2]) + ... of shared w [n], n >= 1, and,
// with c (shared, not w), every partial sum.
__device__ __noinline__ double block_seq_sum(const double* __restrict__ w, double* __restrict__ c, int n)
{
    __shared__ SeqStep part[8];
    __shared__ unsigned long long sM;
    __shared__ double sS;
    __shared__ int sAt;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    // small sets, the first terms, and sets with a negative, infinite or NaN
    // term in order
    int first = n;
    if (n > kSeqSerial) {
        bool plain = true;
        for (int i = threadIdx.x; i < n; i += blockDim.x)
            plain &= (unsigned long long)__double_as_longlong(w[i]) < 0x7ff0000000000000ull;
        if (__syncthreads_and(plain)) first = 16;
    }
    if (threadIdx.x == 0) {
        if (c) {
            c[0] = w[0];
            sS = serial_sum<true>(w[0], w + 1, c + 1, first - 1);
        } else {
            sS = serial_sum<false>(w[0], w + 1, nullptr, first - 1);
        }
    }
    __syncthreads();
    double s = sS;
    for (int i0 = first; i0 < n;) {
        const unsigned long long bits = (unsigned long long)__double_as_longlong(s);
        int e = (int)(bits >> 52);
        if (e >= 0x7fe) {                      // the largest binade: no room to test for its end
            if (threadIdx.x == 0) {
                sS = c ? serial_sum<true>(s, w + i0, c + i0, n - i0)
                       : serial_sum<false>(s, w + i0, nullptr, n - i0);
            }
            __syncthreads();
            s = sS;
            break;
        }
        const unsigned long long m = (bits & ((1ull << 52) - 1)) | (e ? 1ull << 52 : 0ull);
        if (e == 0) e = 1;
        // the sum of like terms doubles from i0 to 2 i0
        const int win = min(n - i0, min(kSeqWindow, max((int)blockDim.x, 2 * i0)));
        const int per = (win + blockDim.x - 1) / blockDim.x;
        const int a = i0 + min(win, (int)threadIdx.x * per), b = i0 + min(win, ((int)threadIdx.x + 1) * per);
        SeqStep t = {0ull, 0ull};
        for (int i = a; i < b; i++) t = seq_join(t, seq_step(w[i], e));
        const SeqStep own = t;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            SeqStep u;
            u.d0 = __shfl_up_sync(0xffffffffu, t.d0, o);
            u.d1 = __shfl_up_sync(0xffffffffu, t.d1, o);
            if (lane >= o) t = seq_join(u, t);
        }
        if (lane == 31) part[wid] = t;
        if (threadIdx.x == 0) sAt = n;
        SeqStep before;
        before.d0 = __shfl_up_sync(0xffffffffu, t.d0, 1);
        before.d1 = __shfl_up_sync(0xffffffffu, t.d1, 1);
        if (lane == 0) before = {0ull, 0ull};
        __syncthreads();
        SeqStep all = part[lane & 7];          // the warps before this one
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) {
            SeqStep u;
            u.d0 = __shfl_up_sync(0xffffffffu, all.d0, o, 8);
            u.d1 = __shfl_up_sync(0xffffffffu, all.d1, o, 8);
            if ((lane & 7) >= o) all = seq_join(u, all);
        }
        all.d0 = __shfl_sync(0xffffffffu, all.d0, (wid + 7) & 7);
        all.d1 = __shfl_sync(0xffffffffu, all.d1, (wid + 7) & 7);
        if (wid == 0) all = {0ull, 0ull};
        all = seq_join(all, before);
        unsigned long long mi = m + (m & 1ull ? all.d1 : all.d0);
        const unsigned long long end = mi + (mi & 1ull ? own.d1 : own.d0);
        if (!c && end < kSeqTop) {
            if (b == i0 + win && a < b) sM = end;
        } else if (mi < kSeqTop) {
            for (int i = a; i < b; i++) {
                const SeqStep u = seq_step(w[i], e);
                const unsigned long long mn = mi + (mi & 1ull ? u.d1 : u.d0);
                if (mn >= kSeqTop) {           // one thread finds the binade's end
                    sAt = i;
                    sM = mi;
                    break;
                }
                mi = mn;
                if (c) c[i] = seq_value(mi, e);
                if (i == i0 + win - 1) sM = mi;
            }
        }
        __syncthreads();
        const int at = sAt;
        s = seq_value(sM, e);
        if (at < n) {
            s = __dadd_rn(s, w[at]);
            if (c && threadIdx.x == 0) c[at] = s;
            i0 = at + 1;
        } else {
            i0 += win;
        }
        __syncthreads();
    }
    __syncthreads();
    return s;
}

__global__ void __launch_bounds__(256)
k_resample(int ld, const double* __restrict__ uIn, const double* __restrict__ wIn,
           const int* __restrict__ perm, const double* __restrict__ u0s,
           const double* __restrict__ peaks, int ldo, const int* __restrict__ nPer,
           int* __restrict__ src, double* __restrict__ wOut, int* __restrict__ top,
           int* __restrict__ flag)
{
    // ld / ldo: pitches of the inputs / outputs of a particle; its own set has
    // n = nPer[b] entries (all ld without nPer) and it draws nOut = n of them
    // (ldo without nPer)
    extern __shared__ double sm[];
    double* u = sm;                 // [ld]
    double* w = u + ld;             // [ld]
    double* cdf = w + ld;           // [max(ld, ldo)]
    int* idx = reinterpret_cast<int*>(cdf + (ld > ldo ? ld : ldo));   // [ld]
    __shared__ double sval[32];
    __shared__ int sidx[32];
    __shared__ double sh;
    __shared__ uint2 cnt[2][8];
    __shared__ unsigned long long skey;
    __shared__ int bad;
    const int b = blockIdx.x;
    const int n = nPer ? nPer[b] : ld;
    const int nOut = nPer ? n : ldo;
    const double* ub = uIn + (size_t)b * ld;
    const double* wb = wIn + (size_t)b * ld;
    const int* pb = perm + (size_t)b * ld;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    if (threadIdx.x == 0) bad = 0;
    // maximum of u (exact in any order)
    double mx = -CUDART_INF;
    for (int i = threadIdx.x; i < n; i += blockDim.x) mx = fmax(mx, ub[i]);
    for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if (lane == 0) sval[wid] = mx;
    __syncthreads();
    if (threadIdx.x == 0) {
        double m = sval[0];
        for (int i = 1; i < nw; i++) m = fmax(m, sval[i]);
        sh = m;
    }
    __syncthreads();
    const double umax = sh;
    double pf = peaks ? peaks[b] : 0.0;
    if (isnan(pf)) {
        // value of rank n/8 in descending order (Particle::setPeakFactor):
        // the largest key x with more than n/8 keys >= x; key: the IEEE
        // pattern in unsigned order (negatives reflected).  Small sets count
        // for every entry (n / 8 steps a thread are fewer than the 32 rounds of
        // the search by two bits: 6 against 9 us at n = 256, 58 against 10 at
        // 1,000).
        const int k = n / 8;
        unsigned long long* key = reinterpret_cast<unsigned long long*>(cdf);   // unused yet
        for (int i = threadIdx.x; i < n; i += blockDim.x) {
            const double x = ub[i];
            const long long bits = __double_as_longlong(x == 0.0 ? 0.0 : x);
            key[i] = (unsigned long long)(bits ^ (bits >> 63 | (long long)0x8000000000000000ull));
        }
        __syncthreads();
        unsigned long long x = 0ull;
        if (n <= 256) {
            if (threadIdx.x < n) {
                const unsigned long long v = key[threadIdx.x];
                int gt = 0, ge = 0;
                for (int j = 0; j < n; j++) {
                    gt += key[j] > v;
                    ge += key[j] >= v;
                }
                if (gt <= k && k < ge) skey = v;     // all writers store the same value
            }
            __syncthreads();
            x = skey;
        } else {
            for (int bit = 62; bit >= 0; bit -= 2) {
                // how many keys reach x + 1, 2 and 3 steps (counts below 2^16)
                const unsigned long long c1 = x | 1ull << bit, c2 = x | 2ull << bit,
                                         c3 = x | 3ull << bit;
                unsigned g12 = 0, g3 = 0;
                for (int i = threadIdx.x; i < n; i += blockDim.x) {
                    const unsigned long long v = key[i];
                    g12 += (v >= c1 ? 1u : 0u) + (v >= c2 ? 65536u : 0u);
                    g3 += v >= c3;
                }
                g12 = __reduce_add_sync(0xffffffffu, g12);
                g3 = __reduce_add_sync(0xffffffffu, g3);
                uint2* c = cnt[bit >> 1 & 1];
                if (lane == 0) c[wid] = make_uint2(g12, g3);
                __syncthreads();
                uint2 t = c[lane & 7];
                t.x = __reduce_add_sync(0xffffffffu, lane < 8 ? t.x : 0u);
                t.y = __reduce_add_sync(0xffffffffu, lane < 8 ? t.y : 0u);
                x = (int)t.y > k ? c3 : (int)(t.x >> 16) > k ? c2 : (int)(t.x & 65535u) > k ? c1 : x;
            }
        }
        const unsigned long long back = x & 0x8000000000000000ull ? x ^ 0x8000000000000000ull : ~x;
        const double ranked = __longlong_as_double((long long)back);
        __syncthreads();               // the keys' storage becomes the cumulative sum
        const double r = __ddiv_rn(ranked, umax);
        pf = fmax(1e-3, fmin(0.5, r));
    }
    const double hh = pf > 0 ? __dmul_rn(umax, pf) : 0.0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        double ui = ub[i];
        if (pf > 0) ui = (ui < hh) ? 0.0 : __dsub_rn(ui, hh);
        const int d = pb[i];
        if (d < 0 || d >= n) { bad = 1; continue; }
        u[d] = ui;
        w[d] = wb[i];
        idx[d] = i;
    }
    __syncthreads();
    if (bad) {
        if (threadIdx.x == 0) atomicOr(flag, 1);
        return;
    }
    // best sample, last index among equal maxima (gsl_sort_largest_index)
    double bv = -CUDART_INF;
    int bi = -1;
    for (int i = threadIdx.x; i < n; i += blockDim.x)
        if (u[i] >= bv) { bv = u[i]; bi = i; }
    for (int o = 16; o > 0; o >>= 1) {
        double ov = __shfl_xor_sync(0xffffffffu, bv, o);
        int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (ov > bv || (ov == bv && oi > bi)) { bv = ov; bi = oi; }
    }
    if (lane == 0) { sval[wid] = bv; sidx[wid] = bi; }
    __syncthreads();
    if (threadIdx.x == 0) {
        double v = sval[0];
        int ii = sidx[0];
        for (int i = 1; i < nw; i++)
            if (sval[i] > v || (sval[i] == v && sidx[i] > ii)) { v = sval[i]; ii = sidx[i]; }
        top[b] = ii >= 0 ? idx[ii] : 0;
    }
    for (int i = threadIdx.x; i < n; i += blockDim.x) w[i] = __dmul_rn(w[i], u[i]);
    __syncthreads();
    const double ws = block_seq_sum(w, nullptr, n);
    if (!(ws > 0.0)) {
        if (threadIdx.x == 0) atomicOr(flag, 2);
        return;
    }
    for (int i = threadIdx.x; i < n; i += blockDim.x) w[i] = __ddiv_rn(w[i], ws);
    __syncthreads();
    const double last = block_seq_sum(w, cdf, n);
    for (int i = threadIdx.x; i < n; i += blockDim.x) cdf[i] = __ddiv_rn(cdf[i], last);
    __syncthreads();
    const double u0 = u0s[b];
    int* so = src + (size_t)b * ldo;
    for (int j = threadIdx.x; j < nOut; j += blockDim.x) {
        const double uj = __dadd_rn(u0, __ddiv_rn((double)j, (double)nOut));
        int lo = 0, hi = n - 1;       // first i with cdf[i] >= uj
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (uj > cdf[mid]) lo = mid + 1; else hi = mid;
        }
        so[j] = idx[lo];
        // new prior 1 / u of the source (PARTICLE_PRIOR_ONE), in place of w
        // (its values are in cdf), the overhang of nOut > n in the output
        const double v = __ddiv_rn(1.0, u[lo]);
        if (j < n) w[j] = v;
        else wOut[(size_t)b * ldo + j] = v;
    }
    __syncthreads();
    double s2 = block_seq_sum(w, nullptr, min(n, nOut));
    if (nOut > n) {
        if (threadIdx.x == 0) {
            for (int j = n; j < nOut; j++) s2 = __dadd_rn(s2, wOut[(size_t)b * ldo + j]);
            sh = s2;
        }
        __syncthreads();
        s2 = sh;
    }
    for (int j = threadIdx.x; j < nOut; j += blockDim.x)
        wOut[(size_t)b * ldo + j] = __ddiv_rn(j < n ? w[j] : wOut[(size_t)b * ldo + j], s2);
}

// ------------------------------------------------------------------------
// Insertion of one weighted, shifted slice per CTA into the interleaved
// (F.re, F.im, T, 0) accumulator (Reconstructor::insertP,
// src/Reconstructor.cpp:782-863).  The image is first shifted by
// -(t - offset) (translate, src/Image/ImageFunctions.cpp:471-492, as in
// Optimiser::reconstructRef, src/Optimiser.cpp:7115-7136).
//   MKB: every voxel with tab[rint(r^2 n / b)] != 0 inside the radius
//        (Volume::addFT(value, x, y, z, a, TabFunction),
//        src/Image/Volume.cpp:399-431; entries past the kernel support are
//        zero, so the loop covers only the support);
//   trilinear: the eight corners (Volume::addFT(value, x, y, z),
//        src/Image/Volume.cpp:334-369).
// Voxels with x < 0 are mirrored and conjugated (Volume::iFT).
// Per-draw parameters of the insertion, one thread per draw: the FP32
// rotation (quat_to_mat in FP64, rounded), the shift t - offset and the
// image weight, 16 floats per draw; and the bookkeeping: O3D -= R (t -
// offset, 0) (insertDir, src/Optimiser.cpp:7180-7186), summed per block
// before one atomic per component, and the draw counter.
// With nC (the multi-class InsertFT), draw m of image l is inserted only
// when m < nC[l] (kernel_getRandomR / kernel_InsertF, gpu/src/Kernel.cu:
// 1847-1899, 2552-2600): a skipped draw gets weight 0, which the insertion
// skips, and adds nothing to O3D or the counter.
__global__ void __launch_bounds__(256)
k_insert_draws(int nDraws, int drawsPerImage, const double* __restrict__ quat,
               const double* __restrict__ trans, const double* __restrict__ offset,
               const float* __restrict__ wgt, float* __restrict__ params,
               double* __restrict__ O3D, int* __restrict__ counter, const int* __restrict__ nC)
{
    __shared__ double part[3][8];
    const int d = blockIdx.x * blockDim.x + threadIdx.x;
    // the insertion's work counter, after the draws
    if (d == 0) *reinterpret_cast<unsigned long long*>(params + 16 * (size_t)nDraws) = 0ull;
    double o[3] = {0.0, 0.0, 0.0};
    const bool active = d < nDraws && (!nC || d % drawsPerImage < nC[d / drawsPerImage]);
    if (d < nDraws && !active) {
        float* pd = params + 16 * (size_t)d;
        for (int i = 0; i < 12; i++) pd[i] = 0.f;
    }
    if (active) {
        const int l = d / drawsPerImage;
        double q[4] = {quat[4 * (size_t)d], quat[4 * (size_t)d + 1], quat[4 * (size_t)d + 2],
                       quat[4 * (size_t)d + 3]};
        double md[9];
        quat_to_mat(q, md);
        const double tx = trans[2 * (size_t)d] - (offset ? offset[2 * (size_t)l] : 0.0);
        const double ty = trans[2 * (size_t)d + 1] - (offset ? offset[2 * (size_t)l + 1] : 0.0);
        float* pd = params + 16 * (size_t)d;
        for (int i = 0; i < 9; i++) pd[i] = (float)md[i];
        pd[9] = (float)tx;
        pd[10] = (float)ty;
        pd[11] = wgt[l];
        o[0] = -(md[0] * tx + md[1] * ty);
        o[1] = -(md[3] * tx + md[4] * ty);
        o[2] = -(md[6] * tx + md[7] * ty);
    }
    if (O3D) {
        const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
        for (int k = 0; k < 3; k++) {
            double v = o[k];
            for (int sft = 16; sft; sft >>= 1) v += __shfl_xor_sync(0xffffffffu, v, sft);
            if (lane == 0) part[k][wid] = v;
        }
        __syncthreads();
        if (threadIdx.x < 3) {
            double v = 0.0;
            for (int w = 0; w < (int)(blockDim.x >> 5); w++) v += part[threadIdx.x][w];
            atomicAdd(O3D + threadIdx.x, v);
        }
    }
    if (counter) {
        const int n = __syncthreads_count(active);
        if (threadIdx.x == 0 && n > 0) atomicAdd(counter, n);
    }
}

// A draw's pixel: its value times CTF and weight, shifted by -(t - offset) (times
// exp(+2 pi i k.t / N)), its CTF^2 and weight, its place in the volume.
struct InsertPixel {
    float vr, vi, vt, x, y, z;
};

struct InsertData {          // what a draw has at a pixel
    float2 X;
    float c;
    int col, row;
};

__device__ __forceinline__ InsertData insert_load(const float2* __restrict__ dat,
                                                  const float* __restrict__ ctf,
                                                  const int* __restrict__ iCol,
                                                  const int* __restrict__ iRow, int K, int d, int l,
                                                  int ctfPerDraw, int p)
{
    return {__ldg(dat + (size_t)l * K + p), __ldg(ctf + (ctfPerDraw ? (size_t)d : (size_t)l) * K + p),
            __ldg(iCol + p), __ldg(iRow + p)};
}

__device__ __forceinline__ InsertPixel insert_pixel(const InsertData& q,
                                                    const float* __restrict__ pd, int pf, int idim)
{
    InsertPixel o;
    const float tx = __ldg(pd + 9), ty = __ldg(pd + 10), w = __ldg(pd + 11);
    const float invN = 1.0f / (float)idim, fpf = (float)pf;
    const float f = ((float)q.col * tx + (float)q.row * ty) * invN;
    float s, co;
    sincospif(2.0f * f, &s, &co);
    const float cw = q.c * w;
    o.vr = (q.X.x * co - q.X.y * s) * cw;
    o.vi = (q.X.x * s + q.X.y * co) * cw;
    o.vt = q.c * q.c * w;
    const float a = (float)q.col * fpf, b = (float)q.row * fpf;
    o.x = __ldg(pd + 0) * a + __ldg(pd + 1) * b;
    o.y = __ldg(pd + 3) * a + __ldg(pd + 4) * b;
    o.z = __ldg(pd + 6) * a + __ldg(pd + 7) * b;
    return o;
}

// Trilinear insertion.  CTA (share of the pixels, draw); parameters from
// k_insert_draws.
__global__ void __launch_bounds__(256)
k_insert(float4* __restrict__ acc, int vdim, const float2* __restrict__ dat,
         const float* __restrict__ ctf, const float* __restrict__ params,
         const int* __restrict__ iCol, const int* __restrict__ iRow, int K, int pf, int idim,
         int d0, int drawsPerImage, int ctfPerDraw)
{
    const int d = d0 + blockIdx.y;            // draw; blockIdx.x: share of its pixels
    const float* pd = params + 16 * (size_t)d;
    if (__ldg(pd + 11) == 0.f) return;        // a skipped draw (or one of weight 0)
    const int nx = vdim / 2 + 1;
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < K; p += gridDim.x * blockDim.x) {
        InsertPixel v = insert_pixel(
            insert_load(dat, ctf, iCol, iRow, K, d, d / drawsPerImage, ctfPerDraw, p), pd, pf, idim);
        if (v.x < 0.f) { v.x = -v.x; v.y = -v.y; v.z = -v.z; v.vi = -v.vi; }
        const float xf = floorf(v.x), yf = floorf(v.y), zf = floorf(v.z);
        const int x0 = (int)xf, y0 = (int)yf, z0 = (int)zf;
        const float fx = v.x - xf, fy = v.y - yf, fz = v.z - zf;
        const float wx[2] = {1.f - fx, fx}, wy[2] = {1.f - fy, fy}, wz[2] = {1.f - fz, fz};
#pragma unroll
        for (int k = 0; k < 2; k++)
#pragma unroll
            for (int j = 0; j < 2; j++)
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    const float ww = wx[i] * wy[j] * wz[k];
                    int yy = y0 + j, zz = z0 + k;
                    yy = yy < 0 ? yy + vdim : yy;
                    zz = zz < 0 ? zz + vdim : zz;
                    atomicAdd(acc + ((size_t)zz * vdim + yy) * nx + (x0 + i),
                              make_float4(v.vr * ww, v.vi * ww, v.vt * ww, 0.f));
                }
    }
}

// MKB insertion: every voxel within the support of a pixel's place gets the
// pixel's value times the kernel's table at rint(r^2 n / b) (entries 0 ..
// tabNz).  The support is less than 4 voxels wide, so the candidates are the 4^3
// from ceil(x - rs).  Four lanes take a pixel, a lane one column of candidates
// along x and its 16 rows: a warp's atomics then come as runs of up to four
// neighbouring float4, a request of L2 instead of four, and what a lane works
// out for a column (its distance, its side of x = 0) serves 16 voxels.  Voxels
// of x < 0 are their Friedel mates: a lane of such a column takes the negative
// rows.  The table (100 KB at padding 2) is looked up in shared memory (kShared;
// padding 1 has 400 KB and leaves it in L2): the latency of lookups that missed
// the L1 was what the insertion waited for.  Persistent; a warp takes 64 pixels
// of a draw at a time from a counter (the SMs do not all get the same share of
// L2: in equal shares the slowest ran a quarter longer than the mean), the next
// pixel's data loaded behind the atomics.  2,000 draws of 9,930 pixels: 2.86 ms
// (a thread a pixel, lookups and rows one after another: 4.85 ms).
// With `order`, the runs of 8 pixels sorted by radius, the items go by radius
// first and draws second: the warps then work in one shell of the volume, which
// stays in L2, where whole draws one after another touch all of it (142 MB at
// radius 160).
constexpr int kInsertThreads = 1024;
constexpr int kInsertItem = 64;
constexpr int kInsertRun = 8;
constexpr size_t kInsertL2 = (size_t)48 << 20;

// order[i] = the run of i-th radius (of its middle pixel), equal ones in their
// own order: a thread a run, its rank counted over all of them.
__global__ void __launch_bounds__(256)
k_insert_order(const int* __restrict__ iCol, const int* __restrict__ iRow, int K, int nRuns,
               int* __restrict__ order)
{
    __shared__ int key[1024];
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    auto radius = [&](int q) {
        const int p = min(q * kInsertRun + kInsertRun / 2, K - 1);
        return q < nRuns ? iCol[p] * iCol[p] + iRow[p] * iRow[p] : INT_MAX;
    };
    const int mine = radius(r);
    int rank = 0;
    for (int q0 = 0; q0 < nRuns; q0 += 1024) {
        __syncthreads();
        for (int i = threadIdx.x; i < 1024; i += blockDim.x) key[i] = radius(q0 + i);
        __syncthreads();
#pragma unroll 16
        for (int i = 0; i < 1024; i++)
            rank += key[i] < mine || (key[i] == mine && q0 + i < r) ? 1 : 0;
    }
    if (r < nRuns) order[rank] = r;
}

template <bool kShared>
__global__ void __launch_bounds__(kInsertThreads, 1)
k_insert_mkb(float4* __restrict__ acc, int vdim, const float* __restrict__ tabG, int tabNz,
             float tabInvStep, float rs, const float2* __restrict__ dat,
             const float* __restrict__ ctf, const float* __restrict__ params,
             const int* __restrict__ iCol, const int* __restrict__ iRow, int K, int pf, int idim,
             int nDraws, int drawsPerImage, int ctfPerDraw, unsigned long long* __restrict__ next,
             const int* __restrict__ order)
{
    extern __shared__ float tabS[];              // [tabNz + 1]
    if (kShared) {
        for (int i = threadIdx.x; i <= tabNz; i += blockDim.x) tabS[i] = tabG[i];
        __syncthreads();
    }
    const float* tab = kShared ? tabS : tabG;
    const int nx = vdim / 2 + 1, half = vdim / 2;
    const int lane = threadIdx.x & 31;
    const int tiles = (K + kInsertItem - 1) / kInsertItem;
    const unsigned long long items = (unsigned long long)tiles * nDraws;
    for (;;) {
        unsigned long long it = lane ? 0 : atomicAdd(next, 1ull);
        it = __shfl_sync(0xffffffffu, it, 0);
        if (it >= items) break;
        const int d = (int)(order ? it % nDraws : it / tiles), l = d / drawsPerImage;
        const int tile = (int)(order ? it / nDraws : it % tiles);
        const float* pd = params + 16 * (size_t)d;
        if (__ldg(pd + 11) == 0.f) continue;     // a skipped draw (or one of weight 0)
        // lanes 0 - 7: the item's runs
        int run = tile * (kInsertItem / kInsertRun) + (lane & 7);
        if (order) run = run * kInsertRun < K ? __ldg(order + run) : K;
        int p = __shfl_sync(0xffffffffu, run, 0) * kInsertRun + lane / 4;
        InsertData data = insert_load(dat, ctf, iCol, iRow, K, d, l, ctfPerDraw, min(p, K - 1));
        for (int g = 1; g <= kInsertItem / kInsertRun; g++) {
            const bool in = p < K;
            const InsertPixel v = insert_pixel(data, pd, pf, idim);
            p = __shfl_sync(0xffffffffu, run, g & 7) * kInsertRun + lane / 4;
            data = insert_load(dat, ctf, iCol, iRow, K, d, l, ctfPerDraw, min(p, K - 1));
            if (!in) continue;
            const int i = (int)ceilf(v.x - rs) + (threadIdx.x & 3);
            const int j0 = (int)ceilf(v.y - rs), k0 = (int)ceilf(v.z - rs);
            // a candidate outside the volume is out of reach
            const float far = 1e15f;
            const float dx = abs(i) <= half ? v.x - (float)i : far;
            const int side = i < 0 ? -1 : 1;
            const float vi = i < 0 ? -v.vi : v.vi;
            float dy[4];
            int row[4];
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const int j = j0 + u, y = side * j;
                dy[u] = j >= -half && j < half ? v.y - (float)j : far;
                row[u] = (y < 0 ? y + vdim : y) * nx + abs(i);
            }
#pragma unroll 2
            for (int s = 0; s < 4; s++) {
                const int k = k0 + s, z = side * k;
                const float dz = k >= -half && k < half ? v.z - (float)k : far;
                float4* plane = acc + (size_t)(z < 0 ? z + vdim : z) * vdim * nx;
                unsigned ti[4];
                float kv[4];
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const float dyz = fmaf(dy[u], dy[u], dz * dz);
                    // rint by the addition of 1.5 2^23 (not a number, or out of
                    // reach: past the table)
                    const float t = __fmul_rn(fmaf(dx, dx, dyz), tabInvStep);
                    ti[u] = t < 4e6f ? __float_as_uint(__fadd_rn(t, 12582912.f)) - 0x4b400000u : ~0u;
                    const unsigned at = min(ti[u], (unsigned)tabNz);
                    kv[u] = kShared ? tab[at] : __ldg(tab + at);
                }
#pragma unroll
                for (int u = 0; u < 4; u++)
                    if (ti[u] <= (unsigned)tabNz)
                        atomicAdd(plane + row[u],
                                  make_float4(v.vr * kv[u], vi * kv[u], v.vt * kv[u], 0.f));
            }
        }
    }
}

// ------------------------------------------------------------------------
// MKB insertion as a gather (same sums as k_insert, one atomic per voxel).
//
// Stage: CTA (tile, draw) writes cells of the draw's dense half-plane grid
// [2 Rg + 1 rows][Rg + 1 columns] of float4: the shifted, weighted value
// (c w X e^{2 pi i k.t/N}, c^2 w) of the cell's pixel, zero where no pixel
// lies (cellPix < 0).  CTA (0, draw) also writes the draw's FP32 rotation
// and does its bookkeeping (O3D, counter) exactly as k_insert.
__global__ void __launch_bounds__(256)
k_insert_stage(float4* __restrict__ grid, int cells, float* __restrict__ rot,
               const int* __restrict__ cellPix, const int* __restrict__ iCol,
               const int* __restrict__ iRow, const float2* __restrict__ dat,
               const float* __restrict__ ctf, const double* __restrict__ quat,
               const double* __restrict__ trans, const double* __restrict__ offset,
               const float* __restrict__ wgt, int K, int idim, int d0, int drawsPerImage,
               int ctfPerDraw, double* __restrict__ O3D, int* __restrict__ counter)
{
    const int dl = blockIdx.y;                // draw within the chunk
    const int d = d0 + dl;
    const int l = d / drawsPerImage;
    const double txd = trans[2 * (size_t)d] - (offset ? offset[2 * (size_t)l] : 0.0);
    const double tyd = trans[2 * (size_t)d + 1] - (offset ? offset[2 * (size_t)l + 1] : 0.0);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        double q[4] = {quat[4 * (size_t)d], quat[4 * (size_t)d + 1], quat[4 * (size_t)d + 2],
                       quat[4 * (size_t)d + 3]};
        double md[9];
        quat_to_mat(q, md);
        for (int i = 0; i < 9; i++) rot[16 * (size_t)dl + i] = (float)md[i];
        if (O3D) {
            atomicAdd(O3D + 0, -(md[0] * txd + md[1] * tyd));
            atomicAdd(O3D + 1, -(md[3] * txd + md[4] * tyd));
            atomicAdd(O3D + 2, -(md[6] * txd + md[7] * tyd));
        }
        if (counter) atomicAdd(counter, 1);
    }
    const float tx = (float)txd, ty = (float)tyd, w = wgt[l];
    const float invN = 1.0f / (float)idim;
    float4* g = grid + (size_t)dl * cells;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < cells; i += gridDim.x * blockDim.x) {
        const int p = cellPix[i];
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (p >= 0) {
            const size_t di = (size_t)l * K + p;
            const float c = ctf[(ctfPerDraw ? (size_t)d : (size_t)l) * K + p];
            const float2 X = dat[di];
            float f = ((float)iCol[p] * tx + (float)iRow[p] * ty) * invN;
            float sn, co;
            sincospif(2.0f * f, &sn, &co);
            const float cw = c * w;
            v = make_float4((X.x * co - X.y * sn) * cw, (X.x * sn + X.y * co) * cw, c * c * w,
                            0.f);
        }
        g[i] = v;
    }
}

// Gather: CTA (tile, draw); each thread takes rows (x-runs of fixed y, z) of
// the stored half volume that cross the draw's slab |h| <= hs, h = e3 . v,
// inside the cylinder of in-plane radius Rp + hs.  Each voxel v = (x, y, z)
// takes its plane coordinates (a, b, h) = R^T v and sums the MKB-weighted
// values of the grid cells within the support: a pixel (c, r) at
// (pf c, pf r, 0) directly, and, for x > 0, the Friedel mate of pixel (c, r)
// at (-pf c, -pf r, 0), conjugated.  This is the set of writes k_insert
// makes to v (direct writes to x >= 0, mirrored writes from x < 0 to x > 0).
__global__ void __launch_bounds__(256, 4)
k_insert_gather(float4* __restrict__ acc, int vdim, const float4* __restrict__ grid, int gw,
                int Rg, const float* __restrict__ rot, const float* __restrict__ tab, int tabNz,
                float tabInvStep, int pf, float Rp, float hs)
{
    const int dl = blockIdx.y;
    const float* mr = rot + 16 * (size_t)dl;
    const float e1x = __ldg(mr + 0), e1y = __ldg(mr + 3), e1z = __ldg(mr + 6);
    const float e2x = __ldg(mr + 1), e2y = __ldg(mr + 4), e2z = __ldg(mr + 7);
    const float e3x = __ldg(mr + 2), e3y = __ldg(mr + 5), e3z = __ldg(mr + 8);
    const float4* g = grid + (size_t)dl * gw * (2 * Rg + 1);
    const int half = vdim / 2, nx = half + 1;
    const float Rc = Rp + hs;                           // cylinder radius
    const float R2 = Rc * Rc + hs * hs;                 // |v|^2 bound
    const int Y = min(half - 1, (int)ceilf(Rc * sqrtf(fmaxf(0.f, 1.f - e3y * e3y)) +
                                           hs * fabsf(e3y)));
    const int Z = min(half - 1, (int)ceilf(Rc * sqrtf(fmaxf(0.f, 1.f - e3z * e3z)) +
                                           hs * fabsf(e3z)));
    const int ny = 2 * Y + 1;
    const int nRows = ny * (2 * Z + 1);
    const float fpf = (float)pf, inv_pf = 1.0f / fpf;

    for (int row = blockIdx.x * blockDim.x + threadIdx.x; row < nRows;
         row += gridDim.x * blockDim.x) {
        const int y = row % ny - Y, z = row / ny - Z;
        const float fy = (float)y, fz = (float)z;
        const float rem = R2 - fy * fy - fz * fz;
        if (rem < 0.f) continue;
        const float hyz = e3y * fy + e3z * fz;
        float lo = 0.f, hi = fminf(sqrtf(rem), (float)(half - 1));
        if (fabsf(e3x) > 1e-6f) {
            const float ta = (-hs - hyz) / e3x, tb = (hs - hyz) / e3x;
            lo = fmaxf(lo, fminf(ta, tb));
            hi = fminf(hi, fmaxf(ta, tb));
        } else if (fabsf(hyz) > hs) {
            continue;
        }
        if (hi < lo) continue;
        const int xa = max((int)ceilf(lo - 1e-3f), 0);
        const int xb = min((int)floorf(hi + 1e-3f), half - 1);
        const float ayz = e1y * fy + e1z * fz, byz = e2y * fy + e2z * fz;
        float4* line = acc + ((size_t)(z < 0 ? z + vdim : z) * vdim + (y < 0 ? y + vdim : y)) * nx;
        for (int x = xa; x <= xb; x++) {
            const float fx = (float)x;
            const float a = fmaf(e1x, fx, ayz);
            const float b = fmaf(e2x, fx, byz);
            const float h = fmaf(e3x, fx, hyz);
            const float h2 = h * h;
            const int c0 = (int)ceilf((a - hs) * inv_pf), c1 = (int)floorf((a + hs) * inv_pf);
            const int q0 = max((int)ceilf((b - hs) * inv_pf), -Rg);
            const int q1 = min((int)floorf((b + hs) * inv_pf), Rg);
            float sr = 0.f, si = 0.f, st = 0.f;
            for (int c = c0; c <= c1; c++) {
                const float dx = a - fpf * (float)c;
                const float dx2h = fmaf(dx, dx, h2);
                for (int r = q0; r <= q1; r++) {
                    const float dy = b - fpf * (float)r;
                    const int ti = __float2int_rn(fmaf(dy, dy, dx2h) * tabInvStep);
                    if (ti > tabNz) continue;
                    const float kv = __ldg(tab + ti);
                    if (c >= 0 && c <= Rg) {
                        const float4 v = __ldg(g + (r + Rg) * gw + c);
                        sr = fmaf(kv, v.x, sr);
                        si = fmaf(kv, v.y, si);
                        st = fmaf(kv, v.z, st);
                    }
                    if (x > 0 && c <= 0 && -c <= Rg) {
                        const float4 v = __ldg(g + (Rg - r) * gw - c);
                        sr = fmaf(kv, v.x, sr);
                        si = fmaf(-kv, v.y, si);
                        st = fmaf(kv, v.z, st);
                    }
                }
            }
            if (sr != 0.f || si != 0.f || st != 0.f)
                atomicAdd(line + x, make_float4(sr, si, st, 0.f));
        }
    }
}

// ------------------------------------------------------------------------
// Projection banks: one class's projections at a fixed rotation set, made
// once (k_project) and gathered by index for every particle that uses them.
// Planes: hi = bf16(x), lo = bf16(x - hi), the rounding of the split store.
__global__ void k_bank_planes(const float* __restrict__ f32, int nB, int K, int Kp,
                              __nv_bfloat16* __restrict__ hi, __nv_bfloat16* __restrict__ lo,
                              float* __restrict__ abs2)
{
    const size_t pairs = (size_t)nB * (Kp / 2);
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < pairs;
         i += (size_t)gridDim.x * blockDim.x) {
        const size_t row = i / (Kp / 2);
        const int p = (int)(i % (Kp / 2));
        const float2 v = reinterpret_cast<const float2*>(f32 + row * Kp)[p];
        __nv_bfloat162 h = __floats2bfloat162_rn(v.x, v.y);
        const float2 hf = __bfloat1622float2(h);
        reinterpret_cast<__nv_bfloat162*>(hi + row * Kp)[p] = h;
        reinterpret_cast<__nv_bfloat162*>(lo + row * Kp)[p] =
            __floats2bfloat162_rn(v.x - hf.x, v.y - hf.y);
        if (p < K) abs2[row * K + p] = v.x * v.x + v.y * v.y;
    }
}

// CTA (particle, group of 64 rows): w = sigRcp ctf^2 of the particle in
// shared memory; a warp per row copies the bank row in 16-byte units and
// sums its norm with shuffles.
constexpr int kBankRows = 64;

__global__ void __launch_bounds__(256)
k_bank_gather(const BankView* __restrict__ table, const int* __restrict__ cls,
              const int* __restrict__ idx, int nR, int K, int Kp,
              const float* __restrict__ sigRcp, const float* __restrict__ ctf,
              float* __restrict__ P, long long splitLo, float* __restrict__ nrm,
              int* __restrict__ flag)
{
    extern __shared__ float w[];                 // [K]
    const int l = blockIdx.x;
    const BankView b = table[cls ? cls[l] : 0];
    for (int p = threadIdx.x; p < K; p += blockDim.x) {
        const float c = ctf[(size_t)l * K + p];
        w[p] = sigRcp[(size_t)l * K + p] * c * c;
    }
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int j1 = min(nR, (blockIdx.y + 1) * kBankRows);
    const int n16 = Kp / 4;                      // 16-byte units of a row (4 floats / 8 bf16)
    for (int j = blockIdx.y * kBankRows + warp; j < j1; j += 8) {
        const size_t row = (size_t)l * nR + j;
        const int r = idx[row];
        const bool ok = r >= 0 && r < b.nB;
        if (!ok && lane == 0) atomicOr(flag, 1 << 16);
        const size_t rs = (size_t)(ok ? r : 0);
        if (splitLo == 0) {
            const float4* src = reinterpret_cast<const float4*>(b.f32 + rs * Kp);
            float4* dst = reinterpret_cast<float4*>(P + row * Kp);
            for (int u = lane; u < n16; u += 32)
                dst[u] = ok ? __ldg(src + u) : make_float4(0.f, 0.f, 0.f, 0.f);
        } else {
            __nv_bfloat16* hp = reinterpret_cast<__nv_bfloat16*>(P);
            const uint4* sh = reinterpret_cast<const uint4*>(b.hi + rs * Kp);
            const uint4* sl = reinterpret_cast<const uint4*>(b.lo + rs * Kp);
            uint4* dh = reinterpret_cast<uint4*>(hp + row * Kp);
            uint4* dl = reinterpret_cast<uint4*>(hp + splitLo + row * Kp);
            const uint4 z = make_uint4(0u, 0u, 0u, 0u);
            for (int u = lane; u < n16 / 2; u += 32) {
                dh[u] = ok ? __ldg(sh + u) : z;
                dl[u] = ok ? __ldg(sl + u) : z;
            }
        }
        float acc = 0.f;
        if (ok) {
            const float* a2 = b.abs2 + rs * K;
            for (int p = lane; p < K; p += 32) acc = fmaf(w[p], __ldg(a2 + p), acc);
        }
        for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if (lane == 0) nrm[row] = acc;
    }
}

// Fourier shell correlation of two half volumes [vdim][vdim][vdim/2+1] of
// complex values (FSC(vec&, const Volume&, const Volume&),
// src/Functions/Spectrum.cpp:302-329): shell u = rint(|k|) in voxel units,
// for u < nShell, of sum Re(A conj B), sum |A|^2, sum |B|^2 in FP64.  Each
// CTA sums its voxels per shell in shared memory, then adds its shells once.
__global__ void __launch_bounds__(256)
k_fsc_shells(const float2* __restrict__ A, const float2* __restrict__ B, int vdim, int nShell,
             double* __restrict__ sums)
{
    extern __shared__ double sacc[];             // [3][nShell]
    for (int i = threadIdx.x; i < 3 * nShell; i += blockDim.x) sacc[i] = 0.0;
    __syncthreads();
    const int nx = vdim / 2 + 1, half = vdim / 2;
    const size_t n = (size_t)vdim * vdim * nx;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
         i += (size_t)gridDim.x * blockDim.x) {
        const int x = (int)(i % nx);
        const size_t zy = i / nx;
        const int y = (int)(zy % vdim), z = (int)(zy / vdim);
        const int fy = y < half ? y : y - vdim, fz = z < half ? z : z - vdim;
        const int u = __double2int_rn(sqrt((double)x * x + (double)fy * fy + (double)fz * fz));
        if (u >= nShell) continue;
        const float2 a = A[i], b = B[i];
        atomicAdd(sacc + u, (double)a.x * b.x + (double)a.y * b.y);
        atomicAdd(sacc + nShell + u, (double)a.x * a.x + (double)a.y * a.y);
        atomicAdd(sacc + 2 * nShell + u, (double)b.x * b.x + (double)b.y * b.y);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 3 * nShell; i += blockDim.x)
        if (sacc[i] != 0.0) atomicAdd(sums + i, sacc[i]);
}

__global__ void k_fsc_finish(const double* __restrict__ sums, int nShell, double* __restrict__ fsc)
{
    const int u = blockIdx.x * blockDim.x + threadIdx.x;
    if (u >= nShell) return;
    const double xy = sums[u], xx = sums[nShell + u], yy = sums[2 * nShell + u];
    fsc[u] = (xx * yy == 0.0) ? 0.0 : xy / sqrt(xx * yy);
}

// V = F / T where T > floor, else 0: the inserted slices' average at every
// voxel of the accumulator.
__global__ void k_acc_ratio(const float4* __restrict__ acc, size_t n, float floor_,
                            float2* __restrict__ V)
{
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
         i += (size_t)gridDim.x * blockDim.x) {
        const float4 a = acc[i];
        V[i] = a.z > floor_ ? make_float2(a.x / a.z, a.y / a.z) : make_float2(0.f, 0.f);
    }
}

__global__ void k_acc_read(const float4* __restrict__ acc, size_t n, float2* __restrict__ F,
                           float* __restrict__ T, int accumulate)
{
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
         i += (size_t)gridDim.x * blockDim.x) {
        const float4 a = acc[i];
        if (accumulate) {
            float2 f = F[i];
            F[i] = make_float2(f.x + a.x, f.y + a.y);
            T[i] += a.z;
        } else {
            F[i] = make_float2(a.x, a.y);
            T[i] = a.z;
        }
    }
}

inline int grid_for(size_t n, int block, int cap = 152 * 16)
{
    size_t g = (n + block - 1) / block;
    if (g > (size_t)cap) g = cap;
    return (int)(g ? g : 1);
}

}  // namespace

// ---------------------------------------------------------------- launchers
cudaError_t launch_rotmat(const double* quat, int n, double* mat, cudaStream_t st)
{
    k_rotmat<<<(n + 127) / 128, 128, 0, st>>>(quat, n, mat);
    return cudaGetLastError();
}

cudaError_t launch_translate(const double* trans, int nT, int idim, const int* iCol,
                             const int* iRow, int K, float2* out, int ldo2, cudaStream_t st)
{
    dim3 grid((ldo2 + 255) / 256, nT);
    k_translate<<<grid, 256, 0, st>>>(trans, nT, idim, iCol, iRow, K, out, ldo2);
    return cudaGetLastError();
}

cudaError_t launch_ctf(const float* attr, int nImg, float px, int idim, const int* iCol,
                       const int* iRow, int K, float* out, cudaStream_t st)
{
    dim3 grid(nImg);
    k_ctf<<<grid, 256, 0, st>>>(attr, nImg, px, idim, iCol, iRow, K, out);
    return cudaGetLastError();
}

size_t volume_block_count(int vdim)
{
    return (size_t)cubes_x(vdim) * cubes_yz(vdim) * cubes_yz(vdim) * 32768;
}

cudaError_t launch_volume_blocks(const float2* vol, int vdim, float4* blocks, cudaStream_t st)
{
    size_t n = (size_t)vdim * vdim * (vdim / 2 + 1);
    k_volume_blocks<<<grid_for(n, 256), 256, 0, st>>>(vol, vdim, blocks);
    return cudaGetLastError();
}

cudaError_t launch_rot_f32(const double* quat, const double* mat, int rows, float* mf,
                           cudaStream_t st)
{
    if (rows <= 0) return cudaSuccess;
    k_rot_f32<<<grid_for((size_t)rows, 256), 256, 0, st>>>(quat, mat, rows, mf);
    return cudaGetLastError();
}

int project_chunks(int ldo) { return (ldo / 2 + kProjChunk - 1) / kProjChunk; }

size_t project_scratch_floats(int rows, int ldo)
{
    return (size_t)rows * (9 + project_chunks(ldo));
}

cudaError_t launch_project(float4* const* volTable, const int* cls, const float4* vol,
                           int vdim, int pf, const double* quat, const double* mat,
                           int rows, int rowsPerParticle, const int* iCol,
                           const int* iRow, int K, float* out, int ldo,
                           const float* sigRcp, const float* ctf, float* nrm, float* scratch,
                           int* flag, long long splitLo, cudaStream_t st, int form, int group)
{
    if (rows <= 0) return cudaSuccess;
    if (!scratch || rows % rowsPerParticle) return cudaErrorInvalidValue;
    static_assert(kProjChunk % 256 == 0, "one lane per pixel takes whole 256-pixel passes");
    const int nP = rows / rowsPerParticle;
    if (group != 4 && group != 8 && group != 16) return cudaErrorInvalidValue;
    // the rotation group of a CTA: kProjG for forms 0 - 2, `group` for 3 and 4
    const int G = form >= 3 ? group : kProjG;
    const int nGroups = (rowsPerParticle + G - 1) / G;
    const int nChunks = project_chunks(ldo);
    const long long grid = (long long)nP * nChunks * nGroups;
    if (grid > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
    float* mf = scratch;
    float* nrmPart = scratch + (size_t)rows * 9;
    k_rot_f32<<<grid_for((size_t)rows, 256), 256, 0, st>>>(quat, mat, rows, mf);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    const size_t tabBytes = sizeof(int) * ((size_t)vdim / 2 + 1 + 2 * (size_t)vdim);
    auto kern = form == 4   ? (G == 4 ? k_project_xchg<true, 4> : G == 16 ? k_project_xchg<true, 16>
                                                                   : k_project_xchg<true, 8>)
                : form == 3 ? (G == 4 ? k_project_xchg<false, 4> : G == 16 ? k_project_xchg<false, 16>
                                                                    : k_project_xchg<false, 8>)
                : form == 2 ? k_project_lane<true>
                : form == 1 ? k_project_lane<false>
                            : k_project;
    if (tabBytes > 48 * 1024) {
        e = allow_shared(kern);
        if (e != cudaSuccess) return e;
    }
    kern<<<(unsigned)grid, 256, form == 4 ? 0 : tabBytes, st>>>(volTable, cls, vol, vdim, pf, mf, rowsPerParticle,
                                                nGroups, nChunks, iCol, iRow, K, out, ldo, sigRcp,
                                                ctf, nrm ? nrmPart : nullptr, flag, splitLo);
    e = cudaGetLastError();
    if (e != cudaSuccess || !nrm) return e;
    k_norm_reduce<<<grid_for((size_t)rows, 256), 256, 0, st>>>(nrmPart, rows, nChunks, nrm);
    return cudaGetLastError();
}

cudaError_t launch_shift_bank(const float2* dat, const float* ctf, const float* sigRcp,
                              const double* trans, const float2* bank, int nP, int nT,
                              int idim, const int* iCol, const int* iRow, int K, float* out,
                              int ldo, long long splitLo, cudaStream_t st, int nD)
{
    if (nD < 1 || nT < 1) return cudaErrorInvalidValue;
    // groups of at most SHIFT_T translations, as even as possible (25 as
    // 7 + 7 + 7 + 4, not 8 + 8 + 8 + 1: every CTA reloads its pixels)
    const int groups = (nT + SHIFT_T - 1) / SHIFT_T;
    const int tPer = (nT + groups - 1) / groups;
    dim3 grid((unsigned)nP * nD, (nT + tPer - 1) / tPer);
    // the separable phase tables when they fit the default shared memory
    const size_t tab = bank ? 0 : sizeof(float2) * SHIFT_T * (size_t)(3 * (idim / 2) + 2);
    const int useTab = (!bank && idim >= 2 && tab <= 48 * 1024) ? 1 : 0;
    k_shift_bank<<<grid, 256, useTab ? tab : 0, st>>>(dat, ctf, sigRcp, trans, bank, nT, nD, idim,
                                                      iCol, iRow, K, out, ldo, splitLo, useTab,
                                                      tPer);
    return cudaGetLastError();
}

cudaError_t launch_norm_defocus(const float* P, long long splitLo, int nP, int nR, int nD, int K,
                                int Kp, const float* sigRcp, const float* ctf, float* nrm,
                                cudaStream_t st)
{
    if (nD < 1 || nD > kMaxDefocus) return cudaErrorInvalidValue;
    k_norm_defocus<<<dim3(nP, (nR + 7) / 8), 256, 0, st>>>(P, splitLo, nP, nR, nD, K, Kp, sigRcp,
                                                           ctf, nrm);
    return cudaGetLastError();
}

cudaError_t launch_project2d(const float2* img, int vdim, int pf, const double* rot, int nR,
                             const int* iCol, const int* iRow, int K, float* out, int ldo,
                             long long splitLo, cudaStream_t st)
{
    if (nR <= 0 || nR > 65535) return cudaErrorInvalidValue;
    k_project2d<<<dim3((ldo / 2 + 255) / 256, nR), 256, 0, st>>>(img, vdim, pf, rot, iCol, iRow,
                                                                K, out, ldo, splitLo);
    return cudaGetLastError();
}

cudaError_t launch_insert2d(float4* acc, int vdim, const float2* dat, const float* ctf,
                            int ctfPerDraw, const float* w, const double* offS, const int* nC,
                            const double* nR, const double* nT, const int* iCol, const int* iRow,
                            int K, int pf, int idim, int nDraws, int drawsPerImage, double* O2D,
                            int* counter, cudaStream_t st)
{
    const int tiles = std::max(1, std::min(1024, (K + 255) / 256));
    for (int d0 = 0; d0 < nDraws; d0 += 65535) {
        const int n = std::min(65535, nDraws - d0);
        k_insert2d<<<dim3(tiles, n), 256, 0, st>>>(acc, vdim, dat, ctf, ctfPerDraw, w, offS, nC, nR,
                                                   nT, iCol, iRow, K, pf, idim, d0,
                                                   drawsPerImage, O2D, counter);
    }
    return cudaGetLastError();
}

cudaError_t launch_draw_attr(const float* attr, const double* nD, int nDraws, int drawsPerImage,
                             float* out, cudaStream_t st)
{
    k_draw_attr<<<(nDraws + 255) / 256, 256, 0, st>>>(attr, nD, nDraws, drawsPerImage, out);
    return cudaGetLastError();
}

cudaError_t launch_ctf_defocus(const float* defO, const float* freQ, const double* dpara, int nD,
                               int K, double k1, double k2, double phaseShift, double conT,
                               float* ctf, cudaStream_t st)
{
    k_ctf_defocus<<<dim3((K + 255) / 256, nD), 256, 0, st>>>(defO, freQ, dpara, K, k1, k2,
                                                            phaseShift, conT, ctf);
    return cudaGetLastError();
}

cudaError_t launch_repeat_rows(const double* src, int rows, int len, int nRep, double* dst,
                               cudaStream_t st)
{
    k_repeat_rows<<<grid_for((size_t)rows * nRep * len, 256), 256, 0, st>>>(src, rows, len, nRep,
                                                                          dst);
    return cudaGetLastError();
}

cudaError_t launch_merge_defocus(int nP, int nD, int nR, int nT, const double* wCb,
                                 const double* wRb, const double* wTb, const double* baseb,
                                 const double* pwD, double* wC, double* wR, double* wT,
                                 double* wD, double* base, cudaStream_t st)
{
    if (nD < 1 || nD > kMaxDefocus) return cudaErrorInvalidValue;
    k_merge_defocus<<<nP, 256, 0, st>>>(nD, nR, nT, wCb, wRb, wTb, baseb, pwD, wC, wR, wT, wD,
                                        base);
    return cudaGetLastError();
}

cudaError_t launch_x0(const float2* dat, const float* sigRcp, int nP, int K, double* x0,
                      cudaStream_t st)
{
    k_x0<<<nP, 256, 0, st>>>(dat, sigRcp, K, x0);
    return cudaGetLastError();
}

cudaError_t launch_gemm_nt_fp32(const float* A, long long sA, int lda, const float* B,
                                long long sB, int ldb, int M, int N, int Kd, int batch,
                                float* C, long long sC, int ldc, const float* nrm,
                                long long sN, float alpha, cudaStream_t st, int cGroup,
                                long long cGroupStride)
{
    // The tile that the cost below prefers: N = 100 takes 112 columns, not 128,
    // and small problems take small tiles.  Measured at 2 x 1,000 x 100: 1.68 ms
    // at TM 16, 0.96, 0.91, 0.81 at 8, 4, 2; at 6,912 x 16,317: 2.8, 3.0, 3.6,
    // 6.3 ms.
    int TM = 16, TN = 8;
    long long best = -1;
    for (int tm = 16; tm >= 2; tm /= 2) {
        if (Kd % std::min(128 / tm, 32)) break;
        for (int tn = 8; tn >= 1; tn--) {
            const long long tiles =
                (long long)((N + 16 * tn - 1) / (16 * tn)) * ((M + 8 * tm - 1) / (8 * tm)) * batch;
            // cycles a step of k, fitted to measured shapes: a tile alone on
            // its SM waits for its K tiles (lone), tiles together share the
            // FP32 pipes (tm tn) and the shared port (4 (tm + tn))
            const long long lone = tm == 16  ? 65 + 15 * tn
                                   : tm == 8 ? 30 + 10 * tn
                                   : tm == 4 ? 18 + 10 * tn
                                             : 14 + 9 * tn;
            const long long shared = (17 * tm * tn + 40 * (tm + tn)) / 20 + 6;
            const long long cost = std::max(lone, (tiles + 151) / 152 * shared);
            if (best < 0 || cost < best) {
                best = cost;
                TM = tm;
                TN = tn;
            }
        }
    }
    dim3 grid((N + 16 * TN - 1) / (16 * TN), (M + 8 * TM - 1) / (8 * TM), batch);
#define TG3_FP32_TILE(tm, tn)                                                                    \
    if (TM == tm && TN == tn)                                                                    \
    k_gemm_nt_fp32<tm, tn><<<grid, 128, 0, st>>>(A, sA, lda, B, sB, ldb, M, N, Kd, C, sC, ldc, nrm, \
                                                 sN, alpha, cGroup, cGroupStride)
#define TG3_FP32_ROWS(tn)                                                                        \
    TG3_FP32_TILE(16, tn);                                                                       \
    TG3_FP32_TILE(8, tn);                                                                        \
    TG3_FP32_TILE(4, tn);                                                                        \
    TG3_FP32_TILE(2, tn)
    TG3_FP32_ROWS(1);
    TG3_FP32_ROWS(2);
    TG3_FP32_ROWS(3);
    TG3_FP32_ROWS(4);
    TG3_FP32_ROWS(5);
    TG3_FP32_ROWS(6);
    TG3_FP32_ROWS(7);
    TG3_FP32_ROWS(8);
#undef TG3_FP32_ROWS
#undef TG3_FP32_TILE
    return cudaGetLastError();
}

// out[i] = sum over the S partial results part[b][i], b = 0 .. S-1 in order
// (the split-K chunks of a GEMM).
__global__ void k_sum_parts(const float* __restrict__ part, int S, size_t cnt,
                            float* __restrict__ out)
{
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < cnt;
         i += (size_t)gridDim.x * blockDim.x) {
        float v = part[i];
        for (int b = 1; b < S; b++) v += part[(size_t)b * cnt + i];
        out[i] = v;
    }
}

__global__ void k_fill_int(int* __restrict__ p, size_t n, int value)
{
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
         i += (size_t)gridDim.x * blockDim.x)
        p[i] = value;
}

cudaError_t launch_fill_int(int* p, size_t n, int value, cudaStream_t st)
{
    k_fill_int<<<grid_for(n, 256), 256, 0, st>>>(p, n, value);
    return cudaGetLastError();
}

cudaError_t launch_sum_parts(const float* part, int S, size_t cnt, float* out, cudaStream_t st)
{
    if (S < 1) return cudaErrorInvalidValue;
    const unsigned blocks = (unsigned)std::min<size_t>((cnt + 255) / 256, 152 * 16);
    k_sum_parts<<<blocks, 256, 0, st>>>(part, S, cnt, out);
    return cudaGetLastError();
}

// Fold the row chunks of k_weights (nc per item): M = max_c base_c, every
// chunk scaled by exp(base_c - M): wC, wT summed over the chunks in order, the
// chunk's wR rows rescaled in place, base = M.  One CTA per item.
__global__ void k_merge_chunks(int nc, int nR, int nT, const double* __restrict__ wCc,
                               const double* __restrict__ wTc, const double* __restrict__ basec,
                               double* __restrict__ wC, double* __restrict__ wR,
                               double* __restrict__ wT, double* __restrict__ base)
{
    extern __shared__ double sc[];   // [nc]
    const int l = blockIdx.x;
    const double* bc = basec + (size_t)l * nc;
    double M = bc[0];
    for (int c = 1; c < nc; c++) M = fmax(M, bc[c]);
    for (int c = threadIdx.x; c < nc; c += blockDim.x) sc[c] = exp(bc[c] - M);
    __syncthreads();
    const int rpb = (nR + nc - 1) / nc;
    for (int r = threadIdx.x; r < nR; r += blockDim.x) wR[(size_t)l * nR + r] *= sc[r / rpb];
    for (int t = threadIdx.x; t < nT; t += blockDim.x) {
        double v = 0.0;
        for (int c = 0; c < nc; c++) v += wTc[((size_t)l * nc + c) * nT + t] * sc[c];
        wT[(size_t)l * nT + t] = v;
    }
    if (threadIdx.x == 0) {
        double v = 0.0;
        for (int c = 0; c < nc; c++) v += wCc[(size_t)l * nc + c] * sc[c];
        wC[l] = v;
        base[l] = M;
    }
}

cudaError_t launch_weights(const float* D, long long sD, int ldc, int nR, int nT, int G,
                           int nBlocks, const float* nrmG, int nrmRS, const double* x0,
                           const double* pwR,
                           long long sR, const double* pwT, long long sT, const double* pwC,
                           double* wC, double* wR, double* wT, double* base, float* dvp,
                           cudaStream_t st, int threads, int nc, double* chunkTmp,
                           const int* best)
{
    if (nc < 1 || (nc > 1 && (G != 1 || !chunkTmp))) return cudaErrorInvalidValue;
    if (threads != 128 && threads != 256 && threads != WEIGHTS_THREADS)
        return cudaErrorInvalidValue;
    const size_t smem = sizeof(float) * (2 + (nT <= 256 ? threads / 32 : 0)) * (size_t)nT;
    if (smem > 48 * 1024) return cudaErrorInvalidValue;
    // nc > 1: per-chunk wC, wT, base in chunkTmp, folded afterwards
    double* cC = nc > 1 ? chunkTmp : wC;
    double* cB = nc > 1 ? chunkTmp + (size_t)nBlocks * nc : base;
    double* cT = nc > 1 ? chunkTmp + 2 * (size_t)nBlocks * nc : wT;
#define TG3_WEIGHTS(TS)                                                                        \
    k_weights<TS><<<nBlocks * nc, threads, smem, st>>>(D, sD, ldc, nR, nT, G, nrmG, nrmRS, x0, \
                                                       pwR, sR, pwT, sT, pwC, cC, wR, cT, cB,  \
                                                       dvp, nc, best)
    if (nT <= 32) TG3_WEIGHTS(1);
    else if (nT <= 64) TG3_WEIGHTS(2);
    else if (nT <= 128) TG3_WEIGHTS(4);
    else if (nT <= 256) TG3_WEIGHTS(8);
    else TG3_WEIGHTS(0);
#undef TG3_WEIGHTS
    if (nc > 1) {
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
        k_merge_chunks<<<nBlocks, 128, sizeof(double) * nc, st>>>(nc, nR, nT, cC, cT, cB, wC, wR,
                                                                  wT, base);
    }
    return cudaGetLastError();
}

cudaError_t launch_merge_class(int nImg, int nK, int kIdx, int nR, int nT, const double* wCn,
                               const double* wRn, const double* wTn, const double* basen,
                               float* wC, float* wR, float* wT, float* baseL, cudaStream_t st,
                               int inStride)
{
    k_merge_class<<<nImg, 256, 0, st>>>(nK, kIdx, nR, nT, wCn, wRn, wTn, basen, wC, wR, wT,
                                         baseL, inStride);
    return cudaGetLastError();
}

// All nK per-(image, class) weight blocks of a multi-class scan folded into
// ExpectGlobal2D's outputs in one pass: relative to the image's best class,
// class k scaled by exp(base_k - max_k base_k) -- the value the running
// baseline of kernel_setBaseLine / kernel_UpdateW reaches class by class.
// One CTA per image; smem: nK doubles.
__global__ void k_merge_classes(int nK, int nR, int nT, const double* __restrict__ wCn,
                                const double* __restrict__ wRn, const double* __restrict__ wTn,
                                const double* __restrict__ basen, float* __restrict__ wC,
                                float* __restrict__ wR, float* __restrict__ wT,
                                float* __restrict__ baseL)
{
    extern __shared__ double esc[];
    __shared__ double Bm;
    const size_t l = blockIdx.x;
    const double* bl = basen + l * nK;
    if (threadIdx.x == 0) {
        double m = bl[0];
        for (int k = 1; k < nK; k++) m = fmax(m, bl[k]);
        Bm = m;
        baseL[l] = (float)m;
    }
    __syncthreads();
    for (int k = threadIdx.x; k < nK; k += blockDim.x) {
        esc[k] = exp(bl[k] - Bm);
        wC[l * nK + k] = (float)(wCn[l * nK + k] * esc[k]);
    }
    __syncthreads();
    const size_t oR = l * nK * nR, oT = l * nK * nT;
    for (int i = threadIdx.x; i < nK * nR; i += blockDim.x)
        wR[oR + i] = (float)(wRn[oR + i] * esc[i / nR]);
    for (int i = threadIdx.x; i < nK * nT; i += blockDim.x)
        wT[oT + i] = (float)(wTn[oT + i] * esc[i / nT]);
}

cudaError_t launch_merge_classes(int nImg, int nK, int nR, int nT, const double* wCn,
                                 const double* wRn, const double* wTn, const double* basen,
                                 float* wC, float* wR, float* wT, float* baseL, cudaStream_t st)
{
    const size_t smem = sizeof(double) * (size_t)nK;
    if (smem > 48 * 1024) return cudaErrorInvalidValue;
    k_merge_classes<<<nImg, 256, smem, st>>>(nK, nR, nT, wCn, wRn, wTn, basen, wC, wR, wT, baseL);
    return cudaGetLastError();
}

__global__ void k_nrm_classes(const float* __restrict__ nrm, int nK, int nR, int n,
                              float* __restrict__ out)
{
    const size_t total = (size_t)nK * nR * n;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total;
         i += (size_t)gridDim.x * blockDim.x) {
        // i walks the output: i = r (n nK) + l nK + k
        const int k = (int)(i % nK);
        const size_t rl = i / nK;
        const int l = (int)(rl % n);
        const int r = (int)(rl / n);
        out[i] = nrm[((size_t)k * nR + r) * n + l];
    }
}

cudaError_t launch_nrm_classes(const float* nrm, int nK, int nR, int n, float* out,
                               cudaStream_t st)
{
    k_nrm_classes<<<grid_for((size_t)nK * nR * n, 256), 256, 0, st>>>(nrm, nK, nR, n, out);
    return cudaGetLastError();
}

cudaError_t prefer_carveouts(bool beside)
{
    // half of the SM's memory as L1: their own full occupancy would take up to
    // 200 KB as shared memory (8 CTAs of 25 KB)
    const int percent = beside ? 50 : cudaSharedmemCarveoutDefault;
    cudaError_t e = cudaFuncSetAttribute(k_shift_bank, cudaFuncAttributePreferredSharedMemoryCarveout,
                                         percent);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_resample, cudaFuncAttributePreferredSharedMemoryCarveout, percent);
    return e;
}

cudaError_t launch_resample(int nP, int n, const double* u, const double* w, const int* perm,
                            const double* u0, const double* peak, int nOut, int* src,
                            double* wOut, int* top, int* flag, cudaStream_t st, const int* nPer)
{
    size_t smem = sizeof(double) * (2 * (size_t)n + (size_t)(n > nOut ? n : nOut))
                + sizeof(int) * (size_t)n;
    cudaError_t e = allow_shared(k_resample);
    if (e != cudaSuccess) return e;
    k_resample<<<nP, 256, smem, st>>>(n, u, w, perm, u0, peak, nOut, nPer, src, wOut, top, flag);
    return cudaGetLastError();
}

size_t insert_param_bytes(int nDraws, int K)
{
    return (size_t)nDraws * 16 * sizeof(float) + sizeof(unsigned long long) +
           sizeof(int) * (size_t)((K + kInsertRun - 1) / kInsertRun);
}

cudaError_t launch_insert(float4* acc, int vdim, int kernel, const float* tab, int tabNz,
                          float tabInvStep, int nDraws, int drawsPerImage, const float2* dat,
                          const float* ctf, const double* quat, const double* trans,
                          const double* offset, const float* w, const int* iCol,
                          const int* iRow, int K, int pf, int idim, double* O3D, int* counter,
                          float* params, cudaStream_t st, double maxRadius, int ctfRows, const int* nC)
{
    if (nDraws <= 0) return cudaSuccess;
    // r^2 bound of the table's support: rint(r^2 n / b) <= tabNz  =>  r^2 < (tabNz + 1/2) b / n
    const float rs2 = (((float)tabNz + 0.5f) / tabInvStep) * (1.0f + 1e-4f);
    if (kernel == TG3_KERNEL_MKB && 2.0f * sqrtf(rs2) >= 4.0f) return cudaErrorInvalidValue;
    k_insert_draws<<<(nDraws + 255) / 256, 256, 0, st>>>(nDraws, drawsPerImage, quat, trans,
                                                         offset, w, params, O3D, counter, nC);
    const int ctfPerDraw = ctfRows == nDraws && drawsPerImage > 1;
    if (kernel == TG3_KERNEL_MKB) {
        const size_t smem = sizeof(float) * ((size_t)tabNz + 1);
        const bool shared = smem <= 200 * 1024;
        const auto kern = shared ? k_insert_mkb<true> : k_insert_mkb<false>;
        if (shared) {
            const cudaError_t e = allow_shared(kern);
            if (e != cudaSuccess) return e;
        }
        const long long items = (long long)((K + kInsertItem - 1) / kInsertItem) * nDraws;
        const long long ctas = (items + kInsertThreads / 32 - 1) / (kInsertThreads / 32);
        auto* next = reinterpret_cast<unsigned long long*>(params + 16 * (size_t)nDraws);
        // The half ball that the draws reach, against the L2: 48 MB of it and up go
        // by radius where there are draws enough to come back to a shell.
        // Measured by draw and by radius: radius 160 (142 MB) 3.19 and 2.86 ms for
        // 2,000 draws, 525 and 450 us for 300, 137 and 163 for 70; radius 124 (67
        // MB) 709 and 682 for 1,000; radius 100 (37 MB) 381 and 389.
        const double R = maxRadius * pf + 2.0;
        int* order = nullptr;
        if (nDraws >= 160 && 2.0 / 3.0 * M_PI * R * R * R * sizeof(float4) > (double)kInsertL2) {
            const int nRuns = (K + kInsertRun - 1) / kInsertRun;
            order = reinterpret_cast<int*>(next + 1);
            k_insert_order<<<(nRuns + 255) / 256, 256, 0, st>>>(iCol, iRow, K, nRuns, order);
        }
        kern<<<(unsigned)std::min<long long>(ctas, 152), kInsertThreads, shared ? smem : 0, st>>>(
            acc, vdim, tab, tabNz, tabInvStep, sqrtf(rs2), dat, ctf, params, iCol, iRow, K, pf, idim,
            nDraws, drawsPerImage, ctfPerDraw, next, order);
        return cudaGetLastError();
    }
    // one pixel per thread: the draw's pixels spread over ceil(K / 256) CTAs
    const int tiles = std::max(1, std::min(1024, (K + 255) / 256));
    for (int d0 = 0; d0 < nDraws; d0 += 65535) {
        const int n = std::min(65535, nDraws - d0);
        k_insert<<<dim3(tiles, n), 256, 0, st>>>(acc, vdim, dat, ctf, params, iCol, iRow, K, pf, idim,
                                                 d0, drawsPerImage, ctfPerDraw);
    }
    return cudaGetLastError();
}

size_t insert_draw_bytes(int Rg)
{
    return (size_t)(Rg + 1) * (2 * Rg + 1) * sizeof(float4) + 16 * sizeof(float);
}

cudaError_t launch_insert_gather(float4* acc, int vdim, const float* tab, int tabNz,
                                 float tabInvStep, int nDraws, int drawsPerImage,
                                 const float2* dat, const float* ctf, const double* quat,
                                 const double* trans, const double* offset, const float* w,
                                 const int* cellPix, const int* iCol, const int* iRow, int K,
                                 int pf, int idim, int Rg, float Rp, double* O3D, int* counter,
                                 void* scratch, size_t scratchBytes, cudaStream_t st, int ctfRows)
{
    if (nDraws <= 0) return cudaSuccess;
    const int ctfPerDraw = ctfRows == nDraws && drawsPerImage > 1;
    const int gw = Rg + 1, cells = gw * (2 * Rg + 1);
    const size_t gridBytes = (size_t)cells * sizeof(float4);
    const size_t chunkMax = scratchBytes / insert_draw_bytes(Rg);
    if (chunkMax < 1) return cudaErrorInvalidValue;
    const int chunk = (int)std::min<size_t>(std::min<size_t>((size_t)nDraws, chunkMax), 65535);
    float4* grid = static_cast<float4*>(scratch);
    float* rot = reinterpret_cast<float*>(static_cast<char*>(scratch) + gridBytes * chunk);
    // slab half thickness: rint(r^2 n / b) <= tabNz  <=>  r^2 < (tabNz + 1/2) b / n
    const float hs = sqrtf(((float)tabNz + 0.5f) / tabInvStep) + 1e-3f;
    const int stageTiles = std::max(1, std::min(64, (cells + 1023) / 1024));
    for (int d0 = 0; d0 < nDraws; d0 += chunk) {
        const int n = std::min(chunk, nDraws - d0);
        k_insert_stage<<<dim3(stageTiles, n), 256, 0, st>>>(grid, cells, rot, cellPix, iCol, iRow,
                                                            dat, ctf, quat, trans, offset, w, K,
                                                            idim, d0, drawsPerImage, ctfPerDraw,
                                                            O3D, counter);
        // about two waves of resident CTAs (152 SMs x 8 CTAs of 256 threads)
        const int tiles = std::max(1, std::min(128, (2 * 152 * 8 + n - 1) / n));
        k_insert_gather<<<dim3(tiles, n), 256, 0, st>>>(acc, vdim, grid, gw, Rg, rot, tab, tabNz,
                                                        tabInvStep, pf, Rp, hs);
    }
    return cudaGetLastError();
}

cudaError_t launch_bank_planes(const float* f32, int nB, int K, int Kp, __nv_bfloat16* hi,
                               __nv_bfloat16* lo, float* abs2, cudaStream_t st)
{
    k_bank_planes<<<grid_for((size_t)nB * (Kp / 2), 256), 256, 0, st>>>(f32, nB, K, Kp, hi, lo,
                                                                       abs2);
    return cudaGetLastError();
}

cudaError_t launch_bank_gather(const BankView* table, const int* cls, const int* idx, int nP,
                               int nR, int K, int Kp, const float* sigRcp, const float* ctf,
                               float* P, long long splitLo, float* nrm, int* flag,
                               cudaStream_t st)
{
    if (Kp % 8) return cudaErrorInvalidValue;
    const size_t smem = sizeof(float) * (size_t)K;
    if (smem > 48 * 1024) {
        if (smem > 200 * 1024) return cudaErrorInvalidValue;
        cudaError_t e = allow_shared(k_bank_gather);
        if (e != cudaSuccess) return e;
    }
    dim3 grid(nP, (nR + kBankRows - 1) / kBankRows);
    k_bank_gather<<<grid, 256, smem, st>>>(table, cls, idx, nR, K, Kp, sigRcp, ctf, P, splitLo,
                                           nrm, flag);
    return cudaGetLastError();
}

cudaError_t launch_fsc(const float2* A, const float2* B, int vdim, int nShell, double* sums,
                       double* fsc, cudaStream_t st)
{
    cudaError_t e = cudaMemsetAsync(sums, 0, sizeof(double) * 3 * (size_t)nShell, st);
    if (e != cudaSuccess) return e;
    const size_t smem = sizeof(double) * 3 * (size_t)nShell;
    e = allow_shared(k_fsc_shells);
    if (e != cudaSuccess) return e;
    const size_t n = (size_t)vdim * vdim * (vdim / 2 + 1);
    k_fsc_shells<<<grid_for(n, 256, 152 * 4), 256, smem, st>>>(A, B, vdim, nShell, sums);
    k_fsc_finish<<<(nShell + 127) / 128, 128, 0, st>>>(sums, nShell, fsc);
    return cudaGetLastError();
}

cudaError_t launch_acc_ratio(const float4* acc, size_t n, float floor_, float2* V, cudaStream_t st)
{
    k_acc_ratio<<<grid_for(n, 256), 256, 0, st>>>(acc, n, floor_, V);
    return cudaGetLastError();
}

cudaError_t launch_acc_read(const float4* acc, size_t n, float2* F, float* T, int accumulate,
                            cudaStream_t st)
{
    k_acc_read<<<grid_for(n, 256), 256, 0, st>>>(acc, n, F, T, accumulate);
    return cudaGetLastError();
}

}  // namespace tg3
