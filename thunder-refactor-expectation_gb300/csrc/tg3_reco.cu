// Reconstruction of a map from the insertion accumulators (Reconstructor::
// reconstruct, src/Reconstructor.cpp:1129-1790, 3-D, no symmetry), on the
// padded half grid vdim = N pf, coordinates (x, y, z) with x in [0, vdim/2]
// and y, z wrapped:
//   Wiener filter from the FSC (RECONSTRUCTOR_WIENER_FILTER_FSC, :1236-1262):
//     for (5 pf)^2 <= |k|^2 < (maxR pf)^2, u = rint(|k|): f = FSC[u / pf]
//     (0 past its end), clamped to [1e-3, 1 - 1e-3], f = sqrt(2 f / (1 + f))
//     when the half maps are joined; T /= f;
//   T = max(T, 1e-25); W = 1 inside maxR pf, 0 outside (:1268-1300);
//   grid correction (:1318-1460): up to 30 rounds of C = T W,
//     C = FT(iFT(C) kRL(r^2) / nf) (convoluteC, :2593-2660; kRL the MKB
//     kernel's real-space form at r = |x| / (N pf), nf = kRL(0)),
//     W /= max(|C|, 1e-6) inside maxR pf, stopping when max ||C| - 1| < 1e-2
//     or, after 10 rounds, when it failed twice in a row to fall below 0.95 x
//     the previous (checkC with RECONSTRUCTOR_CHECK_C_MAX, :2520-2590);
//     without it W = 1 / max(|T|, 1e-6) (:1463-1490);
//   V = F W inside maxR pf; the inverse transform (1 / vdim^3); the central
//   N^3 kept (VOL_EXTRACT_RL); divided by the kernel's real-space transform
//   at |x| / (pf N): j0(pi r)^2 for the trilinear kernel (TIK_RL), MKB_RL(r,
//   a pf, alpha) / MKB_RL(0, a pf, alpha) for MKB (:1700-1790).
// MKB_RL (src/Functions/Functions.cpp:128-160, order 0): with u = 2 pi a r and
// v = sqrt(|alpha^2 - u^2|), (2 pi)^1.5 a^3 / I0(alpha) I_1.5(v) / v^1.5 for
// u <= alpha, J_1.5(v) / v^1.5 beyond; the half-integer Bessel functions in
// their closed forms.
#include <cufft.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <vector>

#include "tg3_fft.cuh"
#include "tg3_internal.cuh"

namespace tg3 {
namespace {

// I_1.5(v) / v^1.5 and J_1.5(v) / v^1.5 (closed forms; series near 0)
__host__ __device__ double i15_over(double v)
{
    if (v < 1e-3) return (1.0 + v * v / 10.0) / (3.0 * sqrt(M_PI / 2.0));
    return sqrt(2.0 / M_PI) * (cosh(v) - sinh(v) / v) / (v * v);
}

__host__ __device__ double j15_over(double v)
{
    if (v < 1e-3) return (1.0 - v * v / 10.0) / (3.0 * sqrt(M_PI / 2.0));
    return sqrt(2.0 / M_PI) * (sin(v) / v - cos(v)) / (v * v);
}

// the modified Bessel function I0 by its power series (alpha is O(10))
__host__ __device__ double bessel_i0(double x)
{
    double s = 1.0, t = 1.0;
    const double q = x * x / 4.0;
    for (int k = 1; k < 200; k++) {
        t *= q / ((double)k * k);
        s += t;
        if (t < 1e-17 * s) break;
    }
    return s;
}

__host__ __device__ double mkb_rl(double r, double a, double alpha, double i0a)
{
    const double u = 2.0 * M_PI * a * r;
    const double w = pow(2.0 * M_PI, 1.5) * a * a * a / i0a;
    if (u <= alpha) return w * i15_over(sqrt(alpha * alpha - u * u));
    return w * j15_over(sqrt(u * u - alpha * alpha));
}

__device__ double tik_rl(double r)
{
    const double x = M_PI * r;
    const double j0 = x < 1e-8 ? 1.0 : sin(x) / x;
    return j0 * j0;
}

__device__ __forceinline__ int wrapc(int i, int n) { return i < n / 2 ? i : i - n; }

// Wiener-filtered, floored T and the initial W (1 inside the radius)
__global__ void k_reco_init(const float4* __restrict__ acc, int vdim, int nz, int pf,
                            const double* __restrict__ fsc, int nFsc, int joinHalf,
                            long long r2max, float* __restrict__ T, float* __restrict__ W)
{
    const int nx = vdim / 2 + 1;
    const size_t n = (size_t)nz * vdim * nx;
    const long long r2min = 25LL * pf * pf;
    for (size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x; idx < n;
         idx += (size_t)gridDim.x * blockDim.x) {
        const unsigned u32 = (unsigned)idx, row = u32 / (unsigned)nx;
        const int x = (int)(u32 - row * (unsigned)nx);
        const int y = wrapc((int)(row % (unsigned)vdim), vdim);
        const int z = nz > 1 ? wrapc((int)(row / (unsigned)vdim), vdim) : 0;
        const long long q = (long long)x * x + (long long)y * y + (long long)z * z;
        double t = acc[idx].z;
        if (fsc && q >= r2min && q < r2max) {
            // rint(sqrt(q)) in FP32 is exact here: no integer q lies within
            // FP32 rounding of a half-integer radius below 2^11
            const int u = (int)rintf(sqrtf((float)q));
            double f = (u / pf >= nFsc) ? 0.0 : fsc[u / pf];
            f = fmax(1e-3, fmin(1.0 - 1e-3, f));
            if (joinHalf) f = sqrt(2.0 * f / (1.0 + f));
            t /= f;
        }
        T[idx] = (float)fmax(t, 1e-25);
        W[idx] = q < r2max ? 1.f : 0.f;
    }
}

// C = T W (real, as a complex half grid)
__global__ void k_reco_tw(const float* __restrict__ T, const float* __restrict__ W, size_t n,
                          float2* __restrict__ C)
{
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
         i += (size_t)gridDim.x * blockDim.x)
        C[i] = make_float2(T[i] * W[i], 0.f);
}

// A radial function of the integer squared radius q, tabulated once per call
// (the kernels depend on x^2 + y^2 + z^2 only): tab[q] = scale k(sqrt(q) / s)
// with k the MKB real-space form (mkb) or j0(pi r)^2.  r2step > 0 takes the
// kernel at r^2 rounded to the nearest multiple of r2step, as a TabFunction
// of r^2 looks it up (src/TabFunction.cpp:42-45; the balancing kernel
// Reconstructor::_kernelRL is one over [0, 1] in 1e5 steps,
// src/Reconstructor.cpp:76-85).
__global__ void k_radial_table(float* __restrict__ tab, int nq, double s, int mkb, double a,
                               double alpha, double i0a, double scale, double r2step)
{
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < nq; q += gridDim.x * blockDim.x) {
        double r = sqrt((double)q) / s;
        if (r2step > 0) r = sqrt(rint((double)q / (s * s) / r2step) * r2step);
        tab[q] = (float)(scale * (mkb ? mkb_rl(r, a, alpha, i0a) : tik_rl(r)));
    }
}

// real-space C (after the unnormalised inverse) times kRL(r^2) / nf / vdim^3
// (the table holds kRL / nf / vdim^3)
__global__ void k_reco_kernel_rl(float* __restrict__ c, int vdim, int nz,
                                 const float* __restrict__ tab)
{
    const size_t n = (size_t)nz * vdim * vdim;
    for (size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x; idx < n;
         idx += (size_t)gridDim.x * blockDim.x) {
        const unsigned u32 = (unsigned)idx, row = u32 / (unsigned)vdim;
        const int x = wrapc((int)(u32 - row * (unsigned)vdim), vdim);
        const int y = wrapc((int)(row % (unsigned)vdim), vdim);
        const int z = nz > 1 ? wrapc((int)(row / (unsigned)vdim), vdim) : 0;
        c[idx] *= tab[x * x + y * y + z * z];
    }
}

// W /= max(|C|, 1e-6) inside the radius; diff = max ||C| - 1| there (float
// bits compared as ints: the values are non-negative); then C <- T W for the
// next round (the inverse transform consumes C)
__global__ void k_reco_update(float2* __restrict__ C, const float* __restrict__ T, int vdim,
                              int nz, long long r2max, float* __restrict__ W,
                              unsigned* __restrict__ diffBits)
{
    const int nx = vdim / 2 + 1;
    const size_t n = (size_t)nz * vdim * nx;
    float dmax = 0.f;
    for (size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x; idx < n;
         idx += (size_t)gridDim.x * blockDim.x) {
        const unsigned u32 = (unsigned)idx, row = u32 / (unsigned)nx;
        const int x = (int)(u32 - row * (unsigned)nx);
        const int y = wrapc((int)(row % (unsigned)vdim), vdim);
        const int z = nz > 1 ? wrapc((int)(row / (unsigned)vdim), vdim) : 0;
        const long long q = (long long)x * x + (long long)y * y + (long long)z * z;
        float w = W[idx];
        if (q < r2max) {
            const float m = sqrtf(C[idx].x * C[idx].x + C[idx].y * C[idx].y);
            w = w / fmaxf(m, 1e-6f);
            W[idx] = w;
            dmax = fmaxf(dmax, fabsf(m - 1.f));
        }
        C[idx] = make_float2(T[idx] * w, 0.f);
    }
    for (int o = 16; o; o >>= 1) dmax = fmaxf(dmax, __shfl_xor_sync(0xffffffffu, dmax, o));
    if ((threadIdx.x & 31) == 0) atomicMax(diffBits, __float_as_uint(dmax));
}

// without grid correction: W = 1 / max(|T|, 1e-6) inside the radius
__global__ void k_reco_w_from_t(const float* __restrict__ T, int vdim, int nz, long long r2max,
                                float* __restrict__ W)
{
    const int nx = vdim / 2 + 1;
    const size_t n = (size_t)nz * vdim * nx;
    for (size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x; idx < n;
         idx += (size_t)gridDim.x * blockDim.x) {
        const unsigned u32 = (unsigned)idx, row = u32 / (unsigned)nx;
        const int x = (int)(u32 - row * (unsigned)nx);
        const int y = wrapc((int)(row % (unsigned)vdim), vdim);
        const int z = nz > 1 ? wrapc((int)(row / (unsigned)vdim), vdim) : 0;
        const long long q = (long long)x * x + (long long)y * y + (long long)z * z;
        if (q < r2max) W[idx] = 1.f / fmaxf(fabsf(T[idx]), 1e-6f);
    }
}

// V = F W inside the radius, 0 outside
__global__ void k_reco_fw(const float4* __restrict__ acc, const float* __restrict__ W, int vdim,
                          int nz, long long r2max, float2* __restrict__ V)
{
    const int nx = vdim / 2 + 1;
    const size_t n = (size_t)nz * vdim * nx;
    for (size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x; idx < n;
         idx += (size_t)gridDim.x * blockDim.x) {
        const unsigned u32 = (unsigned)idx, row = u32 / (unsigned)nx;
        const int x = (int)(u32 - row * (unsigned)nx);
        const int y = wrapc((int)(row % (unsigned)vdim), vdim);
        const int z = nz > 1 ? wrapc((int)(row / (unsigned)vdim), vdim) : 0;
        const long long q = (long long)x * x + (long long)y * y + (long long)z * z;
        const float4 a = acc[idx];
        V[idx] = q < r2max ? make_float2(a.x * W[idx], a.y * W[idx]) : make_float2(0.f, 0.f);
    }
}

// The column x = 0 before a real inverse transform by the library: points k and
// -k become conjugates, (C[k] + conj C[-k]) / 2 each, which leaves the real part
// of the column's sums.  Insertion writes the two from different pixels, so they
// are not; and what the library then gives differs by side: this real part at
// most, a map off by 3 % of its peak at 1,024^3 and by 0.5 % at 2,048^2.
__global__ void k_reco_pair(float2* __restrict__ C, int vdim, int nz)
{
    const int n = nz * vdim, nx = vdim / 2 + 1;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int y = i % vdim, z = i / vdim;
        const int j = (z ? nz - z : 0) * vdim + (y ? vdim - y : 0);
        if (j < i) continue;
        const float2 a = C[(size_t)i * nx], b = C[(size_t)j * nx];
        const float re = 0.5f * (a.x + b.x), im = 0.5f * (a.y - b.y);
        C[(size_t)i * nx] = make_float2(re, im);
        if (j != i) C[(size_t)j * nx] = make_float2(re, -im);
    }
}

// the central N^3 of the padded real-space map, in centred order (index i +
// N/2 for coordinate i), divided by the kernel's real-space transform
// (the table holds the kernel's real-space transform times vdim^3)
__global__ void k_reco_extract(const float* __restrict__ pad, int vdim, int nz, int N,
                               const float* __restrict__ tab, float* __restrict__ out)
{
    const size_t n = (size_t)(nz > 1 ? N : 1) * N * N;
    for (size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x; idx < n;
         idx += (size_t)gridDim.x * blockDim.x) {
        const int x = (int)(idx % N) - N / 2;
        const int y = (int)((idx / N) % N) - N / 2;
        const int z = nz > 1 ? (int)(idx / ((size_t)N * N)) - N / 2 : 0;
        const int px = x < 0 ? x + vdim : x, py = y < 0 ? y + vdim : y, pz = z < 0 ? z + vdim : z;
        out[idx] = pad[((size_t)pz * vdim + py) * vdim + px] / tab[x * x + y * y + z * z];
    }
}

// accumulator <- (F, T): the sums of several contexts or ranks loaded back
__global__ void k_acc_load(const float2* __restrict__ F, const float* __restrict__ T, size_t n,
                           float4* __restrict__ acc)
{
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
         i += (size_t)gridDim.x * blockDim.x)
        acc[i] = make_float4(F[i].x, F[i].y, T[i], 0.f);
}

// ----------------------------------------------------------- own passes --
// The 3-D reconstruction on grids whose side is in TG3_RECO_SIDES, as passes
// over one half-complex array C [z][y][px], each line transformed on chip
// (tg3_fft.cuh).  A balancing round:
//   z: forward along z, W and C = T W updated, inverse along z;
//   y: inverse;  x: inverse to two real rows, the kernel product, forward;
//   y: forward.
// C is zero and not looked at outside the sphere |k|^2 < r2max, so C keeps the
// columns x < rmax only, the y passes read (inverse) or write (forward) the
// rows inside the circle of their column, and the z pass visits those lines
// only.  Bound by the latency of loads, exchanges and stores at 12 warps an SM (DRAM
// at a quarter to a half of its rate): a thread holds 24 to 32 points at up to 168
// registers, and 12 of the 17 z passes spill some of them (8 to 216 bytes; 12 at
// 32 x 16, whose y pass spills 80).  A round moves about 3.9 GB at 512^3 with rmax
// 240 and takes 1.2 ms, where the library's six transform kernels and two passes
// between them took 2.35 ms.
struct Pass3 {
    const float2* tw;        // the n-th roots of unity
    float2* C;               // [n][n][px]
    int nxr, px;             // columns in use, their pitch
    long long r2max;
};

using fft::c64;

template <int A, int B>
__device__ __forceinline__ const float2* pass_roots(const Pass3& p, c64* buf)
{
    float2* tw = reinterpret_cast<float2*>(buf + fft::Shape<A, B>::floats2);
    for (int k = threadIdx.x; k < A * B; k += blockDim.x) tw[k] = p.tw[k];
    return tw;
}

// largest |y| with x0^2 + y^2 < r2max (x0 in use)
__device__ __forceinline__ int rows_inside(long long r2max, int x0)
{
    const int q = (int)(r2max - 1 - (long long)x0 * x0);
    int y = (int)sqrtf((float)q);
    while ((long long)y * y > q) y--;
    while ((long long)(y + 1) * (y + 1) <= q) y++;
    return y;
}

__device__ __forceinline__ void copy16(float* dst, const float* src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                     (uint32_t)__cvta_generic_to_shared(dst)),
                 "l"(src)
                 : "memory");
}

__device__ __forceinline__ c64 load_c(const float2* p) { return *reinterpret_cast<const c64*>(p); }

// CTA (8 columns, plane z): lines along y.
template <int A, int B>
__global__ void __launch_bounds__(fft::Shape<A, B>::threads, 384 / fft::Shape<A, B>::threads)
k_reco_pass_y(const Pass3 p, int inverse, int planes)
{
    using S = fft::Shape<A, B>;
    extern __shared__ __align__(16) c64 fsm[];
    constexpr int n = S::n;
    const int x0 = blockIdx.x * kFftLines, line = threadIdx.x % kFftLines, t = threadIdx.x / kFftLines;
    const float2* tw = pass_roots<A, B>(p, fsm);
    // planes < n: the central ones (coordinates -planes / 2 .. planes / 2 - 1)
    const int z = blockIdx.y < planes / 2 ? blockIdx.y : blockIdx.y + n - planes;
    float2* C = p.C + (size_t)z * n * p.px + x0 + line;
    const int yr = rows_inside(p.r2max, x0);
    c64 v[S::I1][A], o[S::I2][B];
#pragma unroll
    for (int i = 0; i < S::I1; i++)
#pragma unroll
        for (int r = 0; r < A; r++) {
            const int y = t + i * S::TL + r * B;
            v[i][r] = 0;
            if (t + i * S::TL < B && (!inverse || y <= yr || n - y <= yr)) {
                v[i][r] = load_c(C + (size_t)y * p.px);
                if (inverse) v[i][r] = fft::swapped(v[i][r]);
            }
        }
    __syncthreads();
    fft::run<A, B, S::TL>(v, o, fsm, tw, t, line);
#pragma unroll
    for (int i = 0; i < S::I2; i++)
#pragma unroll
        for (int s = 0; s < B; s++) {
            const int y = t + i * S::TL + s * A;
            if (t + i * S::TL < A && (inverse || y <= yr || n - y <= yr))
                *reinterpret_cast<c64*>(C + (size_t)y * p.px) =
                    inverse ? fft::swapped(o[i][s]) : o[i][s];
        }
}

// CTA (8 columns, row y inside their circle): lines along z.  Mode 0: T from
// the accumulator and the FSC (rfsc [nFsc + 1]: 1 / f of a shell, the last for
// shells past its end), W = 1, C = T; 1: a round's update; 2: C = F W; 3: C = F /
// T, no grid correction.  Then the inverse along z.
template <int A, int B>
__global__ void __launch_bounds__(fft::Shape<A, B>::threads, 384 / fft::Shape<A, B>::threads)
k_reco_pass_z(const Pass3 p, int mode, const float4* __restrict__ acc,
              const double* __restrict__ rfsc, int nFsc, int pf, float* __restrict__ T,
              float* __restrict__ W, unsigned* __restrict__ diffBits)
{
    using S = fft::Shape<A, B>;
    extern __shared__ __align__(16) c64 fsm[];
    constexpr int n = S::n;
    const int x0 = blockIdx.x * kFftLines, line = threadIdx.x % kFftLines, t = threadIdx.x / kFftLines;
    const int rmax = rows_inside(p.r2max, 0);
    const int yc = (int)blockIdx.y - rmax;
    if ((long long)x0 * x0 + (long long)yc * yc >= p.r2max) return;
    const float2* tw = pass_roots<A, B>(p, fsm);
    const int y = yc < 0 ? yc + n : yc, x = x0 + line;
    const size_t at0 = (size_t)y * p.px + x, plane = (size_t)n * p.px;
    const int xy = x * x + yc * yc, r2 = (int)p.r2max;
    const int xa = min(x, n / 2);
    c64 v[S::I1][A], o[S::I2][B];
    // a round's W and T of the inside of the line, copied behind the first
    // transform
    float* sW = reinterpret_cast<float*>(fsm + S::smem / sizeof(c64));
    float* sT = sW + n * kFftLines;
    if (mode == 1) {
        const int zr = rows_inside(p.r2max - yc * yc, x0);
        for (int i = threadIdx.x; i < n * 2; i += S::threads) {
            const int z = i >> 1, e = 4 * (i & 1);
            if (z > zr && n - z > zr) continue;
            const size_t g = z * plane + (size_t)y * p.px + x0 + e;
            copy16(sW + z * kFftLines + e, W + g);
            copy16(sT + z * kFftLines + e, T + g);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
#pragma unroll
        for (int i = 0; i < S::I1; i++)
#pragma unroll
            for (int r = 0; r < A; r++) {
                const int z = t + i * S::TL + r * B;
                v[i][r] = t + i * S::TL < B ? load_c(p.C + z * plane + at0) : 0;
            }
        __syncthreads();
        fft::run<A, B, S::TL>(v, o, fsm, tw, t, line);
        asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
    float dmax = 0.f;
    // points outside the sphere read an inside one's neighbourhood of their
    // line (z = 0 lies inside), so that a group's loads go out together
    constexpr int G = 8;
#pragma unroll
    for (int i = 0; i < S::I2; i++)
#pragma unroll
        for (int s0 = 0; s0 < B; s0 += G) {
            float4 f[G];
            float w[G], tt[G];
            bool in[G];
#pragma unroll
            for (int g = 0; g < G; g++) {
                const int z = t + i * S::TL + (s0 + g) * A;
                const int zc = z < n / 2 ? z : z - n;
                in[g] = s0 + g < B && t + i * S::TL < A && xy + zc * zc < r2;
                const int zl = in[g] ? z : 0;
                const size_t at = zl * plane + at0;
                if (mode == 1) {
                    w[g] = sW[zl * kFftLines + line];
                    tt[g] = sT[zl * kFftLines + line];
                }
                if (mode == 2) w[g] = W[at];
                if (mode != 1) f[g] = acc[((size_t)zl * n + y) * (n / 2 + 1) + xa];
            }
#pragma unroll
            for (int g = 0; g < G; g++) {
                if (s0 + g >= B) break;
                const int z = t + i * S::TL + (s0 + g) * A;
                const int zc = z < n / 2 ? z : z - n;
                const int q = xy + zc * zc;
                const size_t at = z * plane + at0;
                float2 c = make_float2(0.f, 0.f);
                if (mode == 1) {
                    const float2 u = fft::unpack(o[i][s0 + g]);
                    const float m = sqrtf(u.x * u.x + u.y * u.y);
                    const float wn = w[g] / fmaxf(m, 1e-6f);
                    if (in[g]) {
                        W[at] = wn;
                        dmax = fmaxf(dmax, fabsf(m - 1.f));
                        c.x = tt[g] * wn;
                    }
                } else if (in[g]) {
                    float tf = 0.f;
                    if (mode != 2) {
                        double d = f[g].z;
                        if (rfsc && q >= 25 * pf * pf)
                            d *= rfsc[min((int)rintf(sqrtf((float)q)) / pf, nFsc)];
                        tf = (float)fmax(d, 1e-25);
                    }
                    if (mode == 0) {
                        c.x = tf;
                        T[at] = tf;
                        W[at] = 1.f;
                    } else {
                        const float wn = mode == 2 ? w[g] : 1.f / fmaxf(tf, 1e-6f);
                        c = make_float2(f[g].x * wn, f[g].y * wn);
                    }
                }
                o[i][s0 + g] = fft::pack(c.y, c.x);   // exchanged: the inverse transform
            }
        }
    fft::run<B, A, S::TL>(o, v, fsm, tw, t, line);
#pragma unroll
    for (int i = 0; i < S::I1; i++)
#pragma unroll
        for (int r = 0; r < A; r++)
            if (t + i * S::TL < B)
                *reinterpret_cast<c64*>(p.C + (t + i * S::TL + r * B) * plane + at0) =
                    fft::swapped(v[i][r]);
    if (mode == 1) {
        for (int k = 16; k; k >>= 1) dmax = fmaxf(dmax, __shfl_xor_sync(0xffffffffu, dmax, k));
        if ((threadIdx.x & 31) == 0) atomicMax(diffBits, __float_as_uint(dmax));
    }
}

// CTA (8 pairs of rows, plane z): pair l holds the rows y = l and n - l (0 and
// n / 2 for l = 0), whose points share the kernel's argument, as the real and
// the imaginary part of one complex line.  With out: the real rows' central N
// points over tab to out [N][N][N]; else times the kernel and forward again.
// The kernel comes as a grid over one octant, kgrid [z][l / 8][x][8]: looked up
// in tab (over the integer squared radius) every point costs a sector of L2,
// four times the bytes of C; tab serves the row n / 2 of the pair 0.
template <int A, int B>
__global__ void __launch_bounds__(fft::Shape<A, B>::threads, 384 / fft::Shape<A, B>::threads)
k_reco_pass_x(const Pass3 p, const float* __restrict__ tab, const float* __restrict__ kgrid, int N,
              float* __restrict__ out)
{
    using S = fft::Shape<A, B>;
    extern __shared__ __align__(16) c64 fsm[];
    constexpr int n = S::n, h = n / 2;
    const int line = threadIdx.x % kFftLines, t = threadIdx.x / kFftLines;
    const int l = blockIdx.x * kFftLines + line;
    const float2* tw = pass_roots<A, B>(p, fsm);
    const int z = !out || blockIdx.y < N / 2 ? blockIdx.y : blockIdx.y + n - N;
    const int zc = z < h ? z : z - n;
    float2* C = p.C + (size_t)z * n * p.px;
    const int ll = min(l, h - 1);               // lines past the last pair are not stored
    // the 16 rows, copied whole and read in both directions (from global memory
    // every access would touch eight rows); their pitch spreads eight rows
    // over the banks
    const int pitch = (p.px + 15) / 16 * 16 + 2;
    float2* rows = reinterpret_cast<float2*>(fsm + S::smem / sizeof(c64));
    for (int i = threadIdx.x; i < 2 * kFftLines * (p.px / 2); i += S::threads) {
        const int r = i / (p.px / 2), e = 2 * (i % (p.px / 2));
        const int q = min(blockIdx.x * kFftLines + r % kFftLines, h - 1);
        const int y = r < kFftLines ? q : (q ? n - q : h);
        copy16(reinterpret_cast<float*>(rows + r * pitch + e),
               reinterpret_cast<const float*>(C + (size_t)y * p.px + e));
    }
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    const float2* row0 = rows + line * pitch;
    const float2* row1 = row0 + kFftLines * pitch;
    c64 v[S::I1][A], o[S::I2][B];
#pragma unroll
    for (int i = 0; i < S::I1; i++)
#pragma unroll
        for (int r = 0; r < A; r++) {
            const int k = t + i * S::TL + r * B;
            const int m = k < p.nxr ? k : n - k;     // the stored column, or the mirrored one
            const bool in = t + i * S::TL < B && m < p.nxr;
            const int ml = min(m, p.nxr - 1);
            const float2 a = row0[ml], b = row1[ml];
            // a + i b, real and imaginary part exchanged: the inverse transform
            const float2 u = k == 0      ? make_float2(b.x, a.x)
                             : k < p.nxr ? make_float2(a.y + b.x, a.x - b.y)
                                         : make_float2(b.x - a.y, a.x + b.y);
            v[i][r] = in ? fft::pack(u.x, u.y) : 0;
        }
    fft::run<A, B, S::TL>(v, o, fsm, tw, t, line);
    if (out) {
#pragma unroll
        for (int i = 0; i < S::I2; i++)
#pragma unroll
            for (int s = 0; s < B; s++) {
                const int x = t + i * S::TL + s * A;
                const int xc = x < h ? x : x - n, y1 = l ? -l : -h;
                if (t + i * S::TL >= A || l >= h || xc < -N / 2 || xc >= N / 2) continue;
                const float2 u = fft::unpack(o[i][s]);        // (row 1, row 0)
                const size_t at = ((size_t)(zc + N / 2) * N + N / 2) * N + xc + N / 2;
                if (l < N / 2) out[at + (long long)l * N] = u.y / tab[xc * xc + l * l + zc * zc];
                if (y1 >= -N / 2)
                    out[at + (long long)y1 * N] = u.x / tab[xc * xc + y1 * y1 + zc * zc];
            }
        return;
    }
    const int c = zc * zc + ll * ll;
    const float* kg = kgrid + ((size_t)abs(zc) * gridDim.x + blockIdx.x) * ((h + 1) * kFftLines) + line;
#pragma unroll
    for (int i = 0; i < S::I2; i++) {
        float kv[B];
#pragma unroll
        for (int s = 0; s < B; s++) {
            const int x = min(t + i * S::TL, A - 1) + s * A;
            const int xc = x <= h ? x : n - x;
            kv[s] = __ldg(kg + xc * kFftLines);
        }
#pragma unroll
        for (int s = 0; s < B; s++) {
            const int x = min(t + i * S::TL, A - 1) + s * A;
            const int xc = x <= h ? x : n - x;
            const float k1 = ll ? kv[s] : __ldg(tab + xc * xc + c + h * h);
            const float2 u = fft::unpack(o[i][s]);            // (row 1, row 0)
            o[i][s] = fft::pack(u.y * kv[s], u.x * k1);
        }
    }
    fft::run<B, A, S::TL>(o, v, fsm, tw, t, line);
    // the two rows' spectra from the line's at k and n - k, a warp along a row
    constexpr int lp = n + 2;
#pragma unroll
    for (int i = 0; i < S::I1; i++)
#pragma unroll
        for (int r = 0; r < A; r++)
            if (t + i * S::TL < B) fsm[line * lp + t + i * S::TL + r * B] = v[i][r];
    __syncthreads();
    for (int i = threadIdx.x; i < kFftLines * p.px; i += S::threads) {
        const int q = i / p.px, k = i % p.px, y = blockIdx.x * kFftLines + q;
        if (y >= h || k >= p.nxr) continue;
        const float2 a = fft::unpack(fsm[q * lp + k]), b = fft::unpack(fsm[q * lp + (k ? n - k : 0)]);
        C[(size_t)y * p.px + k] = make_float2(0.5f * (a.x + b.x), 0.5f * (a.y - b.y));
        C[(size_t)(y ? n - y : h) * p.px + k] = make_float2(0.5f * (a.y + b.y), 0.5f * (b.x - a.x));
    }
}

// kgrid [z][lt][x][8] = tab[x^2 + l^2 + z^2] for z, x <= h, l = 8 lt + lane
__global__ void k_reco_kernel_grid(const float* __restrict__ tab, int h, int lt,
                                   float* __restrict__ kgrid)
{
    const size_t total = (size_t)(h + 1) * lt * (h + 1) * kFftLines;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total;
         i += (size_t)gridDim.x * blockDim.x) {
        const unsigned u = (unsigned)(i / kFftLines);
        const int x = (int)(u % (h + 1)), w = (int)(u / (h + 1));
        const int l = min(w % lt * kFftLines + (int)(i % kFftLines), h), z = w / lt;
        kgrid[i] = tab[x * x + l * l + z * z];
    }
}

// sides with their two factors (the larger first)
#define TG3_RECO_SIDES(X)                                                                        \
    X(12, 8) X(16, 8) X(12, 12) X(16, 10) X(15, 12) X(16, 12) X(18, 12) X(16, 15) X(16, 16)      \
        X(18, 16) X(20, 16) X(20, 18) X(24, 16) X(20, 20) X(24, 18) X(24, 20) X(32, 16)

struct PassKernels {
    void (*y)(Pass3, int, int);
    void (*z)(Pass3, int, const float4*, const double*, int, int, float*, float*, unsigned*);
    void (*x)(Pass3, const float*, const float*, int, float*);
    int threads;
    size_t smem;
};

bool pass_kernels(int n, PassKernels* k)
{
#define X(a, b)                                                                                    \
    if (n == a * b) {                                                                              \
        *k = {k_reco_pass_y<a, b>, k_reco_pass_z<a, b>, k_reco_pass_x<a, b>,                       \
              fft::Shape<a, b>::threads, fft::Shape<a, b>::smem};                                  \
        return true;                                                                               \
    }
    TG3_RECO_SIDES(X)
#undef X
    return false;
}

// 1 / f of every shell of the FSC, f clamped and joined as in k_reco_init
__global__ void k_reco_rfsc(const double* __restrict__ fsc, int nFsc, int joinHalf,
                            double* __restrict__ rfsc)
{
    for (int u = blockIdx.x * blockDim.x + threadIdx.x; u <= nFsc; u += gridDim.x * blockDim.x) {
        double f = u < nFsc ? fsc[u] : 0.0;
        f = fmax(1e-3, fmin(1.0 - 1e-3, f));
        if (joinHalf) f = sqrt(2.0 * f / (1.0 + f));
        rfsc[u] = 1.0 / f;
    }
}

struct Plan3 {
    tg3_ctx* c;
    int vdim, nz, type;
    cufftHandle h;
};
std::vector<Plan3> g_plans3;
std::mutex g_plans3Lock;

// cuFFT plan of the padded grid: vdim^3 (nz = vdim) or vdim^2 (nz = 1)
int plan3(tg3_ctx* c, int vdim, int nz, cufftType type, cufftHandle* out)
{
    std::lock_guard<std::mutex> g(g_plans3Lock);
    for (auto& p : g_plans3)
        if (p.c == c && p.vdim == vdim && p.nz == nz && p.type == (int)type) {
            *out = p.h;
            return TG3_OK;
        }
    cufftHandle h;
    const cufftResult r = nz > 1 ? cufftPlan3d(&h, vdim, vdim, vdim, type)
                                 : cufftPlan2d(&h, vdim, vdim, type);
    if (r != CUFFT_SUCCESS) return fail(TG3_ERR_CUDA, "cuFFT plan creation failed");
    g_plans3.push_back({c, vdim, nz, (int)type, h});
    *out = h;
    return TG3_OK;
}

// ---- PrepareTF: normalisation and symmetrisation of the accumulators
constexpr int kMaxSym = 64;     // symmetry elements (the icosahedral group has 59 besides E)

struct SymMats {
    double m[kMaxSym * 9];
};

// src = acc, scaled by 1 / T at the origin when normalising (allReduceT's
// RECONSTRUCTOR_NORMALISE_T_F, src/Reconstructor.cpp:2453-2480).
__global__ void k_acc_scaled_copy(const float4* __restrict__ acc, size_t n, int normalise,
                                  float4* __restrict__ src)
{
    const float sf = normalise ? 1.0f / acc[0].z : 1.0f;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
         i += (size_t)gridDim.x * blockDim.x) {
        const float4 v = acc[i];
        src[i] = make_float4(v.x * sf, v.y * sf, v.z * sf, 0.f);
    }
}

// Trilinear sample of the (F, T) half grid at (x, y, z), the Friedel mate
// conjugated for x < 0 (Volume::getByInterpolationFT, LINEAR_INTERP).
__device__ __forceinline__ float3 sample_ft(const float4* __restrict__ v, int vdim, float x,
                                            float y, float z)
{
    float sgn = 1.f;
    if (x < 0.f) {
        x = -x;
        y = -y;
        z = -z;
        sgn = -1.f;
    }
    const int nx = vdim / 2 + 1;
    const float xf = floorf(x), yf = floorf(y), zf = floorf(z);
    const int x0 = (int)xf, y0 = (int)yf, z0 = (int)zf;
    const float fx = x - xf, fy = y - yf, fz = z - zf;
    const float wx[2] = {1.f - fx, fx}, wy[2] = {1.f - fy, fy}, wz[2] = {1.f - fz, fz};
    float3 o = make_float3(0.f, 0.f, 0.f);
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const int zz = z0 + k < 0 ? z0 + k + vdim : z0 + k;
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const int yy = y0 + j < 0 ? y0 + j + vdim : y0 + j;
            const float4* row = v + ((size_t)zz * vdim + yy) * nx + x0;
#pragma unroll
            for (int i = 0; i < 2; i++) {
                const float w = wx[i] * wy[j] * wz[k];
                const float4 c = __ldg(row + i);
                o.x += c.x * w;
                o.y += c.y * w;
                o.z += c.z * w;
            }
        }
    }
    o.y *= sgn;
    return o;
}

// acc = src + sum over the symmetry elements R of src sampled at R v for
// |R v|^2 < r2 (SYMMETRIZE_FT, include/Geometry/Transformation.h:170-196),
// T floored at 1e-25 (PrepareTF's symmetrizeT).  R v and its squared norm are
// formed in FP64 in the reference's order, ((m0 i + m1 j) + m2 k) and
// (a^2 + b^2) + c^2, with every product and sum rounded on its own (no fused
// multiply-add): a voxel whose rotated image lies on the sphere |u| = r up to
// rounding is then kept or dropped as the reference keeps or drops it.
__device__ __forceinline__ double dot3_rn(const double* m, double i, double j, double k)
{
    return __dadd_rn(__dadd_rn(__dmul_rn(m[0], i), __dmul_rn(m[1], j)), __dmul_rn(m[2], k));
}

__global__ void k_symmetrize(float4* __restrict__ acc, const float4* __restrict__ src, int vdim,
                             const SymMats mats, int nSym, double r2)
{
    const int nx = vdim / 2 + 1, half = vdim / 2;
    const size_t n = (size_t)vdim * vdim * nx;
    for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < n;
         q += (size_t)gridDim.x * blockDim.x) {
        const int i = (int)(q % nx);
        const int y = (int)((q / nx) % vdim), z = (int)(q / ((size_t)nx * vdim));
        const int j = y < half ? y : y - vdim, k = z < half ? z : z - vdim;
        float4 v = src[q];
        // a rotation keeps |v|: voxels well outside the sphere have nothing to add
        if ((double)(i * i + j * j + k * k) <= r2 + 1.0) {
            for (int s = 0; s < nSym; s++) {
                const double* m = mats.m + 9 * s;
                const double a = dot3_rn(m, i, j, k), b = dot3_rn(m + 3, i, j, k),
                             c = dot3_rn(m + 6, i, j, k);
                const double nn = __dadd_rn(__dadd_rn(__dmul_rn(a, a), __dmul_rn(b, b)),
                                            __dmul_rn(c, c));
                if (nn < r2) {
                    const float3 w = sample_ft(src, vdim, (float)a, (float)b, (float)c);
                    v.x += w.x;
                    v.y += w.y;
                    v.z += w.z;
                }
            }
        }
        v.z = fmaxf(v.z, 1e-25f);
        acc[q] = v;
    }
}

}  // namespace

void reco_release(tg3_ctx* c)
{
    std::lock_guard<std::mutex> g(g_plans3Lock);
    for (size_t i = 0; i < g_plans3.size();) {
        if (g_plans3[i].c == c) {
            cufftDestroy(g_plans3[i].h);
            g_plans3.erase(g_plans3.begin() + i);
        } else {
            i++;
        }
    }
}

}  // namespace tg3

using namespace tg3;

extern "C" int tg3_ctx_insert_load_d(tg3_ctx* c, const float* F, const float* T)
{
    int st = check_ctx(c);
    if (st) return st;
    if (!c->ins.acc) return fail(TG3_ERR_STATE, "no insertion accumulator (tg3_ctx_insert_begin)");
    if (!F || !T) return fail(TG3_ERR_ARG, "null device pointer");
    const int vdim = c->ins.vdim;
    const size_t n = (size_t)vdim * vdim * (vdim / 2 + 1);
    k_acc_load<<<152 * 8, 256, 0, c->stream>>>(reinterpret_cast<const float2*>(F), T, n, c->ins.acc);
    TG3_LAUNCH_CHECK("accumulator load");
    return TG3_OK;
}

namespace {

// The stopping rule of the balancing rounds: round m's largest ||C| - 1| read
// back and compared.
struct Balance {
    float diff = 3.4e38f;
    int noDecrease = 0;
    bool done(int m, float d)
    {
        noDecrease = d > diff * 0.95f ? noDecrease + 1 : 0;
        diff = d;
        return d < 1e-2f || (m >= 10 && noDecrease == 2);
    }
};

int read_diff(tg3_ctx* c, const unsigned* dBits, float* d)
{
    unsigned bits = 0;
    TG3_CUDA(cudaMemcpyAsync(&bits, dBits, sizeof(unsigned), cudaMemcpyDeviceToHost, c->stream));
    TG3_CUDA(cudaStreamSynchronize(c->stream));
    std::memcpy(d, &bits, sizeof(float));
    return TG3_OK;
}

// 3-D reconstruction by the passes above.
int reconstruct_passes(tg3_ctx* c, const PassKernels& k, const float4* acc, int n, int pf,
                       const double* fsc, int nFsc, int joinHalf, int maxRadius, int gridCorr,
                       int kernel, float a, float alpha, float* vol, int* rounds)
{
    int st = TG3_OK;
    const int N = n / pf, rmax = maxRadius * pf;
    Pass3 p;
    p.nxr = rmax;
    p.px = (rmax + kFftLines - 1) / kFftLines * kFftLines;
    p.r2max = (long long)rmax * rmax;
    const size_t cells = (size_t)n * n * p.px;
    auto up = [](size_t x) { return (x + 255) / 256 * 256; };
    const int nqPad = 3 * (n / 2) * (n / 2) + 1, nqBox = 3 * (N / 2) * (N / 2) + 1;
    const size_t oT = 0, oW = up(4 * cells), oC = oW + up(4 * cells), oD = oC + up(8 * cells),
                 oK = oD + 256, oE = oK + up(4 * (size_t)nqPad), oR = oE + up(4 * (size_t)nqBox),
                 oF = oR + up(8 * (size_t)n), oG = oF + up(8 * (size_t)(nFsc + 1));
    const int h = n / 2, lt = (h + kFftLines - 1) / kFftLines;
    const size_t total =
        oG + (gridCorr ? up(4 * (size_t)(h + 1) * lt * (h + 1) * kFftLines) : 256);
    char* b = (char*)ws_get(c, WS_RECO, total, &st);
    if (!b) return st;
    float* T = (float*)(b + oT);
    float* W = (float*)(b + oW);
    p.C = (float2*)(b + oC);
    unsigned* dBits = (unsigned*)(b + oD);
    float* tabK = (float*)(b + oK);
    float* tabE = (float*)(b + oE);
    p.tw = (float2*)(b + oR);
    double* rfsc = fsc ? (double*)(b + oF) : nullptr;
    float* kgrid = (float*)(b + oG);
    cudaStream_t s = c->stream;
    const size_t smemZ = k.smem + 2 * sizeof(float) * (size_t)n * kFftLines;
    const size_t smemX = k.smem + sizeof(float2) * 2 * kFftLines * ((p.px + 15) / 16 * 16 + 2);
    TG3_CUDA(allow_shared(k.y));
    TG3_CUDA(allow_shared(k.x));
    TG3_CUDA(allow_shared(k.z));
    const double i0a = bessel_i0(alpha), cellsD = (double)n * n * n;
    const double invNf = gridCorr ? 1.0 / mkb_rl(0.0, a, alpha, i0a) : 0.0;
    fft::k_roots<<<(n + 127) / 128, 128, 0, s>>>(const_cast<float2*>(p.tw), n);
    if (gridCorr) {
        k_radial_table<<<(nqPad + 255) / 256, 256, 0, s>>>(tabK, nqPad, (double)N * pf, 1, a, alpha,
                                                            i0a, invNf / cellsD, 1.0 / 100000);
        k_reco_kernel_grid<<<152 * 8, 256, 0, s>>>(tabK, h, lt, kgrid);
    }
    if (rfsc) k_reco_rfsc<<<(nFsc + 128) / 128, 128, 0, s>>>(fsc, nFsc, joinHalf, rfsc);
    const int xt = p.px / kFftLines;
    const dim3 gz(xt, 2 * rmax - 1), gy(xt, n), gx(lt, n);
    if (gridCorr)
        k.z<<<gz, k.threads, smemZ, s>>>(p, 0, acc, rfsc, nFsc, pf, T, W, nullptr);
    TG3_LAUNCH_CHECK("reconstruction set-up");
    Balance bal;
    int m = 0;
    for (m = 0; gridCorr && m < 30; m++) {
        k.y<<<gy, k.threads, k.smem, s>>>(p, 1, n);
        k.x<<<gx, k.threads, smemX, s>>>(p, tabK, kgrid, N, nullptr);
        k.y<<<gy, k.threads, k.smem, s>>>(p, 0, n);
        TG3_CUDA(cudaMemsetAsync(dBits, 0, sizeof(unsigned), s));
        k.z<<<gz, k.threads, smemZ, s>>>(p, 1, nullptr, nullptr, 0, pf, T, W, dBits);
        TG3_LAUNCH_CHECK("balancing round");
        float d = 0.f;
        if ((st = read_diff(c, dBits, &d))) return st;
        if (bal.done(m, d)) break;
    }
    if (rounds) *rounds = gridCorr ? std::min(m + 1, 30) : 0;
    const int mkb = kernel == TG3_KERNEL_MKB;
    const double nf = mkb ? mkb_rl(0.0, (double)a * pf, alpha, i0a) : 1.0;
    k_radial_table<<<(nqBox + 255) / 256, 256, 0, s>>>(tabE, nqBox, (double)pf * N, mkb,
                                                        (double)a * pf, alpha, i0a, cellsD / nf, 0.0);
    if (gridCorr)
        k.z<<<gz, k.threads, smemZ, s>>>(p, 2, acc, nullptr, 0, pf, T, W, nullptr);
    else
        k.z<<<gz, k.threads, smemZ, s>>>(p, 3, acc, rfsc, nFsc, pf, T, W, nullptr);
    k.y<<<dim3(xt, N), k.threads, k.smem, s>>>(p, 1, N);
    k.x<<<dim3(gx.x, N), k.threads, smemX, s>>>(p, tabE, nullptr, N, vol);
    TG3_LAUNCH_CHECK("map from F W");
    return TG3_OK;
}

// The reconstruction chain on an accumulator acc of vdim x vdim x (vdim/2+1)
// cells (nz = vdim, 3-D) or vdim x (vdim/2+1) (nz = 1, 2-D), into out: the
// central N^3 or N^2 of the padded real-space result, N = vdim / pf.
int reconstruct_core(tg3_ctx* c, const float4* acc, int vdim, int nz, int pf, const double* fsc,
                     int nFsc, int joinHalf, int maxRadius, int gridCorr, int kernel, float a,
                     float alpha, float* vol, int* rounds)
{
    int st = TG3_OK;
    const int N = vdim / pf;
    // 3-D grids of the listed sides: own transforms fused with the rounds' other
    // passes (512^3, 19 rounds: 48 -> 25 ms); other sides and the
    // single-plane grids of a 2-D class by the library's
    PassKernels own;
    if (nz > 1 && N * pf == vdim && N % 2 == 0 && pass_kernels(vdim, &own))
        return reconstruct_passes(c, own, acc, vdim, pf, fsc, nFsc, joinHalf, maxRadius, gridCorr,
                                  kernel, a, alpha, vol, rounds);
    const double cells = nz > 1 ? (double)vdim * vdim * vdim : (double)vdim * vdim;
    const size_t nh = (size_t)nz * vdim * (vdim / 2 + 1), nr = (size_t)nz * vdim * vdim;
    auto up = [](size_t x) { return (x + 255) / 256 * 256; };
    const int nqPad = 3 * (vdim / 2) * (vdim / 2) + 1, nqBox = 3 * (N / 2) * (N / 2) + 1;
    const size_t oT = 0, oW = up(4 * nh), oC = oW + up(4 * nh), oR = oC + up(8 * nh),
                 oD = oR + up(4 * nr), oK = oD + 256, oE = oK + up(4 * (size_t)nqPad),
                 total = oE + up(4 * (size_t)nqBox);
    char* b = (char*)ws_get(c, WS_RECO, total, &st);
    if (!b) return st;
    float* T = (float*)(b + oT);
    float* W = (float*)(b + oW);
    float2* C = (float2*)(b + oC);
    float* R = (float*)(b + oR);
    unsigned* dBits = (unsigned*)(b + oD);
    float* tabK = (float*)(b + oK);
    float* tabE = (float*)(b + oE);
    cudaStream_t s = c->stream;
    const long long r2max = (long long)maxRadius * pf * maxRadius * pf;
    const int G = 152 * 8;
    k_reco_init<<<G, 256, 0, s>>>(acc, vdim, nz, pf, fsc, nFsc, joinHalf, r2max, T, W);
    TG3_LAUNCH_CHECK("reconstruction set-up");
    const double i0a = bessel_i0(alpha);
    int m = 0;
    if (gridCorr) {
        cufftHandle inv, fwd;
        if ((st = plan3(c, vdim, nz, CUFFT_C2R, &inv)) || (st = plan3(c, vdim, nz, CUFFT_R2C, &fwd)))
            return st;
        if (cufftSetStream(inv, s) != CUFFT_SUCCESS || cufftSetStream(fwd, s) != CUFFT_SUCCESS)
            return fail(TG3_ERR_CUDA, "cuFFT stream");
        const double invNf = 1.0 / mkb_rl(0.0, a, alpha, i0a);
        k_radial_table<<<(nqPad + 255) / 256, 256, 0, s>>>(tabK, nqPad, (double)N * pf, 1, a, alpha,
                                                            i0a, invNf / cells, 1.0 / 100000);
        TG3_LAUNCH_CHECK("balancing kernel table");
        Balance bal;
        k_reco_tw<<<G, 256, 0, s>>>(T, W, nh, C);
        TG3_LAUNCH_CHECK("balancing C = T W");
        for (m = 0; m < 30; m++) {
            k_reco_pair<<<G, 256, 0, s>>>(C, vdim, nz);
            if (cufftExecC2R(inv, reinterpret_cast<cufftComplex*>(C), R) != CUFFT_SUCCESS)
                return fail(TG3_ERR_CUDA, "cuFFT inverse transform failed");
            k_reco_kernel_rl<<<G, 256, 0, s>>>(R, vdim, nz, tabK);
            TG3_LAUNCH_CHECK("balancing kernel product");
            if (cufftExecR2C(fwd, R, reinterpret_cast<cufftComplex*>(C)) != CUFFT_SUCCESS)
                return fail(TG3_ERR_CUDA, "cuFFT forward transform failed");
            TG3_CUDA(cudaMemsetAsync(dBits, 0, sizeof(unsigned), s));
            k_reco_update<<<G, 256, 0, s>>>(C, T, vdim, nz, r2max, W, dBits);
            TG3_LAUNCH_CHECK("balancing update");
            float d = 0.f;
            if ((st = read_diff(c, dBits, &d))) return st;
            if (bal.done(m, d)) break;
        }
    } else {
        k_reco_w_from_t<<<G, 256, 0, s>>>(T, vdim, nz, r2max, W);
        TG3_LAUNCH_CHECK("W from T");
    }
    if (rounds) *rounds = gridCorr ? std::min(m + 1, 30) : 0;
    cufftHandle inv;
    if ((st = plan3(c, vdim, nz, CUFFT_C2R, &inv))) return st;
    if (cufftSetStream(inv, s) != CUFFT_SUCCESS) return fail(TG3_ERR_CUDA, "cuFFT stream");
    k_reco_fw<<<G, 256, 0, s>>>(acc, W, vdim, nz, r2max, C);
    k_reco_pair<<<G, 256, 0, s>>>(C, vdim, nz);
    TG3_LAUNCH_CHECK("F W");
    if (cufftExecC2R(inv, reinterpret_cast<cufftComplex*>(C), R) != CUFFT_SUCCESS)
        return fail(TG3_ERR_CUDA, "cuFFT inverse transform failed");
    const int mkb = kernel == TG3_KERNEL_MKB;
    const double nf = mkb ? mkb_rl(0.0, (double)a * pf, alpha, i0a) : 1.0;
    // gridding correction: the map (times the cell count after the
    // unnormalised inverse) over the kernel's real-space transform at
    // |x| / (pf N)
    k_radial_table<<<(nqBox + 255) / 256, 256, 0, s>>>(tabE, nqBox, (double)pf * N, mkb,
                                                        (double)a * pf, alpha, i0a, cells / nf, 0.0);
    TG3_LAUNCH_CHECK("gridding correction table");
    k_reco_extract<<<G, 256, 0, s>>>(R, vdim, nz, N, tabE, vol);
    TG3_LAUNCH_CHECK("extract and gridding correction");
    return TG3_OK;
}

}  // namespace

extern "C" int tg3_ctx_reconstruct_d(tg3_ctx* c, const double* fsc, int nFsc, int joinHalf,
                                     int maxRadius, int gridCorr, int kernel, float a,
                                     float alpha, float* vol, int* rounds)
{
    int st = check_ctx(c);
    if (st) return st;
    if (!c->ins.acc) return fail(TG3_ERR_STATE, "no insertion accumulator (tg3_ctx_insert_begin)");
    if (!vol || maxRadius <= 0 || (fsc && nFsc <= 0) ||
        (kernel != TG3_KERNEL_MKB && kernel != TG3_KERNEL_TRILINEAR))
        return fail(TG3_ERR_ARG, "bad reconstruction arguments");
    if ((gridCorr || kernel == TG3_KERNEL_MKB) && !(a > 0 && alpha > 0))
        return fail(TG3_ERR_ARG, "MKB parameters a and alpha must be positive");
    const int vdim = c->ins.vdim, pf = c->ins.pf;
    if (maxRadius * pf > vdim / 2) return fail(TG3_ERR_ARG, "maxRadius beyond the padded grid");
    // 32-bit voxel indices in the kernels
    if ((size_t)vdim * vdim * vdim >= (1ull << 31)) return fail(TG3_ERR_UNSUPPORTED, "padded grid above 1290^3");
    return reconstruct_core(c, c->ins.acc, vdim, vdim, pf, fsc, nFsc, joinHalf, maxRadius,
                            gridCorr, kernel, a, alpha, vol, rounds);
}

// The offsets' symmetrisation of Reconstructor::symmetrizeO (src/Reconstructor.cpp,
// under RECONSTRUCTOR_SYMMETRIZE_DURING_RECONSTRUCT): O += sum_s R_s O over
// the symmetry elements besides the identity (each R_s applied to the
// unsymmetrised O), counter *= 1 + nSym.  Host arithmetic.
extern "C" int tg3_SymmetrizeO(double* O3D, int* counter, const double* symMat, int nSym)
{
    if (!O3D || !counter || nSym < 0 || (nSym > 0 && !symMat))
        return fail(TG3_ERR_ARG, "bad symmetrizeO arguments");
    const double o[3] = {O3D[0], O3D[1], O3D[2]};
    double r[3] = {o[0], o[1], o[2]};
    for (int e = 0; e < nSym; e++) {
        const double* m = symMat + 9 * e;
        for (int i = 0; i < 3; i++) r[i] += m[3 * i] * o[0] + m[3 * i + 1] * o[1] + m[3 * i + 2] * o[2];
    }
    O3D[0] = r[0];
    O3D[1] = r[1];
    O3D[2] = r[2];
    *counter *= 1 + nSym;
    return TG3_OK;
}

// 2-D reconstruction (Reconstructor::reconstruct(Image&), MODE_2D): the same
// chain on one class's 2-D accumulators, host buffers in and out.
extern "C" int tg3_Reconstruct2D(const float* F2D, const float* T2D, int vdim, int pf,
                                 const double* fsc, int nFsc, int joinHalf, int maxRadius,
                                 int gridCorr, int kernel, float a, float alpha, float* img,
                                 int* rounds)
{
    if (!F2D || !T2D || !img || vdim < 4 || (vdim & 1) || pf < 1 || vdim % pf ||
        maxRadius <= 0 || maxRadius * pf > vdim / 2 || (fsc && nFsc <= 0) ||
        (kernel != TG3_KERNEL_MKB && kernel != TG3_KERNEL_TRILINEAR))
        return fail(TG3_ERR_ARG, "bad 2-D reconstruction arguments");
    if ((gridCorr || kernel == TG3_KERNEL_MKB) && !(a > 0 && alpha > 0))
        return fail(TG3_ERR_ARG, "MKB parameters a and alpha must be positive");
    int dev = 0;
    TG3_CUDA(cudaGetDevice(&dev));
    static std::mutex mu;
    static tg3_ctx* ctxs[64] = {};
    if (dev < 0 || dev >= 64) return fail(TG3_ERR_ARG, "device ordinal out of range");
    int st = TG3_OK;
    tg3_ctx* c = nullptr;
    {
        std::lock_guard<std::mutex> lk(mu);
        if (!ctxs[dev] && (st = tg3_ctx_create(&ctxs[dev], dev))) return st;
        c = ctxs[dev];
    }
    const size_t nh = (size_t)vdim * (vdim / 2 + 1);
    const int N = vdim / pf;
    const size_t oA = 0, oF = (sizeof(float4) * nh + 255) / 256 * 256,
                 oT = oF + (sizeof(float2) * nh + 255) / 256 * 256,
                 oO = oT + (sizeof(float) * nh + 255) / 256 * 256,
                 total = oO + sizeof(float) * (size_t)N * N;
    char* b = (char*)ws_get(c, WS_RECO2D, total, &st);
    if (!b) return st;
    cudaStream_t s = c->stream;
    double* dFsc = nullptr;
    if (fsc) {
        dFsc = (double*)ws_get(c, WS_MISC, sizeof(double) * nFsc, &st);
        if (!dFsc) return st;
        TG3_CUDA(cudaMemcpyAsync(dFsc, fsc, sizeof(double) * nFsc, cudaMemcpyHostToDevice, s));
    }
    TG3_CUDA(cudaMemcpyAsync(b + oF, F2D, sizeof(float2) * nh, cudaMemcpyHostToDevice, s));
    TG3_CUDA(cudaMemcpyAsync(b + oT, T2D, sizeof(float) * nh, cudaMemcpyHostToDevice, s));
    float4* acc = (float4*)(b + oA);
    k_acc_load<<<152 * 2, 256, 0, s>>>((const float2*)(b + oF), (const float*)(b + oT), nh, acc);
    TG3_LAUNCH_CHECK("2-D accumulator load");
    if ((st = reconstruct_core(c, acc, vdim, 1, pf, dFsc, nFsc, joinHalf, maxRadius, gridCorr,
                               kernel, a, alpha, (float*)(b + oO), rounds)))
        return st;
    TG3_CUDA(cudaMemcpyAsync(img, b + oO, sizeof(float) * (size_t)N * N, cudaMemcpyDeviceToHost,
                             s));
    return tg3_ctx_sync(c);
}

extern "C" int tg3_ctx_prepare_tf_d(tg3_ctx* c, const double* symMat, int nSym, int maxRadius,
                                    int normalise)
{
    int st = check_ctx(c);
    if (st) return st;
    if (!c->ins.acc) return fail(TG3_ERR_STATE, "no insertion accumulator (tg3_ctx_insert_begin)");
    if (nSym < 0 || nSym > kMaxSym || (nSym > 0 && !symMat))
        return fail(TG3_ERR_ARG, "symmetry elements: 0 to 64 matrices");
    const int vdim = c->ins.vdim, pf = c->ins.pf;
    const double r = (double)maxRadius * pf + 1.0;
    if (maxRadius <= 0 || r + 1.0 > vdim / 2)
        return fail(TG3_ERR_ARG, "maxRadius x pf + 2 must not exceed vdim / 2");
    SymMats mats;
    for (int i = 0; i < 9 * nSym; i++) mats.m[i] = symMat[i];
    const size_t n = (size_t)vdim * vdim * (vdim / 2 + 1);
    float4* src = (float4*)ws_get(c, WS_RECO, sizeof(float4) * n, &st);
    if (!src) return st;
    cudaStream_t s = c->stream;
    k_acc_scaled_copy<<<152 * 8, 256, 0, s>>>(c->ins.acc, n, normalise, src);
    TG3_LAUNCH_CHECK("accumulator copy");
    k_symmetrize<<<152 * 16, 256, 0, s>>>(c->ins.acc, src, vdim, mats, nSym, r * r);
    TG3_LAUNCH_CHECK("symmetrisation");
    return TG3_OK;
}

extern "C" int tg3_PrepareTF(float* F3D, float* T3D, int vdim, const double* symMat, int nSym,
                             int maxRadius, int pf)
{
    if (!F3D || !T3D || vdim < 4 || (vdim & 1) || pf < 1)
        return fail(TG3_ERR_ARG, "bad PrepareTF arguments");
    int dev = 0;
    TG3_CUDA(cudaGetDevice(&dev));
    static std::mutex mu;
    static tg3_ctx* ctxs[64] = {};
    if (dev < 0 || dev >= 64) return fail(TG3_ERR_ARG, "device ordinal out of range");
    tg3_ctx* c = nullptr;
    int st = TG3_OK;
    {
        std::lock_guard<std::mutex> lk(mu);
        if (!ctxs[dev] && (st = tg3_ctx_create(&ctxs[dev], dev))) return st;
        c = ctxs[dev];
    }
    if ((st = tg3_ctx_insert_begin(c, vdim, pf))) return st;
    const size_t n = (size_t)vdim * vdim * (vdim / 2 + 1);
    float* d = (float*)ws_get(c, WS_D2H, sizeof(float) * 3 * n, &st);
    if (!d) return st;
    cudaStream_t s = c->stream;
    TG3_CUDA(cudaMemcpyAsync(d, F3D, sizeof(float) * 2 * n, cudaMemcpyHostToDevice, s));
    TG3_CUDA(cudaMemcpyAsync(d + 2 * n, T3D, sizeof(float) * n, cudaMemcpyHostToDevice, s));
    if ((st = tg3_ctx_insert_load_d(c, d, d + 2 * n))) return st;
    if ((st = tg3_ctx_prepare_tf_d(c, symMat, nSym, maxRadius, 1))) return st;
    if ((st = tg3_ctx_insert_read_d(c, d, d + 2 * n, 0))) return st;
    TG3_CUDA(cudaMemcpyAsync(F3D, d, sizeof(float) * 2 * n, cudaMemcpyDeviceToHost, s));
    TG3_CUDA(cudaMemcpyAsync(T3D, d + 2 * n, sizeof(float) * n, cudaMemcpyDeviceToHost, s));
    TG3_CUDA(cudaStreamSynchronize(s));
    return TG3_OK;
}
