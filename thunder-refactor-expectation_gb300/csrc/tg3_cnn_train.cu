// tg3_cnn_train.cu -- the pose network's convolutions in FP32 on the CUDA
// cores: forward, gradient with respect to the input, gradient with respect
// to the weights.
//
// Activations and gradients stay FP32 [n][channel][row][column]; the weights
// come repacked (k_repack), rounded to bf16 where the network uses them so.
// All three are bound by the FP32 pipe and built on fma.rn.f32x2 (two
// multiply-adds an issue): 8 x 8 outputs a thread (forward and data
// gradient) or 8 output channels x 9 taps over pixel pairs (weight
// gradient), so that a warp's shared loads (a cycle for every 128 bytes
// returned) stay below its multiply-adds.  At 256 images the six layers take
// 0.76 ms forward (47 TFLOP/s), 0.82 ms data gradient, 1.36 ms weight gradient;
// with one output pixel x 16 channels a thread, loads from global memory and
// scalar multiply-adds they took 2.8, 12.8 and 13.1 ms.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "tg3_internal.cuh"

namespace tg3 {
namespace {

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

__device__ __forceinline__ void fma2(uint64_t& d, uint64_t a, uint64_t b)
{
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}

// 4-byte asynchronous copy to shared memory, zeros when !ok
__device__ __forceinline__ void cp4(float* dst, const float* src, bool ok)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(
                     (uint32_t)__cvta_generic_to_shared(dst)),
                 "l"(src), "r"(ok ? 4 : 0)
                 : "memory");
}

__device__ __forceinline__ void cp16(float* dst, const float* src, bool ok)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(
                     (uint32_t)__cvta_generic_to_shared(dst)),
                 "l"(src), "r"(ok ? 16 : 0)
                 : "memory");
}

__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }

template <int N>
__device__ __forceinline__ void cp_wait()
{
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// ------------------------------------------------- forward / data gradient --
// y[n][co][p] = epilogue(sum over ci, tap row r, tap column c of
//               Wt[(ci NK + r NKX + c)][co] x[n][ci][p S + (r, c) - pad])
// on an HO x HO grid of output pixels, pad 1 for 3 taps and 0 for fewer.
//   3 x 3, S 1 or 2: the forward convolution; S 1 also the data gradient of a
//     stride-1 layer (flipped taps).
//   1 or 2 taps a side, S 1: one parity class of a stride-2 layer's data
//     gradient -- the input pixels (2 oy + py, 2 ox + px) take 1 + py rows and
//     1 + px columns of taps, and the class writes them only.
// Every output is one chain of fused multiply-adds over ci, r, c ascending.
//
// CTA: 256 output pixels x 8 NW output channels, a warp per 8 channels; a
// lane takes two groups of 4 neighbouring pixels of a row (64 accumulators in
// pairs of channels).  Per input channel and tap row a lane reads its 4 +
// taps - 1 columns once for all taps, and 8 weights a tap (uniform over the
// warp): 12 floats for 32 paired multiply-adds.  Slices of CI input channels
// go through two shared buffers by cp.async (zeros at the borders).  For
// S 2 a staged row holds the odd columns (from -1) and the even columns apart,
// so both strides read neighbouring floats.  The lanes of a quarter warp
// take rows whose offsets differ by whole groups of banks (row_of).
template <int NKY, int NKX, int S, int HO>
struct ConvShape {
    static constexpr int RT = HO < 256 / HO ? HO : 256 / HO;      // output rows of an image
    static constexpr int IT = 256 / (RT * HO);                    // images of a tile
    static constexpr int HI = HO * S;
    static constexpr int PAD = NKX == 3 ? 1 : 0;
    static constexpr int RI = (RT - 1) * S + NKY;                 // staged rows of an image
    static constexpr int CW = (HO - 1) * S + NKX;                 // staged columns
    static constexpr int PO = HO + 4;                             // S 2: odd columns, padded
    static constexpr int PW = S == 2     ? PO + HO
                              : HO == 16 ? 20
                              : HO == 8  ? 12
                                         : (HO + NKX - 1 + 3) / 4 * 4;
    static constexpr int CS = IT * RI * PW;                       // floats of a staged channel
    static constexpr int NE = IT * RI * CW;                       // copied ones
    // image and row of lane group g (0 .. 31) of the first 128 pixels
    __device__ static void row_of(int g, int* img, int* row, int* col)
    {
        if (HO >= 32) {
            *img = 0;
            *row = g / (HO / 4);
            *col = g % (HO / 4);
        } else if (HO == 16) {
            const int h = (g >> 2) & 1, q = g >> 3;
            *img = 0;
            *col = g & 3;
            *row = S == 2 ? (q & 1) + 2 * h + 4 * (q >> 1) : q + 4 * h;
        } else {
            const int h = (g >> 1) & 3, q = g >> 3;
            *img = q >> 1;
            *col = g & 1;
            *row = S == 2 ? h + 4 * (q & 1) : (q & 1) + 2 * h;
        }
    }
};

struct ConvArgs {
    const float* x;      // [n][cin][HI][HI]
    const float* wt;     // [cin taps][cout]
    const float* bias;   // forward: [cout]; null for the data gradient
    const float* act;    // data gradient: the ReLU output that the result passes back through
    float* y;
    int n, cin, cout;
};

template <int NKY, int NKX, int S, int HO, int CI, int NW>
__host__ __device__ constexpr size_t conv_smem()
{
    return 2 * sizeof(float) *
           (size_t)(CI * ConvShape<NKY, NKX, S, HO>::CS + CI * NKY * NKX * 8 * NW);
}

// py, px >= 0: a parity class of a stride-2 data gradient
template <int NKY, int NKX, int S, int HO, int CI, int NW>
__device__ __forceinline__ void conv_tile(const ConvArgs& p, float* sm, int tile, int cob, int py,
                                          int px)
{
    using Sh = ConvShape<NKY, NKX, S, HO>;
    constexpr int NT = 32 * NW, NK = NKY * NKX, CO = 8 * NW, HI = Sh::HI;
    constexpr int XS = CI * Sh::CS, WS = CI * NK * CO;       // floats of a stage
    constexpr int NP = (Sh::NE + NT - 1) / NT;               // copied positions a thread
    float* xs = sm;
    float* wsm = sm + 2 * XS;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int TPI = HO / Sh::RT;                         // tiles of an image (IT == 1)
    const int n0 = Sh::IT > 1 ? tile * Sh::IT : tile / TPI;
    const int oy0 = Sh::IT > 1 ? 0 : tile % TPI * Sh::RT;
    // the staged positions of this thread, the same for every channel
    int gsrc[NP], sdst[NP];
#pragma unroll
    for (int i = 0; i < NP; i++) {
        const int e = tid + i * NT;
        const int im = e / (Sh::RI * Sh::CW), r = e / Sh::CW % Sh::RI, c = e % Sh::CW;
        const int iy = oy0 * S + r - (NKY == 3 ? 1 : 0), ix = c - Sh::PAD;
        const bool in = e < Sh::NE && n0 + im < p.n && iy >= 0 && iy < HI && ix >= 0 && ix < HI;
        gsrc[i] = in ? im * p.cin * HI * HI + iy * HI + ix : -1;
        sdst[i] = e < Sh::NE ? (im * Sh::RI + r) * Sh::PW +
                                   (S == 2 ? ((c & 1) ? Sh::PO + (c >> 1) : (c >> 1)) : c)
                             : -1;
    }
    const float* xn = p.x + (size_t)n0 * p.cin * HI * HI;
    auto stage = [&](int ci0, int buf) {
        float* xd = xs + buf * XS;
#pragma unroll
        for (int ci = 0; ci < CI; ci++) {
            const float* src = xn + (size_t)(ci0 + ci) * HI * HI;
#pragma unroll
            for (int i = 0; i < NP; i++)
                if (sdst[i] >= 0)
                    cp4(xd + ci * Sh::CS + sdst[i], src + max(gsrc[i], 0), gsrc[i] >= 0);
        }
        const float* ws = p.wt + (size_t)ci0 * NK * p.cout + cob * CO;
        float* wd = wsm + buf * WS;
        for (int e = tid; e < WS / 4; e += NT) {
            const int row = e / (CO / 4), q = e % (CO / 4);
            cp16(wd + row * CO + 4 * q, ws + (size_t)row * p.cout + 4 * q, true);
        }
        cp_commit();
    };
    int im, row, col;
    Sh::row_of(lane, &im, &row, &col);
    // the second group: the next 128 pixels
    constexpr int DI = HO == 8 ? 2 : 0, DR = HO == 8 ? 0 : 128 / HO;
    const int xo = (im * Sh::RI + row * S) * Sh::PW + 4 * col;
    constexpr int xd2 = (DI * Sh::RI + DR * S) * Sh::PW;
    uint64_t acc[4][8];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 8; j++) acc[i][j] = 0ull;
    const int ns = p.cin / CI;
    stage(0, 0);
    for (int s = 0; s < ns; s++) {
        if (s + 1 < ns) {
            stage((s + 1) * CI, (s + 1) & 1);
            cp_wait<1>();
        } else {
            cp_wait<0>();
        }
        __syncthreads();
        const float* xb = xs + (s & 1) * XS + xo;
        const float* wb = wsm + (s & 1) * WS + warp * 8;
#pragma unroll 1
        for (int ci = 0; ci < CI; ci++) {
#pragma unroll
            for (int r = 0; r < NKY; r++) {
                // this tap row's columns: v[g][c + j] is tap column c of pixel j (S 1);
                // S 2: odd columns v[g][0 .. 4], even columns u[g][0 .. 3]
                float v[2][6], u[2][4];
#pragma unroll
                for (int g = 0; g < 2; g++) {
                    const float* q = xb + ci * Sh::CS + r * Sh::PW + g * xd2;
                    const float4 a = *reinterpret_cast<const float4*>(q);
                    v[g][0] = a.x;
                    v[g][1] = a.y;
                    v[g][2] = a.z;
                    v[g][3] = a.w;
                    if (S == 2) {
                        v[g][4] = q[4];
                        const float4 b = *reinterpret_cast<const float4*>(q + Sh::PO);
                        u[g][0] = b.x;
                        u[g][1] = b.y;
                        u[g][2] = b.z;
                        u[g][3] = b.w;
                    } else if (NKX == 3) {
                        const float2 b = *reinterpret_cast<const float2*>(q + 4);
                        v[g][4] = b.x;
                        v[g][5] = b.y;
                    } else if (NKX == 2) {
                        v[g][4] = q[4];
                    }
                }
#pragma unroll
                for (int c = 0; c < NKX; c++) {
                    const float* wq = wb + (ci * NK + r * NKX + c) * CO;
                    const ulonglong2 w0 = *reinterpret_cast<const ulonglong2*>(wq);
                    const ulonglong2 w1 = *reinterpret_cast<const ulonglong2*>(wq + 4);
#pragma unroll
                    for (int j = 0; j < 8; j++) {
                        const int g = j >> 2, k = j & 3;
                        const float xv = S == 2 ? (c == 1 ? u[g][k] : v[g][k + (c >> 1)])
                                                : v[g][k + c];
                        const uint64_t xx = pack2(xv, xv);
                        fma2(acc[0][j], w0.x, xx);
                        fma2(acc[1][j], w0.y, xx);
                        fma2(acc[2][j], w1.x, xx);
                        fma2(acc[3][j], w1.y, xx);
                    }
                }
            }
        }
        __syncthreads();
    }
    const int co0 = cob * CO + warp * 8;
#pragma unroll
    for (int g = 0; g < 2; g++) {
        const int n = n0 + im + g * DI, oy = oy0 + row + g * DR;
        if (n >= p.n) continue;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            float2 o[4];
#pragma unroll
            for (int k = 0; k < 4; k++) o[k] = unpack2(acc[i][4 * g + k]);
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int co = co0 + 2 * i + h;
                float4 v = h ? make_float4(o[0].y, o[1].y, o[2].y, o[3].y)
                             : make_float4(o[0].x, o[1].x, o[2].x, o[3].x);
                if (py >= 0) {
                    const size_t at = ((size_t)n * p.cout + co) * (4 * HO * HO) +
                                      (size_t)(2 * oy + py) * (2 * HO) + 8 * col + px;
                    const float w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                    for (int k = 0; k < 4; k++)
                        p.y[at + 2 * k] = p.act[at + 2 * k] > 0.f ? w[k] : 0.f;
                    continue;
                }
                const size_t at = (((size_t)n * p.cout + co) * HO + oy) * HO + 4 * col;
                if (p.bias) {
                    const float b = p.bias[co];
                    v = make_float4(fmaxf(v.x + b, 0.f), fmaxf(v.y + b, 0.f), fmaxf(v.z + b, 0.f),
                                    fmaxf(v.w + b, 0.f));
                } else {
                    const float4 a = *reinterpret_cast<const float4*>(p.act + at);
                    v = make_float4(a.x > 0.f ? v.x : 0.f, a.y > 0.f ? v.y : 0.f,
                                    a.z > 0.f ? v.z : 0.f, a.w > 0.f ? v.w : 0.f);
                }
                *reinterpret_cast<float4*>(p.y + at) = v;
            }
        }
    }
}

template <int S, int HO, int CI, int NW>
__global__ void __launch_bounds__(32 * NW, 16 / NW)
k_conv(const ConvArgs p)
{
    extern __shared__ __align__(16) float sm[];
    conv_tile<3, 3, S, HO, CI, NW>(p, sm, blockIdx.x, blockIdx.y, -1, -1);
}

// The four parity classes of a stride-2 layer's data gradient (blockIdx.z,
// the one with most taps first); the class's weights follow one another in wt.
template <int HO, int NW>
__global__ void __launch_bounds__(32 * NW, 16 / NW)
k_conv_classes(const ConvArgs p)
{
    extern __shared__ __align__(16) float sm[];
    ConvArgs q = p;
    const size_t cc = (size_t)p.cin * p.cout;
    if (blockIdx.z == 0) {
        conv_tile<2, 2, 1, HO, 8, NW>(q, sm, blockIdx.x, blockIdx.y, 1, 1);
    } else if (blockIdx.z == 1) {
        q.wt = p.wt + 4 * cc;
        conv_tile<2, 1, 1, HO, 8, NW>(q, sm, blockIdx.x, blockIdx.y, 1, 0);
    } else if (blockIdx.z == 2) {
        q.wt = p.wt + 6 * cc;
        conv_tile<1, 2, 1, HO, 8, NW>(q, sm, blockIdx.x, blockIdx.y, 0, 1);
    } else {
        q.wt = p.wt + 8 * cc;
        conv_tile<1, 1, 1, HO, 8, NW>(q, sm, blockIdx.x, blockIdx.y, 0, 0);
    }
}

// -------------------------------------------------------- weight gradient --
// dW[co][ci][tap] += sum over images and pixels of dy[co][p] x[ci][p S + tap -
// 1], db[co] += sum dy[co].  CTA: 32 output x 32 input channels over a share
// of the batch's chunks of 64 output pixels; a warp takes 8 output channels, a
// lane one input channel: 8 x 9 sums, each as a pair over even and odd
// columns (the operands' own layout, no move), added at the end.  Per 4
// pixels a lane reads 32 gradients (uniform over the warp) and 18 (S 1) or 27
// (S 2) inputs for 144 paired multiply-adds.  Chunks go through two shared
// buffers by cp.async; the channel pitch over 4 is odd, so a quarter warp's
// float4 reads fall in distinct banks.
//
// Sums of a batch are long (262,144 terms a weight at 256 images of 32 x 32
// pixels), so they are taken in three steps: a thread's FP32 chains end after
// kGradChain terms and are added to its place in the CTA's part (global memory,
// which stays in L2), and the CTAs' parts meet in 48 bits and FP64 in a fixed order
// (k_grad_sum).  Error of a layer's gradient at 256 images, restated on the CPU:
// 0.9 to 1.3e-7 of its norm; with one chain a CTA and atomic adds 2.0 to 3.8e-7.
//
// A gradient of zero takes no part, whatever it would be multiplied with: the
// ReLU maps what is not a number to zero and passes no gradient there.  The
// chains multiply all pairs; a CTA that meets a sum that is not finite does
// its share again, leaving out the zeros.
constexpr int kGradChain = 64;                               // a multiple of a chunk's 32
constexpr int kGradPart = 72 * 128;                          // sums of a CTA
constexpr int kGradCtas = 320;                               // most CTAs of a launch

// the CTA's sums v[i][k] added to its part (or the first of it); whether all
// are finite
__device__ __forceinline__ bool add_to_part(uint64_t (&acc)[8][9], float* part, bool first)
{
    bool finite = true;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        float old[9];
#pragma unroll
        for (int k = 0; k < 9; k++) old[k] = first ? 0.f : part[(i * 9 + k) * 128];
#pragma unroll
        for (int k = 0; k < 9; k++) {
            const float2 v = unpack2(acc[i][k]);
            const float s = v.x + v.y + old[k];
            finite &= fabsf(s) < INFINITY;
            part[(i * 9 + k) * 128] = s;
            acc[i][k] = 0ull;
        }
    }
    return finite;
}

template <int S, int HO>
struct GradShape {
    static constexpr int RT = 64 / HO;                       // output rows of a chunk
    static constexpr int HI = HO * S;
    static constexpr int RI = (RT - 1) * S + 3;
    static constexpr int CW = (HO - 1) * S + 3;
    static constexpr int PO = HO + 4;
    static constexpr int PW = S == 2 ? PO + HO : (HO + 2 + 3) / 4 * 4;
    static constexpr int CS = (RI * PW / 4) % 2 ? RI * PW : RI * PW + 4;
    static constexpr int XS = 32 * CS, YS = 32 * 64;         // floats of a stage
    static constexpr size_t bytes = 2 * sizeof(float) * (XS + YS);
};

template <int S, int HO>
__global__ void __launch_bounds__(128, 2)
k_conv_grad(const float* __restrict__ x, const float* __restrict__ dy, float* __restrict__ parts,
            float* __restrict__ biasParts, int n, int cin, int cout)
{
    using G = GradShape<S, HO>;
    constexpr int HI = G::HI, CPI = HO / G::RT;              // chunks of an image
    extern __shared__ __align__(16) float sm[];
    float* xs = sm;
    float* ys = sm + 2 * G::XS;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int co0 = blockIdx.x * 32, ci0 = blockIdx.y * 32;
    const int chunks = n * CPI;
    const int c0 = (int)((long long)chunks * blockIdx.z / gridDim.z);
    const int c1 = (int)((long long)chunks * (blockIdx.z + 1) / gridDim.z);
    auto stage = [&](int ch, int buf) {
        const int im = ch / CPI, oy0 = ch % CPI * G::RT;
        const float* xn = x + ((size_t)im * cin + ci0) * HI * HI;
        float* xd = xs + buf * G::XS;
        for (int e = tid; e < 32 * G::RI * G::CW; e += 128) {
            const int ci = e / (G::RI * G::CW), r = e / G::CW % G::RI, c = e % G::CW;
            const int iy = oy0 * S + r - 1, ix = c - 1;
            const bool in = iy >= 0 && iy < HI && ix >= 0 && ix < HI;
            cp4(xd + ci * G::CS + r * G::PW + (S == 2 ? ((c & 1) ? G::PO + (c >> 1) : (c >> 1)) : c),
                xn + (in ? ((size_t)ci * HI + iy) * HI + ix : 0), in);
        }
        const float* yn = dy + (((size_t)im * cout + co0) * HO + oy0) * HO;
        float* yd = ys + buf * G::YS;
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const int co = (tid + 128 * e) / 16, q = (tid + 128 * e) % 16;
            cp16(yd + co * 64 + 4 * q, yn + (size_t)co * HO * HO + 4 * q, true);
        }
        cp_commit();
    };
    uint64_t acc[8][9];
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
        for (int k = 0; k < 9; k++) acc[i][k] = 0ull;
    double sb = 0.0;
    const bool bias = blockIdx.y == 0;
    float* part = parts + ((size_t)blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x * kGradPart +
                  (size_t)blockIdx.x * kGradPart + tid;
    bool finite = true, first = true;
    if (c0 < c1) stage(c0, 0);
    for (int ch = c0; ch < c1; ch++) {
        const int buf = (ch - c0) & 1;
        if (ch + 1 < c1) {
            stage(ch + 1, buf ^ 1);
            cp_wait<1>();
        } else {
            cp_wait<0>();
        }
        __syncthreads();
        const float* xb = xs + buf * G::XS + lane * G::CS;
        const float* yb = ys + buf * G::YS + warp * 8 * 64;
        float sc = 0.f;
#pragma unroll 1
        for (int q = 0; q < 16; q++) {
            const int oy = q / (HO / 4), c4 = 4 * (q % (HO / 4));
            ulonglong2 g[8];
#pragma unroll
            for (int i = 0; i < 8; i++)
                g[i] = *reinterpret_cast<const ulonglong2*>(yb + i * 64 + 4 * q);
            if (bias) {
                const float4 t = *reinterpret_cast<const float4*>(yb + (lane & 7) * 64 + 4 * q);
                sc += (t.x + t.y) + (t.z + t.w);
            }
#pragma unroll
            for (int r = 0; r < 3; r++) {
                const float* xr = xb + (oy * S + r) * G::PW + c4;
                const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(xr);
                const float2 a0 = unpack2(a.x), a1 = unpack2(a.y);
                uint64_t t[3][2];                       // [tap column][pixel pair]
                t[0][0] = a.x;
                t[0][1] = a.y;
                if (S == 1) {
                    const uint64_t b = *reinterpret_cast<const uint64_t*>(xr + 4);
                    t[1][0] = pack2(a0.y, a1.x);
                    t[1][1] = pack2(a1.y, unpack2(b).x);
                    t[2][0] = a.y;
                    t[2][1] = b;
                } else {
                    const ulonglong2 e = *reinterpret_cast<const ulonglong2*>(xr + G::PO);
                    t[1][0] = e.x;
                    t[1][1] = e.y;
                    t[2][0] = pack2(a0.y, a1.x);
                    t[2][1] = pack2(a1.y, xr[4]);
                }
#pragma unroll
                for (int c = 0; c < 3; c++)
#pragma unroll
                    for (int i = 0; i < 8; i++) {
                        fma2(acc[i][3 * r + c], g[i].x, t[c][0]);
                        fma2(acc[i][3 * r + c], g[i].y, t[c][1]);
                    }
            }
        }
        __syncthreads();
        sb += sc;
        if ((ch + 1 - c0) % (kGradChain / 32) == 0 || ch + 1 == c1) {
            finite &= add_to_part(acc, part, first);
            first = false;
        }
    }
    if (bias && lane < 8) biasParts[(size_t)blockIdx.z * cout + co0 + warp * 8 + lane] = (float)sb;
    if (!__syncthreads_or(!finite)) return;
    for (int i = 0; i < 8; i++) {
        double sum[9] = {};
        for (int ch = c0; ch < c1; ch++) {
            const int im = ch / CPI, oy0 = ch % CPI * G::RT;
            const float* xc = x + ((size_t)im * cin + ci0 + lane) * HI * HI;
            const float* yc = dy + (((size_t)im * cout + co0 + warp * 8 + i) * HO + oy0) * HO;
            float a[9] = {};
            for (int p = 0; p < 64; p++) {
                const float g = yc[p];
                if (g == 0.f) continue;
                for (int k = 0; k < 9; k++) {
                    const int iy = (oy0 + p / HO) * S + k / 3 - 1, ix = p % HO * S + k % 3 - 1;
                    if (iy >= 0 && iy < HI && ix >= 0 && ix < HI) a[k] = fmaf(g, xc[iy * HI + ix], a[k]);
                }
            }
            for (int k = 0; k < 9; k++) sum[k] += a[k];
        }
        for (int k = 0; k < 9; k++) part[(i * 9 + k) * 128] = (float)sum[k];
    }
}

// The first layer's weight gradient (one input channel, 64 x 64): a lane per
// 4 neighbouring pixels, straight from global memory (each gradient is read
// once: bound by HBM).  Chains, parts and zeros as above; a part has a sum of
// every lane.
__global__ void __launch_bounds__(128, 2)
k_conv1_grad(const float* __restrict__ x, const float* __restrict__ dy, float* __restrict__ parts,
             float* __restrict__ biasParts, int n)
{
    constexpr int H = 64, GR = H * H / 4;                    // groups of 4 pixels an image
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint64_t acc[8][9];
    float sb[8];
    double sum[8] = {};
#pragma unroll
    for (int i = 0; i < 8; i++) {
        sb[i] = 0.f;
#pragma unroll
        for (int k = 0; k < 9; k++) acc[i][k] = 0ull;
    }
    float* part = parts + (size_t)blockIdx.x * kGradPart + threadIdx.x;
    const int total = n * GR, step = gridDim.x * 32;
    bool finite = true, first = true;
    int done = 0;
    for (int e = blockIdx.x * 32 + lane; e < total; e += step) {
        const int im = e / GR, oy = e % GR / (H / 4), c4 = 4 * (e % (H / 4));
        const float* yp = dy + ((size_t)im * 32 + warp * 8) * (H * H) + oy * H + c4;
        ulonglong2 g[8];
#pragma unroll
        for (int i = 0; i < 8; i++) {
            g[i] = __ldg(reinterpret_cast<const ulonglong2*>(yp + (size_t)i * H * H));
            const float2 a = unpack2(g[i].x), b = unpack2(g[i].y);
            sb[i] += (a.x + a.y) + (b.x + b.y);
        }
#pragma unroll
        for (int r = 0; r < 3; r++) {
            const int iy = oy + r - 1;
            if (iy < 0 || iy >= H) continue;
            const float* xr = x + (size_t)im * H * H + iy * H + c4;
            const float4 m = __ldg(reinterpret_cast<const float4*>(xr));
            const float l = c4 > 0 ? __ldg(xr - 1) : 0.f, h = c4 + 4 < H ? __ldg(xr + 4) : 0.f;
            const uint64_t t[3][2] = {{pack2(l, m.x), pack2(m.y, m.z)},
                                      {pack2(m.x, m.y), pack2(m.z, m.w)},
                                      {pack2(m.y, m.z), pack2(m.w, h)}};
#pragma unroll
            for (int c = 0; c < 3; c++)
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    fma2(acc[i][3 * r + c], g[i].x, t[c][0]);
                    fma2(acc[i][3 * r + c], g[i].y, t[c][1]);
                }
        }
        if (++done % (kGradChain / 2) == 0 || e + step >= total) {
            finite &= add_to_part(acc, part, first);
            first = false;
#pragma unroll
            for (int i = 0; i < 8; i++) {
                sum[i] += sb[i];
                sb[i] = 0.f;
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 8; i++) {
        for (int o = 16; o; o >>= 1) sum[i] += __shfl_xor_sync(0xffffffffu, sum[i], o);
        if (lane == 0) biasParts[(size_t)blockIdx.x * 32 + warp * 8 + i] = (float)sum[i];
    }
    if (!__syncthreads_or(!finite)) return;
    for (int i = 0; i < 8; i++) {
        double s[9] = {};
        for (int e = blockIdx.x * 32 + lane; e < total; e += step) {
            const int im = e / GR, oy = e % GR / (H / 4), c4 = 4 * (e % (H / 4));
            const float* yp = dy + ((size_t)im * 32 + warp * 8 + i) * (H * H) + oy * H + c4;
            for (int p = 0; p < 4; p++) {
                const float g = yp[p];
                if (g == 0.f) continue;
                for (int k = 0; k < 9; k++) {
                    const int iy = oy + k / 3 - 1, ix = c4 + p + k % 3 - 1;
                    if (iy >= 0 && iy < H && ix >= 0 && ix < H)
                        s[k] += (double)g * x[(size_t)im * H * H + iy * H + ix];
                }
            }
        }
        for (int k = 0; k < 9; k++) part[(i * 9 + k) * 128] = (float)s[k];
    }
}

// dW += the sum of Z CTAs' parts [z][blocks][kGradPart] and db += that of
// biasParts [z][cout], always in the same order.  A thread sums its share in a
// pair of FP32, the sum and what its roundings lost (Knuth's two-sum, 48 bits
// together), and the shares meet in FP64.  The twelve launches of a batch of 256
// take 97 us (177 with FP64 additions, two lanes a clock).  CTA: 32 sums, 8
// shares of the parts; the last cout / 32 CTAs have the biases.  With lanes
// (the first layer) the 32 sums are the lanes' of one weight.
__global__ void __launch_bounds__(256)
k_grad_sum(const float* __restrict__ parts, const float* __restrict__ biasParts, int Z, int cin,
           int cout, int lanes, float* __restrict__ dW, float* __restrict__ db)
{
    __shared__ double red[8][32];
    const int t = threadIdx.x & 31, share = threadIdx.x >> 5;
    const int xb = cout / 32, blocks = lanes ? 1 : xb * (cin / 32), nW = blocks * (kGradPart / 32);
    const bool bias = (int)blockIdx.x >= nW;
    const int e = ((int)blockIdx.x - (bias ? nW : 0)) * 32 + t;
    const size_t pitch = bias ? (size_t)cout : (size_t)blocks * kGradPart;
    const float* src = (bias ? biasParts : parts) + e;
    float sum = 0.f, lost = 0.f;
#pragma unroll 8
    for (int z = share; z < Z; z += 8) {
        const float v = __ldg(src + z * pitch), u = sum + v, w = u - sum;
        lost += (sum - (u - w)) + (v - w);
        sum = u;
    }
    double s = fabsf(sum) < INFINITY ? (double)sum + lost : (double)sum;
    red[share][t] = s;
    __syncthreads();
    if (share) return;
    for (int i = 1; i < 8; i++) s += red[i][t];
    if (bias) {
        db[e] += (float)s;
        return;
    }
    const int b = e / kGradPart, j = e % kGradPart;
    const int ik = j / 128, co = b % xb * 32 + j % 128 / 32 * 8 + ik / 9, ci = b / xb * 32 + t;
    if (!lanes) {
        dW[((size_t)co * cin + ci) * 9 + ik % 9] += (float)s;
        return;
    }
    for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (t == 0) dW[co * 9 + ik % 9] += (float)s;
}

// ------------------------------------------------------------ weight layout --
// One layer's weights W [co][ci][3][3] as the kernels above read them, rounded
// to bf16 when `round`: fwd [(ci, tap)][co]; bwd, for stride 1 [(co, flipped
// tap)][ci], for stride 2 the four classes (py, px) = (1, 1), (1, 0), (0, 1),
// (0, 0), each [(co, its taps)][ci].
__global__ void k_repack_conv(const float* __restrict__ W, int cin, int cout, int stride, int round,
                              float* __restrict__ fwd, float* __restrict__ bwd)
{
    const int total = cin * cout * 9;
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < total; e += gridDim.x * blockDim.x) {
        const int k = e % 9, ci = e / 9 % cin, co = e / (9 * cin);
        const int ky = k / 3, kx = k % 3;
        const float w = round ? __bfloat162float(__float2bfloat16_rn(W[e])) : W[e];
        if (fwd) fwd[(size_t)(ci * 9 + k) * cout + co] = w;
        if (!bwd) continue;
        if (stride == 1) {
            bwd[(size_t)(co * 9 + 8 - k) * cin + ci] = w;
        } else {
            // tap 1 serves even input rows (one tap), taps 2 and 0 odd ones (two, in that order)
            const int py = ky != 1, px = kx != 1;
            const int nx = 1 + px, nk = (1 + py) * nx;
            const int r = ky == 0, c = kx == 0;
            const int before = py ? (px ? 0 : 4) : (px ? 6 : 8);
            bwd[(size_t)before * cin * cout + (size_t)(co * nk + r * nx + c) * cin + ci] = w;
        }
    }
}

template <typename K>
cudaError_t set_smem(K kern, size_t bytes)
{
    return bytes > 48 * 1024 ? cudaFuncSetAttribute(
                                   kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes)
                             : cudaSuccess;
}

template <int S, int HO, int CI, int NW>
cudaError_t run_conv(const ConvArgs& a, cudaStream_t st)
{
    using Sh = ConvShape<3, 3, S, HO>;
    constexpr size_t smem = conv_smem<3, 3, S, HO, CI, NW>();
    cudaError_t e = set_smem(k_conv<S, HO, CI, NW>, smem);
    if (e != cudaSuccess) return e;
    const int tiles = Sh::IT > 1 ? (a.n + Sh::IT - 1) / Sh::IT : a.n * (HO / Sh::RT);
    k_conv<S, HO, CI, NW><<<dim3(tiles, a.cout / (8 * NW)), 32 * NW, smem, st>>>(a);
    return cudaGetLastError();
}

// 32 output channels a CTA; 16 where that leaves SMs without a CTA (a batch of
// 256 at 8 x 8 is 256 tiles of 32 channels on 152 SMs)
template <int S, int HO, int CI>
cudaError_t run_conv(const ConvArgs& a, cudaStream_t st)
{
    using Sh = ConvShape<3, 3, S, HO>;
    const int tiles = Sh::IT > 1 ? (a.n + Sh::IT - 1) / Sh::IT : a.n * (HO / Sh::RT);
    return (long long)tiles * (a.cout / 32) < 4 * 152 ? run_conv<S, HO, CI, 2>(a, st)
                                                      : run_conv<S, HO, CI, 4>(a, st);
}

template <int HO>
cudaError_t run_classes(const ConvArgs& a, cudaStream_t st)
{
    using Sh = ConvShape<2, 2, 1, HO>;
    constexpr size_t smem = std::max(
        std::max(conv_smem<2, 2, 1, HO, 8, 4>(), conv_smem<2, 1, 1, HO, 8, 4>()),
        std::max(conv_smem<1, 2, 1, HO, 8, 4>(), conv_smem<1, 1, 1, HO, 8, 4>()));
    cudaError_t e = set_smem(k_conv_classes<HO, 4>, smem);
    if (e != cudaSuccess) return e;
    const int tiles = Sh::IT > 1 ? (a.n + Sh::IT - 1) / Sh::IT : a.n * (HO / Sh::RT);
    k_conv_classes<HO, 4><<<dim3(tiles, a.cout / 32, 4), 128, smem, st>>>(a);
    return cudaGetLastError();
}

cudaError_t sum_grad(const float* parts, const float* biasParts, int Z, int cin, int cout, int lanes,
                     float* dW, float* db, cudaStream_t st)
{
    const int sums = (lanes ? 1 : (cout / 32) * (cin / 32)) * kGradPart + cout;
    k_grad_sum<<<sums / 32, 256, 0, st>>>(parts, biasParts, Z, cin, cout, lanes, dW, db);
    return cudaGetLastError();
}

template <int S, int HO>
cudaError_t run_grad(const float* x, const float* dy, float* dW, float* db, int n, int cin,
                     int cout, float* parts, cudaStream_t st)
{
    using G = GradShape<S, HO>;
    cudaError_t e = set_smem(k_conv_grad<S, HO>, G::bytes);
    if (e != cudaSuccess) return e;
    // two CTAs an SM share the chunks
    const int blocks = (cout / 32) * (cin / 32), chunks = n * (HO / G::RT);
    const int split = std::max(1, std::min(chunks, (2 * 152 + blocks - 1) / blocks));
    if (split * blocks > kGradCtas) return cudaErrorInvalidValue;
    float* biasParts = parts + (size_t)kGradCtas * kGradPart;
    k_conv_grad<S, HO><<<dim3(cout / 32, cin / 32, split), 128, G::bytes, st>>>(x, dy, parts, biasParts,
                                                                             n, cin, cout);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    return sum_grad(parts, biasParts, split, cin, cout, 0, dW, db, st);
}

}  // namespace

cudaError_t launch_repack_conv(const float* W, int cin, int cout, int stride, int round, float* fwd,
                               float* bwd, cudaStream_t st)
{
    const int total = cin * cout * 9;
    k_repack_conv<<<std::min((total + 255) / 256, 152 * 8), 256, 0, st>>>(W, cin, cout, stride,
                                                                          round, fwd, bwd);
    return cudaGetLastError();
}

// The network's six convolutions by layer: inputs [n][cin][hin][hin].
cudaError_t launch_conv_fwd(int layer, const float* x, const float* wt, const float* bias, float* y,
                            int n, int cin, int cout, cudaStream_t st)
{
    const ConvArgs a = {x, wt, bias, nullptr, y, n, cin, cout};
    switch (layer) {
    case 0: return run_conv<1, 64, 1, 4>(a, st);
    case 1: return run_conv<2, 32, 4>(a, st);
    case 2: return run_conv<1, 32, 8>(a, st);
    case 3: return run_conv<2, 16, 4>(a, st);
    case 4: return run_conv<1, 16, 8>(a, st);
    case 5: return run_conv<2, 8, 4>(a, st);
    default: return cudaErrorInvalidValue;
    }
}

// dx [n][cin][hin][hin] from dy [n][cout][hout][hout], zeroed where act (the
// layer's input, a ReLU output) is not positive.
cudaError_t launch_conv_bwd_data(int layer, const float* dy, const float* wt, const float* act,
                                 float* dx, int n, int cin, int cout, cudaStream_t st)
{
    const ConvArgs a = {dy, wt, nullptr, act, dx, n, cout, cin};
    switch (layer) {
    case 1: return run_classes<32>(a, st);
    case 2: return run_conv<1, 32, 8>(a, st);
    case 3: return run_classes<16>(a, st);
    case 4: return run_conv<1, 16, 8>(a, st);
    case 5: return run_classes<8>(a, st);
    default: return cudaErrorInvalidValue;
    }
}

// the CTAs' parts of a layer's weights, then of its biases
size_t conv_grad_part_floats() { return (size_t)kGradCtas * (kGradPart + 32); }

cudaError_t launch_conv_bwd_weight(int layer, const float* x, const float* dy, float* dW, float* db,
                                   int n, int cin, int cout, float* parts, cudaStream_t st)
{
    switch (layer) {
    case 0: {
        const int ctas = std::min(n * 32, 152 * 2);
        float* biasParts = parts + (size_t)kGradCtas * kGradPart;
        k_conv1_grad<<<ctas, 128, 0, st>>>(x, dy, parts, biasParts, n);
        const cudaError_t e = cudaGetLastError();
        return e != cudaSuccess ? e : sum_grad(parts, biasParts, ctas, 1, 32, 1, dW, db, st);
    }
    case 1: return run_grad<2, 32>(x, dy, dW, db, n, cin, cout, parts, st);
    case 2: return run_grad<1, 32>(x, dy, dW, db, n, cin, cout, parts, st);
    case 3: return run_grad<2, 16>(x, dy, dW, db, n, cin, cout, parts, st);
    case 4: return run_grad<1, 16>(x, dy, dW, db, n, cin, cout, parts, st);
    case 5: return run_grad<2, 8>(x, dy, dW, db, n, cin, cout, parts, st);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace tg3
