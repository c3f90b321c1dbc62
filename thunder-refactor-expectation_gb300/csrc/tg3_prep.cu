// Image preprocessing ahead of the expectation: real-space particle images
// to the complex pixel data the scoring kernels read (Optimiser::initImg,
// src/Optimiser.cpp:4600-4760, and allocPreCal, src/Optimiser.cpp:7995-8030).
// With r = maskRadius / pixelSize and centred coordinates (i, j), i, j in
// [-N/2, N/2) about the file's pixel (N/2, N/2):
//   substractBgImg (:4917): the mean m and standard deviation s (n - 1) of
//     the pixels with i^2 + j^2 > r^2 (bgMeanStddev, src/Image/
//     ImageFunctions.cpp:607-620); y = (x - m) / s;
//   statImg (:4796): stdN = the mean over the images of the same region's
//     standard deviation of y about 0 (bgStddev, ImageFunctions.cpp:585-596);
//   maskImg (:4953, zeroMask): y (u < r), y (1 - w) for r <= u <= r + 6 with
//     w = 0.5 - 0.5 cos((u - r) / 6 pi), 0 beyond (softMask, src/Functions/
//     Mask.cpp:363-385; EDGE_WIDTH_RL = 6); u = sqrt(i^2 + j^2);
//   normaliseImg (:4987): y / stdN;
//   fwImg (:5003): unnormalised forward r2c transform of the image with its
//     centre at index 0 (ImageFile's MESH_IMAGE_INDEX layout);
//   allocPreCal: dat[l][p] = FT at (iCol[p], iRow[p] mod N).
// The unmasked form (the reference's _imgOri) skips the mask.  The noise-
// filled mask of the non-zeroMask option draws from the reference's GSL
// random stream and is not offered.
#include <cufft.h>

#include <algorithm>
#include <mutex>
#include <vector>

#include "tg3_fft.cuh"
#include "tg3_internal.cuh"

namespace tg3 {
namespace {

__device__ double prep_block_sum(double v, double* scratch)
{
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    __syncthreads();
    if (lane == 0) scratch[wid] = v;
    __syncthreads();
    if (wid == 0) {
        double r = lane < nw ? scratch[lane] : 0.0;
        for (int o = 16; o; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
        if (lane == 0) scratch[0] = r;
    }
    __syncthreads();
    return scratch[0];
}

// The soft mask as a function of the integer squared radius q = i^2 + j^2: 1 for
// q <= qIn, tab[q - qIn] up to qOut, 0 beyond.
struct SoftMask {
    const float* tab;        // [qOut - qIn + 1], tab[0] = 1
    int qIn, qOut;
};

// (x - m) f as (x - high part of m) f - (low part of m) f: the mean rounded to
// FP32 would shift every pixel alike, which the lowest frequencies add up.
struct Scaling {
    float m, f, c;
};

__device__ __forceinline__ float scaled(const Scaling& a, float x) { return fmaf(x - a.m, a.f, a.c); }

__device__ __forceinline__ float masked(float v, int q, const SoftMask& k, const float* tab)
{
    const float w = tab[min(max(q - k.qIn, 0), k.qOut - k.qIn)];
    return q > k.qOut ? 0.f : v * w;
}

// Tables of a call, spread over the CTAs of k_bg_stats: the soft mask's edge, w =
// 1 - (0.5 - 0.5 cos((u - r) / ew pi)); the transform's twiddles w_N^(r j)
// [A][B]; and where the pixels lie in the transform's columns.
struct PrepTables {
    float* mask;
    int qIn, nMask;          // entries
    float r, ew;
    float2* tw;
    int A, B;                // 0: no twiddles, no slots
    int* slot;               // [K] (CTA of the image << 20) + place
    const int *iCol, *iRow;
    int K, cols, maxCol, W;
};

// a total and the part its roundings lost (Knuth's two-sum)
struct Total {
    float s, lost;
    __device__ __forceinline__ void add(float v)
    {
        const float t = s + v, b = t - s;
        lost += (s - (t - b)) + (v - b);
        s = t;
    }
    __device__ __forceinline__ void add_square(float v) { add(v * v); }
    __device__ __forceinline__ double value() const { return (double)s + lost; }
    __device__ __forceinline__ void warp_sum()
    {
        for (int o = 16; o; o >>= 1) {
            const float v = __shfl_xor_sync(0xffffffffu, s, o);
            lost += __shfl_xor_sync(0xffffffffu, lost, o);
            add(v);
        }
    }
};

// a total in FP64, for sums that leave FP32
struct WideTotal {
    double s, none;
    __device__ __forceinline__ void add(float v) { s += v; }
    __device__ __forceinline__ void add_square(float v) { s += (double)v * v; }
    __device__ __forceinline__ double value() const { return s; }
    __device__ __forceinline__ void warp_sum()
    {
        for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    }
};

// The sums of d and d^2 over an image's background pixels only, d = x minus the
// corner pixel (always background); i^2 + j^2 > bgAbove = floor(r^2) in
// integers.  A warp takes four rows at a time, lanes over what lies left and
// right of the circle, eight loads in flight.  A lane sums kTogether pixels in
// pairs in FP32 and adds that to its totals (T): a pair of FP32 (the sum and what
// its roundings lost, 48 bits together), which become FP64 at the end: FP64 sums
// on the way, two lanes a clock, took most of the time.  Lanes past a row's end
// read the pivot, which adds nothing.  CTA: one image; rows in bands of the
// table `rows`, (left, right) of the circle.
//
// kTogether is 8 from 256 pixels a side and 2 below, where an image has fewer
// sums for their roundings to cancel over: the deviation of a 64 pixel image is
// then off by 7.1e-9 (FP32 sums of a row in FP64: 7.0e-9, 8 pixels 8.3e-9), of a
// 256 pixel one by 4.7e-9 (4.9e-9), root mean squares over images of noise.
constexpr int kBgBand = 5888;        // 46 KB of rows; a multiple of a CTA's 32

template <int kTogether, class T>
__device__ __forceinline__ void bg_sums(const float* im, int N, int bgAbove, int2* rows,
                                        double (&sums)[2])
{
    __shared__ T part[2][8];
    const int half = N / 2;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const float pivot = im[0];
    T t1{}, t2{};
    for (int band = 0; band < N; band += kBgBand) {
        const int end = min((N + 3) / 4 * 4, band + kBgBand);
        __syncthreads();
        for (int y = band + threadIdx.x; y < end; y += blockDim.x) {
            const int j = y - half, q = bgAbove - j * j;
            int h = -1;                              // the row inside: |i| <= h
            if (q >= 0) {
                h = (int)sqrtf((float)q);
                while (h * h > q) h--;
                while ((h + 1) * (h + 1) <= q) h++;
            }
            rows[y - band] = y >= N   ? make_int2(0, 0)
                             : h < 0 ? make_int2(N, 0)
                                     : make_int2(max(half - h, 0), max(half - h - 1, 0));
        }
        __syncthreads();
        for (int y0 = band + 4 * warp; y0 < end; y0 += 4 * nw) {
            int left[4], n[4], most = 0;
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const int2 r = rows[y0 - band + k];
                left[k] = r.x;
                n[k] = r.x + r.y;
                most = max(most, n[k]);
            }
            for (int e = lane; e < most; e += 64) {
                float d[8];
#pragma unroll
                for (int k = 0; k < 8; k++) {
                    const int f = e + 32 * (k & 1), r = k >> 1;
                    const int x = (y0 + r) * N + (f < left[r] ? f : N - n[r] + f);
                    d[k] = __ldg(im + (f < n[r] ? x : 0));
                }
#pragma unroll
                for (int k = 0; k < 8; k++) d[k] -= pivot;
                if constexpr (kTogether == 1) {
#pragma unroll
                    for (int k = 0; k < 8; k++) {
                        t1.add(d[k]);
                        t2.add_square(d[k]);
                    }
                } else {
                    float a[4], b[4];
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        a[k] = d[2 * k] + d[2 * k + 1];
                        b[k] = fmaf(d[2 * k], d[2 * k], d[2 * k + 1] * d[2 * k + 1]);
                    }
                    if constexpr (kTogether == 2) {
#pragma unroll
                        for (int k = 0; k < 4; k++) {
                            t1.add(a[k]);
                            t2.add(b[k]);
                        }
                    } else {
                        t1.add((a[0] + a[1]) + (a[2] + a[3]));
                        t2.add((b[0] + b[1]) + (b[2] + b[3]));
                    }
                }
            }
        }
    }
    t1.warp_sum();
    t2.warp_sum();
    if (lane == 0) {
        part[0][warp] = t1;
        part[1][warp] = t2;
    }
    __syncthreads();
    if (threadIdx.x < 2) {
        double s = 0.0;
        for (int w = 0; w < nw; w++) s += part[threadIdx.x][w].value();
        sums[threadIdx.x] = s;
    }
    __syncthreads();
}

// apart, so that it takes no registers from the usual sums
__device__ __noinline__ void bg_sums_wide(const float* im, int N, int bgAbove, int2* rows,
                                          double (&sums)[2])
{
    bg_sums<1, WideTotal>(im, N, bgAbove, rows, sums);
}

// Per-image background statistics: st[l] = (m, s, sN, 1 / s), sN the background
// standard deviation of (x - m) / s about 0.  Sums that leave FP32 (pixels
// beyond about 1e17 at 256 a side) are taken again in FP64.  CTA per image; 1,024
// images of 256^2: 50 us (a load at a time and FP64 sums: 124).
template <int kTogether>
__global__ void __launch_bounds__(256)
k_bg_stats(const float* __restrict__ img, int N, int bgAbove, double cnt, double* __restrict__ st,
           float* __restrict__ st32, const PrepTables t)
{
    extern __shared__ int2 rows[];               // [N rounded up to 4, kBgBand at most]
    __shared__ double sums[2];
    const size_t l = blockIdx.x;
    if (threadIdx.x < 32)
        for (int e = blockIdx.x * 32 + threadIdx.x; e < t.A * t.B; e += gridDim.x * 32) {
            double s, c;
            sincospi(-2.0 * (e / t.B * (e % t.B)) / (t.A * t.B), &s, &c);
            t.tw[e] = make_float2((float)c, (float)s);
        }
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < max(t.nMask, t.K);
         i += gridDim.x * blockDim.x) {
        if (i < t.nMask) {
            const float u = sqrtf((float)(t.qIn + i));
            t.mask[i] = i ? 1.f - (0.5f - 0.5f * cospif((u - t.r) / t.ew)) : 1.f;
        }
        if (t.A && i < t.K) {
            const int k = t.iCol[i], b = k / t.cols, c0 = b * t.cols;
            const int nc = min(t.cols, t.maxCol + 1 - c0);
            const int r = t.iRow[i], y = r < 0 ? r + N : r;
            t.slot[i] = (b << 20) + (y < N / 2 ? y * t.W : (y - N / 2) * t.W + nc) + k - c0;
        }
    }
    const float* im = img + l * N * N;
    bg_sums<kTogether, Total>(im, N, bgAbove, rows, sums);
    if (!(fabs(sums[0]) < INFINITY && fabs(sums[1]) < INFINITY))
        bg_sums_wide(im, N, bgAbove, rows, sums);
    if (threadIdx.x == 0) {
        const float pivot = im[0];
        const double s1 = sums[0], s2 = sums[1];
        const double mu = s1 / cnt;                 // mean about the pivot
        const double ss = fmax(s2 - s1 * mu, 0.0);  // sum of (x - m)^2
        const double sd = sqrt(ss / (cnt - 1.0));
        // sum of ((x - m) / sd)^2 over the background, over (n - 1)
        const double o[4] = {pivot + mu, sd, sqrt(ss / (sd * sd) / (cnt - 1.0)), 1.0 / sd};
        for (int i = 0; i < 4; i++) {
            st[4 * l + i] = o[i];
            if (st32 && i < 3) st32[3 * l + i] = (float)o[i];
        }
    }
}

// stdN: the given value, or the mean of the images' sN; then every image's
// scaling by 1 / (s stdN).  One CTA.
__global__ void __launch_bounds__(256)
k_stdn(const double* __restrict__ st, int n, float given, Scaling* __restrict__ out)
{
    __shared__ double red[32];
    double s = 0.0;
    for (int l = threadIdx.x; l < n; l += blockDim.x) s += st[4 * (size_t)l + 2];
    s = prep_block_sum(s, red);
    const double scale = 1.0 / (given > 0.f ? (double)given : s / n);
    for (int l = threadIdx.x; l < n; l += blockDim.x) {
        const double mean = st[4 * (size_t)l], f = scale * st[4 * (size_t)l + 3];
        const float m = (float)mean;
        out[l] = {m, (float)f, (float)((m - mean) * f)};
    }
}

constexpr int kPrepRows = 4;   // image rows per CTA of k_prep_image

// Normalise, mask and scale rows of an image, written with the image's centre
// at index 0, for the library's transform.  CTA (kPrepRows rows, image l);
// threads over the columns, a thread's rows loaded together; pixels outside
// the mask are not read.
__global__ void k_prep_image(const float* __restrict__ img, int N, const SoftMask mask,
                             const Scaling* __restrict__ scaling, float* __restrict__ out)
{
    const size_t l = blockIdx.y;
    const Scaling sc = scaling[l];
    const int half = N / 2, y0 = blockIdx.x * kPrepRows;
    const float* im = img + l * N * N;
    for (int x = threadIdx.x; x < N; x += blockDim.x) {
        const int i = x - half;
        float v[kPrepRows];
        int q[kPrepRows];
#pragma unroll
        for (int k = 0; k < kPrepRows; k++) {
            const int j = min(y0 + k, N - 1) - half;
            q[k] = i * i + j * j;
            v[k] = __ldg(im + (q[k] <= mask.qOut ? (size_t)(j + half) * N + x : 0));
        }
#pragma unroll
        for (int k = 0; k < kPrepRows; k++) {
            const int j = y0 + k - half;
            const int ci = i < 0 ? i + N : i, cj = j < 0 ? j + N : j;
            if (y0 + k < N)
                out[l * N * N + (size_t)cj * N + ci] = masked(scaled(sc, v[k]), q[k], mask, mask.tab);
        }
    }
}

// Normalisation, mask, 2-D transform and pixel gather of one image by one CTA,
// the transform on chip (tg3_fft.cuh has its two-step form; N = A B, A even).
// A warp holds one line, or two of up to 16 lanes, and needs no other warp:
//   rows: the rows y and y + N/2 of the centred image are the real and the
//     imaginary part of one line; of its transform Z the columns k and N - k of
//     this CTA's range c0 <= k < c0 + cols stay in shared memory;
//   columns: a lane's inputs of column k at y and y + N/2 are (Z[k] +
//     conj Z[N - k]) / 2 and (Z[k] - conj Z[N - k]) / 2i of that line, so the
//     two rows part on the way in; the result takes the column's place;
//   then the pixels are read out in the list's order.
// Images whose columns do not fit take several CTAs, each with a range of the
// columns and all rows; they meet in L2.  Bound by instruction issue at one CTA an
// SM (115,000 warp instructions an image of 256^2 at 0.46 a cycle and
// scheduler); the image is read once, inside the mask, and only the list's
// pixels are written.  1,024 images of 256^2, 9,930 pixels: 200 us, where the
// normalised images, the library's two transform kernels and the gather took
// 495.
struct PrepFt {
    const float* img;
    int A, B, lanes;         // lanes of a line: 16 or 32
    int ex;                  // exchange buffer of a line
    int cols, maxCol, W;     // columns of a CTA, the last one of the list, row pitch
    SoftMask mask;
    const float2* tw;
    const Scaling* scaling;
    const int* slot;         // (CTA of the image << 20) + place of a pixel
    int K;
    float2* dat;
};

#define TG3_RADIX_A(X) X(6) X(8) X(10) X(12) X(14) X(16) X(18) X(20)
#define TG3_RADIX_B(X) \
    X(4) X(5) X(6) X(7) X(8) X(9) X(10) X(11) X(12) X(13) X(14) X(15) X(16) X(18) X(20)

template <int R>
struct Radix {
    static constexpr int value = R;
};

template <class F>
__device__ __forceinline__ void with_a(int r, F f)
{
    switch (r) {
#define X(n) case n: f(Radix<n>()); break;
        TG3_RADIX_A(X)
#undef X
    }
}
template <class F>
__device__ __forceinline__ void with_b(int r, F f)
{
    switch (r) {
#define X(n) case n: f(Radix<n>()); break;
        TG3_RADIX_B(X)
#undef X
    }
}

using fft::c64;

// first step's output of item t to the line's exchange buffer
template <int R>
__device__ __forceinline__ void prep_exchange(c64 (&v)[R], c64* xb, const float2* tw, int B, int t)
{
    fft::dft<R>(v);
#pragma unroll
    for (int r = 0; r < R; r++) {
        const float2 w = tw[r * B + t];
        xb[r * (B | 1) + t] = r ? fft::times(v[r], w.x, w.y) : v[r];
    }
}

// x, as a value of this iteration: what hangs on it is worked out again instead
// of being kept in registers over the loop, where it does not fit
__device__ __forceinline__ int again(int x)
{
    asm volatile("" : "+r"(x));
    return x;
}

// the two rows' pixels of item t of line y
struct PrepRows {
    float a[20], b[20];
};

template <int R>
__device__ __forceinline__ void prep_load(const PrepFt& p, size_t l, int N, int y, int t, PrepRows& v)
{
    const int half = N / 2, B = p.B;
    // rows of the coordinates y and y - N/2, from column 0
    const float* r0 = p.img + (l * N + y + half) * N + half;
    const float* r1 = p.img + (l * N + y) * N + half;
    const int q0 = y * y, q1 = (half - y) * (half - y);
#pragma unroll
    for (int r = 0; r < R; r++) {
        const int i = t + (r < R / 2 ? r : r - R) * B;
        v.a[r] = __ldg(r0 + (i * i + q0 <= p.mask.qOut ? i : 0));
        v.b[r] = __ldg(r1 + (i * i + q1 <= p.mask.qOut ? i : 0));
    }
}

__global__ void __launch_bounds__(512, 1) k_prep_ft(const PrepFt p)
{
    extern __shared__ __align__(16) c64 psm[];
    const int A = p.A, B = p.B, N = A * B, half = N / 2, W = p.W;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int per = 32 / p.lanes, sub = lane / p.lanes;
    c64* big = psm;
    c64* xb = big + half * W + (warp * per + sub) * p.ex;
    float2* tw = reinterpret_cast<float2*>(big + half * W + nw * per * p.ex);
    float* tab = reinterpret_cast<float*>(tw + N);
    const size_t l = blockIdx.y;
    // the first rows' pixels are on their way while the tables are copied, the
    // next ones' behind each line's second step
    PrepRows px;
    with_a(A, [&](auto radix) {
        constexpr int R = decltype(radix)::value;
        const int t = lane % p.lanes;
        if (t < B) prep_load<R>(p, l, N, min(warp * per + sub, half - 1), t, px);
    });
    for (int i = threadIdx.x; i < N; i += blockDim.x) tw[i] = p.tw[i];
    for (int i = threadIdx.x; i <= p.mask.qOut - p.mask.qIn; i += blockDim.x) tab[i] = p.mask.tab[i];
    const int c0 = blockIdx.x * p.cols, nc = min(p.cols, p.maxCol + 1 - c0);
    Scaling sc = p.scaling[l];
    sc.f *= 0.5f;                                // for the columns' halves
    sc.c *= 0.5f;
    __syncthreads();

    for (int base = warp * per; base < half; base += nw * per) {
        const int y = base + sub, t = again(lane % p.lanes);
        const int yl = min(y, half - 1), next = min(y + nw * per, half - 1);
        const int q0 = yl * yl, q1 = (half - yl) * (half - yl);
        with_a(A, [&](auto radix) {
            constexpr int R = decltype(radix)::value;
            if (t >= B) return;
            c64 v[R];
#pragma unroll
            for (int r = 0; r < R; r++) {
                const int i = t + (r < R / 2 ? r : r - R) * B;
                v[r] = fft::pack(masked(scaled(sc, px.a[r]), i * i + q0, p.mask, tab),
                                 masked(scaled(sc, px.b[r]), i * i + q1, p.mask, tab));
            }
            prep_exchange<R>(v, xb, tw, B, t);
            prep_load<R>(p, l, N, next, t, px);
        });
        __syncwarp();
        with_b(B, [&](auto radix) {
            constexpr int R = decltype(radix)::value;
            if (t >= A || y >= half) return;
            c64 o[R];
#pragma unroll
            for (int s = 0; s < R; s++) o[s] = xb[t * (R | 1) + s];
            fft::dft<R>(o);
            c64* row = big + y * W;
#pragma unroll
            for (int s = 0; s < R; s++) {
                const int k = t + A * s, d = k - c0, e = (k ? N - k : 0) - c0;
                if (d >= 0 && d < nc) row[d] = o[s];
                if (e >= 0 && e < nc) row[nc + e] = o[s];
            }
        });
        __syncwarp();
    }
    __syncthreads();
    for (int base = warp * per; base < nc; base += nw * per) {
        const int k = base + sub, kl = min(k, nc - 1), t = again(lane % p.lanes);
        with_a(A, [&](auto radix) {
            constexpr int R = decltype(radix)::value;
            if (t >= B) return;
            c64 v[R];
#pragma unroll
            for (int r = 0; r < R / 2; r++) {
                const c64* row = big + (t + r * B) * W + kl;
                const float2 a = fft::unpack(row[0]), b = fft::unpack(row[nc]);
                v[r] = fft::pack(a.x + b.x, a.y - b.y);            // the 1/2 is in the scaling
                v[r + R / 2] = fft::pack(a.y + b.y, b.x - a.x);
            }
            prep_exchange<R>(v, xb, tw, B, t);
        });
        __syncwarp();
        with_b(B, [&](auto radix) {
            constexpr int R = decltype(radix)::value;
            if (t >= A || k >= nc) return;
            c64 o[R];
#pragma unroll
            for (int s = 0; s < R; s++) o[s] = xb[t * (R | 1) + s];
            fft::dft<R>(o);
#pragma unroll
            for (int s = 0; s < R; s++) {
                const int y = t + A * s;
                big[y < half ? y * W + k : (y - half) * W + nc + k] = o[s];
            }
        });
        __syncwarp();
    }
    __syncthreads();
    float2* dat = p.dat + l * p.K;
    constexpr int G = 8;
    for (int i0 = threadIdx.x; i0 < p.K; i0 += G * blockDim.x) {
        int at[G];
#pragma unroll
        for (int g = 0; g < G; g++) at[g] = __ldg(p.slot + min(i0 + g * (int)blockDim.x, p.K - 1));
#pragma unroll
        for (int g = 0; g < G; g++) {
            const int i = i0 + g * blockDim.x;
            if (i < p.K && at[g] >> 20 == (int)blockIdx.x)
                dat[i] = fft::unpack(big[at[g] & 0xfffff]);
        }
    }
}

// The factors of N (A even, both in the kernel's lists, the nearest to each
// other), and the launch that takes the fewest CTAs an image (each repeats the
// rows: 1,000 images of 256^2 take 200 us with one and, for 102 columns, 314
// with two, the separate kernels 500), then the most warps an SM.  0 where N has
// no such factors (254: the library's transform by 127 stays) or four CTAs
// cannot hold the columns.
struct PrepLaunch {
    int A = 0, B = 0, lanes = 0, ex = 0, cols = 0, W = 0, blocks = 0, threads = 0;
    size_t smem = 0;
};

PrepLaunch prep_launch(int N, int maxCol, int nMask)
{
    PrepLaunch o;
    const int as[] = {
#define X(n) n,
        TG3_RADIX_A(X)};
    const int bs[] = {TG3_RADIX_B(X)};
#undef X
    for (int a : as)
        for (int b : bs)
            if (a * b == N && (!o.A || std::abs(a - b) < std::abs(o.A - o.B))) o.A = a, o.B = b;
    if (!o.A) return o;
    o.lanes = std::max(o.A, o.B) <= 16 ? 16 : 32;
    o.ex = o.A * (o.B | 1);
    for (o.blocks = 1; o.blocks <= 4; o.blocks++) {
        o.cols = (maxCol + o.blocks) / o.blocks;
        o.W = 2 * o.cols | 1;                      // odd: a column's rows spread over the banks
        auto bytes = [&](int warps) {
            return sizeof(c64) * ((size_t)N / 2 * o.W + (size_t)warps * (32 / o.lanes) * o.ex + N) +
                   sizeof(float) * nMask;
        };
        int warps = 2 * (bytes(8) + 1024) <= kSmemSm ? 8 : 16;
        while (warps >= 8 && bytes(warps) > kSmemCta) warps -= 4;
        if (warps >= 8) {
            o.threads = 32 * warps;
            o.smem = bytes(warps);
            return o;
        }
    }
    return PrepLaunch();
}

// dat[l][p] = FT[l][iRow mod N][iCol]
__global__ void k_gather_pixels(const float2* __restrict__ ft, int N, const int* __restrict__ iCol,
                                const int* __restrict__ iRow, int K, float2* __restrict__ dat)
{
    const size_t l = blockIdx.y;
    const int nx = N / 2 + 1;
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < K; p += gridDim.x * blockDim.x) {
        const int row = iRow[p] < 0 ? iRow[p] + N : iRow[p];
        dat[l * K + p] = ft[(l * N + row) * nx + iCol[p]];
    }
}

// ------------------------------------------------------------ sigma^2 --
// Noise spectrum of the images against their best poses (Optimiser::
// allReduceSigma, src/Optimiser.cpp:6355-6630, with OPTIMISER_SIGMA_RANK1ST
// and OPTIMISER_SIGMA_WHOLE_FREQUENCY).  Per image l, with its model
// M = ctf P(R) S(t) and the unmasked model N = ctf P(R) S(t - offset) over the
// pixels of shells u = rint(|k|) < rSig (powerSpectrum, src/Functions/
// Spectrum.cpp:161-190, shell means):
//   vSigM[u] = <|datM - M|^2>, vSigN[u] = <|datN - N|^2>,
//   svd[u] = sqrt(<|M|^2> / <|datM|^2>);
// its group accumulates vSigM / 2, vSigN / 2, svd and a count.  CTA per
// image; shell sums in shared memory (FP32), group sums in FP64.
__global__ void __launch_bounds__(256)
k_sigma_image(const float2* __restrict__ P, int ldp, const float2* __restrict__ datM,
              const float2* __restrict__ datN, const float* __restrict__ ctf,
              const double* __restrict__ trans, const double* __restrict__ offset,
              const int* __restrict__ group, int byGroup, const int* __restrict__ iCol,
              const int* __restrict__ iRow, int K, int N, int rSig, double* __restrict__ acc)
{
    extern __shared__ float sh[];
    float* pM = sh;               // [rSig] each
    float* pN = pM + rSig;
    float* pS = pN + rSig;
    float* pD = pS + rSig;
    int* cnt = reinterpret_cast<int*>(pD + rSig);
    const size_t l = blockIdx.x;
    for (int u = threadIdx.x; u < rSig; u += blockDim.x) {
        pM[u] = pN[u] = pS[u] = pD[u] = 0.f;
        cnt[u] = 0;
    }
    __syncthreads();
    const float invN = 1.0f / (float)N;
    const float tx = (float)trans[2 * l], ty = (float)trans[2 * l + 1];
    const float ox = offset ? (float)offset[2 * l] : 0.f, oy = offset ? (float)offset[2 * l + 1] : 0.f;
    for (int p = threadIdx.x; p < K; p += blockDim.x) {
        const int i = iCol[p], j = iRow[p];
        const int u = (int)rintf(sqrtf((float)(i * i + j * j)));
        if (u >= rSig || i * i + j * j >= rSig * rSig) continue;
        const float2 pr = P[l * ldp + p];
        const float c = ctf[l * K + p];
        float sn, cs;
        // S(t) = exp(-2 pi i (i tx + j ty) / N)
        sincospif(-2.0f * ((float)i * tx + (float)j * ty) * invN, &sn, &cs);
        const float mr = c * (pr.x * cs - pr.y * sn), mi = c * (pr.x * sn + pr.y * cs);
        float so, co;
        sincospif(2.0f * ((float)i * ox + (float)j * oy) * invN, &so, &co);
        const float nr = mr * co - mi * so, ni = mr * so + mi * co;   // S(t - offset)
        const float2 a = datM[l * K + p], b = datN[l * K + p];
        atomicAdd(pM + u, (a.x - mr) * (a.x - mr) + (a.y - mi) * (a.y - mi));
        atomicAdd(pN + u, (b.x - nr) * (b.x - nr) + (b.y - ni) * (b.y - ni));
        atomicAdd(pS + u, mr * mr + mi * mi);
        atomicAdd(pD + u, a.x * a.x + a.y * a.y);
        atomicAdd(cnt + u, 1);
    }
    __syncthreads();
    const int g = byGroup ? group[l] - 1 : 0;
    double* ag = acc + (size_t)g * (3 * rSig + 1);
    for (int u = threadIdx.x; u < rSig; u += blockDim.x) {
        const double n = (double)cnt[u];
        atomicAdd(ag + u, 0.5 * pM[u] / n);
        atomicAdd(ag + rSig + u, 0.5 * pN[u] / n);
        atomicAdd(ag + 2 * rSig + u, sqrt((double)pS[u] / (double)pD[u]));
    }
    if (threadIdx.x == 0) atomicAdd(ag + 3 * rSig, 1.0);
}

// sig = ratio sigM + (1 - ratio) alpha sigN, ratio = min(1, svd); all groups
// copy group 0 when the images were pooled.  One thread per (group, shell).
__global__ void k_sigma_finish(const double* __restrict__ acc, int nGroup, int rSig, int byGroup,
                               double alpha, double* __restrict__ sig, double* __restrict__ sigRcp)
{
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= nGroup * rSig) return;
    const int g = idx / rSig, u = idx % rSig;
    const double* ag = acc + (size_t)(byGroup ? g : 0) * (3 * rSig + 1);
    const double w = ag[3 * rSig];
    const double sM = ag[u] / w, sN = ag[rSig + u] / w, svd = ag[2 * rSig + u] / w;
    const double ratio = fmin(1.0, svd);
    const double s = ratio * sM + (1.0 - ratio) * alpha * sN;
    sig[idx] = s;
    sigRcp[idx] = -0.5 / s;
}

// batched r2c plans, one per (context, size, batch), kept until the context goes
struct Plan {
    tg3_ctx* c;
    int N, batch;
    cufftHandle h;
};
std::vector<Plan> g_plans;
std::mutex g_planLock;

// Batched 2-D plans of a context, forward (real to complex) or inverse.
int get_plan(tg3_ctx* c, int N, int batch, cufftHandle* out, bool inverse = false)
{
    std::lock_guard<std::mutex> g(g_planLock);
    const int key = inverse ? -batch : batch;
    for (auto& p : g_plans)
        if (p.c == c && p.N == N && p.batch == key) {
            *out = p.h;
            return TG3_OK;
        }
    cufftHandle h;
    int n[2] = {N, N};
    const cufftResult r =
        inverse ? cufftPlanMany(&h, 2, n, nullptr, 1, N * (N / 2 + 1), nullptr, 1, N * N,
                                CUFFT_C2R, batch)
                : cufftPlanMany(&h, 2, n, nullptr, 1, N * N, nullptr, 1, N * (N / 2 + 1),
                                CUFFT_R2C, batch);
    if (r != CUFFT_SUCCESS) return fail(TG3_ERR_CUDA, "cuFFT plan creation failed");
    g_plans.push_back({c, N, key, h});
    *out = h;
    return TG3_OK;
}

// ReMask's real-space step: x / N^2 (the normalisation of the inverse
// transform, FFT::bw) times the soft mask of radius r and edge ew about the
// centre at index 0 (kernel_SoftMask / kernel_MulMask, gpu/src/Kernel.cu:
// 5249-5316): 1 inside r, 0.5 + 0.5 cos((u - r) / ew pi) on the edge, 0
// beyond r + ew, u from the wrapped indices.
__global__ void k_remask_real(float* __restrict__ real, int N, float r, float ew, size_t n)
{
    const float inv = 1.0f / ((float)N * (float)N);
    const size_t per = (size_t)N * N;
    for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < n * per;
         q += (size_t)gridDim.x * blockDim.x) {
        const int x = (int)(q % N), y = (int)((q / N) % N);
        const int i = x < N / 2 ? x : x - N, j = y < N / 2 ? y : y - N;
        const float u = sqrtf((float)(i * i + j * j));
        const float m = u > r + ew ? 0.f : (u >= r ? 0.5f + 0.5f * cospif((u - r) / ew) : 1.f);
        real[q] = real[q] * inv * m;
    }
}

// The img x img rfft grid in the particle transforms' order: pixel
// p = r (img/2 + 1) + i holds column i and row j = r (r < img/2), r - img.
__global__ void k_image_grid(int img, int* __restrict__ iCol, int* __restrict__ iRow)
{
    const int h = img / 2, n = img * (h + 1);
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
        const int r = p / (h + 1), i = p % (h + 1);
        iCol[p] = i;
        iRow[p] = r < h ? r : r - img;
    }
}

// One CTA per image: the centred image (index 0 moved to the middle, as an
// fftshift), minus its mean, over its unbiased standard deviation; the sums
// in FP64.
__global__ void k_centre_normalise(const float* __restrict__ real, int img,
                                   float* __restrict__ out)
{
    __shared__ double s1[32], s2[32];
    const int n = img * img, h = img / 2;
    const float* src = real + (size_t)blockIdx.x * n;
    float* dst = out + (size_t)blockIdx.x * n;
    double a = 0.0, b = 0.0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const double v = src[i];
        a += v;
        b += v * v;
    }
    for (int o = 16; o; o >>= 1) {
        a += __shfl_xor_sync(0xffffffffu, a, o);
        b += __shfl_xor_sync(0xffffffffu, b, o);
    }
    if ((threadIdx.x & 31) == 0) {
        s1[threadIdx.x >> 5] = a;
        s2[threadIdx.x >> 5] = b;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double ta = 0.0, tb = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); w++) {
            ta += s1[w];
            tb += s2[w];
        }
        const double mean = ta / n;
        const double var = fmax((tb - ta * mean) / (n - 1), 0.0);
        s1[0] = mean;
        s2[0] = var > 0.0 ? 1.0 / sqrt(var) : 0.0;
    }
    __syncthreads();
    const double mean = s1[0], rs = s2[0];
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const int y = i / img, x = i % img;
        const int ys = y + h < img ? y + h : y + h - img, xs = x + h < img ? x + h : x + h - img;
        dst[(size_t)y * img + x] = (float)(((double)src[(size_t)ys * img + xs] - mean) * rs);
    }
}

}  // namespace

extern "C" int tg3_ctx_render_references_d(tg3_ctx* c, int cls, const double* rotMat, int n,
                                           int img, float* out)
{
    int st = check_ctx(c);
    if (st) return st;
    if (cls < 0 || cls >= kMaxClasses || !c->vol[cls].blocks)
        return fail(TG3_ERR_STATE, "volume not set");
    if (!rotMat || !out || n <= 0 || img < 8 || (img & 1))
        return fail(TG3_ERR_ARG, "bad reference rendering arguments");
    const Volume& v = c->vol[cls];
    const int h = img / 2, K = img * (h + 1);
    // the grid's farthest pixel, (h, h) pf voxels out, with its trilinear
    // corners, must lie inside the stored half grid
    if ((int)ceil(1.41422 * h * v.pf) + 2 > v.vdim / 2)
        return fail(TG3_ERR_ARG, "reference image grid reaches past the volume");
    const int IB = std::min(n, 4096);
    const size_t oCol = 0, oRow = (sizeof(int) * K + 255) / 256 * 256,
                 oP = oRow + (sizeof(int) * K + 255) / 256 * 256,
                 oR = oP + (sizeof(float2) * (size_t)K * IB + 255) / 256 * 256,
                 total = oR + sizeof(float) * (size_t)img * img * IB;
    char* b = (char*)ws_get(c, WS_RENDER, total, &st);
    if (!b) return st;
    float* pscr = (float*)ws_get(c, WS_PROJ, sizeof(float) * project_scratch_floats(IB, 2 * K), &st);
    if (!pscr) return st;
    int* gCol = (int*)(b + oCol);
    int* gRow = (int*)(b + oRow);
    float* P = (float*)(b + oP);
    float* R = (float*)(b + oR);
    cudaStream_t s = c->stream;
    k_image_grid<<<(K + 255) / 256, 256, 0, s>>>(img, gCol, gRow);
    TG3_LAUNCH_CHECK("image grid");
    cufftHandle plan;
    for (int r0 = 0; r0 < n; r0 += IB) {
        const int m = std::min(IB, n - r0);
        TG3_CUDA(launch_project(nullptr, nullptr, v.blocks, v.vdim, v.pf, nullptr,
                                rotMat + 9 * (size_t)r0, m, m, gCol, gRow, K, P, 2 * K, nullptr,
                                nullptr, nullptr, pscr, c->d_flag, 0, s));
        if ((st = get_plan(c, img, m, &plan, true))) return st;
        if (cufftSetStream(plan, s) != CUFFT_SUCCESS ||
            cufftExecC2R(plan, reinterpret_cast<cufftComplex*>(P), R) != CUFFT_SUCCESS)
            return fail(TG3_ERR_CUDA, "cuFFT inverse transform failed");
        k_centre_normalise<<<m, 256, 0, s>>>(R, img, out + (size_t)r0 * img * img);
        TG3_LAUNCH_CHECK("reference centring");
    }
    return TG3_OK;
}

void prep_release(tg3_ctx* c)
{
    std::lock_guard<std::mutex> g(g_planLock);
    for (size_t i = 0; i < g_plans.size();) {
        if (g_plans[i].c == c) {
            cufftDestroy(g_plans[i].h);
            g_plans.erase(g_plans.begin() + i);
        } else {
            i++;
        }
    }
}

}  // namespace tg3

using namespace tg3;

extern "C" int tg3_sigma_d(tg3_ctx* c, int cls, int nImg, const float* datM, const float* datN,
                           const float* ctf, const double* rotMat, const double* trans,
                           const double* offset, const int* group, int nGroup, int byGroup,
                           int rSig, float maskRadius, float pixelSize, double* sig,
                           double* sigRcp)
{
    int st = check_ctx(c);
    if (st) return st;
    if (cls < 0 || cls >= kMaxClasses || !c->vol[cls].blocks)
        return fail(TG3_ERR_STATE, "volume of the class not set");
    if (!datM || !datN || !ctf || !rotMat || !trans || !sig || !sigRcp || (byGroup && !group))
        return fail(TG3_ERR_ARG, "null device pointer");
    if (nImg <= 0 || nGroup <= 0 || rSig <= 0 || rSig > 2048 || !(pixelSize > 0))
        return fail(TG3_ERR_ARG, "bad sigma arguments");
    const Volume& v = c->vol[cls];
    if ((st = check_geometry(c, v.vdim, v.pf))) return st;
    const int K = c->px.K, N = c->px.idim;
    if (rSig > N / 2) return fail(TG3_ERR_ARG, "rSig beyond the image's Nyquist shell");
    const int IB = std::min(nImg, 2048);
    auto up = [](size_t x) { return (x + 255) / 256 * 256; };
    const size_t accN = (size_t)nGroup * (3 * rSig + 1);
    const size_t oA = 0, oP = up(sizeof(double) * accN), total = oP + sizeof(float2) * (size_t)K * IB;
    char* b = (char*)ws_get(c, WS_PREP, total, &st);
    if (!b) return st;
    double* acc = (double*)(b + oA);
    float* P = (float*)(b + oP);
    float* pscr = (float*)ws_get(c, WS_PROJ, sizeof(float) * project_scratch_floats(IB, 2 * K), &st);
    if (!pscr) return st;
    cudaStream_t s = c->stream;
    TG3_CUDA(cudaMemsetAsync(acc, 0, sizeof(double) * accN, s));
    const size_t smem = (4 * sizeof(float) + sizeof(int)) * (size_t)rSig;
    for (int l0 = 0; l0 < nImg; l0 += IB) {
        const int n = std::min(IB, nImg - l0);
        TG3_CUDA(launch_project(nullptr, nullptr, v.blocks, v.vdim, v.pf, nullptr,
                                rotMat + 9 * (size_t)l0, n, n, c->px.iCol, c->px.iRow, K, P, 2 * K,
                                nullptr, nullptr, nullptr, pscr, c->d_flag, 0, s));
        const size_t o = (size_t)l0 * K;
        k_sigma_image<<<n, 256, smem, s>>>(
            reinterpret_cast<const float2*>(P), K, reinterpret_cast<const float2*>(datM) + o,
            reinterpret_cast<const float2*>(datN) + o, ctf + o, trans + 2 * (size_t)l0,
            offset ? offset + 2 * (size_t)l0 : nullptr, byGroup ? group + l0 : nullptr, byGroup,
            c->px.iCol, c->px.iRow, K, N, rSig, acc);
        TG3_LAUNCH_CHECK("sigma per image");
    }
    const double rm = (double)maskRadius / ((double)N * (double)pixelSize);
    const double alpha = sqrt(M_PI * rm * rm);
    k_sigma_finish<<<(nGroup * rSig + 255) / 256, 256, 0, s>>>(acc, nGroup, rSig, byGroup, alpha,
                                                                sig, sigRcp);
    TG3_LAUNCH_CHECK("sigma finish");
    return TG3_OK;
}

extern "C" int tg3_prepare_images_d(tg3_ctx* c, const float* img, int nImg, int N,
                                    float maskRadiusPx, int mask, float stdN, float* dat,
                                    float* stats)
{
    int st = check_ctx(c);
    if (st) return st;
    if (!img || !dat || nImg <= 0 || N < 4 || (N & 1) || !(maskRadiusPx > 0))
        return fail(TG3_ERR_ARG, "bad preprocessing arguments");
    if (!c->px.iCol || c->px.idim != N)
        return fail(TG3_ERR_STATE, "the active pixel set was not made for this image size");
    if (maskRadiusPx >= N / 2 * 1.4142135f)
        return fail(TG3_ERR_ARG, "mask radius leaves no background pixels");
    const int K = c->px.K;
    const float r = maskRadiusPx, ew = 6.0f;
    // the background's pixels, and the mask's edge in squared radii, compared as
    // the FP32 radii u = sqrt(q) are: u < r inside, u > r + ew outside
    const int half = N / 2, bgAbove = (int)std::floor((double)r * (double)r);
    long long cnt = 0;
    for (int j = -half; j < half; j++) {
        const long long q = (long long)bgAbove - (long long)j * j;
        int h = q < 0 ? -1 : (int)std::sqrt((double)q);
        while (h >= 0 && (long long)h * h > q) h--;
        while (q >= 0 && (h + 1LL) * (h + 1) <= q) h++;
        cnt += h < 0 ? N : std::max(half - h, 0) + std::max(half - h - 1, 0);
    }
    SoftMask sm{nullptr, 2 * half * half, 2 * half * half};
    if (mask) {
        sm.qIn = (int)std::min((double)r * r + 2, 2.0 * half * half);
        while (sm.qIn > 0 && !(std::sqrt((float)sm.qIn) < r)) sm.qIn--;
        sm.qOut = (int)std::min(((double)r + ew) * ((double)r + ew) + 2, 2.0 * half * half);
        while (sm.qOut > sm.qIn && std::sqrt((float)sm.qOut) > r + ew) sm.qOut--;
    }
    const int nMask = sm.qOut - sm.qIn + 1;
    const PrepLaunch pl = prep_launch(N, std::min(c->px.maxAbs, half), nMask);
    const int IB = std::min(nImg, pl.A ? 65535 : 2048);
    const size_t img2 = (size_t)N * N, ft2 = (size_t)N * (half + 1);
    auto up = [](size_t x) { return (x + 255) / 256 * 256; };
    const size_t oSt = 0, oN = up(sizeof(double) * 4 * (size_t)nImg),
                 oM = oN + up(sizeof(Scaling) * (size_t)nImg), oT = oM + up(sizeof(float) * nMask),
                 oL = oT + up(sizeof(float2) * (pl.A ? N : 0)),
                 oR = oL + up(sizeof(int) * (pl.A ? K : 0)),
                 oF = up(oR + (pl.A ? 0 : sizeof(float) * img2 * IB)),
                 total = oF + (pl.A ? 0 : sizeof(float2) * ft2 * IB);
    char* b = (char*)ws_get(c, WS_PREP, total, &st);
    if (!b) return st;
    double* stv = (double*)(b + oSt);
    Scaling* sc = (Scaling*)(b + oN);
    float* real = (float*)(b + oR);
    cufftComplex* ft = (cufftComplex*)(b + oF);
    cudaStream_t s = c->stream;
    sm.tab = (float*)(b + oM);
    const int maxCol = std::min(c->px.maxAbs, half);
    const PrepTables tabs{(float*)(b + oM), sm.qIn, nMask, r, ew, (float2*)(b + oT), pl.A, pl.B,
                          (int*)(b + oL), c->px.iCol, c->px.iRow, pl.A ? K : 0, pl.cols, maxCol,
                          pl.W};
    const size_t rowsB = sizeof(int2) * (size_t)std::min((N + 3) / 4 * 4, kBgBand);
    (N < 256 ? k_bg_stats<2> : k_bg_stats<8>)<<<nImg, 256, rowsB, s>>>(img, N, bgAbove, (double)cnt,
                                                                      stv, stats, tabs);
    TG3_LAUNCH_CHECK("background statistics");
    k_stdn<<<1, 256, 0, s>>>(stv, nImg, stdN, sc);
    TG3_LAUNCH_CHECK("noise level");
    if (pl.A)
        TG3_CUDA(allow_shared(k_prep_ft));
    for (int l0 = 0; l0 < nImg; l0 += IB) {
        const int n = std::min(IB, nImg - l0);
        float2* out = reinterpret_cast<float2*>(dat) + (size_t)l0 * K;
        if (pl.A) {
            const PrepFt f{img + (size_t)l0 * img2, pl.A, pl.B, pl.lanes, pl.ex, pl.cols,
                           maxCol, pl.W, sm, tabs.tw, sc + l0, tabs.slot, K, out};
            k_prep_ft<<<dim3(pl.blocks, n), pl.threads, pl.smem, s>>>(f);
            TG3_LAUNCH_CHECK("normalise, mask, transform and gather");
            continue;
        }
        k_prep_image<<<dim3((N + kPrepRows - 1) / kPrepRows, n), std::min(N, 256), 0, s>>>(
            img + (size_t)l0 * img2, N, sm, sc + l0, real);
        TG3_LAUNCH_CHECK("normalise and mask");
        cufftHandle h;
        if ((st = get_plan(c, N, n, &h))) return st;
        if (cufftSetStream(h, s) != CUFFT_SUCCESS || cufftExecR2C(h, real, ft) != CUFFT_SUCCESS)
            return fail(TG3_ERR_CUDA, "cuFFT forward transform failed");
        k_gather_pixels<<<dim3((K + 255) / 256, n), 256, 0, s>>>(
            reinterpret_cast<const float2*>(ft), N, c->px.iCol, c->px.iRow, K, out);
        TG3_LAUNCH_CHECK("pixel gather");
    }
    return TG3_OK;
}

extern "C" int tg3_remask_d(tg3_ctx* c, const float* imgFT, int nImg, int N, float maskRadiusPx,
                            float edgeWidth, float* out)
{
    int st = check_ctx(c);
    if (st) return st;
    if (!imgFT || !out || nImg <= 0 || N < 4 || (N & 1) || !(maskRadiusPx > 0) ||
        !(edgeWidth > 0))
        return fail(TG3_ERR_ARG, "bad re-mask arguments");
    const int IB = std::min(nImg, 2048);
    const size_t img2 = (size_t)N * N, ft2 = (size_t)N * (N / 2 + 1);
    // the inverse transform overwrites its input: it reads a copy
    const size_t oR = 0, oF = (sizeof(float) * img2 * IB + 255) / 256 * 256,
                 total = oF + sizeof(float2) * ft2 * IB;
    char* b = (char*)ws_get(c, WS_PREP, total, &st);
    if (!b) return st;
    float* real = (float*)(b + oR);
    cufftComplex* ft = (cufftComplex*)(b + oF);
    cudaStream_t s = c->stream;
    for (int l0 = 0; l0 < nImg; l0 += IB) {
        const int n = std::min(IB, nImg - l0);
        TG3_CUDA(cudaMemcpyAsync(ft, imgFT + 2 * ft2 * (size_t)l0, sizeof(float2) * ft2 * n,
                                 cudaMemcpyDeviceToDevice, s));
        cufftHandle hi, hf;
        if ((st = get_plan(c, N, n, &hi, true))) return st;
        if ((st = get_plan(c, N, n, &hf, false))) return st;
        if (cufftSetStream(hi, s) != CUFFT_SUCCESS || cufftExecC2R(hi, ft, real) != CUFFT_SUCCESS)
            return fail(TG3_ERR_CUDA, "cuFFT inverse transform failed");
        const size_t cnt = img2 * n;
        k_remask_real<<<(unsigned)std::min<size_t>((cnt + 255) / 256, 152 * 32), 256, 0, s>>>(
            real, N, maskRadiusPx, edgeWidth, n);
        TG3_LAUNCH_CHECK("re-mask");
        if (cufftSetStream(hf, s) != CUFFT_SUCCESS ||
            cufftExecR2C(hf, real, reinterpret_cast<cufftComplex*>(out) + ft2 * (size_t)l0) !=
                CUFFT_SUCCESS)
            return fail(TG3_ERR_CUDA, "cuFFT forward transform failed");
    }
    return TG3_OK;
}

extern "C" int tg3_ReMask(float* const* images, int nImg, int idim, float maskRadius,
                          float pixelSize, float ew)
{
    if (!images || nImg <= 0 || idim <= 0 || !(pixelSize > 0))
        return fail(TG3_ERR_ARG, "bad ReMask arguments");
    int st = TG3_OK;
    tg3_ctx* c = nullptr;
    {
        int dev = 0;
        TG3_CUDA(cudaGetDevice(&dev));
        static std::mutex mu;
        static tg3_ctx* ctxs[64] = {};
        if (dev < 0 || dev >= 64) return fail(TG3_ERR_ARG, "device ordinal out of range");
        std::lock_guard<std::mutex> lk(mu);
        if (!ctxs[dev] && (st = tg3_ctx_create(&ctxs[dev], dev))) return st;
        c = ctxs[dev];
    }
    const size_t ft2 = (size_t)idim * (idim / 2 + 1);
    const int IB = std::min(nImg, 1024);
    float* d = (float*)ws_get(c, WS_H2D, sizeof(float2) * ft2 * IB, &st);
    if (!d) return st;
    cudaStream_t s = c->stream;
    for (int l0 = 0; l0 < nImg; l0 += IB) {
        const int n = std::min(IB, nImg - l0);
        for (int i = 0; i < n; i++)
            TG3_CUDA(cudaMemcpyAsync(d + 2 * ft2 * i, images[l0 + i], sizeof(float2) * ft2,
                                     cudaMemcpyHostToDevice, s));
        if ((st = tg3_remask_d(c, d, n, idim, maskRadius / pixelSize, ew, d))) return st;
        for (int i = 0; i < n; i++)
            TG3_CUDA(cudaMemcpyAsync(images[l0 + i], d + 2 * ft2 * i, sizeof(float2) * ft2,
                                     cudaMemcpyDeviceToHost, s));
        TG3_CUDA(cudaStreamSynchronize(s));
    }
    return TG3_OK;
}
