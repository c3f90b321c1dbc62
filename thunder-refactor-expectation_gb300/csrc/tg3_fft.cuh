// tg3_fft.cuh -- FP32 complex transforms of many lines by a CTA, for kernels
// that do something else with the data on the way in or out (the
// reconstruction's passes, the image preprocessing).
//
// A line of n = A B points is transformed by TL threads in two steps of whole
// small transforms in registers, with one exchange through shared memory
// between them:
//   first:  thread j holds x[j + r B], r < A: a transform of A, times w_n^(r j);
//   second: thread k holds the B values of its k < A: a transform of B, whose
//           outputs are X[k + A s], s < B.
// The outputs are spread over the threads as the inputs of a transform with A
// and B exchanged, so a pass that transforms, changes the points and transforms
// back (B, A) needs no exchange but the two inside.  The inverse is the forward
// transform of the points with real and imaginary part exchanged, exchanged
// back (unnormalised, as the forward one).
//
// The small transforms are unrolled from radix 2, 3, 4, 5 and (by their definition) 7, 11, 13 with constant
// twiddles; the twiddles between the steps come from one table of the n-th
// roots of unity (each rounded from an accurate sine and cosine), so the error
// is that of the additions.  Additions work on (re, im) pairs.  A CTA has
// kFftLines lines, consecutive threads on consecutive lines: global and shared
// accesses are whole 64-byte rows.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace tg3 {

constexpr int kFftLines = 8;

namespace fft {

typedef uint64_t c64;   // (re, im)

__device__ __forceinline__ c64 pack(float x, float y)
{
    c64 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ float2 unpack(c64 v)
{
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ c64 add(c64 a, c64 b)
{
    c64 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ c64 mad(c64 a, c64 b, c64 c)
{
    c64 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ c64 sub(c64 a, c64 b) { return mad(b, pack(-1.f, -1.f), a); }
__device__ __forceinline__ c64 scale(c64 a, float s)
{
    c64 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(pack(s, s)));
    return r;
}
// a times -i
__device__ __forceinline__ c64 rot(c64 a)
{
    const float2 v = unpack(a);
    return pack(v.y, -v.x);
}
__device__ __forceinline__ c64 swapped(c64 a)
{
    const float2 v = unpack(a);
    return pack(v.y, v.x);
}
__device__ __forceinline__ c64 times(c64 a, float wx, float wy)
{
    const float2 v = unpack(a);
    return pack(v.x * wx - v.y * wy, v.x * wy + v.y * wx);
}

// cos and sin of 2 pi k / n, by their power series after reduction to an
// eighth of the circle
struct Root {
    double c, s;
};
constexpr Root root(int k, int n)
{
    k %= n;
    bool flip = false, half = false, quarter = false;
    // angle 2 pi k / n in units of 8 n: first into [0, pi], then [0, pi / 2], [0, pi / 4]
    long long a = 8LL * k, N = 8LL * n;
    if (2 * a > N) {
        a = N - a;
        flip = true;
    }
    if (4 * a > N) {
        a = N / 2 - a;
        half = true;
    }
    if (8 * a > N) {
        a = N / 4 - a;
        quarter = true;
    }
    const double x = 6.28318530717958647692528676655900577 * (double)a / (double)N;
    double c = 1.0, s = x, tc = 1.0, ts = x;
    for (int i = 1; i < 12; i++) {
        tc *= -x * x / ((2 * i - 1) * (2 * i));
        ts *= -x * x / ((2 * i) * (2 * i + 1));
        c += tc;
        s += ts;
    }
    if (quarter) {
        const double t = c;
        c = s;
        s = t;
    }
    if (half) c = -c;
    if (flip) s = -s;
    return {c, s};
}

// a times exp(-2 pi i K / N)
template <int K, int N>
__device__ __forceinline__ c64 twiddle(c64 a)
{
    constexpr int k = K % N;
    if constexpr (k == 0) {
        return a;
    } else if constexpr (4 * k == N) {
        return rot(a);
    } else if constexpr (2 * k == N) {
        return scale(a, -1.f);
    } else {
        constexpr Root w = root(k, N);
        return times(a, (float)w.c, (float)-w.s);
    }
}

// factors of a small transform: R = kP * Q
constexpr int first_factor(int r)
{
    return r % 8 == 0 && r > 8 && r != 16 ? r / 8    // 24 = 3 8, 32 = 4 8
           : r % 4 == 0 && r > 4          ? 4
           : r % 3 == 0                   ? 3
           : r % 5 == 0                   ? 5
                                          : 2;
}

template <int R>
__device__ __forceinline__ void dft(c64* v);

// cosines and sines of 2 pi k / R
template <int R>
struct Circle {
    float c[R] = {}, s[R] = {};
    constexpr Circle()
    {
        for (int k = 0; k < R; k++) {
            const Root w = root(k, R);
            c[k] = (float)w.c;
            s[k] = (float)w.s;
        }
    }
};

template <int R, int P, int Q, int I>
__device__ __forceinline__ void twiddle_all(c64* u)
{
    if constexpr (I < R) {
        u[I] = twiddle<(I / Q) * (I % Q), R>(u[I]);
        twiddle_all<R, P, Q, I + 1>(u);
    }
}

// v[0 .. R - 1] to its transform, in order
template <int R>
__device__ __forceinline__ void dft(c64* v)
{
    if constexpr (R == 1) {
    } else if constexpr (R == 2) {
        const c64 a = v[0];
        v[0] = add(a, v[1]);
        v[1] = sub(a, v[1]);
    } else if constexpr (R == 3) {
        const c64 s = add(v[1], v[2]), t = scale(rot(sub(v[1], v[2])), 0.86602540378443864676f);
        const c64 m = mad(s, pack(-0.5f, -0.5f), v[0]);
        v[0] = add(v[0], s);
        v[1] = add(m, t);
        v[2] = sub(m, t);
    } else if constexpr (R == 4) {
        const c64 s = add(v[0], v[2]), t = sub(v[0], v[2]), u = add(v[1], v[3]),
                  w = rot(sub(v[1], v[3]));
        v[0] = add(s, u);
        v[2] = sub(s, u);
        v[1] = add(t, w);
        v[3] = sub(t, w);
    } else if constexpr (R == 5) {
        const float c1 = 0.30901699437494742410f, c2 = -0.80901699437494742410f;
        const float s1 = 0.95105651629515357212f, s2 = 0.58778525229247312917f;
        const c64 a1 = add(v[1], v[4]), a2 = add(v[2], v[3]);
        const c64 b1 = rot(sub(v[1], v[4])), b2 = rot(sub(v[2], v[3]));
        const c64 m1 = mad(a2, pack(c2, c2), mad(a1, pack(c1, c1), v[0]));
        const c64 m2 = mad(a2, pack(c1, c1), mad(a1, pack(c2, c2), v[0]));
        const c64 t1 = mad(b2, pack(s2, s2), scale(b1, s1));
        const c64 t2 = mad(b2, pack(-s1, -s1), scale(b1, s2));
        v[0] = add(v[0], add(a1, a2));
        v[1] = add(m1, t1);
        v[4] = sub(m1, t1);
        v[2] = add(m2, t2);
        v[3] = sub(m2, t2);
    } else if constexpr (R == 7 || R == 11 || R == 13) {
        // X[k], X[R - k] = v[0] + sum_j (v[j] + v[R - j]) cos(2 pi j k / R)
        //                  -+ i (v[j] - v[R - j]) sin(2 pi j k / R)
        constexpr Circle<R> w;
        constexpr int H = R / 2;
        c64 a[H], b[H], sum = v[0];
#pragma unroll
        for (int j = 1; j <= H; j++) {
            a[j - 1] = add(v[j], v[R - j]);
            b[j - 1] = rot(sub(v[j], v[R - j]));
            sum = add(sum, a[j - 1]);
        }
#pragma unroll
        for (int k = 1; k <= H; k++) {
            c64 m = v[0], t = scale(b[0], w.s[k]);
#pragma unroll
            for (int j = 1; j <= H; j++) {
                m = mad(a[j - 1], pack(w.c[j * k % R], w.c[j * k % R]), m);
                if (j > 1) t = mad(b[j - 1], pack(w.s[j * k % R], w.s[j * k % R]), t);
            }
            v[k] = add(m, t);
            v[R - k] = sub(m, t);
        }
        v[0] = sum;
    } else {
        // x[q + Q p]: transforms of P over p, twiddles, transforms of Q over q
        constexpr int P = first_factor(R), Q = R / P;
        c64 u[R];
#pragma unroll
        for (int q = 0; q < Q; q++) {
            c64 t[P];
#pragma unroll
            for (int p = 0; p < P; p++) t[p] = v[q + Q * p];
            dft<P>(t);
#pragma unroll
            for (int p = 0; p < P; p++) u[p * Q + q] = t[p];
        }
        twiddle_all<R, P, Q, 0>(u);
#pragma unroll
        for (int p = 0; p < P; p++) {
            dft<Q>(u + p * Q);
#pragma unroll
            for (int q = 0; q < Q; q++) v[p + P * q] = u[p * Q + q];
        }
    }
}

// Threads of a line and the items of the two steps.
template <int A, int B>
struct Shape {
    static constexpr int n = A * B;
    // as many threads as the smaller step count divides, else one a larger item
    static constexpr int TL = A % B == 0 ? B : A;
    static constexpr int threads = TL * kFftLines;
    static constexpr int I1 = (B + TL - 1) / TL;     // first-step items of a thread
    static constexpr int I2 = (A + TL - 1) / TL;     // second-step items
    // exchange buffer of either order: A rows of B or B rows of A, odd pitches;
    // or the lines one after another, n + 2 apart
    static constexpr int rows = A * (B | 1) > B * (A | 1) ? A * (B | 1) : B * (A | 1);
    static constexpr int floats2 = (rows > n + 2 ? rows : n + 2) * kFftLines;
    static constexpr size_t smem = sizeof(float2) * (floats2 + n);   // and the roots
};

// The transform of n = A B: v[i][r] = x[(t + i TL) + r B] (i < items of the
// first step, t the thread of the line) to o[i][s] = X[(t + i TL) + A s].  buf:
// the exchange buffer; tw: the n-th roots (shared).  All threads of the CTA.
template <int A, int B, int TL, int I1, int I2>
__device__ __forceinline__ void run(c64 (&v)[I1][A], c64 (&o)[I2][B], c64* buf,
                                    const float2* __restrict__ tw, int t, int line)
{
    constexpr int pitch = B | 1;
#pragma unroll
    for (int i = 0; i < I1; i++) {
        const int j = t + i * TL;
        if (j < B) {
            dft<A>(v[i]);
#pragma unroll
            for (int r = 0; r < A; r++) {
                const float2 w = tw[r * j];
                buf[(r * pitch + j) * kFftLines + line] = r ? times(v[i][r], w.x, w.y) : v[i][r];
            }
        }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < I2; i++) {
        const int k = t + i * TL;
        if (k < A) {
#pragma unroll
            for (int s = 0; s < B; s++) o[i][s] = buf[(k * pitch + s) * kFftLines + line];
            dft<B>(o[i]);
        }
    }
    __syncthreads();
}

// exp(-2 pi i k / n) for k < n into global tw, once for the kernels of a call
static __global__ void k_roots(float2* __restrict__ tw, int n)
{
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        double s, c;
        sincospi(-2.0 * k / n, &s, &c);
        tw[k] = make_float2((float)c, (float)s);
    }
}

}  // namespace fft
}  // namespace tg3
