// fft_reg.cuh -- register-resident, fully unrolled mixed-radix FFT on packed FP32 pairs.
//
// A thread's transform of length N runs as transforms of length N/4 (or N/2) over its
// sub-sequences x[r + 4m].  Two sub-sequences share one set of twiddles, so they run together
// in the two lanes of packed FP32 instructions (add/mul/fma.f32x2): cplx<float2> holds the
// same element of both, real parts in one 64-bit register pair, imaginary parts in another.
// Neighbouring elements (x[2j], x[2j + 1]) are exactly such a pair, and they are what wide
// loads of a row bring in, so packing costs no moves.  Only the last combination across the
// sub-sequences is scalar.
//
// What bounds it: a packed instruction does two FP32 operations in one issue slot but
// occupies the FP32 pipe for two (measured 126 adds, 118 multiply-adds per SM and clock,
// scalar 122), and the kernels around it are bound by issue slots, not by that pipe.  A
// 32-point transform takes about 290 instructions against 432 in scalar form.
//
// Rounding: every product and sum is the one the scalar form rounds, in the same order, so
// packed and scalar results are identical; fft_first_product() says which of a twiddle's two
// products is rounded before the fused multiply-add.
//
// Natural order in, natural order out, unnormalised: INV = false uses exp(-2*pi*i*k*n/N),
// INV = true exp(+2*pi*i*k*n/N).  Decimation in time, radix 4 where possible, then 2 and 3
// (every length is a multiple of 4 of the form 4 * 2^a * 3^b).  Twiddles are compile-time
// immediates (piv_common.cuh).
#pragma once

#include "piv_common.cuh"

namespace piv {

template <class V>
struct cplx {
    V re, im;
};

__device__ __forceinline__ float vadd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float vsub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float vmul(float a, float c) { return __fmul_rn(a, c); }
__device__ __forceinline__ float vfma(float a, float c, float b) { return __fmaf_rn(a, c, b); }
__device__ __forceinline__ float2 vadd(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 vsub(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.f, -1.f), a); }
__device__ __forceinline__ float2 vmul(float2 a, float c) { return __fmul2_rn(a, make_float2(c, c)); }
__device__ __forceinline__ float2 vfma(float2 a, float c, float2 b) { return __ffma2_rn(a, make_float2(c, c), b); }

// exp(-2 pi i E/N) in quarter turns (0..3), or -1 when it is none
constexpr int quarter_turns(int N, int E)
{
    const int e = ((E % N) + N) % N;
    return (4 * e) % N == 0 ? 4 * e / N : -1;
}
// the quarter turns left over by twiddle(), which multiplies by everything else
constexpr int left_turns(int N, int E) { return quarter_turns(N, E) < 0 ? 0 : quarter_turns(N, E); }

// a + t*b with t = (-i)^Q forward, (+i)^Q inverse: the turn is a choice of operands and signs
template <bool INV, int Q, class V>
__device__ __forceinline__ cplx<V> add_turned(cplx<V> a, cplx<V> b)
{
    constexpr int q = INV ? (4 - (Q & 3)) & 3 : Q & 3;  // in units of -i
    if constexpr (q == 0) return {vadd(a.re, b.re), vadd(a.im, b.im)};
    else if constexpr (q == 1) return {vadd(a.re, b.im), vsub(a.im, b.re)};
    else if constexpr (q == 2) return {vsub(a.re, b.re), vsub(a.im, b.im)};
    else return {vsub(a.re, b.im), vadd(a.im, b.re)};
}

// The imaginary part re*s + im*c is fma(re, s, im*c), or fma(im, c, re*s) where this is true.
constexpr bool fft_first_product(int N, int e, bool inv) { return !inv && 0 < 4 * e && 4 * e < N && 8 * e != N; }

// v * exp(-/+ 2*pi*i*E/N), quarter turns excepted (left to add_turned)
template <int N, bool INV, int E, class V>
__device__ __forceinline__ cplx<V> twiddle(cplx<V> v)
{
    constexpr int e = ((E % N) + N) % N;
    if constexpr (quarter_turns(N, e) >= 0) {
        return v;
    } else {
        constexpr CosSin cs = cossin_2pi(e, N);
        constexpr float c = (float)cs.c;
        constexpr float s = INV ? (float)cs.s : (float)(-cs.s);
        cplx<V> r;
        r.re = vfma(v.re, c, vmul(v.im, -s));
        if constexpr (fft_first_product(N, e, INV)) r.im = vfma(v.im, c, vmul(v.re, s));
        else r.im = vfma(v.re, s, vmul(v.im, c));
        return r;
    }
}

constexpr int pick_radix(int n) { return n % 4 == 0 ? 4 : (n % 2 == 0 ? 2 : 3); }

// one radix-4 combination: X[0..3] of a, b, c, d, still to be turned by qb, qc, qd quarters
template <bool INV, int qb, int qc, int qd, class V>
__device__ __forceinline__ void combine4(cplx<V> a, cplx<V> b, cplx<V> c, cplx<V> d, cplx<V> &x0, cplx<V> &x1,
                                         cplx<V> &x2, cplx<V> &x3)
{
    const cplx<V> t0 = add_turned<INV, qc>(a, c), t1 = add_turned<INV, qc + 2>(a, c);
    const cplx<V> t2 = add_turned<INV, qd - qb + 4>(b, d), t3 = add_turned<INV, qd - qb + 6>(b, d);
    x0 = add_turned<INV, qb>(t0, t2);
    x1 = add_turned<INV, qb + 1>(t1, t3);
    x2 = add_turned<INV, qb + 2>(t0, t2);
    x3 = add_turned<INV, qb + 3>(t1, t3);
}

// In-place transform of length N of every lane of V.
template <int N, bool INV, class V>
__device__ __forceinline__ void fft(cplx<V> (&x)[N])
{
    if constexpr (N == 1) {
    } else if constexpr (N == 3) {
        // X1 = a - (b+c)/2 -/+ i*sqrt(3)/2*(b-c), X2 = the other sign
        constexpr float h = 0.86602540378443864676f;  // sqrt(3)/2
        constexpr float hs = INV ? -h : h;
        const cplx<V> a = x[0], b = x[1], c = x[2];
        const cplx<V> t1 = add_turned<INV, 0>(b, c), t2 = add_turned<INV, 2>(b, c);
        const cplx<V> m = {vfma(t1.re, -0.5f, a.re), vfma(t1.im, -0.5f, a.im)};
        x[0] = add_turned<INV, 0>(a, t1);
        x[1] = {vfma(t2.im, hs, m.re), vfma(t2.re, -hs, m.im)};
        x[2] = {vfma(t2.im, -hs, m.re), vfma(t2.re, hs, m.im)};
    } else {
        constexpr int R = pick_radix(N), M = N / R;
        static_assert(R * M == N, "lengths of factors 2 and 3");
        cplx<V> sub[R][M];
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
            for (int m = 0; m < M; ++m) sub[r][m] = x[r + R * m];
#pragma unroll
        for (int r = 0; r < R; ++r) fft<M, INV>(sub[r]);
        static_for<0, M>([&](auto kc) {
            constexpr int k = decltype(kc)::value;
            const cplx<V> a = sub[0][k], b = twiddle<N, INV, k>(sub[1][k]);
            if constexpr (R == 2) {
                x[k] = add_turned<INV, left_turns(N, k)>(a, b);
                x[k + M] = add_turned<INV, left_turns(N, k) + 2>(a, b);
            } else if constexpr (R == 4) {
                combine4<INV, left_turns(N, k), left_turns(N, 2 * k), left_turns(N, 3 * k)>(
                    a, b, twiddle<N, INV, 2 * k>(sub[2][k]), twiddle<N, INV, 3 * k>(sub[3][k]), x[k], x[k + M],
                    x[k + 2 * M], x[k + 3 * M]);
            } else {
                cplx<V> t[3] = {a, b, twiddle<N, INV, 2 * k>(sub[2][k])};
                fft<3, INV>(t);
                x[k] = t[0];
                x[k + M] = t[1];
                x[k + 2 * M] = t[2];
            }
        });
    }
}

// Inverse transforms of 32 points and more split radix-2 first, all others radix-4 first.
template <int N, bool INV>
constexpr bool radix2_first() { return INV && N >= 32; }

// One thread's transform of length N (a multiple of 4): p[j] = (x[2j], x[2j + 1]) in,
// x in natural order out.  Radix-4 first: p's even entries hold (x[4m], x[4m + 1]), its odd
// ones (x[4m + 2], x[4m + 3]).  Radix-2 first: p holds the even and the odd half.
template <int N, bool INV>
__device__ __forceinline__ void fft_thread(cplx<float2> (&p)[N / 2], cplx<float> (&x)[N])
{
    static_assert(N % 4 == 0, "length divisible by 4");
    if constexpr (radix2_first<N, INV>()) {
        constexpr int H = N / 2, Q = N / 4;
        fft<H, INV>(p);
        static_for<0, Q>([&](auto jc) {
            constexpr int j = decltype(jc)::value;
            constexpr int q = left_turns(N, j);
            const cplx<float> e0 = {p[j].re.x, p[j].im.x}, e1 = {p[j + Q].re.x, p[j + Q].im.x};
            const cplx<float> o0 = twiddle<N, INV, j>(cplx<float>{p[j].re.y, p[j].im.y});
            const cplx<float> o1 = twiddle<N, INV, j>(cplx<float>{p[j + Q].re.y, p[j + Q].im.y});
            x[j] = add_turned<INV, q>(e0, o0);
            x[j + H] = add_turned<INV, q + 2>(e0, o0);
            x[j + Q] = add_turned<INV, q + 1>(e1, o1);
            x[j + Q + H] = add_turned<INV, q + 3>(e1, o1);
        });
    } else {
        constexpr int M = N / 4;
        cplx<float2> u[M], v[M];
#pragma unroll
        for (int m = 0; m < M; ++m) {
            u[m] = p[2 * m];
            v[m] = p[2 * m + 1];
        }
        fft<M, INV>(u);
        fft<M, INV>(v);
        static_for<0, M>([&](auto kc) {
            constexpr int k = decltype(kc)::value;
            constexpr int qb = left_turns(N, k), qc = left_turns(N, 2 * k), qd = left_turns(N, 3 * k);
            const cplx<float> a = {u[k].re.x, u[k].im.x};
            const cplx<float> b = twiddle<N, INV, k>(cplx<float>{u[k].re.y, u[k].im.y});
            const cplx<float> c = twiddle<N, INV, 2 * k>(cplx<float>{v[k].re.x, v[k].im.x});
            const cplx<float> d = twiddle<N, INV, 3 * k>(cplx<float>{v[k].re.y, v[k].im.y});
            if constexpr (qc == 0 && qd == qb) {
                // the first butterflies of (a, c) and (b, d) are alike: packed
                const cplx<float2> ab = {make_float2(a.re, b.re), make_float2(a.im, b.im)};
                const cplx<float2> cd = {make_float2(c.re, d.re), make_float2(c.im, d.im)};
                const cplx<float2> s = add_turned<INV, 0>(ab, cd), t = add_turned<INV, 2>(ab, cd);
                x[k] = add_turned<INV, qb>(cplx<float>{s.re.x, s.im.x}, cplx<float>{s.re.y, s.im.y});
                x[k + M] = add_turned<INV, qb + 1>(cplx<float>{t.re.x, t.im.x}, cplx<float>{t.re.y, t.im.y});
                x[k + 2 * M] = add_turned<INV, qb + 2>(cplx<float>{s.re.x, s.im.x}, cplx<float>{s.re.y, s.im.y});
                x[k + 3 * M] = add_turned<INV, qb + 3>(cplx<float>{t.re.x, t.im.x}, cplx<float>{t.re.y, t.im.y});
            } else {
                combine4<INV, qb, qc, qd>(a, b, c, d, x[k], x[k + M], x[k + 2 * M], x[k + 3 * M]);
            }
        });
    }
}

}  // namespace piv
