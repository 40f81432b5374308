// Counter-based random numbers for the fluctuated forward.
//
// Philox-4x32-10: J. K. Salmon, M. A. Moraes, R. O. Dror, D. E. Shaw,
// "Parallel random numbers: as easy as 1, 2, 3", SC'11.  Every draw is a pure
// function of (key, counter), so a kernel can regenerate the same variate in
// another pass, in any order, on any thread.
//
// Binomial variates (IRandom::binomial, iface/inc/WireCellIface/IRandom.h;
// gen/src/Random.cxx draws them with std::binomial_distribution):
//   * n * min(p, 1-p) < 10: inversion by sequential search from 0 using
//     f(x+1) = f(x) * (n - x) / (x + 1) * p / (1 - p);
//   * otherwise: transformed rejection with squeeze, algorithm BTRS of
//     W. Hormann, "The generation of binomial random variates", J. Statist.
//     Comput. Simul. 46 (1993) 101-110: accept k when
//     log(v * alpha / (a / us^2 + b)) <= log f(k) - log f(m), m the mode,
//     with log x! = (x + 1/2) log(x + 1) - (x + 1) + log(2 pi) / 2 + fc(x),
//     fc the Stirling correction (exact values below 10, the series
//     1/12 (x+1)^-1 - 1/360 (x+1)^-3 + 1/1260 (x+1)^-5 above).
// Both are exact samplers (up to floating-point rounding).
#pragma once

#include <cuda_runtime.h>
#include <cstdint>

namespace wctb200 {

// One block of Philox-4x32-10.
__device__ __forceinline__ uint4 philox_block(uint32_t k0, uint32_t k1, uint32_t x0, uint32_t x1, uint32_t x2,
                                              uint32_t x3)
{
#pragma unroll
    for (int r = 0; r < 10; ++r) {
        const uint32_t lo0 = 0xD2511F53u * x0, hi0 = __umulhi(0xD2511F53u, x0);
        const uint32_t lo1 = 0xCD9E8D57u * x2, hi1 = __umulhi(0xCD9E8D57u, x2);
        const uint32_t y0 = hi1 ^ x1 ^ k0, y2 = hi0 ^ x3 ^ k1;
        x0 = y0;
        x1 = lo1;
        x2 = y2;
        x3 = lo0;
        k0 += 0x9E3779B9u;
        k1 += 0xBB67AE85u;
    }
    return make_uint4(x0, x1, x2, x3);
}

// A 32-bit unsigned integer as a double: the low word of 2^52 + w (an addition,
// where a conversion has a quarter of its rate).
__device__ __forceinline__ double u32_double(uint32_t w)
{
    return __hiloint2double(0x43300000, (int)w) - 4503599627370496.0;
}

// Uniform double in (0, 1], 53 random bits: (x + 1/2) 2^-53. From x = 2^52 on
// the half rounds to an even number, so the largest x gives exactly 1. (Kept
// below 1 by three integer operations a word, the noise of a 2560 x 6000 frame
// takes 2 % longer; box_muller and the samplers take the 1 instead: BTRS finds
// its proposal out of range and draws again, inversion ends its search.)
__device__ __forceinline__ double uniform53(uint32_t hi, uint32_t lo)
{
    const double x = fma(u32_double(hi), 2097152.0, u32_double(lo >> 11));  // exact
    return (x + 0.5) * 1.1102230246251565404e-16;
}

// The uniforms of the stream (key0, key1) x (ctr0, ctr1, ctr2) in order, two a
// block; the fourth counter word numbers the blocks.
struct Philox {
    uint32_t k0, k1, c0, c1, c2, c3;
    uint32_t hi, lo;  // the block's second pair, while have is set
    bool have;

    __device__ __forceinline__ void init(uint32_t key0, uint32_t key1, uint32_t ctr0, uint32_t ctr1, uint32_t ctr2)
    {
        k0 = key0;
        k1 = key1;
        c0 = ctr0;
        c1 = ctr1;
        c2 = ctr2;
        c3 = 0;
        have = false;
    }

    __device__ __forceinline__ double uniform()
    {
        if (have) {
            have = false;
            return uniform53(hi, lo);
        }
        const uint4 o = philox_block(k0, k1, c0, c1, c2, c3++);
        hi = o.z;
        lo = o.w;
        have = true;
        return uniform53(o.x, o.y);
    }
};

// Box-Muller for u1, u2 in (0, 1], sqrt(-2 log u1) cos(2 pi u2), in double precision to about 1e-11
// and rounded to float.  The series are Taylor's, on the ranges that exact
// reductions leave: the logarithm as e log 2 + 2 atanh((m - 1) / (m + 1)) with m
// in [sqrt(1/2), sqrt(2)), sine and cosine within pi / 4 of a quarter turn; the
// root starts from the single-precision one and takes one Newton step.
// Integers become doubles by additions: conversions run at a quarter of their
// rate.  (The library's log, sincospi and sqrt, to the last bit of a double, took
// four times the operations: 248 us for the noise of a 2560 x 6000 frame, 15 M
// normals, with the generic transform; now 194 us: half the FP64 chains, a quarter each Philox
// and transform.)
__device__ __forceinline__ float box_muller(double u1, double u2)
{
    // u1 = m 2^e
    long long bits = __double_as_longlong(u1);
    int e = (int)(bits >> 52) - 1023;
    double m = __longlong_as_double((bits & 0x000fffffffffffffll) | 0x3ff0000000000000ll);
    if (m > 1.4142135623730951) {
        m *= 0.5;
        ++e;
    }
    // 1 / d on [1.7, 2.42]: a parabola good to 0.16 %, and two Newton steps
    const double d = m + 1.0;
    double r = fma(fma(0.1175, d, -0.7253), d, 1.4810);
    r = r * fma(-d, r, 2.0);
    r = r * fma(-d, r, 2.0);
    const double s = (m - 1.0) * r, s2 = s * s;
    double p = 1.0 / 13.0;
    p = fma(p, s2, 1.0 / 11.0);
    p = fma(p, s2, 1.0 / 9.0);
    p = fma(p, s2, 1.0 / 7.0);
    p = fma(p, s2, 1.0 / 5.0);
    p = fma(p, s2, 1.0 / 3.0);
    p = fma(p * s2, s, s);  // atanh s
    const double ed = __hiloint2double(0x43300000, e ^ 0x80000000) - 4503601774854144.0;  // e + 2^31 + 2^52
    const double x = -2.0 * fma(ed, 0.69314718055994531, 2.0 * p);
    double y = (double)rsqrtf(fmaxf((float)x, 1e-30f));  // u1 = 1: x = 0, and the normal is 0
    y = y * fma(-0.5 * x * y, y, 1.5);
    // 4 u2 = q + f, f in [-1/2, 1/2]
    const double v = 4.0 * u2, w = v + 6755399441055744.0;  // 1.5 2^52: rounds, the quarter in the low bits
    const double f = (v - (w - 6755399441055744.0)) * 1.5707963267948966, f2 = f * f;
    double c = 1.0 / 479001600.0, z = 1.0 / 6227020800.0;  // 12!, 13!
    c = fma(c, f2, -1.0 / 3628800.0);
    c = fma(c, f2, 1.0 / 40320.0);
    c = fma(c, f2, -1.0 / 720.0);
    c = fma(c, f2, 1.0 / 24.0);
    c = fma(c, f2, -0.5);
    c = fma(c, f2, 1.0);
    z = fma(z, f2, -1.0 / 39916800.0);
    z = fma(z, f2, 1.0 / 362880.0);
    z = fma(z, f2, -1.0 / 5040.0);
    z = fma(z, f2, 1.0 / 120.0);
    z = fma(z, f2, -1.0 / 6.0);
    z = fma(z * f2, f, f);
    const int turn = __double2loint(w) & 3;
    const double t = (turn & 1) ? z : c;
    return (float)(x * y * (turn == 1 || turn == 2 ? -t : t));
}

// Stirling correction fc(x) = log x! - [(x + 1/2) log(x + 1) - (x + 1) + log(2 pi)/2].
__device__ __forceinline__ double stirling_fc(int x)
{
    if (x < 10) {
        const double t[10] = {0.08106146679532733,  0.041340695955409457, 0.027677925684997717,
                              0.020790672103765839, 0.016644691189821259, 0.013876128823072875,
                              0.011896709945893313, 0.010411265261973668, 0.0092554621827094508,
                              0.0083305634333594725};
        return t[x];
    }
    const double r = 1.0 / ((double)x + 1.0), r2 = r * r;
    return r * (1.0 / 12.0 - r2 * (1.0 / 360.0 - r2 * (1.0 / 1260.0)));
}

// log x! up to the terms that cancel in the ratios below: (x + 1/2) log(x + 1) + fc(x).
__device__ __forceinline__ double logfact_part(int x)
{
    return ((double)x + 0.5) * log((double)x + 1.0) + stirling_fc(x);
}

// Binomial(n, p) for 0 <= p <= 1/2.
__device__ __forceinline__ int binomial_low(int n, double p, Philox& g)
{
    const double q = 1.0 - p;
    const double np = (double)n * p;
    if (np < 10.0) {
        const double s = p / q;
        const double f0 = exp((double)n * log1p(-p));  // q^n, >= exp(-10 * 1.39)
        for (int attempt = 0; attempt < 64; ++attempt) {
            double u = g.uniform();
            double f = f0;
            int x = 0;
            // at most n steps; the tail below one part in 2^53 ends the search
            while (u > f && x < n) {
                u -= f;
                f *= s * (double)(n - x) / (double)(x + 1);
                ++x;
                if (f < 1e-300) break;
            }
            if (u <= f || x == n) return x;
            // rounding left u above the remaining mass: draw again
        }
        return (int)floor(np);
    }
    // BTRS
    const double spq = sqrt(np * q);
    const double b = 1.15 + 2.53 * spq;
    const double a = -0.0873 + 0.0248 * b + 0.01 * p;
    const double c = np + 0.5;
    const double vr = 0.92 - 4.2 / b;
    const double alpha = (2.83 + 5.1 / b) * spq;
    const double lpq = log(p / q);
    const int m = (int)floor((double)(n + 1) * p);
    const double lfm = logfact_part(m) + logfact_part(n - m);
    for (int attempt = 0; attempt < 1000; ++attempt) {
        const double u = g.uniform() - 0.5;
        const double v = g.uniform();
        const double us = 0.5 - fabs(u);
        const int k = (int)floor((2.0 * a / us + b) * u + c);
        if (k < 0 || k > n) continue;
        if (us >= 0.07 && v <= vr) return k;  // squeeze
        const double lv = log(v * alpha / (a / (us * us) + b));
        // log f(k) - log f(m); the -(x+1) and log(2 pi)/2 terms of the four factorials cancel
        const double lratio = lfm - logfact_part(k) - logfact_part(n - k) + (double)(k - m) * lpq;
        if (lv <= lratio) return k;
    }
    return m;  // not reached in practice (acceptance probability per try is above 0.5)
}

// Binomial(n, p) in double precision throughout, drawing from the stream g.
static __device__ __noinline__ int binomial_double(int n, double p, Philox g)
{
    if (p <= 0.5) return binomial_low(n, p, g);
    return n - binomial_low(n, 1.0 - p, g);
}

// log x! correction of stirling_fc in single precision.
__device__ __forceinline__ float stirling_fcf(int x)
{
    if (x < 10) {
        const float t[10] = {0.08106147f,  0.04134070f,  0.02767793f,  0.02079067f,  0.01664469f,
                             0.01387613f,  0.01189671f,  0.01041127f,  0.009255462f, 0.008330563f};
        return t[x];
    }
    const float r = __fdividef(1.0f, (float)x + 1.0f), r2 = r * r;
    return r * (0.083333333f - r2 * (0.0027777778f - r2 * 0.00079365079f));
}

// The draws of binomial_low for 0 < p <= 1/2 with the transcendentals in
// single precision: the same uniforms, and every comparison that decides the
// draw is answered "in doubt" when its two sides are closer than a bound on the
// single-precision error; the caller then runs the double-precision draw.  So
// the result, where there is one, is the double-precision draw.
constexpr int kDrawDoubt = -1;    // take the double-precision draw
constexpr int kDrawReject = -2;   // BTRS: next attempt
constexpr int kDrawOpen = -3;     // BTRS: the squeeze did not decide

// Inversion, n p < 10.  The cumulated probabilities are below 1; each of at
// most about 30 terms is known to (|n log(1-p)| + 4 x) 3e-7 of itself and a
// sum of them to 1e-5 (margin 2e-5).
__device__ __forceinline__ int draw_inversion(int n, float p, float u)
{
    const float s = __fdividef(p, 1.0f - p);
    float f = expf((float)n * log1pf(-p));
    float c = f, left = (float)n;
    for (int x = 0;; ++x) {
        if (fabsf(u - c) < 2e-5f) return kDrawDoubt;
        if (u < c || x == n) return x;
        f *= s * __fdividef(left, (float)(x + 1));
        left -= 1.0f;
        c += f;
    }
}

// BTRS, n p >= 10: one attempt with the uniforms u (less one half) and v.  The
// proposal k = floor(y) needs y to 5e-7 of its distance from the mode; the
// acceptance ratio's logarithms are taken as log1p of (m - k) / (k + 1) and the
// like, differences that do not cancel, good to 3e-7 (|k - m| + 20).
template <bool SQUEEZE_ONLY>
__device__ __forceinline__ int draw_btrs(int n, double p, double u, float v)
{
    const double np = (double)n * p;
    const float pf = (float)p, qf = 1.0f - pf;
    const float spq = sqrtf((float)np * qf);
    const float b = 1.15f + 2.53f * spq;
    const float a = -0.0873f + 0.0248f * b + 0.01f * pf;
    const float ib = __fdividef(1.0f, b);
    const float us = (float)(0.5 - fabs(u));
    const double dy = (double)(__fdividef(2.0f * a, us) + b) * u;
    const double y = dy + (np + 0.5), yk = floor(y);
    const float frac = (float)(y - yk), tol = 2e-6f * (1.0f + fabsf((float)dy));
    if (frac < tol || frac > 1.0f - tol) return kDrawDoubt;
    if (!(yk >= 0.0 && yk <= (double)n)) return kDrawReject;
    const int k = (int)yk;
    if (fabsf(us - 0.07f) < 1e-6f) return kDrawDoubt;
    if (us > 0.07f) {
        const float vr = 0.92f - 4.2f * ib;
        if (fabsf(v - vr) < 1e-5f) return kDrawDoubt;
        if (v < vr) return k;
    }
    if (SQUEEZE_ONLY) return kDrawOpen;
    const int m = (int)floor((double)(n + 1) * p);
    const float alpha = (2.83f + 5.1f * ib) * spq;
    const float lv = logf(__fdividef(v * alpha, __fdividef(a, us * us) + b));
    const float dk = (float)(k - m), k1 = (float)k + 1.0f, nk1 = (float)(n - k) + 1.0f;
    const float lr = ((float)m + 0.5f) * log1pf(__fdividef(-dk, k1)) +
                     ((float)(n - m) + 0.5f) * log1pf(__fdividef(dk, nk1)) +
                     dk * logf(__fdividef(nk1, k1) * __fdividef(pf, qf)) + (stirling_fcf(m) - stirling_fcf(k)) +
                     (stirling_fcf(n - m) - stirling_fcf(n - k));
    if (!(fabsf(lv - lr) > 4e-5f + 3e-6f * fabsf(dk))) return kDrawDoubt;
    return lv < lr ? k : kDrawReject;
}

// binomial_low's draw from the stream g, or kDrawDoubt.
__device__ __forceinline__ int binomial_low_single(int n, double p, Philox& g)
{
    if ((double)n * p < 10.0) return draw_inversion(n, (float)p, (float)g.uniform());
    for (int attempt = 0; attempt < 8; ++attempt) {
        const double u = g.uniform() - 0.5;
        const float v = (float)g.uniform();
        const int k = draw_btrs<false>(n, p, u, v);
        if (k != kDrawReject) return k;
    }
    return kDrawDoubt;
}

// Binomial(n, p) from the stream g, just initialised; p >= 1 gives n
// (GaussianDiffusion.cxx:196-198), p <= 0 gives 0.
__device__ __forceinline__ int binomial(int n, double p, const Philox& g)
{
    if (n <= 0 || !(p > 0.0)) return 0;
    if (p >= 1.0) return n;
    int k = kDrawDoubt;
    if (p <= 0.5) {
        Philox h = g;
        k = binomial_low_single(n, p, h);
    }
    return k >= 0 ? k : binomial_double(n, p, g);
}

// Counter-stream tags (first counter word's top bits are the plane, the
// drift uses its own tag).
constexpr uint32_t kRngDriftTag = 0xFFFFu;
constexpr uint32_t kRngSampleTag = 0xFFFEu;  // bulk draws of the sampling entry point

}  // namespace wctb200
