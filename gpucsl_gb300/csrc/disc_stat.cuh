// P-values of the chi-squared tests, shared by the discrete test kernels (discrete.cu,
// disc_bits.cu).
#pragma once

#include "common.cuh"

namespace gcsl {

// ---------------------------------------------------------------- p-value
// Ibbetson (CACM Alg. 209) normal tail as coded by Perlman; the polynomial
// coefficients are those of the published algorithm.
__device__ inline double poz_dev(double z) {
    double x;
    if (z == 0.0) {
        x = 0.0;
    } else {
        double y = 0.5 * fabs(z);
        if (y >= 3.0) {
            x = 1.0;
        } else if (y < 1.0) {
            const double w = y * y;
            double t = 0.000124818987;
            t = __dadd_rn(__dmul_rn(t, w), -0.001075204047);
            t = __dadd_rn(__dmul_rn(t, w), 0.005198775019);
            t = __dadd_rn(__dmul_rn(t, w), -0.019198292004);
            t = __dadd_rn(__dmul_rn(t, w), 0.059054035642);
            t = __dadd_rn(__dmul_rn(t, w), -0.151968751364);
            t = __dadd_rn(__dmul_rn(t, w), 0.319152932694);
            t = __dadd_rn(__dmul_rn(t, w), -0.531923007300);
            t = __dadd_rn(__dmul_rn(t, w), 0.797884560593);
            x = __dmul_rn(__dmul_rn(t, y), 2.0);
        } else {
            y -= 2.0;
            double t = -0.000045255659;
            t = __dadd_rn(__dmul_rn(t, y), 0.000152529290);
            t = __dadd_rn(__dmul_rn(t, y), -0.000019538132);
            t = __dadd_rn(__dmul_rn(t, y), -0.000676904986);
            t = __dadd_rn(__dmul_rn(t, y), 0.001390604284);
            t = __dadd_rn(__dmul_rn(t, y), -0.000794620820);
            t = __dadd_rn(__dmul_rn(t, y), -0.002034254874);
            t = __dadd_rn(__dmul_rn(t, y), 0.006549791214);
            t = __dadd_rn(__dmul_rn(t, y), -0.010557625006);
            t = __dadd_rn(__dmul_rn(t, y), 0.011630447319);
            t = __dadd_rn(__dmul_rn(t, y), -0.009279453341);
            t = __dadd_rn(__dmul_rn(t, y), 0.005353579108);
            t = __dadd_rn(__dmul_rn(t, y), -0.002141268741);
            t = __dadd_rn(__dmul_rn(t, y), 0.000535310849);
            x = __dadd_rn(__dmul_rn(t, y), 0.999936657524);
        }
    }
    return z > 0.0 ? ((x + 1.0) * 0.5) : ((1.0 - x) * 0.5);
}

__device__ __forceinline__ double ex_dev(double x) { return (x < -20.0) ? 0.0 : exp(x); }

// Upper tail of chi^2 (Hill & Pike, CACM Alg. 299, with the 1985 rounding remark, in
// Perlman's formulation): the finite series of the even / odd df cases.
__device__ inline double pchisq_dev(double x, long long df) {
    if (x <= 0.0 || df < 1) return 1.0;
    const double a = 0.5 * x;
    const bool even = (df & 1) == 0;
    const double y = (df > 1) ? ex_dev(-a) : 0.0;
    double s = even ? y : 2.0 * poz_dev(-sqrt(x));
    if (df <= 2) return s;
    const double half = 0.5 * ((double)df - 1.0);
    double z = even ? 1.0 : 0.5;
    if (a > 20.0) {
        double e = even ? 0.0 : 0.5723649429247000870717135;
        const double c = log(a);
        while (z <= half) {
            e = __dadd_rn(log(z), e);
            s = __dadd_rn(s, ex_dev(__dsub_rn(__dsub_rn(__dmul_rn(c, z), a), e)));
            z += 1.0;
        }
        return s;
    }
    double e = even ? 1.0 : 0.5641895835477562869480795 / sqrt(a);
    double c = 0.0;
    while (z <= half) {
        e = __dmul_rn(e, a / z);
        c = __dadd_rn(c, e);
        z += 1.0;
    }
    return __dadd_rn(__dmul_rn(c, y), s);
}

// Tables of ln Gamma(z + 1), the running sum of log z of the series above, for its two
// rows z = 1, 2, .. (even df) and z = 1/2, 3/2, .. (odd df): LG_TERMS entries each, built
// once per solve.  A term beyond the table calls lgamma.
constexpr int LG_TERMS = 512;
constexpr int LG_BLOCKS = 2 * LG_TERMS / 256;

// Entries [256 b, 256 (b + 1)) of the two tables by one 256-thread block.
__device__ __forceinline__ void lgam_build(double *__restrict__ lg, int b) {
    const int k = b * 256 + threadIdx.x;
    if (k < 2 * LG_TERMS) lg[k] = lgamma(k < LG_TERMS ? k + 2.0 : (k - LG_TERMS) + 1.5);
}

__device__ __forceinline__ double lgam_term(const double *__restrict__ lg, bool even, long long k) {
    if (k < LG_TERMS) return __ldg(lg + (even ? k : LG_TERMS + k));
    return lgamma((even ? 2.0 : 1.5) + (double)k);
}

// pchisq_dev with the logarithms of its a > 20 series taken from the tables.  Terms whose
// exponent is below -20 are zero there, and the exponent c z - a - ln Gamma(z + 1) rises
// with z up to z = a: the terms are taken from the last one down and the loop ends at the
// first zero term below a.  In the other series a term too small to change the sum ends
// the loop (every later one is smaller).
__device__ inline double pchisq_tab(double x, long long df, const double *__restrict__ lg) {
    if (x <= 0.0 || df < 1) return 1.0;
    const double a = 0.5 * x;
    const bool even = (df & 1) == 0;
    const double y = (df > 1) ? ex_dev(-a) : 0.0;
    double s = even ? y : 2.0 * poz_dev(-sqrt(x));
    if (df <= 2) return s;
    const double z0 = even ? 1.0 : 0.5;
    const long long K = (df - 1) / 2;  // z = z0, z0 + 1, .. <= (df - 1) / 2
    if (a > 20.0) {
        const double c = log(a);
        for (long long k = K - 1; k >= 0; --k) {
            const double z = z0 + (double)k;
            const double t = c * z - a - lgam_term(lg, even, k);
            if (t >= -20.0) s += exp(t);
            else if (z < a) break;
        }
        return s;
    }
    double e = even ? 1.0 : 0.5641895835477562869480795 / sqrt(a);
    double c = 0.0;
    for (long long k = 0; k < K; ++k) {
        const double z = z0 + (double)k;
        e *= a / z;
        const double c1 = c + e;
        if (c1 == c && z > a) break;
        c = c1;
    }
    return c * y + s;
}

// The same by the 32 lanes of one warp (the terms of the long series of large tables in
// parallel).  All lanes call it; every lane returns the value.
__device__ inline double pchisq_tab_warp(double x, long long df, const double *__restrict__ lg) {
    const int lane = threadIdx.x & 31;
    if (x <= 0.0 || df < 1) return 1.0;
    const double a = 0.5 * x;
    const bool even = (df & 1) == 0;
    const double y = (df > 1) ? ex_dev(-a) : 0.0;
    double s = even ? y : 2.0 * poz_dev(-sqrt(x));
    if (df <= 2) return s;
    const double z0 = even ? 1.0 : 0.5;
    const long long K = (df - 1) / 2;
    if (a > 20.0) {
        const double c = log(a);
        double part = 0.0;
        for (long long k0 = (K - 1) / 32 * 32; k0 >= 0; k0 -= 32) {  // blocks of 32 terms, the last first
            const long long k = k0 + lane;
            const double z = z0 + (double)k;
            double t = -1.0e300;
            if (k < K) t = c * z - a - lgam_term(lg, even, k);
            if (t >= -20.0) part += exp(t);
            // every term of the block zero and all of it on the rising side: so are the rest
            if (!__any_sync(GCSL_FULL_MASK, t >= -20.0) && z0 + (double)k0 < a) break;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(GCSL_FULL_MASK, part, o);
        return s + part;
    }
    double e = even ? 1.0 : 0.5641895835477562869480795 / sqrt(a);
    double c = 0.0;
    for (long long k = 0; k < K; ++k) {
        const double z = z0 + (double)k;
        e *= a / z;
        const double c1 = c + e;
        if (c1 == c && z > a) break;
        c = c1;
    }
    return c * y + s;
}

// The p-value jumps where the published formulation changes branch: at chi^2 = 4 and 36 (pieces
// of the normal tail) and 40 (the two series, their first term).  chi^2 of few samples is a small
// fraction and may lie on a jump exactly, or the p-value on alpha; the last bit would then decide.
// Such a test is evaluated once more in the published order (chi^2 cell by cell, pchisq_dev), by
// one thread.  (A term's cut at exponent -20 is met by chance only: the exponent has a logarithm.)
//
// On it: the 32 bits of two doubles from the fifth-last exponent bit on differ by at most one, a
// window of at least 2^-28 relative, above the difference of the two evaluations (below 1e-9 up to
// 2^32 samples) and met by chance once in millions of tests.
__device__ __forceinline__ unsigned tie_bits(double x) {
    return __funnelshift_l((unsigned)__double2loint(x), (unsigned)__double2hiint(x), 8);
}
__device__ __forceinline__ bool pvalue_tie(double chi2, double pv, double alpha) {
    const unsigned k = tie_bits(chi2);  // 4, 36, 40: from one step below
    return (k - 0x0fffffffu <= 1u) | (k - 0x41ffffffu <= 1u) | (k - 0x43ffffffu <= 1u) |
           (tie_bits(pv) - tie_bits(alpha) + 1u <= 2u);
}

// A cell's term of a lower bound of chi^2 in FP32: e = N_a N_b / N_s and d = N - e carry
// relative errors of a few 2^-24 of N + e, taken off |d|.  The error of a sum of these terms
// and of its quotients is far inside a factor 0.999, which the caller applies.
__device__ __forceinline__ float chi2_floor_term(float o, float e) {
    const float d = fmaxf(fabsf(o - e) - 1e-6f * (o + e), 0.f);
    return __fdividef(d * d, e);
}

// True when the p-value of any chi^2 >= x with df degrees of freedom is exactly zero: past
// x = 40 the first terms of the series are cut off (exp(-x / 2) below exp(-20), the normal
// tail from sqrt(x) >= 6), and the largest term, the one at z = (df - 1) / 2 below a = x / 2,
// is at most exp(z ln(a / z) - a + z - ln(2 pi z) / 2) by Stirling's lower bound of Gamma;
// it falls as a grows.  One unit of margin covers the rounding (a relative 1e-6 of a + z).
__device__ __forceinline__ bool pvalue_zero(float x, int df) {
    if (!(x > 42.f)) return false;
    if (df <= 2) return true;
    const float a = 0.5f * x, z = 0.5f * (float)(df - 1);
    if (!(a > z + 1.f)) return false;
    const float g = z * logf(a / z) - a + z - 0.5f * logf(6.2831853f * z);
    return g + 2e-6f * (a + z) < -21.f;
}

}  // namespace gcsl
