// The transcendental functions of the box-mass form (box_math.cuh), branch-free so that a thread's calls
// interleave and a warp never splits over a call's cases.  Errors are absolute ones at rounding level (the box
// masses are sums of terms of order one): arctangent of [0, 1] by one polynomial in x^2, logarithm by the
// classical reduction to m in [sqrt(1/2), sqrt(2)) and 2 atanh((m - 1) / (m + 1)).  The polynomials interpolate at
// Chebyshev points (tables/gen_box_tables.py).  CUDA's own atan and log1p branch on their argument and carry
// a full-range reduction and a division each.  Every product-sum is an explicit fma, so that the values do
// not depend on how a caller is compiled.
#pragma once

#include <math.h>
#include <stdint.h>
#include <string.h>

#include "box_tables.h"
#include "kiwi_math.cuh"

namespace kiwi_b200 {

// 1 / d for normal d > 0, to rounding: the hardware's approximation y (at least 18 bits), then
// y (1 + e + e^2 + e^3) with e = 1 - d y.
KIWI_HD double fm_rcp(double d) {
#ifdef __CUDA_ARCH__
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
    const double e = fma(-d, y, 1.0);
    return fma(y, fma(fma(e, e, e), e, e), y);
#else
    return 1.0 / d;
#endif
}

// 1 / sqrt(a) for normal a > 0, to rounding: y (1 + e/2 + 3 e^2 / 8 + 5 e^3 / 16) with e = 1 - a y^2.
KIWI_HD double fm_rsqrt(double a) {
#ifdef __CUDA_ARCH__
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a));
    const double e = fma(-(a * y), y, 1.0);
    return fma(y, fma(fma(0.3125, e, 0.375), e, 0.5) * e, y);
#else
    return 1.0 / sqrt(a);
#endif
}

// atan(x), 0 <= x <= 1: x times two interleaved Horner chains in x^4.
KIWI_HD double fm_atan01(double x) {
    constexpr double c[KIWI_N_ATAN] = {KIWI_ATAN_COEFS};
    static_assert(KIWI_N_ATAN % 2 == 0, "paired coefficients");
    const double z = x * x, z2 = z * z;
    double e = c[KIWI_N_ATAN - 2], o = c[KIWI_N_ATAN - 1];
#ifdef __CUDACC__
#pragma unroll
#endif
    for (int k = KIWI_N_ATAN - 4; k >= 0; k -= 2) {
        e = fma(e, z2, c[k]);
        o = fma(o, z2, c[k + 1]);
    }
    return x * fma(o, z, e);
}

// atan(u) for u > 0 given with its reciprocal.
KIWI_HD double fm_atan_pos(double u, double iu) {
    const bool lo = u <= 1.0;
    const double a = fm_atan01(lo ? u : iu);
    return lo ? a : 0.5 * kPi - a;
}

// log(v) for normal v > 0, to rounding in absolute terms.
KIWI_HD double fm_log(double v) {
    constexpr double c[KIWI_N_LOG] = {KIWI_LOG_COEFS};
    constexpr double kLn2 = 0.69314718055994530942;
#ifdef __CUDA_ARCH__
    const int hi = __double2hiint(v), lo = __double2loint(v);
    // v = m 2^k, m in [sqrt(1/2), sqrt(2)): the exponent read off with the high word biased by sqrt(2)'s
    const int k = (hi - 0x3fe6a09e) >> 20;
    const double m = __hiloint2double(hi - (k << 20), lo);
    const double dk = __hiloint2double(0x43300000, k ^ (int)0x80000000) - 4503601774854144.0;  // (double)k
#else
    int64_t bits;
    memcpy(&bits, &v, 8);
    const int hi = (int)(bits >> 32);
    const int k = (hi - 0x3fe6a09e) >> 20;
    bits -= (int64_t)k << 52;
    double m;
    memcpy(&m, &bits, 8);
    const double dk = (double)k;
#endif
    // log(1 + f) = f - (f^2/2 - s (f^2/2 + s^2 R)), s = f / (2 + f): the leading term is exact (the arrangement
    // of fdlibm's log)
    const double f = m - 1.0, s = f * fm_rcp(m + 1.0);
    const double z = s * s, z2 = z * z, hf = 0.5 * f * f;
    double e = c[KIWI_N_LOG - 2], o = c[KIWI_N_LOG - 1];  // 2 (atanh(s)/s - 1) / z
    static_assert(KIWI_N_LOG % 2 == 1, "paired coefficients");
#ifdef __CUDACC__
#pragma unroll
#endif
    for (int j = KIWI_N_LOG - 4; j >= 1; j -= 2) {
        e = fma(e, z2, c[j]);
        o = fma(o, z2, c[j + 1]);
    }
    const double R = fma(o, z, e) * (z + z);
    return fma(dk, kLn2, f - fma(-s, hf + R, hf));
}

}  // namespace kiwi_b200
