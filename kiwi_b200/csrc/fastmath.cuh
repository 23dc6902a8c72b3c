// The transcendental functions of the box-mass form (box_math.cuh), branch-free so that a thread's calls
// interleave and a warp never splits over a call's cases.  Errors are absolute ones at rounding level (the box
// masses are sums of terms of order one): arctangent of [0, 1] by one polynomial in x^2, logarithm by a table of
// reciprocals and a short polynomial.  The polynomials interpolate at
// Chebyshev points (tables/gen_box_tables.py).  The product-sums of these functions are explicit fmas.  Their callers
// are not free of contraction (a sum that takes a function's last product, a difference of products), so the bodies of
// one kernel could differ in the last place with how they are compiled; that every entry point gives the same bits is
// tested for each kernel (tests/test_gpu_entry_points.py).  Rounding those products on their own, so that it could not
// happen, cost 1 to 3 % (registers; 2 M particles on 256^3, cubic: 71.5 -> 73.7 ms).
#pragma once

#include <math.h>
#include <stdint.h>
#include <string.h>

#include "box_tables.h"
#include "kiwi_math.cuh"

namespace kiwi_b200 {

// a b, rounded on its own: a sum that takes it is not contracted into an fma.
KIWI_HD double fm_mul(double a, double b) {
#ifdef __CUDA_ARCH__
    return __dmul_rn(a, b);
#else
    return fma(a, b, -0.0);
#endif
}

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

#ifdef __CUDACC__
static __device__ const double fm_log_table[2 << KIWI_LOG_BITS] __attribute__((aligned(16))) = {KIWI_LOG_TABLE};
#endif

// log(v) for normal v > 0, to rounding in absolute terms: v = m 2^k, m in [sqrt(1/2), sqrt(2)), and m = (1 + f) / inv with
// the reciprocal of the middle of m's cell (64 cells), log v = k ln 2 - log inv + log(1 + f); f is exact to the last
// place and small, so that a polynomial of degree 6 and no division are left (reduction by a table as in P. T. P.
// Tang, "Table-driven implementation of the logarithm function", 1990).  In the cell that holds 1, inv = 1, so that
// the result keeps its relative accuracy there.  The table is 1 KB, in L1 for as long as a kernel uses it.
// Against 2 atanh(f / (2 + f)) over the whole of [sqrt(1/2), sqrt(2)), with its division: 9 k particles on
// 37 x 41 x 149, quintic spline, 3.22 -> 3.09 ms; 100 k on 128^3, Wendland C4, 8.5 -> 8.3 ms; cubic maps 1 %.
KIWI_HD double fm_log(double v) {
    constexpr double c[KIWI_N_LOG] = {KIWI_LOG_COEFS};
    constexpr double kLn2 = 0.69314718055994530942;
#ifdef __CUDA_ARCH__
    const int hi = __double2hiint(v), lo = __double2loint(v);
    const int at = hi - KIWI_LOG_HI0, k = at >> 20;
    const double2 cell = __ldg(reinterpret_cast<const double2*>(fm_log_table) + ((at >> (20 - KIWI_LOG_BITS)) & ((1 << KIWI_LOG_BITS) - 1)));
    const double inv = cell.x, L = cell.y;
    const double m = __hiloint2double(hi - (k << 20), lo);
    const double dk = __hiloint2double(0x43300000, k ^ (int)0x80000000) - 4503601774854144.0;  // (double)k
#else
    static const double table[2 << KIWI_LOG_BITS] = {KIWI_LOG_TABLE};
    int64_t bits;
    memcpy(&bits, &v, 8);
    const int at = (int)(bits >> 32) - KIWI_LOG_HI0, k = at >> 20;
    const int i = (at >> (20 - KIWI_LOG_BITS)) & ((1 << KIWI_LOG_BITS) - 1);
    const double inv = table[2 * i], L = table[2 * i + 1];
    bits -= (int64_t)k << 52;
    double m;
    memcpy(&m, &bits, 8);
    const double dk = (double)k;
#endif
    const double f = fma(m, inv, -1.0), f2 = f * f;
    static_assert(KIWI_N_LOG == 5, "the polynomial below");
    const double q = fma(fma(c[4], f2, c[2]), f2, fma(fma(c[3], f2, c[1]), f, c[0]));
    return fma(dk, kLn2, L + fma(f2, q, f));
}

}  // namespace kiwi_b200
