// Box masses: the kernel mass T(x, y, z) of the box spanned by a particle and a lattice point at offsets
// x, y, z > 0, from per-plane and per-edge-line records shared by every point on that plane or line.  A cell
// of a Cartesian grid is the alternating sum of its eight corners' T (their signs are the offsets').  The
// reference forms the same number as 6 faces x 4 edges x 2 vertex pyramids with a series per pyramid
// (src/cartesian_grid.cpp:246-259, src/kernel_integral.cpp:356-400, src/kernel_integral_generic.cpp:119-221);
// here the kernel's polynomial pieces are integrated over the box directly (the formulas and their derivation
// stand in tables/gen_box_tables.py), so a point needs one root, three logarithms and two arctangents for any of
// the six kernels, no reciprocal beyond its planes', and a point beyond the support nothing but its
// records' constants.
//
// Lengths are in units of the support radius H.  A plane at signed offset u has the record
//   [0] u   [1] 1 / |u|   [2 + k] a_k   [2 + NP + k] W_{k+1}   [2 + 2 NP + k] f_k   [2 + 3 NP + k] h_k
// (k = 0 .. NP-1, at |u|; W_k = -(pi/2) sum_{s<k} h_s is the wall's part of a point in piece k, NP being "beyond
// the support"), and an edge line at distances p, q from the particle (in its two planes) has
//   [k] pq Q_k(p, q)   [NP + k] K_k,  k = 0 .. NP-1,   [2 NP] K_NP
// with K_k = -pq Q_k ln sqrt(p^2 + q^2) + sum_{s<k} g_s; entries k below the line's own piece are never
// read (a point on the line is at least as far) and not written.
#pragma once

#include "fastmath.cuh"

namespace kiwi_b200 {

// The tables' kernels with their pieces and largest power: the gathers are compiled for each, so that the records'
// strides and the polynomials' lengths are constants (100 k particles on 128^3, Wendland C4: 19.9 ms with them
// read from the table, 8.7 ms so; 9 k column, quintic: 14.2 and 4.6 ms).
#define KIWI_BOX_OTHERS(X) X(1, 3, 4) X(2, 3, 5) X(3, 1, 5) X(4, 1, 8) X(5, 1, 11)
#define KIWI_BOX_KERNELS(X) X(0, 2, 3) KIWI_BOX_OTHERS(X)

// Offsets below this fraction of H count as zero: the box's mass is below 1e-100 there, and its reciprocals stay
// finite.
constexpr double kBoxTiny = 1e-100;

// Record strides in doubles for n pieces (eight consecutive records start on different banks).
KIWI_HD constexpr int box_plane_stride(int n) { return 2 + 4 * n; }
KIWI_HD constexpr int box_edge_stride(int n) { return 2 * n + 1; }

// Horner's rule over c[0 .. n].
KIWI_HD double box_horner(const double* c, int n, double x) {
    double s = c[n];
#ifdef __CUDACC__
#pragma unroll
#endif
    for (int i = n - 1; i >= 0; --i) s = fma(s, x, c[i]);
    return s;
}

// C(r, e2, e3) of a kernel with powers up to deg, s = r - c (coefficient order of the tables' C).
constexpr int kBoxC = 39;
KIWI_HD double box_c(const double* c, int deg, double s, double e2, double e3) {
    double v = box_horner(c, deg + 1, s);
    if (deg >= 3) {
        double t = box_horner(c + 13, deg - 3, s);
        if (deg >= 7) {
            double u = box_horner(c + 22, deg - 7, s);
            if (deg >= 11) u = fma(c[37], e2, u);
            t = fma(u, e2, t);
        }
        v = fma(t, e2, v);
    }
    if (deg >= 5) {
        double t = box_horner(c + 27, deg - 5, s);
        if (deg >= 9) t = fma(box_horner(c + 34, deg - 9, s), e2, t);
        if (deg >= 11) t = fma(c[38], e3, t);
        v = fma(t, e3, v);
    }
    return v;
}

// Q(P, S), weighted degree D >= 1 (coefficient order of the tables' Q).
KIWI_HD double box_q(const double* c, int D, double P, double S) {
    double s = P * box_horner(c, D - 1, P);
    if (D >= 2) {
        double t = box_horner(c + 6, D - 2, P);
        if (D >= 4) {
            double u = box_horner(c + 11, D - 4, P);
            if (D >= 6) u = fma(c[14], S, u);
            t = fma(u, S, t);
        }
        s = fma(t, S, s);
    }
    return s;
}

// G(P, S), weighted degree D (coefficient order of the tables' G).
KIWI_HD double box_g(const double* c, int D, double P, double S) {
    double s = box_horner(c, D, P);
    if (D >= 2) {
        double t = box_horner(c + 6, D - 2, P);
        if (D >= 4) t = fma(box_horner(c + 10, D - 4, P), S, t);
        s = fma(t, S, s);
    }
    return s;
}

// Degrees of a kernel whose pieces have powers up to deg (DEG > 0: known when compiling).
template <int DEG>
struct BoxDegree {
    int deg;
    KIWI_HD int even() const { return (DEG ? DEG : deg) / 2; }             // fp's terms past p c1
    KIWI_HD int odd() const { return ((DEG ? DEG : deg) - 1) / 2; }        // a has odd() + 1 terms
    KIWI_HD int q() const { return ((DEG ? DEG : deg) + 1) / 2; }          // of Q
};

// The record of the plane at signed offset u (in units of H); |u| >= kBoxTiny, else the record's u is 0 and
// the rest is not formed.  Returns through w.
template <int NP, int DEG>
KIWI_HD void box_plane(const KiwiBoxTable& T, double u, double* rec) {
    const int n = NP ? NP : T.npiece;
    const BoxDegree<DEG> d{T.deg};
    const double p = fabs(u), p2 = p * p;
    if (p < kBoxTiny) {
        rec[0] = 0.0;
        return;
    }
    rec[0] = u;
    rec[1] = 1.0 / p;
    double w = 0.0;
#ifdef __CUDACC__
#pragma unroll
#endif
    for (int k = 0; k < n; ++k) {
        const KiwiBoxScale& s = T.scale[k];
        const double v = s.b - p;
        double f = 0.0, h = 0.0;
        if (v > 0.4 * s.b) {
            f = p * box_horner(s.fp, d.even() + 1, p2);
            h = s.m + fma(p2 * p2, box_horner(s.ap, d.odd(), p2), -f);
        } else if (v > 0.0) {
            f = box_horner(s.f, 2 * d.even() + 3, v);
            h = box_horner(s.h, (DEG ? DEG : T.deg) + 3, v);
        }
        w = fma(-0.5 * kPi, h, w);
        rec[2 + k] = (p2 * p2) * box_horner(T.reg[k].a, d.odd(), p2);
        rec[2 + n + k] = w;
        rec[2 + 2 * n + k] = f;
        rec[2 + 3 * n + k] = h;
    }
}

// The octant's mass (pi/2) sum_{s<k} m_s: the constant of a point in piece k (k = NP: beyond the support).
template <int NP>
KIWI_HD double box_centre(const KiwiBoxTable& T, int k) {
    double c = 0.0;
    const int n = NP ? NP : T.npiece;
#ifdef __CUDACC__
#pragma unroll
#endif
    for (int s = 0; s < n; ++s)
        if (s < k) c += 0.5 * kPi * T.scale[s].m;
    return c;
}

// phi - ang of a wall at p with the line at q and the leg t on the sphere of radius b > p: the difference of the two
// arctangents as one, tan = t q (b - p) / (q^2 b + p t^2).
KIWI_HD double box_delta(double t, double t2, double p, double q, double b) {
    const double num = t * (q * (b - p)), den = fma(q * q, b, p * t2);
    const bool lo = num <= den;
    const double a = fm_atan01((lo ? num : den) * fm_rcp(lo ? den : num));
    return lo ? a : 0.5 * kPi - a;
}

// The record of the edge line of the planes with records A, B (offsets p, q), whose own piece is c: P = p^2 + q^2
// lies in [scale[c-1].b^2, scale[c].b^2).
template <int NP, int DEG>
KIWI_HD void box_edge(const KiwiBoxTable& T, int c, const double* A, const double* B, double* rec) {
    const int n = NP ? NP : T.npiece;
    const BoxDegree<DEG> d{T.deg};
    const double p = fabs(A[0]), q = fabs(B[0]), ip = A[1], iq = B[1];
    const double P = fma(p, p, q * q), pq = p * q, S = pq * pq;
    const double lr = 0.5 * fm_log(P);  // ln of the line's distance (P >= kBoxTiny^2: normal)
    double gsum = 0.0, Qn = pq * box_q(T.reg[c].Q, d.q(), P, S);
#ifdef __CUDACC__
#pragma unroll
#endif
    for (int k = 0; k < n; ++k) {
        if (k < c) continue;
        const double Qk = Qn;
        rec[k] = Qk;
        Qn = k + 1 < n ? pq * box_q(T.reg[k + 1].Q, d.q(), P, S) : 0.0;
        rec[n + k] = fma(-Qk, lr, gsum);
        const KiwiBoxScale& s = T.scale[k];
        const double t2 = fma(s.b, s.b, -P);
        if (t2 > 0.0 && p < s.b && q < s.b) {
            const double it = fm_rsqrt(t2), t = t2 * it, ib = s.ib;
            const double anp = fm_atan_pos((p * ib) * (t * iq), (s.b * ip) * (q * it));
            const double anq = fm_atan_pos((q * ib) * (t * ip), (s.b * iq) * (p * it));
            double g = pq * (t * box_g(s.G, (DEG ? DEG : T.deg) / 2, P, S));
            g = fma(Qk - Qn, fm_log(s.b + t) - lr, g);
            g = fma(-box_delta(t, t2, p, q, s.b), A[2 + 2 * n + k], g);
            g = fma(-box_delta(t, t2, q, p, s.b), B[2 + 2 * n + k], g);
            g = fma(anp, A[2 + 3 * n + k], g);
            g = fma(anq, B[2 + 3 * n + k], g);
            gsum += g;
        }
    }
    rec[2 * n] = gsum;
}

// T without the walls' W and the centre: offsets x, y, z > 0, r2 = x^2 + y^2 + z^2; C the table of the point's
// piece and c0 its centre; the lines' pq Q and K of that piece (qz, kz the line at (x, y), along z, and so
// on); for the angles, the smallest offset s0 with its a, and the other two with their reciprocals and a.
template <int DEG>
KIWI_HD double box_inside(const double* C, double c0, int deg, double x, double y, double z, double r2, double qx,
                          double kx, double qy, double ky, double qz, double kz, double s0, double a0, double s1,
                          double i1, double a1, double s2, double i2, double a2) {
    const double ir = fm_rsqrt(r2);
    double r = r2 * ir;
    r = fma(0.5 * ir, fma(-r, r, r2), r);
    const int top = DEG ? DEG : deg;
    double e2 = 0.0, e3 = 0.0;
    if (top >= 3) {
        const double x2 = x * x, y2 = y * y, z2 = z * z;
        e2 = fma(x2, y2, (x2 + y2) * z2);
        if (top >= 5) e3 = (x2 * y2) * z2;
    }
    const double c = box_c(C, top, r - c0, e2, e3);
    // A_1 and A_2 are at most pi/4 each; A_0 = pi/2 - A_1 - A_2
    const double w = s0 * ir;
    const double A1 = fm_atan01((w * s2) * i1), A2 = fm_atan01((w * s1) * i2);
    const double lx = fma(-x, ir, fm_log(r + x)), ly = fma(-y, ir, fm_log(r + y)), lz = fma(-z, ir, fm_log(r + z));
    double t = (fma(qx, lx, kx) + fma(qy, ly, ky)) + fma(qz, lz, kz);
    t = fma(((x * y) * z) * ir, c, t);
    double v = -0.5 * kPi * a0;
    v = fma(-(a1 - a0), A1, v);
    v = fma(-(a2 - a0), A2, v);
    return t + v;
}

}  // namespace kiwi_b200
