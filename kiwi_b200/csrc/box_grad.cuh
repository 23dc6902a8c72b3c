// Derivatives of the box masses (box_math.cuh): dT/dx is the kernel's integral over the box's face at x, from the
// same root, logarithms and angles as T itself, so a point's value and three derivatives cost about a third
// more than its value.  (Forward-mode dual numbers through the same formulas cost four times the value, and
// four times its registers.)
//
// Records, in units of the support radius, k = piece 0 .. NP-1; a plane's:
//   [0] u   [1] 1 / |u|   then NP entries each of   a_k, a'_k, W_{k+1}, W'_{k+1}, f_k, h_k, f'_k, h'_k
// an edge line's, at distances p, q:
//   [3 k + 0..2]          pq Q_k,   q R_k(p^2, q^2)  (of d/dp),   p R_k(q^2, p^2)  (of d/dq)
//   [3 NP + 3 k + 0..2]   K_k and the constants of d/dp and d/dq,   k = 0 .. NP
#pragma once

#include "box_math.cuh"

namespace kiwi_b200 {

KIWI_HD constexpr int box_grad_plane_stride(int n) { return 2 + 8 * n; }
KIWI_HD constexpr int box_grad_edge_stride(int n) { return 6 * n + 3; }
// offsets in a plane record
KIWI_HD constexpr int bg_a(int, int k) { return 2 + k; }
KIWI_HD constexpr int bg_da(int n, int k) { return 2 + n + k; }
KIWI_HD constexpr int bg_w(int n, int k) { return 1 + 2 * n + k; }   // k = 1 .. NP
KIWI_HD constexpr int bg_dw(int n, int k) { return 1 + 3 * n + k; }  // k = 1 .. NP
KIWI_HD constexpr int bg_f(int n, int k) { return 2 + 4 * n + k; }
KIWI_HD constexpr int bg_h(int n, int k) { return 2 + 5 * n + k; }
KIWI_HD constexpr int bg_df(int n, int k) { return 2 + 6 * n + k; }
KIWI_HD constexpr int bg_dh(int n, int k) { return 2 + 7 * n + k; }

// Horner's rule and the derivative with respect to x.
KIWI_HD double box_horner_d(const double* c, int n, double x, double& dv) {
    double s = c[n], d = 0.0;
#ifdef __CUDACC__
#pragma unroll
#endif
    for (int i = n - 1; i >= 0; --i) {
        d = fma(d, x, s);
        s = fma(s, x, c[i]);
    }
    dv = d;
    return s;
}

// sum_{i=0..D} X^i (polynomial of degree D - i in P), coefficient order of the tables' R and A with total degree
// `full` in the table.
KIWI_HD double box_xp(const double* c, int full, int D, double X, double P) {
    double s = 0.0;
#ifdef __CUDACC__
#pragma unroll
#endif
    for (int i = D; i >= 0; --i) s = fma(s, X, box_horner(c + i * (full + 1) - i * (i - 1) / 2, D - i, P));
    return s;
}

// The record of the plane at signed offset u.  T is odd in u: on a plane through the particle it is 0, and so are its
// derivatives along the plane, but not the one across it, whose terms tend to their values at u = 0.  Such a plane's record is
// that of the smallest offset, by which bg_on tells it.
KIWI_HD bool bg_on(double u) { return fabs(u) <= kBoxTiny; }
template <int NP, int DEG>
KIWI_HD void box_grad_plane(const KiwiBoxTable& T, double u, double* rec) {
    const int n = NP ? NP : T.npiece;
    const BoxDegree<DEG> d{T.deg};
    const bool on = fabs(u) < kBoxTiny;
    const double p = on ? kBoxTiny : fabs(u), p2 = p * p;
    rec[0] = on ? kBoxTiny : u;
    rec[1] = 1.0 / p;
    double w = 0.0, dw = 0.0;
#ifdef __CUDACC__
#pragma unroll
#endif
    for (int k = 0; k < n; ++k) {
        const KiwiBoxScale& s = T.scale[k];
        const double v = s.b - p;
        double f = 0.0, h = 0.0, df = 0.0, dh = 0.0, t, dt;
        if (v > 0.4 * s.b) {
            t = box_horner_d(s.fp, d.even() + 1, p2, dt);  // f = p t(p^2)
            f = p * t;
            df = fma(2.0 * p2, dt, t);
            t = box_horner_d(s.ap, d.odd(), p2, dt);       // a = p^4 t(p^2)
            h = s.m + fma(p2 * p2, t, -f);
            dh = fma((p * p2) * 2.0, fma(p2, dt, 2.0 * t), -df);
        } else if (v > 0.0) {
            f = box_horner_d(s.f, 2 * d.even() + 3, v, dt);
            df = -dt;
            h = box_horner_d(s.h, (DEG ? DEG : T.deg) + 3, v, dt);
            dh = -dt;
        }
        w = fma(-0.5 * kPi, h, w);
        dw = fma(-0.5 * kPi, dh, dw);
        t = box_horner_d(T.reg[k].a, d.odd(), p2, dt);
        rec[bg_a(n, k)] = (p2 * p2) * t;
        rec[bg_da(n, k)] = (p * p2) * 2.0 * fma(p2, dt, 2.0 * t);
        rec[bg_w(n, k + 1)] = w;
        rec[bg_dw(n, k + 1)] = dw;
        rec[bg_f(n, k)] = f;
        rec[bg_h(n, k)] = h;
        rec[bg_df(n, k)] = df;
        rec[bg_dh(n, k)] = dh;
    }
}

// The record of the edge line of the planes with records A, B, whose own piece is c.
template <int NP, int DEG>
KIWI_HD void box_grad_edge(const KiwiBoxTable& T, int c, const double* A, const double* B, double* rec) {
    const int n = NP ? NP : T.npiece;
    const int deg = DEG ? DEG : T.deg;
    const BoxDegree<DEG> d{T.deg};
    const double p = fabs(A[0]), q = fabs(B[0]), ip = A[1], iq = B[1];
    const double p2 = p * p, q2 = q * q;
    const double P = fma(p, p, q2), pq = p * q, S = pq * pq;
    const double lr = 0.5 * fm_log(P);
    double gs = 0.0, gp = 0.0, gq = 0.0;
    double Qn = pq * box_q(T.reg[c].Q, d.q(), P, S), Rn = q * box_xp(T.reg[c].R, 6, d.q(), p2, P),
           Sn = p * box_xp(T.reg[c].R, 6, d.q(), q2, P);
#ifdef __CUDACC__
#pragma unroll
#endif
    for (int k = 0; k < n; ++k) {
        if (k < c) continue;
        const double Qk = Qn, Rk = Rn, Sk = Sn;
        rec[3 * k] = Qk;
        rec[3 * k + 1] = Rk;
        rec[3 * k + 2] = Sk;
        rec[3 * (n + k)] = fma(-Qk, lr, gs);
        rec[3 * (n + k) + 1] = fma(-Rk, lr, gp);
        rec[3 * (n + k) + 2] = fma(-Sk, lr, gq);
        const bool more = k + 1 < n;
        Qn = more ? pq * box_q(T.reg[more ? k + 1 : 0].Q, d.q(), P, S) : 0.0;
        Rn = more ? q * box_xp(T.reg[more ? k + 1 : 0].R, 6, d.q(), p2, P) : 0.0;
        Sn = more ? p * box_xp(T.reg[more ? k + 1 : 0].R, 6, d.q(), q2, P) : 0.0;
        const KiwiBoxScale& s = T.scale[k];
        const double t2 = fma(s.b, s.b, -P);
        if (t2 > 0.0 && p < s.b && q < s.b) {
            const double it = fm_rsqrt(t2), t = t2 * it, ib = s.ib;
            const double anp = fm_atan_pos((p * ib) * (t * iq), (s.b * ip) * (q * it));
            const double anq = fm_atan_pos((q * ib) * (t * ip), (s.b * iq) * (p * it));
            const double dep = box_delta(t, t2, p, q, s.b), deq = box_delta(t, t2, q, p, s.b);
            const double L = fm_log(s.b + t) - lr;
            double g = pq * (t * box_g(s.G, deg / 2, P, S));
            g = fma(Qk - Qn, L, g);
            g = fma(-dep, A[bg_f(n, k)], g);
            g = fma(-deq, B[bg_f(n, k)], g);
            g = fma(anp, A[bg_h(n, k)], g);
            g = fma(anq, B[bg_h(n, k)], g);
            gs += g;
            double v = (q * t) * box_xp(s.A, 5, deg / 2, p2, P);
            v = fma(Rk - Rn, L, v);
            v = fma(-dep, A[bg_df(n, k)], v);
            gp += fma(anp, A[bg_dh(n, k)], v);
            v = (p * t) * box_xp(s.A, 5, deg / 2, q2, P);
            v = fma(Sk - Sn, L, v);
            v = fma(-deq, B[bg_df(n, k)], v);
            gq += fma(anq, B[bg_dh(n, k)], v);
        }
    }
    rec[6 * n] = gs;
    rec[6 * n + 1] = gp;
    rec[6 * n + 2] = gq;
}

// A piece's D as polynomials in X and S: the coefficients p(r) of X^i S^j (their order that of the tables' D).
constexpr int kBoxD = 84;
struct BoxD {
    double c[16];
};
KIWI_HD void box_d_coefs(const double* D, int deg, double s, BoxD& out) {
    // first coefficient of each X^i S^j in D, row by row in j
    constexpr int at[16] = {0, 13, 24, 33, 40, 45, 48, 49, 58, 65, 70, 73, 74, 79, 82, 83};
    constexpr int wt[16] = {0, 2, 4, 6, 8, 10, 12, 4, 6, 8, 10, 12, 8, 10, 12, 12};
#ifdef __CUDACC__
#pragma unroll
#endif
    for (int i = 0; i < 16; ++i) out.c[i] = wt[i] <= deg + 1 ? box_horner(D + at[i], deg + 1 - wt[i], s) : 0.0;
}
KIWI_HD double box_d(const BoxD& p, int deg, double X, double S) {
    double s = 0.0;
    if (deg >= 11) s = p.c[15] * S;
    if (deg >= 7) s = (s + fma(fma(p.c[14], X, p.c[13]), X, p.c[12])) * S;
    if (deg >= 3) s = (s + fma(fma(fma(fma(p.c[11], X, p.c[10]), X, p.c[9]), X, p.c[8]), X, p.c[7])) * S;
    return s + fma(fma(fma(fma(fma(fma(p.c[6], X, p.c[5]), X, p.c[4]), X, p.c[3]), X, p.c[2]), X, p.c[1]), X, p.c[0]);
}

// A point within the support: out = T and dT/d|x|, dT/d|y|, dT/d|z| (per H) without the walls' W, W' and the
// centre.  C, D, c0: the piece's tables; rx, ry, rz: its planes' records; ez, ey, ex: the records of the lines
// (x, y), (x, z), (y, z); n the number of pieces, k the point's.
template <int DEG>
KIWI_HD void box_inside_grad(const double* C, const double* D, double c0, int deg, int n, int k, const double* rx,
                             const double* ry, const double* rz, const double* ex, const double* ey, const double* ez,
                             double* out) {
    const int top = DEG ? DEG : deg;
    const double x = fabs(rx[0]), y = fabs(ry[0]), z = fabs(rz[0]);
    const double x2 = x * x, y2 = y * y, z2 = z * z;
    const double r2 = fma(x, x, fma(y, y, z2));
    const double ir = fm_rsqrt(r2);
    double r = r2 * ir;
    r = fma(0.5 * ir, fma(-r, r, r2), r);
    const double lx = fma(-x, ir, fm_log(r + x)), ly = fma(-y, ir, fm_log(r + y)), lz = fma(-z, ir, fm_log(r + z));
    // the two larger offsets' angles are at most pi/4
    const bool mx = x <= y && x <= z, my = !mx && y <= z;
    const double s0 = mx ? x : (my ? y : z), s1 = mx ? y : x, s2 = mx || my ? z : y;
    const double i1 = mx ? ry[1] : rx[1], i2 = mx || my ? rz[1] : ry[1];
    const double w = s0 * ir;
    const double A1 = fm_atan01((w * s2) * i1), A2 = fm_atan01((w * s1) * i2), A0 = 0.5 * kPi - (A1 + A2);
    const double Ax = mx ? A0 : A1, Ay = mx ? A1 : (my ? A0 : A2), Az = mx || my ? A2 : A0;
    double e2 = 0.0, e3 = 0.0;
    if (top >= 3) e2 = fma(x2, y2, (x2 + y2) * z2);
    if (top >= 5) e3 = (x2 * y2) * z2;
    const int q = 3 * k, m = 3 * (n + k);
    double t = (fma(ex[q], lx, ex[m]) + fma(ey[q], ly, ey[m])) + fma(ez[q], lz, ez[m]);
    t = fma(((x * y) * z) * ir, box_c(C, top, r - c0, e2, e3), t);
    t = fma(-rx[bg_a(n, k)], Ax, t);
    t = fma(-ry[bg_a(n, k)], Ay, t);
    out[0] = fma(-rz[bg_a(n, k)], Az, t);
    BoxD p;
    box_d_coefs(D, top, r - c0, p);
    // a line's [1] entries are of its first plane's axis, its [2] entries of its second's
    t = fma(ez[q + 1], lz, ez[m + 1]) + fma(ey[q + 1], ly, ey[m + 1]);
    t = fma((y * z) * ir, box_d(p, top, x2, y2 * z2), t);
    out[1] = fma(-rx[bg_da(n, k)], Ax, t);
    t = fma(ez[q + 2], lz, ez[m + 2]) + fma(ex[q + 1], lx, ex[m + 1]);
    t = fma((x * z) * ir, box_d(p, top, y2, x2 * z2), t);
    out[2] = fma(-ry[bg_da(n, k)], Ay, t);
    t = fma(ey[q + 2], ly, ey[m + 2]) + fma(ex[q + 2], lx, ex[m + 2]);
    t = fma((x * y) * ir, box_d(p, top, z2, x2 * y2), t);
    out[3] = fma(-rz[bg_da(n, k)], Az, t);
}

}  // namespace kiwi_b200
