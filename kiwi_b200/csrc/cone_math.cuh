// Face integrals of general polyhedral cells with the box masses' formulas: a face's integral is the sum over its
// edges of the kernel masses of the cones from the particle over the right triangles between the particle's foot
// point on the face's plane, the foot point's projection on the edge line and the edge's two vertices
// (face_integral_impl, src/kernel_integral.cpp:471-647), each cone from the polynomial moments of the kernel's
// pieces (tables/gen_box_tables.py) instead of a series per vertex.  A cone needs a root, a logarithm and one or
// two arctangents; the edge line's share of a cone that leaves a piece is formed once per edge, and only if the
// two cones' shares do not cancel.  Where the reference takes R_0 = r12 sqrt(1 - cos^2) and the angles' cosines,
// the distances here come from the cross and dot products (no cancellation near a vertex).
#pragma once

#include "box_grad.cuh"

namespace kiwi_b200 {

// V(r, X, P) of a kernel with powers up to deg, s = r - c (coefficient order of the cone tables' V).
KIWI_HD double cone_v(const double* c, int deg, double s, double X, double P) {
    // first coefficient of the groups i + j = d
    constexpr int first[7] = {0, 13, 35, 62, 90, 115, 133};
    const int dmax = (deg + 1) / 2;
    double v = 0.0;
#ifdef __CUDACC__
#pragma unroll
#endif
    for (int i = dmax; i >= 0; --i) {  // Horner in X over polynomials in P
        double q = 0.0;
#ifdef __CUDACC__
#pragma unroll
#endif
        for (int j = dmax - i; j >= 0; --j) {
            const int d = i + j, len = 13 - 2 * d;
            q = fma(q, P, box_horner(c + first[d] + i * len, deg + 1 - 2 * d, s));
        }
        v = fma(v, X, q);
    }
    return v;
}

// The functions of a face's plane: a_k, h_k, f_k at its distance r0 (in units of H).
template <int NP, int DEG>
struct ConeWall {
    double a[NP], h[NP], f[NP];
    KIWI_HD void set(const KiwiConeTable& T, double p) {
        const BoxDegree<DEG> d{DEG};
        const double p2 = p * p;
#ifdef __CUDACC__
#pragma unroll
#endif
        for (int k = 0; k < NP; ++k) {
            const KiwiConeScale& s = T.scale[k];
            const double v = s.b - p;
            f[k] = h[k] = 0.0;
            if (v > 0.4 * s.b) {
                f[k] = p * box_horner(s.fp, d.even() + 1, p2);
                h[k] = s.m + fma(p2 * p2, box_horner(s.ap, d.odd(), p2), -f[k]);
            } else if (v > 0.0) {
                f[k] = box_horner(s.f, 2 * d.even() + 3, v);
                h[k] = box_horner(s.h, DEG + 3, v);
            }
            a[k] = (p2 * p2) * box_horner(T.reg[k].a, d.odd(), p2);
        }
    }
};

// The normal of a face's plane from its first three vertices, u and w the second's and third's offsets from the first,
// with the roundings of face_integral_impl (src/kernel_integral.cpp:471-647): products rounded on their own, so that three vertices in
// a line give exactly 0 as there, and not what an fma leaves of a product.
struct FaceNormal {
    double x, y, z;
};
KIWI_HD FaceNormal face_normal(double ux, double uy, double uz, double wx, double wy, double wz) {
    return {fm_mul(uy, wz) - fm_mul(wy, uz), fm_mul(uz, wx) - fm_mul(wz, ux), fm_mul(ux, wy) - fm_mul(wx, uy)};
}

// The integral of a face with vertices V (nv of them, in order) for a particle at (x0, y0, z0), iH = 1 / H.  R: the
// table's pieces, where the caller keeps them (threads differ in piece).
template <int NP, int DEG, class Verts>
KIWI_HD double cone_face(const KiwiConeTable& T, const KiwiConeRegion* R, const Verts& V, int nv, double x0, double y0,
                         double z0, double iH) {
    if (nv < 3) return 0.0;
    const double x1 = V.x(0), y1 = V.y(0), z1 = V.z(0);
    const FaceNormal nrm = face_normal(V.x(1) - x1, V.y(1) - y1, V.z(1) - z1, V.x(2) - x1, V.y(2) - y1, V.z(2) - z1);
    const double n2 = fma(nrm.x, nrm.x, fma(nrm.y, nrm.y, fm_mul(nrm.z, nrm.z)));
    if (!(n2 > 0.0)) return 0.0;  // no plane: the reference's angles are undefined there and it adds nothing
    const double in = 1.0 / sqrt(n2), A = nrm.x * in, B = nrm.y * in, C = nrm.z * in;
    const double rs = fma(A, x0 - x1, fma(B, y0 - y1, C * (z0 - z1)));  // signed distance
    const double r0 = fabs(rs) * iH;
    if (!(r0 > kBoxTiny)) return 0.0;
    const double xp = fma(-rs, A, x0), yp = fma(-rs, B, y0), zp = fma(-rs, C, z0);  // the foot point
    ConeWall<NP, DEG> w;
    w.set(T, r0);
    const double X = r0 * r0;
    double total = 0.0;
    double ax = (V.x(0) - xp) * iH, ay = (V.y(0) - yp) * iH, az = (V.z(0) - zp) * iH;
    const double fx = ax, fy = ay, fz = az;
    for (int j = 0; j < nv; ++j) {
        const bool wrap = j == nv - 1;
        const double bx = wrap ? fx : (V.x(j + 1) - xp) * iH, by = wrap ? fy : (V.y(j + 1) - yp) * iH,
                     bz = wrap ? fz : (V.z(j + 1) - zp) * iH;
        const double ex = bx - ax, ey = by - ay, ez = bz - az;
        const double len2 = fma(ex, ex, fma(ey, ey, ez * ez));
        // twice the signed area of the triangle (foot, a, b) about the normal
        const double side = fma(A, fma(ay, bz, -(az * by)), fma(B, fma(az, bx, -(ax * bz)), C * fma(ax, by, -(ay * bx))));
        if (len2 > 1e-200) {
            const double il = fm_rsqrt(len2);
            const double R0 = fabs(side) * il;
            const double sa = fma(ax, ex, fma(ay, ey, az * ez)) * il, sb = fma(bx, ex, fma(by, ey, bz * ez)) * il;
            if (R0 > kBoxTiny) {
                const double Y = R0 * R0, P = X + Y, rR = r0 * R0;
                const double lr = 0.5 * fm_log(P);
                double sum = 0.0;
                int net[NP];  // how often each difference kernel's edge share enters: -2 .. 2
#ifdef __CUDACC__
#pragma unroll
#endif
                for (int s = 0; s < NP; ++s) net[s] = 0;
#ifdef __CUDACC__
#pragma unroll 1
#endif
                for (int e = 0; e < 2; ++e) {  // the cones to b (positive) and a (negative), odd in the leg
                    const double sl = e == 0 ? sb : sa, t = fabs(sl);
                    if (t <= kBoxTiny) continue;
                    const bool minus = (sl < 0.0) != (e == 1);
                    const double r2 = fma(t, t, P), ir = fm_rsqrt(r2);
                    double r = r2 * ir;
                    r = fma(0.5 * ir, fma(-r, r, r2), r);
                    int k = 0;
#ifdef __CUDACC__
#pragma unroll
#endif
                    for (int s = 0; s < NP; ++s) k += r2 >= T.scale[s].b * T.scale[s].b;
                    // phi - ang: tan = t R0 (r - r0) / (R0^2 r + t^2 r0), r - r0 = (R0^2 + t^2) / (r + r0)
                    const double tt = t * t;
                    double num = t * (R0 * (Y + tt)), den = (r + r0) * fma(Y, r, tt * r0);
                    bool lo = num <= den;
                    double de = fm_atan01((lo ? num : den) * fm_rcp(lo ? den : num));
                    if (!lo) de = 0.5 * kPi - de;
                    double c = 0.0;
                    if (k > 0) {
                        lo = t <= R0;
                        double ph = fm_atan01((lo ? t : R0) * fm_rcp(lo ? R0 : t));
                        if (!lo) ph = 0.5 * kPi - ph;
#ifdef __CUDACC__
#pragma unroll
#endif
                        for (int s = 0; s < NP; ++s)
                            if (s < k) {
                                c = fma(T.scale[s].m, de, fma(-w.h[s], ph, c));
                                net[s] += minus ? -1 : 1;
                            }
                    }
                    if (k < NP) {
                        const KiwiConeRegion& g = R[k];
                        double ak = w.a[0];
#ifdef __CUDACC__
#pragma unroll
#endif
                        for (int s = 1; s < NP; ++s) ak = k == s ? w.a[s] : ak;
                        const double q = t * ir;
                        double v = q * cone_v(g.V, DEG, r - g.c, X, P);
                        v = fma(box_xp(g.B, 6, (DEG + 1) / 2, X, P), (fm_log(r + t) - lr) - q, v);
                        c = fma(rR, v, fma(-de, ak, c));
                    }
                    sum += minus ? -c : c;
                }
#ifdef __CUDACC__
#pragma unroll
#endif
                for (int s = 0; s < NP; ++s) {
                    const KiwiConeScale& g = T.scale[s];
                    const double t2 = fma(g.b, g.b, -P);
                    if (net[s] != 0 && t2 > 0.0 && r0 < g.b) {
                        const double it = fm_rsqrt(t2), t = t2 * it, ib = g.ib, iR = fm_rcp(R0);
                        const double ang = fm_atan_pos((r0 * ib) * (t * iR), (g.b * R0) * (it * fm_rcp(r0)));
                        const double dB = box_xp(T.reg[s].B, 6, (DEG + 1) / 2, X, P) -
                                          (s + 1 < NP ? box_xp(T.reg[s + 1 < NP ? s + 1 : 0].B, 6, (DEG + 1) / 2, X, P) : 0.0);
                        double v = t * box_xp(g.A, 5, DEG / 2, X, P);
                        v = fma(dB, fm_log(g.b + t) - lr, v);
                        v = fma(rR, v, fma(ang, w.h[s], -(box_delta(t, t2, r0, R0, g.b) * w.f[s])));
                        sum = fma((double)net[s], v, sum);
                    }
                }
                total += side > 0.0 ? sum : -sum;
            }
        }
        ax = bx;
        ay = by;
        az = bz;
    }
    return rs > 0.0 ? total : -total;
}

// A face's plane from its first three vertices, as the reference takes it: unit normal (x, y, z) and offset w.
struct FacePlane {
    double x, y, z, w;
};
KIWI_HD FacePlane face_plane(const double* q) {
    const FaceNormal n = face_normal(q[3] - q[0], q[4] - q[1], q[5] - q[2], q[6] - q[0], q[7] - q[1], q[8] - q[2]);
    const double in = 1.0 / sqrt(n.x * n.x + n.y * n.y + n.z * n.z);
    return {n.x * in, n.y * in, n.z * in, -(n.x * q[0] + n.y * q[1] + n.z * q[2]) * in};
}

// Whether the kernel reaches a face: face_reachable's rule (the reference's, src/kernel_integral.cpp:533-645) decided
// from squared lengths and products, without its three roots, two divisions and two arccosines per vertex; 1 or 0
// where the decision has a margin, -1 where it has none (the caller then takes face_reachable).  What the two may differ by:
// the plane's distance, the foot point and with them every length by the roundings of the coordinates, below err = 1e-14 of
// their size (each is a handful of sums of products with a unit normal, formed from the same A, B, C); R_0 = r12 sqrt(1 - cos^2)
// and the legs from arccosines by up to 1e-8 of the face's extent.  The margins are err and 1e-5 of the radius, for faces of
// up to 100 radii and coordinates of up to 1e7 radii (beyond which the answer is -1 unless the plane alone decides); for the
// side tests, whose threshold is 1e-9 of max(extent, 1), err and a tenth of the threshold.  So it answers in any unit of length,
// and only where coordinates leave the radius fewer than seven digits it does not.  Of 400 k tests
// about the cells of a jittered tessellation none was left to face_reachable.  (Walk of 64 k particles: 30.3 ms with
// face_reachable and the visited marks in global memory, 9.2 ms.)
template <class Plane>
KIWI_HD int face_reach_fast(double x0, double y0, double z0, double radius, const Plane pl, const double* v, int nv) {
    const double mag = (fabs(x0) + fabs(y0) + fabs(z0)) + (fabs(v[0]) + fabs(v[1]) + fabs(v[2])), err = 1e-14 * mag;
    const double r0 = fma(pl.x, x0, fma(pl.y, y0, fma(pl.z, z0, pl.w)));
    const double ar0 = fabs(r0), tol = fma(1e-9, radius, err);
    if (ar0 >= radius + tol) return 0;
    if (!(ar0 < radius - tol) || !(mag < 1e7 * radius)) return -1;
    const double rr = radius * radius, near = rr * (1.0 - 1e-5), r02 = r0 * r0;
    const double xp = fma(-r0, pl.x, x0), yp = fma(-r0, pl.y, y0), zp = fma(-r0, pl.z, z0);
    bool inside = true, have = false, positive = false, sure = true;
    double min2 = INFINITY;
    const double fx = xp - v[0], fy = yp - v[1], fz = zp - v[2];
    double ax = fx, ay = fy, az = fz;  // foot - vertex
    double a2 = fma(ax, ax, fma(ay, ay, az * az));
    const double f2 = a2;
    for (int j = 0; j < nv; ++j) {
        const bool wrap = j == nv - 1;
        const double* q = v + 3 * (wrap ? 0 : j + 1);
        const double bx = wrap ? fx : xp - q[0], by = wrap ? fy : yp - q[1], bz = wrap ? fz : zp - q[2];
        const double b2 = wrap ? f2 : fma(bx, bx, fma(by, by, bz * bz));
        const double ex = ax - bx, ey = ay - by, ez = az - bz;
        const double len2 = fma(ex, ex, fma(ey, ey, ez * ez)), dot = fma(ex, ax, fma(ey, ay, ez * az));
        sure = sure && len2 > 1e-200 && a2 < 1e4 * rr;
        const double d2 = dot <= 0.0 || dot >= len2 ? fmin(a2, b2) : fma(-dot * dot, fm_rcp(len2), a2);
        min2 = fmin(min2, d2);
        if (sure && r02 + d2 < near) return 1;  // within reach whatever the side tests say
        const double side = fma(fma(ey, az, -(ez * ay)), pl.x, fma(fma(ez, ax, -(ex * az)), pl.y, fma(ex, ay, -(ey * ax)) * pl.z));
        const double m = fmax(fmax(fabs(ax), fabs(ay)), fmax(fabs(az), 1.0));
        const double lo = fmax(fma(0.9e-9, m, -err), 0.0), hi = fma(1.1e-9, m, err), s2 = side * side;
        if (s2 >= lo * lo * len2 && s2 <= hi * hi * len2) sure = false;
        if (s2 > hi * hi * len2) {
            if (!have) {
                positive = side > 0.0;
                have = true;
            } else if ((side > 0.0) != positive) {
                inside = false;
            }
        }
        ax = bx;
        ay = by;
        az = bz;
        a2 = b2;
    }
    if (!sure || !(min2 < INFINITY)) return -1;
    if (inside) return 1;  // the plane's distance, which is below the radius
    const double d2 = r02 + min2;
    if (fabs(d2 - rr) < 1e-5 * rr) return -1;
    return d2 < rr;
}

}  // namespace kiwi_b200
