// Test-only: compiles the box-mass maths (kiwi_b200/csrc/box_math.cuh) for the host, and the face integrals
// (cone_math.cuh) for the host, so that tests/test_box_math.py can check them against the float128 oracle without a
// GPU.
#include "../kiwi_b200/csrc/cone_math.cuh"

using namespace kiwi_b200;

namespace {

int piece(const KiwiBoxTable& T, double d2) {
    int k = 0;
    while (k < T.npiece && !(d2 < T.scale[k].b * T.scale[k].b)) ++k;
    return k;
}

template <int NP, int DEG>
double box_mass(const KiwiBoxTable& T, const double* o) {
    const int n = T.npiece;
    double pl[3][16], e[3][8];  // e[i]: the edge line of the two other axes' planes
    for (int a = 0; a < 3; ++a) box_plane<NP, DEG>(T, o[a], pl[a]);
    for (int i = 0; i < 3; ++i) {
        const double *A = pl[i == 0 ? 1 : 0], *B = pl[i == 2 ? 1 : 2];
        const int c = piece(T, fma(A[0], A[0], B[0] * B[0]));
        e[i][2 * n] = 0.0;
        if (c < n) box_edge<NP, DEG>(T, c, A, B, e[i]);
    }
    const double r2 = fma(o[0], o[0], fma(o[1], o[1], o[2] * o[2]));
    const int k = piece(T, r2);
    double t = box_centre<NP>(T, k);
    if (k > 0) t += pl[0][1 + n + k] + pl[1][1 + n + k] + pl[2][1 + n + k];
    if (k == n) return t + (e[0][2 * n] + e[1][2 * n] + e[2][2 * n]);
    const int m = o[0] <= o[1] && o[0] <= o[2] ? 0 : (o[1] <= o[2] ? 1 : 2), a = (m + 1) % 3, b = (m + 2) % 3;
    return t + box_inside<DEG>(T.reg[k].C, T.reg[k].c, T.deg, o[0], o[1], o[2], r2, e[0][k], e[0][n + k], e[1][k],
                               e[1][n + k], e[2][k], e[2][n + k], o[m], pl[m][2 + k], o[a], pl[a][1], pl[a][2 + k], o[b],
                               pl[b][1], pl[b][2 + k]);
}

// The same with its derivatives: out = T, dT/dx, dT/dy, dT/dz.
template <int NP, int DEG>
void box_mass_grad(const KiwiBoxTable& T, const double* o, double* out) {
    const int n = T.npiece;
    double pl[3][32], e[3][32];
    for (int a = 0; a < 3; ++a) box_grad_plane<NP, DEG>(T, o[a], pl[a]);
    for (int i = 0; i < 3; ++i) {
        const double *A = pl[i == 0 ? 1 : 0], *B = pl[i == 2 ? 1 : 2];
        const int c = piece(T, fma(A[0], A[0], B[0] * B[0]));
        for (int j = 0; j < 3; ++j) e[i][6 * n + j] = 0.0;
        if (c < n) box_grad_edge<NP, DEG>(T, c, A, B, e[i]);
    }
    const int k = piece(T, fma(o[0], o[0], fma(o[1], o[1], o[2] * o[2])));
    if (k < n) {
        box_inside_grad<DEG>(T.reg[k].C, T.reg[k].D, T.reg[k].c, T.deg, n, k, pl[0], pl[1], pl[2], e[0], e[1], e[2], out);
    } else {
        const double *x = e[0] + 6 * n, *y = e[1] + 6 * n, *z = e[2] + 6 * n;
        out[0] = x[0] + y[0] + z[0];
        out[1] = z[1] + y[1];
        out[2] = z[2] + x[1];
        out[3] = y[2] + x[2];
    }
    out[0] += box_centre<NP>(T, k);
    for (int a = 0; a < 3 && k > 0; ++a) {
        out[0] += pl[a][bg_w(n, k)];
        out[1 + a] += pl[a][bg_dw(n, k)];
    }
}

}  // namespace

extern "C" {

double bx_log(double v) { return fm_log(v); }
double bx_atan01(double v) { return fm_atan01(v); }
// The box's mass at offsets > 0 in units of the support radius; fixed: the cubic spline with its sizes known when
// compiling, as its kernel has them.
double bx_mass(int kernel, int fixed, const double* offsets) {
    const KiwiBoxTable& T = kiwi_box_tables[kernel];
    return fixed ? box_mass<2, 3>(T, offsets) : box_mass<0, 0>(T, offsets);
}
void bx_mass_grad(int kernel, int fixed, const double* offsets, double* out) {
    const KiwiBoxTable& T = kiwi_box_tables[kernel];
    if (fixed) box_mass_grad<2, 3>(T, offsets, out);
    else box_mass_grad<0, 0>(T, offsets, out);
}
// A face's integral for a particle with support H, and whether the kernel reaches the face: the quick answer (-1: none)
// and face_reachable's.
double bx_face(int kernel, const double* verts, int nv, const double* p, double H) {
    const FlatVerts V{verts};
    const KiwiConeTable& T = kiwi_cone_tables[kernel];
    switch (kernel) {
#define FACE(K, NP, DEG) \
    case K: return cone_face<NP, DEG>(T, T.reg, V, nv, p[0], p[1], p[2], 1.0 / H);
        KIWI_BOX_KERNELS(FACE)
#undef FACE
    }
    return NAN;
}
int bx_reach(const double* verts, int nv, const double* p, double radius, int* exact) {
    const FlatVerts V{verts};
    *exact = face_reachable(p[0], p[1], p[2], radius, V, nv) ? 1 : 0;
    return face_reach_fast(p[0], p[1], p[2], radius, face_plane(verts), verts, nv);
}
double bx_cone_coef_sum(int kernel) {
    const KiwiConeTable& T = kiwi_cone_tables[kernel];
    double s = 0.0;
    for (int k = 0; k < T.npiece; ++k) {
        for (double c : T.reg[k].V) s += fabs(c);
        for (double c : T.reg[k].B) s += fabs(c);
        for (double c : T.reg[k].a) s += fabs(c);
        for (double c : T.scale[k].A) s += fabs(c);
        for (double c : T.scale[k].fp) s += fabs(c);
        for (double c : T.scale[k].ap) s += fabs(c);
    }
    return s;
}
// The sum of the absolute values of a kernel's coefficients, for error bounds.
double bx_coef_sum(int kernel) {
    const KiwiBoxTable& T = kiwi_box_tables[kernel];
    double s = 0.0;
    for (int k = 0; k < T.npiece; ++k) {
        for (double c : T.reg[k].C) s += fabs(c);
        for (double c : T.reg[k].Q) s += fabs(c);
        for (double c : T.reg[k].a) s += fabs(c);
        for (double c : T.scale[k].G) s += fabs(c);
    }
    return s;
}
}
