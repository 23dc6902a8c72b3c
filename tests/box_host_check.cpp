// Test-only: compiles the box-mass maths (kiwi_b200/csrc/box_math.cuh) for the host, so that tests/test_box_math.py
// can check it against the float128 oracle without a GPU.
#include "../kiwi_b200/csrc/box_math.cuh"

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
// The sum of the absolute values of a kernel's coefficients, for error bounds.
double bx_coef_sum(int kernel) {
    const KiwiBoxTable& T = kiwi_box_tables[kernel];
    double s = 0.0;
    for (int k = 0; k < T.npiece; ++k) {
        for (double c : T.reg[k].C) s += fabs(c);
        for (double c : T.reg[k].Q) s += fabs(c);
        for (double c : T.reg[k].a) s += fabs(c);
        for (double c : T.scale[k].G) s += fabs(c);
        for (double c : T.scale[k].Q) s += fabs(c);
    }
    return s;
}
}
