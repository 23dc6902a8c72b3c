"""The box masses of the Cartesian kernels (kiwi_b200/csrc/box_math.cuh, compiled for the host) against the
float128 oracle: each cell of a particle's support box as the alternating sum of its corners' masses."""
import ctypes as C
import os
import subprocess
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
KERNELS = ["M4", "M5", "M6", "WC2", "WC4", "WC6"]
SUPPORT = [2.0, 2.5, 3.0, 2.0, 2.0, 2.0]
EPS = 2.0 ** -53


@pytest.fixture(scope="module")
def bx(tmp_path_factory):
    out = tmp_path_factory.mktemp("bx") / "libbx.so"
    subprocess.run(["g++", "-O2", "-fPIC", "-shared", "-std=c++17", "-ffp-contract=off", "-o", str(out),
                    os.path.join(ROOT, "tests", "box_host_check.cpp")], check=True)
    L = C.CDLL(str(out))
    for f in ("bx_log", "bx_atan01"):
        getattr(L, f).restype, getattr(L, f).argtypes = C.c_double, [C.c_double]
    L.bx_mass.restype, L.bx_mass.argtypes = C.c_double, [C.c_int, C.c_int, C.POINTER(C.c_double)]
    L.bx_coef_sum.restype, L.bx_coef_sum.argtypes = C.c_double, [C.c_int]
    return L


@pytest.fixture(scope="module")
def quad_oracle():
    from oracle.oracle import Oracle

    return Oracle(quad=True)


def test_tables_are_current():
    gen = os.path.join(ROOT, "kiwi_b200", "tables", "gen_box_tables.py")
    assert subprocess.run([sys.executable, gen, "--check"]).returncode == 0


def test_functions(bx):
    """Rounding level in absolute terms: the reduction's and the polynomial's few roundings of values up to |f|."""
    x = np.concatenate([[0.0, 1e-300, 1e-17, 1.0], np.random.default_rng(1).random(2000)])
    assert max(abs(bx.bx_atan01(v) - np.arctan(np.longdouble(v))) for v in x) <= 4 * EPS
    v = np.concatenate([[1.0, np.sqrt(0.5), np.sqrt(2.0), 2.0, 1e-200], np.exp(np.random.default_rng(2).uniform(-40, 3, 2000))])
    for t in v:
        want = np.log(np.longdouble(t))
        assert abs(bx.bx_log(t) - want) <= 4 * EPS * max(1.0, abs(want))


@pytest.mark.parametrize("kernel", range(6), ids=KERNELS)
def test_cells_against_float128(bx, quad_oracle, kernel):
    """Particles at a general place, near planes (offsets of 1e-3, 1e-9 and 1e-15 of a cell) and with a support that
    ends on planes; a wide and a narrow support.  Bound: each of a cell's eight corner masses carries at most 16
    roundings of terms no larger than the table's coefficients allow."""
    n = 6
    bound = 8 * 16 * EPS * max(1.0, bx.bx_coef_sum(kernel))
    for frac, H in (((0.31, 0.57, 0.44), 0.42), ((1e-3, 0.5, 1 - 1e-3), 0.3), ((1e-9, 1e-15, 0.7), 0.25),
                    ((0.5, 0.5, 0.5), 0.25), ((0.2, 0.9, 1e-9), 0.06)):
        pos = [(2 + f) / n for f in frac]
        P = {k: np.array([v]) for k, v in zip(("x", "y", "z", "vx", "vy", "vz", "m", "h"),
                                             (*pos, 0.0, 0.0, 0.0, 1.0, H / SUPPORT[kernel]))}
        truth = quad_oracle.sph_to_grid(P, (0.0, 1.0) * 3, (n, n, n), kernel=-1 if kernel == 0 else kernel,
                                        support_in_h=SUPPORT[kernel])[4][0].reshape(n, n, n)
        H = SUPPORT[kernel] * P["h"][0]
        d = 1.0 / n
        off = [(np.arange(n + 1) * d - p) / H for p in pos]
        for fixed in ((0, 1) if kernel == 0 else (0,)):
            T = np.zeros((n + 1,) * 3)
            for i in np.ndindex(T.shape):
                u = [off[a][i[a]] for a in range(3)]
                if 0.0 not in u:
                    T[i] = np.sign(u).prod() * bx.bx_mass(kernel, fixed, (C.c_double * 3)(*np.abs(u)))
            cells = np.diff(np.diff(np.diff(T, axis=0), axis=1), axis=2)
            assert np.max(np.abs(np.maximum(cells, 0.0) - truth.astype(float))) <= bound


@pytest.mark.parametrize("kernel", range(6), ids=KERNELS)
def test_derivatives_against_differences(bx, kernel):
    """dT/dx, dT/dy, dT/dz against extrapolated central differences of T over the pieces, near their breakpoints,
    near a plane and beyond the support.  Bound: the kernels' third derivative jumps, so the differences err by
    step^3 times the size of the kernel's coefficients, plus T's roundings over the step."""
    bx.bx_mass_grad.argtypes = [C.c_int, C.c_int, C.POINTER(C.c_double), C.POINTER(C.c_double)]
    rng = np.random.default_rng(5)
    pts = np.concatenate([rng.uniform(0.02, 1.1, (60, 3)), 10.0 ** rng.uniform(-2, 0, (40, 3)),
                          [[0.3, 0.4, 0.0051], [0.5, 0.5, 0.7071], [0.6, 0.8, 0.02], [0.2, 0.33, 0.999], [1.2, 1.3, 1.1]]])
    step, size = 2.5e-4, max(1.0, bx.bx_coef_sum(kernel))
    bound = 2 * step ** 3 * size + 16 * 8 * EPS * size / step
    mass = lambda f, p: bx.bx_mass(kernel, f, (C.c_double * 3)(*p))  # noqa: E731
    for fixed in ((0, 1) if kernel == 0 else (0,)):
        for p in pts:
            got = (C.c_double * 4)()
            bx.bx_mass_grad(kernel, fixed, (C.c_double * 3)(*p), got)
            assert abs(got[0] - mass(fixed, p)) <= 16 * EPS * size
            for a in range(3):
                d = [(mass(fixed, p + np.eye(3)[a] * s) - mass(fixed, p - np.eye(3)[a] * s)) / (2 * s) for s in (step, 2 * step)]
                assert abs(got[1 + a] - (4 * d[0] - d[1]) / 3) <= bound


def _polygon(rng, n, scale, squash=1.0):
    """A convex planar polygon of n vertices in a random plane."""
    a = np.sort(rng.uniform(0, 2 * np.pi, n))
    q, _ = np.linalg.qr(rng.standard_normal((3, 3)))
    return (np.stack([np.cos(a), squash * np.sin(a), 0 * a], 1) * scale) @ q.T + rng.standard_normal(3) * scale


@pytest.mark.parametrize("kernel", range(6), ids=KERNELS)
def test_faces_against_float128(bx, quad_oracle, kernel):
    """Faces of 3 to 9 vertices, slivers among them, particles anywhere about them, near a vertex, near an edge line
    and near the plane.  Bound: each of the face's cones carries at most 16 roundings of terms no larger than the
    table's coefficients allow, two cones and an edge share per vertex."""
    dp = C.POINTER(C.c_double)
    bx.bx_face.restype, bx.bx_face.argtypes = C.c_double, [C.c_int, dp, C.c_int, dp, C.c_double]
    bx.bx_cone_coef_sum.restype, bx.bx_cone_coef_sum.argtypes = C.c_double, [C.c_int]
    rng = np.random.default_rng(17)
    size = max(1.0, bx.bx_cone_coef_sum(kernel))
    for i in range(160):
        n = 3 + i % 7
        v = np.ascontiguousarray(_polygon(rng, n, 0.3, 1.0 if i % 4 else 0.02))
        H = rng.uniform(0.2, 1.5)
        p = v.mean(0) + rng.standard_normal(3) * 0.5 * H
        if i % 5 == 1:
            p = v[0] + rng.standard_normal(3) * 1e-5
        if i % 5 == 2:
            p = 0.5 * (v[0] + v[1]) + rng.standard_normal(3) * 1e-4
        if i % 5 == 3:
            p = v.mean(0) + rng.standard_normal(3) * 1e-7
        want = quad_oracle.face_integral(*p, v, kernel=-1 if kernel == 0 else kernel, h=H / SUPPORT[kernel],
                                         support=H)[0]
        got = bx.bx_face(kernel, v.ctypes.data_as(dp), n, p.ctypes.data_as(dp), H)
        assert abs(got - want) <= 3 * n * 16 * EPS * size, (i, got, want)


def test_quick_reach_agrees(bx):
    """Where the quick test answers, it answers as the reference's rule does: over scales, slivers, repeated vertices,
    distances about the radius (down to 1e-9 of it), particles in the plane and beside vertices; and it does
    answer almost always where the distance has a margin."""
    dp = C.POINTER(C.c_double)
    bx.bx_reach.argtypes = [dp, C.c_int, dp, C.c_double, C.POINTER(C.c_int)]
    rng = np.random.default_rng(23)
    open_, far = 0, 0
    for i in range(20_000):
        scale = 10.0 ** rng.integers(-9, 4) if i % 3 == 0 else 0.3
        n = 3 + i % 8
        v = _polygon(rng, n, scale, (1.0, 0.05, 1e-6)[i % 17 % 3])
        if i % 11 == 0:
            v[n - 1] = v[n - 2]
        v = np.ascontiguousarray(v)
        p = v.mean(0) + rng.standard_normal(3) * scale * 10.0 ** rng.uniform(-6, 1)
        if i % 7 == 0:
            p = v[0] + rng.standard_normal(3) * scale * 10.0 ** rng.uniform(-9, -1)
        radius = scale * rng.uniform(0.1, 4.0)
        if i % 2:  # a radius at a chosen distance from the face's vertices or plane
            d = np.linalg.norm(p - v[rng.integers(n)])
            radius = d * (1 + rng.choice([-1, 1]) * 10.0 ** rng.uniform(-9, -1))
        ex = C.c_int(0)
        got = bx.bx_reach(v.ctypes.data_as(dp), n, np.ascontiguousarray(p).ctypes.data_as(dp), radius, C.byref(ex))
        assert got in (-1, ex.value), (i, got, ex.value)
        if i % 2 == 0 and i % 3 and i % 11:
            far += 1
            open_ += got < 0
    assert open_ < 0.02 * far
