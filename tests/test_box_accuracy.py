"""How exact the box masses and the face integrals are (csrc/box_math.cuh and cone_math.cuh, compiled for the host), against
the float128 oracle: bounds at six times what each kernel showed when they were set, so that a table or a
polynomial that loses a digit shows here.  (The bounds of test_box_math.py hold for any evaluation that rounds its terms;
a thousand times the rounding of the logarithm passes them.)"""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from test_box_math import KERNELS, SUPPORT, _polygon, quad_oracle  # noqa: F401

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
DP = C.POINTER(C.c_double)
EPS = 2.0 ** -53
# largest errors measured (kernel mass 1), over a whole 32^3 grid too: cells 1.1e-15, 3.4e-15, 9.9e-15, 1.4e-15, 7.9e-15, 8.6e-14
CELL = [7e-15, 2e-14, 6e-14, 9e-15, 5e-14, 5e-13]
# and faces 1.2e-16, 4.1e-16, 9.5e-16, 2.0e-16, 1.6e-15, 1.2e-14
FACE = [8e-16, 2.5e-15, 6e-15, 1.3e-15, 1e-14, 7e-14]


@pytest.fixture(scope="module")
def bx(tmp_path_factory):
    out = tmp_path_factory.mktemp("accuracy") / "libbx.so"
    subprocess.run(["g++", "-O2", "-fPIC", "-shared", "-std=c++17", "-ffp-contract=off", "-o", str(out),
                    os.path.join(ROOT, "tests", "box_host_check.cpp")], check=True)
    L = C.CDLL(str(out))
    L.bx_mass.restype, L.bx_mass.argtypes = C.c_double, [C.c_int, C.c_int, DP]
    L.bx_face.restype, L.bx_face.argtypes = C.c_double, [C.c_int, DP, C.c_int, DP, C.c_double]
    return L


@pytest.mark.parametrize("kernel", range(6), ids=KERNELS)
def test_cells(bx, quad_oracle, kernel):  # noqa: F811
    """A coarse grid, where a cell holds much of the kernel, and blocks of a fine one (1/32, supports of 0.45), where corners
    nearly cancel: about the particle, on the way out and at the support's end."""
    for lo, n, cell, pos, H in ((0.0, 6, 1 / 6, (2.31 / 6, 2.57 / 6, 2.44 / 6), 0.42), (0.0, 6, 1 / 6, (2 / 6 + 1e-10, 2 / 6, 0.45), 0.25),
                                (0.0, 6, 1 / 6, (2.5 / 6, 2.5 / 6, 2.5 / 6), 0.25), (0.375, 7, 1 / 32, (0.4788, 0.4866, 0.4825), 0.45),
                                (0.5, 6, 1 / 32, (0.4788, 0.4866, 0.4825), 0.45), (0.625, 6, 1 / 32, (0.4788, 0.4866, 0.4825), 0.45)):
        P = {k: np.array([v]) for k, v in zip(("x", "y", "z", "vx", "vy", "vz", "m", "h"),
                                             (*pos, 0.0, 0.0, 0.0, 1.0, H / SUPPORT[kernel]))}
        truth = quad_oracle.sph_to_grid(P, (lo, lo + n * cell) * 3, (n, n, n), kernel=-1 if kernel == 0 else kernel,
                                        support_in_h=SUPPORT[kernel])[4][0].reshape(n, n, n)
        d = (lo + n * cell - lo) / n
        off = [(lo + np.arange(n + 1) * d - p) / (SUPPORT[kernel] * P["h"][0]) for p in pos]
        T = np.zeros((n + 1,) * 3)
        for i in np.ndindex(T.shape):
            u = [off[a][i[a]] for a in range(3)]
            if 0.0 not in u:
                T[i] = np.sign(u).prod() * bx.bx_mass(kernel, 0, (C.c_double * 3)(*np.abs(u)))
        cells = np.diff(np.diff(np.diff(T, axis=0), axis=1), axis=2)
        assert np.max(np.abs(np.maximum(cells, 0.0) - truth.astype(float))) <= CELL[kernel], (lo, pos)


@pytest.mark.parametrize("kernel", range(6), ids=KERNELS)
def test_faces(bx, quad_oracle, kernel):  # noqa: F811
    rng = np.random.default_rng(31)
    worst = 0.0
    for i in range(60):
        n = 3 + i % 7
        v = np.ascontiguousarray(_polygon(rng, n, 0.3))
        H = rng.uniform(0.2, 1.5)
        p = v.mean(0) + rng.standard_normal(3) * 0.5 * H
        want = quad_oracle.face_integral(*p, v, kernel=-1 if kernel == 0 else kernel, h=H / SUPPORT[kernel], support=H)[0]
        worst = max(worst, abs(bx.bx_face(kernel, v.ctypes.data_as(DP), n, p.ctypes.data_as(DP), H) - want))
    assert worst <= FACE[kernel], worst


@pytest.mark.parametrize("kernel", range(6), ids=KERNELS)
def test_cells_about_the_particle(bx, quad_oracle, kernel):  # noqa: F811
    """Relative to their own mass, cells of 0.02 and 0.05 of the support about the particle, where the box masses are small.
    Bound: a cell's eight corners hold at most eight times its mass, each with some four roundings."""
    for cell in (0.02, 0.05):
        pos, n, lo = (0.31 * cell, 0.77 * cell, 0.45 * cell), 4, -2 * cell
        P = {k: np.array([v]) for k, v in zip(("x", "y", "z", "vx", "vy", "vz", "m", "h"),
                                             (*pos, 0.0, 0.0, 0.0, 1.0, 1.0 / SUPPORT[kernel]))}
        truth = quad_oracle.sph_to_grid(P, (lo, -lo) * 3, (n, n, n), kernel=-1 if kernel == 0 else kernel,
                                        support_in_h=SUPPORT[kernel])[4][0].reshape(n, n, n).astype(float)
        off = [(lo + np.arange(n + 1) * (-2 * lo / n) - p) / (SUPPORT[kernel] * P["h"][0]) for p in pos]
        T = np.zeros((n + 1,) * 3)
        for i in np.ndindex(T.shape):
            u = [off[a][i[a]] for a in range(3)]
            T[i] = np.sign(u).prod() * bx.bx_mass(kernel, 0, (C.c_double * 3)(*np.abs(u)))
        cells = np.diff(np.diff(np.diff(T, axis=0), axis=1), axis=2)
        assert np.max(np.abs(cells - truth) / truth) <= 8 * 8 * 4 * EPS
