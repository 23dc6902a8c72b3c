"""The derivatives of the box masses (kiwi_b200/csrc/box_grad.cuh, compiled for the host) on a plane through the particle."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
DP = C.POINTER(C.c_double)
EPS = 2.0 ** -53


@pytest.fixture(scope="module")
def bx(tmp_path_factory):
    out = tmp_path_factory.mktemp("planes") / "libbx.so"
    subprocess.run(["g++", "-O2", "-fPIC", "-shared", "-std=c++17", "-ffp-contract=off", "-o", str(out),
                    os.path.join(ROOT, "tests", "box_host_check.cpp")], check=True)
    L = C.CDLL(str(out))
    L.bx_mass.restype, L.bx_mass.argtypes = C.c_double, [C.c_int, C.c_int, DP]
    L.bx_mass_grad.argtypes = [C.c_int, C.c_int, DP, DP]
    L.bx_coef_sum.restype, L.bx_coef_sum.argtypes = C.c_double, [C.c_int]
    return L


@pytest.mark.parametrize("kernel", range(6))
def test_derivative_across_a_plane_through_the_particle(bx, kernel):
    """T is odd in each offset, so dT/dx at x = 0 is the limit of T / x: against its extrapolation from two steps, for
    points within the support, in its outer part and beyond it.  Bound: the steps' third-order remainder and T's
    roundings over the step, as for the derivatives elsewhere."""
    step, size = 2.5e-4, max(1.0, bx.bx_coef_sum(kernel))
    bound = 2 * step ** 3 * size + 16 * 8 * EPS * size / step
    rng = np.random.default_rng(11)
    for y, z in np.concatenate([rng.uniform(0.02, 0.7, (30, 2)), rng.uniform(0.7, 1.3, (10, 2)), [[1e-3, 0.5], [0.4, 1.0]]]):
        for axis in range(3):
            at = lambda x: (C.c_double * 3)(*np.insert([y, z], axis, x))  # noqa: E731
            d = [bx.bx_mass(kernel, 0, at(s)) / s for s in (step, 2 * step)]
            got = (C.c_double * 4)()
            bx.bx_mass_grad(kernel, 0, at(0.0), got)
            assert abs(got[1 + axis] - (4 * d[0] - d[1]) / 3) <= bound
            assert abs(got[0]) <= 16 * EPS * size
            for other in {0, 1, 2} - {axis}:
                assert abs(got[1 + other]) <= 16 * 8 * EPS * size
