"""The device forms of the functions behind the box masses (kiwi_b200/csrc/fastmath.cuh: the hardware's approximations
refined, the logarithm's table) against extended precision, over the ranges that their callers reach.  (The host
forms, which tests/test_box_math.py checks, take other paths.)"""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
DP = C.POINTER(C.c_double)
EPS = 2.0 ** -53
RNG = np.random.default_rng(41)


@pytest.fixture(scope="module")
def apply(tmp_path_factory):
    from kiwi_b200.build import ARCH, nvcc

    so = tmp_path_factory.mktemp("functions") / "libfm.so"
    subprocess.run([nvcc(), *ARCH, "-O3", "-std=c++17", "--expt-relaxed-constexpr", "-Xcompiler", "-fPIC", "-shared", "-o",
                    str(so), os.path.join(ROOT, "tests", "fastmath_device_check.cu")], check=True)
    L = C.CDLL(str(so))
    L.fm_apply.argtypes = [C.c_int, C.c_int, DP, DP]

    def run(which, x):
        x = np.ascontiguousarray(x, dtype=np.float64)
        y = np.empty_like(x)
        assert L.fm_apply(which, x.size, x.ctypes.data_as(DP), y.ctypes.data_as(DP)) == 0
        return y

    return run


def _wide():
    """Log-uniform over 1e-290 .. 1e290, and every last place about 1, 2 and 4."""
    near = [np.array(c) * (1 + np.arange(-40, 40) * 2 * EPS) for c in (1.0, 2.0, 4.0)]
    return np.concatenate([10.0 ** RNG.uniform(-290, 290, 40_000), 10.0 ** RNG.uniform(-3, 1, 40_000), *near])


def test_reciprocal(apply):
    """To rounding: half a place of the last fma and the refinement's own, far below it; at most two roundings."""
    x = _wide()
    assert np.max(np.abs(apply(0, x).astype(np.longdouble) * x - 1)) <= 2 * EPS


def test_reciprocal_root(apply):
    """a y is rounded once before its residual (a quarter of a place in the result) and the result once."""
    x = _wide()
    y = apply(1, x).astype(np.longdouble)
    assert np.max(np.abs(y * np.sqrt(x.astype(np.longdouble)) - 1)) <= 2 * EPS


def test_logarithm(apply):
    """In absolute terms, as its callers need it: a rounding of the table's entry, of the polynomial, of their sum and of the
    exponent's part.  Both sides of every cell of the table, at several exponents, and the range of the callers."""
    hi0 = np.float64(np.sqrt(0.5)).view(np.int64) >> 32
    edges = np.array([((int(hi0) + (j << 14)) << 32) for j in range(-64, 130)], dtype=np.int64).view(np.float64)
    edges = np.concatenate([np.nextafter(edges, 0), edges, np.nextafter(edges, 4)])
    cuts = np.array([np.sqrt(0.5), np.sqrt(2.0), 1.0, 2.0])
    cuts = np.concatenate([np.nextafter(cuts, 0), cuts, np.nextafter(cuts, 4)])
    x = np.concatenate([np.concatenate([edges, cuts]) * 2.0 ** k for k in (-660, -30, -2, -1, 0, 1, 3)] +
                       [10.0 ** RNG.uniform(-200, 1, 40_000), RNG.uniform(0.5, 2.0, 40_000)])
    want = np.log(x.astype(np.longdouble))
    assert np.max(np.abs(apply(2, x) - want) / np.maximum(1.0, np.abs(want))) <= 4 * EPS


def test_arctangent(apply):
    x = np.concatenate([[0.0, 1e-300, 1e-17, 1.0, np.nextafter(1.0, 0)], RNG.random(60_000), 10.0 ** RNG.uniform(-20, 0, 20_000)])
    want = np.arctan(x.astype(np.longdouble))
    assert np.max(np.abs(apply(3, x) - want)) <= 4 * EPS
    assert np.max(np.abs(apply(3, x[x > 0]) / want[x > 0] - 1)) <= 6 * EPS
