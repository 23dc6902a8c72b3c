"""The Voronoi map's face integrals (kiwi_b200/csrc/cone_math.cuh, compiled for the host) on faces the general tests do
not hold."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
DP = C.POINTER(C.c_double)
EPS = 2.0 ** -53
SUPPORT = [2.0, 2.5, 3.0, 2.0, 2.0, 2.0]


@pytest.fixture(scope="module")
def bx(tmp_path_factory):
    out = tmp_path_factory.mktemp("cone") / "libbx.so"
    subprocess.run(["g++", "-O2", "-fPIC", "-shared", "-std=c++17", "-ffp-contract=off", "-o", str(out),
                    os.path.join(ROOT, "tests", "box_host_check.cpp")], check=True)
    L = C.CDLL(str(out))
    L.bx_face.restype, L.bx_face.argtypes = C.c_double, [C.c_int, DP, C.c_int, DP, C.c_double]
    L.bx_reach.argtypes = [DP, C.c_int, DP, C.c_double, C.POINTER(C.c_int)]
    return L


def _ptr(a):
    return np.ascontiguousarray(a).ctypes.data_as(DP)


@pytest.mark.parametrize("kernel", range(6))
def test_first_three_vertices_in_a_line(bx, oracle, kernel):
    """A face that starts with a vertex on an edge (a hanging node: the offsets of its second and third vertex are exact
    multiples) has no plane by the reference's rule, and the reference adds exactly 0 for it; listed from another
    vertex on, it is the face it is."""
    rng = np.random.default_rng(3)
    for i in range(40):
        q, _ = np.linalg.qr(rng.standard_normal((3, 3)))
        square = np.array([[0, 0, 0], [1, 0, 0], [2, 0, 0], [2, 2, 0], [0, 2, 0]]) * 2.0 ** -int(rng.integers(0, 4))
        v = square @ (q.T if i else np.eye(3))
        v[1:3] = np.outer([1.0, 2.0], v[1])
        p = v.mean(0) + rng.standard_normal(3) * 0.2
        h = 0.5
        want = oracle.face_integral(*p, v, kernel=-1 if kernel == 0 else kernel, h=h, support=SUPPORT[kernel] * h)[0]
        assert want == 0.0
        assert bx.bx_face(kernel, _ptr(v), 5, _ptr(p), SUPPORT[kernel] * h) == 0.0, i
        assert bx.bx_face(kernel, _ptr(np.roll(v, -2, axis=0)), 5, _ptr(p), SUPPORT[kernel] * h) != 0.0


def _polygon(rng, n, scale, squash):
    a = np.sort(rng.uniform(0, 2 * np.pi, n))
    q, _ = np.linalg.qr(rng.standard_normal((3, 3)))
    return (np.stack([np.cos(a), squash * np.sin(a), 0 * a], 1) * scale) @ q.T


@pytest.mark.parametrize("offset,scale", [(0.0, 1e-6), (0.0, 1e16), (3e4, 1.0), (3e4, 1e-4), (3e4, 1e-6), (3e4, 1e-7), (2e5, 1e3),
                                          (1e8, 1.0), (3e18, 1e16), (3e18, 1e12), (1.0, 1e-10)])
def test_quick_reach_far_from_the_origin(bx, offset, scale):
    """The quick test answers as the reference's rule does wherever the face lies and in whatever unit, also where the
    coordinates' roundings are no longer small against the radius and the particle is within 1e-7 of it; and it does answer
    where they leave the radius more than seven digits."""
    rng = np.random.default_rng(29)
    undecided = tests = 0
    for i in range(6000):
        n = 3 + i % 8
        v = np.ascontiguousarray(_polygon(rng, n, scale, (1.0, 0.05, 1e-3)[i % 3]) + offset * rng.uniform(0.5, 1, 3))
        p = v.mean(0) + rng.standard_normal(3) * scale * 10.0 ** rng.uniform(-3, 0.5)
        radius = scale * rng.uniform(0.1, 4.0)
        if i % 2:
            radius = np.linalg.norm(p - v[rng.integers(n)]) * (1 + rng.choice([-1, 1]) * 10.0 ** rng.uniform(-7, -2))
        ex = C.c_int(0)
        got = bx.bx_reach(_ptr(v), n, _ptr(p), radius, C.byref(ex))
        assert got in (-1, ex.value), (i, got, ex.value)
        if i % 2 == 0 and 6 * max(offset, scale) < 1e7 * radius:
            tests += 1
            undecided += got < 0
    assert undecided <= 0.02 * tests
