"""Voronoi maps of tessellations and particles that the other tests do not hold."""
import numpy as np
import pytest

from conftest import random_particles
from test_gpu_voronoi import _cells_as_lists, _lists_as_cells, lattice_cells

pytestmark = pytest.mark.gpu


def _home(P, n, d):
    return ((np.floor(P["x"] / d) * n + np.floor(P["y"] / d)) * n + np.floor(P["z"] / d)).astype(np.int32)


def _close(got, want):
    for band, tol in ((1e-2, 4e-10), (1e-4, 4e-9), (1e-6, 1e-7)):
        m = want > band * want.max()
        assert np.max(np.abs(got[m] - want[m]) / want[m]) < tol, band


def test_face_that_starts_on_an_edge(kiwi, ctx, oracle):
    """A cell whose faces start with a vertex on an edge (three vertices in a line) has no plane there by the reference's
    rule: such faces add 0 and every walk passes them.  The tessellation is turned, so that the offsets' products
    round."""
    n = 8
    geo, d = lattice_cells(n, 0.0, 1.0)
    cells = _cells_as_lists(geo)
    c = (4 * n + 3) * n + 4
    turn, _ = np.linalg.qr(np.random.default_rng(9).standard_normal((3, 3)))
    for i, (v, b) in enumerate(cells[c]):
        step = 0.5 * (v[1] - v[0])
        cells[c][i] = (np.concatenate([v[:1], [v[0] + step], v[1:]]), b)
    P = random_particles(60, 21, box=(0.3, 0.7), hmin=0.05, hmax=0.12)
    home = _home(P, n, d)
    g = _lists_as_cells(cells, geo["volume"])
    g["vxyz"] = np.ascontiguousarray((g["vxyz"].reshape(-1, 3) @ turn.T).reshape(-1))
    # the second and third vertices' offsets from the first exactly in the ratio 1 : 2 after the turn
    vx, vo = g["vxyz"].reshape(-1, 3), g["vert_off"]
    for f in range(g["face_off"][c], g["face_off"][c + 1]):
        a = vo[f]
        half = np.round(0.5 * (vx[a + 2] - vx[a]) * 2.0 ** 40) / 2.0 ** 40
        vx[a] = np.round(vx[a] * 2.0 ** 40) / 2.0 ** 40
        vx[a + 1], vx[a + 2] = vx[a] + half, vx[a] + 2 * half
        assert not np.any(np.cross(vx[a + 1] - vx[a], vx[a + 2] - vx[a]))
    X = np.stack([P["x"], P["y"], P["z"]], 1) @ turn.T
    P["x"], P["y"], P["z"] = (np.ascontiguousarray(X[:, i]) for i in range(3))
    o = oracle.map_voronoi(P, home, g)
    v = kiwi.map_voronoi(P, home, g, raw=True, ctx=ctx)
    assert v.stats["visited_pairs"] == o[5]
    _close(v.raw[0], o[4][0])


@pytest.mark.parametrize("unit,shift", [(2.0 ** 21, 0.0), (2.0 ** 62, 0.0), (1.0, 3.0e4), (2.0 ** -10, 3.0)])
def test_units_and_offsets(kiwi, ctx, oracle, unit, shift):
    """Any unit of length, and a domain far from the origin: the walk visits the reference's pairs."""
    n = 8
    geo, d = lattice_cells(n, 0.0, 1.0)
    P = random_particles(60, 33, box=(0.2, 0.8), hmin=0.04, hmax=0.12)
    home = _home(P, n, d)
    g = dict(geo, vxyz=np.ascontiguousarray(geo["vxyz"].reshape(-1) * unit + shift), volume=geo["volume"] * unit ** 3)
    for k in ("x", "y", "z"):
        P[k] = P[k] * unit + shift
    P["h"] = P["h"] * unit
    o = oracle.map_voronoi(P, home, g)
    v = kiwi.map_voronoi(P, home, g, raw=True, ctx=ctx)
    assert v.stats["visited_pairs"] == o[5]
    if shift == 0.0:  # (else the coordinates' roundings, which the two take differently, are in the masses)
        _close(v.raw[0], o[4][0])


# walks longer than the shared table holds (640 cells; here up to all 4,096), alone, and one in seven among short ones
@pytest.mark.parametrize("n_part,every", [(3, 1), (300, 7)])
@pytest.mark.parametrize("kernel", [0, 4])
def test_long_walks(kiwi, oracle, n_part, every, kernel):
    """The walks that outgrow the shared table run in a launch of their own: the reference's pairs, and the same bits from
    a context's first map (two walks), its second (one, staged), a larger map after a smaller one (the staging area
    overflows), the single-launch gather and the inverse map's pairs."""
    n = 16
    geo, d = lattice_cells(n, 0.0, 1.0)
    P = random_particles(n_part, 7, box=(0.05, 0.95), hmin=0.04, hmax=0.13)
    P["h"][::every] = np.linspace(0.25, 0.9, len(P["h"][::every]))
    home = _home(P, n, d)
    ki = kiwi.KernelIntegrator(kernel=kernel)
    o = oracle.map_voronoi(P, home, geo, kernel=kernel if kernel > 0 else -1, support_in_h=2.0)
    assert o[5] > 640 * len(P["h"][::every])
    ctx = kiwi.Context(0)
    maps = [kiwi.map_voronoi(P, home, geo, kernel=ki, raw=True, ctx=ctx) for _ in range(2)]
    ctx.set_voronoi_face_tables(False)
    maps.append(kiwi.map_voronoi(P, home, geo, kernel=ki, raw=True, ctx=ctx))
    other = kiwi.Context(0)
    kiwi.map_voronoi({k: v[:2] for k, v in P.items()}, home[:2], geo, kernel=ki, ctx=other)
    maps.append(kiwi.map_voronoi(P, home, geo, kernel=ki, raw=True, ctx=other))
    for v in maps:
        assert v.stats["visited_pairs"] == o[5]
        assert np.array_equal(v.raw, maps[0].raw)
    assert np.max(np.abs(maps[0].raw[0] - o[4][0])) <= 1e-9 * o[4][0].max()
    inv = [kiwi.inverse_map_voronoi(P, home, geo, kernel=ki, ctx=c) for c in (other, kiwi.Context(0))]
    assert np.array_equal(inv[0].m_recovered, inv[1].m_recovered)


def test_short_walks_hold_no_global_arrays(kiwi):
    """A map of short walks takes memory for its cells, faces and pairs alone: 27,000 cells under 100 MB."""
    torch = pytest.importorskip("torch")
    n = 30
    geo, d = lattice_cells(n, 0.0, 1.0)
    P = random_particles(20, 5, box=(0.2, 0.8), hmin=0.02, hmax=0.05)
    ctx = kiwi.Context(0)
    tiny, dt = lattice_cells(3, 0.0, 1.0)
    kiwi.map_voronoi(P, _home(P, 3, dt), tiny, ctx=ctx)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    kiwi.map_voronoi(P, _home(P, n, d), geo, ctx=ctx)
    torch.cuda.synchronize()
    assert free - torch.cuda.mem_get_info()[0] < 100e6
