"""Grids whose every tile has a long particle list: the raw sums of the lists' segments stay bounded, the tiles being taken in
several runs, and the cells are those of a call that needs one run."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

SHAPE, BOUNDS = (160, 160, 160), (0.0, 160.0) * 3


def _particles(per_corner, seed):
    """Particles about the corners that eight tiles share (supports of a fifth of a cell): 8 entries each."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    c = torch.arange(1, 20, device="cuda", dtype=torch.float64) * 8.0
    at = torch.stack(torch.meshgrid(c, c, c, indexing="ij"), -1).reshape(-1, 3).repeat(per_corner, 1)
    n = at.shape[0]
    at = at + 0.3 * (torch.rand(n, 3, dtype=torch.float64, device="cuda", generator=g) - 0.5)
    P = {k: at[:, i].contiguous() for i, k in enumerate(("x", "y", "z"))}
    P.update({k: torch.randn(n, dtype=torch.float64, device="cuda", generator=g) for k in ("vx", "vy", "vz")})
    P["m"] = 0.5 + torch.rand(n, dtype=torch.float64, device="cuda", generator=g)
    P["h"] = torch.full((n,), 0.1, dtype=torch.float64, device="cuda")
    return P


def _new():
    nc = int(np.prod(SHAPE))
    return {"density": torch.full((nc,), np.nan, dtype=torch.float64, device="cuda"),
            "raw4": torch.full((4 * nc,), np.nan, dtype=torch.float64, device="cuda")}


def _free():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_sums_are_bounded(kiwi):
    """All 57,040 segments would take 0.93 GB (1.17 with the scratch pool's quarter); 16,384 of them take 0.34 GB.  Then with
    less memory left than that: smaller runs, the same cells.  And a batch of two such grids, in several runs."""
    P = _particles(1200, 1)
    ctx = kiwi.Context(0)
    parts = _new()
    for p in range(8):  # (one run each)
        kiwi.sph_to_grid_device(P, BOUNDS, SHAPE, parts, ctx=ctx, part=p, n_parts=8)
    assert not torch.isnan(parts["raw4"]).any()
    whole, free = _new(), _free()
    kiwi.sph_to_grid_device(P, BOUNDS, SHAPE, whole, ctx=ctx)
    assert free - _free() < 400e6
    assert all(torch.equal(whole[k], parts[k]) for k in whole)
    halves = _new()
    for p in range(2):  # (two runs each, over a part's own tiles)
        kiwi.sph_to_grid_device(P, BOUNDS, SHAPE, halves, ctx=ctx, part=p, n_parts=2)
    assert all(torch.equal(halves[k], parts[k]) for k in halves)
    # a context whose sums hold one part's at the time the memory is taken
    ctx, little = kiwi.Context(0), _new()
    for p in range(8):
        kiwi.sph_to_grid_device(P, BOUNDS, SHAPE, little, ctx=ctx, part=p, n_parts=8)
    little = _new()
    torch.cuda.empty_cache()
    hold = torch.empty(max(_free() - 150_000_000, 0), dtype=torch.uint8, device="cuda")
    kiwi.sph_to_grid_device(P, BOUNDS, SHAPE, little, ctx=ctx)
    del hold
    torch.cuda.empty_cache()
    assert all(torch.equal(little[k], parts[k]) for k in little)
    two = [_new(), _new()]
    b = kiwi.Batch([{"particles": P, "bounds": BOUNDS, "shape": SHAPE, "out": o} for o in two], ctx=kiwi.Context(0))
    for _ in range(2):
        for o in two:
            for k in o:
                o[k].fill_(np.nan)
        torch.cuda.synchronize()
        b.run()
        assert all(torch.equal(o[k], parts[k]) for o in two for k in o)
    b.close()


def test_table_blocks_are_given_back(kiwi):
    """The tabulated integral's block copy of the table (0.73 GB) makes way for a call's own scratch: 5 M particles with
    300 MB left map as with all the memory."""
    n, shape = 5_000_000, (64, 64, 64)
    g = torch.Generator(device="cuda").manual_seed(3)
    P = {k: torch.rand(n, dtype=torch.float64, device="cuda", generator=g) for k in ("x", "y", "z", "vx", "vy", "vz", "m")}
    P["h"] = torch.full((n,), 1e-3, dtype=torch.float64, device="cuda")
    ki = kiwi.make_kernel_integrator("cubic_spline", use_tabulated_integral=True)

    def density(Q, ctx, out):
        kiwi.sph_to_grid_device(Q, (0.0, 1.0) * 3, shape, {"density": out}, kernel=ki, ctx=ctx)
        torch.cuda.synchronize()
        return out

    outs = [torch.empty(64 ** 3, dtype=torch.float64, device="cuda") for _ in range(2)]
    want = density(P, kiwi.Context(0), outs[0])
    ctx = kiwi.Context(0)
    density({k: v[:1000].contiguous() for k, v in P.items()}, ctx, outs[1])
    torch.cuda.empty_cache()
    hold = torch.empty(max(_free() - 300_000_000, 0), dtype=torch.uint8, device="cuda")
    got = density(P, ctx, outs[1])
    del hold
    torch.cuda.empty_cache()
    assert torch.equal(got, want)
