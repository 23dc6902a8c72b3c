"""Tiles whose particle lists are cut into segments (box_segment in csrc/box_tile.cuh): every entry point adds the
same numbers in the same order, and the sums agree with the reference-order form."""
import ctypes as C

import numpy as np
import pytest
from gpu_checks import assert_band_tolerance

pytestmark = pytest.mark.gpu


def _particles(torch, n, hmax, seed):
    rng = np.random.default_rng(seed)
    P = {k: rng.uniform(0.0, 1.0, n) for k in ("x", "y", "z")}
    P.update({k: rng.standard_normal(n) for k in ("vx", "vy", "vz")})
    P["m"], P["h"] = rng.uniform(0.5, 1.5, n), rng.uniform(0.03, hmax, n)
    return {k: torch.from_numpy(v).cuda() for k, v in P.items()}


# lists just below and above one segment of 128 entries, of several, and 40 k particles on one tile (the cap on the
# number of segments)
@pytest.mark.parametrize("kernel,n,shape", [("cubic_spline", 128, (8, 8, 8)), ("cubic_spline", 129, (8, 8, 8)),
                                            ("cubic_spline", 3000, (17, 16, 9)), ("wendland_c4", 900, (16, 16, 16)),
                                            ("cubic_spline", 40_000, (6, 7, 8))])
def test_entry_points_agree(kiwi, ctx, kernel, n, shape):
    import torch

    ki = kiwi.make_kernel_integrator(kernel)
    bounds, nc = (0.0, 1.0) * 3, int(np.prod(shape))
    dP = _particles(torch, n, 0.12 if n < 10_000 else 0.05, n)

    def new():
        out = {k: torch.full((nc,), np.nan, dtype=torch.float64, device="cuda") for k in ("density", "vx", "vy", "vz")}
        out["raw4"] = torch.full((4 * nc,), np.nan, dtype=torch.float64, device="cuda")
        return out

    torch.cuda.synchronize()
    whole = new()
    torch.cuda.synchronize()
    st = kiwi.sph_to_grid_device(dP, bounds, shape, whole, kernel=ki, ctx=ctx)
    parts, n_parts = new(), 3
    batch_out, na = new(), new()
    torch.cuda.synchronize()
    for p in range(n_parts):
        kiwi.sph_to_grid_device(dP, bounds, shape, parts, kernel=ki, ctx=ctx, part=p, n_parts=n_parts)
    batch = kiwi.Batch([{"particles": dP, "bounds": bounds, "shape": shape, "kernel": ki, "out": batch_out}], ctx=ctx)
    _, tot = batch.run()
    batch.close()
    f = kiwi.load_library().kiwi_sph_to_grid_device_noalloc
    f.restype = C.c_int
    f.argtypes = [C.c_void_p, C.POINTER(kiwi.KiwiParticles), C.POINTER(kiwi.KiwiCartGrid), C.POINTER(kiwi.KiwiKernelSel),
                  C.c_int] + [C.POINTER(C.c_double)] * 5 + [C.POINTER(kiwi.KiwiStats), C.c_char_p, C.c_size_t]
    Ps, _ = kiwi._particles_struct(dP, device=True)
    err = C.create_string_buffer(256)
    ptr = [C.cast(C.c_void_p(int(na[k].data_ptr())), C.POINTER(C.c_double)) for k in ("density", "vx", "vy", "vz", "raw4")]
    sel, stn = ki.sel(), kiwi.KiwiStats()
    rc = f(None, C.byref(Ps), C.byref(kiwi.KiwiCartGrid((C.c_double * 6)(*bounds), *shape)), C.byref(sel), kiwi.KIWI_FP64,
           *ptr, C.byref(stn), err, 256)
    torch.cuda.synchronize()
    assert rc == 0, err.value
    assert tot["sphere_pairs"] == st["sphere_pairs"] == stn.sphere_pairs
    for k in whole:
        assert not torch.isnan(whole[k]).any()
        for other in (parts, batch_out, na):
            assert torch.equal(other[k], whole[k]), k
    if n < 10_000:
        ref = new()
        torch.cuda.synchronize()
        kiwi.sph_to_grid_device(dP, bounds, shape, ref, kernel=ki, ctx=ctx, precision="fp64_reference_order")
        assert_band_tolerance(whole["density"].cpu().numpy(), ref["density"].cpu().numpy(), (4e-10, 4e-9, 1e-7))


def test_tabulated_parts_agree(kiwi, ctx):
    """The tabulated integral's tiles are cut the same way: parts equal the whole, and the whole agrees with the
    per-cell form to the rounding of the lookups' indices."""
    import torch

    ki = kiwi.make_kernel_integrator("cubic_spline", use_tabulated_integral=True)
    bounds, shape, n = (0.0, 1.0) * 3, (17, 16, 9), 3000
    nc = int(np.prod(shape))
    dP = _particles(torch, n, 0.12, 5)
    outs = []
    for parts, form in ((1, "fp64"), (3, "fp64"), (1, "fp64_reference_order")):
        out = {"density": torch.full((nc,), np.nan, dtype=torch.float64, device="cuda")}
        torch.cuda.synchronize()
        for p in range(parts):
            st = kiwi.sph_to_grid_device(dP, bounds, shape, out, kernel=ki, ctx=ctx, part=p, n_parts=parts, precision=form)
        outs.append((out["density"], st))
    assert torch.equal(outs[0][0], outs[1][0])
    assert_band_tolerance(outs[0][0].cpu().numpy(), outs[2][0].cpu().numpy(), (4e-10, 4e-9, 1e-7))


# small boxes (chunks of 32 entries), boxes that fill their tiles (chunks of two or three) and both mixed
@pytest.mark.parametrize("kernel", ["cubic_spline", "quintic_spline", "wendland_c4"])
@pytest.mark.parametrize("hmin,hmax", [(0.002, 0.02), (0.3, 0.5), (0.002, 0.5)])
def test_adjoint_does_not_depend_on_the_other_particles(kiwi, ctx, kernel, hmin, hmax):
    """At given cotangents a particle's gradient is its own entries' sums: the same bits whatever else is mapped."""
    import torch

    ki = kiwi.make_kernel_integrator(kernel)
    bounds, shape, n = (0.0, 1.0) * 3, (17, 16, 23), 200
    dP = _particles(torch, n, 0.5, 3)
    dP["h"] = hmin + (dP["h"] - dP["h"].min()) / 0.5 * (hmax - hmin)
    cot = torch.from_numpy(np.random.default_rng(4).standard_normal(4 * int(np.prod(shape)))).cuda()

    def gradients(P):
        g = {k: torch.full((P["x"].numel(),), np.nan, dtype=torch.float64, device="cuda") for k in P}
        torch.cuda.synchronize()
        kiwi.sph_to_grid_adjoint_device(P, bounds, shape, cot, g, kernel=ki, ctx=ctx)
        return g

    every = gradients(dP)
    assert all(torch.isfinite(v).all() for v in every.values())
    for idx in (slice(0, 1), slice(0, None, 7), slice(5, 120)):
        some = gradients({k: v[idx].contiguous() for k, v in dP.items()})
        for k in every:
            assert torch.equal(some[k], every[k][idx]), k
