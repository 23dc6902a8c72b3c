"""Gradients of particles that lie on planes of the grid (a lattice of particles aligned with it, an ordinary initial
condition), against central differences of the forward pass (test_gpu_adjoint.py's recipe and tolerance)."""
import numpy as np
import pytest

from test_gpu_adjoint import FD_TOL, KEYS, _dev, _fd, _one, _rel_errors

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("kernel", ["cubic_spline", "quartic_spline", "quintic_spline", "wendland_c2", "wendland_c4",
                                    "wendland_c6"])
def test_particles_on_planes(kiwi, ctx, kernel):
    """Particles on one, two and three planes of a grid of cell 1/8 (exact offsets of 0), on the planes between tiles, one
    an ulp off a plane, with supports within a cell and over many."""
    bounds, shape = (0.0, 2.0) * 3, (16, 16, 16)
    ki = kiwi.make_kernel_integrator(kernel)
    pos = [(0.75, 0.8, 0.9), (0.8, 1.0, 0.93), (0.77, 0.81, 1.125), (0.75, 0.875, 0.93), (1.0, 0.81, 1.0), (0.75, 1.0, 1.25),
           (1.0, 1.0, 1.0), (np.nextafter(0.75, 1.0), 1.0, 0.9)]
    P = {k: np.repeat(np.array([p[a] for p in pos]), 3) for a, k in enumerate(("x", "y", "z"))}
    rng = np.random.default_rng(6)
    n = len(P["x"])
    P.update({k: rng.standard_normal(n) for k in ("vx", "vy", "vz")})
    P["m"], P["h"] = rng.uniform(0.5, 1.5, n), np.tile([0.03, 0.11, 0.24], len(pos))
    cot = rng.standard_normal(4 * int(np.prod(shape)))
    Pd = _dev(P)
    g = {k: torch.empty_like(Pd[k]) for k in KEYS}
    kiwi.sph_to_grid_adjoint_device(Pd, bounds, shape, torch.tensor(cot, device="cuda"), g, kernel=ki, ctx=ctx)
    ad = {k: v.cpu().numpy() for k, v in g.items()}

    def loss(P1):
        return float(kiwi.sph_to_grid(P1, bounds, shape, kernel=ki, raw=True, ctx=ctx).raw.reshape(-1) @ cot)

    for i in range(n):
        assert max(_rel_errors(ad, _fd(loss, _one(P, i), float(P["h"][i])), i)) <= FD_TOL, i
