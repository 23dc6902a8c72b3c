"""Masses and velocities that are not finite show in the cells that their particle reaches, and nowhere else."""
import numpy as np
import pytest

from conftest import random_particles

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel", ["cubic_spline", "wendland_c4", "tabulated"])
@pytest.mark.parametrize("m,vx", [(np.nan, 0.5), (np.inf, 0.5), (1.0, np.nan), (1.0, np.inf), (0.0, np.nan)])
def test_values_that_are_not_finite(kiwi, ctx, kernel, m, vx):
    tabulated = kernel == "tabulated"
    shape, h, at = (20, 17, 9), 0.1, np.array([0.41, 0.52, 0.47])
    P = random_particles(40, 1, box=(0.0, 1.0), hmin=0.03, hmax=0.12)
    P["x"][3], P["y"][3], P["z"][3] = at
    P["h"][3], P["m"][3], P["vx"][3] = h, m, vx
    ki = kiwi.make_kernel_integrator("cubic_spline" if tabulated else kernel, use_tabulated_integral=tabulated)
    raw = kiwi.sph_to_grid(P, (0.0, 1.0) * 3, shape, kernel=ki, raw=True, ctx=ctx).raw
    # each cell's nearest and farthest distance from the particle, and its box of cells
    ax = [np.arange(k + 1) / k for k in shape]
    lo = np.meshgrid(*[np.maximum(np.maximum(a[:-1] - c, c - a[1:]), 0.0) for a, c in zip(ax, at)], indexing="ij")
    hi = np.meshgrid(*[np.maximum(abs(a[:-1] - c), abs(a[1:] - c)) for a, c in zip(ax, at)], indexing="ij")
    near, far = np.sqrt(sum(v * v for v in lo)).ravel(), np.sqrt(sum(v * v for v in hi)).ravel()
    outside = np.maximum(np.maximum(*lo[:2]), lo[2]).ravel() > 2 * h if tabulated else near > 2 * h
    inside = far < 1.9 * h
    assert inside.sum() > 20 and outside.sum() > 20
    assert np.isfinite(raw[:, outside]).all()
    assert np.isfinite(raw[2:]).all() == np.isfinite(m)
    assert not np.isfinite(raw[1][inside]).any()
    assert np.isfinite(raw[0][inside]).all() == np.isfinite(m)
