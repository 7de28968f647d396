"""Renderer records of particles outside the grid, up to positions whose cell index does
not fit 32 bits: the density is interpolated from the cells that exist, with the weights
of the formula, and is zero where there are none."""
import numpy as np
import pytest

from fluid_simulator_gb300 import native as N

pytestmark = pytest.mark.gpu


def test_density_outside_the_grid(gpu):
    shape, h = (5, 6, 7), np.float32(1 / 7)
    far = [-np.inf, -1e30, -2147483648.0 / 7, -2.0, -0.01, 0.0, 0.06, 0.5, 0.99, 1.02, 5.0, 2147483520.0 / 7,
           2147483648.0 / 7, 1e12, np.inf]
    rng = np.random.default_rng(3)
    pos = np.array([(x, y, z) for x in far for y in far for z in (0.4, 1.1, 3e38, np.inf, -1e9)], np.float32)
    pos = np.concatenate([pos, rng.uniform(-0.3, 1.3, (500, 3)).astype(np.float32)])
    sim = N.Simulation(7, N.default_params(resolution=7), dims=[(n + 0.01) / 7 for n in shape])
    assert sim.shape == shape
    avg = rng.uniform(1, 9, shape).astype(np.float32)
    sim.set_grid(N.F_AVGPNUM, avg)
    sim.set_particles(pos, np.zeros_like(pos))
    got = sim.gfx()[:, 4]
    sim.close()
    with np.errstate(over="ignore", invalid="ignore"):
        g = pos.astype(np.float64) * 7 - 0.5
        ref = np.zeros(len(pos))
        b = np.trunc(np.clip(g, -1e6, 1e6)).astype(np.int64)  # the int conversion, saturated
        for k in range(8):
            c = b + [k >> 2, (k >> 1) & 1, k & 1]
            ok = np.all((c >= 0) & (c < shape), axis=1)
            w = np.prod(1 - np.abs(g - c), axis=1)
            cc = np.where(ok[:, None], c, 0)
            ref[ok] += (w * avg[cc[:, 0], cc[:, 1], cc[:, 2]])[ok]
    # coordinates below 14 cells, FP32: each weight is off by up to 2^-20, eight cells of at most 9
    near = np.all(np.abs(pos) < 2.5, axis=1)
    assert near.sum() > 500 and np.abs(got - ref)[near].max() <= 8 * 9 * 27 * 2.0 ** -20
    assert np.all(got[~near & (ref == 0)] == 0)
