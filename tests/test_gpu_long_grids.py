"""The multigrid solve on long thin grids, whose small levels halve along one axis only:
all of them together do not fit one CTA's shared memory, although each does.  Against
the all-FP64 red-black IC solve."""
import numpy as np
import pytest

from fluid_simulator_gb300 import native as N
from test_gpu_multigrid import problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(3, 3, 16384), (3, 8192, 3), (3, 16384, 8), (8192, 3, 3), (4, 4, 16001)])
def test_solve_on_long_thin_grids(gpu, shape):
    rng = np.random.default_rng(7)
    flags = np.full(shape, N.SOLID, np.uint8)
    inner = flags[1:-1, 1:-1, 1:-1]
    # an air cell among eight on average: short runs of fluid, so the problem is well conditioned
    inner[...] = np.where(rng.random(inner.shape) < 0.125, N.AIR, N.WATER)
    rhs = np.where(flags == N.WATER, rng.standard_normal(shape), 0.0)
    h = 1.0 / max(shape)
    prm = N.default_params(resolution=max(shape), tol=1e-9, tol_mode=N.TOL_REL_L2, max_iters=4000)
    sim = N.Simulation(max(shape), prm, dims=[(n + 0.01) * h for n in shape])
    assert sim.shape == shape
    sim.set_grid(N.F_FLAGS, flags)
    p, s = sim.solve_pressure(rhs, h * h, precision=N.PREC_MIXED, tol=1e-9, max_iters=400)
    q, t = sim.solve_pressure(rhs, h * h, precision=N.PREC_FP64, tol=1e-11, max_iters=4000)
    assert s.converged and t.converged
    # runs of fluid between air cells are below 150 cells long (probability 1e-5 among 16384):
    # condition number of their chains below 150^2
    assert np.abs(p - q).max() <= 1e-9 * 150 ** 2 * np.abs(q).max()
    sim.close()


@pytest.mark.parametrize("kind", ["surface", "mask"])
@pytest.mark.parametrize("shape", [(10, 200, 200), (8, 128, 256), (20, 150, 150), (9, 180, 130)])
def test_solve_on_thin_boxes(gpu, shape, kind):
    """Small levels thin in x: their slabs of the thread-block cluster's shared memory are too
    large, so the cluster runs them in global memory."""
    flags, rhs = problem(shape, kind, sum(shape))
    h = 1.0 / max(shape)
    prm = N.default_params(resolution=max(shape), tol=1e-9, tol_mode=N.TOL_REL_L2, max_iters=4000)
    sim = N.Simulation(max(shape), prm, dims=[(n + 0.01) * h for n in shape])
    assert sim.shape == shape
    sim.set_grid(N.F_FLAGS, flags)
    p, s = sim.solve_pressure(rhs, h * h, precision=N.PREC_MIXED, tol=1e-9, max_iters=400)
    q, t = sim.solve_pressure(rhs, h * h, precision=N.PREC_FP64, tol=1e-10, max_iters=4000)
    sim.close()
    assert s.converged and t.converged
    # condition number below 10 * 200^2 (the longest axis and its open faces)
    assert np.abs(p - q).max() <= 4e-4 * np.abs(q).max()
    assert s.pcg_iterations <= 24  # nine decades, as on other boxes
