"""The default (multigrid) solve on the smallest grids fsim_create takes, 3 or 4 cells
per axis, where the hierarchy has one coarse level of at most 2 cells per axis, against
the all-FP64 red-black IC solve, which does not use the hierarchy."""
import numpy as np
import pytest

from fluid_simulator_gb300 import native as N

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(3, 3, 3), (4, 4, 4), (3, 4, 4), (4, 3, 3), (3, 3, 4), (4, 4, 5)])
@pytest.mark.parametrize("hole", [False, True])
def test_solve_on_the_smallest_grids(gpu, shape, hole):
    rng = np.random.default_rng(sum(shape))
    flags = np.full(shape, N.SOLID, np.uint8)
    flags[1:-1, 1:-1, 1:-1] = N.WATER
    flags[1:-1, -1, 1:-1] = N.AIR  # open above: the problem has a solution for every right-hand side
    if hole:
        flags[1, 1, 1] = N.AIR if max(shape) > 3 else N.WATER
    rhs = np.where(flags == N.WATER, rng.standard_normal(shape), 0.0)
    h = 1.0 / max(shape)
    prm = N.default_params(resolution=max(shape), tol=1e-9, tol_mode=N.TOL_REL_L2, max_iters=200)
    sim = N.Simulation(max(shape), prm, dims=[(n + 0.01) * h for n in shape])
    assert sim.shape == shape
    sim.set_grid(N.F_FLAGS, flags)
    p, s = sim.solve_pressure(rhs, h * h, precision=N.PREC_MIXED, tol=1e-9, max_iters=200)
    q, t = sim.solve_pressure(rhs, h * h, precision=N.PREC_FP64, tol=1e-12, max_iters=200)
    assert s.converged and t.converged
    # at most 12 unknowns with a Dirichlet face each: condition number below 100; a relative
    # residual of 1e-9, and the result is read back in FP32
    assert np.abs(p - q).max() <= 1e-6 * np.abs(q).max()
    assert s.pcg_iterations <= 24
    sim.close()
