"""Sweep counts changed between the solves of one context: every solve runs the V-cycle
of its own counts, as a new context does, bit for bit (the solver is deterministic)."""
import numpy as np
import pytest

from fluid_simulator_gb300 import native as N

pytestmark = pytest.mark.gpu
SHAPE = (64, 64, 64)


def params(**kw):
    return N.default_params(resolution=64, tol=1e-6, tol_mode=N.TOL_REL_L2, max_iters=2000, **kw)


def solve(sim):
    rng = np.random.default_rng(1)
    flags = np.full(SHAPE, N.SOLID, np.uint8)
    flags[1:-1, 1:-1, 1:-1] = N.AIR
    flags[1:-1, 1:30, 1:-1] = N.WATER
    sim.set_grid(N.F_FLAGS, flags)
    for f in (N.F_V2X, N.F_V2Y, N.F_V2Z):
        sim.set_grid(f, rng.standard_normal(SHAPE))
    s = sim.solve_current(1.0 / 480, N.WARM_ZERO)
    assert s.converged
    return sim.grid(N.F_PRESSURE), s.pcg_iterations


@pytest.mark.parametrize("first,second", [
    (dict(mg_coarse_sweeps=1, mg_cluster_sweeps=100), dict(mg_coarse_sweeps=2)),
    (dict(precond=N.PRECOND_RBIC, mg_sweeps=100), dict()),
    (dict(mg_sweeps=1, mg_coarse_sweeps=2), dict()),
    (dict(mg_boundary_sweeps=2), dict(mg_boundary_sweeps=-1))])
def test_each_solve_uses_its_own_sweep_counts(gpu, first, second):
    sim = N.Simulation(64, params(**first))
    solve(sim)
    sim.set_params(params(**second))
    got = solve(sim)
    sim.close()
    new = N.Simulation(64, params(**second))
    want = solve(new)
    new.close()
    assert got[1] == want[1] and np.array_equal(got[0], want[0])
