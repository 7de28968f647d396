"""The multigrid preconditioner's coarse operator and interpolation on shapes
where they can go wrong: odd and flat grids (a coarse cell with one child per
axis), obstacles (partly closed coarse faces), porous masks (coarse cells cut by
the free surface everywhere), grids with and without separately launched coarse
levels.  The pressure is checked against the all-FP64 red-black IC solve, which
does not use the hierarchy; the iteration count shows that the cycle converges
as multigrid should (about one decade per 1.5 iterations, whatever the size)."""
import numpy as np
import pytest

from fluid_simulator_gb300 import native as N

pytestmark = pytest.mark.gpu


def problem(shape, kind, seed):
    """Cell types (solid walls) and a random right-hand side on the fluid cells."""
    rng = np.random.default_rng(seed)
    flags = np.full(shape, N.SOLID, np.uint8)
    inner = flags[1:-1, 1:-1, 1:-1]
    inner[...] = N.AIR
    x, y, z = np.meshgrid(*[(np.arange(1, n - 1) + 0.5) / n for n in shape], indexing="ij")
    if kind == "mask":
        f = rng.standard_normal(inner.shape)
        for a in range(3):
            f = f + np.roll(f, 1, a) + np.roll(f, 2, a)
        inner[f > np.median(f)] = N.WATER  # never all fluid: that has no solution
    else:
        inner[y < 0.55 + 0.1 * np.sin(7 * x) * np.cos(9 * z)] = N.WATER
    if kind == "obstacle":
        inner[(x - 0.5) ** 2 + (y - 0.4) ** 2 + (z - 0.5) ** 2 < 0.2 ** 2] = N.SOLID
        inner[(np.abs(x - 0.3) < 0.02) & (y < 0.4)] = N.SOLID  # a thin wall
    rhs = np.where(flags == N.WATER, rng.standard_normal(shape), 0.0)
    return flags, rhs


@pytest.mark.parametrize("kind", ["surface", "obstacle", "mask"])
@pytest.mark.parametrize("shape", [(5, 5, 5), (9, 33, 18), (33, 34, 35), (64, 17, 40), (71, 45, 50), (96, 96, 96)])
def test_multigrid_converges_at_any_shape(gpu, shape, kind):
    flags, rhs = problem(shape, kind, sum(shape))
    h = 1.0 / max(shape)
    prm = N.default_params(resolution=max(shape), tol=1e-9, tol_mode=N.TOL_REL_L2, max_iters=4000)
    sim = N.Simulation(max(shape), prm, dims=[(n + 0.01) * h for n in shape])
    assert sim.shape == shape
    sim.set_grid(N.F_FLAGS, flags)
    dt = h * h  # scale 1
    p, s = sim.solve_pressure(rhs, dt, precision=N.PREC_MIXED, tol=1e-9, max_iters=400)
    q, t = sim.solve_pressure(rhs, dt, precision=N.PREC_FP64, tol=1e-10, max_iters=4000)
    assert s.converged and t.converged
    # relative residual 1e-9 bounds the relative error by 1e-9 times the condition number (< 1e4 at 96 cells)
    assert np.abs(p - q).max() <= 1e-5 * np.abs(q).max()
    # nine decades in at most 24 iterations (the shapes above take 6 to 16)
    assert s.pcg_iterations <= 24, s.pcg_iterations
    sim.close()
