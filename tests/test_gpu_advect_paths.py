"""Advection's short path (particles that surely meet no wall and no obstacle) against
the general one.  A box sink that covers the whole box sends every particle through
the general path and, with despawning off, changes nothing: both runs must agree in
every bit.  Particles are drawn in the interior, on and around the walls' clamp band
and the obstacles' surfaces, at rest, slow, exactly reaching a wall and fast enough to
bounce several times."""
import numpy as np
import pytest

from fluid_simulator_gb300 import native as N

pytestmark = pytest.mark.gpu


def run(pos, vel, obstacles, dt, dims, transfer):
    p = N.default_params(resolution=32, transfer=transfer)
    p.despawning_enabled = 0
    sim = N.Simulation(32, p, dims=dims, track_ids=True)
    sim.set_particles(pos, vel)
    sim.set_obstacles(obstacles)
    sim.stage(N.STAGE_ADVECT, dt)
    out = sim.particles()
    sim.close()
    return [np.asarray(a) for a in out[:2]]


@pytest.mark.parametrize("dt", [0.0, 1.0 / 480.0, 1.0 / 60.0])
@pytest.mark.parametrize("dims", [(1.0, 1.0, 1.0), (1.3, 0.7, 0.9)])
@pytest.mark.parametrize("which", [(), ("sphere",), ("box",), ("sphere", "box", "source")])
def test_short_path_is_the_general_path(gpu, dt, dims, which):
    rng = np.random.default_rng(len(which) + int(dt * 1e4))
    d = np.array(dims)
    h = 1.0 / 32
    n = 4099
    pos = rng.uniform(1.2 * h, d - 1.2 * h, (n, 3))
    vel = rng.standard_normal((n, 3)) * rng.choice([0.0, 1e-7, 0.3, 2.0, 40.0], (n, 1))
    # on and around the walls, moving along, into and away from them
    wall = rng.integers(0, 3, n)
    for a in range(3):
        near = (rng.random(n) < 0.3) & (wall == a)
        band = h * 1.01 / 1.0 + rng.choice([0.0, 1e-7, 1e-4, 5e-3], n)
        pos[near, a] = np.where(rng.random(n) < 0.5, band, d[a] - band)[near]
    if dt > 0:  # a step ends on the wall, to rounding
        k = rng.random(n) < 0.1
        vel[k, 0] = (d[0] - 1.01 * h - pos[k, 0]) / dt
    obs = []
    c = d * 0.5
    if "sphere" in which:
        obs.append(N.obstacle(N.OBS_SPHERE, tuple(c), r=0.15, speed=(0.5, 0.0, -0.2)))
        k = rng.random(n) < 0.2
        u = rng.standard_normal((n, 3))
        u /= np.linalg.norm(u, axis=1)[:, None]
        pos[k] = (c + u * (0.15 + rng.choice([-0.05, 0.0, 0.005, 0.01], (n, 1))))[k]
    if "box" in which:
        b = d * np.array([0.25, 0.3, 0.7])
        obs.append(N.obstacle(N.OBS_BOX, tuple(b), size=(0.2, 0.1, 0.15), speed=(0.0, 0.4, 0.0)))
        k = rng.random(n) < 0.2
        pos[k] = (b + rng.uniform(-0.55, 0.55, (n, 3)) * np.array([0.22, 0.12, 0.17]))[k]
    if "source" in which:
        obs.append(N.obstacle(N.OBS_SOURCE, tuple(d * 0.75), r=0.08))
    pos = np.clip(pos, 1.0001 * h, d - 1.0001 * h).astype(np.float32)
    vel = vel.astype(np.float32)
    cover = N.obstacle(N.OBS_BOX_SINK, tuple(c), size=tuple(4 * d))
    short = run(pos, vel, obs, dt, dims, N.FLIP)
    general = run(pos, vel, obs + [cover], dt, dims, N.FLIP)
    for a, b in zip(short, general):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
