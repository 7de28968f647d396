"""What a frame costs follows from what it shows: device times of frames that differ in one
thing, the least of many, on an otherwise idle GPU.  The bounds leave room for noise; the
faults they are set against cost factors of 1.2 and more."""
import numpy as np
import pytest

from fluid_simulator_gb300 import native as N

pytestmark = pytest.mark.gpu


def frame_ms(r, pts, cam, prm, frames=30):
    ms = []
    for _ in range(frames):
        r.frame(pts, cam, prm)
        ms.append(r.stats()[0])
    return min(ms)


def camera(w, h, eye=(2.5, 1.7, 2.8)):
    yaw, pitch = N.look_at_angles(eye, (0.5, 0.5, 0.5))
    return N.camera(eye, yaw, pitch, fov=40.0, aspect=w / h, near=0.05, far=60.0)


def test_background_costs_no_weights(gpu):
    """An empty frame: the Gaussian filter, whose weights are 676 exponentials, costs what the
    bilateral one with 36 does (1.3 with a table per block)."""
    w, h = 3840, 2160
    r = N.Renderer(w, h)
    none = np.zeros((0, 5), np.float32)
    g, b = (frame_ms(r, none, camera(w, h), N.default_render_params(bilateral_filter=f)) for f in (0, 1))
    r.close()
    assert g <= 1.1 * b


def test_spray_costs_what_surface_does(gpu):
    """2048 sprites as spray and as surface (spray: 5 times as long from one block)."""
    rng = np.random.default_rng(2)
    r = N.Renderer(1000, 1000)
    prm = N.default_render_params(particle_radius=0.02, smoothing_size=0.06, transparency_blur_size=0.06)
    pts = rng.random((2048, 5)).astype(np.float32)
    ms = []
    for density in (0.0, 8.0):
        pts[:, 4] = density
        ms.append(frame_ms(r, pts, camera(1000, 1000), prm))
    r.close()
    assert ms[0] <= 1.5 * ms[1]


def test_few_sprites_cost_the_same_in_a_large_frame(gpu):
    """What a thousand sprites of a pixel or two add to an empty frame does not grow with the
    frame (16 times the pixels; with an eye ray tabulated for every pixel it did)."""
    prm = N.default_render_params(particle_radius=0.001, smoothing_size=0.06, transparency_blur_size=0.06)
    pts = np.random.default_rng(4).random((1000, 5)).astype(np.float32)
    pts[:, 4] = 8.0
    add = []
    for w, h in ((960, 540), (3840, 2160)):
        r = N.Renderer(w, h)
        some, none = (frame_ms(r, q, camera(w, h), prm) for q in (pts, pts[:0]))
        add.append(some - none)
        r.close()
    assert add[1] <= 3 * add[0]
