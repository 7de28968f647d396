"""Frames that are all spray, with particle counts at which a block gathers 256, 512 and
768 particles (eight blocks per SM first) and the last block is partly filled, against
the oracle's depth: the spray is drawn on the smoothed surface, here the empty one."""
import numpy as np
import pytest

from fluid_simulator_gb300 import native as N
from oracle import oracle as O
from test_render import scene_camera

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 255, 257, 5000, 400001, 700001])
def test_all_spray(gpu, port_lib, n):
    w, h = 96, 72
    rng = np.random.default_rng(n)
    pts = rng.random((n, 5)).astype(np.float32)
    pts[:, 4] = 0.5
    cam = scene_camera(w, h)
    prm = N.default_render_params(particle_radius=1 / 48, smoothing_size=0.05, transparency_blur_size=0.05)
    r = N.Renderer(w, h)
    r.frame(pts, cam, prm)
    ref = O.render_frame(pts, cam, prm, w, h)
    assert np.all(r.read(N.IMG_RAW_DEPTH) == 1.0)
    assert np.array_equal(r.read(N.IMG_DEPTH), ref["depth"])
    r.close()
