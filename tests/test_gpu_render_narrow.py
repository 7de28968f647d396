"""Near and far planes within a thousandth of each other and sprites of a ten-thousandth:
window depths come out of differences of large products, so their rounding is far above
the depth of a sprite.  The tests for hidden fragments and for sprites between the planes
must leave the sprite depth as it is, bit for bit."""
import numpy as np
import pytest

from fluid_simulator_gb300 import native as N
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("near,far", [(2.4, 2.402), (2.4, 2.41), (2.4, 2.5), (0.05, 20.0)])
def test_depth_with_a_narrow_range(gpu, port_lib, near, far):
    w, h, n, r = 67, 61, 4000, 1e-4
    rng = np.random.default_rng(int(far * 1000))
    half = 2.4 * np.tan(np.radians(0.02))
    pts = np.empty((n, 5), np.float32)
    pts[:, :2] = rng.uniform(-half, half, (n, 2))
    pts[:, 2] = -rng.uniform(2.4005, 2.4015, n)
    pts[: n // 4, 2] = -rng.uniform(near - 2 * r, near + 2 * r, n // 4)  # cut by the near plane
    pts[n // 4 : n // 2, 2] = -rng.uniform(far - 2 * r, far + 2 * r, n // 4)
    pts[:, 3], pts[:, 4] = 0.0, 8.0
    cam = N.camera((0.0, 0.0, 0.0), -90.0, 0.0, fov=0.04, aspect=w / h, near=near, far=far)
    prm = N.default_render_params(particle_radius=r, smoothing_size=4e-4, transparency_blur_size=4e-4)
    rr = N.Renderer(w, h)
    rr.frame(pts, cam, prm)
    ref = O.render_frame(pts, cam, prm, w, h)
    raw = rr.read(N.IMG_RAW_DEPTH)
    rr.close()
    assert (ref["raw_depth"] < 1).mean() > 0.5
    assert np.array_equal(raw, ref["raw_depth"])
