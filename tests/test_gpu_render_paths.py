"""The renderer's shortcuts against the oracle: image sizes that are no multiple of the
shading tiles (32 x 8), particle counts around the spray gather (2048), a near plane
that cuts through the fluid (clip tests and depths on both sides of it), an orthographic
projection (no shortcut applies) and a scene depth.  The depth is bit-exact, thickness
sums run in any order (1e-5 of the largest)."""
import numpy as np
import pytest

from fluid_simulator_gb300 import native as N
from oracle import oracle as O
from test_render import scene_camera, scene_particles

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,n,view,spray,scene", [
    (33, 9, 2047, "far", 1, False), (64, 8, 2049, "far", 1, True), (97, 41, 4097, "near", 1, False),
    (161, 121, 12000, "near", 0, True), (70, 50, 9000, "ortho", 1, False), (31, 7, 1, "far", 1, False)])
def test_splat_paths(gpu, port_lib, w, h, n, view, spray, scene):
    import torch

    pts = scene_particles(seed=n)[:n]
    cam = scene_camera(w, h)
    if view == "near":  # the eye is ~2.3 away from the middle of the fluid
        eye = (1.6, 1.1, 2.0)
        yaw, pitch = N.look_at_angles(eye, (0.4, 0.3, 0.5))
        cam = N.camera(eye, yaw, pitch, fov=40.0, aspect=w / h, near=2.2, far=2.6)
    if view == "ortho":  # 1.5 x 1.5 units, depth 0.05 .. 20
        P = np.diag([1 / 0.75, 1 / 0.75, -2 / 19.95, 1.0])
        P[2, 3] = -20.05 / 19.95
        cam.proj[:] = P.T.ravel().astype(np.float32).tolist()
        cam.proj_inv[:] = np.linalg.inv(P).T.ravel().astype(np.float32).tolist()
    prm = N.default_render_params(particle_radius=1 / 48, smoothing_size=0.05, transparency_blur_size=0.05,
                                  spray_enabled=spray, noise_scale=9.0, background=(0.1, 0.2, 0.3, 1.0))
    sd = None
    if scene:
        sd = np.ones((h, w), np.float32)
        sd[:, : w // 2] = 0.97
    r = N.Renderer(w, h)
    r.frame(pts, cam, prm, **({"scene_depth": torch.from_numpy(sd).cuda()} if scene else {}))
    ref = O.render_frame(pts, cam, prm, w, h, **({"scene_depth": sd} if scene else {}))
    assert np.array_equal(r.read(N.IMG_RAW_DEPTH), ref["raw_depth"])
    th, scale = r.read(N.IMG_THICKNESS), float(ref["thickness"].max())
    # (a kernel size on the other side of an integer: the shaders' int(extent * width))
    assert (np.abs(th - ref["thickness"]) > 1e-5 * max(scale, 1e-30)).mean() <= 0.002
    bad = np.abs(r.read(N.IMG_COLOR) - ref["color"]).max(axis=-1) > 2e-3
    assert bad.mean() <= 0.005
    r.close()
