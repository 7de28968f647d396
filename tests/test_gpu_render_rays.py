"""Eye rays: projections whose inverse keeps x and y apart (rays tabulated by axis) and
ones that do not (rolled, tilted), with few sprites and with many, against the oracle's
sprite depth bit for bit; the thickness sums run in any order."""
import numpy as np
import pytest

from fluid_simulator_gb300 import native as N
from oracle import oracle as O
from test_render import scene_camera

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("view", ["plain", "rolled", "tilted", "offset"])
@pytest.mark.parametrize("w,h,n", [(97, 63, 3000), (1, 40, 500), (64, 1, 500), (96, 64, 200001)])
def test_rays(gpu, port_lib, view, w, h, n):
    rng = np.random.default_rng(n)
    pts = rng.random((n, 5)).astype(np.float32)
    pts[:, 4] = 3.0 * rng.random(n)  # some below the spray threshold
    cam = scene_camera(w, h)
    P = np.array(cam.proj[:], np.float64).reshape(4, 4).T
    M = np.eye(4)
    c, s = np.cos(0.2), np.sin(0.2)
    if view == "rolled":
        M[:2, :2] = [[c, -s], [s, c]]
    if view == "tilted":
        M[1:3, 1:3] = [[c, -s], [s, c]]
    if view == "offset":  # an off-centre frustum
        M[0, 2], M[1, 2] = 0.1, -0.05
    if view != "plain":
        P = P @ M
        cam.proj[:] = P.T.ravel().astype(np.float32).tolist()
        cam.proj_inv[:] = np.linalg.inv(P).T.ravel().astype(np.float32).tolist()
    prm = N.default_render_params(particle_radius=1 / 40, smoothing_size=0.05, transparency_blur_size=0.05)
    r = N.Renderer(w, h)
    r.frame(pts, cam, prm)
    ref = O.render_frame(pts, cam, prm, w, h)
    raw = r.read(N.IMG_RAW_DEPTH)
    # (64 pixels of 1.8 units in one row: the centres miss most sprites)
    assert (h == 1 or (raw < 1).any()) and np.array_equal(raw, ref["raw_depth"])
    th = r.read(N.IMG_THICKNESS)
    assert (np.abs(th - ref["thickness"]) > 1e-5 * max(ref["thickness"].max(), 1e-30)).mean() <= 0.002
    r.close()


@pytest.mark.parametrize("bilateral", [0, 1])
def test_large_frame(gpu, port_lib, bilateral):
    """More pixels than two waves of blocks (a blur thread takes several), no multiple of a
    block's: mostly background, a few sprites."""
    w, h = 2051, 1303
    rng = np.random.default_rng(1)
    pts = (rng.random((60, 5)) * [1, 1, 1, 0, 3]).astype(np.float32)
    cam = scene_camera(w, h)
    prm = N.default_render_params(particle_radius=1 / 80, smoothing_size=0.02, transparency_blur_size=0.02,
                                  bilateral_filter=bilateral, noise_scale=9.0)
    r = N.Renderer(w, h)
    r.frame(pts, cam, prm)
    ref = O.render_frame(pts, cam, prm, w, h)
    assert np.array_equal(r.read(N.IMG_RAW_DEPTH), ref["raw_depth"])
    d = r.read(N.IMG_DEPTH)
    assert np.array_equal(d < 1, ref["depth"] < 1) and np.abs(d - ref["depth"]).max() <= 2e-6
    th = r.read(N.IMG_THICKNESS)
    assert (np.abs(th - ref["thickness"]) > 1e-5 * ref["thickness"].max()).mean() <= 0.001
    r.close()
