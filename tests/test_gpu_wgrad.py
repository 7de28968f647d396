"""The weight-gradient kernel at the edges of its tiles (8 x 16 x 4 voxels; 8 x 16 x 2
pointwise), chunks (32 input channels; 128 pointwise) and output splits: volumes
smaller than a tile, ragged on every axis, several samples (the planes of two
samples must not mix), several tiles per CTA, partly used channel chunks."""
import numpy as np
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


def bf(a):
    return torch.tensor(np.asarray(a, np.float32)).bfloat16().float().numpy()


@pytest.mark.parametrize("taps,shape,cin,cout", [
    (27, (1, 1, 1, 1), 16, 16), (27, (2, 1, 8, 8), 16, 16), (27, (3, 5, 17, 9), 16, 48), (27, (2, 4, 33, 24), 48, 16),
    (27, (5, 3, 16, 8), 80, 32), (27, (2, 40, 48, 40), 32, 64), (27, (2, 64, 64, 64), 16, 16),
    (1, (1, 1, 1, 1), 16, 16), (1, (3, 3, 17, 9), 144, 48), (1, (2, 5, 16, 10), 64, 64), (1, (2, 32, 32, 32), 128, 32)])
def test_weight_gradient_at_tile_edges(gpu, taps, shape, cin, cout):
    from fluid_simulator_gb300 import native as N

    rng = np.random.default_rng(sum(shape) + cin)
    n, d, h, w = shape
    vox = int(np.prod(shape))
    x, g = bf(rng.standard_normal((vox, cin))), bf(rng.standard_normal((vox, cout)))
    xt = F.pad(torch.tensor(x).view(n, d, h, w, cin), (0, 0) + (1, 1) * 3 if taps == 27 else (0, 0))
    gt = torch.tensor(g).view(vox, cout).double()
    ref = np.empty((taps, cout, cin))
    for t in range(taps):
        a, b, c = (t // 9, t // 3 % 3, t % 3) if taps == 27 else (0, 0, 0)
        sl = xt[:, a:a + d, b:b + h, c:c + w].reshape(vox, cin).double()
        ref[t] = (gt.t() @ sl).numpy()
    dw = N.net_conv(taps, 2, x, None, g, shape=shape, cin=cin, cout=cout).astype(np.float64)
    # products of BF16 values are exact in FP32; sums of vox terms of size ~1 in FP32, any order:
    # each rounding is below 2^-24 of a partial sum of size <~ 4 sqrt(vox)
    assert np.abs(dw - ref).max() <= 2.0 ** -24 * vox * 4 * np.sqrt(vox) / 16 + 1e-5
