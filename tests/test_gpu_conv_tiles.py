"""The 3x3x3 convolution at the edges of its tiles: 8 (w) x 16 (h) x 2, 4 or 8 (d)
voxels and 16 to 64 output channels per CTA, chosen by size.  An input plane's
products go to three output planes at once, fewer at either end of a tile, so
volumes of 1 to 9 planes, ragged last tiles and neighbouring samples are drawn,
forward and input gradient (the same kernel with the taps reversed)."""
import numpy as np
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


def bf(a):
    return torch.tensor(np.asarray(a, np.float32)).bfloat16().float().numpy()


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("shape,cin,cout", [
    ((1, 1, 1, 1), 16, 16), ((2, 2, 8, 8), 16, 32), ((3, 3, 17, 9), 48, 48), ((2, 9, 16, 15), 32, 128),
    ((1, 40, 40, 41), 16, 16), ((1, 61, 70, 67), 16, 16), ((2, 63, 50, 45), 16, 48), ((1, 57, 66, 80), 32, 32),
    ((1, 16, 16, 16), 64, 64), ((1, 32, 31, 33), 64, 64), ((1, 33, 48, 64), 96, 32)])
def test_convolution_at_tile_edges(gpu, mode, shape, cin, cout):
    from fluid_simulator_gb300 import native as N

    rng = np.random.default_rng(sum(shape) + cin + mode)
    n, d, h, w = shape
    vox = int(np.prod(shape))
    kin, kout = (cin, cout) if mode == 0 else (cout, cin)
    a = bf(rng.standard_normal((vox, kin)))
    wgt = bf(rng.standard_normal((27, cout, cin)) * 0.1)
    y = N.net_conv(27, mode, *((a, wgt) if mode == 0 else (None, wgt, a)), shape=shape, cin=cin, cout=cout)
    k = torch.tensor(wgt).double().permute(1, 2, 0).reshape(cout, cin, 3, 3, 3)
    if mode == 1:  # correlation with the transposed, reversed taps
        k = k.transpose(0, 1).flip(2, 3, 4)

    def conv(u, v):
        return F.conv3d(u.view(n, d, h, w, kin).permute(0, 4, 1, 2, 3), v, padding=1).permute(0, 2, 3, 4, 1).reshape(vox, kout).numpy()

    x = torch.tensor(a).double()
    ref, size = conv(x, k), conv(x.abs(), k.abs())
    # products of BF16 values are exact in FP32; 27 kin additions, each off by at most 2^-23 of the
    # sum of sizes (the tensor core truncates); then one rounding to BF16 (2^-9 relative)
    assert (np.abs(y - ref) <= np.abs(ref) * 2.0 ** -8 + 27 * kin * 2.0 ** -23 * size + 1e-30).all()
