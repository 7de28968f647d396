"""The weight gradient's long sums.  The tensor core truncates when it adds to its
accumulator, so its error grows with the number of additions in a row; the kernel drains
the accumulators every 64 at most."""
import numpy as np
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


def test_long_sums_do_not_drift(gpu):
    from fluid_simulator_gb300 import native as N

    n, d, h, w, c = 8, 64, 64, 64, 16
    vox = n * d * h * w
    gen = torch.Generator().manual_seed(4)
    x, g = (torch.randn((vox, c), generator=gen).bfloat16().float() for _ in range(2))
    dw = N.net_conv(27, 2, x.numpy(), None, g.numpy(), shape=(n, d, h, w), cin=c, cout=c).astype(np.float64)
    xt = F.pad(x.view(n, d, h, w, c), (0, 0) + (1, 1) * 3).double()
    gt = g.double()
    ref = np.empty((27, c, c))
    for t in range(27):
        a, b, e = t // 9, t // 3 % 3, t % 3
        ref[t] = (gt.t() @ xt[:, a:a + d, b:b + h, e:e + w].reshape(vox, c)).numpy()
    err = dw - ref
    # An addition to a partial sum s truncates by 2^-24 |s| on average.  16 products of unit variance
    # an addition, |s| ~ 4 sqrt(k) after k: a chain of K is off by 2^-24 * 4 * (2/3) K^1.5, with its sum's
    # sign.  2 M voxels over 152 CTAs, two planes to an addition, are 432 each: as chains of 32 the 2,000
    # errors of 2.9e-5 add up to 1.3e-3 (RMS), as one chain the 152 of 1.4e-3 to 1.8e-2.  The FP32 sums
    # of the chains are below that.  Bounds: three times the first, a fifth of the second; extremes of
    # 6,912 values at four times that.
    assert np.sqrt((err ** 2).mean()) <= 4e-3
    assert np.abs(err).max() <= 1.6e-2
