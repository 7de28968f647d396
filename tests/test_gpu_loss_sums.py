"""The loss's sums of squares against FP64, for targets from 1e-18 to 1e18 (squares and
sums that FP32 does not hold) and for samples and volumes around the kernel's blocks of
512 voxels.  The untrained network predicts zero, so the residual is the target's."""
import numpy as np
import pytest
import torch

import net_ref
from fluid_simulator_gb300 import native as N

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 8, 8, 8), (3, 8, 16, 24), (2, 24, 8, 40)])
@pytest.mark.parametrize("scale", [1e-18, 1e-15, 1.0, 1e15, 1e18])
def test_loss_of_the_zero_guess(gpu, shape, scale):
    rng = np.random.default_rng(5)
    kind = rng.integers(0, 3, shape)
    x = np.zeros(shape + (4,), np.float32)
    x[..., 0] = np.where(kind == 0, rng.standard_normal(shape), 0)
    for k in range(3):
        x[..., 1 + k] = kind == (0, 2, 1)[k]
    m = (kind == 0).astype(np.uint8)
    t = np.where(kind == 0, rng.standard_normal(shape) * scale, 0).astype(np.float32)
    net = N.WarmStartNet(seed=1)
    assert np.all(net.forward(x, train=True) == 0)
    loss = net.backward(t, m)
    net.close()
    b = torch.tensor(x[..., 0]).bfloat16().double().numpy() * m
    r = net_ref.operator(-torch.tensor(t).double(), torch.tensor(m).double(), torch.tensor(x[..., 2]).double()).numpy()
    ax = (1, 2, 3)
    ref = float((np.sqrt((r ** 2).sum(ax)) / np.sqrt((b ** 2).sum(ax)) + 0.1).mean())
    # each residual is a sum of seven FP32 terms (below 8 * 2^-24 of the largest, independent over
    # the voxels); the loss itself comes back in FP32
    assert abs(loss - ref) <= 1e-6 * ref
