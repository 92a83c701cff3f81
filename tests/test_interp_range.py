"""The separable interpolation carries images as FP16 hi/lo planes of their own
scale, so they keep FP32's range, and ILT gradients are FP32 throughout: inputs
scaled by a power of two give the same bits, scaled (every other operation is
FP32 and far from its limits)."""
import numpy as np
import pytest

import highuvlith_b200 as HB
from highuvlith_b200 import ilt

pytestmark = pytest.mark.gpu


def _engine(n, flare=0.0):
    return HB.SimulationEngine(HB.SourceConfig.euv(0.5), HB.OpticsConfig(0.33, flare, 1.0, "euv"),
                               grid=HB.GridConfig(n, 1.0), max_kernels=8)


def _maps(n, clips):
    import torch
    rng = np.random.default_rng(n)
    m = rng.integers(0, 2, (clips, n // 16, n // 16)).repeat(16, 1).repeat(16, 2)
    return torch.from_numpy((0.1 + 0.8 * m + 0.05 * rng.random(m.shape)).astype(np.float32)).cuda()


# 256: narrow-band field kernel; 1024: 160-point register-radix field pass
@pytest.mark.parametrize("dtype", ["float32", "complex64"])
@pytest.mark.parametrize("power", [-45, -36, 20])
@pytest.mark.parametrize("n", [256, 1024])
def test_images(n, power, dtype):
    import torch
    eng, x = _engine(n, 0.03), _maps(n, 2).to(getattr(torch, dtype))
    ref = eng.compute_batch(x, pixel_transfer=False).double()
    out = eng.compute_batch(x * 2.0 ** power, pixel_transfer=False).double()
    assert torch.equal(out * 2.0 ** (-2 * power), ref)


@pytest.mark.parametrize("power", [-30, -22, 15])
@pytest.mark.parametrize("n", [256, 512, 1024])
def test_gradients(n, power):
    """Image cost against a zero target without regularisers: dC/dtheta is
    proportional to the dose squared."""
    import torch
    eng, theta = _engine(n), _maps(n, 2) - 0.5
    grads = [ilt.cost_and_gradient(eng, theta, torch.zeros_like(theta),
                                   ilt.IltSettings(cost="image", regularization=0.0, dose=d))[1].double()
             for d in (1.0, 2.0 ** power)]
    assert torch.equal(grads[1] * 2.0 ** (-2 * power), grads[0])
