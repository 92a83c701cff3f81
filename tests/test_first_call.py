"""The first call of an engine or a network on a stream of its own (which does
not wait for the legacy stream that its tables are copied on) equals the later
ones bit for bit."""
import numpy as np
import pytest

import highuvlith_b200 as HB
from highuvlith_b200 import ilt
from highuvlith_b200.fno import FnoSurrogate

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,form,kernels", [(256, "auto", 20), (512, "fft", 30), (1024, "auto", 32), (512, "tc", 20),
                                            (2048, "auto", 48)])
def test_images(n, form, kernels):
    import torch
    st = torch.cuda.Stream()
    x = (torch.rand(1, n // 8, n // 8, device="cuda") > 0.5).to(torch.uint8).repeat_interleave(8, 1).repeat_interleave(8, 2)
    torch.cuda.synchronize()
    for _ in range(3):
        eng = HB.SimulationEngine(HB.SourceConfig(13.5, "annular", (0.4, 0.7)), HB.OpticsConfig.euv_nxe_033(),
                                  grid=HB.GridConfig(n, 1.0), max_kernels=kernels, source_points_per_axis=9)
        with torch.cuda.stream(st):
            first = eng.compute_batch(x, form=form, stream=st).clone()
            assert torch.equal(first, eng.compute_batch(x, form=form, stream=st))


def test_gradients_and_rectangles():
    import torch
    st = torch.cuda.Stream()
    theta = torch.rand(2, 256, 256, device="cuda") - 0.5
    target = (theta > 0).float()
    many = [[(float(i % 50) * 4 - 100, float(i // 50) * 4 - 90, 2.5, 3.0) for i in range(2100)]]  # resolved on the host
    torch.cuda.synchronize()
    for _ in range(3):
        eng = HB.SimulationEngine(HB.SourceConfig.euv(0.5), HB.OpticsConfig.euv_nxe_033(), grid=HB.GridConfig(256, 1.0),
                                  max_kernels=12)
        with torch.cuda.stream(st):
            a = eng.compute_batch_rects(many, stream=st).clone()
            assert torch.equal(a, eng.compute_batch_rects(many, stream=st))
            c0, g0 = ilt.cost_and_gradient(eng, theta, target, ilt.IltSettings(), stream=st)
            c1, g1 = ilt.cost_and_gradient(eng, theta, target, ilt.IltSettings(), stream=st)
            assert np.array_equal(c0, c1) and torch.equal(g0, g1)


@pytest.mark.parametrize("n", [64, 128])
def test_networks(n):
    import torch
    st = torch.cuda.Stream()
    x = torch.rand(2, n, n, device="cuda")
    torch.cuda.synchronize()
    for seed in range(3):
        f = FnoSurrogate(n, 8, 2, seed=seed)
        with torch.cuda.stream(st):
            first = f.forward(x, stream=st).clone()
            assert torch.equal(first, f.forward(x, stream=st))
