"""ILT gradients of bands wider than a block of the radix-4 adjoint (more than
256 orders), against the FP64 objective (oracle/ilt.py); tolerances as in
tests/test_ilt_small.py."""
import numpy as np
import pytest

import highuvlith_b200 as HB
from highuvlith_b200 import ilt
from oracle import ilt as OI

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pixel,kernels", [(10.0, 3), (12.0, 6)])
def test_gradient_matches_the_fp64_objective(pixel, kernels):
    import torch
    n = 512
    eng = HB.SimulationEngine(HB.SourceConfig.euv(0.5), HB.OpticsConfig(0.33, 0.0, 1.0, "euv"),
                              grid=HB.GridConfig(n, pixel), max_kernels=kernels, source_points_per_axis=9)
    assert 2 * eng.imaging_diagnostics()["band_half_width"] + 1 > 256
    rng = np.random.default_rng(kernels)
    target = rng.integers(0, 2, (2, n // 8, n // 8)).repeat(8, 1).repeat(8, 2).astype(np.float32)
    theta = (target - 0.5 + 0.1 * rng.standard_normal(target.shape)).astype(np.float32)
    st = ilt.IltSettings(cost="resist", threshold=0.3, steepness=25.0)
    cost, grad = ilt.cost_and_gradient(eng, torch.from_numpy(theta).cuda(), torch.from_numpy(target).cuda(), st)
    ev, ker = eng.kernels()
    cfg = OI.IltConfig(cost="resist", threshold=0.3, steepness=25.0)
    for m in range(2):
        c, g = OI.IltProblem(ev, ker, target[m], cfg).cost_and_gradient(theta[m].astype(np.float64))
        assert abs(cost[m] - c) <= 1e-5 * c
        assert np.max(np.abs(grad[m].cpu().numpy() - g)) <= 1e-4 * np.max(np.abs(g)), m
