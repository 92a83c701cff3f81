"""The ILT gradient on the evaluation grids whose images go through the tcgen05
interpolation (128 and 160, output grids that are multiples of 256), against
the FP64 objective (oracle/ilt.py), at both ends of the bands that these grids
serve, with one kernel and with several.

Tolerance as in tests/test_ilt_small.py: FP32 transforms through a resist
sigmoid of steepness 25, 1e-4 of the largest gradient."""
import numpy as np
import pytest

import highuvlith_b200 as HB
from highuvlith_b200 import ilt
from oracle import ilt as OI

pytestmark = pytest.mark.gpu


def _case(n, pixel, kernels, masks, flare):
    eng = HB.SimulationEngine(HB.SourceConfig.euv(0.5), HB.OpticsConfig(0.33, flare, 1.0, "euv"),
                              grid=HB.GridConfig(n, pixel), max_kernels=kernels, source_points_per_axis=17)
    rng = np.random.default_rng(n + kernels)
    target = rng.integers(0, 2, (masks, n // 16, n // 16)).repeat(16, 1).repeat(16, 2).astype(np.float32)
    theta = (target - 0.5 + 0.1 * rng.standard_normal(target.shape)).astype(np.float32)
    return eng, theta, target


@pytest.mark.parametrize("n,pixel,h,kernels,masks,focus,flare", [
    (512, 0.87, 16, 1, 3, 0.0, 0.0), (512, 1.65, 30, 1, 2, 0.0, 0.04), (512, 1.77, 33, 1, 3, 20.0, 0.0),
    (512, 2.09, 39, 1, 2, 0.0, 0.0), (512, 0.87, 16, 5, 1, 30.0, 0.0), (256, 3.55, 33, 6, 2, 0.0, 0.0)])
def test_gradient_matches_the_fp64_objective(n, pixel, h, kernels, masks, focus, flare):
    import torch
    eng, theta, target = _case(n, pixel, kernels, masks, flare)
    assert eng.imaging_diagnostics()["band_half_width"] == h
    st = ilt.IltSettings(cost="resist", threshold=0.3, steepness=25.0, defocus_nm=focus)
    cost, grad = ilt.cost_and_gradient(eng, torch.from_numpy(theta).cuda(), torch.from_numpy(target).cuda(), st)
    ev, ker = eng.kernels(focus)
    cfg = OI.IltConfig(cost="resist", threshold=0.3, steepness=25.0, flare=flare)
    for m in {0, masks - 1}:
        c, g = OI.IltProblem(ev, ker, target[m], cfg).cost_and_gradient(theta[m].astype(np.float64))
        assert abs(cost[m] - c) <= 1e-5 * c
        assert np.max(np.abs(grad[m].cpu().numpy() - g)) <= 1e-4 * np.max(np.abs(g)), m
