"""The narrow-band ILT adjoint (ilt_adj_small, csrc/cuda/field_small.cu) on its
three grids at their widest bands, against the FP64 objective
(oracle/ilt.py): kernel counts that leave a round or a cluster block short, in
focus (folded kernels) and out of focus (the set itself), with flare.

Tolerance: FP32 transforms (errors of a few 1e-6 of the largest value each way)
through a resist sigmoid of steepness 25, whose slope multiplies the image
error by up to 25/4: 1e-4 of the largest gradient."""
import numpy as np
import pytest

import highuvlith_b200 as HB
from highuvlith_b200 import ilt
from oracle import ilt as OI

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pixel,h,kernels,masks,focus,flare", [
    (0.34, 3, 31, 2, 0.0, 0.0), (0.34, 3, 5, 1, 20.0, 0.0), (0.79, 7, 9, 3, 0.0, 0.04), (0.79, 7, 1, 1, 0.0, 0.0),
    (1.65, 15, 20, 2, 0.0, 0.0), (1.65, 15, 7, 1, 30.0, 0.04), (1.0, 9, 12, 150, 0.0, 0.0)])
def test_adjoint_matches_the_fp64_objective(pixel, h, kernels, masks, focus, flare):
    import torch
    n = 256
    eng = HB.SimulationEngine(HB.SourceConfig.euv(0.5), HB.OpticsConfig(0.33, flare, 1.0, "euv"),
                              grid=HB.GridConfig(n, pixel), max_kernels=kernels)
    assert eng.imaging_diagnostics()["band_half_width"] == h
    rng = np.random.default_rng(kernels)
    target = rng.integers(0, 2, (masks, n // 16, n // 16)).repeat(16, 1).repeat(16, 2).astype(np.float32)
    theta = (target - 0.5 + 0.1 * rng.standard_normal(target.shape)).astype(np.float32)
    st = ilt.IltSettings(cost="resist", threshold=0.3, steepness=25.0, defocus_nm=focus)
    cost, grad = ilt.cost_and_gradient(eng, torch.from_numpy(theta).cuda(), torch.from_numpy(target).cuda(), st)
    ev, ker = eng.kernels(focus)
    cfg = OI.IltConfig(cost="resist", threshold=0.3, steepness=25.0, flare=flare)
    for m in {0, masks - 1}:
        c, g = OI.IltProblem(ev, ker, target[m], cfg).cost_and_gradient(theta[m].astype(np.float64))
        assert abs(cost[m] - c) <= 1e-5 * c
        assert np.max(np.abs(grad[m].cpu().numpy() - g)) <= 1e-4 * np.max(np.abs(g)), m
