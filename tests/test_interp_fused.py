"""The one-kernel separable interpolation (csrc/cuda/interp_tc.cu) against the
plain FP32-FFT form of the same engine: one clip (row tiles split over CTAs),
odd counts and more than one wave of CTAs, the smallest and largest output
grids, evaluation grids with and without a half-filled last K box.

Tolerance: each of the two products errs by at most (3 2^-22 + n 2^-23) of
the sum of |P| over a row (FP16 hi/lo splits with lo.lo dropped, n = 3 M / 16
truncating accumulations), and that sum is below 5 for these Dirichlet
kernels: (7.2e-7 + 30 * 1.2e-7) (5 + 25) = 1.3e-4 of the largest intensity.
"""
import numpy as np
import pytest

import highuvlith_b200 as HB

pytestmark = pytest.mark.gpu

TOL = 1.3e-4


@pytest.mark.parametrize("n,pixel,grid,clips", [(256, 4.0, 160, 1), (256, 4.0, 160, 151), (512, 2.0, 160, 3),
                                                (1024, 1.0, 160, 1), (1024, 1.0, 160, 5), (2048, 0.5, 160, 2),
                                                (512, 1.0, 128, 7)])
def test_fused_interpolation_matches_fft_form(n, pixel, grid, clips):
    import torch
    eng = HB.SimulationEngine(HB.SourceConfig.euv(0.5), HB.OpticsConfig.euv_nxe_033(), grid=HB.GridConfig(n, pixel),
                              max_kernels=6)
    rng = np.random.default_rng(n + clips)
    x = torch.from_numpy(rng.integers(0, 2, (clips, n // 8, n // 8), dtype=np.uint8).repeat(8, 1).repeat(8, 2)).cuda()
    ref = eng.compute_batch(x, form="fft", eval_grid=n)
    out = eng.compute_batch(x, form="hybrid", eval_grid=grid)
    eng.device_status()
    err = (out - ref).abs().amax(dim=(1, 2)) / ref.amax(dim=(1, 2))
    assert float(err.max()) < TOL
