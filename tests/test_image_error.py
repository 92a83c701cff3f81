"""Images of every evaluation grid of the narrow-band field kernel and of the
one-kernel interpolation against the same kernels summed in FP64 (numpy).

Tolerance: 1e-5 of the largest intensity, as for the FP32-FFT form in
tests/test_focus_sweep.py.  A dropped or misplaced plane of a split FP16
product is 2^-12 = 2.4e-4 of its operand, which the worst-case bounds of
tests/test_field_small.py and tests/test_interp_fused.py could hide."""
import numpy as np
import pytest

import highuvlith_b200 as HB

pytestmark = pytest.mark.gpu


def _fp64(eng, t, focus, flare):
    ev, ker = eng.kernels(focus)
    spec = np.fft.fft2(t.astype(np.complex128))
    img = sum(v * np.abs(np.fft.ifft2(k * spec)) ** 2 for v, k in zip(ev, ker))
    return (1.0 - flare) * img + flare * img.mean()


# n, pixel, grid (None: automatic), band half-width, kernels, focus, flare
@pytest.mark.parametrize("n,pixel,grid,h,kernels,focus,flare", [
    (256, 0.34, None, 3, 9, 0.0, 0.0), (256, 0.79, None, 7, 12, 25.0, 0.03), (256, 1.2, None, 11, 7, 0.0, 0.0),
    (256, 1.65, None, 15, 20, 0.0, 0.03), (256, 2.05, None, 19, 5, 40.0, 0.0), (256, 2.5, None, 23, 16, 0.0, 0.0),
    (256, 2.75, 128, 25, 8, 0.0, 0.0), (512, 1.65, 128, 30, 6, 30.0, 0.03), (256, 3.55, 160, 33, 8, 0.0, 0.0),
    (512, 2.09, 160, 39, 5, 0.0, 0.03), (1024, 1.0, 160, 37, 4, 20.0, 0.0), (1024, 1.0, 160, 37, 7, 0.0, 0.0)])
@pytest.mark.parametrize("dtype", ["float32", "complex64"])
def test_against_fp64(n, pixel, grid, h, kernels, focus, flare, dtype):
    import torch
    eng = HB.SimulationEngine(HB.SourceConfig.euv(0.5), HB.OpticsConfig(0.33, flare, 1.0, "euv"),
                              grid=HB.GridConfig(n, pixel), max_kernels=kernels, source_points_per_axis=13)
    assert eng.imaging_diagnostics()["band_half_width"] == h
    rng = np.random.default_rng(n + kernels)
    m = rng.integers(0, 2, (2, n // 8, n // 8)).repeat(8, 1).repeat(8, 2)
    t = (0.05 + 0.9 * m).astype(np.float32)
    if dtype == "complex64":
        t = (t * np.exp(0.4j * m)).astype(np.complex64)
    out = eng.compute_batch(torch.from_numpy(t).cuda(), focus_nm=focus, pixel_transfer=False,
                            **({} if grid is None else dict(form="hybrid", eval_grid=grid)))
    eng.device_status()
    for c in range(2):
        ref = _fp64(eng, t[c], focus, flare)
        assert np.max(np.abs(out[c].cpu().numpy() - ref)) < 1e-5 * np.max(ref)
