"""The narrow-band field kernel (csrc/cuda/field_small.cu): every evaluation
grid 16 .. 96 at its widest band, kernel counts that leave a round or a
cluster block short, real and complex inputs, focus planes in one launch.

Against the plain FP32-FFT form on the full grid.  Tolerance as for the
interpolation it feeds (FP16 hi/lo operands, at most 18 truncating
accumulations per product, row sums of |P| below 5):
(7.2e-7 + 18 * 1.2e-7) (5 + 25) = 8.7e-5 of the largest intensity.
"""
import numpy as np
import pytest

import highuvlith_b200 as HB

pytestmark = pytest.mark.gpu

TOL = 8.7e-5


def _engine(pixel, kernels, n=256, optics=None):
    return HB.SimulationEngine(HB.SourceConfig.euv(0.5), optics or HB.OpticsConfig.euv_nxe_033(),
                               grid=HB.GridConfig(n, pixel), max_kernels=kernels)


def _clips(n, count, seed):
    import torch
    rng = np.random.default_rng(seed)
    return torch.from_numpy(rng.integers(0, 2, (count, n // 8, n // 8), dtype=np.uint8).repeat(8, 1).repeat(8, 2)).cuda()


# pixel size -> band half-width h = floor(0.33 * 1.5 / 13.5 * 256 * pixel), grid
# = the smallest multiple of 16 above 4h
@pytest.mark.parametrize("pixel,h,kernels,clips,focus", [
    (0.05, 0, 3, 1, 0.0), (0.34, 3, 31, 2, 0.0), (0.34, 3, 40, 1, 30.0), (0.79, 7, 5, 3, 0.0), (0.79, 7, 31, 1, 0.0),
    (1.2, 11, 1, 1, 0.0), (1.2, 11, 31, 5, 25.0), (1.65, 15, 20, 1, 0.0), (1.65, 15, 2, 150, 0.0),
    (2.05, 19, 26, 2, 0.0), (2.5, 23, 9, 3, 20.0)])
def test_every_grid_matches_fft_form(pixel, h, kernels, clips, focus):
    eng = _engine(pixel, kernels)
    assert eng.imaging_diagnostics()["band_half_width"] == h
    x = _clips(256, clips, clips + kernels)
    ref = eng.compute_batch(x, form="fft", eval_grid=256, focus_nm=focus)
    out = eng.compute_batch(x, focus_nm=focus)
    eng.device_status()
    assert float(((out - ref).abs().amax(dim=(1, 2)) / ref.amax(dim=(1, 2))).max()) < TOL
    # complex transmittance, and an image does not depend on its batch
    c = (x.float() - 0.3j * (1 - x.float()))[:1].contiguous()
    ref = eng.compute_batch(c, form="fft", eval_grid=256, focus_nm=focus, pixel_transfer=False)
    out1 = eng.compute_batch(c, focus_nm=focus, pixel_transfer=False)
    assert float((out1 - ref).abs().max() / ref.max()) < TOL
    assert bool((eng.compute_batch(x[-1:], focus_nm=focus) == out[-1:]).all())


def test_flare_and_normalisation_match_fft_form():
    eng = HB.SimulationEngine(HB.SourceConfig.arf_laser(0.7), HB.OpticsConfig(0.93, 0.05), grid=HB.GridConfig(512, 2.0),
                              max_kernels=12, normalization="absolute")
    x = _clips(512, 3, 5)
    ref = eng.compute_batch(x, form="fft", eval_grid=512)
    assert float((eng.compute_batch(x) - ref).abs().max() / ref.max()) < TOL


def test_sweep_of_many_planes_is_the_single_planes():
    eng = _engine(1.0, 20)
    x = _clips(256, 3, 9)
    z = [float(v) for v in np.linspace(-90.0, 90.0, 19)] + [0.0]
    out = eng.compute_batch_through_focus(x, z)
    for p, f in enumerate(z):
        assert bool((out[p] == eng.compute_batch(x, focus_nm=f)).all()), f
