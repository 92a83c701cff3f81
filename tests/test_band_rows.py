"""Row transforms of f32 and complex rasters (band_rows_img, csrc/cuda/
socs_fft.cu) at every length they serve and for narrow and wide bands, against
numpy's FFT through the SOCS sum with the engine's own kernels.

Tolerance: FP32 transforms of up to 2048 points, a few 1e-7 each: 5e-6 of the
largest intensity (FFT form)."""
import numpy as np
import pytest

import highuvlith_b200 as HB

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,pixel,kernels", [(128, 1.0, 5), (128, 6.0, 3), (256, 1.0, 4), (256, 6.0, 3), (512, 0.3, 5),
                                             (512, 3.0, 3), (1024, 1.0, 3), (2048, 0.7, 2)])
@pytest.mark.parametrize("dtype", ["f32", "c64"])
def test_maps_match_numpy(n, pixel, kernels, dtype):
    import torch
    eng = HB.SimulationEngine(HB.SourceConfig.euv(0.5), HB.OpticsConfig.euv_nxe_033(), grid=HB.GridConfig(n, pixel),
                              max_kernels=kernels)
    rng = np.random.default_rng(n)
    x = rng.random((2, n, n)).astype(np.float32)
    if dtype == "c64":
        x = (x * np.exp(1j * rng.random((2, n, n)))).astype(np.complex64)
    ev, ker = eng.kernels()
    for form in ("fft", "auto"):
        out = eng.compute_batch(torch.from_numpy(x).cuda(), pixel_transfer=False, form=form).cpu().numpy()
        for c in range(2):
            spec = np.fft.fft2(x[c].astype(np.complex128))
            ref = sum(l * np.abs(np.fft.ifft2(k * spec)) ** 2 for l, k in zip(ev, ker))
            assert np.max(np.abs(out[c] - ref)) < (5e-6 if form == "fft" else 1.3e-4) * ref.max(), (form, c)
