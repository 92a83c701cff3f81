"""Focus sweeps of rectangle clips (huv_image_focus_sweep with
HUV_INPUT_RECTS).  The batch's own defocus_nm is no part of a sweep: whatever
it holds, every plane is the single-plane image bit for bit, also where the
engine's plane cache has no room for another plane."""
import ctypes as C

import numpy as np
import pytest

import highuvlith_b200 as HB
from highuvlith_b200 import _lib as L

pytestmark = pytest.mark.gpu


def _clips(seed, clips=3, count=9):
    rng = np.random.default_rng(seed)
    return [[tuple(v) for v in np.concatenate([rng.uniform(-100, 100, (count, 2)), rng.uniform(8, 50, (count, 2))], 1)]
            for _ in range(clips)]


def _sweep(eng, clips, z, ignored, form="auto"):
    import torch
    view = eng._rect_clips(clips, 1.0, 0.0)
    z = np.asarray(z, dtype=np.float64)
    n = eng.grid.size
    out = torch.empty((len(z), len(clips), n, n), dtype=torch.float32, device="cuda")
    b = L.Batch(len(clips), L.INPUT_RECTS, C.addressof(view), 0, ignored, L.FORM[form], 0)
    L.check(L.lib().huv_image_focus_sweep(eng.handle, C.byref(b), z.ctypes.data, len(z), out.data_ptr(),
                                          torch.cuda.current_stream().cuda_stream))
    return out


@pytest.mark.parametrize("ignored", [0.0, 77.0, float("nan"), float("inf")])
@pytest.mark.parametrize("form", ["auto", "fft"])
def test_the_batch_s_defocus_is_ignored(ignored, form):
    import torch
    eng = HB.SimulationEngine(HB.SourceConfig.euv(0.5), HB.OpticsConfig.euv_nxe_033(), grid=HB.GridConfig(256, 1.0),
                              max_kernels=12, kernel_cache_capacity=3)
    clips, z = _clips(1), [-40.0, 0.0, 25.0, 60.0]  # the cache's three planes and the one in focus
    for _ in range(2):  # planes built in the call, then held
        out = _sweep(eng, clips, z, ignored, form)
        for p, zz in enumerate(z):
            assert torch.equal(out[p], eng.compute_batch_rects(clips, focus_nm=zz, form=form)), zz


def test_an_engine_of_one_plane_sweeps_that_plane():
    import torch
    src = HB.SimulationEngine(HB.SourceConfig.euv(0.5), HB.OpticsConfig.euv_nxe_033(), grid=HB.GridConfig(256, 1.0),
                              max_kernels=12)
    values, kernels = src.kernels()
    eng = HB.SimulationEngine.from_kernel_set(values, kernels, defocus_nm=30.0)
    clips = _clips(2)
    one = eng.compute_batch_rects(clips, focus_nm=30.0)
    out = _sweep(eng, clips, [30.0, 30.0], 5.0)
    assert torch.equal(out[0], one) and torch.equal(out[1], one)
