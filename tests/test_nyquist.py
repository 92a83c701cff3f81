"""Bands that reach the grid's Nyquist order (2 h = N): the orders -h and +h are
one bin of the transform, in images, gradients and the allocation-free entry
point, against the same kernels in FP64 (numpy), and the same bits each time.

Tolerances as in tests/test_image_error.py (1e-5 of the largest intensity) and
tests/test_ilt_small.py (1e-4 of the largest gradient)."""
import ctypes as C

import numpy as np
import pytest

import highuvlith_b200 as HB
from highuvlith_b200 import _lib as L
from highuvlith_b200 import ilt
from oracle import ilt as OI

pytestmark = pytest.mark.gpu


def _engine(n, pixel, flare=0.03):
    kernels = 9 if n < 512 else 5  # what the allocation-free entry point holds
    eng = HB.SimulationEngine(HB.SourceConfig.euv(0.5), HB.OpticsConfig(0.33, flare, 1.0, "euv"),
                              grid=HB.GridConfig(n, pixel), max_kernels=kernels, source_points_per_axis=9)
    assert 2 * eng.imaging_diagnostics()["band_half_width"] == n
    return eng


SIZES = [(8, 80.0), (16, 40.0), (64, 20.0), (128, 32.0), (256, 16.0), (512, 16.0)]  # 257 and 513 orders: past a block


@pytest.mark.parametrize("dtype", ["float32", "complex64"])
@pytest.mark.parametrize("n,pixel", SIZES)
def test_images(n, pixel, dtype):
    import torch
    eng = _engine(n, pixel)
    rng = np.random.default_rng(n)
    t = (0.1 + 0.8 * rng.random((3, n, n))).astype(np.float32)
    if dtype == "complex64":
        t = (t * np.exp(1j * rng.random(t.shape))).astype(np.complex64)
    x = torch.from_numpy(t).cuda()
    ev, ker = eng.kernels()
    out = eng.compute_batch(x, pixel_transfer=False)
    free = torch.empty_like(out)
    b = L.Batch(3, eng._kind(x), x.data_ptr(), 0, 0.0, L.FORM["fft"], 0)
    L.check(L.lib().huv_image_batch_noalloc(eng.handle, C.byref(b), free.data_ptr(),
                                            torch.cuda.current_stream().cuda_stream))
    for c in range(3):
        spec = np.fft.fft2(t[c].astype(np.complex128))
        img = sum(v * np.abs(np.fft.ifft2(k * spec)) ** 2 for v, k in zip(ev, ker))
        ref = 0.97 * img + 0.03 * img.mean()
        for o in (out, free):
            assert np.max(np.abs(o[c].cpu().numpy() - ref)) < 1e-5 * np.max(ref)
    for _ in range(5):
        assert torch.equal(out, eng.compute_batch(x, pixel_transfer=False))


@pytest.mark.parametrize("n,pixel", SIZES[1:])
def test_gradients(n, pixel):
    import torch
    eng = _engine(n, pixel)
    rng = np.random.default_rng(n)
    target = rng.integers(0, 2, (2, n // 4, n // 4)).repeat(4, 1).repeat(4, 2).astype(np.float32)
    theta = (target - 0.5 + 0.1 * rng.standard_normal(target.shape)).astype(np.float32)
    th, tg = torch.from_numpy(theta).cuda(), torch.from_numpy(target).cuda()
    st = ilt.IltSettings(cost="resist", threshold=0.3, steepness=25.0)
    cost, grad = ilt.cost_and_gradient(eng, th, tg, st)
    ev, ker = eng.kernels()
    cfg = OI.IltConfig(cost="resist", threshold=0.3, steepness=25.0, flare=0.03)
    for m in range(2):
        c, g = OI.IltProblem(ev, ker, target[m], cfg).cost_and_gradient(theta[m].astype(np.float64))
        assert abs(cost[m] - c) <= 1e-5 * c
        assert np.max(np.abs(grad[m].cpu().numpy() - g)) <= 1e-4 * np.max(np.abs(g)), m
    for _ in range(3):
        assert torch.equal(grad, ilt.cost_and_gradient(eng, th, tg, st)[1])
