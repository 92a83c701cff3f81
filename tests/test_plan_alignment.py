"""Clips of an uneven plan that lie anywhere: a view some elements into a
buffer, alone or in a run of contiguous clips (read where it lies), with the
tuned and the default form, against single calls on aligned clips as
tests/test_uneven_plan.py compares them (1e-4 of the largest intensity: a
plan's form may be the split-BF16 one).
"""
import numpy as np
import pytest

import highuvlith_b200 as HB

pytestmark = pytest.mark.gpu


def _engine(n):
    return HB.SimulationEngine(HB.SourceConfig.euv(0.5), HB.OpticsConfig.euv_nxe_033(), grid=HB.GridConfig(n, 1.0),
                               max_kernels=10)


def _maps(n, clips, dtype):
    import torch
    rng = np.random.default_rng(n + clips)
    m = rng.integers(0, 2, (clips, n // 16, n // 16)).repeat(16, 1).repeat(16, 2)
    if dtype == "uint8":
        return torch.from_numpy(m.astype(np.uint8)).cuda()
    if dtype == "float32":
        return torch.from_numpy((m * 0.8 + 0.1 * rng.random(m.shape)).astype(np.float32)).cuda()
    return torch.from_numpy((m * np.exp(0.2j * rng.random(m.shape))).astype(np.complex64)).cuda()


def _view(x, skip):
    """x's values, `skip` elements into a larger buffer."""
    import torch
    buf = torch.zeros(skip + x.numel(), dtype=x.dtype, device="cuda")
    v = buf[skip:].view(x.shape)
    v.copy_(x)
    return v


def _images(eng, x, out, autotune):
    import torch
    plan = HB.UnevenPlan([(eng, 10, x[i], out[i]) for i in range(x.shape[0])], pixel_transfer=x.dtype == torch.uint8,
                         autotune=autotune)
    out.zero_()
    plan.launch()
    torch.cuda.synchronize()
    return out.clone(), plan.describe()


@pytest.mark.parametrize("autotune", [False, True])
@pytest.mark.parametrize("clips", [1, 3])
@pytest.mark.parametrize("n,dtype,skip", [(128, "float32", 1), (256, "float32", 1), (256, "float32", 3),
                                          (512, "float32", 2), (1024, "float32", 1), (256, "complex64", 1),
                                          (512, "complex64", 1), (256, "uint8", 5), (2048, "uint8", 1)])
def test_inputs(n, dtype, skip, clips, autotune):
    import torch
    eng, x = _engine(n), _maps(n, clips, dtype)
    out = torch.empty((clips, n, n), device="cuda")
    ref = eng.compute_batch(x, pixel_transfer=dtype == "uint8", form="fft")
    got, groups = _images(eng, _view(x, skip), out, autotune)
    assert len(groups) == 1 and groups[0]["contiguous"] == 1
    assert float((got - ref).abs().max() / ref.max()) < 1e-4


@pytest.mark.parametrize("autotune", [False, True])
@pytest.mark.parametrize("clips", [1, 3])
@pytest.mark.parametrize("n,dtype,skip", [(128, "uint8", 2), (256, "uint8", 1), (256, "uint8", 2), (512, "uint8", 2),
                                          (512, "float32", 3), (256, "complex64", 2)])
def test_outputs(n, dtype, skip, clips, autotune):
    import torch
    eng, x = _engine(n), _maps(n, clips, dtype)
    ref = eng.compute_batch(x, pixel_transfer=dtype == "uint8", form="fft")
    buf = torch.full((clips * n * n + 2 * skip,), -7.0, device="cuda")
    out = buf[skip:skip + clips * n * n].view(clips, n, n)
    got, _ = _images(eng, x, out, autotune)
    assert float((got - ref).abs().max() / ref.max()) < 1e-4
    assert bool((buf[:skip] == -7.0).all()) and bool((buf[-skip:] == -7.0).all())


def test_complex_maps_between_elements():
    import torch
    eng, x = _engine(256), _maps(256, 2, "complex64")
    buf = torch.zeros(2 * x.numel() + 1, device="cuda")
    buf[1:].copy_(torch.view_as_real(x).reshape(-1))
    out = torch.empty((2, 256, 256), device="cuda")
    bytes_per = 8 * 256 * 256
    from highuvlith_b200 import _lib as L
    import ctypes as C
    arr = (L.Clip * 2)(*[L.Clip(eng.handle, 10, L.INPUT_C64, buf.data_ptr() + 4 + bytes_per * i, out[i].data_ptr())
                         for i in range(2)])
    h = C.c_void_p()
    L.check(L.lib().huv_plan_create(arr, 2, 0, 0, C.byref(h)))
    L.check(L.lib().huv_plan_launch(h, torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    L.lib().huv_plan_destroy(h)
    ref = eng.compute_batch(x, pixel_transfer=False, form="fft")
    assert float((out - ref).abs().max() / ref.max()) < 1e-4
