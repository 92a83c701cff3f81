"""The give-up path of the FNO's projection backward: with
huv_debug_probe_wait one warp of each CTA waits, at the end, for a barrier
phase that never comes, for a short time.  The wait runs out, the other warps
do not wait for it at the sum of the output bias, the kernel returns and the
call reports HUV_ERR_DEVICE_TIMEOUT; the next call's gradients are whole."""
import numpy as np
import pytest

import highuvlith_b200 as HB
from highuvlith_b200 import _lib as L
from highuvlith_b200.fno import FnoSurrogate

pytestmark = pytest.mark.gpu


def test_one_warp_s_wait_runs_out():
    import torch
    f = FnoSurrogate(128, 8, 2, seed=3)
    g = torch.Generator(device="cuda").manual_seed(1)
    x = torch.rand(2, 128, 128, generator=g, device="cuda")
    dout = torch.rand(2, 128, 128, generator=g, device="cuda")
    _, ref, dx = f.backward(x, dout=dout, want_input_grad=True)
    L.check(L.lib().huv_debug_probe_wait(200_000))  # 0.2 ms
    try:
        with pytest.raises(HB.HuvError) as ex:
            f.backward(x, dout=dout, want_input_grad=True)
        assert ex.value.status == 10  # HUV_ERR_DEVICE_TIMEOUT
    finally:
        L.check(L.lib().huv_debug_probe_wait(0))
    f.device_status()  # the flag was cleared by the report
    _, got, dx2 = f.backward(x, dout=dout, want_input_grad=True)
    assert torch.equal(dx, dx2)  # no atomics in the input gradient
    # parameter gradients: FP32 sums by atomics, another order each time
    assert float((got - ref).abs().max() / ref.abs().max()) < 1e-5
