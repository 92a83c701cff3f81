"""Focus sweeps of more planes than one launch holds (65,535 images): planes may
repeat, and each is the single-plane image bit for bit."""
import numpy as np
import pytest

import highuvlith_b200 as HB

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("planes,clips", [(1024, 1), (1025, 2), (65540, 1)])
def test_planes_past_one_launch(planes, clips):
    import torch
    eng = HB.SimulationEngine(HB.SourceConfig.euv(0.5), HB.OpticsConfig.euv_nxe_033(), grid=HB.GridConfig(256, 1.0),
                              max_kernels=3)
    x = (torch.rand(clips, 16, 16, device="cuda") > 0.5).to(torch.uint8)
    x = x.repeat_interleave(16, 1).repeat_interleave(16, 2).contiguous()
    distinct = [0.0, 20.0, -35.0]
    z = [distinct[(p * p + p // 7) % 3] for p in range(planes)]
    out = eng.compute_batch_through_focus(x, z)
    one = {f: eng.compute_batch(x, focus_nm=f) for f in distinct}
    rng = np.random.default_rng(planes)
    for p in {0, 15, 16, 1023, planes - 1, *rng.integers(0, planes, 200).tolist()}:
        assert torch.equal(out[p], one[z[p]]), p
