"""A plan's tuned choice holds for sets that do the same work: of two engines of
one grid, band and kernel count, the one whose set does not fold (no symmetry
under inversion) is timed for itself."""
import numpy as np
import pytest

import highuvlith_b200 as HB

pytestmark = pytest.mark.gpu


def test_sets_that_fold_and_sets_that_do_not():
    import torch
    n, clips = 512, 12
    eng = HB.SimulationEngine(HB.SourceConfig.euv(0.5), HB.OpticsConfig.euv_nxe_033(), grid=HB.GridConfig(n, 1.3),
                              max_kernels=23)
    ev, ker = eng.kernels()
    f = np.fft.fftfreq(n) * n
    skew = np.exp(1j * (0.3 * np.sin(f[None, :] + 0.2 * f[:, None] ** 2) + 0.1 * f[:, None]))  # no inversion symmetry
    other = HB.SimulationEngine.from_kernel_set(ev, ker * skew, pixel_nm=1.3)
    x = (torch.rand(clips, n // 8, n // 8, device="cuda") > 0.5).to(torch.uint8)
    x = x.repeat_interleave(8, 1).repeat_interleave(8, 2).contiguous()
    out = torch.empty((clips, n, n), device="cuda")
    told = []
    for e in (eng, other, eng):
        plan = HB.UnevenPlan([(e, len(ev), x[i], out[i]) for i in range(clips)])
        told.append(plan.describe()[0])
        plan.launch()
        torch.cuda.synchronize()
        ref = e.compute_batch(x, form="fft")
        assert float((out - ref).abs().max() / ref.max()) < 1e-4
        del plan
    assert told[0]["K"] == told[1]["K"] and told[0]["h"] == told[1]["h"]
    assert told[2]["ms_per_clip"] == told[0]["ms_per_clip"]  # the same set: the choice is kept
    assert told[1]["ms_per_clip"] != told[0]["ms_per_clip"]  # a timing of its own
