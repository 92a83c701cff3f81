"""Rectangle clips resolved on the GPU against the host's resolution of the
same union (csrc/cuda/rects.cu): a clip of more than 2048 rectangles goes
through the host, so each clip is also given with its rectangles repeated past
that.  Overlapping, nested, touching, zero-size and partly or wholly outside
rectangles; counts around the sort's powers of two; an empty clip.

Both sum the same FP64 terms in another order (1e-13 of the spectrum) and
round to FP32 once: 1e-6 of the largest intensity.
"""
import numpy as np
import pytest

import highuvlith_b200 as HB

pytestmark = pytest.mark.gpu


def _clip(rng, count):
    w = rng.uniform(0.0, 60.0, (count, 2))
    c = rng.uniform(-140.0, 140.0, (count, 2))
    r = np.concatenate([c, w], axis=1)
    if count > 4:
        r[1] = [r[0, 0] + r[0, 2], r[0, 1], r[0, 2], r[0, 3]]  # touches the first
        r[2] = [r[0, 0], r[0, 1], r[0, 2] / 2, r[0, 3] / 2]    # inside it
        r[3, 2] = 0.0                                          # empty
        r[4] = [400.0, 0.0, 50.0, 50.0]                        # outside the field
    return [tuple(v) for v in r.tolist()]


@pytest.mark.parametrize("form", ["auto", "fft"])
def test_device_and_host_resolution_give_one_image(form):
    eng = HB.SimulationEngine(HB.SourceConfig.euv(0.5), HB.OpticsConfig.euv_nxe_033(), grid=HB.GridConfig(256, 1.0),
                              max_kernels=12)
    rng = np.random.default_rng(4)
    clips = [_clip(rng, n) for n in (1, 2, 5, 31, 32, 33, 64, 65, 700, 2048)] + [[]]
    many = [c * (2048 // max(len(c), 1) + 1) for c in clips]
    a = eng.compute_batch_rects(clips, form=form)
    b = eng.compute_batch_rects(many, form=form)
    assert float((a - b).abs().max() / b.max()) < 1e-6
    assert float(a[-1].abs().max()) < 1e-12
    # amplitudes and background; a clip alone is the clip in its batch
    c = eng.compute_batch_rects(clips[:4], feature=-0.25 + 0.1j, background=1.0, form=form)
    d = eng.compute_batch_rects(many[:4], feature=-0.25 + 0.1j, background=1.0, form=form)
    assert float((c - d).abs().max() / d.max()) < 1e-6
    assert bool((eng.compute_batch_rects(clips[5:6], form=form)[0] == a[5]).all())
