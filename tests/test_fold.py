"""Kernel sets of real masks (csrc/host/fold.cpp): in focus, two kernels of a
symmetric source become one complex transform.  On the host against the set
itself (tests/fold_check.cpp); on the GPU against the same masks given as
complex maps, which are imaged with the set as it is."""
import os
import subprocess
import tempfile

import numpy as np
import pytest

import highuvlith_b200 as HB

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


def test_folded_sets_give_the_set_s_intensity():
    with tempfile.TemporaryDirectory() as d:
        exe = os.path.join(d, "fold_check")
        host = os.path.join(ROOT, "highuvlith_b200", "csrc", "host")
        subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", "-I", os.path.join(ROOT, "include"),
                        os.path.join(HERE, "fold_check.cpp")]
                       + [os.path.join(host, f) for f in ("fold.cpp", "kernels.cpp", "source.cpp")] + ["-o", exe],
                       check=True)
        out = subprocess.run([exe], capture_output=True, text=True, check=True, timeout=300).stdout
    seen = {}
    for line in out.splitlines():
        name, k, ok, err = line.split()
        seen.setdefault(name, []).append((int(k), int(ok)))
        # dropped energy below 1e-13 of the set's, FP64 sums of at most a few thousand terms
        assert float(err) < 1e-11, line
    for name, cases in seen.items():
        for k, ok in cases:
            if name in ("defocus", "nyquist", "asymmetric"):
                assert not ok, (name, k)
            else:
                assert ok == (k >= 2), (name, k)


# Two FP32 evaluations of one image, each within 2e-6 of it (the errors of the
# forms against FP64); the TC form's BF16 split is within 2.4e-5.
@pytest.mark.gpu
@pytest.mark.parametrize("form,tol", [("auto", 5e-6), ("fft", 5e-6), ("tc", 5e-5), ("tc_rows", 5e-5)])
@pytest.mark.parametrize("fill,par,kernels", [("conventional", (0.5,), 31), ("annular", (0.6, 0.85), 24),
                                              ("quasar", (0.7, 0.9, 45.0), 17), ("dipole", (0.7, 0.15, 30.0), 2)])
def test_real_masks_match_the_complex_path(form, tol, fill, par, kernels):
    import torch
    for n, pixel in ((512, 2.0), (512, 0.6)):
        eng = HB.SimulationEngine(HB.SourceConfig(13.5, fill, par), HB.OpticsConfig(0.33, 0.03, 1.0, "euv"),
                                  grid=HB.GridConfig(n, pixel), max_kernels=kernels)
        rng = np.random.default_rng(kernels)
        x = torch.from_numpy(rng.integers(0, 2, (3, n // 8, n // 8), dtype=np.uint8).repeat(8, 1).repeat(8, 2)).cuda()
        grey = x.float() * 0.8 + 0.1
        for real, transfer in ((x, True), (grey, False)):
            ref = eng.compute_batch(real.to(torch.complex64), pixel_transfer=transfer, form=form)
            out = eng.compute_batch(real, pixel_transfer=transfer, form=form)
            assert float((out - ref).abs().max() / ref.max()) < tol, (n, pixel, transfer)
