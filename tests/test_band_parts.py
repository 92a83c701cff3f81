"""The workspace of the flare mean's partial sums holds one per block of the
column pass: two columns per block at 2048 (complex maps) and 4096 points, one
at 8192.  The rule on the host (tests/band_parts_check.cu); on the GPU chunks of
many clips on such grids against single clips, with flare."""
import os
import shutil
import subprocess
import tempfile

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.skipif(shutil.which("nvcc") is None, reason="nvcc not on PATH")
def test_every_block_has_its_partial_sum():
    with tempfile.TemporaryDirectory() as d:
        exe = os.path.join(d, "band_parts_check")
        subprocess.run(["nvcc", "-O2", "-std=c++17", "--expt-relaxed-constexpr", "-Wno-deprecated-gpu-targets",
                        "-x", "cu", os.path.join(HERE, "band_parts_check.cu"), "-o", exe], check=True)
        out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout
    rows = [[int(v) for v in line.split()] for line in out.splitlines()]
    assert len(rows) == 11 and all(cases > 0 and short == 0 for _, cases, short in rows), rows


@pytest.mark.gpu
@pytest.mark.parametrize("n,pixel,clips,dtype", [(2048, 1.0, 40, "complex64"), (2048, 1.0, 3, "uint8"),
                                                 (4096, 0.5, 9, "uint8")])
def test_large_grids_with_flare(n, pixel, clips, dtype):
    import torch
    import highuvlith_b200 as HB
    eng = HB.SimulationEngine(HB.SourceConfig(13.5, "annular", (0.7, 0.9)), HB.OpticsConfig(0.33, 0.05, 1.0, "euv"),
                              grid=HB.GridConfig(n, pixel), max_kernels=2, source_points_per_axis=9)
    rng = np.random.default_rng(n)
    m = torch.from_numpy(rng.integers(0, 2, (clips, n // 64, n // 64), dtype=np.uint8)).cuda()
    x = m.repeat_interleave(64, 1).repeat_interleave(64, 2).to(getattr(torch, dtype))
    out = eng.compute_batch(x, form="fft", pixel_transfer=False)
    for c in (0, clips // 2, clips - 1):  # a clip does not depend on its chunk
        assert torch.equal(out[c], eng.compute_batch(x[c], form="fft", pixel_transfer=False)[0])
