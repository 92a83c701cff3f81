"""The folded kernels in FP32 are the FP64 ones rounded (tests/fold_f32_check.cpp)."""
import os
import subprocess
import tempfile

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


def test_fp32_kernels_are_the_fp64_ones_rounded():
    with tempfile.TemporaryDirectory() as d:
        exe = os.path.join(d, "check")
        host = os.path.join(ROOT, "highuvlith_b200", "csrc", "host")
        subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", "-I", os.path.join(ROOT, "include"),
                        os.path.join(HERE, "fold_f32_check.cpp")]
                       + [os.path.join(host, f) for f in ("fold.cpp", "kernels.cpp", "source.cpp")] + ["-o", exe],
                       check=True)
        out = subprocess.run([exe], capture_output=True, text=True, check=True, timeout=300).stdout
    rows = [[int(x) for x in line.split()] for line in out.splitlines()]
    assert len(rows) == 6
    for k, folded, differing, misplaced in rows:
        assert folded == 1 and differing == 0 and misplaced == 0, rows
