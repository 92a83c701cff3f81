"""The FNO layers' BF16 GELU is the rounding of the FP32 formula for every
input (tests/gelu_check.cu runs all 2^32 bit patterns)."""
import os
import subprocess
import tempfile

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.gpu
def test_every_input_rounds_as_the_plain_formula():
    with tempfile.TemporaryDirectory() as d:
        exe = os.path.join(d, "gelu_check")
        subprocess.run([os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc"), "-O3", "-std=c++17", "-gencode",
                        "arch=compute_100a,code=sm_100a", os.path.join(HERE, "gelu_check.cu"), "-o", exe], check=True)
        out = subprocess.run([exe], capture_output=True, text=True, timeout=300, check=True)
        assert int(out.stdout) == 0
