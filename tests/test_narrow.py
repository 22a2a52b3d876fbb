"""The fold's FP64 to FP32 rounding on the integer pipe (narrow_bits, csrc/narrow.cuh), checked on the host:
tests/narrow_check.cu compiles the same header and compares it with the host's conversion."""
import os
import subprocess

import pytest

from gpu_ppm_b200 import build as B

HERE = os.path.dirname(os.path.abspath(__file__))


def test_narrow_rounds_to_nearest_even(tmp_path):
    if not os.path.exists(B.NVCC):
        pytest.skip("nvcc not available")
    exe = tmp_path / "narrow_check"
    subprocess.run([B.NVCC, "-std=c++17", "-O2", *B.ARCH, "-I", B.CSRC, os.path.join(HERE, "narrow_check.cu"), "-o",
                    str(exe)], check=True, capture_output=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split()
    assert out == ["409600", "0"]
