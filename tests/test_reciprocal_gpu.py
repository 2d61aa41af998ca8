"""The differentiable march's reciprocal over its range
(tests/cuda/reciprocal_check.cu): half an ulp of the final rounding and the
2^-46 that one Newton step leaves of the approximation's 2^-23."""

import os
import shutil
import subprocess

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "pyvr_gb300", "csrc")


def test_reciprocal_exhaustive(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = str(tmp_path / "reciprocal_check")
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "--fmad=false", "-std=c++17",
                    f"-I{CSRC}", os.path.join(HERE, "cuda", "reciprocal_check.cu"), "-o", exe],
                   check=True, capture_output=True, text=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True, timeout=300).stdout.split()
    worst, n = (int(x) for x in out)
    assert n == 150 * 2 ** 23 + 1
    assert worst <= 510000, f"{worst / 1e6} ulp"
