"""The exact arithmetic's exp and reciprocal square root, for every float
(tests/cuda/special_functions_check.cu)."""

import os
import shutil
import subprocess

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "pyvr_gb300", "csrc")


def test_special_functions_exhaustive(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = str(tmp_path / "special_functions_check")
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "--fmad=false", "-std=c++17",
                    f"-I{CSRC}", os.path.join(HERE, "cuda", "special_functions_check.cu"), "-o", exe],
                   check=True, capture_output=True, text=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True, timeout=300).stdout.split()
    assert [int(x) for x in out] == [0, 0], out
