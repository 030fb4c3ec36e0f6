"""The branch-free FP64 reciprocal, quotient and square root are CUDA's operators' bit for bit over
their range (150 million operands of each)."""
import os
import subprocess

import pytest

from lica_boiling1d_b200 import build

pytestmark = pytest.mark.gpu


def test_fp64_rn_bitwise(tmp_path):
    src = os.path.join(os.path.dirname(__file__), "abi", "fp64_rn.cu")
    exe = str(tmp_path / "fp64_rn")
    subprocess.run([build.NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-fmad=false",
                    "-I", os.path.join(build.HERE, "csrc"), "-o", exe, src], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True, timeout=120).stdout
    assert out.split() == ["0", "0", "0"], out
