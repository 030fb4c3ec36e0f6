"""The flags of the branch-free FP64 root, and its cheap test of operands, on 75 million operands in
range, mantissas of all ones among them.  A root whose last correction is formed from a remainder
without rounding error misses the rounded value only within about 2^-50 units of a midpoint, so next
to none may be flagged (one in a million here); `plain` refuses one random operand in 2^32."""
import os
import subprocess

import pytest

from lica_boiling1d_b200 import build

pytestmark = pytest.mark.gpu


def test_flags(tmp_path):
    src = os.path.join(os.path.dirname(__file__), "abi", "fp64_rn_flags.cu")
    exe = str(tmp_path / "fp64_rn_flags")
    subprocess.run([build.NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-fmad=false",
                    "-I", os.path.join(build.HERE, "csrc"), "-o", exe, src], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True, timeout=120).stdout
    wrong, flagged, too_plain, wrong_recip, refused = map(int, out.split())
    assert (wrong, too_plain, wrong_recip) == (0, 0, 0), out
    assert flagged <= 75 and refused <= 10, out
