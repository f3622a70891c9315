"""The mixed form's arithmetic off the FP64 unit (gbh_df.cuh): the reciprocal
is the FP64 Newton step to its last place, so no further from 1/b, and the
conversion of a double-float is the FP64 sum of its parts, rounded to nearest.
tests/cuda/mixed_arith.cu compares them over 3e7 operands."""
import os
import subprocess

import pytest

from gbhsolve import build

pytestmark = pytest.mark.gpu


def test_reciprocal_and_conversion(tmp_path, gpu_engine):
    exe = str(tmp_path / "mixed_arith")
    src = os.path.join(os.path.dirname(os.path.abspath(__file__)), "cuda", "mixed_arith.cu")
    subprocess.run([build.nvcc()] + build.ARCH + ["-O2", "-std=c++17", "--fmad=false", "-I" + build.CSRC, src, "-o",
                                                  exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stderr
    got = {a: int(b) for a, b in (line.split() for line in out.stdout.splitlines())}
    assert got["convert"] == 0, got
    # the step's residual has up to 54 bits, of which its FMA keeps 53: at most
    # the last place of the result shows it
    assert got["step"] <= 1, got
    assert got["step_int"] <= got["step64"] + 1, got
