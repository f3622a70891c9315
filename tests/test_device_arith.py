"""The kernels' FP64 divisions, comparisons and table rows that run partly on
the integer and FP32 units (gbh_df.cuh, gbh_devfn.cuh) give IEEE's bits; the
mixed form's reciprocal and its double-float to double conversion are within
their stated errors. tests/cuda/arith.cu compares them with CUDA's IEEE
operations over 3e7 operands of each kind."""
import os
import subprocess

import pytest

from gbhsolve import build

pytestmark = pytest.mark.gpu


def test_device_arithmetic(tmp_path, gpu_engine):
    exe = str(tmp_path / "arith")
    src = os.path.join(os.path.dirname(os.path.abspath(__file__)), "cuda", "arith.cu")
    subprocess.run([build.nvcc()] + build.ARCH + ["-O2", "-std=c++17", "--fmad=false", "-I" + build.CSRC, src, "-o",
                                                  exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stderr
    got = {a: int(b) for a, b in (line.split() for line in out.stdout.splitlines())}
    for k in ("div", "rcp", "special", "key", "row", "volt"):
        assert got[k] == 0, got
    # against the FP64 Newton step: residual below 2^-22 (rcp.approx is within
    # 2^-23 of 1/m in [1/2, 1]); it and its product round at 2^-24 of it each,
    # the divisor's low part at 2^-47
    assert got["seed"] <= 320, got
    # with both products' low parts: the residual of the significand's first 24
    # bits alone rounds, at 2^-47 of a reciprocal of 1/2 or more
    assert got["step"] <= 136, got
    assert got["df"] <= 2, got        # truncated at 2^-52
