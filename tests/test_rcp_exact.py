"""Reciprocals that are results of their own -- the gradient's tape holds them
-- are the correctly rounded ones, also where 1/b lies next to the middle
between two doubles."""
import os
import re
import subprocess

import pytest

from gbhsolve import build


@pytest.mark.gpu
def test_reciprocals_next_to_the_middle(tmp_path, gpu_engine):
    exe = str(tmp_path / "rcp_exact")
    src = os.path.join(os.path.dirname(os.path.abspath(__file__)), "cuda", "rcp_exact.cu")
    subprocess.run([build.nvcc()] + build.ARCH + ["-O2", "-std=c++17", "--fmad=false", "-I" + build.CSRC, src, "-o",
                                                  exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stderr
    got = {a: int(b) for a, b in (line.split() for line in out.stdout.splitlines())}
    assert got["hard"] == 0 and got["random"] == 0, got


def test_the_tape_keeps_exact_reciprocals():
    text = open(os.path.join(build.CSRC, "gbh_adjoint.cuh")).read()
    assert not re.search(r"\brcp_(rn|seed|step)\(", text)
