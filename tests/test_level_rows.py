"""Depth of the passive rows of a tree (static_levels, gbh_decode.h), which the
choice between level elimination and the specialised kernels looks at. A neuron
without any channel has only passive rows, its root among them. Built with
AddressSanitizer; no GPU."""
import os
import shutil
import subprocess

import pytest

from gbhsolve import build

SRC = r"""
#include <stdio.h>
#include <stdlib.h>
#include "gbh_decode.h"
int main(int argc, char **argv)
{
    const int nstatic = atoi(argv[1]);
    std::vector<int> parent;
    for (int i = 2; i < argc; ++i) parent.push_back(atoi(argv[i]));
    printf("%d\n", gbh::static_levels(parent, nstatic));
    return 0;
}
"""

CASES = [                                                    # parents per row, passive rows, levels
    ([1, 2, 3, 4, 5, 6, 7, -1], 7, 7),                       # a cable's dendrites
    ([1, 2, 3, 4, 5, 6, 7, -1], 8, 8),                       # the same without a channel anywhere
    ([8, 8, 8, 8, 8, 8, 8, 8, -1], 8, 1),                    # a star
    ([8, 8, 8, 8, 8, 8, 8, 8, -1], 9, 2),
    ([2, 2, 6, 5, 5, 6, 7, -1], 6, 2),                       # two rows with channels
    ([-1], 0, 0),
    ([-1], 1, 1),
]


@pytest.fixture(scope="module")
def levels(tmp_path_factory):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("no g++")
    d = tmp_path_factory.mktemp("levels")
    (d / "levels.cpp").write_text(SRC)
    exe = str(d / "levels")
    subprocess.run([gxx, "-std=c++17", "-O1", "-g", "-fsanitize=address", "-I" + build.CSRC, "-I" + build.INCLUDE,
                    str(d / "levels.cpp"), "-o", exe], check=True)
    env = dict(os.environ, ASAN_OPTIONS="detect_leaks=0")
    return lambda nstatic, parent: subprocess.run([exe, str(nstatic)] + [str(p) for p in parent], env=env,
                                                  capture_output=True, text=True)


@pytest.mark.parametrize("parent,nstatic,want", CASES)
def test_static_levels(levels, parent, nstatic, want):
    r = levels(nstatic, parent)
    assert r.returncode == 0, r.stderr
    assert int(r.stdout) == want
