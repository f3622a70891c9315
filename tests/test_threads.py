"""Kernels are compiled on threads of their own; where the host gives no more of
them, the rest is compiled on the calling thread (in_threads, gbh_parallel.h)
and the process lives on. No GPU."""
import os
import re
import shutil
import subprocess

import pytest

from gbhsolve import build

SRC = r"""
#include <atomic>
#include <stdio.h>
#include <stdlib.h>
#include <system_error>
#include "gbh_parallel.h"
static int allowed;
struct Thread {
    std::thread t;
    template <class F> Thread(F f, size_t i)
    {
        if (allowed-- <= 0) throw std::system_error(EAGAIN, std::generic_category());
        t = std::thread(f, i);
    }
    Thread(Thread &&) = default;
    void join() { t.join(); }
};
int main(int, char **argv)
{
    allowed = atoi(argv[1]);
    std::atomic<int> seen[10] = {};
    gbh::in_threads<Thread>(10, [](size_t i) { return i != 4; }, [&](size_t i) { seen[i]++; });
    for (int i = 0; i < 10; ++i) printf("%d", (int)seen[i]);
    return 0;
}
"""


@pytest.mark.parametrize("allowed", [0, 1, 3, 8, 10])
def test_the_rest_runs_here(tmp_path, allowed):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("no g++")
    (tmp_path / "t.cpp").write_text(SRC)
    exe = str(tmp_path / "t")
    subprocess.run([gxx, "-std=c++17", "-O1", "-pthread", "-I" + build.CSRC, str(tmp_path / "t.cpp"), "-o", exe],
                   check=True)
    r = subprocess.run([exe, str(allowed)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    assert r.stdout == "1111011111"


def test_kernels_are_compiled_through_it():
    text = open(os.path.join(build.CSRC, "gbh_engine.cu")).read()
    for m in re.finditer(r"jit_compile\(", text):
        assert "in_threads(" in text[max(0, m.start() - 300):m.start()]
