"""A Vm that is no longer finite is reported by the step that meets it, wherever
in the tree it is: the mixed form's conversions turn it into a finite value near
2^128, which the couplings along a long dendrite take to any size by the time
it reaches another row."""
import numpy as np
import pytest

from gbhsolve import configs, model

pytestmark = pytest.mark.gpu


def _lose(eng, at, value):
    vm = eng.vm()
    vm[at] = value
    eng.set_state(vm=vm)
    with pytest.raises(RuntimeError, match="NaN or infinite"):
        eng.run(1)
    eng.close()


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("row", [0, 150, 299])
@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_row_parallel_cable(gpu_engine, prec, row, value):
    hs = [model.build(configs.cables(1, ncomp=300, gk_dend=36.0)[0]) for _ in range(3)]
    p = gpu_engine.PREC_FP64 if prec == "fp64" else gpu_engine.PREC_MIXED
    _lose(gpu_engine.Engine(hs, precision=p, jit=4), 300 + row, value)


@pytest.mark.parametrize("row", ["leaf", "top", "root"])
@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_level_tree(gpu_engine, prec, row):
    from test_level import _trees
    hs = _trees(5, 60, 8, tops=4)
    p = gpu_engine.PREC_FP64 if prec == "fp64" else gpu_engine.PREC_MIXED
    eng = gpu_engine.Engine(hs, precision=p, steps_per_launch=16)
    assert eng.stats().stack_tiles == eng.stats().tiles
    _lose(eng, 60 * 2 + {"leaf": 0, "top": 56, "root": 59}[row], np.nan)


@pytest.mark.parametrize("kw", [dict(jit=False, wide_min=-1), dict(jit=1, wide_min=-1), dict(jit=2, wide_min=-1),
                                dict(jit=False, wide_min=32)])
@pytest.mark.parametrize("row", [0, 20, 39])
def test_mixed_channel_rows(gpu_engine, kw, row):
    """Rows with channels under the other mappings: lane-mapped interpreted,
    specialised and compact, and one neuron per block."""
    hs = [model.build(configs.cables(1, ncomp=40, gk_dend=36.0)[0]) for _ in range(40)]
    _lose(gpu_engine.Engine(hs, precision=gpu_engine.PREC_MIXED, steps_per_launch=10, **kw), 40 * 33 + row, np.nan)
