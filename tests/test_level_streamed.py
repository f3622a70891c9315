"""The level kernel's streamed form (constants in global memory), which one
neuron of more passive rows than shared memory holds with their constants runs
-- some 3,500 in FP64, 4,100 mixed -- beside small trees that keep theirs
resident. FP64 equals the oracle bit for bit; the mixed form stays within the
1e-9 V of the other mappings."""
import numpy as np
import pytest

from gbhsolve import configs, model
from test_level import _trees

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("method", [model.BEULER, model.CRANK])
def test_large_neuron_streams_its_constants(oracle, gpu_engine, method, prec):
    hs = _trees(2, 4501, 90, method) + _trees(5, 60, 91, method)
    mixed = prec == "mixed"
    eng = gpu_engine.Engine(hs, precision=gpu_engine.PREC_MIXED if mixed else gpu_engine.PREC_FP64,
                            steps_per_launch=16, wide_min=-1)
    assert eng.stats().stack_tiles == eng.stats().tiles == 2
    assert eng.stats().jit_kernels == 1        # one program of the soma, in both forms
    refs = [oracle.Solver(h) for h in hs]
    rows = [(i, int(h.compchips[r]) + 1) for i, h in enumerate(hs) for r in (h.ncompts - 1, 0)]
    eng.register_inputs(np.array([r[0] for r in rows], np.int32), np.array([r[1] for r in rows]))
    for k, steps in enumerate((1, 33, 18)):
        v = np.random.default_rng(k).uniform(0.0, 5e-10, size=len(rows))
        eng.set_inputs_async(v, 0)
        for (i, c), x in zip(rows, v):
            refs[i].chip[c] = x
        eng.run(steps)
        st = eng.get_state()
        for i, r in enumerate(refs):
            r.run(steps)
            if mixed:
                assert np.max(np.abs(st["vm"][i] - r.vm)) <= 1e-9
            else:
                np.testing.assert_array_equal(st["vm"][i], r.vm)
                np.testing.assert_array_equal(st["chip"][i], r.chip)
    eng.close()


def test_kernel_count(gpu_engine):
    """jit_kernels counts what was compiled: the resident form alone where no
    neuron needs the other, and the row-parallel kernel."""
    eng = gpu_engine.Engine(_trees(5, 60, 91), steps_per_launch=16)
    assert eng.stats().jit_kernels == 1
    eng.close()
    hs = [model.build(m) for m in configs.cables(3, ncomp=120, gk_dend=36.0, per_neuron_solvers=True)]
    eng = gpu_engine.Engine(hs, jit=4)
    assert eng.stats().jit_kernels == 1
    eng.close()
