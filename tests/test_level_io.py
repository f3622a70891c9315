"""Per-step inputs and outputs of trees with passive dendrites inside the level
kernel's launches (run_io): on the soma, on the channel rows below it and on
passive rows, for some neurons only, against the oracle stepped one by one. FP64
bit for bit, mixed within 1e-9 V. The steps of a block run in one launch, so a
recorded run costs about what the same run without recording does."""
import numpy as np
import pytest

from gbhsolve import configs, model
from test_level import _trees

pytestmark = pytest.mark.gpu


def _batch(name, method):
    if name == "sizes":                    # several groups and tiles, a partial one
        return _trees(40, 48, 70, method) + _trees(7, 130, 71, method) + _trees(3, 9, 72, method)
    if name == "tops":                     # channel rows above the passive ones
        return _trees(35, 40, 73, method, tops=4)
    if name == "uniform":                  # one tree many times: several neurons a group
        h = _trees(1, 33, 74, method)[0]
        return configs.replicate(h, 500, inject=np.linspace(0.0, 5e-10, 500))
    return _trees(2, 4501, 75, method)     # "streamed": constants in global memory


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("method", [model.BEULER, model.CRANK])
@pytest.mark.parametrize("name", ["sizes", "tops", "uniform", "streamed"])
def test_recorded_runs_equal_oracle(oracle, gpu_engine, name, method, prec):
    hs = _batch(name, method)
    n = len(hs)
    fp64 = prec == "fp64"
    eng = gpu_engine.Engine(hs, precision=gpu_engine.PREC_FP64 if fp64 else gpu_engine.PREC_MIXED,
                            steps_per_launch=16, wide_min=-1)
    assert eng.stats().stack_tiles == eng.stats().tiles
    rng = np.random.default_rng(7)
    ins, outs = [], []                     # every neuron's soma, a leaf, a middle and the row below the soma of some
    for i, h in enumerate(hs):
        for r in sorted({h.ncompts - 1, 0, h.ncompts // 2, h.ncompts - 2}):
            if r == h.ncompts - 1 or rng.random() < 0.4:
                ins.append((i, r))
            if r == h.ncompts - 1 or rng.random() < 0.4:
                outs.append((i, r))
    eng.register_inputs(np.array([i for i, _ in ins], np.int32),
                        np.array([int(hs[i].compchips[r]) + 1 for i, r in ins]))
    eng.register_outputs(np.array([i for i, _ in outs], np.int32), np.array([r for _, r in outs], np.int32))
    idx = sorted(set(range(0, n, max(1, n // 8))) | {n - 1})
    refs = {i: oracle.Solver(hs[i]) for i in idx}
    for steps, block in ((1, 0), (37, 16), (8, 3)):
        stim = rng.uniform(0.0, 5e-10, size=(steps, len(ins)))
        rec = np.zeros((steps, len(outs)))
        before = eng.stats().launches
        eng.run_io(stim, rec, steps, block)
        blocks = -(-steps // (block or 16))
        assert eng.stats().launches - before <= blocks * 4 * -(-n // 32), "steps of a block share a launch"
        for q in range(steps):
            for j, (i, r) in enumerate(ins):
                if i in refs:
                    refs[i].chip[int(hs[i].compchips[r]) + 1] = stim[q, j]
            for i in idx:
                refs[i].run(1)
            for j, (i, r) in enumerate(outs):
                if i in refs:
                    if fp64:
                        assert rec[q, j] == refs[i].vm[r], (q, i, r)
                    else:
                        assert abs(rec[q, j] - refs[i].vm[r]) <= 1e-9
        eng.run(5)                         # the last inputs stay in their fields
        st = eng.get_state()
        for i in idx:
            refs[i].run(5)
            if fp64:
                np.testing.assert_array_equal(st["vm"][i], refs[i].vm)
                np.testing.assert_array_equal(st["chip"][i], refs[i].chip)
    eng.close()


def test_outputs_alone_and_inputs_alone(oracle, gpu_engine):
    hs = _trees(33, 40, 80)
    eng = gpu_engine.Engine(hs, steps_per_launch=16, wide_min=-1)
    refs = [oracle.Solver(h) for h in hs]
    n = len(hs)
    eng.register_outputs(np.arange(n, dtype=np.int32), np.zeros(n, np.int32))
    rec = np.zeros((20, n))
    eng.run_io(None, rec, 20)
    for q in range(20):
        for r in refs:
            r.run(1)
        assert (rec[q] == [r.vm[0] for r in refs]).all()
    slots = np.array([int(h.compchips[0]) + 1 for h in hs])
    eng.register_inputs(np.arange(n, dtype=np.int32), slots)
    stim = np.random.default_rng(1).uniform(0.0, 5e-10, size=(20, n))
    eng.run_io(stim, None, 20)
    for q in range(20):
        for i, r in enumerate(refs):
            r.chip[slots[i]] = stim[q, i]
            r.run(1)
    vm = eng.get_state()["vm"]
    for i, r in enumerate(refs):
        np.testing.assert_array_equal(vm[i], r.vm)
    eng.close()
