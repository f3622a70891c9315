"""Single steps of trees with passive dendrites may take another plan than runs
of several (the autotuner times both): runs that alternate between the two, with
inputs on passive rows, a state write and givals between them, equal the
oracle's sequential steps bit for bit whichever plan either takes."""
import re

import numpy as np
import pytest

from gbhsolve import configs, model
from test_level import _trees

pytestmark = pytest.mark.gpu


def _steps(eng, refs, idx, sequence, rows, seed):
    rng = np.random.default_rng(seed)
    for steps in sequence:
        v = rng.uniform(0.0, 5e-10, size=len(rows))
        eng.set_inputs_async(v, 0)
        for (i, c), x in zip(rows, v):
            if i in refs:
                refs[i].chip[c] = x
        eng.run(steps)
        vm = eng.get_state()["vm"]
        for i in idx:
            refs[i].run(steps)
            np.testing.assert_array_equal(vm[i], refs[i].vm)


@pytest.mark.parametrize("batch", ["few", "many", "uniform"])
def test_alternating_run_lengths(oracle, gpu_engine, monkeypatch, capfd, batch):
    if batch == "uniform":
        h = model.build(configs.random_trees(1, size_range=(96, 96), seed=96)[0])
        hs = configs.replicate(h, 12000, inject=np.linspace(0.0, 1e-9, 12000))
    else:
        hs = _trees(40, 60, 1) + _trees(3, 300, 2)
        if batch == "many":
            hs = hs * 200
    monkeypatch.setenv("GBH_VERBOSE", "1")
    eng = gpu_engine.Engine(hs, wide_min=-1)
    err = capfd.readouterr().err
    if "level elimination\n" in err and batch != "few":       # (a few blocks have the SMs to themselves: not timed)
        assert re.search(r"trial single steps: level elimination [\d.]+ us/step, lanes [\d.]+", err), err
    idx = sorted(set(range(0, len(hs), max(1, len(hs) // 7))) | {len(hs) - 1})
    refs = {i: oracle.Solver(hs[i]) for i in idx}
    rows = [(i, int(hs[i].compchips[r]) + 1) for i in range(len(hs)) for r in (hs[i].ncompts - 1, 0)]
    eng.register_inputs(np.array([r[0] for r in rows], np.int32), np.array([r[1] for r in rows]))
    _steps(eng, refs, idx, (1, 1, 9, 1, 70, 1), rows, 1)
    st = eng.get_state()
    for i in idx:                               # a passive row's diagonal term
        c = int(hs[i].compchips[0]) + 3
        st["chip"][i][c] *= 1.03
        refs[i].chip[c] = st["chip"][i][c]
    eng.set_state(chip=st["chip"])
    _steps(eng, refs, idx, (1, 5, 1), rows, 2)
    eng.enable_givals(True)
    _steps(eng, refs, idx, (1, 4), rows, 3)
    eng.enable_givals(False)
    _steps(eng, refs, idx, (1, 3), rows, 4)
    out = np.zeros(len(hs))                     # the pipelined form, one step a call
    eng.register_outputs(np.arange(len(hs), dtype=np.int32), np.array([h.ncompts - 1 for h in hs], np.int32))
    for _ in range(3):
        eng.step_io(None, out)
    eng.io_sync()
    for i in idx:
        refs[i].run(3)
        assert out[i] == refs[i].vm[-1]
    eng.close()
