"""The row-parallel kernels (gbh_rows.cuh) with the plan forced (jit=4) instead
of chosen by a timing: every case runs them, in both precisions, whatever a
trial would have found. Cases and comparisons as in test_rows."""
import numpy as np
import pytest

from gbhsolve import configs, model
from test_rows import CASES, _active_trees

pytestmark = pytest.mark.gpu


def _forced(gpu_engine, hs, prec, capfd, monkeypatch, **kw):
    monkeypatch.setenv("GBH_VERBOSE", "1")
    eng = gpu_engine.Engine(hs, precision=gpu_engine.PREC_FP64 if prec == "fp64" else gpu_engine.PREC_MIXED, jit=4,
                            **kw)
    err = capfd.readouterr().err
    groups = [line for line in err.splitlines() if "launch group" in line]
    assert groups and all(line.endswith(" row-parallel") for line in groups), err
    return eng


@pytest.mark.parametrize("spl", [0, 16])
@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("method", [model.BEULER, model.CRANK])
@pytest.mark.parametrize("case", sorted(CASES))
def test_forced_rows_equal_oracle(oracle, gpu_engine, monkeypatch, capfd, case, method, prec, spl):
    hs = CASES[case](method)
    eng = _forced(gpu_engine, hs, prec, capfd, monkeypatch, steps_per_launch=spl)
    assert eng.stats().wide_tiles == 0
    n = len(hs)
    idx = sorted(set(range(0, n, max(1, n // 5))) | {n - 1})
    refs = {i: oracle.Solver(hs[i]) for i in idx}
    eng.register_inputs(np.arange(n, dtype=np.int32), np.array([configs.inject_slot(h) for h in hs]))
    eng.register_outputs(np.arange(n, dtype=np.int32), np.array([h.ncompts - 1 for h in hs], np.int32))
    worst = 0.0
    for k, steps in enumerate((1, 37, 20)):
        if k == 1:
            stim = np.random.default_rng(k).uniform(0.0, 5e-10, size=(steps, n))
            rec = np.zeros_like(stim)
            eng.run_io(stim, rec, steps)
            for i in idx:
                for q in range(steps):
                    refs[i].chip[configs.inject_slot(hs[i])] = stim[q, i]
                    refs[i].run(1)
                    if prec == "fp64":
                        assert rec[q, i] == refs[i].vm[-1]
        else:
            eng.run(steps)
            for i in idx:
                refs[i].run(steps)
        st = eng.get_state()
        for i in idx:
            if prec == "fp64":
                np.testing.assert_array_equal(st["vm"][i], refs[i].vm)
                np.testing.assert_array_equal(st["chip"][i], refs[i].chip)
                np.testing.assert_array_equal(st["conc"][i], refs[i].conc[:len(st["conc"][i])])
            else:
                worst = max(worst, float(np.max(np.abs(st["vm"][i] - refs[i].vm))))
    assert worst <= 1e-9, worst
    eng.close()


def test_forced_rows_elsewhere_specialise(oracle, gpu_engine):
    """A batch the plan does not serve (point cells) runs as with jit=1."""
    h = model.build(configs.ap_verify(40))
    eng = gpu_engine.Engine([h], jit=4)
    ref = oracle.Solver(h)
    eng.run(50)
    ref.run(50)
    np.testing.assert_array_equal(eng.vm(), ref.vm)
    assert eng.stats().jit_kernels == 1
    eng.close()


def test_forced_rows_small_and_large(gpu_engine, capfd, monkeypatch):
    """One tree and the largest batch the plan takes."""
    for n, size in ((1, 5), (1216, 33)):
        eng = _forced(gpu_engine, _active_trees(n, size, 4, model.BEULER), "mixed", capfd, monkeypatch)
        eng.run(3)
        assert np.isfinite(eng.vm()).all()
        eng.close()
