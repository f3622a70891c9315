"""Row-parallel steps (gbh_rows.cuh): small batches of neurons with channels
along their dendrites, one thread per compartment, the elimination depth by
depth. FP64 results equal the oracle (the reference's sequential step) bit for
bit; the mixed form stays within the 1e-9 V of the other mixed mappings."""
import numpy as np
import pytest

from gbhsolve import configs, engine, model

pytestmark = pytest.mark.gpu


def _active_trees(n, size, seed, method):
    """Trees with Na and K on every compartment."""
    trees, (na, k) = configs.grad_trees(n, ncomp=size, seed=seed)
    return [model.build(t.model(na, k, dt=2e-5, method=method)) for t in trees]


def _classes(n, method):
    """Cables of several program classes: the soma with a Ca channel, a
    Ca-dependent K channel and their pool besides, no channel on every third
    dendrite."""
    soma = configs.random_trees(1, size_range=(2, 2), seed=1)[0].compartments[0].children
    ms = configs.cables(n, ncomp=31, method=method, gk_dend=36.0, per_neuron_solvers=True)
    for m in ms:
        m.compartments[0].children = list(soma)
        for c in m.compartments[3::3]:
            c.children = []
    return [model.build(m) for m in ms]


CASES = {     # tile and group edges: one neuron, full and partial tiles, rows over and under a block's threads
    "one-cell": lambda m: _active_trees(1, 70, 1, m),
    "cables": lambda m: [model.build(x) for x in configs.cables(300, ncomp=23, method=m, gk_dend=36.0,
                                                                per_neuron_solvers=True)],
    "trees": lambda m: _active_trees(37, 40, 2, m) + _active_trees(3, 33, 3, m),
    "classes": lambda m: _classes(33, m),
    "long": lambda m: _active_trees(3, 700, 5, m),
}


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("method", [model.BEULER, model.CRANK])
@pytest.mark.parametrize("case", sorted(CASES))
def test_rows_equal_oracle(oracle, gpu_engine, monkeypatch, capfd, case, method, prec):
    hs = CASES[case](method)
    monkeypatch.setenv("GBH_VERBOSE", "1")
    eng = gpu_engine.Engine(hs, precision=gpu_engine.PREC_FP64 if prec == "fp64" else gpu_engine.PREC_MIXED)
    err = capfd.readouterr().err
    assert "trial row-parallel" in err
    if prec == "fp64" or case not in ("cables", "classes"):    # (mixed cables are as fast lane-mapped)
        assert " row-parallel\n" in err                        # the plan the trial kept
    idx = sorted(set(range(0, len(hs), max(1, len(hs) // 9))) | {len(hs) - 1})
    refs = {i: oracle.Solver(hs[i]) for i in idx}
    n = len(hs)
    eng.register_inputs(np.arange(n, dtype=np.int32), np.array([configs.inject_slot(h) for h in hs]))
    eng.register_outputs(np.arange(n, dtype=np.int32), np.array([h.ncompts - 1 for h in hs], np.int32))
    worst = 0.0
    for k, steps in enumerate((1, 60, 33)):
        if k == 1:                                 # per-step inputs and outputs inside the launches
            stim = np.random.default_rng(k).uniform(0.0, 5e-10, size=(steps, n))
            rec = np.zeros_like(stim)
            eng.run_io(stim, rec, steps)
            want = {}
            for i in idx:
                tr = []
                for q in range(steps):
                    refs[i].chip[configs.inject_slot(hs[i])] = stim[q, i]
                    refs[i].run(1)
                    tr.append(refs[i].vm[-1])
                want[i] = np.array(tr)
        else:
            eng.enable_givals(k == 2)
            eng.run(steps)
            for i in idx:
                refs[i].run(steps)
        st = eng.get_state()
        for i in idx:
            if prec == "fp64":
                np.testing.assert_array_equal(st["vm"][i], refs[i].vm)
                np.testing.assert_array_equal(st["chip"][i], refs[i].chip)
                np.testing.assert_array_equal(st["conc"][i], refs[i].conc[:len(st["conc"][i])])
                if k == 1:
                    np.testing.assert_array_equal(rec[:, i], want[i])
            else:
                worst = max(worst, float(np.max(np.abs(st["vm"][i] - refs[i].vm))))
    assert worst <= 1e-9, worst
    eng.close()


def test_rows_carry_the_table_bracket(oracle, gpu_engine, monkeypatch, capfd):
    """As test_wide's: a compartment exactly on a table node that a fresh
    lookup puts one row lower, after a compartment inside the upper row."""
    from test_wide import _bracket_edge
    h = model.build(configs.cables(1, ncomp=48, gk_dend=36.0)[0])
    edge = _bracket_edge(h)
    if edge is None:
        pytest.skip("no rounding edge in this table")
    r, x = edge
    vm = np.array(h.vm, copy=True)
    vm[10], vm[11], vm[30], vm[31] = x + 0.3 / h.invdx, x, x + 0.6 / h.invdx, x
    h.vm = vm
    monkeypatch.setenv("GBH_VERBOSE", "1")
    eng = gpu_engine.Engine([h])
    assert " row-parallel\n" in capfd.readouterr().err
    ref = oracle.Solver(h)
    for _ in range(3):
        eng.run(1)
        ref.run(1)
        st = eng.get_state()
        np.testing.assert_array_equal(st["vm"][0], ref.vm)
        np.testing.assert_array_equal(st["chip"][0], ref.chip)
    eng.close()
