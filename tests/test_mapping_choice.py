"""Which mapping a batch gets where the level and row-parallel kernels do not
serve all of it, or are not certain to be the faster ones: the other mappings
are timed too. Only what was timed is asserted, not which mapping won; FP64
results equal the oracle whatever did."""
import numpy as np
import pytest

from gbhsolve import configs, model

pytestmark = pytest.mark.gpu


def _types(n, ncomp, per):
    """n programs with channels everywhere, each with one gate power of its own
    on some dendrite, so that no two share a kernel."""
    hs = []
    for j in range(n):
        m = configs.cables(1, ncomp=ncomp, gk_dend=36.0, per_neuron_solvers=True)[0]
        k = m.compartments[1].children[0]
        for q in range(1, 2 + j):      # j + 1 dendrites with j + 2 channels each
            m.compartments[q].children = [type(k)(k.ctype, Gbar=k.Gbar / (j + 2)) for _ in range(j + 2)]
        hs += [model.build(m) for _ in range(per)]
    return hs


def _create(gpu_engine, monkeypatch, capfd, hs, **kw):
    monkeypatch.setenv("GBH_VERBOSE", "1")
    eng = gpu_engine.Engine(hs, **kw)
    return eng, capfd.readouterr().err


def _check(eng, oracle, hs, steps=40):
    idx = sorted(set(range(0, len(hs), max(1, len(hs) // 6))) | {len(hs) - 1})
    for k in (1, steps):
        eng.run(k)
    vm = eng.get_state()["vm"]
    for i in idx:
        r = oracle.Solver(hs[i])
        r.run(1 + steps)
        np.testing.assert_array_equal(vm[i], r.vm)
    eng.close()


@pytest.mark.parametrize("n,timed", [(8, False), (12, True)])
def test_more_programs_than_kernels(oracle, gpu_engine, monkeypatch, capfd, n, timed):
    hs = _types(n, 60, 2)
    eng, err = _create(gpu_engine, monkeypatch, capfd, hs)
    assert ("mapping trial wide_min 32" in err) == timed, err
    _check(eng, oracle, hs)


@pytest.mark.parametrize("ncomp,n,timed", [(200, 5, True), (200, 700, True), (120, 3, True)])
def test_long_passive_cables_are_timed(oracle, gpu_engine, monkeypatch, capfd, ncomp, n, timed):
    """One row a level: the stack elimination may be the faster one."""
    h = model.build(configs.cables(1, ncomp=ncomp, per_neuron_solvers=True)[0])
    hs = configs.replicate(h, n, inject=np.linspace(0.0, 5e-10, n))
    eng, err = _create(gpu_engine, monkeypatch, capfd, hs)
    assert ("mapping trial wide_min 32" in err) == timed, err
    _check(eng, oracle, hs)


def test_large_uniform_population_times_levels_and_lanes(oracle, gpu_engine, monkeypatch, capfd):
    h = model.build(configs.random_trees(1, size_range=(16, 16), seed=16)[0])
    hs = configs.replicate(h, 11000, inject=np.linspace(0.0, 1e-9, 11000))
    eng, err = _create(gpu_engine, monkeypatch, capfd, hs)
    assert "trial level elimination" in err and "form 0" in err, err
    _check(eng, oracle, hs)
    small, err = _create(gpu_engine, monkeypatch, capfd, hs[:300])
    assert "trial level elimination" not in err and "form 0" not in err, err
    _check(small, oracle, hs[:300])


def test_branched_trees_need_no_trial(oracle, gpu_engine, monkeypatch, capfd):
    hs = [model.build(m) for m in configs.random_trees(20, size_range=(100, 200), seed=5)]
    eng, err = _create(gpu_engine, monkeypatch, capfd, hs)
    assert "mapping trial" not in err, err
    assert eng.stats().stack_tiles == eng.stats().tiles
    _check(eng, oracle, hs)


def test_channels_everywhere_compile_no_lane_kernels(oracle, gpu_engine, monkeypatch, capfd):
    """A small batch of active trees runs row-parallel: the specialised forms it
    would never use are not compiled."""
    trees, (na, k) = configs.grad_trees(5, ncomp=64, seed=3)
    hs = [model.build(t.model(na, k, dt=2e-5)) for t in trees]
    eng, err = _create(gpu_engine, monkeypatch, capfd, hs)
    assert eng.stats().jit_kernels == 1, err
    assert "mapping trial" not in err and "form 0" not in err, err
    _check(eng, oracle, hs)


@pytest.mark.parametrize("active", [True, False])
def test_many_dendrites_on_one_soma(oracle, gpu_engine, monkeypatch, capfd, active):
    """450 dendrites on the soma are more than a lane's elimination stack holds
    and than its shared-memory columns do: only some mappings take the neuron."""
    m = configs.cables(1, ncomp=451, gk_dend=36.0 if active else 0.0, per_neuron_solvers=True)[0]
    for c in m.compartments[1:]:
        c.parent = 0
    hs = [model.build(m) for _ in range(3)]
    eng, err = _create(gpu_engine, monkeypatch, capfd, hs)
    assert "mapping trial wide_min 32" in err, err
    _check(eng, oracle, hs, 20)
