"""Networks whose runs are replayed from graphs: the cooperative plan is timed
against the replay, and runs below its own limit are replayed beside longer
cooperative ones. Spikes and Vm equal the oracle's bit for bit whichever plan
each run takes."""
import numpy as np
import pytest

from test_network_parity import _network, _oracle_net

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,p", [(10, 0.5), (300, 0.1)])
def test_run_lengths_mix(oracle, gpu_engine, monkeypatch, capfd, n, p):
    rng = np.random.default_rng(41)
    hs, esyn, child = _network(n, p, seed=42, inject=rng.uniform(0.05e-9, 0.3e-9, size=n))
    monkeypatch.setenv("GBH_VERBOSE", "1")
    eng = gpu_engine.Engine(hs, synapses=esyn, use_graph=True)
    assert "trial graph replay" in capfd.readouterr().err
    total = 0
    for m in (1, 200, 8, 15, 16, 8, 300, 5, 40, 1):
        eng.run(m)
        total += m
    solvers, ref_spikes = _oracle_net(oracle, hs, esyn, child, total)
    assert ref_spikes.any()
    np.testing.assert_array_equal(eng.spike_counts(), ref_spikes)
    np.testing.assert_array_equal(eng.vm(), np.concatenate([s.vm for s in solvers]))
    eng.close()
