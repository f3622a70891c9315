"""The autotuner's trial steps run on the live engine: the state they leave
must be the one the engine was created with, also when the saved copies are
large (their copies take longer than a launch)."""
import numpy as np
import pytest

from gbhsolve import configs

pytestmark = pytest.mark.gpu


def test_trials_leave_the_initial_state(gpu_engine):
    hs, _ = configs.cables_replicated(100_000, 16, seed=3, gk_dend=36.0)
    eng = gpu_engine.Engine(hs, precision=gpu_engine.PREC_MIXED)
    b = eng.batch
    np.testing.assert_array_equal(eng.vm(), b.vm)
    chip = np.concatenate(eng.get_state()["chip"])
    # the mixed form holds fields as double-float pairs (48 bits)
    np.testing.assert_allclose(chip, b.chip, rtol=2.0 ** -47, atol=0.0)
    eng.close()


def test_trials_leave_no_pending_event(oracle, gpu_engine):
    """Weights per synapse: the events the trials leave under way (the cells
    fire throughout, up to 90 steps' delay) are taken back together with the
    bits that name their synapses."""
    from test_network_parity import _network, _oracle_net, _weighted
    n = 96
    hs, esyn, child = _network(n, 0.2, seed=21, inject=np.random.default_rng(20).uniform(0.2e-9, 0.5e-9, size=n))
    ws = _weighted(esyn, 22, zero_frac=0.1, max_delay=90)
    auto = gpu_engine.Engine(hs, synapses=ws)
    plain = gpu_engine.Engine(hs, synapses=ws, steps_per_launch=1)
    for m in (100, 500):
        auto.run(m)
        plain.run(m)
        np.testing.assert_array_equal(auto.spike_counts(), plain.spike_counts())
        np.testing.assert_array_equal(auto.vm(), plain.vm())
    solvers, ref_spikes = _oracle_net(oracle, hs, ws, child, 600)
    assert ref_spikes.sum() > n
    np.testing.assert_array_equal(auto.spike_counts(), ref_spikes)
    np.testing.assert_array_equal(auto.vm(), np.concatenate([s.vm for s in solvers]))
    auto.close()
    plain.close()
