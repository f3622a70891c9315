"""Work that creating an engine leaves on the device is done before steps on a
stream of the caller's start."""
import os

import numpy as np
import pytest

from gbhsolve import build

gpu = pytest.mark.gpu


def test_creation_waits_for_the_trials_last_work():
    """What the autotuner puts on the engine's stream (clears of the trials'
    spikes and itotal sums, the factors' new generation) is done when it
    returns: a first step may run on any other stream."""
    text = open(os.path.join(build.CSRC, "gbh_engine.cu")).read()
    start = text.index("\nint autotune(gbh_engine *e)\n")
    body = text[start:text.index("\n}\n", start)]
    queued = max(body.rindex(s) for s in ("autotune_trials(e", "stack_invalidate(e, e->stream)"))
    assert "cudaStreamSynchronize(e->stream)" in body[queued:]


@gpu
@pytest.mark.parametrize("n", [40, 4000])
def test_first_step_on_a_foreign_stream(gpu_engine, n):
    """Steps issued on the caller's stream right after creation: their spikes
    are the ones of steps on the engine's own."""
    import torch
    from test_network_parity import _network
    hs, esyn, _ = _network(n, 0.02, seed=31, inject=np.full(n, 0.4e-9))
    for h in hs:
        h.vm = np.full_like(h.vm, 0.02)      # above the threshold: every cell fires in the first step
    st = torch.cuda.Stream()
    eng = gpu_engine.Engine(hs, synapses=esyn)
    eng.run_async(1, st.cuda_stream)
    st.synchronize()
    assert eng.get_spiked().all()
    np.testing.assert_array_equal(eng.spike_counts(), np.ones(n, dtype=np.int64))
    eng.close()
