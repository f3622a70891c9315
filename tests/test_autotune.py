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
