"""A solver whose buffers for redistribution over the whole GPU do not fit (by the
test hook): one cluster decides long lists from then on, with the same moves."""
import numpy as np
import pytest

import oracle
from sdr_b200 import _lib
from tests.gpu_common import make_pair
from tests.test_gpu_errors import _checkerboard

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hook", [True, False])
def test_redistribution_without_the_rounds_buffers(hook):
    gpu, orc, _ = make_pair()
    pos = _checkerboard(gpu, orc)
    gpu.set_profiling(True)
    if hook:
        _lib.check(_lib.load().sdr_debug_inject(_lib.FAULT_LAZY_BUFFERS))
    gpu.run_phase(_lib.PHASE_REDISTRIBUTE)
    orc.phase(oracle.PHASE_REDISTRIBUTE)
    pg, po = gpu.particles()[0], orc.particles()[0]
    moved = np.any(po != pos, axis=1)
    assert moved.sum() > 20
    assert np.array_equal(np.any(pg != pos, axis=1), moved)
    # one block takes up to 8,192 candidates beside a cluster, 2,048 beside the whole GPU
    assert gpu.profile()["redist_candidates"] > 2048
    assert gpu.profile()["redist_long_sweeps"] >= (0 if hook else 1)
    gpu.run_phase(_lib.PHASE_REDISTRIBUTE)  # and again with what the first call left
    orc.phase(oracle.PHASE_REDISTRIBUTE)
    assert np.array_equal(np.any(gpu.particles()[0] != pg, axis=1), np.any(orc.particles()[0] != po, axis=1))
