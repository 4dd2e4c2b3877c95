"""A solver whose tiled-solve buffers do not fit (by the test hook): it frees
them, solves with the other kernels from then on, and never launches the tiled
kernel on what it has not got. Against the oracle's solve with the reference dot
order, bit for bit."""
import numpy as np
import pytest

import oracle
from sdr_b200 import _lib
from tests.test_gpu_tiles import _pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel", [_lib.PCG_AUTO, _lib.PCG_TILES])
@pytest.mark.parametrize("dims", [(21, 33, 16), (34, 65, 65)])  # one cluster; the cooperative grid
def test_solve_without_the_tiles_buffers(dims, kernel):
    gpu, orc = _pair("sparse", dims)
    gpu.set_pcg_kernel(kernel)
    gpu.set_dot_order(True)
    gpu.set_profiling(True)
    faces = [gpu.face(w) for w in range(3)]
    orc.phase(oracle.PHASE_PROJECT, 1e-3)
    _lib.check(_lib.load().sdr_debug_inject(_lib.FAULT_LAZY_BUFFERS))
    for _ in range(2):  # the second solve must not take the tiles either
        for w in range(3):
            gpu.set_face(w, faces[w])
        gpu.run_phase(_lib.PHASE_PROJECT, 1e-3)
        assert gpu.profile()["pcg_tile_launches"] == 0
        assert gpu.last_pcg_iters == orc.scalars()["last_pcg_iters"]
        assert np.array_equal(gpu.pressure().view(np.uint64), orc.pressure().view(np.uint64))
    other, _ = _pair("sparse", dims)  # the hook was one-shot
    other.set_profiling(True)
    other.run_phase(_lib.PHASE_PROJECT, 1e-3)
    assert other.profile()["pcg_tile_launches"] == 1
