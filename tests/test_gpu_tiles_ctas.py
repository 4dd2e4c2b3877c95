"""The tiled solve's cooperative grid on fewer CTAs than SMs: the first solve of a
solver takes all of them, later ones what the last solve's fluid cells and tiles
ask for; a grid of 169 tiles has more tiles than CTAs. Every solve against the
oracle's, bit for bit in the reference dot order."""
import numpy as np
import pytest

import oracle
from sdr_b200 import _lib
from tests.test_gpu_tiles import _pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("case", ["full", "sparse", "corners", "seam"])
@pytest.mark.parametrize("dims", [(34, 65, 65), (6, 90, 47), (2, 200, 200)])
def test_later_solves_on_fewer_ctas(case, dims):
    gpu, orc = _pair(case, dims)
    gpu.set_dot_order(True)
    gpu.set_profiling(True)
    faces = [gpu.face(w) for w in range(3)]
    orc.phase(oracle.PHASE_PROJECT, 1e-3)
    ref = orc.pressure().view(np.uint64)
    for solves in (1, 2, 3):
        for w in range(3):
            gpu.set_face(w, faces[w])
        gpu.run_phase(_lib.PHASE_PROJECT, 1e-3)
        assert gpu.profile()["pcg_tile_launches"] == solves
        assert gpu.last_pcg_iters == orc.scalars()["last_pcg_iters"]
        assert np.array_equal(gpu.pressure().view(np.uint64), ref)
