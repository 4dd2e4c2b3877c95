"""The kernels that skip bricks of 8 x 8 x 8 nodes away from the liquid, at the
bricks' edges: grids that end at, before and after a brick's last node, and
liquid in corners, on seams and scattered. Every face is compared, so a brick
skipped wrongly shows. Tolerances: a P2G face is an f64 sum rounded to f32
(2^-24 relative, doubled for the oracle's f64 order); an extrapolated face is
four times in a row a mean of at most six f32 values (six roundings each)."""
import numpy as np
import pytest

import oracle
from sdr_b200 import _lib
from tests.test_gpu_tiles import _pair

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -24


def _rel(a, b):
    return float(np.max(np.abs(a - b))) / max(float(np.max(np.abs(b))), 1e-30)


@pytest.mark.parametrize("case", ["full", "sparse", "corners", "seam"])
@pytest.mark.parametrize("dims", [(2, 2, 2), (7, 8, 9), (16, 15, 17), (33, 24, 8), (41, 7, 26)])
def test_brick_kernels_match_oracle(case, dims):
    gpu, orc = _pair(case, dims)
    gpu.run_phase(_lib.PHASE_EXTRAPOLATE)
    orc.phase(oracle.PHASE_EXTRAPOLATE)
    for w in range(3):
        assert _rel(gpu.face(w), orc.face(w)) <= 24 * EPS
    speed = np.sqrt(sum(float(np.max(np.abs(gpu.face(w)))) ** 2 for w in range(3)))
    assert gpu.cfl()[1] == speed

    rng = np.random.default_rng(7)
    pos, _ = gpu.particles()
    pos = (pos + rng.uniform(-0.49e-3, 0.49e-3, pos.shape)).astype(np.float32).astype(np.float64)
    vel = rng.normal(0.0, 1.0, pos.shape).astype(np.float32).astype(np.float64)
    for s in (gpu, orc):
        s.set_particles(pos, vel)
    gpu.run_phase(_lib.PHASE_P2G)
    orc.phase(oracle.PHASE_P2G)
    orc.phase(oracle.PHASE_SAVE_GRID)
    for w in range(6):
        assert _rel(gpu.face(w), orc.face(w)) <= 2 * EPS
