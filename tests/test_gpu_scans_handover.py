"""Scans at the edges of their tiles (4,096 items; up to eight tiles each block
adds up the items before its own) and the candidate list's length from which the
whole GPU decides a redistribution sweep (2,048). Tolerances: a P2G face is an
f64 sum rounded to f32 (2^-24 relative, doubled for the oracle's f64 order); the
particles that stay, and which ones move, are exact."""
import numpy as np
import pytest

import oracle
from sdr_b200 import _lib
from tests.gpu_common import f32, make_pair
from tests.gpu_states import sync_faces
from tests.test_gpu_tiles import DX, _pair

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -24


@pytest.mark.parametrize("dims, n", [((15, 13, 21), 4095), ((16, 16, 16), 4096), ((17, 16, 16), 4097),
                                     ((33, 32, 31), 32768), ((32, 32, 32), 32769), ((41, 47, 39), 70001)])
def test_scans_at_tile_edges(dims, n):
    gpu, orc = _pair("corners", dims)
    rng = np.random.default_rng(n)
    pos = f32(rng.uniform(-0.05, 1.05, (n, 3)) * (np.array(dims) * DX))  # some outside: dropped
    vel = f32(rng.normal(0.0, 1.0, pos.shape))
    for s in (gpu, orc):
        s.set_particles(pos, vel)
    gpu.run_phase(_lib.PHASE_BOUNDS)
    orc.phase(oracle.PHASE_BOUNDS)
    (pg, vg), (po, vo) = gpu.particles(), orc.particles()
    assert 0 < len(po) < n
    assert np.array_equal(pg, po) and np.array_equal(vg, vo)
    gpu.run_phase(_lib.PHASE_P2G)
    orc.phase(oracle.PHASE_P2G)
    for w in range(3):
        a, b = gpu.face(w), orc.face(w)
        assert float(np.max(np.abs(a - b))) <= 2 * EPS * float(np.max(np.abs(b)))


@pytest.mark.parametrize("n", [2047, 2048, 2049, 4500])
def test_redistribution_handover_exact(n):
    gpu, orc, _ = make_pair()
    nx, ny, nz = gpu.grid_dims
    st = gpu.stats()
    cav = gpu.cavity_mask().reshape(nz, ny, nx).astype(bool)
    inner = cav.copy()
    for ax in range(3):
        for sh in (-1, 1):
            inner &= np.roll(cav, sh, axis=ax)
    k, j, i = (int(x) for x in np.argwhere(inner)[len(np.argwhere(inner)) // 2])
    rng = np.random.default_rng(n)
    pos = f32(np.array([st.origin.x, st.origin.y, st.origin.z]) +
              (np.array([i, j, k]) + 0.5 + rng.uniform(-0.3, 0.3, (n, 3))) * gpu.dx)
    vel = np.zeros_like(pos)
    for s in (gpu, orc):
        s.set_particles(pos, vel)
    sync_faces(gpu, orc)
    gpu.set_profiling(True)
    gpu.run_phase(_lib.PHASE_REDISTRIBUTE)
    orc.phase(oracle.PHASE_REDISTRIBUTE)
    pg, po = gpu.particles()[0], orc.particles()[0]
    assert (gpu.profile()["redist_long_sweeps"] >= 1) == (n > 2048)
    moved = np.any(po != pos, axis=1)
    assert moved.sum() > 20
    assert np.array_equal(np.any(pg != pos, axis=1), moved)
