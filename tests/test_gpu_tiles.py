"""The tiled pressure solve at the edges of its tiles: grids of one tile, of up
to 16 (one cluster) and of more (the cooperative grid), lines that end inside a
tile, tiles without a fluid cell, and scattered fluid whose levels have gaps.
Against the oracle's solve with the reference dot order, bit for bit, and
against the one-block kernel with the default dots."""
import numpy as np
import pytest

import oracle
from sdr_b200 import _lib
from sdr_b200 import scene as sc

pytestmark = pytest.mark.gpu

DX = 1e-3


def _fluid(case, dims, rng):
    nx, ny, nz = dims
    full = np.ones((nz, ny, nx), dtype=bool)
    if case == "full":
        return full
    if case == "sparse":
        return rng.random((nz, ny, nx)) < 0.35
    if case == "corners":  # two far corners: every tile between them is empty, the level ranges are disjoint
        m = np.zeros_like(full)
        m[:2, :2, :2] = True
        m[-3:, -2:, -2:] = True
        return m
    m = np.zeros_like(full)  # "seam": a slab across the tile seams, one cell thick in places
    m[:, ny // 3: ny // 3 + 1, :] = True
    m[nz // 2, :, ::2] = True
    return m


def _pair(case, dims):
    """A GPU and an oracle solver whose every cell is inside, one particle at the centre of each fluid cell and
    random faces."""
    from sdr_b200.solver import Sdf, Solver
    nx, ny, nz = dims
    rng = np.random.default_rng(nx * 10007 + ny * 101 + nz)
    data = np.full((nz + 1, ny + 1, nx + 1), -1.0)
    fluid = sc.FluidParams()
    needle = sc.Needle(tip=(0.0, 0.0, 0.0), axis=(0.0, 1.0, 0.0), radius=4e-4, flow_rate=0.0)
    gpu = Solver(Sdf((0.0, 0.0, 0.0), DX, data), DX, fluid, needle)
    orc = oracle.Solver(oracle.SdfGrid((0.0, 0.0, 0.0), DX, data), DX,
                        oracle.Fluid(fluid.density, fluid.gravity, fluid.flip_ratio, fluid.particles_per_cell,
                                     fluid.volume_stiffness, fluid.redistribute, fluid.redist_cap_factor),
                        oracle.Needle(needle.tip, needle.axis, needle.radius, needle.flow_rate, needle.inject_until))
    gpu.solve = sc.SolveParams(60, 1e-6)
    orc.set_solve(60, 1e-6)
    k, j, i = np.nonzero(_fluid(case, dims, rng))
    pos = (np.stack([i, j, k], axis=1) + 0.5) * DX
    pos = pos.astype(np.float32).astype(np.float64)
    for s in (gpu, orc):
        s.set_particles(pos, np.zeros_like(pos))
    for w, n in enumerate(((nx + 1) * ny * nz, nx * (ny + 1) * nz, nx * ny * (nz + 1))):
        f = rng.uniform(-1.0, 1.0, n).astype(np.float32).astype(np.float64)
        gpu.set_face(w, f)
        orc.set_face(w, f)
    gpu.run_phase(_lib.PHASE_CLASSIFY)
    orc.phase(oracle.PHASE_CLASSIFY)
    return gpu, orc


@pytest.mark.parametrize("case", ["full", "sparse", "corners", "seam"])
@pytest.mark.parametrize("dims", [(2, 2, 2), (5, 16, 16), (3, 17, 15), (21, 33, 16), (13, 64, 64), (9, 80, 17),
                                  (34, 65, 65), (6, 90, 47)])
def test_tiled_solve_bit_exact(case, dims):
    gpu, orc = _pair(case, dims)
    gpu.set_pcg_kernel(_lib.PCG_TILES)
    gpu.set_dot_order(True)
    gpu.set_profiling(True)
    gpu.run_phase(_lib.PHASE_PROJECT, 1e-3)
    orc.phase(oracle.PHASE_PROJECT, 1e-3)
    assert gpu.profile()["pcg_tile_launches"] == 1
    assert gpu.last_pcg_iters == orc.scalars()["last_pcg_iters"]
    assert np.array_equal(gpu.pressure().view(np.uint64), orc.pressure().view(np.uint64))

    runs = []
    for kernel in (_lib.PCG_TILES, _lib.PCG_ONE_BLOCK):
        g, _ = _pair(case, dims)
        g.set_pcg_kernel(kernel)
        g.run_phase(_lib.PHASE_PROJECT, 1e-3)
        runs.append((g.last_pcg_iters, g.pressure()))
        g.close()
    assert runs[0][0] == runs[1][0]
    assert np.array_equal(runs[0][1].view(np.uint64), runs[1][1].view(np.uint64))
