"""The closed-mesh SDF path against the pass over all node-triangle pairs, bit
for bit: nested and separate shells, inside-out meshes, nodes far outside and
on the surface, grids smaller than a brick and with ragged bricks, and meshes
the path must leave to the full pass (an open one, a sliver, a single
triangle). The full pass is reached through sdr_sdf_from_mesh_noalloc, which
knows no other."""
import ctypes as C

import numpy as np
import pytest

from sdr_b200 import _lib
from sdr_b200.cavity import icosphere, perturbed_ellipsoid

pytestmark = pytest.mark.gpu


def _sphere(subdiv, radius, centre=(0.0, 0.0, 0.0)):
    v, f = icosphere(subdiv)
    return (v * radius + np.asarray(centre))[f]  # (T, 3, 3)


def _box(lo, hi):
    c = np.array([[x, y, z] for z in (lo, hi) for y in (lo, hi) for x in (lo, hi)], dtype=np.float64)
    q = [(0, 2, 3, 1), (4, 5, 7, 6), (0, 1, 5, 4), (2, 6, 7, 3), (0, 4, 6, 2), (1, 3, 7, 5)]
    return np.array([c[list(t)] for a, b, d, e in q for t in ((a, b, d), (a, d, e))])


def _mesh(name):
    if name == "cavity":
        return perturbed_ellipsoid(3, subdiv=4).tris.reshape(-1, 3, 3)
    if name == "cavity_inside_out":
        return perturbed_ellipsoid(4, subdiv=3).tris.reshape(-1, 3, 3)[:, ::-1]
    if name == "two_spheres":
        return np.concatenate([_sphere(3, 4e-3, (-6e-3, 0, 0)), _sphere(2, 3e-3, (5e-3, 1e-3, 0))])
    if name == "shell":  # a ball with a hollow: the inner surface faces inwards
        return np.concatenate([_sphere(3, 8e-3), _sphere(3, 5e-3)[:, ::-1]])
    if name == "overlapping":  # winding number 2 where they overlap
        return np.concatenate([_sphere(3, 6e-3, (-2e-3, 0, 0)), _sphere(3, 6e-3, (2e-3, 0, 0))])
    if name == "box_on_nodes":
        return _box(-4e-3, 4e-3)
    if name == "open":
        return _sphere(3, 6e-3)[1:]
    if name == "sliver":  # closed, with a fan vertex put almost on an edge
        t = _box(-4.05e-3, 4.1e-3)
        a, b, c = t[0]
        m = 0.5 * (a + b) + 1e-14 * (c - a)
        return np.concatenate([t[1:], np.array([[a, m, c], [m, b, c], [a, b, m]])])
    if name == "one_triangle":
        return _sphere(1, 5e-3)[:1]
    raise KeyError(name)


GRIDS = {"around": ((-11e-3, -12e-3, -11e-3), 1.0e-3, (23, 25, 22)),
         "fine": ((-7.03e-3, -6.01e-3, -6.5e-3), 3.7e-4, (39, 33, 37)),
         "small": ((1e-3, -1e-3, 0.5e-3), 0.9e-3, (3, 1, 2)),
         "far": ((0.5, 0.4, -0.3), 1e-3, (9, 5, 6))}


@pytest.mark.parametrize("grid", list(GRIDS))
@pytest.mark.parametrize("mesh", ["cavity", "cavity_inside_out", "two_spheres", "shell", "overlapping", "box_on_nodes",
                                  "open", "sliver", "one_triangle"])
def test_closed_mesh_field_has_the_full_pass_bits(mesh, grid):
    import torch
    lib = _lib.load()
    tris = np.ascontiguousarray(_mesh(mesh), dtype=np.float64).reshape(-1, 9)
    origin, dx, dims = GRIDS[grid]
    nx, ny, nz = dims
    cdims = (C.c_uint64 * 3)(*dims)
    got = np.empty((nz, ny, nx))
    dp = C.POINTER(C.c_double)
    _lib.check(lib.sdr_sdf_from_mesh(tris.ctypes.data_as(dp), len(tris), _lib.Vec3(*origin), dx, cdims,
                                     got.ctypes.data_as(dp)))
    dev = torch.tensor(tris, device="cuda")
    out = torch.full((nx * ny * nz,), float("nan"), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    _lib.check(lib.sdr_sdf_from_mesh_noalloc(C.c_void_p(dev.data_ptr()), len(tris), _lib.Vec3(*origin), dx, cdims,
                                             C.c_void_p(out.data_ptr()), C.c_void_p(0)))
    ref = out.cpu().numpy().reshape(nz, ny, nx)
    assert np.array_equal(got.view(np.uint64), ref.view(np.uint64))
