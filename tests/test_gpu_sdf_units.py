"""The closed-mesh SDF path in other units of length, against the pass over all
node-triangle pairs, bit for bit. Its f32 distances form products of four
lengths: beyond about 1e9 these leave f32, below about 1e-9 they are denormal.
A power of two scales every coordinate exactly."""
import ctypes as C

import numpy as np
import pytest

from sdr_b200 import _lib
from tests.test_gpu_sdf_closed import GRIDS, _mesh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mesh", ["cavity", "shell"])
@pytest.mark.parametrize("power", [-29, -24, -20, -12, 0, 20, 32, 36, 40, 46])
def test_field_in_other_units(mesh, power):
    import torch
    lib = _lib.load()
    unit = 2.0 ** power
    tris = np.ascontiguousarray(_mesh(mesh), dtype=np.float64).reshape(-1, 9) * unit
    origin, dx, dims = GRIDS["fine"]
    origin, dx = tuple(o * unit for o in origin), dx * unit
    cdims = (C.c_uint64 * 3)(*dims)
    n = int(np.prod(dims))
    got = np.empty(n)
    dp = C.POINTER(C.c_double)
    _lib.check(lib.sdr_sdf_from_mesh(tris.ctypes.data_as(dp), len(tris), _lib.Vec3(*origin), dx, cdims,
                                     got.ctypes.data_as(dp)))
    dev = torch.tensor(tris, device="cuda")
    out = torch.full((n,), float("nan"), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    _lib.check(lib.sdr_sdf_from_mesh_noalloc(C.c_void_p(dev.data_ptr()), len(tris), _lib.Vec3(*origin), dx, cdims,
                                             C.c_void_p(out.data_ptr()), C.c_void_p(0)))
    assert np.array_equal(got.view(np.uint64), out.cpu().numpy().view(np.uint64))
