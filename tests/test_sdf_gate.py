"""The gate of the closed-mesh SDF path, which the blocks of a launch may open
while others of it start: a block has to leave as one, as its warps share lists
in shared memory. Read off the source, and on the GPU with boxes whose faces lie
on nodes, on a grid of more bricks (2,744) than run at once, against the pass
over all node-triangle pairs, bit for bit."""
import ctypes as C
import os
import re

import numpy as np
import pytest

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sdr_b200", "csrc", "sdf.cuh")


def test_blocks_leave_as_one():
    text = re.sub(r"//[^\n]*", "", open(SRC).read())
    kernels = re.split(r"(?=__global__)", text)[1:]
    both = 0
    for k in kernels:
        if not re.search(r"\*a\.gate = 1u", k):
            continue
        rest = re.sub(r"\*a\.gate = 1u", "", k)
        rest = re.sub(r"\*\(volatile uint32_t\*\)a\.gate", "*a.gate", rest)
        reads = len(re.findall(r"\*a\.gate", rest))
        if reads:
            both += 1
            assert reads == len(re.findall(r"__syncthreads_or\((?:tid == 0 && )?\*a\.gate != 0u\)", rest)), k[:80]
    assert both == 2  # the distances and the roots


@pytest.mark.gpu
@pytest.mark.parametrize("place", ["first", "middle", "last", "all"])
def test_box_on_nodes_of_many_bricks(place):
    import torch
    from sdr_b200 import _lib
    from tests.test_gpu_sdf_closed import _box
    lib = _lib.load()
    lo, hi = {"first": (-13.0, -11.5), "middle": (-3.0, 2.5), "last": (11.5, 13.0), "all": (-13.0, 13.0)}[place]
    tris = np.ascontiguousarray(_box(lo, hi)).reshape(-1, 9)
    origin, dx, dims = (-13.0, -13.0, -13.0), 0.5, (53, 53, 53)  # nodes at whole multiples of 0.5: exact
    cdims = (C.c_uint64 * 3)(*dims)
    dp = C.POINTER(C.c_double)
    dev = torch.tensor(tris, device="cuda")
    out = torch.full((53 ** 3,), float("nan"), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    _lib.check(lib.sdr_sdf_from_mesh_noalloc(C.c_void_p(dev.data_ptr()), len(tris), _lib.Vec3(*origin), dx, cdims,
                                             C.c_void_p(out.data_ptr()), C.c_void_p(0)))
    ref = out.cpu().numpy()
    assert (ref == 0.0).any()  # nodes on the surface
    for _ in range(5):
        got = np.empty(53 ** 3)
        _lib.check(lib.sdr_sdf_from_mesh(tris.ctypes.data_as(dp), len(tris), _lib.Vec3(*origin), dx, cdims,
                                         got.ctypes.data_as(dp)))
        assert np.array_equal(got.view(np.uint64), ref.view(np.uint64))


@pytest.mark.gpu
def test_ball_centred_on_a_node():
    """The centre's node is as far from every triangle: its brick takes the whole mesh, in many lists, and meanwhile
    the nodes at the ball's poles open the gate. Without those nodes the lists run to their end."""
    import torch
    from sdr_b200 import _lib
    from tests.test_gpu_sdf_closed import _sphere
    lib = _lib.load()
    dp = C.POINTER(C.c_double)
    for radius, on_nodes in ((8.0, True), (7.9, False)):
        tris = np.ascontiguousarray(_sphere(5, radius)).reshape(-1, 9)
        origin, dx, dims = (-9.5, -9.5, -9.5), 0.5, (39, 39, 39)
        cdims = (C.c_uint64 * 3)(*dims)
        dev = torch.tensor(tris, device="cuda")
        out = torch.full((39 ** 3,), float("nan"), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        _lib.check(lib.sdr_sdf_from_mesh_noalloc(C.c_void_p(dev.data_ptr()), len(tris), _lib.Vec3(*origin), dx, cdims,
                                                 C.c_void_p(out.data_ptr()), C.c_void_p(0)))
        ref = out.cpu().numpy()
        assert bool((np.abs(ref) < 1e-9).any()) == on_nodes
        got = np.empty(39 ** 3)
        _lib.check(lib.sdr_sdf_from_mesh(tris.ctypes.data_as(dp), len(tris), _lib.Vec3(*origin), dx, cdims,
                                         got.ctypes.data_as(dp)))
        assert np.array_equal(got.view(np.uint64), ref.view(np.uint64))
