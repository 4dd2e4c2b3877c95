"""Default solvers on several threads of one process: their solves run beside each
other, so none may keep the others off the GPU while it iterates, and each gives
the bits it gives alone."""
import os
import re
import threading

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sdr_b200", "csrc")


@pytest.mark.parametrize("file, kernel, body", [("pressure_tiles.cuh", "k_pcg_tiles_cluster", "tw_solve"),
                                                ("pressure.cuh", "k_pcg", "k_pcg_body")])
def test_solves_let_the_next_launch_begin_behind_their_iterations(file, kernel, body):
    """Blocks of the next kernel that are set up early hold their places for as long as the solve runs."""
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, file)).read())
    entry = text[re.search(r"__global__[^;{]*\b%s\(" % kernel, text).end():]
    entry = entry[:entry.index("}\n")]
    assert "pdl_wait()" in entry and "pdl_begin()" not in entry
    solve = text[re.search(r"\b%s\([^;{]*\{" % body, text).end():]
    solve = solve[:solve.index("a.p_dense[")]  # the result, behind the iterations
    loop = solve.index("it < a.max_iters")
    assert "pdl_next()" not in solve[:loop] and solve[loop:].count("pdl_next()") == 1
    assert solve.rindex("pdl_next()") > solve.rindex("beta")


# 2 x 2 x 2 cells; one cluster of 8 and of 16 CTAs; the cooperative grid
DIMS = [(2, 2, 2), (21, 22, 17), (9, 64, 48), (34, 65, 65), (40, 80, 33)]


@pytest.mark.gpu
def test_threads_give_the_bits_of_each_alone():
    from sdr_b200 import _lib
    from tests.test_gpu_tiles import _pair

    def solve(gpu, faces):
        out = []
        for _ in range(6):
            for w in range(3):
                gpu.set_face(w, faces[w])
            gpu.run_phase(_lib.PHASE_PROJECT, 1e-3)
            out.append((gpu.last_pcg_iters, gpu.pressure().tobytes()))
        return out

    solvers = [_pair(case, dims)[0] for dims in DIMS for case in ("full", "sparse")]
    faces = [[s.face(w) for w in range(3)] for s in solvers]
    alone = [solve(s, f) for s, f in zip(solvers, faces)]
    got = [None] * len(solvers)
    failed = []

    def work(k):
        try:
            got[k] = solve(solvers[k], faces[k])
        except Exception as e:  # reported below, by the main thread
            failed.append((k, e))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(solvers))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed
    assert all(np.all([a == b for a, b in zip(x, y)]) for x, y in zip(alone, got))
    assert all(it[0] >= 1 for runs in alone for it in runs)
