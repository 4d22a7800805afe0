"""Builds of different worlds on several host threads and streams at once."""
import threading

import numpy as np
import pytest

from pixels_gb300 import _lib, config
from pixels_gb300.ir import Program
from pixels_gb300.shapes import box, rotateY, sphere
from pixels_gb300.world import MODE_FP64, MODE_MIXED, VoxelWorld

import pyoracle

VPM, DIMS = 40.0, (96, 80, 88)


def scene(seed, n):
    rng = np.random.default_rng(seed)
    prog = Program()
    with config.using(VPM):
        for k in range(n):
            c = tuple(float(v) for v in rng.uniform(0.3, 1.7, 3))
            r = float(rng.uniform(0.05, 0.3))
            prog.add_op(k % 3, rotateY(box(c, (r, r, r)), 0.3, c) if k % 2 else sphere(c, r), k % 50 + 1)
    return prog.to_bytes()


@pytest.mark.gpu
def test_worlds_on_threads_of_their_own(built_lib):
    """Four threads, each with a world and a stream: every build equals the oracle, and reports its own
    launches, whatever the others launch meanwhile."""
    import torch
    torch.cuda.init()
    jobs = [(scene(s, n), mode) for s, (n, mode) in enumerate([(40, MODE_MIXED), (900, MODE_MIXED), (40, MODE_FP64), (7, MODE_MIXED)])]
    grids = [pyoracle.OracleWorld(ir, VPM, DIMS).grid for ir, _ in jobs]
    launches = [set() for _ in jobs]
    errors = []

    def work(i, builds):
        try:
            ir, mode = jobs[i]
            s = torch.cuda.Stream()
            w = VoxelWorld(*DIMS, vpm=VPM, mode=mode)
            for _ in range(builds):
                _lib.world_reset(w._h, stream=s.cuda_stream)
                _lib.submit_ops(w._h, ir)
                _lib.build(w._h, mode, s.cuda_stream)
                launches[i].add(w.stats()["kernel_launches"])
                s.synchronize()
                np.testing.assert_array_equal(w.grid, grids[i])
            w.close()
        except BaseException as e:  # reported by the test's thread
            errors.append((i, e))

    for i in range(len(jobs)):
        work(i, 2)
    alone = [set(x) for x in launches]
    threads = [threading.Thread(target=work, args=(i, 60)) for i in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    assert launches == alone and all(len(x) == 1 for x in launches), (alone, launches)
