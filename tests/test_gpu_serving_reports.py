"""What a serving run reports: the ops it applied, and each edit's outcome."""
import ctypes

import numpy as np
import pytest

from pixels_gb300 import _lib, config, serving
from pixels_gb300.ir import Program
from pixels_gb300.shapes import box
from pixels_gb300.world import MODE_MIXED, VoxelWorld

VPM, DIMS = 40.0, (128, 96, 112)


def world():
    prog = Program()
    with config.using(VPM):
        prog.add_op(0, box((1.6, 1.2, 1.4), (1.2, 0.8, 1.0)), 3)
        prog.add_op(0, box((1.6, 1.2, 1.4), (0.3, 1.1, 0.3)), 4)
    w = VoxelWorld(*DIMS, vpm=VPM, mode=MODE_MIXED)
    w._pending = prog
    w.build()
    return w


def edits(n, seed=1):
    rng = np.random.default_rng(seed)
    out = []
    for _ in range(n):
        c = tuple(float(v) for v in rng.uniform(0.3, 0.7, 3) * np.array(DIMS) / VPM)
        out.append((serving.SPHERE, c, c, float(rng.uniform(0.02, 0.1))))
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("n,max_batch", [(0, 8), (1, 8), (8, 8), (40, 8), (45, 16), (30, 1)])
def test_ops_applied_counts_each_edit_once(built_lib, n, max_batch):
    w = world()
    total = 2
    for run in range(2):
        serving.serve(w, edits(n, run), np.zeros(n), max_batch=max_batch)
        total += n
        assert w.stats()["ops_applied"] == total
    with config.using(VPM):
        w.submit(1, box((1.6, 1.2, 1.4), (0.1, 0.1, 0.1)), 0)
    w.build()
    assert w.stats()["ops_applied"] == total + 1
    w.close()
