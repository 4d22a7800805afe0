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


@pytest.mark.gpu
@pytest.mark.parametrize("max_batch", [4, 100])
def test_a_run_that_fails_reports_every_edit(built_lib, max_batch):
    """A mode that no build takes: the first step cannot be queued.  No edit is reported as
    applied, and none is left queued for the world's next build."""
    w = world()
    before, used = w.grid.copy(), w.poolUsed
    n = 20
    es = (_lib.Edit * n)()
    for e, (shape, a, b, r) in zip(es, edits(n)):
        e.shape, e.r = shape, r
        e.a[:], e.b[:] = a, b
    res, order, applied = (_lib.EditResult * n)(), (ctypes.c_uint64 * n)(), ctypes.c_size_t()
    rc = _lib.load().px_serve_run(w._h, es, (ctypes.c_double * n)(), n, max_batch, 1 << 40, 7, None, res, order,
                                  ctypes.byref(applied))
    assert rc == 1 and applied.value == 0  # PX_E_INVALID_ARG
    assert all(r.status != 0 for r in res)
    w.build()
    np.testing.assert_array_equal(w.grid, before)
    assert w.poolUsed == used
    serving.serve(w, edits(n), np.zeros(n), max_batch=max_batch)  # and the world serves
    assert w.stats()["ops_applied"] == 2 + n
    w.close()
