"""A requeued list is culled by the table that is on the device.

The op tables of the last build stay on the device, and px_world_reset(requeue) builds
from them.  Lists of each form of the cull table -- op order, spatial order, the few
(op, tile) pairs of an edit -- are built, then a list of no ops is queued and dropped by
the reset (or refused), or the world goes into a batch: the rebuild equals the oracle's
world of the last list.  Whole numbers, equal or wrong.
"""
import numpy as np
import pytest

from pixels_gb300 import _lib, config, serving
from pixels_gb300.batch import Batch
from pixels_gb300.ir import Program
from pixels_gb300.shapes import box, capsule, sphere
from pixels_gb300.world import MODE_FP64, MODE_MIXED, VoxelWorld

import pyoracle

VPM, DIMS = 20.0, (328, 296, 312)  # 41 x 37 x 39 bricks, 1,100 tiles


def scene(form):
    """Ops in rows along x (their order is spatial: CULL_SEQ), the same kind scattered
    (CULL_SORTED), or one stroke (CULL_FEW: fewer tiles than half the world's)."""
    n = 1 if form == "few" else 300
    rng = np.random.default_rng(n)
    ext = np.array(DIMS) / VPM
    prog = Program()
    with config.using(VPM):
        for k in range(n):
            c = rng.uniform(0.05, 0.95, 3) * ext
            if form == "rows":
                c[0] = (k + 0.5) / n * ext[0]
            c = tuple(float(v) for v in c)
            r = float(rng.uniform(0.2, 0.7))
            s = (sphere(c, r), box(c, (r, 0.5 * r, r)), capsule(c, (c[0] + r, c[1], c[2] - r), 0.4 * r))[k % 3]
            prog.add_op(0 if k % 4 else 1, s, k % 60 + 1) if k else prog.add_op(0, s, 7)
    return prog


def check(w, o):
    grid = w.grid
    np.testing.assert_array_equal(grid, o.grid)
    assert w.poolUsed == o.pool_used
    np.testing.assert_array_equal(w.freeBricks(), o.free_holes)
    live = np.nonzero((o.grid != 0) & ((o.grid & 0x80000000) == 0))[0]
    idx = o.grid[live].astype(np.int64) - 1
    np.testing.assert_array_equal(w.pool.reshape(-1, 512)[idx], o.pool.reshape(-1, 512)[idx])


@pytest.mark.gpu
@pytest.mark.parametrize("mode", [MODE_MIXED, MODE_FP64])
@pytest.mark.parametrize("form", ["rows", "scattered", "few"])
@pytest.mark.parametrize("between", ["empty", "empty twice", "refused", "batch"])
def test_requeue_after_a_list_that_is_not_built(built_lib, form, between, mode):
    prog = scene(form)
    o = pyoracle.OracleWorld(prog.to_bytes(), VPM, DIMS, threads=8)
    w = VoxelWorld(*DIMS, vpm=VPM, mode=mode)
    w._pending = prog
    w.build()
    empty = Program().to_bytes()
    if between == "refused":
        with pytest.raises(_lib.PxError):
            _lib.submit_ops(w._h, scene("few").to_bytes()[:-8])
    else:
        for _ in range(2 if between == "empty twice" else 1):
            _lib.submit_ops(w._h, empty)
    if between == "batch":
        with Batch([w], n_streams=1, pairs_per_block=0) as b:
            b.run()
            check(w, o)
    else:
        _lib.world_reset(w._h, True)
        _lib.build(w._h, mode)
        check(w, o)
    w.close()


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["rows", "scattered", "few"])
@pytest.mark.parametrize("n", [0, 5])
def test_requeue_after_serving_that_builds_nothing(built_lib, form, n):
    """px_serve_run grows the op tables for its largest step before the first edit; with no
    edit, or none that fits the pool, nothing is uploaded into them.  The requeued list is not
    in the grown tables: it has to be uploaded again."""
    prog = scene(form)
    o = pyoracle.OracleWorld(prog.to_bytes(), VPM, DIMS, threads=8)
    w = VoxelWorld(*DIMS, vpm=VPM, mode=MODE_MIXED)
    w._pending = prog
    w.build()
    edits = [(0, (5.0, 5.0, 5.0 + i), (0.0, 0.0, 0.0), 1.0) for i in range(n)]
    res, order = serving.serve(w, edits, np.zeros(n), max_batch=4096, pool_budget=w.liveBricks)
    assert len(order) == 0 and (res["status"] == 3).all()
    check(w, o)
    for _ in range(2):  # uploaded again, then resident
        _lib.world_reset(w._h, True)
        _lib.build(w._h, MODE_MIXED)
        check(w, o)
    w.close()


@pytest.mark.gpu
@pytest.mark.parametrize("mode", [MODE_MIXED, MODE_FP64])
@pytest.mark.parametrize("first,second", [("scattered", "few"), ("few", "scattered"), ("rows", "rows"), ("few", "few")])
def test_two_lists_queued_and_requeued(built_lib, first, second, mode):
    """Two lists queued before one build: their cull table is made at the build, and requeued with
    the tables; then a list of another form, and the two again as one."""
    parts = [scene(first), scene(second)]
    whole = Program()
    for p in parts:
        code, par = len(whole.code), len(whole.params)
        whole.ops += [tuple(o[:5]) + (o[5] + code,) + tuple(o[6:]) for o in p.ops]
        whole.code += [(w0, off + par) for w0, off in p.code]
        whole.params += p.params
    o = pyoracle.OracleWorld(whole.to_bytes(), VPM, DIMS, threads=8)
    w = VoxelWorld(*DIMS, vpm=VPM, mode=mode)
    for p in parts:
        _lib.submit_ops(w._h, p.to_bytes())
    _lib.build(w._h, mode)
    check(w, o)
    _lib.world_reset(w._h, True)
    _lib.build(w._h, mode)
    check(w, o)
    _lib.world_reset(w._h)
    _lib.submit_ops(w._h, scene("few").to_bytes())
    _lib.build(w._h, mode)
    _lib.world_reset(w._h)
    _lib.submit_ops(w._h, whole.to_bytes())
    _lib.build(w._h, mode)
    check(w, o)
    w.close()
