"""Short op lists in a large world: the tile lists of the few tiles they touch.

A list whose (op, tile) pairs are fewer than half the world's tiles is culled by one
warp per pair, anything else by one per tile.  Lists at the edges of a 32-op group, of one
op, of ops outside the world (no pair at all), overlapping and apart, on both sides of
the rule, as a first build, as an edit of the built world and requeued, against the
oracle: whole numbers, equal or wrong.
"""
import numpy as np
import pytest

from pixels_gb300 import _lib, config
from pixels_gb300.ir import Program
from pixels_gb300.shapes import box, capsule, sphere
from pixels_gb300.world import MODE_MIXED, VoxelWorld

import pyoracle

VPM, DIMS = 20.0, (328, 296, 312)  # 41 x 37 x 39 bricks, 1,100 tiles


def add_ops(prog, n, size, seed):
    rng = np.random.default_rng(seed)
    ext = np.array(DIMS) / VPM
    with config.using(VPM):
        for k in range(n):
            c = tuple(float(v) for v in (rng.uniform(0, 1, 3) if k % 3 else rng.uniform(0.4, 0.45, 3)) * ext)
            r = float(rng.uniform(0.3, 1.0) * size)
            if k % 7 == 6:
                c = (c[0] + 40.0, c[1], c[2])  # outside the world: no tile
            s = (sphere(c, r), box(c, (r, 0.5 * r, r)), capsule(c, (c[0] + r, c[1], c[2] - r), 0.4 * r))[k % 3]
            prog.add_op((0, 0, 1, 2)[int(rng.integers(4))], s, int(rng.integers(1, 60)))


def check(w, o):
    grid = w.grid
    np.testing.assert_array_equal(grid, o.grid)
    assert w.poolUsed == o.pool_used
    np.testing.assert_array_equal(w.freeBricks(), o.free_holes)
    live = np.nonzero((o.grid != 0) & ((o.grid & 0x80000000) == 0))[0]
    idx = o.grid[live].astype(np.int64) - 1
    np.testing.assert_array_equal(w.pool.reshape(-1, 512)[idx], o.pool.reshape(-1, 512)[idx])


@pytest.mark.gpu
@pytest.mark.parametrize("n,size", [(1, 0.2), (7, 0.2), (31, 0.3), (32, 0.3), (33, 0.3), (64, 0.5), (100, 1.5), (1024, 0.05),
                                    (1025, 0.05), (33, 6.0)])
def test_short_lists(built_lib, n, size):
    w = VoxelWorld(*DIMS, vpm=VPM, mode=MODE_MIXED)
    both = Program()
    for seed in (1, 2):  # a first build, then an edit of the built world
        part = Program()
        add_ops(part, n, size, 100 * n + seed)
        add_ops(both, n, size, 100 * n + seed)
        w._pending = part
        w.build()
    check(w, pyoracle.OracleWorld(both.to_bytes(), VPM, DIMS, threads=8))
    _lib.world_reset(w._h, True)  # the last list again, from its device tables
    _lib.build(w._h, MODE_MIXED)
    check(w, pyoracle.OracleWorld(part.to_bytes(), VPM, DIMS, threads=8))
    w.close()


@pytest.mark.gpu
def test_no_op_in_the_world(built_lib):
    w = VoxelWorld(*DIMS, vpm=VPM, mode=MODE_MIXED)
    prog = Program()
    with config.using(VPM):
        prog.add_op(0, sphere((60.0, 1.0, 1.0), 0.5), 7)
    w._pending = prog
    w.build()
    assert not w.grid.any() and w.poolUsed == 0
    _lib.world_reset(w._h, True)
    _lib.build(w._h, MODE_MIXED)
    assert not w.grid.any()
    w.close()
