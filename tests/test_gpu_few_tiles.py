"""Op lists of up to 1,024 ops that touch few tiles of a large world: every group of 32.

Lists whose (op, tile) pairs are fewer than half the world's tiles are culled by one warp
per pair, which finds its op by a 32-way search and holds one ballot word per group of 32
ops.  Lists around the edges of groups, of search steps and of the largest length; tiles that
ops of the first, middle and last groups share; runs of ops without any pair at the steps'
boundaries.  Each parameter set states on which side of the rule it lies, counted as the host
does.  Against the oracle: whole numbers, equal or wrong.
"""
import numpy as np
import pytest

from pixels_gb300 import _lib, config
from pixels_gb300.ir import Program, decode
from pixels_gb300.shapes import box, capsule, sphere
from pixels_gb300.world import MODE_FP64, MODE_MIXED, VoxelWorld

import pyoracle

VPM, DIMS = 20.0, (640, 320, 512)  # 80 x 40 x 64 bricks: 20 x 10 x 16 = 3,200 tiles
MAX_FEW = 1024


def op_list(n, seed, spread, outside):
    """n small ops, two thirds of them in one corner a few tiles wide (`spread`: a third all over),
    those that `outside` names beyond the world."""
    rng = np.random.default_rng(seed)
    ext = np.array(DIMS) / VPM
    prog = Program()
    with config.using(VPM):
        for k in range(n):
            c = rng.uniform(0.02, 0.98, 3) * ext if spread and k % 3 == 1 else 3.0 + rng.uniform(0, 2.5, 3)
            if outside(k):
                c = c + np.array([100.0, 0.0, 0.0])
            c = tuple(float(v) for v in c)
            r = float(rng.uniform(0.05, 0.15))
            s = (sphere(c, r), box(c, (r, 0.5 * r, r)), capsule(c, (c[0] + r, c[1], c[2] - r), 0.5 * r))[int(rng.integers(3))]
            prog.add_op((0, 0, 0, 1, 2)[int(rng.integers(5))], s, int(rng.integers(1, 60)))
    return prog


def tile_pairs(prog):
    """(op, tile) pairs of a list: tiles of 4^3 bricks in each op's brick box (shapes.ts:341-347)."""
    ops = decode(prog.to_bytes())[0]
    v0 = np.maximum(0, np.floor(ops["min"] * VPM - 0.5))
    v1 = np.minimum(np.array(DIMS) - 1, np.ceil(ops["max"] * VPM + 0.5))
    t = (v1 // 32 - v0 // 32 + 1).prod(axis=1)
    return int(t[(v0 <= v1).all(axis=1)].sum())


def check(w, o):
    grid = w.grid
    np.testing.assert_array_equal(grid, o.grid)
    assert w.poolUsed == o.pool_used
    np.testing.assert_array_equal(w.freeBricks(), o.free_holes)
    live = np.nonzero((o.grid != 0) & ((o.grid & 0x80000000) == 0))[0]
    idx = o.grid[live].astype(np.int64) - 1
    np.testing.assert_array_equal(w.pool.reshape(-1, 512)[idx], o.pool.reshape(-1, 512)[idx])


OUTSIDE = {"none": lambda k: False, "runs": lambda k: k % 32 in (0, 1, 31) or 200 <= k < 300 or k >= 1000,
           "most": lambda k: k % 33 != 7}


@pytest.mark.gpu
@pytest.mark.parametrize("n,spread,outside,few", [
    (65, True, "none", True), (96, True, "runs", True), (97, True, "none", True), (100, True, "none", True),
    (512, True, "runs", True), (512, False, "none", True), (993, False, "runs", True), (1023, False, "runs", True),
    (1024, False, "runs", True), (1024, True, "most", True), (1025, True, "most", False), (1024, True, "none", False)])
def test_lists_of_many_groups(built_lib, n, spread, outside, few):
    prog = op_list(n, n, spread, OUTSIDE[outside])
    pairs, tiles = tile_pairs(prog), np.prod([(d // 8 + 3) // 4 for d in DIMS])
    assert (n <= MAX_FEW and 2 * pairs < tiles) == few, (pairs, tiles)
    w = VoxelWorld(*DIMS, vpm=VPM, mode=MODE_MIXED)
    _lib.submit_ops(w._h, prog.to_bytes())
    w.build()
    o = pyoracle.OracleWorld(prog.to_bytes(), VPM, DIMS, threads=8)
    check(w, o)
    _lib.world_reset(w._h, True)  # the same list from its device tables
    _lib.build(w._h, MODE_MIXED)
    check(w, o)
    w.close()


@pytest.mark.gpu
@pytest.mark.parametrize("mode", [MODE_MIXED, MODE_FP64])
@pytest.mark.parametrize("gap", [30, 31, 32, 33, 63, 64, 65, 200])
def test_ops_without_pairs_between(built_lib, gap, mode):
    """Runs of `gap` ops outside the world between single ones of a few pairs each: the ops of
    32 neighbouring (op, brick) pairs lie far apart in the list."""
    prog = op_list(20 * (gap + 1), gap, False, lambda k: k % (gap + 1) != gap // 2)
    w = VoxelWorld(*DIMS, vpm=VPM, mode=mode)
    _lib.submit_ops(w._h, prog.to_bytes())
    w.build()
    assert w.poolUsed > 0
    check(w, pyoracle.OracleWorld(prog.to_bytes(), VPM, DIMS, threads=8))
    w.close()
