"""The apply pass on crowded bricks against the oracle, bit for bit.

A warp of the apply pass takes one brick at a time, or four where every warp
has many; it looks up the first entries of a brick's tile list together and the
rest 32 at a time, and fetches the next painted pair's values ahead.  Lists just
below, at and beyond those sizes, with constant and procedural paints, adds,
carves and repaints mixed, in both takes: whole numbers, so equal or wrong.
"""
import numpy as np
import pytest

from pixels_gb300 import config
from pixels_gb300.ir import Program
from pixels_gb300.paints import noise, tufted
from pixels_gb300.shapes import box, capsule, rotateY, roundBox, sphere
from pixels_gb300.world import MODE_FP64, MODE_MIXED, VoxelWorld

import pyoracle


def crowded(vpm, dims, n_ops, seed, cover):
    rng = np.random.default_rng(seed)
    ext = np.array(dims) / vpm
    prog = Program()
    with config.using(vpm):
        if cover:  # every brick is in some op's list
            prog.add_op(0, box(tuple(ext / 2), tuple(ext)), 0x0105)
        for _ in range(n_ops):
            c = tuple(float(v) for v in rng.uniform(0, 1, 3) * ext)
            h = float(rng.uniform(0.1, 0.5) * ext.min())
            s = [lambda: sphere(c, h), lambda: roundBox(c, (h, 0.6 * h, 0.8 * h), 0.2 * h),
                 lambda: rotateY(box(c, (h, h, 0.5 * h)), float(rng.uniform(0, 3)), c),
                 lambda: capsule(c, tuple(float(v) for v in c + rng.normal(size=3) * h), 0.5 * h)][int(rng.integers(4))]()
            kind = int(rng.choice([0, 0, 0, 1, 2, 2]))
            value = int(rng.integers(1, 60)) | int(rng.integers(256)) << 8
            if kind != 1 and rng.random() < 0.4:
                f = rng.uniform(0.5, 4, 3)
                value = noise(int(rng.integers(1 << 31)), float(np.float32(rng.uniform(10, 80))), float(np.float32(f[0])),
                              float(np.float32(f[1])), float(np.float32(f[2])), 0.1, value, int(rng.integers(3)))
            prog.add_op(kind, s, value if kind != 1 else 0)
    return prog


@pytest.mark.gpu
@pytest.mark.parametrize("mode", [MODE_FP64, MODE_MIXED])
@pytest.mark.parametrize("vpm,dims,n_ops,cover", [
    (20.0, (8, 8, 8), 1, False), (20.0, (24, 16, 24), 31, False), (20.0, (24, 16, 24), 32, False),
    (20.0, (16, 24, 16), 33, False), (20.0, (16, 16, 16), 64, False), (20.0, (24, 24, 16), 150, False),
    # enough bricks that a warp takes four at a time, most of them with more than eight entries
    (20.0, (344, 344, 344), 24, True),
])
def test_crowded_bricks(built_lib, mode, vpm, dims, n_ops, cover):
    if cover and mode == MODE_FP64:
        pytest.skip("the apply pass is the same in both forms; the large world once")
    prog = crowded(vpm, dims, n_ops, n_ops, cover)
    o = pyoracle.OracleWorld(prog.to_bytes(), vpm, dims, threads=8)
    w = VoxelWorld(*dims, initialPoolBricks=4, vpm=vpm, mode=mode)
    w._pending = prog
    w.build()
    grid = w.grid
    np.testing.assert_array_equal(grid, o.grid)
    assert w.poolUsed == o.pool_used
    np.testing.assert_array_equal(w.freeBricks(), o.free_holes)
    live = np.nonzero((o.grid != 0) & ((o.grid & 0x80000000) == 0))[0]
    idx = o.grid[live].astype(np.int64) - 1
    np.testing.assert_array_equal(w.pool.reshape(-1, 512)[idx], o.pool.reshape(-1, 512)[idx])
    w.close()


@pytest.mark.gpu
@pytest.mark.parametrize("mode", [MODE_FP64, MODE_MIXED])
def test_paints_past_the_slot_budget(built_lib, mode):
    """A painted op over 65^3 bricks has more (op, brick) pairs than there are paint slots
    (262,144): its paints are called by the apply pass, the costly kind keeps its slots."""
    vpm, dims = 20.0, (520, 520, 520)
    prog = Program()
    with config.using(vpm):
        prog.add_op(0, sphere((9.0, 9.0, 9.0), 2.5), 0x0305)
        prog.add_op(0, capsule((0.5, 0.5, 0.5), (25.5, 25.5, 25.5), 0.4), noise(77, 31.0, 1.5, 2.5, 0.75, 0.1, 0x0107, 9))
        prog.add_op(2, capsule((25.5, 0.5, 0.5), (0.5, 25.5, 25.5), 0.6), noise(5, 12.0, 2.5, 0.5, 3.0, -0.1, 0x0211, 0x0312))
        prog.add_op(0, roundBox((12.0, 12.0, 11.0), (1.0, 0.6, 0.8), 0.1), tufted(11.0, 11.4, 21))
        prog.add_op(1, sphere((12.6, 12.2, 11.2), 0.7), 0)
    o = pyoracle.OracleWorld(prog.to_bytes(), vpm, dims, threads=8)
    assert o.stats["paint_evals"] > 0
    w = VoxelWorld(*dims, vpm=vpm, mode=mode)
    w._pending = prog
    w.build()
    assert w.stats()["pairs"] > 2 * 262144
    grid = w.grid
    np.testing.assert_array_equal(grid, o.grid)
    assert w.poolUsed == o.pool_used
    live = np.nonzero((o.grid != 0) & ((o.grid & 0x80000000) == 0))[0]
    idx = o.grid[live].astype(np.int64) - 1
    np.testing.assert_array_equal(w.pool.reshape(-1, 512)[idx], o.pool.reshape(-1, 512)[idx])
    w.close()
