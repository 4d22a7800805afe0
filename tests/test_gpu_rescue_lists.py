"""Long lists of voxels left to intervals and float64, on grids of any size.

Faces that pass through voxel centres leave every one of their voxels to the rescue
list.  Builds that share the GPU run on as few blocks as their pairs ask for; the
warps that take the list follow its length, on one block as on the whole GPU.  Lists
shorter than one warp's round, at the edges of a round, and longer than what half the
blocks take in one round each, against the oracle: whole numbers, equal or wrong.
"""
import statistics

import numpy as np
import pytest

from pixels_gb300 import _lib, config
from pixels_gb300.batch import Batch
from pixels_gb300.ir import Program
from pixels_gb300.shapes import box, rotateY
from pixels_gb300.world import MODE_MIXED, VoxelWorld

import pyoracle

VPM, DIMS = 64.0, (256, 128, 128)


def boxes(n, side, shift, paint=5):
    """n boxes under a rotation by zero (no lone box: evaluated per voxel), faces `shift`
    voxels from voxel centres."""
    rng = np.random.default_rng(100 * n + side)
    prog = Program()
    with config.using(VPM):
        for i in range(n):
            lo = rng.integers(4, np.array(DIMS) - side - 4)
            c = tuple(float(v) for v in (lo + 0.5 + shift + side / 2) / VPM)
            prog.add_op(i % 3 == 2, rotateY(box(c, (side / 2 / VPM,) * 3), 0.0, c), paint)
    return prog


def built(prog):
    w = VoxelWorld(*DIMS, vpm=VPM, mode=MODE_MIXED)
    w._pending = prog
    w.build()
    return w


@pytest.mark.gpu
@pytest.mark.parametrize("pairs_per_block", [0, 64, 1 << 20])
@pytest.mark.parametrize("n,side", [(1, 1), (1, 2), (1, 3), (1, 30), (1, 100), (12, 24)])
def test_long_rescue_lists(built_lib, n, side, pairs_per_block):
    prog = boxes(n, side, 0.0)
    o = pyoracle.OracleWorld(prog.to_bytes(), VPM, DIMS)
    w = built(prog)
    with Batch([w], n_streams=1, pairs_per_block=pairs_per_block) as b:
        b.run()
        assert w.stats()["rescued_voxel"] >= 6 * (side - 1) ** 2
        np.testing.assert_array_equal(w.grid, o.grid)
        live = np.nonzero((o.grid != 0) & ((o.grid & 0x80000000) == 0))[0]
        idx = o.grid[live].astype(np.int64) - 1
        np.testing.assert_array_equal(w.pool.reshape(-1, 512)[idx], o.pool.reshape(-1, 512)[idx])
    w.close()


@pytest.mark.gpu
def test_a_long_list_on_one_block_uses_the_block(built_lib):
    """One block, 60,002 voxels to resolve: eight warps take 4 times what the same boxes half a
    voxel aside cost, one warp alone took 16 times."""
    ms = []
    for shift in (0.0, 0.3):
        w = built(boxes(1, 100, shift))
        with Batch([w], n_streams=1, pairs_per_block=1 << 20) as b:
            b.run()
            ms.append(statistics.median(b.run() for _ in range(5)))
        w.close()
    assert ms[0] < 8 * ms[1], ms
