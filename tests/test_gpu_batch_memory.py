"""Host memory of batched worlds: the op-list conversion's workspace is given back.

Worlds keep the arrays an op list was converted in for the next list.  A batched world
queues no list, so those arrays go when the batch is made; many worlds side by side then
hold their op tables only.
"""
import ctypes

import numpy as np
import pytest

from pixels_gb300.batch import Batch
from pixels_gb300.scenes.synthetic import synthetic_program
from pixels_gb300.world import MODE_MIXED, VoxelWorld


class _Info(ctypes.Structure):
    _fields_ = [(n, ctypes.c_size_t) for n in ("arena", "ordblks", "smblks", "hblks", "hblkhd", "usmblks", "fsmblks",
                                               "uordblks", "fordblks", "keepcost")]


def in_use():
    """Bytes the C allocator has handed out."""
    libc = ctypes.CDLL("libc.so.6")
    libc.mallinfo2.restype = _Info
    m = libc.mallinfo2()
    return m.uordblks + m.hblkhd


@pytest.mark.gpu
def test_batched_worlds_give_their_workspace_back(built_lib):
    dims, n = (160, 88, 120), 12
    progs = [synthetic_program(k + 1, 2000, 40.0, (4.0, 2.2, 3.0)).to_bytes() for k in range(n)]
    worlds = [VoxelWorld(*dims, vpm=40.0, mode=MODE_MIXED) for _ in range(n)]
    with Batch(_built(worlds[:1], progs[:1])):  # what the first batch of a process sets up
        pass
    base = in_use()
    _built(worlds[1:], progs[1:])
    built = in_use()
    with Batch(worlds[1:]) as b:
        b.run()
        batched = in_use()
        grids = [w.grid for w in worlds[1:]]
    # op tables and the workspace, about as large; a batch holds a second copy of the tables
    assert batched - built < 0.25 * (built - base), (base, built, batched)
    for w, g, p in zip(worlds[1:], grids, progs[1:]):  # and the next list still queues
        w._lib.world_reset(w._h)
        w._lib.submit_ops(w._h, p)
        w.build()
        np.testing.assert_array_equal(w.grid, g)
    for w in worlds:
        w.close()


def _built(worlds, progs):
    for w, p in zip(worlds, progs):
        w._lib.submit_ops(w._h, p)
        w.build()
    return worlds
