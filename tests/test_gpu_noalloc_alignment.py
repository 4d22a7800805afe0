"""px_derive_noalloc on pools off the 16-byte boundary and ragged grids.

A pool that starts on a 16-byte boundary is read 16 bytes at a time, any other
4 bytes at a time; super cells on the far faces are partial; a grid may refer to
a pool brick twice or not at all.  Counts and bytes, equal or wrong.
"""
import numpy as np
import pytest

from pixels_gb300 import _lib

from test_zz_no_alloc import _expected, _run_twice


@pytest.mark.gpu
@pytest.mark.parametrize("offset", [0, 4, 8, 12])
@pytest.mark.parametrize("bricks", [(1, 1, 1), (4, 4, 4), (9, 6, 5), (33, 18, 21)])
def test_pool_offsets_and_ragged_grids(built_lib, bricks, offset):
    import torch
    rng = np.random.default_rng(offset + bricks[0])
    n = bricks[0] * bricks[1] * bricks[2]
    n_pool = max(1, n // 2)
    grid = np.where(rng.random(n) < 0.7, rng.integers(1, n_pool + 1, n), 0).astype(np.uint32)
    uni = rng.random(n) < 0.2
    grid[uni] = 0x80000000 | rng.integers(1, 64, int(uni.sum())).astype(np.uint32)
    pool = rng.integers(0, 70, n_pool * 512).astype(np.uint16)
    pool[rng.random(pool.size) < 0.4] = 0
    g_d = torch.from_numpy(grid.view(np.int32)).cuda()
    p_d = torch.zeros(pool.size + 8, dtype=torch.int16, device="cuda:0")
    p_d[offset // 2: offset // 2 + pool.size] = torch.from_numpy(pool.view(np.int16)).cuda()
    torch.cuda.synchronize()
    sup, den = _expected(grid, pool, bricks)
    s_d, d_d = _run_twice(g_d.data_ptr(), p_d.data_ptr() + offset, bricks, n_pool, sup, den)
    if (grid[(grid & 0x80000000) == 0] == n_pool).any():  # a brick beyond the pool: reported, and its density 0
        with pytest.raises(_lib.PxError) as e:
            _lib.derive_noalloc(g_d.data_ptr(), p_d.data_ptr() + offset, bricks, n_pool - 1, s_d.data_ptr(), d_d.data_ptr())
        assert e.value.code == 1
        bad = grid == n_pool
        den[bad] = 0
        np.testing.assert_array_equal(d_d.cpu().numpy(), den)
    _lib.derive_noalloc(g_d.data_ptr(), p_d.data_ptr() + offset, bricks, n_pool, s_d.data_ptr(), d_d.data_ptr())
