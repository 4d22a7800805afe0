"""Served steps whose work lists run out of room.

A step reserves staging slots from a guess, and pipelined steps cannot grow them: later
ones are queued behind.  Bursts in solid material, where every brick an edit touches ends
mixed, pass the guess.  Such a step is built again alone and the burst goes on: every edit is
applied, in arrival order, and the world equals the oracle's, pool indices and free list
included.
"""
import numpy as np
import pytest

import pyoracle
from pixels_gb300 import _lib, config, serving
from pixels_gb300.ir import Program
from pixels_gb300.shapes import box
from pixels_gb300.world import MODE_FP64, MODE_MIXED, VoxelWorld

from test_gpu_parity import assert_same_world
from test_gpu_serving import _concat_ir

VPM, DIMS = 40.0, (512, 256, 384)
EXT = np.array(DIMS) / VPM


def solid(derive=False, mode=MODE_MIXED):
    prog = Program()
    with config.using(VPM):
        prog.add_op(0, box(tuple(float(v) for v in EXT / 2), tuple(float(v) for v in EXT)), 7)
    w = VoxelWorld(*DIMS, initialPoolBricks=64, vpm=VPM, mode=mode, derive_on_build=derive)
    w._pending = prog
    w.build()
    return prog, w


def burst(n, r, seed):
    """n spheres of radius r apart from each other (each cuts bricks of its own)."""
    rng = np.random.default_rng(seed)
    cells = np.stack(np.meshgrid(*[np.arange(0.4, e - 0.3, 0.6) for e in EXT], indexing="ij"), -1).reshape(-1, 3)
    at = cells[rng.permutation(len(cells))[:n]] + rng.uniform(-0.05, 0.05, (n, 3))
    return [(serving.SPHERE, tuple(float(v) for v in c), tuple(float(v) for v in c), r) for c in at]


@pytest.mark.gpu
@pytest.mark.parametrize("n,max_batch,derive,mode", [
    (700, 700, False, MODE_MIXED), (1400, 512, False, MODE_MIXED), (1400, 512, True, MODE_MIXED), (1400, 256, False, MODE_FP64),
    (900, 1000, False, MODE_MIXED)])
def test_every_brick_of_a_step_ends_mixed(built_lib, n, max_batch, derive, mode):
    prog, w = solid(derive, mode)
    edits = burst(n, 0.21, n)
    for again in range(2):  # the second burst finds a world with the sizes the first one asked for
        res, order = serving.serve(w, edits, np.zeros(n), max_batch=max_batch)
        assert (res["status"] == 0).all()
        assert list(order) == list(range(n))
        assert (res["dev_end_ms"] > res["dev_start_ms"]).all() and (res["done_s"] > 0).all()
        carves = serving.carve_program(edits, order, VPM)
        whole = _concat_ir(prog, carves)
        if not again:
            assert_same_world(w, pyoracle.OracleWorld(whole, VPM, DIMS, threads=8))
            # a plain build of more ops follows the served steps
            extra = Program()
            with config.using(VPM):
                extra.add_op(0, box((3.0, 3.0, 3.0), (1.0, 0.7, 0.9)), 9)
            w._pending = extra
            w.build()
            two = Program()
            for part in (prog, carves, extra):
                two.ops, two.code, two.params = _append(two, part)
            assert_same_world(w, pyoracle.OracleWorld(two.to_bytes(), VPM, DIMS, threads=8))
            _lib.world_reset(w._h)
            w._pending = prog
            w.build()
        else:
            assert_same_world(w, pyoracle.OracleWorld(whole, VPM, DIMS, threads=8))
    w.close()


def _append(a, b):
    from pixels_gb300.ir import decode
    ops, code, params = decode(_concat_ir(a, b))
    return ([tuple(x.tolist() if hasattr(x, "tolist") else x for x in o) for o in ops],
            [tuple(int(v) for v in c) for c in code], [float(v) for v in params])


@pytest.mark.gpu
def test_rejections_between_steps_that_wait_again(built_lib):
    """Edits too large for the pool are rejected once, also where the step behind them failed and
    its own edits had to wait again."""
    prog, w = solid()
    edits = burst(1200, 0.21, 5)
    huge = (serving.SPHERE, (6.0, 3.0, 5.0), (6.0, 3.0, 5.0), 40.0)  # every brick of the world
    edits = edits[:300] + [huge] + edits[300:700] + [huge] + edits[700:]
    res, order = serving.serve(w, edits, np.zeros(len(edits)), max_batch=400, pool_budget=60000)
    ok = [i for i in range(len(edits)) if edits[i] is not huge]
    assert list(np.nonzero(res["status"])[0]) == [300, 701] and (res["status"][[300, 701]] == 3).all()
    assert list(order) == ok
    o = pyoracle.OracleWorld(_concat_ir(prog, serving.carve_program(edits, order, VPM)), VPM, DIMS, threads=8)
    assert_same_world(w, o)
    w.close()
