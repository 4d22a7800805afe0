"""Serving on small worlds that already have holes.

px_serve_run sizes the free lists for its largest step before the first edit; a world built
from a few ops has short ones, and the holes in them have to survive: the next allocations
pop them in LIFO order (VoxelWorld.ts:112-127).  Against the oracle, pool indices and free
list included.
"""
import numpy as np
import pytest

import pyoracle
from pixels_gb300 import config, serving
from pixels_gb300.ir import Program
from pixels_gb300.shapes import box, sphere
from pixels_gb300.world import MODE_FP64, MODE_MIXED, VoxelWorld

from test_gpu_parity import assert_same_world
from test_gpu_serving import _concat_ir

VPM, DIMS = 40.0, (128, 96, 112)


def scene(n_holes):
    """A slab, then spheres added and boxes that clear them: `n_holes` or more freed bricks."""
    prog = Program()
    with config.using(VPM):
        prog.add_op(0, box((1.6, 0.4, 1.4), (1.6, 0.4, 1.4)), 3)
        for k in range(n_holes):
            c = (0.3 + 0.2 * (k % 13), 1.3 + 0.4 * (k // 13), 0.4 + 0.17 * (k % 11))
            prog.add_op(0, sphere(c, 0.05), 5)
            if k % 5 != 4:
                prog.add_op(1, box(c, (0.1, 0.1, 0.1)), 0)
    return prog


@pytest.mark.gpu
@pytest.mark.parametrize("mode", [MODE_MIXED, MODE_FP64])
@pytest.mark.parametrize("n_holes,builds", [(1, 1), (1, 2), (20, 1), (20, 2)])
def test_holes_survive_the_reservation(built_lib, n_holes, builds, mode):
    prog = scene(n_holes)
    w = VoxelWorld(*DIMS, initialPoolBricks=4, vpm=VPM, mode=mode)
    parts = [prog]
    w._pending = prog
    w.build()
    if builds == 2:  # the free list is in the other buffer
        extra = Program()
        with config.using(VPM):
            extra.add_op(0, sphere((2.9, 2.0, 2.5), 0.05), 6)
            extra.add_op(1, box((2.9, 2.0, 2.5), (0.1, 0.1, 0.1)), 0)
        w._pending = extra
        w.build()
        parts.append(extra)
    assert len(w.freeBricks()) > 0
    rng = np.random.default_rng(n_holes)
    edits = []
    for k in range(40):
        c = tuple(float(v) for v in rng.uniform(0.2, 0.8, 3) * np.array([3.2, 0.9, 2.8]))
        edits.append((serving.SPHERE, c, c, float(rng.uniform(0.02, 0.2))))
    res, order = serving.serve(w, edits, np.zeros(len(edits)), max_batch=16)
    assert (res["status"] == 0).all() and len(order) == len(edits)
    whole = Program()
    for p in parts + [serving.carve_program(edits, order, VPM)]:
        whole = _join(whole, p)
    assert_same_world(w, pyoracle.OracleWorld(whole.to_bytes(), VPM, DIMS))
    w.close()


def _join(a, b):
    from pixels_gb300.ir import decode
    p = Program()
    ops, code, params = decode(_concat_ir(a, b))
    p.ops = [tuple(x.tolist() if hasattr(x, "tolist") else x for x in o) for o in ops]
    p.code = [tuple(int(v) for v in c) for c in code]
    p.params = [float(v) for v in params]
    return p
