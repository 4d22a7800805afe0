"""Programs that only the interpreter evaluates, on both sides of the passes' launch rule.

The classify and sub-block passes are compiled for two and for three blocks per SM; interpreted
programs take the latter from a tenth of the pairs on.  Trees of three to five primitives,
alone and among lean programs, around that line, against the oracle.
"""
import numpy as np
import pytest

from pixels_gb300 import config
from pixels_gb300.ir import Program
from pixels_gb300.shapes import box, cylinder, intersect, prism, rotateX, rotateY, rotateZ, sphere, subtract, union
from pixels_gb300.world import MODE_MIXED, VoxelWorld

import pyoracle

VPM, DIMS = 40.0, (320, 128, 320)
LIMIT, WEIGHT = 1 << 19, 10  # two blocks per SM: pairs + WEIGHT * interpreted pairs <= LIMIT


def tree(k, c, r):
    ring = [float(v) for j in range(8) for v in (r * np.cos(j * np.pi / 4), r * np.sin(j * np.pi / 4))]
    a, b, d, p = sphere(c, r), box(c, (r, r / 2, r * 1.2)), cylinder(c, r * 0.6, r * 1.3, "y"), prism(c, ring, c[1] - r, c[1] + r)
    return (union(a, b, d), subtract(union(rotateY(b, 0.4, c), d, p), rotateX(d, 0.8, c), a),
            rotateX(union(rotateZ(subtract(a, b), 0.3, c), rotateY(p, 0.2, c)), 0.5, c), intersect(union(a, b, d), p))[k % 4]


@pytest.mark.gpu
@pytest.mark.parametrize("trees,lean,two", [(40, 0, True), (150, 0, True), (300, 0, True), (310, 0, False), (250, 400, True), (300, 400, False)])
def test_trees_on_both_sides_of_the_rule(built_lib, trees, lean, two):
    rng = np.random.default_rng(trees)
    ext = np.array(DIMS) / VPM
    progs = [Program(), Program()]  # all ops, and the trees alone
    with config.using(VPM):
        for k in range(trees + lean):
            c = tuple(float(v) for v in rng.uniform(0.1, 0.9, 3) * ext)
            r = float(rng.uniform(0.1, 0.5))
            is_tree = k * trees // (trees + lean) != (k + 1) * trees // (trees + lean)
            s = tree(k, c, r) if is_tree else rotateY(box(c, (r, r, r)), 0.3, c)
            for p in progs[: 2 if is_tree else 1]:
                p.add_op(0 if k % 6 else 1, s, k % 60 + 1)
    pairs = []
    for prog in progs:
        w = VoxelWorld(*DIMS, vpm=VPM, mode=MODE_MIXED)
        w._pending = prog
        ir = prog.to_bytes()
        w.build()
        pairs.append(w.stats()["pairs"])
        o = pyoracle.OracleWorld(ir, VPM, DIMS, threads=8)
        np.testing.assert_array_equal(w.grid, o.grid)
        live = np.nonzero((o.grid != 0) & ((o.grid & 0x80000000) == 0))[0]
        idx = o.grid[live].astype(np.int64) - 1
        np.testing.assert_array_equal(w.pool.reshape(-1, 512)[idx], o.pool.reshape(-1, 512)[idx])
        w.close()
    assert (pairs[0] + WEIGHT * pairs[1] <= LIMIT) == two, pairs
