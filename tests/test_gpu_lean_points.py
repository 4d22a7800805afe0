"""Float32 point values of the lean programs against float64, every primitive and stage.

The mixed form decides one- and two-primitive programs from a float32 value and a
bound of its error derived per op.  Every primitive, alone, under each kind of
rotation and a composed run, combined with a second one and offset, is built in
both forms and in validation mode, which evaluates each boundary voxel in float64
as well and counts values outside the bound: none may be.  Sizes lie on both sides
of the largest bound a lean program may have (1/128 voxel), beyond which the op
takes the interval interpreter.  All results are whole numbers, equal to the oracle's.
"""
import numpy as np
import pytest

from pixels_gb300 import config
from pixels_gb300.ir import Program
from pixels_gb300.shapes import (box, capsule, cylinder, ellipsoid, intersect, lathe, prism, rotateX, rotateY, rotateZ,
                                 roundBox, sphere, subtract, torus, union)

from test_gpu_edge_cases import run_both

STAGES = [lambda s, a, c: s, lambda s, a, c: rotateX(s, a, c), lambda s, a, c: rotateY(s, a, c),
          lambda s, a, c: rotateZ(s, a, c), lambda s, a, c: rotateZ(rotateY(rotateZ(s, 0.7 * a, c), a, c), 1.3 * a, c)]


def primitives(rng, c, h):
    """One of each primitive around c, of half extent about h."""
    e = tuple(float(v) for v in h * rng.uniform(0.3, 1.0, 3))
    d = rng.normal(size=3)
    d = d / np.linalg.norm(d) * h
    ys = np.sort(rng.uniform(-h, h, 7))
    prof = [float(v) for y in ys for v in (rng.uniform(0.2, 0.8) * h, y)]
    hexagon = [float(v) for k in range(6) for v in (h * np.cos(k * np.pi / 3 + rng.uniform(-0.3, 0.3)),
                                                   h * np.sin(k * np.pi / 3 + rng.uniform(-0.3, 0.3)))]
    star = [float(v) for k in range(10) for v in (h * (0.4 + 0.6 * (k % 2)) * np.cos(k * np.pi / 5),
                                                h * (0.4 + 0.6 * (k % 2)) * np.sin(k * np.pi / 5))]
    out = [box(c, e), roundBox(c, e, 0.3 * min(e)), sphere(c, h), ellipsoid(c, e),
           capsule(tuple(float(v) for v in c - d), tuple(float(v) for v in c + d), 0.3 * h),
           lathe(c, prof, 0), lathe(c, prof, 0.1 * h), prism(c, hexagon, c[1] - e[1], c[1] + e[1]),
           prism(c, star, c[1] - e[1], c[1] + e[1])]
    return out + [f(c, 0.7 * h, r, axis) for axis in "xyz" for f, r in ((cylinder, e[0]), (torus, 0.2 * h))]


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["one", "two"])
@pytest.mark.parametrize("stage", range(len(STAGES)))
def test_every_primitive_and_stage(built_lib, stage, form):
    vpm, dims = 40.0, (120, 88, 104)
    ext = np.array(dims) / vpm
    rng = np.random.default_rng(10 * stage + len(form))
    prog = Program()
    with config.using(vpm):
        for h in (0.08, 0.35, 1.1):
            for i in range(15):
                c = tuple(float(v) for v in rng.uniform(0.1, 0.9, 3) * ext)
                a = float(rng.uniform(-3, 3))
                s = STAGES[stage](primitives(rng, c, h)[i], a, c)
                if form == "two":
                    c2 = tuple(float(v) for v in np.array(c) + rng.uniform(-0.4, 0.4, 3) * h)
                    t = primitives(rng, c2, 0.8 * h)[int(rng.integers(15))]
                    comb = (subtract, intersect, union)[i % 3]
                    s = comb(s, STAGES[int(rng.integers(len(STAGES)))](t, a, c2))
                prog.add_op(int(rng.integers(2)) if i else 0, s, int(rng.integers(1, 60)))
    _, stats = run_both(prog, vpm, dims)
    assert stats[2]["rescued_voxel"] <= stats[2]["voxel_evals"] // 50


@pytest.mark.gpu
@pytest.mark.parametrize("radius", [0.5, 4.0, 12.0, 20.0, 60.0, 400.0])
def test_large_shapes_around_the_bound(built_lib, radius):
    vpm, dims = 160.0, (64, 48, 56)
    ext = np.array(dims) / vpm
    c = tuple(float(v) for v in ext / 2 + np.array([radius, 0.02, -0.03]))
    prog = Program()
    with config.using(vpm):
        prog.add_op(0, sphere(c, radius), 5)
        prog.add_op(1, rotateY(capsule(c, (c[0], c[1] + radius, c[2]), radius - 0.1), 0.01, c), 0)
        prog.add_op(0, rotateZ(roundBox(c, (radius - 0.15, radius, radius), 0.05), 0.004, c), 9)
    run_both(prog, vpm, dims)
