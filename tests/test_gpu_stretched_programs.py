"""Op lists whose programs stretch distances, against the float64 oracle in both forms.

The C ABI takes any parameters: rotations whose cos and sin are not a unit vector,
ellipsoids and capsules whose derived constants do not fit the rest.  The reference's
closures would evaluate them at every boundary voxel; a voxel decided from its
sub-block's centre must be decided with the program's own Lipschitz constant.  Factors
below and above 1, around the largest constant that decision covers (16), nested, and in
every combination with a primitive: whole numbers, equal to the oracle's or wrong.
"""
import numpy as np
import pytest

from pixels_gb300 import config
from pixels_gb300.ir import OP_CAPSULE, OP_ELLIPSOID, OP_ROT_X, OP_ROT_Z, Program
from pixels_gb300.shapes import (box, capsule, cylinder, ellipsoid, intersect, prism, rotateX, rotateY, rotateZ, roundBox,
                                 sphere, subtract, torus, union)

from test_gpu_edge_cases import run_both

VPM, DIMS = 40.0, (96, 72, 88)


def stretch(prog, rot=1.0, ell=1.0, cap=1.0):
    """Scale every rotation's cos and sin, every ellipsoid's factor, every capsule's |e|^2."""
    for w0, off in prog.code:
        op = w0 & 0xFF
        if OP_ROT_X <= op <= OP_ROT_Z:
            prog.params[off + 2] *= rot
            prog.params[off + 3] *= rot
        elif op == OP_ELLIPSOID:
            prog.params[off + 6] *= ell
        elif op == OP_CAPSULE:
            prog.params[off + 6] *= cap
    return prog


def shapes(rng, n):
    ext = np.array(DIMS) / VPM
    for k in range(n):
        c = tuple(float(v) for v in rng.uniform(0.25, 0.75, 3) * ext)
        h = float(rng.uniform(0.2, 0.6))
        e = tuple(float(v) for v in h * rng.uniform(0.3, 1.0, 3))
        d = rng.normal(size=3)
        d = d / np.linalg.norm(d) * h
        hexagon = [float(v) for j in range(6) for v in (h * np.cos(j * np.pi / 3), h * np.sin(j * np.pi / 3))]
        yield c, float(rng.uniform(-3, 3)), (
            sphere(c, h), box(c, e), roundBox(c, e, 0.2 * min(e)), ellipsoid(c, e), cylinder(c, h, e[0], "xyz"[k % 3]),
            capsule(tuple(float(v) for v in c - d), tuple(float(v) for v in c + d), 0.3 * h),
            torus(c, 0.7 * h, 0.2 * h, "xyz"[k % 3]), prism(c, hexagon, c[1] - e[1], c[1] + e[1]))


@pytest.mark.gpu
@pytest.mark.parametrize("rot", [0.3, 0.999, 1.001, 1.3, 2.0, 4.0, 15.9, 16.1, 1000.0])
def test_rotations_that_scale(built_lib, rot):
    rng = np.random.default_rng(int(rot * 10))
    prog = Program()
    with config.using(VPM):
        for k, (c, a, prims) in enumerate(shapes(rng, 10)):
            s = (rotateX, rotateY, rotateZ)[k % 3](prims[int(rng.integers(8))], a, c)
            if k % 4 == 3:
                s = (subtract, intersect, union)[k % 3](s, prims[int(rng.integers(8))])
            prog.add_op(1 if k % 5 == 4 else 0, s, k + 1)
    run_both(stretch(prog, rot=rot), VPM, DIMS)


@pytest.mark.gpu
@pytest.mark.parametrize("rot", [1.2, 2.5, 2.6, 40.0])
def test_nested_rotations_that_scale(built_lib, rot):
    rng = np.random.default_rng(int(rot * 10) + 1)
    prog = Program()
    with config.using(VPM):
        for k, (c, a, prims) in enumerate(shapes(rng, 6)):
            s = rotateZ(rotateY(rotateX(prims[k], a, c), 0.7 * a, c), 1.3 * a, c)
            prog.add_op(0, s if k % 2 else rotateY(union(s, prims[6]), a, c), k + 1)
    run_both(stretch(prog, rot=rot), VPM, DIMS)


@pytest.mark.gpu
@pytest.mark.parametrize("ell,cap", [(0.5, 0.5), (1.5, 0.4), (2.0, 0.1), (5.0, 3.0), (15.0, 0.06), (17.0, 0.05), (200.0, -0.5)])
def test_constants_that_do_not_fit(built_lib, ell, cap):
    rng = np.random.default_rng(7)
    prog = Program()
    with config.using(VPM):
        for k, (c, a, prims) in enumerate(shapes(rng, 8)):
            s = prims[3] if k % 2 else prims[5]
            prog.add_op(0 if k % 4 else 1, rotateY(s, a, c) if k % 3 else s, k + 1) if k else prog.add_op(0, s, 1)
    run_both(stretch(prog, ell=ell, cap=cap), VPM, DIMS)
