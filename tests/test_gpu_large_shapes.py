"""Lean programs of any size: which path they take, what they build, what they cost.

A one- or two-primitive program takes the lean voxel kernels while the error bound of its
float32 points is below 1/128 voxel, a kernel that evaluates the undecided voxels in line up
to half a voxel, and the interpreter beyond.  The bound grows with the shape, so radii from
one to thousands of metres cross both lines; every primitive, rotated, composed and
combined, must equal the oracle on all of them.
"""
import statistics

import numpy as np
import pytest

from pixels_gb300 import _lib, config
from pixels_gb300.ir import Program
from pixels_gb300.shapes import (Shape, box, capsule, cylinder, ellipsoid, intersect, lathe, prism, rotateX, rotateZ, roundBox,
                                 sphere, subtract, torus, union)
from pixels_gb300.world import MODE_MIXED, VoxelWorld

from test_gpu_edge_cases import run_both

VPM = 160.0


def shapes(ext, R):
    """One of each primitive whose surface crosses the world, of size R; then rotated ones and pairs."""
    x, y, z = (float(v) for v in ext / 2)
    c = (x, y - R, z)
    ring = [float(v) for k in range(12) for v in (R * np.cos(k * np.pi / 6), R * np.sin(k * np.pi / 6))]
    prof = [0.0, -R, 0.7 * R, -0.6 * R, R, 0.0, 0.6 * R, 0.5 * R, 0.0, R]
    one = [sphere(c, R), box((x - R, y - R, z), (R, R, R)), roundBox(c, (R, R, R), 0.1 * R), ellipsoid(c, (R, R, 0.8 * R)),
           cylinder((x - R, y, z), R, 0.2 * y, "y"), cylinder(c, R, 0.2, "x"), capsule((x, y - 2 * R, z), c, R),
           torus((x, y - 1.5 * R, z), R, 0.5 * R, "x"), lathe((x - R, y, z), prof, 0), lathe((x - R, y, z), prof, 0.05),
           prism((x - R * np.cos(np.pi / 12), 0.0, z), ring, 0.3 * y, y)]
    rot = [rotateX(one[6], 0.01, (x, y, z)), rotateZ(one[1], 0.02, (x, y, z)),
           rotateZ(rotateX(one[2], 0.01, (x, y, z)), 0.02, (x, y, z)), rotateX(one[10], 0.01, (x, y, z))]
    two = [subtract(one[0], sphere((x, y - R - 0.05, z), R)), intersect(rot[0], one[4]), union(rot[1], rot[3])]
    return one + rot + two


def scene(ext, shapes_):
    prog = Program()
    with config.using(VPM):
        for k, s in enumerate(shapes_(ext)):
            prog.add_op(1 if k % 5 == 3 else 0, s, k + 1)
    return prog


@pytest.mark.gpu
@pytest.mark.parametrize("radius", [1.0, 8.0, 25.0, 90.0, 300.0, 900.0])
def test_every_primitive_of_any_size(built_lib, radius):
    dims = (64, 56, 72)
    ext = np.array(dims) / VPM

    def all_(e):
        with config.using(VPM):
            return shapes(e, radius)
    run_both(scene(ext, all_), VPM, dims)


def timed(ops, dims):
    w = VoxelWorld(*dims, vpm=VPM, mode=MODE_MIXED)
    prog = Program()
    with config.using(VPM):
        for s in ops:
            prog.add_op(0, s, 5)
    w._pending = prog
    w.build()
    launches = w.stats()["kernel_launches"]
    ms = []
    for _ in range(7):
        _lib.world_reset(w._h, True)
        _lib.build(w._h, MODE_MIXED)
        ms.append(w.stats()["build_ms"])
    w.close()
    return launches, statistics.median(ms)


@pytest.mark.gpu
def test_which_kernels_run(built_lib):
    """Each voxel kernel is launched where a program asks for it: small, large and very large shapes
    together take one launch more for each further kind."""
    small, large, vast = (sphere((0.2, 0.2 - r + 0.1, 0.2), r) for r in (0.1, 300.0, 5000.0))
    n = {k: timed(s, (64, 64, 64))[0] for k, s in (("small", [small]), ("large", [large]), ("vast", [vast]),
                                                   ("two", [small, large]), ("all", [vast, small, large]))}
    assert n["small"] == n["large"] == n["vast"] == n["two"] - 1 == n["all"] - 2, n
    # ten metres at this density are still the lean kernels'
    assert timed([small, sphere((0.2, 0.2 - 10.0, 0.2), 10.0)], (64, 64, 64))[0] == n["small"]


@pytest.mark.gpu
def test_points_decide_large_prisms(built_lib):
    """A 12-sided prism of 30 m, past the lean kernels' bound, against the same prism under two
    offsets of 0 (no lean program: the interpreter's): its points decide nearly all voxels."""
    dims, R = (1024, 256, 1024), 30.0
    x, y, z = (float(v) / 2 / VPM for v in dims)
    with config.using(VPM):
        p = prism((x, 0.0, z - R + z / 2), [float(v) for k in range(12) for v in (R * np.cos(k * np.pi / 6),
                                                                                  R * np.sin(k * np.pi / 6))], y / 2, y)
        q = Shape(("offset", ("offset", p.node, 0.0), 0.0), p.min, p.max)
        alone, interpreted = timed([p], dims)[1], timed([q], dims)[1]
    assert interpreted > 1.2 * alone, (alone, interpreted)
