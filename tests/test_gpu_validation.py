"""Validation mode counts no violation, in either form.

Both forms settle voxels from their sub-block's centre, and the mixed form decides bricks,
sub-blocks and voxels from float32 points; with validation on, one kernel more compares
all of these with the float64 values.  Whole scenes, every primitive and stage, shapes
on both sides of each bound of the points, and programs that stretch distances.
"""
import numpy as np
import pytest

from pixels_gb300 import _lib, config
from pixels_gb300.ir import Program
from pixels_gb300.scenes.penthouse import penthouse_program
from pixels_gb300.scenes.synthetic import synthetic_program
from pixels_gb300.world import MODE_FP64, MODE_MIXED, VoxelWorld

import pyoracle
import test_gpu_large_shapes as large
import test_gpu_lean_points as points
import test_gpu_stretched_programs as stretched


def every_primitive(vpm, dims):
    rng = np.random.default_rng(3)
    ext = np.array(dims) / vpm
    prog = Program()
    with config.using(vpm):
        for k, stage in enumerate(points.STAGES):
            for i in range(15):
                c = tuple(float(v) for v in rng.uniform(0.15, 0.85, 3) * ext)
                prog.add_op(int(i % 5 == 4), stage(points.primitives(rng, c, (0.1, 0.3, 0.6)[i % 3])[i], float(rng.uniform(-3, 3)), c), i + k + 1)
    return prog


def of_size(vpm, dims, radius):
    with config.using(vpm):
        shapes = large.shapes(np.array(dims) / vpm, radius)
    return large.scene(None, lambda _: shapes)


def stretching(vpm, dims, rot):
    prog = Program()
    with config.using(vpm):
        for k, (c, a, prims) in enumerate(stretched.shapes(np.random.default_rng(5), 8)):
            prog.add_op(0, (stretched.rotateX, stretched.rotateY, stretched.rotateZ)[k % 3](prims[k], a, c), k + 1)
    return stretched.stretch(prog, rot=rot)


SCENES = {
    "penthouse": (20.0, config.Config(20.0).dims, lambda v, d: penthouse_program(v)[0]),
    "synthetic": (40.0, config.Config(40.0).dims, lambda v, d: synthetic_program(4, 200, v)),
    "primitives": (40.0, (96, 88, 104), every_primitive),
    "large 25": (160.0, (64, 56, 72), lambda v, d: of_size(v, d, 25.0)),
    "large 300": (160.0, (64, 56, 72), lambda v, d: of_size(v, d, 300.0)),
    "stretched 1.3": (stretched.VPM, stretched.DIMS, lambda v, d: stretching(v, d, 1.3)),
    "stretched 15": (stretched.VPM, stretched.DIMS, lambda v, d: stretching(v, d, 15.0)),
}


@pytest.mark.gpu
@pytest.mark.parametrize("mode", [MODE_FP64, MODE_MIXED])
@pytest.mark.parametrize("name", SCENES)
def test_no_violations(built_lib, name, mode):
    vpm, dims, make = SCENES[name]
    prog = make(vpm, dims)
    o = pyoracle.OracleWorld(prog.to_bytes(), vpm, dims, threads=8)
    launches = []
    for validate in (False, True):
        w = VoxelWorld(*dims, vpm=vpm, mode=mode)
        _lib.set_validation(w._h, validate)
        _lib.submit_ops(w._h, prog.to_bytes())
        w.build()
        st = w.stats()
        launches.append(st["kernel_launches"])
        np.testing.assert_array_equal(w.grid, o.grid)
        assert st["violations"] == 0
        w.close()
    assert launches[1] == launches[0] + 1  # the comparison ran
