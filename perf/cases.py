"""The measured work of the voxeliser: what a program that embeds it has it do.

Every case goes through the C ABI (its ctypes binding ``pixels_gb300._lib``, or
``pixels_gb300.batch``), with the op lists, handles and buffers such a program
keeps, and returns the world's own device buffers: grid, pool, super-grid
counts, density and the GPU free list.  Every output is a whole number or a
byte, equal or wrong.

Kinds of case (``case["kind"]``):

* ``load``   a level is loaded: an op list in host memory is submitted to an
             empty world and built, derived upload buffers included.  Scenes:
             ``penthouse`` (the repository's scene, plus a saved game's damage
             of 64 seeded add / carve strokes) and ``synthetic`` (seeded
             primitives of every kind under rotations and CSG).
* ``graph``  the same scene rebuilt from ops that stay on the device, as a
             captured graph of one world (a program that rebuilds per frame).
* ``batch``  independent scenes of uneven size rebuilt by one graph launch.
* ``edit``   an incremental build on a resident map: sculpting strokes, each an
             added sphere or capsule that a carve then cuts, so that every pass
             changes voxels and moves bricks in and out of the pool.
* ``serve``  a play session: a level is loaded, then a burst of subtract-edits
             goes through the serving loop.
* ``derive`` super-grid counts and density of a grid and pool that the caller
             holds, into buffers it holds (no allocation).
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from pixels_gb300 import _lib, config
from pixels_gb300.batch import Batch
from pixels_gb300.ir import ADD, CARVE, Program
from pixels_gb300.materials import opaque_table, uniform_density_table, vox
from pixels_gb300.scenes.penthouse import penthouse_program
from pixels_gb300.scenes.synthetic import batch_specs, synthetic_program
from pixels_gb300.serving import carve_program, edit_stream
from pixels_gb300.shapes import capsule, sphere
from pixels_gb300.world import MODE_FP64, MODE_MIXED

MAX_BRICKS = 1 << 31      # device limit of the GPU free list: none
EDIT_LISTS = 8            # stroke lists an editing session cycles through
MODES = {"mixed": MODE_MIXED, "fp64": MODE_FP64}


def listed():
    return [
        # the smallest level load: the plain configuration's size, bound by launches and latency
        {"name": "load-penthouse-20", "kind": "load", "scene": "penthouse", "vpm": 20, "mode": "mixed"},
        # the headline scene and size, from a host op list
        {"name": "load-penthouse-80", "kind": "load", "scene": "penthouse", "vpm": 80, "mode": "mixed"},
        # the largest density the reference publishes a build time for
        {"name": "load-penthouse-128", "kind": "load", "scene": "penthouse", "vpm": 128, "mode": "mixed"},
        # the all-float64 form, a user's exact mirror of JavaScript numbers
        {"name": "load-penthouse-40-fp64", "kind": "load", "scene": "penthouse", "vpm": 40, "mode": "fp64"},
        # the headline figure: the scene's resident ops rebuilt as a graph
        {"name": "graph-penthouse-80", "kind": "graph", "scene": "penthouse", "vpm": 80, "mode": "mixed"},
        # scattered rotated primitives, CSG and procedural paint at the synthetic configuration's size
        {"name": "load-synthetic-4096", "kind": "load", "scene": "synthetic", "vpm": 80, "prims": 4096, "mode": "mixed"},
        # ... a smaller one in the float64 form
        {"name": "load-synthetic-512-fp64", "kind": "load", "scene": "synthetic", "vpm": 40, "prims": 512,
         "mode": "fp64"},
        # many uneven scenes in one graph launch (a slice of the batched configuration)
        {"name": "batch-12", "kind": "batch", "scenes": 12, "mode": "mixed"},
        # one brush stroke on a resident map at serving density: the smallest call
        {"name": "edit-1", "kind": "edit", "vpm": 160, "strokes": 1},
        # 256 strokes at once: a serving step at the target's concurrency
        {"name": "edit-256", "kind": "edit", "vpm": 160, "strokes": 256},
        # a burst of subtract-edits through the serving loop
        {"name": "serve-1024", "kind": "serve", "vpm": 80, "edits": 1024},
        # the derived buffers alone, for a renderer with fixed device memory
        {"name": "derive-80", "kind": "derive", "vpm": 80},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _vpm(rng, lo, hi):
    return round(math.exp(rng.uniform(math.log(lo), math.log(hi))), 1)  # any density, ragged world edges


def draw(rng):
    kind = rng.choice(["load", "load", "load", "load", "graph", "batch", "edit", "edit", "serve", "derive"])
    if kind == "load" and rng.random() < 0.5:
        mode = rng.choice(["mixed", "mixed", "fp64"])
        return {"kind": "load", "scene": "penthouse", "vpm": _vpm(rng, 16, 120 if mode == "mixed" else 40), "mode": mode}
    if kind == "load":
        mode = rng.choice(["mixed", "mixed", "fp64"])
        return {"kind": "load", "scene": "synthetic", "vpm": _vpm(rng, 20, 80 if mode == "mixed" else 40),
                "prims": _log(rng, 64, 4000 if mode == "mixed" else 512), "mode": mode}
    if kind == "graph":
        return {"kind": "graph", "scene": "penthouse", "vpm": _vpm(rng, 16, 80), "mode": "mixed"}
    if kind == "batch":
        return {"kind": "batch", "scenes": _log(rng, 2, 12), "mode": "mixed", "content": rng.randrange(1 << 16)}
    if kind == "edit":
        return {"kind": "edit", "vpm": _vpm(rng, 40, 160), "strokes": _log(rng, 1, 256)}
    if kind == "serve":
        return {"kind": "serve", "vpm": _vpm(rng, 20, 80), "edits": _log(rng, 64, 1024)}
    return {"kind": "derive", "vpm": _vpm(rng, 16, 128)}


# ---------------------------------------------------------------------------
# inputs


def _radius(rng):
    return math.exp(rng.uniform(math.log(0.01), math.log(0.4)))  # 1-40 cm, as the serving edits


def _stroke(prog: Program, rng, centre):
    """A sphere (70%) or capsule of a random material added at ``centre``, then bitten by a carve."""
    r = _radius(rng)
    c = tuple(float(v) for v in centre)
    d = rng.normal(size=3)
    d = d / max(float(np.linalg.norm(d)), 1e-9) * r
    material = vox(1 + int(rng.integers(60)), int(rng.integers(256)))
    if rng.random() < 0.7:
        prog.add_op(ADD, sphere(c, r), material)
    else:
        prog.add_op(ADD, capsule(c, tuple(float(v) for v in c + 1.5 * d), r), material)
    prog.add_op(CARVE, sphere(tuple(float(v) for v in c + 0.7 * d), 0.8 * r), 0)


def _volume(vpm):
    return [n / vpm for n in config.Config(vpm).dims]


def _scene(case, seed) -> bytes:
    """The op list of a level, as the bytes the C ABI takes."""
    vpm = float(case["vpm"])
    if case.get("scene") == "synthetic":
        return synthetic_program(seed, case["prims"], vpm).to_bytes()
    prog, _ = penthouse_program(vpm)
    rng = np.random.default_rng(seed)
    vol = _volume(vpm)
    with config.using(vpm):
        for _ in range(64):
            _stroke(prog, rng, [rng.uniform(0, v) for v in vol])
    return prog.to_bytes()


class _Handle:
    """A world handle, as ``Batch`` takes a built world; destroyed with its last user."""

    def __init__(self, dims, vpm, capacity):
        self._h = _lib.world_create(*dims, float(vpm), capacity)

    def _ensure(self):
        pass

    def __del__(self):
        _lib.world_destroy(self._h)


class _View:
    """A device array of a world for torch, without a copy; keeps the world's handle alive."""

    def __init__(self, owner, ptr, n, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (int(ptr), False), "shape": (int(n),), "typestr": typestr, "version": 2}


class _World:
    """A world and torch views of its buffers (as signed integers of the same width)."""

    def __init__(self, dims, vpm, mode, derive, ir, capacity):
        self.cells = dims[0] * dims[1] * dims[2] // 512
        self.supers = math.prod((d // 8 + 3) // 4 for d in dims)
        self.capacity = min(int(capacity), 2 * self.cells + 4096)  # pool bricks, for the scene and for play
        self.handle = _Handle(dims, vpm, self.capacity)
        self.h = self.handle._h
        self.derive = derive
        self.seen = None
        if derive:
            _lib.set_derive_on_build(self.h, MAX_BRICKS)
        # the first build sizes every buffer; pool and free list then start as zeros, so that
        # the bytes no build has written are the same in every program
        _lib.submit_ops(self.h, ir)
        _lib.build(self.h, mode)
        for t in (self.views()[1], *self.views()[4:]):
            t.zero_()
        torch.cuda.synchronize()
        _lib.world_reset(self.h, True)
        _lib.build(self.h, mode)
        self.views()

    def _tensor(self, ptr, n, typestr):
        return torch.as_tensor(_View(self.handle, ptr, n, typestr), device="cuda")

    def views(self):
        """The world's buffers, whole: pool and free list to their capacity."""
        v = _lib.device_view(self.h)
        at = (v.grid, v.pool, v.super_counts, v.density, v.free_list)
        if at != self.seen:
            if _lib.stats(self.h)["pool_capacity"] != self.capacity:
                raise RuntimeError("the pool grew: the case's capacity is too small")
            self.seen = at
            self.out = [self._tensor(v.grid, self.cells, "<i4"), self._tensor(v.pool, self.capacity * 512, "<i2")]
            if self.derive:
                self.out += [self._tensor(v.super_counts, self.supers, "<i4"), self._tensor(v.density, self.cells, "|u1"),
                             self._tensor(v.free_list, max(self.capacity + 98304, 2 * self.capacity), "<i4")]
        return self.out

    def holes(self):
        n = _lib.stats(self.h)["n_holes"]
        return self._tensor(_lib.device_view(self.h).holes, n, "<i4") if n else None


class _Batch:
    def __init__(self, worlds, mode):
        self.worlds = worlds
        self.batch = Batch([w.handle for w in worlds], mode)

    def __del__(self):
        self.batch.close()  # before its worlds' handles go


def _occupied(world, vpm, rng, n):
    """Points in occupied bricks of the built map, uniform over them."""
    bx, by, _ = config.Config(vpm).bricks
    occ = torch.nonzero(world.out[0]).flatten()
    ci = occ[torch.from_numpy(rng.integers(len(occ), size=n)).to(occ.device)].cpu().numpy()
    b = np.stack([ci % bx, (ci // bx) % by, ci // (bx * by)], axis=1)
    return (b * 8 + rng.uniform(0, 8, size=(n, 3))) / vpm


def _capacity(case):
    """Pool bricks of a world: what its scene fills, what a build reserves beside it, and room for play."""
    v2 = float(case["vpm"]) ** 2
    if case["kind"] == "edit":
        return 8192 + 2 * v2 + 4096 * v2 / 25
    if case.get("scene") == "synthetic":
        return 8192 + 2 * v2 + case["prims"] * v2 / 50
    return 8192 + 45 * v2 + (131072 if case["kind"] == "serve" else 0)


def _map(vpm):
    """The op list of the resident map: the synthetic configuration's scene."""
    return synthetic_program(1, 4096, float(vpm)).to_bytes()


def prepare(case, seed):
    kind = case["kind"]
    mode = MODES[case.get("mode", "mixed")]
    state = {"kind": kind, "mode": mode}
    if kind == "batch":
        # sizes are the batched configuration's, the scenes' content the seed's
        worlds = []
        for i, s in enumerate(batch_specs(n=case["scenes"])):
            prog = synthetic_program((seed * 131 + case.get("content", 0)) * 1009 + i, s["n_prims"], s["vpm"], s["volume"])
            worlds.append(_World(s["dims"], s["vpm"], mode, True, prog.to_bytes(), 1 << 30))
        state["batch"] = _Batch(worlds, mode)
        return state
    vpm = float(case["vpm"])
    cfg = config.Config(vpm)
    if kind in ("load", "graph"):
        ir = _scene(case, seed)
        world = _World(cfg.dims, vpm, mode, True, ir, _capacity(case))
        state.update(world=world, ir=ir)
        if kind == "graph":
            state["batch"] = _Batch([world], mode)
    elif kind == "edit":
        world = _World(cfg.dims, vpm, mode, False, _map(vpm), _capacity(case))
        rng = np.random.default_rng(seed)
        lists = []
        with config.using(vpm):
            for _ in range(EDIT_LISTS):
                prog = Program()
                for c in _occupied(world, vpm, rng, case["strokes"]):
                    _stroke(prog, rng, c)
                lists.append(prog.to_bytes())
        state.update(world=world, lists=lists, next=0)
    elif kind == "serve":
        ir = _scene(case, 0)
        world = _World(cfg.dims, vpm, mode, False, ir, _capacity(case))
        n = case["edits"]
        edits, _ = edit_stream(world.out[0].cpu().numpy(), cfg.bricks, vpm, n, rate=0, seed=seed)
        arr = (_lib.Edit * n)()
        for e, (shape, a, b, r) in zip(arr, edits):
            e.shape, e.r = int(shape), float(r)
            e.a[:], e.b[:] = [float(v) for v in a], [float(v) for v in b]
        # the burst as one plain build first: it sizes the staging area, which a serving step cannot grow
        _lib.submit_ops(world.h, carve_program(edits, range(n), vpm).to_bytes())
        _lib.build(world.h, mode)
        state.update(world=world, ir=ir, n=n, edits=arr, arrivals=(ctypes.c_double * n)(), results=(_lib.EditResult * n)(),
                     order=np.zeros(n, np.int64))
    else:  # derive
        world = _World(cfg.dims, vpm, mode, False, _scene(case, seed), _capacity(case))
        grid, pool = world.views()
        grid, pool = grid.clone(), pool[: _lib.stats(world.h)["pool_used"] * 512].clone()
        n_super = math.prod((b + 3) // 4 for b in cfg.bricks)
        state.update(grid=grid, pool=pool, bricks=cfg.bricks, opaque=np.array(opaque_table(), np.uint8),
                     udens=np.array(uniform_density_table(), np.uint8),
                     super=torch.zeros(n_super, dtype=torch.int32, device="cuda"),
                     density=torch.zeros(grid.numel(), dtype=torch.uint8, device="cuda"))
    return state


# ---------------------------------------------------------------------------
# one pass


def run(state):
    kind = state["kind"]
    if kind == "load":
        h = state["world"].h
        _lib.world_reset(h)
        _lib.submit_ops(h, state["ir"])
        _lib.build(h, state["mode"])
        return state["world"].views()
    if kind in ("graph", "batch"):
        b = state["batch"]
        b.batch.run()
        return [w.views() for w in b.worlds]
    if kind == "edit":
        h, lists = state["world"].h, state["lists"]
        _lib.submit_ops(h, lists[state["next"]])
        state["next"] = (state["next"] + 1) % len(lists)
        _lib.build(h, state["mode"])
        return state["world"].views()
    if kind == "serve":
        w, n_app = state["world"], ctypes.c_size_t()
        _lib.world_reset(w.h)
        _lib.submit_ops(w.h, state["ir"])
        _lib.build(w.h, state["mode"])
        rc = _lib.load().px_serve_run(
            w.h, state["edits"], state["arrivals"], state["n"], 256, 1 << 40, state["mode"], None, state["results"],
            state["order"].ctypes.data_as(ctypes.POINTER(ctypes.c_uint64)), ctypes.byref(n_app))
        if rc != _lib.PX_OK:
            raise _lib.PxError(rc, _lib.load().px_last_error(w.h).decode())
        grid, pool = w.views()
        holes = w.holes()
        if holes is not None:  # freed bricks, whose bytes depend on how the burst fell into steps
            pool.view(-1, 512).index_fill_(0, holes.long(), 0)
        return [grid, pool, state["order"][: n_app.value]]
    s = state
    rc = _lib.load().px_derive_noalloc(
        ctypes.c_void_p(s["grid"].data_ptr()), ctypes.c_void_p(s["pool"].data_ptr()), *s["bricks"],
        s["pool"].numel() // 512, s["opaque"].ctypes.data, s["udens"].ctypes.data,
        ctypes.c_void_p(s["super"].data_ptr()), ctypes.c_void_p(s["density"].data_ptr()), None)
    if rc != _lib.PX_OK:
        raise _lib.PxError(rc, "px_derive_noalloc")
    return [s["super"], s["density"]]


# ---------------------------------------------------------------------------
# what a pass cannot do without

FLOPS_PER_EVALUATION = 30  # adds, multiplies, min / max, compares and roots of one signed distance


def _evaluations(st):
    return FLOPS_PER_EVALUATION * (st["brick_evals"] + st["sub_evals"] + st["voxel_evals"])


def work(case):
    """Bytes: the op list in, every live pool brick, grid entry and derived byte out (edits: the
    bricks they cut read and written).  Flops: the distance evaluations the reference's procedure
    prescribes (whole bricks, sub-blocks, boundary voxels), counted by a build of the case."""
    state = prepare(case, 0)
    kind = case["kind"]
    if kind == "derive":
        return {"bytes": sum(state[k].numel() * state[k].element_size() for k in ("grid", "pool", "super", "density")),
                "flops": state["pool"].numel()}
    run(state)
    torch.cuda.synchronize()

    def written(w):  # live pool bricks, grid, super counts, density and the free list (98,304 bricks of room)
        st = _lib.stats(w.h)
        return 1024 * (st["pool_used"] - st["n_holes"]) + 4 * w.cells + (4 * w.supers + w.cells + 4 * 98304) * w.derive

    if kind in ("graph", "batch"):
        worlds = state["batch"].worlds
        return {"bytes": sum(map(written, worlds)), "flops": sum(_evaluations(_lib.stats(w.h)) for w in worlds)}
    st = _lib.stats(state["world"].h)
    if kind == "load":
        return {"bytes": len(state["ir"]) + written(state["world"]), "flops": _evaluations(st)}
    if kind == "edit":  # a partial pair is a brick with 8 sub-block evaluations
        return {"bytes": len(state["lists"][0]) + 2 * 1024 * st["sub_evals"] // 8, "flops": _evaluations(st)}
    return {"bytes": 80 * state["n"] + written(state["world"]), "flops": 2 * _evaluations(st)}
