"""The liquid step's performance cases: what programs ask of this framework,
from a toy pond to a batch of worlds, each through the public entry points
(fluid.LiquidStep, fluid.Batch, serve.GpuBackend, the allocation-free norm).

A case's state is a world (or several) on the device as a program holds it;
one pass is one step of it, launched as a frame loop launches it: with that
frame's Params, asynchronously, with no read-back.  Successive passes step
the world on.

A pass returns the world's buffers, where they live: the cells, the field's
records of the cells and faces (pressure, divergence, density, drift, face
velocities), the counters' words (the sort's counts and starts among them),
the particle count, a free body's words.  Not returned: the relaxation's
rim words and the coarse levels, which a step keeps to itself, and the
particles' records, whose order within a cell is an atomic's and differs
from run to run; the next pass splats every particle into the counters by
sums that do not depend on the order, so it shows them all.
"""
import ctypes

import numpy as np
import torch

from worldinagrain_b200 import abi, fluid, serve
from worldinagrain_b200 import world as W

# The 1e-6 solve with FP64 dot products that the benchmark times; the same
# with 16-bit coarse levels; the reference's own stopping rule and iteration
# cap, which a host that just replaces encodeFluid gets.
RULES = {
    "tight": (abi.STEP_TOLERANCE | abi.STEP_F64_DOTS, 64),
    "mixed": (abi.STEP_TOLERANCE | abi.STEP_F64_DOTS | abi.STEP_MIXED, 64),
    "reference": (0, abi.FLUID_CYCLES),
}
TOLERANCE = 1e-6


def listed():
    return [
        # an interactive toy: a pond of a few thousand cells in a page, the
        # drop-in call of a host that sets nothing; ragged sides
        {"name": "toy_75x52", "kind": "pond", "w": 75, "h": 52, "rule": "reference"},
        # the plain dam break, the smallest configuration of the benchmark
        {"name": "dam_256", "kind": "dam", "w": 256, "h": 256, "rule": "tight"},
        # two liquids, one viscous, with the viscosity sweeps; ragged sides
        {"name": "two_liquids_375x283", "kind": "liquids", "w": 375, "h": 283, "rule": "tight"},
        # free bodies coupled into the solve: a tank with floating, sunk,
        # held and new bodies
        {"name": "bodies_256", "kind": "bodies", "w": 256, "h": 256, "rule": "tight"},
        # a world whose liquid is at rest or absent: the host's bookkeeping step
        {"name": "dry_512", "kind": "dry", "w": 512, "h": 512, "rule": "reference"},
        # a host under its own allocator or capture, asking how far a solve got
        {"name": "norm_1024", "kind": "norm", "w": 1024, "h": 1024, "rule": "tight"},
        # the benchmark's single world, FP32 and mixed
        {"name": "disks_1024", "kind": "disks", "w": 1024, "h": 1024, "rule": "tight"},
        {"name": "disks_1024_mixed", "kind": "disks", "w": 1024, "h": 1024, "rule": "mixed"},
        # the largest single world: the obstacle column at 2 particles a cell
        {"name": "column_2048", "kind": "column", "w": 2048, "h": 2048, "rule": "tight"},
        # many worlds stepped as one: the multi-world set's sizes, FP32 and mixed
        {"name": "batch_48", "kind": "batch", "worlds": 48, "lo": 64, "hi": 512, "rule": "tight"},
        {"name": "batch_48_mixed", "kind": "batch", "worlds": 48, "lo": 64, "hi": 512, "rule": "mixed"},
        # a serving lane's step of small worlds, their scratch lent by the lane's pool
        {"name": "served_24", "kind": "served", "worlds": 24, "lo": 64, "hi": 256, "rule": "tight"},
    ]


def draw(rng):
    def side(lo, hi):
        return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))

    kind = rng.choice(["pond", "dam", "disks", "disks", "column", "liquids", "bodies", "dry", "norm", "batch", "batch",
                       "served"])
    rule = rng.choice(["tight", "tight", "mixed", "reference"])
    if kind in ("batch", "served"):
        lo = side(64, 128)
        return {"kind": kind, "worlds": side(4, 48), "lo": lo, "hi": side(2 * lo, 512 if kind == "batch" else 256),
                "rule": rule}
    lo, hi = {"pond": (40, 200), "dam": (64, 1024), "disks": (200, 1280), "column": (128, 1536), "liquids": (96, 640),
              "bodies": (96, 448), "dry": (64, 1536), "norm": (64, 1000)}[kind]
    w = side(lo, hi)
    h = max(lo, min(hi, int(w * rng.uniform(0.6, 1.6))))
    if kind == "bodies" and rule == "mixed":
        rule = "reference"  # a world with bodies is solved in FP32
    return {"kind": kind, "w": w, "h": h, "rule": rule}


# ---------------------------------------------------------------- worlds

def _world(case, seed):
    kind, w, h = case["kind"], case["w"], case["h"]
    if kind == "pond":
        return W.small_world(w, h, seed=seed, kind="obstacles")
    if kind == "dam":
        return W.dam_break(w, h, seed=seed)
    if kind == "disks":
        # as many disks to the area as the benchmark's world has
        return W.disks_world(w, h, n_disks=max(4, int(200 * w * h / 2 ** 20)), seed=seed)
    if kind == "column":
        return W.obstacle_column(w, h, seed=seed)
    if kind == "liquids":
        return W.two_liquids(w, h, seed=seed)
    if kind == "dry":
        rng = np.random.default_rng(seed)
        world = W.World(w, h)
        world.paint(rng.random((h, w)) < 0.2, abi.WALL)
        world.paint(rng.random((h, w)) < 0.1, abi.SAND)
        world.config = dict(earth_g=W.earth_g_cells())
        return world
    raise ValueError(kind)


class _Memory:
    """Device memory of `owner` as torch can wrap it (the tensor keeps this
    object, and so the owner, alive)."""

    def __init__(self, owner, ptr, n, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": typestr, "data": (ptr, False), "version": 2}


def _view(owner, ptr, n, typestr):
    return torch.as_tensor(_Memory(owner, ptr, n, typestr), device="cuda")


def _outputs(owner, world, b):
    """The buffers of one world a program reads after a step, in place."""
    C, F = world.C, world.L["face_count"]
    counters = _view(owner, b.counters, 11 * C + 2 * F, "<i4")
    return {
        "cells": _view(owner, b.cells, world.L["cells_bytes"] // 4, "<i4"),
        "field": _view(owner, b.field, 4 * (2 * C + F), "<f4"),
        "counts": counters[:11 * C].view(C, 11)[:, :9],
        "faces": counters[11 * C:],
        "particles": _view(owner, b.sorted, 1, "<i4"),
    }


class _Single:
    """A world on its own handle."""

    def __init__(self, case, seed):
        self.seed, self.frame = seed, 0
        self.flags, self.cycles = RULES[case["rule"]]
        self.bodies = None
        elems = W.element_table()
        if case["kind"] == "bodies":
            self.world, bodies = W.bodies_world(case["w"], case["h"], seed=seed, stamps=False)
            elems = W.body_element_table()
        else:
            self.world = _world(case, seed)
        if case["kind"] == "liquids":
            self.flags |= abi.STEP_VISCOUS
        if case["kind"] == "dry":
            self.flags |= abi.STEP_BOOKKEEPING_ONLY
        self.step = fluid.LiquidStep(self.world, elems)
        b = self.step.buffers()
        self.out = _outputs(self.step, self.world, b)
        if case["kind"] == "dry":
            blocks = _view(self.step, b.blocks, self.world.L["blocks_bytes"] // 4, "<i4")
            self.out = {"cells": self.out["cells"], "blocks": blocks[:2 * self.world.L["block_count"]]}
        if case["kind"] == "bodies":
            self.bodies = [torch.from_numpy(a.view(np.int32).copy()).cuda()
                           for a in (bodies.motion, bodies.pushes, bodies.stamps)]
            fluid.check(fluid.lib().wig_fluid_bind_bodies(self.step.h, *(ctypes.c_void_p(t.data_ptr()) for t in self.bodies)),
                        "wig_fluid_bind_bodies")
            self.out["motion"] = self.bodies[0]
        # the world's host copy is not needed any more
        for name in abi.BUFFER_NAMES:
            setattr(self.world, name, None)

    def run(self):
        self.frame += 1
        P = W.make_params(self.world, self.frame, self.seed, self.world.config["earth_g"])
        self.step.step(P, max_cycles=self.cycles, flags=self.flags, tolerance=TOLERANCE)
        return self.out


def _set(case, seed):
    """The multi-world configuration's worlds of these sides (its own sizes and
    fills, whatever the seed), their liquid moving."""
    worlds = W.multi_worlds(case["worlds"], case["lo"], case["hi"])
    rng = np.random.default_rng(seed)
    for w in worlds:
        cells = w.cell_view()
        water = cells[:, :, 0] == abi.WATER
        vel = rng.normal(0.0, 0.2, (int(water.sum()), 2)).astype(np.float32)
        cells[water, 2] = W.f16x2(vel[:, 0], vel[:, 1])
    return worlds


class _Many:
    """Worlds in one batch."""

    def __init__(self, case, seed):
        self.seed, self.frame = seed, 0
        self.flags, self.cycles = RULES[case["rule"]]
        self.worlds = _set(case, seed)
        self.ids = (ctypes.c_uint32 * len(self.worlds))(*range(len(self.worlds)))
        self.batch = fluid.Batch(self.worlds, W.element_table())
        self.out = [_outputs(self.batch, w, self.batch.buffers(k)) for k, w in enumerate(self.worlds)]
        for w in self.worlds:
            for name in abi.BUFFER_NAMES:
                setattr(w, name, None)

    def run(self):
        self.frame += 1
        P = (abi.Params * len(self.worlds))(*[W.make_params(w, self.frame, self.seed, w.config["earth_g"])
                                              for w in self.worlds])
        self.batch.step(self.ids, P, max_cycles=self.cycles, flags=self.flags, tolerance=TOLERANCE)
        return _joined(self.out)


class _Backend(serve.GpuBackend):
    """A serving backend closed with its last user."""

    def __del__(self):
        try:
            self.close()
        except Exception:
            pass


class _Served:
    """Worlds resident in a serving backend with lane pools, stepped on lane 0."""

    def __init__(self, case, seed):
        flags, cycles = RULES[case["rule"]]
        self.worlds = _set(case, seed)
        pool = sum(fluid.world_bytes(w.W, w.H, 4, w.cap) for w in self.worlds)  # room for all of them in one step
        self.backend = _Backend(self.worlds, W.element_table(), flags, cycles, TOLERANCE, pool_bytes=pool,
                                seed=seed)
        self.ids = list(range(len(self.worlds)))
        for k in self.ids:
            self.backend.admit(k)
        self.out = []
        for k, w in enumerate(self.worlds):
            b = abi.Buffers()
            fluid.check(fluid.lib().wig_batch_buffers_of(self.backend.h, k, ctypes.byref(b)), "wig_batch_buffers_of")
            self.out.append(_outputs(self.backend, w, b))

    def run(self):
        self.backend.launch(0, self.ids)
        return _joined(self.out)


def _joined(worlds):
    """The worlds' buffers by name, as many as a pass may return (64): every
    world's field, then the cells, counters and counts of the first ones."""
    names = [(name, k) for name in ("field", "cells", "counts", "faces", "particles") for k in range(len(worlds))]
    return {"%s_%d" % (name, k): worlds[k][name] for name, k in names[:64]}


class _Norm:
    """A host's own field, blocks and cg buffers after a solve: the residual
    norm read without an allocation."""

    def __init__(self, case, seed):
        self.desc = abi.WorldDesc(case["w"], case["h"], 4, 0)
        field, blocks, cg = _solved(case, seed)
        self.bufs = [torch.from_numpy(a).cuda() for a in (field, blocks, cg)]
        self.out = torch.zeros(1, dtype=torch.float64, device="cuda")
        self.fn = fluid.lib().wig_fluid_residual_norm2_noalloc
        self.fn.argtypes = [ctypes.POINTER(abi.WorldDesc)] + [ctypes.c_void_p] * 5
        self.fn.restype = ctypes.c_int

    def run(self):
        fluid.check(self.fn(ctypes.byref(self.desc), *(t.data_ptr() for t in self.bufs), self.out.data_ptr(), None),
                    "wig_fluid_residual_norm2_noalloc")
        return self.out


def _solved(case, seed):
    """Buffers as a solve of a half-full world leaves them: liquid in the
    lower half's blocks (a few walls in it), residuals spread over four
    orders of magnitude."""
    rng = np.random.default_rng(seed)
    w, h = case["w"], case["h"]
    L = abi.layout_py(w, h)
    C, B, bw = L["cell_count"], L["block_count"], L["blocks_wide"]
    field = np.zeros(L["field_bytes"] // 4, dtype=np.float32)
    cg = np.zeros(L["cg_bytes"] // 4, dtype=np.float32)
    blocks = np.zeros(L["blocks_bytes"] // 4, dtype=np.int32)
    y = np.arange(h)[:, None]
    rho = np.where(y < h // 2, 0.0, np.where(rng.random((h, w), dtype=np.float32) < 0.05, -1.0, 1.0)).astype(np.float32)
    field[:8 * C].reshape(C, 8)[:, 2] = rho.ravel()
    r = rng.standard_normal((h, w), dtype=np.float32) * 10.0 ** rng.uniform(-6.0, -2.0, (h, w)).astype(np.float32)
    cg[:4 * C].reshape(C, 4)[:, 1] = r.ravel()
    rows = np.arange(B) // bw
    blocks[B:2 * B] = np.where(8 * rows + 7 >= h // 2, 3, 0)
    return field, blocks, cg


# ---------------------------------------------------------------- the file's functions

def prepare(case, seed):
    if case["kind"] == "norm":
        return _Norm(case, seed)
    if case["kind"] == "batch":
        return _Many(case, seed)
    if case["kind"] == "served":
        return _Served(case, seed)
    return _Single(case, seed)


def run(state):
    return state.run()


# The share of a world's cells that hold liquid, by its kind.
FILLED = {"pond": 0.32, "dam": 0.24, "disks": 0.42, "column": 0.6, "liquids": 0.55, "bodies": 0.62, "dry": 0.0}


def work(case):
    """A step's bytes: each particle's 48 read and written once, and a cell's
    words (its cell record read and written; its counters, field records and
    faces written: 120 bytes), however many iterations the solve takes; two
    flops a cell and an iteration's stencil are below any bound."""
    kind = case["kind"]
    if kind == "norm":
        # the residual and the density of each cell of the blocks worked on
        n = case["w"] * case["h"] / 2
        return {"bytes": 8.0 * n, "flops": 2.0 * n}
    if kind == "dry":
        n = case["w"] * case["h"]
        return {"bytes": 4.0 * n, "flops": 0.0}
    if kind in ("batch", "served"):
        # squares of log-uniform sides, 45% of their cells filled
        lo, hi = float(case["lo"]), float(case["hi"])
        cells = case["worlds"] * (hi * hi - lo * lo) / (2.0 * np.log(hi / lo))
        particles = 0.45 * 4 * cells
    else:
        cells = case["w"] * case["h"]
        particles = FILLED[kind] * (2 if kind == "column" else 4) * cells
    return {"bytes": float(96 * particles + 120 * cells), "flops": float(40 * particles + 100 * cells)}


def exact(case, seed):
    """The norm's sum in 64 bits.  A step has no such value here: its
    classification, sealing and sort decide cell by cell from the particles'
    pseudo-random places, and outside this repository nothing restates them."""
    if case["kind"] != "norm":
        return None
    field, blocks, cg = _solved(case, seed)
    w, h = case["w"], case["h"]
    n = w * h
    active = np.repeat(np.repeat((blocks[((w + 7) // 8) * ((h + 7) // 8):][:((w + 7) // 8) * ((h + 7) // 8)] & 1)
                                 .reshape((h + 7) // 8, (w + 7) // 8), 8, 0), 8, 1)[:h, :w].ravel() != 0
    liquid = field[:8 * n].reshape(n, 8)[:, 2] > 0
    r = cg[:4 * n].reshape(n, 4)[:, 1].astype(np.float64)
    return np.array([np.sum(np.where(active & liquid, r * r, 0.0))])
