"""Liquid beside a block no longer worked on.  The world is a box full of
water; then its upper rows are emptied by the host while a wall is drawn in
on the last row of a block row.  The cells below that wall hold no particles
but stay sealed liquid, so the solve takes the wall cells above them, whose
block retires, for open air at potential 0: what those cells were when they
were last worked on must not reach the solve.  The state is reached by an
edit of the cells, by an upload into a handle that has stepped another
world, and in a pooled lane whose memory another world has used, and every
form's steps are the plain form's bit for bit (the mixed form's a fresh
handle's)."""
import functools

import numpy as np
import pytest

from worldinagrain_b200 import abi
from worldinagrain_b200 import world as W

from .common import compare_worlds, diff_words, params

pytestmark = pytest.mark.gpu

TOL = abi.STEP_TOLERANCE | abi.STEP_F64_DOTS
FORMS = {"fast": 0, "persistent": abi.STEP_PERSISTENT, "bodies": 0, "plain": abi.STEP_PLAIN}
# a cluster's, the loop's and a grid's number of blocks
SIZES = [(64, 64), (256, 240), (520, 520)]
CEILING, SURFACE, FLOOR = 15, 28, 47


def _box(width, height):
    w = W.World(width, height)
    wall = np.zeros((height, width), dtype=bool)
    wall[0, :] = wall[FLOOR:, :] = True
    wall[:, 0] = wall[:, -1] = True
    w.paint(wall, abi.WALL)
    w.paint(~wall, abi.WATER)
    w.config = dict(workload="box", grid=f"{width}x{height}", seed=1, earth_g=W.earth_g_cells())
    return w


def _empty_the_top(w):
    rows = np.zeros((w.H, w.W), dtype=bool)
    rows[1:SURFACE, 1:-1] = True
    w.paint(rows, abi.AIR)
    rows[:] = False
    rows[CEILING, :] = True
    w.paint(rows, abi.WALL)


def _parity(s):
    return abi.STEP_SHIFTED_SET | (abi.STEP_SHIFTED_FIRST if s % 2 else 0)


class _Bytes:
    def __init__(self, ptr, n):
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": (n,), "typestr": "|u1", "version": 2}


def _write_cells(g, w):
    """The host's own copy of the cells, with no call of the library."""
    import torch
    a = np.ascontiguousarray(w.cells).view(np.uint8).reshape(-1)
    torch.cuda.synchronize()
    torch.as_tensor(_Bytes(g.buffers().cells, a.size), device="cuda").copy_(torch.from_numpy(a.copy()))
    torch.cuda.synchronize()


def _handle(world, form):
    from worldinagrain_b200 import fluid
    g = fluid.LiquidStep(world, W.body_element_table())
    if form == "bodies":
        g.bind_bodies(W.Bodies(world.W, world.H))  # none alive
    return g


def _steps(g, world, first, last, flags):
    cycles = []
    for s in range(first, last + 1):
        g.step(params(world, s), max_cycles=64, flags=flags | _parity(s), tolerance=1e-6)
        cycles.append(g.stats(unconverged_ok=True).cycles)
    return cycles


def _beside_idle(w):
    """Liquid cells straight below a cell of a block not worked on."""
    B, bw = w.L["block_count"], w.L["blocks_wide"]
    act = (w.blocks[B:2 * B].reshape(-1, bw) & 1).repeat(8, 0).repeat(8, 1)[: w.H, : w.W] != 0
    rho = w.field_cells()[:, 0, 2].reshape(w.H, w.W) > 0
    return int(np.sum(rho[1:] & act[1:] & ~act[:-1]))


@functools.lru_cache(maxsize=4)
def _edited_plain(size, how, flags):
    return _edited(size, "plain", how, flags)


def _edited(size, form, how, flags):
    """Three steps of the box, the edit, three more; the world and the
    iterations of the last three."""
    w = _box(*size)
    g = _handle(w, form)
    _steps(g, w, 1, 3, flags | FORMS[form])
    g.download()
    _empty_the_top(w)
    if how == "upload":
        g.upload()
    else:
        _write_cells(g, w)
    cycles = _steps(g, w, 4, 6, flags | FORMS[form])
    g.download()
    g.close()
    return w, cycles


@pytest.mark.parametrize("form", ["fast", "persistent", "bodies"])
@pytest.mark.parametrize("how", ["upload", "own_copy"])
@pytest.mark.parametrize("size", SIZES)
@pytest.mark.parametrize("flags", [0, TOL])
def test_an_edited_world_steps_as_plain(size, form, how, flags):
    a, ca = _edited(size, form, how, flags)
    b, cb = _edited_plain(size, how, flags)
    assert _beside_idle(b) > size[0] // 2
    assert ca == cb
    diffs = compare_worlds(a, b, scratch=True)
    assert not diffs, "; ".join(diffs)


@pytest.mark.parametrize("size", SIZES)
@pytest.mark.parametrize("mixed", [0, abi.STEP_MIXED])
def test_a_used_handle_steps_an_upload_as_a_fresh_one(size, mixed):
    saved = _box(*size)
    g = _handle(saved, "plain")
    _steps(g, saved, 1, 3, TOL | abi.STEP_PLAIN)
    g.download()
    _empty_the_top(saved)
    g.upload()
    _steps(g, saved, 4, 4, TOL | abi.STEP_PLAIN)
    g.download()
    g.close()
    got = []
    for used in (True, False):
        w = _box(*size) if used else saved.copy()
        g = _handle(w, "fast")
        if used:
            _steps(g, w, 1, 3, TOL | mixed)
            g.upload(saved)
        cycles = _steps(g, saved, 5, 6, TOL | mixed)
        g.download(w)
        g.close()
        assert _beside_idle(w) > size[0] // 2
        got.append((w, cycles))
    assert got[0][1] == got[1][1]
    diffs = compare_worlds(got[0][0], got[1][0], scratch=True)
    assert not diffs, "; ".join(diffs)


@pytest.mark.parametrize("size", SIZES[:2])
@pytest.mark.parametrize("pooled", [False, True])
def test_a_served_world_beside_another(size, pooled):
    """The edited world steps in lane memory that a box full of water of its
    size was stepped in before (pooled), or after that box in one batch."""
    from worldinagrain_b200 import fluid, serve
    want, _ = _edited_plain(size, "upload", TOL)
    w, other = _box(*size), _box(*size)
    be = serve.GpuBackend([w, other], W.body_element_table(), TOL, 64, 1e-6,
                          pool_bytes=fluid.world_bytes(*size) if pooled else None, seed=0x1234)
    be.admit(0)
    be.admit(1)

    def step(ids):
        be.launch(0, ids)
        be.torch.cuda.synchronize()

    for s in range(1, 4):
        be.first_flags[0] = _parity(s)
        step([0])
    be.fetch(0)
    _empty_the_top(w)
    for which, name in be.names:
        arr = np.ascontiguousarray(getattr(w, name))
        be.fluid.check(be.fluid.lib().wig_batch_upload(be.h, 0, which, arr.ctypes.data, 0, arr.nbytes, None), "upload")
    for s in range(4, 7):
        step([1])
        be.first_flags[0] = _parity(s)
        step([0])
    be.fetch(0)
    be.close()
    assert _beside_idle(w) > size[0] // 2
    names = ("cells", "counters", "blocks") + (() if pooled else ("cg",))
    diffs = compare_worlds(w, want, grid=names, particles=("sorted",), scratch=True)
    n = 4 * (2 * want.C + want.L["face_count"] + 2 * ((want.L["face_count"] + 3) // 4))
    diffs += [d] if (d := diff_words(w.field[:n], want.field[:n], "field")) else []
    assert not diffs, "; ".join(diffs)


@pytest.mark.parametrize("between", ["plain", "bookkeeping", "dispatch"])
@pytest.mark.parametrize("size", SIZES)
def test_blocks_retired_by_another_form(size, between):
    """The blocks retire in a plain step, a bookkeeping-only one or passes
    the host dispatches; the fast steps after it are the plain form's."""
    got = []
    for form in (0, abi.STEP_PLAIN):
        w = _box(*size)
        g = _handle(w, "fast")
        _steps(g, w, 1, 3, TOL | form)
        g.download()
        _empty_the_top(w)
        _write_cells(g, w)
        if between == "plain":
            _steps(g, w, 4, 4, TOL | abi.STEP_PLAIN)
        elif between == "bookkeeping":
            g.step(params(w, 4), max_cycles=64, flags=TOL | form | _parity(4) | abi.STEP_BOOKKEEPING_ONLY, tolerance=1e-6)
        else:
            for name in ("SYNC", "SYNC_PARTICLES", "SYNC_SEED", "COMPACT", "RETIRE"):
                g.dispatch(params(w, 4), name)
        cycles = _steps(g, w, 5, 7, TOL | form)
        g.download()
        g.close()
        assert _beside_idle(w) > size[0] // 2
        got.append((w, cycles))
    assert got[0][1] == got[1][1]
    diffs = compare_worlds(got[0][0], got[1][0], scratch=True)
    assert not diffs, "; ".join(diffs)


@pytest.mark.parametrize("size", SIZES)
def test_blocks_dropped_without_retiring(size):
    """A dam's upper part emptied, and its blocks dropped by a compact that no
    retire follows: the solve's sums take none of theirs."""
    got = []
    for form in (0, abi.STEP_PLAIN):
        w = W.dam_break(*size)
        g = _handle(w, "fast")
        _steps(g, w, 1, 3, TOL | form)
        g.download()
        top = (w.cell_view()[:, :, 0] & 0xff) == abi.WATER
        top[w.H - w.H // 4:, :] = False
        w.paint(top, abi.AIR)
        _write_cells(g, w)
        for name in ("SYNC", "SYNC_PARTICLES", "SYNC_SEED", "COMPACT"):
            g.dispatch(params(w, 4), name)
        cycles = _steps(g, w, 5, 7, TOL | form)
        g.download()
        g.close()
        assert _beside_idle(w) == 0
        got.append((w, cycles))
    assert got[0][1] == got[1][1]
    diffs = compare_worlds(got[0][0], got[1][0], scratch=True)
    assert not diffs, "; ".join(diffs)


@pytest.mark.parametrize("size", SIZES)
def test_a_world_whose_bodies_are_unbound(size):
    """A host writes all of a world's buffers while bodies are bound (which
    needs no bind), then unbinds them."""
    import torch
    saved = _box(*size)
    g = _handle(saved, "plain")
    _steps(g, saved, 1, 3, TOL | abi.STEP_PLAIN)
    g.download()
    _empty_the_top(saved)
    g.upload()
    _steps(g, saved, 4, 4, TOL | abi.STEP_PLAIN)
    g.download()
    g.close()
    got = []
    for form in (0, abi.STEP_PLAIN):
        w = _box(*size)
        g = _handle(w, "bodies")
        _steps(g, w, 1, 3, TOL | form)
        torch.cuda.synchronize()
        for name in abi.BUFFER_NAMES:
            a = np.ascontiguousarray(getattr(saved, name)).view(np.uint8).reshape(-1)
            torch.as_tensor(_Bytes(getattr(g.buffers(), name), a.size), device="cuda").copy_(torch.from_numpy(a.copy()))
        torch.cuda.synchronize()
        g.bind_bodies(None)
        cycles = _steps(g, saved, 5, 6, TOL | form)
        g.download(w)
        g.close()
        assert _beside_idle(w) > size[0] // 2
        got.append((w, cycles))
    assert got[0][1] == got[1][1]
    diffs = compare_worlds(got[0][0], got[1][0], scratch=True)
    assert not diffs, "; ".join(diffs)
