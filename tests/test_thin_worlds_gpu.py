"""Worlds of a few rows or columns: their levels only halve as they coarsen,
so the levels one CTA holds start deeper than a level's own cells say.  They
are made, and every form's steps are the plain form's bit for bit."""
import numpy as np
import pytest

from worldinagrain_b200 import abi
from worldinagrain_b200 import world as W

from .common import compare_worlds, params

pytestmark = pytest.mark.gpu

TOL = abi.STEP_TOLERANCE | abi.STEP_F64_DOTS


def _thin(width, height):
    w = W.World(width, height)
    water = np.zeros((height, width), dtype=bool)
    water[height // 3:, : width // 3] = True
    water[:, : width // 5] = True
    w.paint(water, abi.WATER)
    w.config = dict(workload="thin", grid=f"{width}x{height}", seed=1, earth_g=W.earth_g_cells())
    return w


@pytest.mark.parametrize("form", ["fast", "persistent", "bodies"])
@pytest.mark.parametrize("size", [(8192, 2), (2, 8192), (8192, 8), (16384, 4), (32768, 8), (32768, 16)])
def test_thin_worlds_step_as_plain(size, form):
    from worldinagrain_b200 import fluid
    world = _thin(*size)
    got = []
    for flags in (abi.STEP_PERSISTENT if form == "persistent" else 0, abi.STEP_PLAIN):
        w = world.copy()
        g = fluid.LiquidStep(w, W.body_element_table())
        if form == "bodies":
            g.bind_bodies(W.Bodies(*size))  # none alive
        cycles = []
        for s in range(1, 4):
            g.step(params(w, s), max_cycles=16, flags=TOL | flags, tolerance=1e-6)
            cycles.append(g.stats(unconverged_ok=True).cycles)
        g.download()
        g.close()
        got.append((w, cycles))
    assert got[0][1] == got[1][1]
    diffs = compare_worlds(got[0][0], got[1][0], scratch=True)
    assert not diffs, "; ".join(diffs)


def test_a_thin_world_steps_by_its_bookkeeping_alone():
    from worldinagrain_b200 import fluid
    world = W.World(8192, 2)
    world.config = dict(workload="thin", grid="8192x2", seed=1, earth_g=W.earth_g_cells())
    g = fluid.LiquidStep(world, W.element_table())
    g.step(params(world, 1), flags=abi.STEP_BOOKKEEPING_ONLY)
    assert g.stats().particles == 0
    g.close()
