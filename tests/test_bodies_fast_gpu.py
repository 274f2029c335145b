"""Free bodies coupled into the fast form's solve (one launch, a cluster or
a cooperative grid by the world's size), every buffer the reference's passes
leave bit for bit: against the plain form, which runs them one by one, on
tanks of the sizes either side of the rule that chooses the group."""
import pytest

from worldinagrain_b200 import abi
from worldinagrain_b200 import world as W

from .common import compare_worlds, diff_words, params

pytestmark = pytest.mark.gpu

TOL = abi.STEP_TOLERANCE | abi.STEP_F64_DOTS


@pytest.mark.parametrize("size", [(96, 80), (259, 201), (512, 512), (600, 520)])
@pytest.mark.parametrize("case", ["tolerance", "default", "viscous", "one_cycle"])
def test_fast_steps_with_bodies_equal_plain(size, case):
    from worldinagrain_b200 import fluid
    liquid, flags, cycles = {"tolerance": (abi.WATER, TOL, 64), "default": (abi.WATER, 0, abi.FLUID_CYCLES),
                             "viscous": (W.MUD, abi.STEP_TOLERANCE | abi.STEP_VISCOUS, 64),
                             "one_cycle": (abi.WATER, TOL, 1)}[case]
    world, bodies = W.bodies_world(*size, liquid=liquid, stamps=False)
    got = []
    for form in (0, abi.STEP_PLAIN):
        w, b = world.copy(), bodies.copy()
        g = fluid.LiquidStep(w, W.body_element_table())
        g.bind_bodies(b)
        cyc = []
        for s in range(1, 4):
            g.step(params(w, s), max_cycles=cycles, flags=flags | form, tolerance=1e-6)
            cyc.append(g.stats(unconverged_ok=True).cycles)
        g.download()
        g.download_bodies(b)
        g.close()
        got.append((w, b, cyc))
    (wa, ba, ca), (wb, bb, cb) = got
    assert ca == cb
    diffs = compare_worlds(wa, wb) + [d for n in ("motion", "pushes") if (d := diff_words(getattr(ba, n), getattr(bb, n), n))]
    assert not diffs, "; ".join(diffs)


class _Bytes:
    def __init__(self, ptr, n):
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": (n,), "typestr": "|u1", "version": 2}


def test_a_host_writing_its_buffers_needs_no_rebinding():
    """The world taken back by the host's own copies after 30 steps, blocks
    then worked on idle again; no bind call tells the handle."""
    import numpy as np
    import torch
    from worldinagrain_b200 import fluid
    world, bodies = W.bodies_world(160, 120, stamps=False)
    got = []
    for form in (0, abi.STEP_PLAIN):
        w, b = world.copy(), bodies.copy()
        g = fluid.LiquidStep(w, W.body_element_table())
        g.bind_bodies(b)
        for s in range(1, 31):
            g.step(params(w, s), max_cycles=64, flags=TOL | form, tolerance=1e-6)
        torch.cuda.synchronize()
        at = g.buffers()
        for name in abi.BUFFER_NAMES:
            a = np.ascontiguousarray(getattr(world, name)).view(np.uint8).reshape(-1)
            torch.as_tensor(_Bytes(getattr(at, name), a.size), device="cuda").copy_(torch.from_numpy(a.copy()))
        torch.cuda.synchronize()
        for s in range(1, 4):
            g.step(params(w, s), max_cycles=64, flags=TOL | form, tolerance=1e-6)
        g.download()
        g.download_bodies(b)
        g.close()
        got.append((w, b))
    (wa, ba), (wb, bb) = got
    diffs = compare_worlds(wa, wb) + [d for n in ("motion", "pushes") if (d := diff_words(getattr(ba, n), getattr(bb, n), n))]
    assert not diffs, "; ".join(diffs)
