"""A world whose steps solve in one launch is not tuned: its profiled steps
run other kernels."""
import pytest

from worldinagrain_b200 import abi, tune
from worldinagrain_b200 import world as W

from .common import params


class _OneLaunch:
    shapes = {"coarse_cells": 2048, "level_per_sm": 32, "cg_per_sm": 4, "relax_per_sm": 64}

    def one_launch(self):
        return True

    def launch_shapes(self):
        return dict(self.shapes)

    def get_launch(self, name):
        return self.shapes[name]

    def set_launch(self, name, value):
        raise AssertionError(f"{name} set to {value}")


def test_a_one_launch_world_keeps_its_shapes_without_a_step():
    def step():
        raise AssertionError("stepped")
    assert tune.autotune(_OneLaunch(), step) == (_OneLaunch.shapes, {})


@pytest.mark.gpu
@pytest.mark.parametrize("size,bodies,legacy,own", [((200, 200), False, True, True), ((208, 200), False, False, False),
                                                    ((512, 512), False, False, False), ((520, 512), False, True, False),
                                                    ((300, 240), True, True, True)])
@pytest.mark.parametrize("stream", ["legacy", "own"])
def test_which_worlds_solve_in_one_launch(size, bodies, legacy, own, stream):
    """The library's word on it against the launches a step reports, on the
    legacy stream and on one of its own: the same whatever its iterations, or
    more with each."""
    import torch
    from worldinagrain_b200 import fluid
    one = legacy if stream == "legacy" else own
    s = torch.cuda.Stream()
    if bodies:
        w, table = W.bodies_world(*size, stamps=False)
    else:
        w = W.disks_world(*size, n_disks=8, r_lo=3, r_hi=10, seed=12)
    g = fluid.LiquidStep(w, W.body_element_table(), stream=0 if stream == "legacy" else s.cuda_stream)
    if bodies:
        g.bind_bodies(table)
    assert g.one_launch() is one
    seen = []
    for cycles in (1, 4):
        g.step(params(w, cycles), max_cycles=cycles, flags=abi.STEP_TOLERANCE | abi.STEP_F64_DOTS, tolerance=1e-12)
        st = g.stats(unconverged_ok=True)
        assert st.cycles == cycles
        seen.append(st.launches)
    assert (seen[0] == seen[1]) is one
    g.close()


@pytest.mark.gpu
def test_a_batch_says_it_of_one_world_only():
    from worldinagrain_b200 import fluid
    import torch
    s = torch.cuda.Stream().cuda_stream
    small, large = [W.dam_break(64, 64, seed=2), W.dam_break(96, 64, seed=3)], [W.dam_break(520, 520, seed=2)]
    for ws, one in ((small[:1], (True, True)), (small, (False, False)), (large, (True, False))):
        b = fluid.Batch(ws, W.element_table())
        assert (b.one_launch(), b.one_launch(stream=s)) == one
        b.close()
