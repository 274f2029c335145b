"""A grid of every multiprocessor whose CTAs' barrier waits all run out: the
step reports it, and the handle's next step is the plain form's."""
import pytest

from worldinagrain_b200 import abi
from worldinagrain_b200 import world as W

from .common import compare_worlds, params

pytestmark = pytest.mark.gpu

TOL = abi.STEP_TOLERANCE | abi.STEP_F64_DOTS
SHIFTED = abi.STEP_SHIFTED_SET | abi.STEP_SHIFTED_FIRST


@pytest.fixture
def lowered_limits():
    from worldinagrain_b200 import fluid
    yield fluid.set_wait_limits
    fluid.set_wait_limits(0, 0)


@pytest.mark.parametrize("limit", [1, 3])
def test_every_cta_of_a_full_grid_gives_up(limit, lowered_limits):
    from worldinagrain_b200 import fluid
    world = W.disks_world(520, 520, n_disks=40, r_lo=3, r_hi=10, seed=12)
    g = fluid.LiquidStep(world.copy(), W.element_table())
    lowered_limits(0, limit)
    for s in range(1, 4):
        g.step(params(world, s), max_cycles=64, flags=TOL | abi.STEP_PERSISTENT, tolerance=1e-6)
        with pytest.raises(fluid.WigError, match="WIG_E_STATE.*barrier"):
            g.stats()
    lowered_limits(0, 0)
    got = []
    for form in (abi.STEP_PERSISTENT, abi.STEP_PLAIN):
        g.upload(world)
        g.step(params(world, 1), max_cycles=64, flags=TOL | SHIFTED | form, tolerance=1e-6)
        cycles = g.stats().cycles
        got.append((g.download(world.copy()), cycles))
    g.close()
    assert got[0][1] == got[1][1]
    diffs = compare_worlds(got[0][0], got[1][0], scratch=True)
    assert not diffs, "; ".join(diffs)


def test_the_documented_spin_limits_are_taken(lowered_limits):
    """Up to 2^23 polls are taken, a number from the default up standing for
    it; more are refused, as are more than 2^22 retries."""
    from worldinagrain_b200 import fluid
    for spin in (1, 1 << 20, (1 << 20) + 1, 1 << 22, 1 << 23):
        lowered_limits(0, spin)
    lowered_limits(1 << 22, 0)
    for limits in ((0, (1 << 23) + 1), (0, 0xFFFFFFFF), ((1 << 22) + 1, 0)):
        with pytest.raises(fluid.WigError, match="WIG_E_ARG"):
            lowered_limits(*limits)
