"""The plain form's iterations as a loop on the device: a step cut short at
its cap, one that converges before it, and worlds where the cap, the
stopping rule and the residual slots the skipped iterations clear meet at
every remainder of three, against the oracle bit for bit (which runs every
iteration's passes, the converged ones returning early)."""
import pytest

from worldinagrain_b200 import abi
from worldinagrain_b200 import world as W

from .common import compare_worlds, params

pytestmark = pytest.mark.gpu

TOL = abi.STEP_TOLERANCE | abi.STEP_F64_DOTS


@pytest.mark.parametrize("cycles", [1, 2, 3, 5, 16])
@pytest.mark.parametrize("flags", [0, TOL])
@pytest.mark.parametrize("bodies", [False, True])
def test_plain_steps_at_any_cap_match_oracle(cycles, flags, bodies):
    from oracle.oracle import Oracle
    from worldinagrain_b200 import fluid
    if bodies:
        world, table = W.bodies_world(stamps=False)
        elems = W.body_element_table()
    else:
        world, table = W.small_world(61, 43, seed=4, kind="obstacles"), None
        elems = W.element_table()
    ref = world.copy()
    o = Oracle(ref, elems, table.copy()) if bodies else Oracle(ref, elems)
    g = fluid.LiquidStep(world, elems)
    if bodies:
        g.bind_bodies(table)
    got = world.copy()
    for s in range(1, 4):
        P = params(ref, s)
        ost = o.step(P, max_cycles=cycles, flags=flags, tolerance=1e-6)
        g.step(P, max_cycles=cycles, flags=flags | abi.STEP_PLAIN, tolerance=1e-6)
        st = g.stats(unconverged_ok=True)
        g.download(got)
        diffs = compare_worlds(got, ref, region_links=True)
        assert not diffs, f"step {s}: " + "; ".join(diffs)
        assert st.cycles == ost.cycles <= cycles
    g.close()
