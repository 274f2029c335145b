"""No launch shape takes a small world's step out of its one-launch form."""
import pytest

from worldinagrain_b200 import abi
from worldinagrain_b200 import world as W

from .common import compare_worlds, params

pytestmark = pytest.mark.gpu

TOL = abi.STEP_TOLERANCE | abi.STEP_F64_DOTS


SIZES = [(200, 200), (150, 250)]


def _run(world, cells, flags, profile=False):
    from worldinagrain_b200 import fluid
    w = world.copy()
    g = fluid.LiquidStep(w, W.element_table())
    g.set_launch("coarse_cells", cells)
    st = []
    for s in range(1, 4):
        (g.step_profile if profile else g.step)(params(w, s), max_cycles=64, flags=flags, tolerance=1e-6)
        x = g.stats()
        st.append((x.launches, x.cycles, x.rel_residual))
    g.download()
    g.close()
    return w, st


def _world(size):
    return W.disks_world(*size, n_disks=8, r_lo=3, r_hi=10, seed=12)


@pytest.mark.parametrize("size", SIZES)
def test_coarse_cells_of_the_clusters_range_keep_the_one_launch_solve(size):
    a, sa = _run(_world(size), 16384, TOL)
    b, sb = _run(_world(size), 4096, TOL)
    assert sa == sb
    assert sa[0][0] == sa[1][0]  # a step's launches, whatever its iterations
    diffs = compare_worlds(a, b, scratch=True)
    assert not diffs, "; ".join(diffs)


@pytest.mark.parametrize("size", SIZES)
def test_coarse_cells_still_say_which_levels_the_mixed_form_keeps_in_fp32(size):
    """With the levels from 16384 cells in FP32 on chip, a step and a profiled
    one (the loop's launches) are the same, and not what levels stored in 16
    bits give."""
    flags = TOL | abi.STEP_MIXED
    a, sa = _run(_world(size), 16384, flags)
    b, sb = _run(_world(size), 16384, flags, profile=True)
    c, sc = _run(_world(size), 4096, flags)
    assert [x[1:] for x in sa] == [x[1:] for x in sb] and sa[0][2] != sc[0][2]
    diffs = compare_worlds(a, b, scratch=True)
    assert not diffs, "; ".join(diffs)
