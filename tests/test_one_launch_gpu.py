"""A single world's solve as one launch or as the loop's launches, by its
number of blocks: on a cluster up to 640, the loop's launches up to 4096, a
grid above, whose block sums are shared by the grid above 8192.  Worlds on
either side of each line, and the mixed form there, against the plain form
or the same form by the other route, bit for bit."""
import pytest

from worldinagrain_b200 import abi
from worldinagrain_b200 import world as W

from .common import compare_worlds, params

pytestmark = pytest.mark.gpu

TOL = abi.STEP_TOLERANCE | abi.STEP_F64_DOTS
SIZES = [(200, 200), (208, 200), (512, 512), (520, 512), (720, 728), (728, 728)]


def _run(world, flags, steps=2, profile=False):
    from worldinagrain_b200 import fluid
    g = fluid.LiquidStep(world, W.element_table())
    out = []
    for s in range(1, steps + 1):
        step = g.step_profile if profile else g.step
        step(params(world, s), max_cycles=10, flags=flags, tolerance=1e-6)
        st = g.stats(unconverged_ok=True)
        out.append((st.cycles, st.rel_residual, st.b_norm))
    got = g.download(world.copy())
    g.close()
    return got, out


@pytest.mark.parametrize("size", SIZES)
@pytest.mark.parametrize("flags", [0, TOL])
def test_route_by_size_equals_plain(size, flags):
    world = W.disks_world(*size, n_disks=size[0] * size[1] // 5000, r_lo=3, r_hi=10, seed=12)
    for form in (0, abi.STEP_PERSISTENT):
        a, sa = _run(world, flags | form)
        b, sb = _run(world, flags | abi.STEP_PLAIN)
        assert [x[0] for x in sa] == [x[0] for x in sb] and (flags == 0 or sa == sb)
        diffs = compare_worlds(a, b, scratch=True)
        assert not diffs, "; ".join(diffs)


@pytest.mark.parametrize("size", SIZES)
def test_mixed_route_by_size_equals_the_loop(size):
    """A profiled step runs the loop's launches at any size."""
    world = W.disks_world(*size, n_disks=size[0] * size[1] // 5000, r_lo=3, r_hi=10, seed=12)
    a, sa = _run(world, TOL | abi.STEP_MIXED)
    b, sb = _run(world, TOL | abi.STEP_MIXED, profile=True)
    assert sa == sb
    diffs = compare_worlds(a, b, scratch=True)
    assert not diffs, "; ".join(diffs)


def test_handles_of_other_coarse_sizes_leave_a_handles_launches_valid():
    """The kernels' shared-memory limits are the process's, not a handle's:
    a handle of smaller coarse levels made later takes none away."""
    from worldinagrain_b200 import fluid
    big = W.small_world(500, 420, seed=3, kind="dam")
    small = W.small_world(24, 20, seed=3, kind="dam")
    g = fluid.LiquidStep(big, W.element_table())
    h = fluid.LiquidStep(small, W.element_table())
    for world, step in ((small, h), (big, g)):
        step.step(params(world, 1), max_cycles=8, flags=TOL, tolerance=1e-6)
        assert step.stats(unconverged_ok=True).cycles > 0
        step.close()
