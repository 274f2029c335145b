"""The conjugate gradients' block sums in the fast form, which adds every
block's partial, those not worked on being +0: worlds whose block counts
lie at the edges of its rounds (256 columns of 16 rows, two components or
one), with FP32 and FP64 dots, and handles that change form between steps
while blocks come and go, against the plain form bit for bit (which reads
each block's state)."""
import pytest

from worldinagrain_b200 import abi
from worldinagrain_b200 import world as W

from .common import compare_worlds, params

pytestmark = pytest.mark.gpu

TOL = abi.STEP_TOLERANCE | abi.STEP_F64_DOTS


def _step(g, world, s, flags):
    g.step(params(world, s), max_cycles=8, flags=flags, tolerance=1e-6)
    return g.stats(unconverged_ok=True)


@pytest.mark.parametrize("size", [(8, 8), (121, 130), (512, 512), (520, 505), (1000, 523), (1024, 1030)])
@pytest.mark.parametrize("flags", [0, abi.STEP_TOLERANCE, TOL])
def test_fast_sums_equal_plain_at_round_edges(size, flags):
    from worldinagrain_b200 import fluid
    world = W.disks_world(*size, n_disks=max(2, size[0] * size[1] // 6000), r_lo=2, r_hi=9, seed=9)
    a = fluid.LiquidStep(world, W.element_table())
    b = fluid.LiquidStep(world, W.element_table())
    for s in (1, 2):
        sa, sb = _step(a, world, s, flags), _step(b, world, s, flags | abi.STEP_PLAIN)
        assert sa.cycles == sb.cycles and sa.b_norm == sb.b_norm
        # (a world with nothing to solve has no residual to report)
        assert sb.b_norm == 0.0 or sa.rel_residual == sb.rel_residual
    got, ref = a.download(world.copy()), b.download(world.copy())
    diffs = compare_worlds(got, ref, scratch=True)
    assert not diffs, "; ".join(diffs)
    a.close()
    b.close()


@pytest.mark.parametrize("flags", [abi.STEP_TOLERANCE, TOL])
def test_forms_in_turn_on_one_handle(flags):
    """Falling water leaves blocks and enters others; the forms share the
    partials' arrays."""
    from worldinagrain_b200 import fluid
    world = W.small_world(96, 160, seed=6, kind="moving")
    a = fluid.LiquidStep(world, W.element_table())
    b = fluid.LiquidStep(world, W.element_table())
    forms = [abi.STEP_PLAIN, 0, abi.STEP_PERSISTENT]
    for s in range(1, 61):
        sa, sb = _step(a, world, s, flags | forms[(s // 4) % 3]), _step(b, world, s, flags | abi.STEP_PLAIN)
        assert sa.cycles == sb.cycles and sa.rel_residual == sb.rel_residual, s
    got, ref = a.download(world.copy()), b.download(world.copy())
    diffs = compare_worlds(got, ref, scratch=True)
    assert not diffs, "; ".join(diffs)
    a.close()
    b.close()
