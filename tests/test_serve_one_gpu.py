"""A server of one world: a deferred batch of one, whose memory moves with
each admission, steps as the world alone does, bit for bit, pooled or not."""
import pytest

from worldinagrain_b200 import abi
from worldinagrain_b200 import serve
from worldinagrain_b200 import world as W

from .common import compare_worlds

pytestmark = pytest.mark.gpu

TOL = abi.STEP_TOLERANCE | abi.STEP_F64_DOTS
# the sizes a world alone solves on a cluster, as the loop's launches, on a grid
SIZES = [(48, 40), (256, 240), (520, 520)]


def _params(w, s):
    return W.make_params(w, frame=s, seed=0x5eed, earth_g=w.config["earth_g"])


def _backend(w, flags, pooled):
    from worldinagrain_b200 import fluid
    return serve.GpuBackend([w], W.element_table(), flags, 64, 1e-6,
                            pool_bytes=fluid.world_bytes(w.W, w.H, w.L["liquid_per_cell"], w.cap) if pooled else None)


@pytest.mark.parametrize("flags", [0, TOL, TOL | abi.STEP_MIXED])
@pytest.mark.parametrize("pooled", [False, True])
@pytest.mark.parametrize("size", SIZES)
def test_one_served_world_steps_as_alone(size, pooled, flags):
    from worldinagrain_b200 import fluid
    base = W.disks_world(*size, n_disks=max(1, size[0] * size[1] // 5000), r_lo=2, r_hi=8, seed=9)
    ref = base.copy()
    g = fluid.LiquidStep(ref, W.element_table())
    if flags & abi.STEP_MIXED:
        g.set_launch("coarse_cells", 2048)  # which levels the form stores in 16 bits
    for s in range(1, 7):
        g.step(_params(ref, s), max_cycles=64, flags=flags, tolerance=1e-6)
    cycles = g.stats(unconverged_ok=True).cycles
    g.download()
    g.close()
    w, other = base.copy(), base.copy()
    be, beside = _backend(w, flags, pooled), _backend(other, flags, pooled)
    be.admit(0)
    for s in range(1, 7):
        be.launch(0, [0])
        if s == 3:
            # evicted, its memory taken by another batch's world, admitted again
            be.evict(0)
            beside.admit(0)
            be.admit(0)
    be.torch.cuda.synchronize()
    assert be.stats([0])[0].cycles == cycles
    be.fetch(0)
    be.close()
    beside.close()
    n = 4 * (2 * w.C + w.L["face_count"] + 2 * ((w.L["face_count"] + 3) // 4))
    w.field[n:] = ref.field[n:]
    grid = ("cells", "counters", "field", "blocks") + (() if pooled else ("cg",))
    diffs = compare_worlds(w, ref, grid=grid, particles=("sorted",), region_links=True, scratch=True)
    assert not diffs, "; ".join(diffs)


@pytest.mark.parametrize("pooled", [False, True])
def test_one_served_world_takes_a_batchs_knobs(pooled):
    from worldinagrain_b200 import fluid
    w = W.dam_break(160, 128, seed=4)
    be = _backend(w, TOL, pooled)
    with pytest.raises(fluid.WigError, match="WIG_E_ARG"):
        be.set_launch("coarse_cells", 16384)  # the cluster's range is a world's whose memory stays
    be.admit(0)
    be.launch(0, [0])
    shapes, _ = be.autotune([0])
    assert shapes["coarse_cells"] <= 4096
    be.launch(0, [0])
    assert be.stats([0])[0].rel_residual <= 1e-6
    be.close()
