"""compact against the oracle on worlds either side of the rule that makes
it two launches, with random marks and last states."""
import numpy as np
import pytest

from worldinagrain_b200 import abi
from worldinagrain_b200 import world as W

from .common import params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(8, 8), (512, 512), (520, 512), (1001, 777), (1024, 1024), (2056, 1032)])
def test_compact_matches_oracle(size):
    from oracle.oracle import Oracle
    from worldinagrain_b200 import fluid
    world = W.World(*size, capacity=256)
    world.config = dict(earth_g=W.earth_g_cells())
    B = world.L["block_count"]
    rng = np.random.default_rng(B)
    world.blocks[:B] = np.where(rng.random(B) < 0.08, rng.integers(1, 4, B), 0)
    world.blocks[B:2 * B] = np.where(rng.random(B) < 0.4, 1 | (rng.integers(0, 8, B) << 1), 0)
    ref = world.copy()
    o = Oracle(ref, W.element_table())
    g = fluid.LiquidStep(world, W.element_table())
    P = params(world, 1)
    o.pass_(P, "COMPACT", 0, 0)
    g.dispatch(P, "COMPACT")
    got = g.download(world.copy(), names=("blocks",))
    na, nr = int(ref.blocks[4 * B]), int(ref.blocks[4 * B + 1])
    assert (int(got.blocks[4 * B]), int(got.blocks[4 * B + 1])) == (na, nr) and (na > 0 or B == 1)
    assert np.array_equal(got.blocks[B:2 * B], ref.blocks[B:2 * B])
    assert np.array_equal(got.blocks[2 * B:2 * B + na], ref.blocks[2 * B:2 * B + na])
    assert np.array_equal(got.blocks[3 * B:3 * B + nr], ref.blocks[3 * B:3 * B + nr])
    g.close()
