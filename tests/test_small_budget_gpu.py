"""Renders whose sample budget is below the pool: the paths live in the pool's first slots,
and the fused kernel's blocks take fewer slots each there.  Against the oracle, bit for
bit, with the budget at a tile's edge and the pool ending inside a block."""
import numpy as np
import pytest

from tests.helpers import camera, compare_slots
from tests.test_inner_bounces_gpu import _scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scene,npaths,side,spp,steps", [
    ("cornell", 4097, (40, 36), 2, 6),
    ("mixed", 20001, (64, 64), 1, 9),      # the budget is one tile
    ("mixed", 20001, (64, 64), 2, 30),
    ("spheres", 13000, (41, 100), 1, 12),  # a tile and four
    ("mixed", 400000, (40, 36), 3, 10),    # a pool that takes the persistent cast without a budget
    ("cornell", 160000, (400, 390), 1, 4),  # more than a wave of half spans, fewer than the pool
])
def test_budget_below_the_pool(rg, po, scene, npaths, side, spp, steps):
    sm, osc, camd = _scene(rg, po, scene)
    cam = camera(camd, *side)
    config = rg.render_config(spp=spp, max_depth=5)
    lane = rg.WavefrontLane(0, npaths)
    lane.setup(sm)
    lane.initialize(cam, config)
    lane.step(steps)
    lane.synchronize()
    oacc, oslots, onext = osc.render(po.camera_from_rgr(cam), po.config_from_rgr(config, side[0] * side[1]), npaths,
                                     steps, threads=16)
    assert compare_slots(lane.debug_slots(), oslots) == {}
    assert lane.stats().paths_started == onext
    ga = lane.accumulation().reshape(-1, 4)
    assert (ga[:, 3] == oacc[:, 3]).all()
    np.testing.assert_allclose(ga[:, :3], oacc[:, :3], rtol=1e-12, atol=1e-300)
