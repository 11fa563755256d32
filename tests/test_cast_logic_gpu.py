"""Bounces of small pools (cast and logic in one launch) against the oracle, bit for bit,
at the edges of a block's span of slots and of the rule that chooses the span."""
import numpy as np
import pytest

from tests.helpers import camera, compare_slots
from tests.test_inner_bounces_gpu import _scene

pytestmark = pytest.mark.gpu
WAVE = 152 * 4 * 256  # the largest pool that blocks of 256 slots take in one wave


@pytest.mark.parametrize("scene,npaths,steps,cfg", [
    ("cornell", 1, 3, dict(dof=0.0)),
    ("mixed", 255, 12, {}),
    ("spheres", 257, 12, dict(dof=0.0)),
    ("mixed", 4097, 20, dict(rr_depth=2, spp=5, max_depth=6)),  # slots retire, then none is live
    ("mixed", WAVE, 4, dict(max_depth=2)),
    ("cornell", WAVE + 1, 4, {}),
    ("mixed", WAVE + 513, 6, dict(max_depth=3, spp=120)),
])
def test_fused_bounces(rg, po, scene, npaths, steps, cfg):
    sm, osc, camd = _scene(rg, po, scene)
    cam = camera(camd, 40, 36)
    config = rg.render_config(**cfg)
    lane = rg.WavefrontLane(0, npaths)
    lane.set_render_trace(False)
    lane.setup(sm)
    lane.initialize(cam, config)
    lane.step(steps)
    lane.synchronize()
    oacc, oslots, onext = osc.render(po.camera_from_rgr(cam), po.config_from_rgr(config, 40 * 36), npaths, steps,
                                     threads=16)
    assert compare_slots(lane.debug_slots(), oslots) == {}
    assert lane.stats().paths_started == onext
    ga = lane.accumulation().reshape(-1, 4)
    assert (ga[:, 3] == oacc[:, 3]).all()
    np.testing.assert_allclose(ga[:, :3], oacc[:, :3], rtol=1e-12, atol=1e-300)
