"""Means of the readback kernel, which divides in double only where a float quotient leaves
the half in doubt, against numpy's: bit for bit."""
import numpy as np
import pytest

from raccoongpurender_gb300 import scenes
from tests.helpers import build, camera

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,steps", [(1, 1, 3), (33, 7, 40), (900, 700, 6), (640, 360, 30)])
def test_means(rg, po, w, h, steps):
    mesh, env, camd = scenes.mixed_scene(level=3, seed=3)
    sm, _ = build(mesh, env=env)
    lane = rg.WavefrontLane(0, 1 << 18)
    lane.setup(sm)
    lane.initialize(camera(camd, w, h), rg.render_config())
    lane.step(steps)
    acc, got = lane.accumulation(), lane.intermediate()
    cnt = acc[..., 3:]
    with np.errstate(all="ignore"):
        mean = np.where(cnt > 0, acc[..., :3] / cnt, 0.0).astype(np.float32).astype(np.float16)
    assert (got[..., :3] == mean.view(np.uint16)).all()
    assert (got[..., 3] == (acc[..., 3].astype(np.uint64) & 0xFFFF)).all()
    if w * h * 3 > 500_000:  # values enough that the division decided some
        assert (mean > 0).sum() > 100_000
