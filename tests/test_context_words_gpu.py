"""Contexts beyond those that share one allocation of host words, from several threads:
each render ends by its own words."""
import threading

import numpy as np
import pytest

from raccoongpurender_gb300 import scenes
from tests.helpers import build, camera

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [3, 70])
def test_many_contexts(rg, po, count):
    sm, _ = build(scenes.cornell_box())
    cam = camera(scenes.cornell_camera(), 24, 20)
    out = [None] * count

    def work(ids):
        lanes = []
        for i in ids:
            lane = rg.WavefrontLane(0, 1024)
            lane.setup(sm)
            lane.initialize(cam, rg.render_config(spp=2 + i % 3, max_depth=5))
            lanes.append(lane)
        for i, lane in zip(ids, lanes):
            lane.render_until_done()
            out[i] = lane.accumulation()[..., 3].sum(), lane.stats().active_paths

    threads = [threading.Thread(target=work, args=(range(k, count, 3),)) for k in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    ref = {}
    for spp in (2, 3, 4):
        lane = rg.WavefrontLane(0, 1024)
        lane.setup(sm)
        lane.initialize(cam, rg.render_config(spp=spp, max_depth=5))
        lane.render_until_done()
        ref[spp] = lane.accumulation()[..., 3].sum()
    for i in range(count):
        assert out[i] == (ref[2 + i % 3], 0)
    assert np.unique(list(ref.values())).size == 3
