"""Replayed bounces inside a run (rgr_set_graph_mode(1) with the cast of large pools) against
launched ones, bit for bit: graphs of several bounces with a remainder, renders to their end,
a second render that replays the first one's graph with another camera and seed, batches, and a
frozen guide with selected rows."""
import numpy as np
import pytest

from raccoongpurender_gb300 import scenes
from tests.helpers import build, camera

pytestmark = pytest.mark.gpu


def _same(a, b):
    for k in a[0]:
        assert (np.asarray(a[0][k]).view(np.uint32) == np.asarray(b[0][k]).view(np.uint32)).all(), k
    assert a[2:] == b[2:]
    assert (a[1][..., 3] == b[1][..., 3]).all()
    np.testing.assert_allclose(a[1], b[1], rtol=1e-12, atol=1e-300)


def _renders(rg, lane, cams, cfg, steps):
    out = []
    for seed, cam in enumerate(cams):
        lane.initialize(cam, rg.render_config(seed_offset=seed, **cfg))
        if steps:
            for n in steps:
                lane.step(n)
            ran = sum(steps)
        else:
            ran = lane.render_until_done()
        lane.synchronize()
        st = lane.stats()
        out.append((lane.debug_slots(), lane.accumulation(), ran, st.steps, st.paths_started, st.rays_traced))
    return out


@pytest.mark.parametrize("graph_steps", [1, 4, 7])
@pytest.mark.parametrize("steps,cfg", [((13, 2, 30), {}), ((1, 9), dict(spp=2, max_depth=4)),
                                       ((), dict(spp=12, max_depth=6))])
@pytest.mark.parametrize("guide_cfg", [None, dict(max_depth=2), dict(train_interval=3)])
def test_replayed_runs(rg, po, graph_steps, steps, cfg, guide_cfg):
    mesh, env, camd = scenes.mixed_scene(level=3, seed=3)
    sm, _ = build(mesh, env=env)
    cams = [camera(camd, 40, 36), camera(dict(camd, vfov=camd["vfov"] * 0.7), 40, 36), camera(camd, 33, 20)]
    W, b = rg.Guide(0).weights()
    out = []
    for mode in (True, False):
        lane = rg.WavefrontLane(0, 5000)
        lane.set_graph_mode(mode)
        lane.set_render_trace(True, 12)
        lane.set_render_tuning(4, graph_steps)
        lane.setup(sm)
        if guide_cfg is not None:
            guide = rg.Guide(0, train=0, **guide_cfg)
            guide.set_weights(W * 1.5, b)
            lane.set_guide(guide)
        out.append(_renders(rg, lane, cams, cfg, steps))
    for x, y in zip(*out):
        _same(x, y)


@pytest.mark.parametrize("steps_per_launch", [1, 2, 6])
def test_replayed_batches(rg, po, steps_per_launch):
    from tests.test_batch_gpu import _requests
    out = []
    for mode in (1, 0):
        batch = rg.Batch(0, 5000)
        assert batch._lib.rgr_set_graph_mode(batch._lib.rgr_batch_context(batch._h), mode) == 0
        batch.set_render_trace(12, True)
        ids = [batch.add(sm, cam, cfg) for sm, _, cam, cfg in _requests(po)]
        for order in (rg.ORDER_FIFO, rg.ORDER_SHORTEST_FIRST):  # the second run replays nothing stale
            steps = batch.run(order=order, steps_per_launch=steps_per_launch)
            sums = np.concatenate([batch.accumulation(i).reshape(-1, 4) for i in ids])
            out.append((batch.debug_slots(), sums, steps))
    _same(out[0], out[2])
    _same(out[1], out[3])
