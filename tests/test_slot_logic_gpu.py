"""Fused bounces of scenes of few primitives (one thread a slot) against the oracle, bit
for bit: pools that end inside a block, budgets below the pool, requests of several scenes, and
the scene from which on a block lists its slots."""
import numpy as np
import pytest

from raccoongpurender_gb300 import scenes
from tests.helpers import build, camera, compare_slots
from tests.test_inner_bounces_gpu import _scene

pytestmark = pytest.mark.gpu


def _check(rg, po, sm, osc, cam, config, npaths, steps, npix):
    lane = rg.WavefrontLane(0, npaths)
    lane.set_render_trace(False)
    lane.setup(sm)
    lane.initialize(cam, config)
    lane.step(steps)
    lane.synchronize()
    oacc, oslots, onext = osc.render(po.camera_from_rgr(cam), po.config_from_rgr(config, npix), npaths, steps, threads=16)
    assert compare_slots(lane.debug_slots(), oslots) == {}
    assert lane.stats().paths_started == onext
    ga = lane.accumulation().reshape(-1, 4)
    assert (ga[:, 3] == oacc[:, 3]).all()
    np.testing.assert_allclose(ga[:, :3], oacc[:, :3], rtol=1e-12, atol=1e-300)


@pytest.mark.parametrize("scene,npaths,steps,cfg", [
    ("cornell", 1, 3, dict(dof=0.0)),
    ("spheres", 255, 12, dict(dof=0.0)),
    ("cornell", 257, 20, dict(rr_depth=1, max_depth=0)),
    ("spheres", 4097, 20, dict(dof=0.0, spp=2, max_depth=5)),
    ("cornell", 200001, 4, {}),
])
def test_pools(rg, po, scene, npaths, steps, cfg):
    sm, osc, camd = _scene(rg, po, scene)
    _check(rg, po, sm, osc, camera(camd, 40, 36), rg.render_config(**cfg), npaths, steps, 40 * 36)


@pytest.mark.parametrize("ntris", [1024, 1025])
def test_edge_of_the_rule(rg, po, ntris):
    mesh = scenes.displaced_icosphere(3, seed=9)
    mesh = scenes.Mesh(mesh.points, mesh.indices[:ntris], mesh.materials[:ntris])
    sm, osc = build(mesh, env=scenes.sky_envmap(64, 32))
    cam = camera(dict(eye=(0, 0.3, 3.0), target=(0, 0, 0), up=(0, 1, 0), vfov=40.0), 40, 36)
    _check(rg, po, sm, osc, cam, rg.render_config(max_depth=6), 3000, 12, 40 * 36)


def test_requests_of_several_scenes(rg, po):
    reqs = []
    for k, name in enumerate(("cornell", "spheres", "cornell")):
        sm, osc, camd = _scene(rg, po, name)
        reqs.append((sm, osc, camera(camd, 20 + 7 * k, 30), rg.render_config(dof=0.0, max_depth=5, spp=3 - k)))
    npaths = 700
    b = rg.Batch(0, npaths)
    ids = [b.add(sm, cam, cfg) for sm, _, cam, cfg in reqs]
    steps = b.run(order=rg.ORDER_FIFO, steps_per_launch=3)
    oaccs, oslots = po.render_batch([r[1] for r in reqs], [po.camera_from_rgr(r[2]) for r in reqs],
                                    [po.config_from_rgr(r[3], r[2].image_w * r[2].image_h) for r in reqs], npaths,
                                    steps, threads=16)
    for i, oa in zip(ids, oaccs):
        ga = b.accumulation(i).reshape(-1, 4)
        assert (ga[:, 3] == oa[:, 3]).all()
        np.testing.assert_allclose(ga[:, :3], oa[:, :3], rtol=1e-12, atol=1e-300)
        assert b.request_stats(i).complete_ms > 0
    fields = ["T", "L", "ro", "rd", "rng", "pixel_index", "queue"]
    assert compare_slots(b.debug_slots(), oslots, fields=fields) == {}
