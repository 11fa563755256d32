"""Bounces inside a run (no logic pass between them, launch_inner) against the
oracle: the state after a run of n bounces is bit for bit that of n bounces,
whatever the pool's remainder, the scene's kinds of hit and the ways a path ends."""
import numpy as np
import pytest

from raccoongpurender_gb300 import materials, scenes
from tests.helpers import build, camera, compare_slots

pytestmark = pytest.mark.gpu


def _scene(rg, po, name):
    if name == "mixed":
        mesh, env, camd = scenes.mixed_scene(level=3, seed=3)
        return (*build(mesh, env=env), camd)
    mesh = scenes.cornell_box()
    if name == "cornell":
        return (*build(mesh), scenes.cornell_camera())
    sm = rg.SceneManager()
    sm.addMesh(mesh)
    sph = np.array([[0.0, 1.5, 0.0, 0.3], [-0.5, 1.4, 0.4, 0.2], [0.5, 0.9, 0.3, 0.25]], np.float32)
    sm.addSpheres(sph, [materials.dielectric(), materials.ward(alpha=0.2), materials.specular()])
    sm.buildBVH()
    return sm, po.OracleScene.from_scene(sm, mesh.points, mesh.indices, spheres=sph), scenes.cornell_camera()


@pytest.mark.parametrize("scene,npaths,steps,cfg", [
    ("cornell", 1, 2, dict(dof=0.0)),                          # the smallest pool, one inner bounce
    ("cornell", 4097, 9, dict(dof=0.0, max_depth=3)),          # one slot past a tile, the depth limit
    ("cornell", 5000, 40, dict(rr_depth=1, max_depth=0)),      # Russian roulette from the second segment
    ("cornell", 8192, 30, dict(spp=3, max_depth=5)),           # slots retire, then nothing is in flight
    ("mixed", 8191, 2, {}),
    ("mixed", 12289, 33, {}),                                  # volumes, envmap, every material
    ("mixed", 4096, 24, dict(rr_depth=2, spp=5, max_depth=6, radiance_clamp=5.0)),
    ("spheres", 6000, 20, dict(dof=0.0)),                      # sphere hits carry their type too
])
def test_run_matches_oracle(rg, po, scene, npaths, steps, cfg):
    sm, osc, camd = _scene(rg, po, scene)
    cam = camera(camd, 40, 36)
    config = rg.render_config(**cfg)
    lane = rg.WavefrontLane(0, npaths)
    lane.set_render_trace(True, 12)  # whatever the pool's size
    lane.setup(sm)
    lane.initialize(cam, config)
    lane.step(steps)
    lane.synchronize()
    oacc, oslots, onext = osc.render(po.camera_from_rgr(cam), po.config_from_rgr(config, 40 * 36), npaths, steps,
                                     threads=16)
    assert compare_slots(lane.debug_slots(), oslots) == {}
    st = lane.stats()
    assert st.paths_started == onext and st.steps == steps
    ga = lane.accumulation().reshape(-1, 4)
    assert (ga[:, 3] == oacc[:, 3]).all()
    np.testing.assert_allclose(ga[:, :3], oacc[:, :3], rtol=1e-12, atol=1e-300)


@pytest.mark.parametrize("spp,max_steps", [(1, 1000), (4, 1000), (7, 11)])
def test_until_done_leaves_the_state_of_single_bounces(rg, po, spp, max_steps):
    """render_until_done ends a run at a group's last bounce (or at max_steps); the
    state, counters and sums are those of as many single bounces, and more bounces
    can follow."""
    sm, _, camd = _scene(rg, po, "mixed")
    cam = camera(camd, 48, 40)
    config = rg.render_config(spp=spp, max_depth=6)
    out = []
    for single in (False, True):
        lane = rg.WavefrontLane(0, 5000)
        lane.set_render_trace(True, 12)
        lane.setup(sm)
        lane.initialize(cam, config)
        if single:
            for _ in range(out[0][2]):
                lane.step(1)
            n = out[0][2]
        else:
            n = lane.render_until_done(max_steps)
        lane.synchronize()
        slots, st = lane.debug_slots(), lane.stats()
        acc = lane.accumulation()
        lane.step(3)
        out.append((slots, acc, n, (st.steps, st.paths_started, st.rays_traced, st.active_paths), lane.debug_slots()))
    a, b = out
    for k in a[0]:
        assert (np.asarray(a[0][k]).view(np.uint32) == np.asarray(b[0][k]).view(np.uint32)).all(), k
        assert (np.asarray(a[4][k]).view(np.uint32) == np.asarray(b[4][k]).view(np.uint32)).all(), k
    assert a[3] == b[3]
    assert (a[1][..., 3] == b[1][..., 3]).all()
    np.testing.assert_allclose(a[1], b[1], rtol=1e-12, atol=1e-300)
