"""Runs of a guided render whose guide is frozen (no logic pass between the bounces, the
inference over hits as the cast left them) against as many single bounces: the state, the
counters and the sums are the same."""
import numpy as np
import pytest

from raccoongpurender_gb300 import scenes
from tests.helpers import build, camera

pytestmark = pytest.mark.gpu


def _spheres(rg):
    mesh = scenes.cornell_box()
    sm = rg.SceneManager()
    sm.addMesh(mesh)
    from raccoongpurender_gb300 import materials
    sm.addSpheres(np.array([[0.0, 1.5, 0.0, 0.3], [-0.5, 1.4, 0.4, 0.2]], np.float32),
                  [materials.lambertian(r=(0.5, 0.7, 0.6)), materials.ward(alpha=0.2)])
    sm.buildBVH()
    return sm, scenes.cornell_camera()


@pytest.mark.parametrize("scene,npaths,steps,guide_cfg,cfg", [
    ("mixed", 12289, 9, dict(guide_volumes=1), {}),                       # in-volume vertices are guided too
    ("mixed", 5000, 12, dict(max_depth=2), dict(rr_depth=2)),             # selected rows
    ("spheres", 4097, 7, dict(guide_volumes=0), dict(dof=0.0)),
    ("mixed", 8192, 0, dict(train_interval=3), dict(spp=3, max_depth=6)),  # until done
])
def test_run_equals_single_bounces(rg, po, scene, npaths, steps, guide_cfg, cfg):
    if scene == "mixed":
        mesh, env, camd = scenes.mixed_scene(level=3, seed=3)
        sm, _ = build(mesh, env=env)
    else:
        sm, camd = _spheres(rg)
    cam = camera(camd, 40, 36)
    W, b = rg.Guide(0).weights()
    W *= 1.5  # the initial ones, with more contrast
    out = []
    for single in (False, True):
        g = rg.Guide(0, train=0, **guide_cfg)
        g.set_weights(W, b)
        lane = rg.WavefrontLane(0, npaths)
        lane.set_render_trace(True, 12)
        lane.setup(sm)
        lane.set_guide(g)
        lane.initialize(cam, rg.render_config(seed_offset=11, **cfg))
        if single:
            for _ in range(out[0][2]):
                lane.step(1)
            n = out[0][2]
        elif steps:
            lane.step(steps)
            n = steps
        else:
            n = lane.render_until_done()
        lane.synchronize()
        g.check()
        st = lane.stats()
        out.append((lane.debug_slots(), lane.accumulation(), n, (st.steps, st.paths_started, st.rays_traced,
                                                                  st.active_paths), g.stats()["iterations"]))
    a, b2 = out
    for k in a[0]:
        assert (np.asarray(a[0][k]).view(np.uint32) == np.asarray(b2[0][k]).view(np.uint32)).all(), k
    assert a[3] == b2[3] and a[4] == b2[4]
    assert (a[1][..., 3] == b2[1][..., 3]).all()
    np.testing.assert_allclose(a[1], b2[1], rtol=1e-12, atol=1e-300)
