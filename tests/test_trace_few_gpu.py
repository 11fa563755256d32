"""Closest hits of calls at the edges of the kernels' choice: few rays spread over the
warps, the first calls that whole warps take, the first that are sorted; and rays whose
far clip is not a positive number.  All against the oracle, bit for bit."""
import numpy as np
import pytest

from raccoongpurender_gb300 import materials, scenes
from tests.conftest import bits
from tests.helpers import build

pytestmark = pytest.mark.gpu
WARPS = 152 * 5 * 8  # of the closest-hit kernel's grid


def _hits(lane, rays):
    import torch
    soa = [torch.from_numpy(a).cuda() for a in rays.soa()]
    n = len(rays)
    prim = torch.full((n + 1,), -7, dtype=torch.int32, device="cuda")
    t = torch.full((n + 1,), -7.0, dtype=torch.float32, device="cuda")
    ng = torch.full((n + 1, 3), -7.0, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    lane.trace_closest_device([a.data_ptr() for a in soa], n, prim.data_ptr(), t.data_ptr(), ng.data_ptr())
    lane.synchronize()
    assert prim[n] == -7 and t[n] == -7.0 and (ng[n] == -7.0).all()
    return prim[:n].cpu().numpy(), t[:n].cpu().numpy(), ng[:n].cpu().numpy()


@pytest.mark.parametrize("n", [1, 2, 31, 33, WARPS - 1, WARPS, WARPS + 1, 4 * WARPS, 4 * WARPS + 1,
                               8 * WARPS, 8 * WARPS + 1, 65535, 65536, 65537,
                               131071])
def test_counts(rg, po, n):
    mesh = scenes.displaced_icosphere(5, seed=7)
    sm, osc = build(mesh)
    lane = rg.WavefrontLane(0, 1024)
    lane.setup(sm)
    rays = scenes.random_rays(n, (-1.3, -1.3, -1.3), (1.3, 1.3, 1.3), seed=n)
    rays.tmax[::5] = 0.4
    oprim, ot, ong = osc.trace(rays.packed8(), threads=16)
    for reorder in (0, 1):
        lane.set_trace_reorder(reorder)
        prim, t, ng = _hits(lane, rays)
        assert (prim == oprim).all() and (bits(t) == bits(ot)).all()
        assert (ng[prim < 0] == 0).all()
        assert np.allclose(np.linalg.norm(ng[prim >= 0], axis=1), 1.0, atol=1e-5)
    lane.set_trace_reorder(0)
    hp, ht = lane.trace_closest(rays)
    assert (hp == oprim).all() and (bits(ht) == bits(ot)).all()


@pytest.mark.parametrize("tmax", [0.0, -0.0, -1.0, float("nan"), float("inf"), 1e-30, 0.5])
@pytest.mark.parametrize("n", [64, 30000])
def test_far_clip(rg, po, tmax, n):
    """The slab test's single comparison stands in for the reference's three only for a
    far clip >= 0: any other keeps them."""
    mesh = scenes.displaced_icosphere(4, seed=7)
    sm, osc = build(mesh)
    lane = rg.WavefrontLane(0, 1024)
    lane.setup(sm)
    rays = scenes.random_rays(n, (-1.3, -1.3, -1.3), (1.3, 1.3, 1.3), seed=3)
    rays.tmax[::2] = tmax
    rays.d[::16, 0] = 0.0
    oprim, ot, _ = osc.trace(rays.packed8(), threads=16)
    prim, t, _ = _hits(lane, rays)
    assert (prim == oprim).all()
    assert ((bits(t) == bits(ot)) | (np.isnan(t) & np.isnan(ot))).all()


@pytest.mark.parametrize("leaf", [1, 4, 8])
@pytest.mark.parametrize("n", [5, 8 * WARPS, 9 * WARPS])
def test_deep_tree(rg, po, n, leaf):
    """Triangles at distances that double from one to the next, whose boxes the rays pass
    from the smallest on: more pending links than the stack's entries in shared memory, in
    the lanes that go alone (few rays; the last ones of a warp) and in whole warps."""
    k = np.repeat(np.exp2(np.arange(-20, 20, dtype=np.float64)), 3)
    size = k * 0.3
    p = np.stack([k, np.zeros_like(k), np.zeros_like(k)], 1)
    p[0::3, 1:] = np.stack([-size[0::3], -size[0::3]], 1)
    p[1::3, 1:] = np.stack([size[1::3], -size[1::3]], 1)
    p[2::3, 1:] = np.stack([-size[2::3], size[2::3]], 1)
    tris = np.arange(len(p), dtype=np.uint32).reshape(-1, 3)
    mesh = scenes.Mesh(p.astype(np.float32), tris, [materials.lambertian()] * len(tris))
    sm, osc = build(mesh, leaf=leaf)
    lane = rg.WavefrontLane(0, 1024)
    lane.setup(sm)
    rays = scenes.random_rays(n, (-1e-6, -1e-6, -1e-6), (1e-6, 1e-6, 1e-6), seed=n)
    rng = np.random.default_rng(n)
    yz = rng.uniform(-0.2, 0.31, (n, 2))  # with y + z > 0 past every triangle
    d = np.concatenate([np.ones((n, 1)), yz], 1)
    rays.d[:] = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)
    rays.d[::7] *= -1.0
    oprim, ot, _ = osc.trace(rays.packed8(), threads=16)
    assert n < 100 or 0.1 < (oprim >= 0).mean() < 0.9
    prim, t, _ = _hits(lane, rays)
    assert (prim == oprim).all() and (bits(t) == bits(ot)).all()


@pytest.mark.parametrize("refill", [1, 7, 16, 32])
@pytest.mark.parametrize("n", [8 * 152 * 8 + 1, 100001])
def test_host_runs(rg, po, refill, n):
    """Hits written across the link in runs: short runs and whole ones, more open than a warp
    keeps, a last run cut by the end."""
    mesh = scenes.displaced_icosphere(4, seed=7)
    sm, osc = build(mesh)
    lane = rg.WavefrontLane(0, 1024)
    lane.setup(sm)
    lane.set_trace_tuning(refill, 1)  # one block an SM: many refills a warp
    rays = scenes.random_rays(n, (-1.3, -1.3, -1.3), (1.3, 1.3, 1.3), seed=n + refill)
    rays.tmax[::3] = 0.05  # over at once, beside long ones
    oprim, ot, _ = osc.trace(rays.packed8(), threads=16)
    prim, t = lane.trace_closest(rays)
    assert (prim == oprim).all() and (bits(t) == bits(ot)).all()


@pytest.mark.parametrize("n", [(1 << 19) - 1, 1 << 19, (1 << 19) + 33])
@pytest.mark.parametrize("order", ["one octant", "every octant", "by turns"])
def test_octants(rg, po, n, order):
    """Warps that choose their thresholds by their rays' octants, from 2^19 rays on."""
    mesh = scenes.displaced_icosphere(4, seed=7)
    sm, osc = build(mesh)
    lane = rg.WavefrontLane(0, 1024)
    lane.setup(sm)
    rays = scenes.random_rays(n, (-1.3, -1.3, -1.3), (1.3, 1.3, 1.3), seed=n)
    if order != "every octant":
        turn = np.arange(n) % 256 < 128 if order == "by turns" else np.ones(n, bool)
        rays.d[turn] = np.abs(rays.d[turn])
    oprim, ot, _ = osc.trace(rays.packed8(), threads=16)
    prim, t, _ = _hits(lane, rays)
    assert (prim == oprim).all() and (bits(t) == bits(ot)).all()
