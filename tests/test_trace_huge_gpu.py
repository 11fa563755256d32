"""Closest hits where the triangle test overflows: its determinant is infinite or its products are
NaN, a hit at a distance that is not a number is taken, as the reference takes it, and every
box test after that compares with it.  Against the oracle, bit for bit (a NaN is a NaN)."""
import numpy as np
import pytest

from raccoongpurender_gb300 import scenes
from tests.conftest import bits
from tests.helpers import build

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scene,origin,direction", [
    (1e8, 1e8, 1.0), (1e10, 1e10, 1.0), (1e15, 1e15, 1.0),
    (1e18, 1e18, 1.0), (5e18, 5e18, 1.0), (1e19, 1e19, 1.0), (1e21, 1e21, 1.0), (1e29, 1e29, 1.0),
    (1.0, 1.0, 1e8), (1.0, 1.0, 1e15), (1.0, 1.0, 1e37), (1e10, 1e10, 1e20),
    (1.0, 1e25, 1.0), (1e13, 1e29, 1.0),
])
@pytest.mark.parametrize("n", [2000, 150000])
def test_overflow(rg, po, scene, origin, direction, n):
    mesh = scenes.displaced_icosphere(3, seed=7)
    mesh.points[:] = (mesh.points.astype(np.float64) * scene).astype(np.float32)
    sm, osc = build(mesh)
    lane = rg.WavefrontLane(0, 1024)
    lane.setup(sm)
    rays = scenes.random_rays(n, (-1.3, -1.3, -1.3), (1.3, 1.3, 1.3), seed=3)
    rays.o[:] = (rays.o.astype(np.float64) * origin).astype(np.float32)
    rays.d[:] = (rays.d.astype(np.float64) * direction).astype(np.float32)
    if origin > scene:  # head for the mesh
        rays.d[:] = -rays.o / np.abs(rays.o).max(1, keepdims=True)
    rays.tmax[:] = np.float32(3.0e38)
    oprim, ot, _ = osc.trace(rays.packed8(), threads=16)
    import torch
    soa = [torch.from_numpy(a).cuda() for a in rays.soa()]
    prim = torch.empty(n, dtype=torch.int32, device="cuda")
    t = torch.empty(n, device="cuda")
    torch.cuda.synchronize()
    lane.trace_closest_device([a.data_ptr() for a in soa], n, prim.data_ptr(), t.data_ptr(), 0)
    lane.synchronize()
    for gp, gt in ((prim.cpu().numpy(), t.cpu().numpy()), lane.trace_closest(rays)):
        assert (gp == oprim).all()
        assert ((bits(gt) == bits(ot)) | (np.isnan(gt) & np.isnan(ot))).all()
