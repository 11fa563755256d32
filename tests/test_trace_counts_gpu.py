"""Node and primitive counts of a call of few rays (spread over the warps, lane by lane) against
the same rays' in a large call (whole warps): a ray's walk does not depend on its company."""
import numpy as np
import pytest

from raccoongpurender_gb300 import scenes
from tests.conftest import bits
from tests.helpers import build

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 33, 1000, 30000])
def test_counts_of_few(rg, po, n):
    import torch
    sm, osc = build(scenes.displaced_icosphere(5, seed=7))
    lane = rg.WavefrontLane(0, 1024)
    lane.setup(sm)
    rays = scenes.random_rays(200_000, (-1.3, -1.3, -1.3), (1.3, 1.3, 1.3), seed=n)
    soa = [torch.from_numpy(a).cuda() for a in rays.soa()]
    out = []
    for m in (n, len(rays)):
        prim, nodes, prims = (torch.full((m,), -7, dtype=torch.int32, device="cuda") for _ in range(3))
        t = torch.full((m,), -7.0, device="cuda")
        torch.cuda.synchronize()
        lane.trace_closest_counts_device([a.data_ptr() for a in soa], m, prim.data_ptr(), t.data_ptr(),
                                         nodes.data_ptr(), prims.data_ptr())
        lane.synchronize()
        out.append([a[:n].cpu().numpy() for a in (prim, nodes, prims)] + [bits(t[:n].cpu().numpy())])
    for few, many in zip(*out):
        assert (few == many).all()
    oprim, ot, _ = osc.trace(rays.packed8()[:n], threads=16)
    assert (out[0][0] == oprim).all() and (out[0][3] == bits(ot)).all()
    assert (out[0][1] >= 0).all() and out[0][1].max() > 3
