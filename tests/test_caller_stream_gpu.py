"""Calls that start as dependent launches, on a caller's stream between the caller's own
kernels: their inputs come from a kernel just before, and the next one overwrites inputs and
reads results, without a wait on the host; and the same in a captured graph."""
import numpy as np
import pytest

from oracle import guide_oracle as go
from raccoongpurender_gb300 import scenes
from tests.helpers import build

pytestmark = pytest.mark.gpu
ROUNDS = 12


class _Hits:
    """n rays against one mesh; few are spread over the warps, more go in rounds."""

    def __init__(self, rg, n):
        import torch
        sm, osc = build(scenes.displaced_icosphere(4, seed=7))
        self.lane = rg.WavefrontLane(0, 1024)
        self.lane.setup(sm)
        self.n, self.src, self.want = n, [], []
        for k in range(2):
            rays = scenes.random_rays(n, (-1.3, -1.3, -1.3), (1.3, 1.3, 1.3), seed=50 + k)
            self.src.append([torch.from_numpy(a).cuda() for a in rays.soa()])
            prim, t, _ = osc.trace(rays.packed8(), threads=16)
            self.want.append((torch.from_numpy(prim).cuda(), torch.from_numpy(t).cuda()))
        self.inputs = [torch.empty(n, device="cuda") for _ in range(7)]
        self.outputs = [torch.empty(n, dtype=torch.int32, device="cuda"), torch.empty(n, device="cuda")]

    def call(self, stream):
        self.lane.trace_closest_device([a.data_ptr() for a in self.inputs], self.n, self.outputs[0].data_ptr(),
                                       self.outputs[1].data_ptr(), 0, stream)


class _Rows:
    """The guiding network over n rows."""

    def __init__(self, rg, n):
        import torch
        W, b = go.init_weights(4)
        self.guide = rg.Guide(0)
        self.guide.set_weights(W, b)
        self.guide.set_bounds((-1, -1, -1), (1, 1, 1))
        self.n, self.src, self.want = n, [], []
        self.inputs = [torch.empty((n, 16), device="cuda")]
        self.outputs = [torch.empty((n, go.ROW_OUTPUTS), device="cuda")]
        for k in range(2):
            self.src.append([torch.from_numpy(go.random_samples(n, seed=60 + k)).cuda()])
            self.inputs[0].copy_(self.src[k][0])
            torch.cuda.synchronize()
            self.guide.infer_device(self.inputs[0].data_ptr(), n, self.outputs[0].data_ptr())
            torch.cuda.synchronize()
            self.want.append((self.outputs[0].clone(),))  # a row's result depends on the row alone

    def call(self, stream):
        self.guide.infer_device(self.inputs[0].data_ptr(), self.n, self.outputs[0].data_ptr(), stream)


KINDS = [(_Hits, 1000), (_Hits, 200000), (_Rows, 300), (_Rows, 100000)]


def _same(got, want):
    return all((g.cpu().numpy().view(np.uint32) == w.cpu().numpy().view(np.uint32)).all() for g, w in zip(got, want))


@pytest.mark.parametrize("kind,n", KINDS)
def test_between_the_callers_kernels(rg, po, kind, n):
    import torch
    w = kind(rg, n)
    st = torch.cuda.Stream()
    torch.cuda.synchronize()
    got = []
    with torch.cuda.stream(st):
        for r in range(ROUNDS):
            torch.cuda._sleep(200_000)  # the inputs are late
            for dst, src in zip(w.inputs, w.src[r % 2]):
                torch.mul(src, 1.0, out=dst)
            w.call(st.cuda_stream)
            got.append([torch.mul(o, 1) for o in w.outputs])
            for dst in w.inputs + w.outputs:
                dst.fill_(7)
    torch.cuda.synchronize()
    for r in range(ROUNDS):
        assert _same(got[r], w.want[r % 2]), r


@pytest.mark.parametrize("kind,n", KINDS)
def test_in_a_captured_graph(rg, po, kind, n):
    import torch
    w = kind(rg, n)
    stage = [torch.empty_like(a) for a in w.inputs]
    result = [torch.empty_like(a) for a in w.outputs]
    st = torch.cuda.Stream()
    for a in w.inputs:
        a.zero_()
    torch.cuda.synchronize()
    w.call(st.cuda_stream)  # the first call allocates its scratch
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=st):
        for dst, src in zip(w.inputs, stage):
            torch.mul(src, 1.0, out=dst)
        w.call(st.cuda_stream)
        for dst, src in zip(result, w.outputs):
            torch.mul(src, 1, out=dst)
        for dst in w.inputs + w.outputs:
            dst.fill_(7)
    for r in range(4):
        for dst, src in zip(stage, w.src[r % 2]):
            dst.copy_(src)
        torch.cuda.synchronize()
        g.replay()
        torch.cuda.synchronize()
        assert _same(result, w.want[r % 2]), r
