"""The tcgen05 inference kernel at the edges of its warps (32 rows a bulk copy), tiles
(128 rows), CTAs (five tiles) and grid (152 CTAs, then a second tile each) against the
float64 oracle; nothing is written past the last row."""
import numpy as np
import pytest

from oracle import guide_oracle as go

pytestmark = pytest.mark.gpu
LO, HI, IE = (-1.0, -1.0, -1.0), (1.0, 1.0, 1.0), (0.5, 0.5, 0.5)


@pytest.mark.parametrize("n", [1, 31, 32, 33, 127, 129, 640, 641, 152 * 640 + 1, 200003])
def test_edges(rg, n):
    import torch
    W, b = go.init_weights(4)
    s = go.random_samples(n, seed=n)
    g = rg.Guide(0)
    g.set_weights(W, b)
    g.set_bounds(LO, HI)
    rows = torch.from_numpy(s).cuda()
    out = torch.full((n + 40, go.ROW_OUTPUTS), 7.0, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    g.infer_device(rows.data_ptr(), n, out.data_ptr())
    torch.cuda.synchronize()
    g.check()
    got = out.cpu().numpy()
    assert (got[n:] == 7.0).all() and not got[:n, go.NET_OUTPUTS:].any()
    # the oracle makes every bf16 rounding of the kernel's; what remains is FP32 accumulation
    # order and a value on a rounding boundary now and then: 1 % as in test_guide_gpu,
    # over all rows and over the last tile's
    ref, _ = go.forward(W, b, go.encode(s[:, 0:9], LO, IE), bf16_round=True)
    for part in (slice(0, n), slice(max(0, n - 128), n)):
        d, r = got[part, :go.NET_OUTPUTS] - ref[part], ref[part]
        assert np.linalg.norm(d) <= 1e-2 * np.linalg.norm(r)
