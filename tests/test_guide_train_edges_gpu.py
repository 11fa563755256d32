"""The tcgen05 training iteration at the edges of its tiles (128 samples, two groups
per CTA, one CTA per SM) against the float64 oracle, and its update kernel: the
gradients of a call with the Adam step are those of a call without it, wherever the
caller's gradient buffer starts."""
import numpy as np
import pytest

from oracle import guide_oracle as go

pytestmark = pytest.mark.gpu
LO, HI, IE = (-1.0, -1.0, -1.0), (1.0, 1.0, 1.0), (0.5, 0.5, 0.5)


@pytest.mark.parametrize("n", [1, 31, 128, 129, 256, 257, 152 * 256 + 1])
def test_edges(rg, n):
    import torch
    W, b = go.init_weights(5)
    s = go.random_samples(n, seed=20 + n)
    dev = torch.from_numpy(s).cuda()
    buf = torch.full((rg.Guide.N_PARAMS + 2,), 7.0, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    out = []
    for step in (False, True):
        g = rg.Guide(0)
        g.set_weights(W, b)
        g.set_bounds(LO, HI)
        loss = g.train_device(dev.data_ptr(), n, weight_scale=1.0 / n, apply_adam=step, grads_ptr=buf.data_ptr() + 4)
        g.check()
        assert g.stats()["iterations"] == int(step)
        if step:
            assert g.loss_history()[0] == np.float32(loss)
        out.append((loss, buf.cpu().numpy().copy(), g.weights()))
    # the bytes around the buffer are not written, and the step moves the weights only
    for o in out:
        assert o[1][0] == 7.0 and o[1][-1] == 7.0
    assert (out[0][2][0] == W.astype(np.float32)).all() and not (out[1][2][0] == W.astype(np.float32)).all()
    # the two groups' tiles reach the shared accumulators in either order: FP32 rounding
    np.testing.assert_allclose(out[1][1], out[0][1], rtol=0, atol=1e-5 * np.abs(out[0][1][1:-1]).max())
    grads = out[0][1][1:-1]
    rloss, rdW, rdb = go.gradients(W, b, s, LO, IE, weight_scale=1.0 / n, bf16_round=True)
    # as in test_guide_gpu: FP32 accumulation and transcendentals, bf16 boundaries
    assert abs(out[0][0] - rloss) <= 1e-3 * abs(rloss) + 1e-6
    dW = grads[:go.LAYERS * 64 * 64].reshape(go.LAYERS, 64, 64)
    db = grads[go.LAYERS * 64 * 64:].reshape(go.LAYERS, 64)
    for l in range(go.LAYERS):
        assert np.linalg.norm(dW[l] - rdW[l]) <= 1e-2 * np.linalg.norm(rdW[l])
        assert np.linalg.norm(db[l] - rdb[l]) <= 1e-2 * np.linalg.norm(rdb[l])
