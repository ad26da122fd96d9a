"""The fused training step (csrc/mlp_train.cu) where its blocks and the gradient's layout have edges:
the rows each step draws, prepared while the previous update runs; the update of every parameter; and
the next step's weights."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _philox_x(row, step, seed):
    """First word of Philox4x32-10 on (row, step, 0, "tran"), the key the seed's two halves."""
    m = np.uint64(0xFFFFFFFF)
    c = [row.astype(np.uint64), np.full_like(row, step, np.uint64), np.zeros_like(row, np.uint64),
         np.full_like(row, 0x7472616E, np.uint64)]
    k = [np.uint64(seed & 0xFFFFFFFF), np.uint64(seed >> 32)]
    for _ in range(10):
        a, b = c[0] * np.uint64(0xD2511F53), c[2] * np.uint64(0xCD9E8D57)
        c = [(b >> np.uint64(32)) ^ c[1] ^ k[0], b & m, (a >> np.uint64(32)) ^ c[3] ^ k[1], a & m]
        k = [(k[0] + np.uint64(0x9E3779B9)) & m, (k[1] + np.uint64(0xBB67AE85)) & m]
    return c[0]


def _fused_gradient(engine, torch, mlp, x, t):
    g = torch.full((mlp.n_params,), float("nan"), device="cuda")
    loss = torch.zeros(1, device="cuda")
    engine.check(engine.load().wob_mlp_gradient_fused(mlp._h, x.data_ptr(), t.data_ptr(), x.shape[0], g.data_ptr(),
                                                     loss.data_ptr(), None))
    torch.cuda.synchronize()
    return g.cpu().numpy(), float(loss.item())


@pytest.mark.parametrize("out_dim,batch", [(1, 1), (1, 1000), (15, 64), (16, 65), (17, 63), (64, 8300)])
def test_steps_draw_and_update_what_they_should(engine, cuda, out_dim, batch):
    torch = cuda
    from wobtoolbox_gb300 import cv
    n, seed, lr, steps = 5003, (9 << 32) | 5, 1e-2, 35
    gen = torch.Generator().manual_seed(out_dim)
    x, t = torch.randn(n, 6, generator=gen).cuda(), torch.randn(n, out_dim, generator=gen).cuda()

    def rows(step):
        h = _philox_x(np.arange(batch, dtype=np.uint64), step, seed)
        i = torch.from_numpy(((h * np.uint64(n)) >> np.uint64(32)).astype(np.int64)).cuda()
        return x[i].contiguous(), t[i].contiguous()

    # weights that a vanishing rate leaves alone: each step's loss is its own batch's, bit for bit
    mlp = cv.MLP(32, 4, out_dim, 1.0, 4)
    p0 = mlp.params()[0]
    p0[p0 == 0.0] = 0.01
    mlp.set_params(p0)
    grad, _ = _fused_gradient(engine, torch, mlp, *rows(0))
    want = [_fused_gradient(engine, torch, mlp, *rows(s))[1] for s in range(steps)]
    hist = torch.zeros(steps, device="cuda")
    mlp.train(x, t, n, steps, batch, 1e-30, seed=seed, loss_history=hist)
    assert np.array_equal(mlp.params()[0], p0)
    assert hist.tolist() == want
    mlp.close()

    # the first update divides the gradient by its own magnitude; 1 - 0.999 in FP32 is off by up to 6e-5
    one, two = cv.MLP(32, 4, out_dim, 1.0, 4), cv.MLP(32, 4, out_dim, 1.0, 4)
    one.set_params(p0)
    two.set_params(p0)
    one.train(x, t, n, 1, batch, lr, seed=seed)
    p1 = one.params()[0]
    g64 = grad.astype(np.float64)
    expect = p0 - lr * g64 / (np.abs(g64) + 1e-8)
    assert np.max(np.abs(p1 - expect)) < 1e-4 * lr + 2e-7 * np.max(np.abs(p0))
    # and the second step runs on the weights the first one left
    hist = torch.zeros(2, device="cuda")
    two.train(x, t, n, 2, batch, lr, seed=seed, loss_history=hist)
    assert float(hist[1].item()) == _fused_gradient(engine, torch, one, *rows(1))[1]
    one.close()
    two.close()
