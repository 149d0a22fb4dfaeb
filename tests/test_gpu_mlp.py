"""The warm-start network's device kernels against the CPU restatement
(oracle/mlp_ref.py): forward, loss and gradient (FP32 device vs FP64 oracle,
relative tolerance 1e-4 on the gradient norm and 2e-4 per output), and one
short training run that must lower the loss."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SMALL = (4, 32, 48, 24)


def _data(n, seed):
    rng = np.random.default_rng(seed)
    x = rng.uniform(-1, 1, (n, 4)).astype(np.float32)
    t = np.stack([np.sin(1.3 * x[:, 0] + k * 0.2) * np.cos(x[:, 1] - 0.1 * k) + 0.3 * x[:, 2] * x[:, 3]
                  for k in range(SMALL[3])], axis=1).astype(np.float32)
    return x, t


def test_forward_and_gradient_match_oracle(gpu_ctx):
    from atlas12_b200.warmstart import MLP
    import mlp_ref
    m = MLP(gpu_ctx, shape=SMALL, seed=3)
    p32 = m.params()
    assert p32.size == m.nparam and np.all(np.isfinite(p32)), (p32.size, m.nparam)
    p = p32.astype(np.float64)
    x, t = _data(77, 1)
    y = m.forward(x)
    _, _, yr = mlp_ref.forward(p, x, SMALL)
    assert np.all(np.isfinite(yr)), (np.isfinite(p).all(), np.isfinite(x).all(), mlp_ref.__file__)
    np.testing.assert_allclose(y, yr, rtol=2e-4, atol=2e-5)
    loss, g = m.loss_grad(x, t)
    lr, gr = mlp_ref.loss_grad(p, x, t, SMALL)
    assert abs(loss - lr) <= 1e-4 * lr
    assert np.linalg.norm(g - gr) <= 1e-4 * np.linalg.norm(gr)
    m.close()


def test_training_lowers_loss(gpu_ctx):
    from atlas12_b200.warmstart import MLP
    m = MLP(gpu_ctx, shape=SMALL, seed=5)
    x, t = _data(512, 2)
    l0, _ = m.loss_grad(x, t)
    hist = m.train(x, t, epochs=200, batch=64, lr=3e-3, seed=9)
    l1, _ = m.loss_grad(x, t)
    assert np.all(np.isfinite(hist))
    assert l1 < 0.1 * l0, (l0, l1)
    m.close()


@pytest.mark.parametrize("shape", [(4, 256, 256, 216), (3, 17, 33, 1)])
@pytest.mark.parametrize("n", [1, 15, 16, 17, 64, 129, 2369])
def test_tile_edges(gpu_ctx, shape, n):
    """Sample counts and layer widths around the tile edges, up to where 64x64
    tiles fill the chip.  Sums of at most 2,369 FP32 terms in chunks: relative
    error of a few 1e-6 in norm through three layers, 2e-5 allowed; and the
    same bits when run again."""
    from atlas12_b200.warmstart import MLP
    import mlp_ref
    m = MLP(gpu_ctx, shape=shape, seed=3)
    rng = np.random.default_rng(n)
    x = rng.uniform(-1, 1, (n, shape[0])).astype(np.float32)
    t = rng.normal(size=(n, shape[3])).astype(np.float32)
    p = m.params().astype(np.float64)
    lr, gr = mlp_ref.loss_grad(p, x.astype(np.float64), t.astype(np.float64), shape)
    yr = mlp_ref.forward(p, x.astype(np.float64), shape)[2]
    loss, g = m.loss_grad(x, t)
    y = m.forward(x)
    assert abs(loss - lr) <= 2e-5 * lr
    assert np.linalg.norm(y - yr) <= 2e-5 * np.linalg.norm(yr)
    assert np.linalg.norm(g - gr) <= 2e-5 * np.linalg.norm(gr)
    loss2, g2 = m.loss_grad(x, t)
    assert loss2 == loss and np.array_equal(g, g2)
    m.close()
