"""State that a call sets up on the context's stream: in place for the next call
whatever other streams are doing.
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_new_network_while_the_default_stream_is_busy(gpu_ctx):
    """Weights, Adam moments and the loss counter of a new network are set on the stream
    that reads them: loss, gradient and a short training run are the same bits however
    much work waits on the default stream."""
    from atlas12_b200.warmstart import MLP
    rng = np.random.default_rng(1)
    x = rng.uniform(-1, 1, (64, 4)).astype(np.float32)
    t = rng.normal(size=(64, 24)).astype(np.float32)
    a = torch.ones((4096, 4096), device="cuda")
    torch.cuda.synchronize()
    got = []
    for busy in (False, True, True, True):
        for _ in range(20 if busy else 0):
            a = a @ a * 1e-4
        m = MLP(gpu_ctx, shape=(4, 32, 48, 24), seed=3)
        loss, g = m.loss_grad(x, t)
        hist = m.train(x, t, epochs=3, batch=16, lr=1e-3, seed=5)
        got.append((loss, g, hist, m.params()))
        m.close()
    torch.cuda.synchronize()
    for other in got[1:]:
        assert other[0] == got[0][0]
        for p, q in zip(other[1:], got[0][1:]):
            assert np.array_equal(p, q)
