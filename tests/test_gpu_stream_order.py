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


def test_line_opacity_after_a_call_that_was_captured(tables):
    """line_opacity waits inside, so a stream under capture refuses it; a first call refused
    that way leaves nothing half made for the next (the 1/n^2 table of the direct wings)."""
    from cuda.bindings import runtime as rt
    from atlas12_b200 import _lib
    from atlas12_b200 import synthe as S
    from atlas12_b200._lib import ptr
    length, n = 3000, 40
    rec = S.make_lte_lines(np.arange(n) * 70 + 50, np.ones(n), np.ones(n, int), np.zeros(n), np.full(n, 1e-7),
                           np.zeros(n), np.zeros(n))
    one = torch.ones((1, 1), dtype=torch.float64, device="cuda")
    dop = torch.full((1, 1), 1e-5, dtype=torch.float64, device="cuda")
    cont = torch.full((1, length), 1e-10, dtype=torch.float32, device="cuda")
    lines = torch.from_numpy(rec.view(np.uint8)).cuda()
    out = torch.zeros((1, length), dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()

    def run(ctx):
        ctx.call("atlasgpu_synthe_line_opacity_dev", ptr(lines), n, length, 1, 500000.0, ptr(cont), ptr(one), ptr(dop), 1,
                 ptr(one), ptr(one), ptr(one), S.MAXPROF, ptr(out))
        ctx.synchronize()
        return out.cpu().numpy()

    plain = _lib.Context(0)
    want = run(plain)
    plain.close()
    assert np.count_nonzero(want) == length
    err, stream = rt.cudaStreamCreateWithFlags(rt.cudaStreamNonBlocking)
    assert err == rt.cudaError_t.cudaSuccess
    ctx = _lib.Context(0)
    ctx.set_stream(int(stream))
    err, = rt.cudaStreamBeginCapture(stream, rt.cudaStreamCaptureMode.cudaStreamCaptureModeRelaxed)
    assert err == rt.cudaError_t.cudaSuccess
    with pytest.raises(_lib.AtlasGPUError):
        run(ctx)
    rt.cudaStreamEndCapture(stream)  # (reports the invalidated capture)
    try:
        run(ctx)  # may report the refusal a second time
    except _lib.AtlasGPUError:
        pass
    got = run(ctx)
    ctx.close()
    rt.cudaStreamDestroy(stream)
    np.testing.assert_allclose(got, want, rtol=1e-6)
