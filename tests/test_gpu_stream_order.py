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


class Spectrum:
    """synthe_spectrum_dev on device inputs of one case, with outputs of their own."""

    def __init__(self, width, seed):
        from atlas12_b200 import surrogate, synthetic
        from atlas12_b200 import synthe as S
        c = synthetic.synthe_case(nlines=1, wlbeg=400.0, wlend=400.0 + width, seed=seed, nrhox=48,
                                  ross=surrogate.RossTable(nt=48, np_=48, nwave=300))
        self.grid = S.synthe_grid(c["wlbeg"], c["wlend"], c["resolu"])
        rng = np.random.default_rng(seed)
        op = 10.0 ** rng.uniform(-6.0, 1.0, (48, self.grid["length"]))
        self.v = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (
            c["wledge"], c["contabs"], c["contscat"], c["atm"]["rhox"], c["atm"]["hkt"], op.astype(np.float32))]
        self.out = [torch.zeros(self.grid["length"], dtype=torch.float64, device="cuda") for _ in range(2)]
        torch.cuda.synchronize()

    def call(self, ctx):
        from atlas12_b200._lib import ptr
        we, ca, cs, rx, hk, op = self.v
        g = self.grid
        ctx.call("atlasgpu_synthe_spectrum_dev", ptr(we), we.numel(), ptr(ca), ptr(cs), ca.shape[1], 48, ptr(rx), ptr(hk),
                 g["wbegin"], g["ratio"], g["length"], ptr(op), *[ptr(o) for o in self.out])

    def result(self):
        r = np.stack([o.cpu().numpy() for o in self.out])
        for o in self.out:
            o.zero_()
        torch.cuda.synchronize()
        return r

    def plain(self, tables):
        ctx = spectrum_context(tables)
        self.call(ctx)
        ctx.close()
        return self.result()


def spectrum_context(tables):
    from atlas12_b200 import _lib
    ctx = _lib.Context(0)
    ctx.set_operators(tables["xtau8"], tables["coefj"], tables["coefh"], tables["ch_j"], tables["ck_j"])
    return ctx


@pytest.mark.parametrize("before", [False, True])
def test_spectrum_captured(tables, before):
    """spectrum_dev launches kernels only, so it can be captured, also as a context's first
    call, and the graph goes on giving the same bits after longer calls of the context."""
    from cuda.bindings import runtime as rt
    a, b = Spectrum(1.0, 1), Spectrum(30.0, 2)  # one round, and two of 32,768 wavelengths
    want_a, want_b = a.plain(tables), b.plain(tables)
    assert np.all(want_a > 0.0) and np.all(want_b > 0.0)
    _, stream = rt.cudaStreamCreateWithFlags(rt.cudaStreamNonBlocking)
    ctx = spectrum_context(tables)
    ctx.synchronize()
    ctx.set_stream(int(stream))
    if before:
        a.call(ctx)
        ctx.synchronize()
        assert np.array_equal(a.result(), want_a)
    err, = rt.cudaStreamBeginCapture(stream, rt.cudaStreamCaptureMode.cudaStreamCaptureModeGlobal)
    assert err == rt.cudaError_t.cudaSuccess
    a.call(ctx)
    err, graph = rt.cudaStreamEndCapture(stream)
    assert err == rt.cudaError_t.cudaSuccess
    err, run = rt.cudaGraphInstantiate(graph, 0)
    assert err == rt.cudaError_t.cudaSuccess
    for _ in range(3):
        b.call(ctx)
        assert rt.cudaGraphLaunch(run, stream)[0] == rt.cudaError_t.cudaSuccess
        b.call(ctx)
        ctx.synchronize()
        assert np.array_equal(a.result(), want_a)
        assert np.array_equal(b.result(), want_b)
    rt.cudaGraphExecDestroy(run)
    rt.cudaGraphDestroy(graph)
    ctx.close()
    rt.cudaStreamDestroy(stream)


def test_spectra_of_one_context_on_two_streams(tables):
    """The stream changed between calls that nothing waits for: each has its own result."""
    from cuda.bindings import runtime as rt
    a, b = Spectrum(12.0, 3), Spectrum(25.0, 4)
    want_a, want_b = a.plain(tables), b.plain(tables)
    streams = [rt.cudaStreamCreateWithFlags(rt.cudaStreamNonBlocking)[1] for _ in range(2)]
    ctx = spectrum_context(tables)
    ctx.synchronize()
    for _ in range(5):
        for x, s in ((a, 0), (b, 1), (a, 0), (b, 1)):
            ctx.set_stream(int(streams[s]))
            x.call(ctx)
        torch.cuda.synchronize()
        assert np.array_equal(a.result(), want_a)
        assert np.array_equal(b.result(), want_b)
    ctx.close()
    for s in streams:
        rt.cudaStreamDestroy(s)
