"""Large results: pageable arrays (filled by the context's copier
from 8 MB on) against the same calls on page-locked arrays (copied directly),
bit for bit, at sizes below, at and above the chunk, the ring and the limits,
with ragged ends; and with two contexts on two threads at once.
"""
import threading

import numpy as np
import pytest
import torch

from atlas12_b200 import _lib, operators, surrogate, synthetic
from atlas12_b200._lib import ptr

pytestmark = pytest.mark.gpu


def _pinned(a):
    return torch.from_numpy(np.ascontiguousarray(a)).pin_memory().numpy()


def _out(shape, pinned):
    return _pinned(np.full(shape, 7.0)) if pinned else np.full(shape, 7.0)


def _kapp(ctx, numnu, kw, pinned):
    m = surrogate.grey_model(9000.0, 4.0, nrhox=56, ross=surrogate.RossTable(nt=48, np_=48, nwave=300))
    e = surrogate.eos(m["t"], m["p"])
    ws, _ = synthetic.geometric_waveset(9.0, 160000.0, numnu)
    out = [_out((numnu, kw), pinned) for _ in range(3)]
    vec = [np.ascontiguousarray(v) for v in (m["t"], e["xne"], e["rho"], e["nh"] * (1 - e["xh"]) / 2, e["nh"] * e["xh"])]
    ctx.call("atlasgpu_atlas_kapp_hydrogen", numnu, ptr(ws), 56, kw, *[ptr(v) for v in vec], None, None,
             *[ptr(o) for o in out], None)
    return out


@pytest.fixture(scope="module")
def kapp_ctx():
    from atlas12_b200 import atlas
    ctx = _lib.Context(0, _lib.PREC_FP64)
    A = atlas.Atlas(ctx, operators.load())
    A.set_kapp_tables(operators.load())
    yield ctx, A
    ctx.close()


@pytest.mark.parametrize("numnu,kw", [(100, 56), (586, 56), (6241, 56), (6242, 57), (14043, 56), (15001, 99)])
def test_results_of_all_sizes(kapp_ctx, numnu, kw):
    a, b = (_kapp(kapp_ctx[0], numnu, kw, p) for p in (False, True))
    for x, y in zip(a, b):
        assert np.array_equal(x, y)


def test_window_equals_its_three_calls(kapp_ctx):
    """Synthe.run's one call against continuum, line_opacity and spectrum in a row (the
    order of the FP64 atomic sums differs from run to run: 1e-6, as the batch test)."""
    from atlas12_b200 import synthe as S
    case = synthetic.synthe_case(nlines=300, wlbeg=400.0, wlend=401.3, seed=5, nrhox=64,
                                 ross=surrogate.RossTable(nt=48, np_=48, nwave=300))
    syn = S.Synthe(kapp_ctx[0], operators.load())
    _, flux, cflux, op = syn.run(case)
    g, L, atm = S.synthe_grid(case["wlbeg"], case["wlend"], case["resolu"]), case["lines"], case["atm"]
    lines = S.make_lte_lines(syn.bin_lines(L["wlvac"], g), *(L[k] for k in ("cgf", "nelion", "elo", "gamrf", "gamsf",
                                                                          "gamwf")))
    cont = syn.continuum(case["wledge"], case["continall"], g)
    op3 = syn.line_opacity(lines, g, case["resolu"], cont, *(atm[k] for k in ("xnfdop", "dopple", "xne", "txnxn",
                                                                             "hckt")))
    f3, c3 = syn.spectrum(case["wledge"], case["contabs"], case["contscat"], atm["rhox"], atm["hkt"], g, op3)
    assert np.count_nonzero(op3)
    np.testing.assert_allclose(op, op3, rtol=1e-6)
    np.testing.assert_allclose(flux, f3, rtol=1e-6)
    assert np.array_equal(cflux, c3)


def test_two_contexts_on_two_threads(kapp_ctx):
    from atlas12_b200 import atlas
    ref = _kapp(kapp_ctx[0], 8000, 72, True)
    ctxs = [_lib.Context(0, _lib.PREC_FP64) for _ in range(2)]
    for c in ctxs:
        atlas.Atlas(c, operators.load()).set_kapp_tables(operators.load())
    got = [[], []]

    def run(i):
        for _ in range(4):
            got[i].append(_kapp(ctxs[i], 8000, 72, False))

    th = [threading.Thread(target=run, args=(i,)) for i in range(2)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    for c in ctxs:
        c.close()
    for g in got:
        assert len(g) == 4
        for out in g:
            for x, y in zip(out, ref):
                assert np.array_equal(x, y)
