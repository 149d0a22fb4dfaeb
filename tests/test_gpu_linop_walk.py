"""LINOP1's wing walks where they can go wrong: depth counts around
the coarse gates' groups (lines gated several at a time) and the warp width,
line counts around a chunk, lines at both ends of the grid, wings that run to
their limit of 100 points, and values over the whole range of the
fixed-point words, against the CPU oracle.

Tolerances as the LINOP1 test: FP64 1e-9 per element, mixed precision 1e-6, and
the same nonzero pattern.
"""
import numpy as np
import pytest

from atlas12_b200 import _lib, atlas, surrogate, synthetic

pytestmark = pytest.mark.gpu
NSPEC = 270


@pytest.fixture(scope="module")
def ross():
    return surrogate.RossTable(nt=48, np_=48, nwave=300)


@pytest.fixture(scope="module")
def h_tables(po, tables):
    return po.tabvoigt(tables["tabvi"], tables["tabh1"])


def case(ross, nrhox, numnu, nlines, seed, strength=1.0):
    m = surrogate.grey_model(5000.0, 3.0, nrhox=nrhox, ross=ross)
    pop = surrogate.populations(m["t"], m["p"], 1.5)
    d = pop["dopple"][:, :NSPEC]
    xnfdop = np.where(d > 0, pop["xnfp"][:, :NSPEC] / np.maximum(d, 1e-300) / pop["rho"][:, None], 0.0).T * strength
    dopple = np.where(d > 0, d, 1.0).T
    hkt = surrogate.HPLANCK / (surrogate.KBOL * m["t"])
    ws, _ = synthetic.geometric_waveset(200.0, 2000.0, numnu)
    cut = atlas.cutoff_grid()
    ka, sg = surrogate.continuum_opacity(cut, m["t"], m["p"], pop)
    tab = (ka + sg) * atlas.LINE_CUTOFF / (1.0 - np.exp(-(surrogate.CLIGHT_NMS / cut)[:, None] * hkt[None, :]))
    txnxn = (pop["nh"] * (1 - pop["xh"]) + 0.42 * 0.085 * pop["nh"]) * (m["t"] / 1e4) ** 0.3
    return dict(xnfdop=np.ascontiguousarray(xnfdop), dopple=np.ascontiguousarray(dopple), xne=pop["xne"], txnxn=txnxn,
                hckt=hkt * surrogate.CLIGHT, ws=ws, tabcont=np.vstack([tab, tab[-1:]]), iw=atlas.iwavetab(cut),
                # lines reach a little past both ends of the grid
                lines=synthetic.atlas_lines(nlines, ws[0] * 0.999, ws[-1] * 1.001, seed=seed))


@pytest.mark.parametrize("prec,tol", [(_lib.PREC_FP64, 1e-9), (_lib.PREC_MIXED, 1e-6)])
@pytest.mark.parametrize("nrhox,numnu,nlines,strength", [(16, 50, 1, 1.0), (16, 300, 33, 1e4), (31, 101, 64, 1e4),
                                                         (33, 102, 65, 1.0), (63, 400, 500, 1e6), (72, 2000, 3000, 1e2),
                                                         (96, 500, 257, 1e8), (100, 777, 1000, 1.0)])
def test_linop_walks(po, gpu_ctx, tables, h_tables, ross, nrhox, numnu, nlines, strength, prec, tol):
    c = case(ross, nrhox, numnu, nlines, seed=nrhox, strength=strength)
    atm = dict(xnfdop=c["xnfdop"], dopple=c["dopple"], xne=c["xne"], txnxn=c["txnxn"], hckt=c["hckt"])
    ref, used = po.atlas_linop1(*h_tables, po.build_tablog(), c["lines"], atm, c["tabcont"], c["iw"], c["ws"])
    A = atlas.Atlas(gpu_ctx, tables, *h_tables)
    gpu_ctx.set_precision(prec)
    try:
        got, n = A.linop1(c["lines"], nrhox, c["xnfdop"], c["dopple"], c["xne"], c["txnxn"], c["hckt"], c["tabcont"],
                          c["iw"], c["ws"])
    finally:
        gpu_ctx.set_precision(_lib.PREC_MIXED)
    assert n == used
    np.testing.assert_array_equal(got != 0, ref != 0)
    assert np.max(np.abs(got - ref) / np.maximum(np.abs(ref), 1e-300), initial=0.0) < tol


@pytest.mark.parametrize("prec", [_lib.PREC_FP64, _lib.PREC_MIXED])
@pytest.mark.parametrize("past", [0.004, 0.3, 0.9])
def test_line_past_the_last_wavelength(gpu_ctx, tables, h_tables, ross, past, prec):
    """A line less than 1 nm past the last wavelength adds there at the distance V, as
    on a grid with one more wavelength beyond it (its profile table has no
    negative side).  The same additions in both: equal to rounding."""
    c = case(ross, 72, 60, 1, seed=1, strength=1e8)
    iwl = int(round(np.log(c["ws"][-1] + past) / np.log(1.0 + 1.0 / 2000000.0)))
    lines = c["lines"][:1].copy()
    lines[0, 0] = iwl
    A = atlas.Atlas(gpu_ctx, tables, *h_tables)
    gpu_ctx.set_precision(prec)
    try:
        a, b = (A.linop1(lines, 72, c["xnfdop"], c["dopple"], c["xne"], c["txnxn"], c["hckt"], c["tabcont"], c["iw"],
                         ws)[0] for ws in (c["ws"], np.append(c["ws"], c["ws"][-1] + 5.0)))
    finally:
        gpu_ctx.set_precision(_lib.PREC_MIXED)
    assert np.all(np.isfinite(a)) and np.count_nonzero(a[-1]) > 30 and a.min() >= 0.0
    np.testing.assert_allclose(a[-1], b[-2], rtol=1e-9)


@pytest.mark.parametrize("prec,tol", [(_lib.PREC_FP64, 1e-9), (_lib.PREC_MIXED, 1e-6)])
@pytest.mark.parametrize("nrhox,nlines", [(72, 131072), (40, 131073)])
def test_both_sides_of_the_split(po, gpu_ctx, tables, h_tables, ross, nrhox, nlines, prec, tol):
    """The most lines whose rounds of 32 depths go to warps of their own, and one more.
    (Lines past the last wavelength, whose table index is negative in the oracle, moved inside.)"""
    c = case(ross, nrhox, 400, nlines, seed=nrhox)
    lines = c["lines"].copy()
    lines[:, 0] = np.minimum(lines[:, 0], int(np.log(c["ws"][-1]) / np.log(1.0 + 1.0 / 2000000.0)) - 1)
    atm = dict(xnfdop=c["xnfdop"], dopple=c["dopple"], xne=c["xne"], txnxn=c["txnxn"], hckt=c["hckt"])
    ref, used = po.atlas_linop1(*h_tables, po.build_tablog(), lines, atm, c["tabcont"], c["iw"], c["ws"])
    assert np.all(np.isfinite(ref))
    A = atlas.Atlas(gpu_ctx, tables, *h_tables)
    gpu_ctx.set_precision(prec)
    try:
        got, n = A.linop1(lines, nrhox, c["xnfdop"], c["dopple"], c["xne"], c["txnxn"], c["hckt"], c["tabcont"],
                          c["iw"], c["ws"])
    finally:
        gpu_ctx.set_precision(_lib.PREC_MIXED)
    assert n == used
    np.testing.assert_array_equal(got != 0, ref != 0)
    assert np.max(np.abs(got - ref) / np.maximum(np.abs(ref), 1e-300), initial=0.0) < tol
