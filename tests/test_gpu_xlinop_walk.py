"""XLINOP's walk where it can go wrong: depth counts around the 32 depths of a round, one
warp per record and one per round, wings that end before, at and after the hand-over to
the whole warp with any number of lanes left, up to their limit of 2000 points, and both
ends of the grid, against the CPU oracle.

Tolerances as the XLINOP parity test: FP64 1e-9 per element, mixed precision 1e-6, and the
same nonzero pattern.
"""
import numpy as np
import pytest

from atlas12_b200 import _lib, atlas, surrogate, synthetic

NSPEC = 270


@pytest.fixture(scope="module")
def ross():
    return surrogate.RossTable(nt=48, np_=48, nwave=300)


@pytest.fixture(scope="module")
def h_tables(po, tables):
    return po.tabvoigt(tables["tabvi"], tables["tabh1"])


def case(ross, nrhox, numnu, n, teff, gf):
    m = surrogate.grey_model(teff, 4.0, nrhox=nrhox, ross=ross)
    pop = surrogate.populations(m["t"], m["p"], 1.5)
    d = pop["dopple"][:, :NSPEC]
    xnfdop = np.where(d > 0, pop["xnfp"][:, :NSPEC] / np.maximum(d, 1e-300) / pop["rho"][:, None], 0.0).T
    hkt = surrogate.HPLANCK / (surrogate.KBOL * m["t"])
    cut = atlas.cutoff_grid()
    ka, sg = surrogate.continuum_opacity(cut, m["t"], m["p"], pop)
    tab = (ka + sg) * atlas.LINE_CUTOFF / (1.0 - np.exp(-(surrogate.CLIGHT_NMS / cut)[:, None] * hkt[None, :]))
    ws = np.geomspace(300.0, 600.0, numnu)
    recs = synthetic.nlte_records(n, 299.8, 600.2, seed=nrhox + n, strong=0.2)
    rng = np.random.default_rng(nrhox)
    recs["gf"] *= 10.0 ** rng.uniform(gf - 6.0, gf, n)  # of every strength up to gf
    return dict(xnfdop=np.ascontiguousarray(xnfdop), dopple=np.ascontiguousarray(np.where(d > 0, d, 1.0).T),
                xne=pop["xne"], txnxn=(pop["nh"] * (1 - pop["xh"]) + 0.42 * 0.085 * pop["nh"]) * (m["t"] / 1e4) ** 0.3,
                hckt=hkt * surrogate.CLIGHT, ws=ws, tabcont=np.vstack([tab, tab[-1:]]), iw=atlas.iwavetab(cut),
                recs=recs, contx=synthetic.contx_table())


def oracle(po, h_tables, c):
    atm = {k: c[k] for k in ("xnfdop", "dopple", "xne", "txnxn", "hckt")}
    return po.atlas_xlinop(*h_tables, po.build_tablog(), c["recs"], atm, c["tabcont"], c["iw"], c["ws"], c["contx"],
                           np.zeros((c["ws"].size, c["xnfdop"].shape[1])))[0]


# (the last: more records than get a warp per round of depths, most of them too weak to walk)
CASES = [(16, 50, 40, 9000.0, 2.0), (31, 5000, 200, 9000.0, 2.0), (33, 5000, 200, 4000.0, 3.0), (64, 3000, 100, 9000.0, 1.0),
         (72, 6000, 300, 9000.0, 2.0), (99, 2500, 100, 5777.0, 4.0), (40, 400, 131073, 5777.0, -4.0)]


def test_some_depths_walk_on(po, h_tables, ross):
    """The cases have lines of which only 1 to 16 depths of a round walk past 32 points, and wings of 2000."""
    reach = []
    for nrhox, numnu, n, teff, gf in CASES[1:6]:
        c = case(ross, nrhox, numnu, n, teff, gf)
        for i in range(n):
            one = dict(c, recs=c["recs"][i:i + 1])
            hit = oracle(po, h_tables, one) != 0
            first, last = np.argmax(hit, 0), numnu - 1 - np.argmax(hit[::-1], 0)
            reach.append(np.where(hit.any(0), last - first, 0)[:32])
    left = [np.count_nonzero(r > 64) for r in reach]
    assert sum(0 < k <= 16 for k in left) > 10 and sum(k > 16 for k in left) > 10
    assert max(r.max() for r in reach) > 2000


@pytest.mark.gpu
@pytest.mark.parametrize("prec,tol", [(_lib.PREC_FP64, 1e-9), (_lib.PREC_MIXED, 1e-6)])
@pytest.mark.parametrize("nrhox,numnu,n,teff,gf", CASES)
def test_xlinop_walks(po, gpu_ctx, tables, h_tables, ross, nrhox, numnu, n, teff, gf, prec, tol):
    c = case(ross, nrhox, numnu, n, teff, gf)
    ref = oracle(po, h_tables, c)
    A = atlas.Atlas(gpu_ctx, tables, *h_tables)
    gpu_ctx.set_precision(prec)
    try:
        got, _ = A.xlinop(c["recs"], nrhox, c["xnfdop"], c["dopple"], c["xne"], c["txnxn"], c["hckt"], c["tabcont"],
                          c["iw"], c["ws"], c["contx"])
    finally:
        gpu_ctx.set_precision(_lib.PREC_MIXED)
    assert np.count_nonzero(ref) > 100
    np.testing.assert_array_equal(got != 0, ref != 0)
    assert np.max(np.abs(got - ref) / np.maximum(ref, 1e-300)) < tol
