"""SELECTLINES on records placed at its cut CENRATIO exp(-E/kT) = 1, where the FP32
estimate that drops most records must decide none of them wrongly: E (or, with E = 0,
log gf) of each record follows from its own CENRATIO, up to CENRATIO of 2**400, where
the estimate's error is largest.
"""
import math

import numpy as np
import pytest

from atlas12_b200 import atlas, linelists, synthetic

CLIGHT_NMS = 2.99792458e17
# scale of the populations: CENRATIO to 2**20, 2**50 and 2**430 (H2O's E ends at 32,767 cm-1)
CASES = [(k, s) for k in range(1, 8) for s in (1.0, 1e8, 1e120) if not (k == 6 and s > 1e8)]
TIO, H2O = 5, 6
QUICK = 0.05  # log2 below the cut from which the estimate decides


@pytest.fixture(scope="module")
def sel(tables):
    wt = tables["wavetab"]
    xn, hckt, tc = synthetic.selectlines_tables(wt)
    return dict(wt=wt, iwt=np.asarray(atlas.iwavetab(wt), np.int64), xn=xn, tc=tc, hckt=hckt,
                tb={k: tables[k] for k in ("molcodes", "isox", "tio_isocorr", "h2o_isocorr")})


def log2_cenratio(sel, kind, recs, xmax):
    """log2 of CEN_PREFAC TABLOG(IGFLOG) XNFDOPMAX / FREQ of each record at the NU it is met with
    (:19262-19767), -inf where its species has no population."""
    tb, wt = sel["tb"], sel["wt"]
    if kind == TIO:
        wl = recs["wl"].astype(float)
        dropped = (recs["code"] != 822) | (recs["iso"] < 46) | (recs["iso"] > 50) | ~(wl > 0.0)  # before the NU advance
        iwl = np.floor(np.log(np.where(dropped, 1.0, wl)) / math.log(1.0 + 1.0 / 2000000.0) + 0.5).astype(np.int64)
        iso = np.clip(recs["iso"] - 46, 0, 4)
        g = np.trunc(np.round(recs["gflog"].astype(float) * 1000.0)).astype(np.int64) + 16384 + tb["tio_isocorr"][iso]
        nel = np.full(iwl.size, 895)
        iwl[dropped] = 0
    elif kind == H2O:
        iwl = np.abs(recs["iwl"].astype(np.int64))
        up, ug = recs["ielo"] > 0, recs["igflog"] > 0
        iso = np.where(up & ug, 0, np.where(up, 1, np.where(ug, 2, 3)))
        g = np.abs(recs["igflog"].astype(np.int64)) + tb["h2o_isocorr"][iso]
        nel = np.full(iwl.size, 940)
    else:
        iwl = recs[:, 0].astype(np.int64)
        code = (recs[:, 1].astype(np.int64) & 0xFFFF).astype(np.int16).astype(np.int64)
        g = (recs[:, 2].astype(np.int64) & 0xFFFF).astype(np.int16).astype(np.int64)
        nel = np.abs(np.trunc(code / 10).astype(np.int64))
        if kind == 4:
            order = np.argsort(tb["molcodes"])
            g = g + tb["isox"][order[np.searchsorted(tb["molcodes"][order], code)]]
        if kind == 7:
            g, nel = g - 1272, np.full(iwl.size, 895)
    if kind in (4, 5, 6, 7):
        g = np.maximum(g, 1)
    nu = np.maximum.accumulate(np.maximum(np.searchsorted(sel["iwt"], iwl, side="right") + 1, 1))
    freq = CLIGHT_NMS / np.where(nu > 1, wt[np.minimum(np.maximum(nu - 2, 0), wt.size - 1)], wt[-1])
    with np.errstate(divide="ignore"):
        x = np.log2(xmax[np.minimum(nu - 1, xmax.shape[0] - 1), nel - 1])
    if kind == TIO:
        x[dropped] = -np.inf
    return math.log2(0.026538 / math.sqrt(math.pi)) + (g - 16384) * 0.001 * math.log2(10.0) + x - np.log2(freq)


def at_the_cut(sel, po, kind, scale, n=60_001):
    """Records with E within a few steps of ln(CENRATIO) / HCKT, the third of them with E = 0
    nearly and log gf within a few steps of CENRATIO = 1; and the distance of each from the
    cut in log2."""
    rng = np.random.default_rng(kind)
    xn = np.minimum(sel["xn"], 1e300 / scale) * scale
    xmax = po.xnfdopmax(72, xn, sel["tc"])
    recs = synthetic.selectlines_records(kind, n, sel["wt"], seed=700 + kind).copy()
    hl = sel["hckt"][-1] / math.log(2.0)
    kdex = 0.001 * math.log2(10.0)
    off = rng.uniform(-0.08, 0.08, n)
    flat = rng.uniform(size=n) < 0.33  # E = 0: the cut is CENRATIO itself
    l2 = log2_cenratio(sel, kind, recs, xmax)
    ok = np.isfinite(l2) & (l2 > 0.1) & (l2 < 440.0)
    if kind == H2O:  # E to 32,767 cm-1 only: bring CENRATIO into reach by log gf
        want = np.where(flat, off, rng.uniform(0.2, 0.9 * 32767 * hl, n))
        g = np.abs(recs["igflog"].astype(np.int64)) + np.rint((want - l2) / kdex).astype(np.int64)
        fits = (g > 300) & (g < 32700)
        recs["igflog"] = np.where(fits, g, np.abs(recs["igflog"])) * np.sign(recs["igflog"])
        l2 = log2_cenratio(sel, kind, recs, xmax)
        ok = np.isfinite(l2)
        e = np.clip(np.rint(np.where(flat, 1.0, (l2 - off) / hl)), 1, 32767)
        recs["ielo"] = (e * np.sign(recs["ielo"])).astype(np.int16)
    else:
        step = np.rint(np.where(np.isfinite(l2), off - l2, 0.0) / kdex).astype(np.int64)
        if kind == TIO:
            fits = flat & np.isfinite(l2)
            recs["gflog"] = np.where(fits, recs["gflog"] + step * 0.001, recs["gflog"]).astype(np.float32)
        else:
            g = (recs[:, 2].astype(np.int64) & 0xFFFF).astype(np.int16) + step
            fits = flat & np.isfinite(l2) & (g > 2000) & (g < 32700)
            recs[:, 2] = np.where(fits, (recs[:, 2] & ~0xFFFF) | (g & 0xFFFF), recs[:, 2]).astype(np.int32)
        l2 = log2_cenratio(sel, kind, recs, xmax)
        want = np.where(fits | ~ok, 1e-6, (l2 - off) / hl)
        want = np.maximum(want, 1e-6)
        if kind == TIO:
            recs["e1"] = want.astype(np.float32) * np.where(rng.uniform(size=n) < 0.5, 1, -1)
            recs["e2"] = recs["e1"] * 2.0
            e = np.minimum(np.abs(recs["e1"]), np.abs(recs["e2"])).astype(float)
        else:
            ie = np.clip(np.rint(16384 + 1000 * np.log10(want)), 1, 32767).astype(np.int64)
            recs[:, 1] = (recs[:, 1] & 0xFFFF) | (ie << 16).astype(np.int32)
            e = 10.0 ** ((ie - 16384) * 0.001)
    return recs, xn, xmax, l2 - e * hl, l2


def reference(po, sel, kind, recs, xmax):
    st = {"nu": 1, "freq": CLIGHT_NMS / sel["wt"][-1], "igr": 5}
    out, err, bad = po.selectlines(sel["tb"], kind, recs, st, xmax, sel["hckt"][-1], sel["iwt"].astype(np.int32),
                                   sel["wt"])
    assert err == 0, (err, bad)
    return out, st


@pytest.mark.parametrize("kind,scale", CASES)
def test_records_lie_at_the_cut(sel, po, kind, scale):
    """Hundreds of records on either side within the estimate's margin, the exact filter
    splitting them as their distance says, among them large CENRATIO."""
    recs, _, xmax, d, l2 = at_the_cut(sel, po, kind, scale)
    out, _ = reference(po, sel, kind, recs, xmax)
    below, above = (d > -2 * QUICK) & (d < -1e-6), (d > 1e-6) & (d < 2 * QUICK)
    assert below.sum() > 500 and above.sum() > 500, (below.sum(), above.sum())
    assert np.sum((d > -1.2 * QUICK) & (d < -0.8 * QUICK)) > 20  # where the estimate begins to decide
    if kind != H2O and scale > 1:
        deep = 0.5 * math.log2(scale)
        assert np.sum((below | above) & (l2 > deep)) > 100
    # (LOWPRED and LOWOBS drop populations of 1e-37 and less whatever CENRATIO is)
    sure, near = np.sum((d > 1e-6) & (l2 > 1e-6)), np.sum((np.abs(d) <= 1e-6) | (np.abs(l2) <= 1e-6))
    assert abs(out.shape[0] - sure) <= near, (out.shape[0], sure, near)


@pytest.mark.gpu
@pytest.mark.parametrize("kind,scale", CASES)
def test_selection_at_the_cut_is_the_exact_one(sel, po, gpu_ctx, kind, scale):
    recs, xn, xmax, _, _ = at_the_cut(sel, po, kind, scale)
    want, wst = reference(po, sel, kind, recs, xmax)
    dev = linelists.SelectLines(gpu_ctx, 72, xn, sel["hckt"], sel["tc"], sel["iwt"].astype(np.int32), sel["wt"])
    st = {"nu": 1, "freq": CLIGHT_NMS / sel["wt"][-1], "igr": 5}
    np.testing.assert_array_equal(dev.select(kind, recs, st), want)
    assert st == wst
