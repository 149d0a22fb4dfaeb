"""Wings of the unit-19 records (metal, Shore, merged-continuum edge, hydrogen)
over windows around the lengths where the walks change form: a warp's step (32),
what it walks by itself (8 steps), a block's step (256), in both directions, and
more unfinished wings than the list holds; against the FP64 oracle.

Tolerance 1e-6 of kappa + kappa_cont per bin, as the other unit-19 tests (REAL(4)
output, 6e-8; FP64 sums in another order).
"""
import numpy as np
import pytest

from atlas12_b200 import _lib, surrogate, synthetic
from atlas12_b200 import synthe as S

pytestmark = pytest.mark.gpu


def _case(po, length, nrhox, teff=7000.0):
    g = dict(po.synthe_grid(400.0, 402.0, 500000.0), length=length)
    m = surrogate.grey_model(teff, 4.0, nrhox=nrhox, ross=surrogate.RossTable(nt=48, np_=48, nwave=300))
    atm = synthetic.synthe_atmosphere(teff, 4.0, 2.0, nrhox, ross=surrogate.RossTable(nt=48, np_=48, nwave=300))
    wav = g["wbegin"] * g["ratio"] ** np.arange(g["length"])
    ka, sg = surrogate.continuum_opacity(wav, m["t"], m["p"], atm["eos"])
    return g, m, atm, wav, np.ascontiguousarray((ka + sg).T, np.float32)


def _records(g, wav, n, seed, types):
    rng = np.random.default_rng(seed)
    r = np.zeros(n, _lib.NLTE_LINE)
    L = synthetic.synthe_lines(n, wav[0] * 0.9995, wav[-1] * 1.0005, seed=seed)
    r["wlvac"], r["elo"], r["gf"], r["nelion"] = np.sort(L["wlvac"]), L["elo"], L["cgf"], L["nelion"]
    r["itype"] = rng.choice(types, n)
    for a, b in (("gammar", "gamrf"), ("gammas", "gamsf"), ("gammaw", "gamwf")):
        r[a] = L[b]
    f = r["itype"] == 1
    r["gammaw"][f] = 10.0 ** rng.uniform(6.0, 9.0, f.sum())
    r["gammas"][f] = r["gammaw"][f] * rng.uniform(-2.0, 2.0, f.sum())
    r["gammar"][f] = 10.0 ** rng.uniform(10.0, 13.0, f.sum())
    r["gf"][r["itype"] == 0] *= 1.0e4
    r["nbuff"] = np.floor(np.log(r["wlvac"]) / g["ratiolg"] + 0.5).astype(int) - g["ixwlbeg"] + 1
    return r


def _compare(po, gpu_ctx, tables, g, atm, cont, recs, wlend, nrhox):
    a = dict(atm, xnfpel=atm["xnfdop"] * atm["dopple"])
    contx = np.zeros((17, 26))
    ref = po.synthe_nlte_opacity(recs, g["length"], g["wbegin"], g["ratio"], wlend, 0.0, cont, a, contx)
    got = S.Synthe(gpu_ctx, tables).nlte_opacity(recs, g, wlend, cont, atm["xnfdop"], atm["dopple"], atm["xne"],
                                                 atm["txnxn"], atm["hckt"], contx,
                                                 np.zeros((nrhox, g["length"]), np.float32), xnfpel=a["xnfpel"])
    assert np.count_nonzero(ref)
    err = np.abs(got.astype(np.float64) - ref) / (ref + cont.astype(np.float64))
    assert err.max() <= 1e-6, err.max()


@pytest.mark.parametrize("length", [1, 31, 33, 256, 257, 288, 512, 513, 1500])
def test_walk_lengths(po, gpu_ctx, tables, length):
    g, _, atm, wav, cont = _case(po, length, 9)
    recs = _records(g, wav, 60, length, [0, 0, 1, 1, 30])
    _compare(po, gpu_ctx, tables, g, atm, cont, recs, wav[-1], 9)


def test_more_wings_than_the_list_holds(po, gpu_ctx, tables):
    """2,200 Shore lines at 64 depths, 1,600 points: 281,600 wings, most of them
    longer than a warp walks alone; the list holds 262,144."""
    g, _, atm, wav, cont = _case(po, 1600, 64)
    recs = _records(g, wav, 2200, 3, [1])
    recs["wlvac"] = np.sort(np.random.default_rng(4).uniform(wav[400], wav[1200], recs.size))
    recs["nbuff"] = np.floor(np.log(recs["wlvac"]) / g["ratiolg"] + 0.5).astype(int) - g["ixwlbeg"] + 1
    recs["gf"], recs["elo"], recs["gammar"] = 1.0, 0.0, 1.0e13
    recs["gammaw"], recs["gammas"] = 1.0e8, 0.0
    recs["nelion"] = 1
    _compare(po, gpu_ctx, tables, g, atm, cont, recs, wav[-1], 64)


@pytest.mark.parametrize("stehle", [False, True], ids=["analytic", "stehle"])
@pytest.mark.parametrize("length,nbuff", [(1, 1), (255, 1), (256, 256), (257, 128), (513, 257), (1100, 700)])
def test_hydrogen_walk_lengths(po, gpu_ctx, tables, length, nbuff, stehle):
    """Alpha, beta and higher members of the Balmer series moved to grid points
    around nbuff (before the window, inside it, past its end)."""
    g, m, atm, wav, cont = _case(po, length, 9, teff=9500.0)
    recs = synthetic.hydrogen_records(380.0, 700.0, g["wbegin"], g["ratio"], series=((2, 3, 6),))
    recs["nbuff"] = nbuff + np.arange(recs.size) - 2
    recs["wlvac"] = g["wbegin"] * g["ratio"] ** (recs["nbuff"] - 1.0)
    h = synthetic.hydrogen_atmosphere()
    a = {k: np.ascontiguousarray(v[40:49]) for k, v in h.items()}
    st = synthetic.stehle_tables() if stehle else None
    ref = po.synthe_hydrogen_opacity(recs, length, g["wbegin"], g["ratio"], wav[-1], 0.0, cont, a,
                                     po.HTab.from_tables(tables, "s_"), st)
    assert np.count_nonzero(ref) > 0.3 * ref.size
    syn = S.Synthe(gpu_ctx, tables)
    syn.set_hydrogen_tables(tables, st)
    got = syn.nlte_opacity(recs, g, wav[-1], cont, a["xnfdop"], a["dopple"], a["xne"], a["txnxn"], a["hckt"],
                           np.zeros((17, 26)), np.zeros((9, length), np.float32), hydrogen=a)
    err = np.abs(got.astype(np.float64) - ref) / (ref + cont.astype(np.float64))
    assert err.max() <= 1e-6, err.max()
