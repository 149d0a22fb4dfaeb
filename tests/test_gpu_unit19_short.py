"""Unit-19 records over windows that a warp walks by itself: one launch for the records
and one for the sum, the same opacity as where the wavelengths come from a table.
"""
import numpy as np
import pytest

from atlas12_b200 import synthe as S
from atlas12_b200 import synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("length,launches", [(1, 2), (50, 2), (256, 2), (1024, 2), (1025, 4)])
def test_launches_and_points(gpu_ctx, tables, length, launches):
    """The first points of a longer window: what a wing adds to a point does not depend on where
    the window ends, as long as the wing starts inside it (one strong Shore line at point 1; its
    sums are single values, so the results are equal to the bit)."""
    g = S.synthe_grid(400.0, 410.0, 500000.0)
    nrhox, full = 16, 2500
    recs = synthetic.nlte_records(1, 400.0, 400.1, seed=1, types=(1,), type_p=(1.0,))
    recs["wlvac"], recs["nbuff"], recs["nelion"], recs["elo"], recs["gf"] = g["wbegin"], 1, 1, 0.0, 1.0
    recs["gammar"], recs["gammas"], recs["gammaw"] = 1.0e13, 3.0e7, 1.0e8
    one = np.ones(nrhox)
    pop = np.ones((nrhox, 2))

    def run(n):
        before = gpu_ctx.launches()
        out = S.Synthe(gpu_ctx, tables).nlte_opacity(
            recs, dict(g, length=n), 410.0, np.full((nrhox, n), 1e-6, np.float32), pop, pop * 1e-5, one, one, one,
            np.zeros((17, 26)), np.zeros((nrhox, n), np.float32), xnfpel=pop)
        return out, gpu_ctx.launches() - before

    got, count = run(length)
    want, _ = run(full)
    assert np.all(got > 0)
    assert np.array_equal(got, want[:, :length])
    assert count == launches


def _shore(po, n, length, nrhox, seed, lo, hi):
    """n strong Shore lines between two points, their wings over the whole window, and the oracle's inputs."""
    g = dict(po.synthe_grid(400.0, 420.0, 500000.0), length=length)
    wav = g["wbegin"] * g["ratio"] ** np.arange(length)
    recs = synthetic.nlte_records(n, wav[0], wav[-1], seed=seed, types=(1,), type_p=(1.0,))
    recs["wlvac"] = np.sort(np.random.default_rng(seed).uniform(wav[lo], wav[hi], n))
    recs["nbuff"] = np.floor(np.log(recs["wlvac"]) / g["ratiolg"] + 0.5).astype(int) - g["ixwlbeg"] + 1
    recs["nelion"], recs["elo"], recs["gf"] = 1, 0.0, 1.0
    recs["gammar"], recs["gammas"], recs["gammaw"] = 1.0e13, 0.0, 1.0e8
    pop = 1.0 + 0.01 * np.arange(nrhox)[:, None] * np.ones((1, 2))
    atm = dict(xnfdop=pop, dopple=np.full((nrhox, 2), 1e-5), xne=np.ones(nrhox), txnxn=np.ones(nrhox),
               hckt=np.ones(nrhox), xnfpel=pop)
    return g, wav, recs, atm, np.full((nrhox, length), 1e-6, np.float32)


@pytest.mark.parametrize("n,length,nrhox,lo,hi", [(60, 2300, 9, 0, -1), (900, 2047, 9, 0, -1), (900, 2049, 9, 0, -1),
                                                  (900, 4200, 9, 0, -1), (2100, 4500, 64, 2100, 2400)])
def test_listed_wings(po, gpu_ctx, tables, n, length, nrhox, lo, hi):
    """Wings listed after 8 steps of a warp (few pairs) and after 64 (2,048 points), and more
    of these than the list holds (268,800 wings, all of them longer).  Tolerance 1e-6 of
    kappa + kappa_cont, as the other unit-19 tests."""
    g, wav, recs, atm, cont = _shore(po, n, length, nrhox, length, lo, hi)
    contx = np.zeros((17, 26))
    ref = po.synthe_nlte_opacity(recs, length, g["wbegin"], g["ratio"], wav[-1], 0.0, cont, atm, contx)
    got = S.Synthe(gpu_ctx, tables).nlte_opacity(recs, g, wav[-1], cont, atm["xnfdop"], atm["dopple"], atm["xne"],
                                                 atm["txnxn"], atm["hckt"], contx, np.zeros((nrhox, length), np.float32),
                                                 xnfpel=atm["xnfpel"])
    assert np.all(ref > 0)
    err = np.abs(got.astype(np.float64) - ref) / (ref + cont.astype(np.float64))
    assert err.max() <= 1e-6, err.max()


@pytest.mark.parametrize("length", [1, 31, 32, 33, 300, 1024, 1025])
def test_hydrogen_by_warps(po, gpu_ctx, tables, length):
    """Analytic hydrogen profiles of 19 waves of blocks, one warp a pair (up to 1,024 points) and
    one block a pair, at both ends of the window and outside it."""
    g = dict(po.synthe_grid(400.0, 410.0, 500000.0), length=length)
    wav = g["wbegin"] * g["ratio"] ** np.arange(length)
    recs = synthetic.hydrogen_records(100.0, 3000.0, g["wbegin"], g["ratio"])
    recs = recs[(recs["nblo"] == 2) | (recs["nblo"] == 3)]
    recs["nbuff"] = np.random.default_rng(length).integers(-2, length + 4, recs.size)
    recs["wlvac"] = g["wbegin"] * g["ratio"] ** (recs["nbuff"] - 1.0)
    h = synthetic.hydrogen_atmosphere()
    nr = h["t"].size
    assert recs.size * nr * 64 >= 2 * 148 * 1024
    cont = np.full((nr, length), 1e-3, np.float32)
    ref = po.synthe_hydrogen_opacity(recs, length, g["wbegin"], g["ratio"], wav[-1], 0.0, cont, h,
                                     po.HTab.from_tables(tables, "s_"), None)
    assert np.count_nonzero(ref) > 0.3 * ref.size
    syn = S.Synthe(gpu_ctx, tables)
    syn.set_hydrogen_tables(tables, None)
    got = syn.nlte_opacity(recs, g, wav[-1], cont, h["xnfdop"], h["dopple"], h["xne"], h["txnxn"], h["hckt"],
                           np.zeros((17, 26)), np.zeros((nr, length), np.float32), hydrogen=h)
    err = np.abs(got.astype(np.float64) - ref) / (ref + cont.astype(np.float64))
    assert err.max() <= 1e-6, err.max()
