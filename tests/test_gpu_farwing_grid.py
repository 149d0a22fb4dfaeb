"""SYNTHE's far wings over grids of every size: sub-tiles without a wing beside ones with
many, one and four warps a sub-tile (far_four_warps), and the tile counters in shared
memory and, from 8,192 tiles on, in global memory, against the FP64 oracle.

Tolerance 1e-5 of kappa_line + kappa_cont per bin, as the line-opacity test.
"""
import numpy as np
import pytest

from atlas12_b200 import synthe as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("length,lines,nrhox,maxprof", [
    (1000, 1, 72, 1000000), (1000, 2000, 3, 1000000),    # one tile: one warp, four warps
    (5000, 600, 16, 1000000), (60000, 600, 16, 1000000),    # the same lines on more tiles
    (200000, 12, 16, 700), (200000, 1, 72, 1000000),     # most sub-tiles without a wing
    (8191 * 1024, 10, 1, 1000000), (8191 * 1024 + 1, 10, 1, 1000000),
    (8192 * 1024, 310000, 1, 200), (8190 * 1024, 310000, 1, 200)])  # blocks of 1,024 records there
def test_grids(po, gpu_ctx, tables, length, lines, nrhox, maxprof):
    rng = np.random.default_rng(length + lines)
    nb = np.sort(rng.integers(1, length + 1, lines))
    nb[0] = 1
    nb[-1] = length
    cgf = 10.0 ** rng.uniform(-3.0, 0.0, lines)
    L = dict(nbuff=nb, cgf=cgf.astype(np.float32), nelion=np.ones(lines, int), elo=np.zeros(lines),
             gamrf=np.full(lines, 1e-7, np.float32), gamsf=np.zeros(lines), gamwf=np.zeros(lines))
    one = np.ones(nrhox)
    atm = dict(xnfdop=1.0 + 0.1 * np.arange(nrhox)[:, None], dopple=np.full((nrhox, 1), 1e-5), xne=one, txnxn=one,
               hckt=one)
    cont = np.full((nrhox, length), 1e-11, np.float32)
    ref = po.synthe_line_opacity(po.FP64, L, length, atm, cont, 500000.0, maxprof)[1]
    rec = S.make_lte_lines(L["nbuff"], L["cgf"], L["nelion"], L["elo"], L["gamrf"], L["gamsf"], L["gamwf"])
    got = S.Synthe(gpu_ctx, tables).line_opacity(rec, dict(length=length), 500000.0, cont, atm["xnfdop"],
                                                 atm["dopple"], one, one, one, maxprof=maxprof)
    assert np.count_nonzero(ref) > 100 * min(lines, 5)
    assert np.max(np.abs(got.astype(np.float64) - ref) / (ref + cont.astype(np.float64))) <= 1e-5
