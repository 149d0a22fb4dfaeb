"""SYNTHE's line-opacity lists where they can go wrong: far-wing counts around
the warp buffer (32) and a block of the list kernels (1,024), short and long
lists (four warps and one warp per sub-tile), one bin, tile edges, wings past
the 1/n^2 table and past the grid, against the FP64 oracle.

Tolerance 1e-5 of kappa_line + kappa_cont per bin, as the line-opacity test
(REAL(4) output; the expansions' truncation is below 1e-8).
"""
import numpy as np
import pytest

from atlas12_b200 import _lib, surrogate, synthetic
from atlas12_b200 import synthe as S

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ross():
    return surrogate.RossTable(nt=48, np_=48, nwave=300)


@pytest.mark.parametrize("prec", [_lib.PREC_FP64, _lib.PREC_MIXED])
@pytest.mark.parametrize("nlines,width,nrhox,strength", [(1, 0.001, 72, 1.0), (31, 0.81, 64, 1e3), (33, 0.82, 72, 1e6),
                                                         (1023, 0.84, 8, 1e2), (1025, 1.7, 9, 1e2),
                                                         (9000, 0.5, 8, 1e4), (40, 60.0, 8, 1e8)])
def test_line_opacity_lists(po, gpu_ctx, tables, ross, nlines, width, nrhox, strength, prec):
    case = synthetic.synthe_case(nlines=nlines, wlbeg=400.0, wlend=400.0 + width, seed=nlines, nrhox=nrhox, ross=ross)
    g = po.synthe_grid(case["wlbeg"], case["wlend"], case["resolu"])
    nb = np.array([po.nbuff(w, g["ratiolg"], g["ixwlbeg"]) for w in case["lines"]["wlvac"]], np.int32)
    L = dict(case["lines"], nbuff=nb, cgf=(case["lines"]["cgf"] * np.float32(strength)).astype(np.float32))
    cont = po.synthe_continuum(po.REF32, case["wledge"], case["continall"], g["wbegin"], g["ratio"], g["length"])
    atm = case["atm"]
    ref = po.synthe_line_opacity(po.FP64, L, g["length"], atm, cont, case["resolu"])[1]
    rec = S.make_lte_lines(L["nbuff"], L["cgf"], L["nelion"], L["elo"], L["gamrf"], L["gamsf"], L["gamwf"])
    gpu_ctx.set_precision(prec)
    try:
        got = S.Synthe(gpu_ctx, tables).line_opacity(rec, g, case["resolu"], cont, atm["xnfdop"], atm["dopple"],
                                                     atm["xne"], atm["txnxn"], atm["hckt"])
    finally:
        gpu_ctx.set_precision(_lib.PREC_MIXED)
    assert np.max(np.abs(got.astype(np.float64) - ref) / (ref + cont.astype(np.float64))) <= 1e-5
