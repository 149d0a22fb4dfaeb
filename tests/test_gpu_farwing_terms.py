"""SYNTHE's far wings x / n^2 of distant lines to FP64 rounding, whatever lines
share a group: the REAL(4) results of a wing over 38,000 bins determine x, as the
common part of their rounding intervals, to about 1e-11, and the bins of one
sub-tile that are off by more than that have no common x with the others.
"""
import numpy as np
import pytest

from atlas12_b200 import _lib
from atlas12_b200 import synthe as S

LENGTH, CENTRE, DEPTHS = 40000, 1500, 100
BINS = np.arange(CENTRE + 1100, LENGTH + 1)
STRENGTH = 1.0 + 0.01 * np.arange(DEPTHS) + 1e-5 * np.arange(DEPTHS) ** 2


def spread(op):
    """How far the rounding intervals of op = REAL(4)(x / n^2) at BINS are from having a
    common x: (largest lower end) / (smallest upper end) - 1, negative when there is one."""
    half = np.spacing(op).astype(np.float64) / 2
    n2 = (BINS - CENTRE).astype(np.float64) ** 2
    return np.max((op - half) * n2) / np.min((op + half) * n2) - 1.0


def test_measure_sees_a_short_expansion():
    """The measure itself: exact wings pass, wings of 8 Taylor terms (1e-9 at 1,100 bins) do not."""
    n = (BINS - CENTRE).astype(np.float64)
    mid = (BINS - 1) // 128 * 128 + 64.5
    short = sum((k + 1) * (-(BINS - mid) / (mid - CENTRE)) ** k for k in range(8)) / (mid - CENTRE) ** 2
    assert max(spread((x / n ** 2).astype(np.float32)) for x in STRENGTH) <= 2e-12
    assert max(spread((x * short).astype(np.float32)) for x in STRENGTH) > 5e-11


@pytest.mark.gpu
@pytest.mark.parametrize("prec", [_lib.PREC_FP64, _lib.PREC_MIXED])
@pytest.mark.parametrize("lines", [1, 33, 5000])  # four warps per sub-tile twice, one warp per sub-tile
def test_wing_of_distant_lines_to_rounding(gpu_ctx, tables, lines, prec):
    """Bins from 1,100 on (16 terms leave out 1e-18 there).  Tolerance 2e-12: the
    FP64 sum of 5,000 equal terms and their coefficients rounds to at most 1e-12."""
    rec = S.make_lte_lines(np.full(lines, CENTRE), np.full(lines, 1.0 / lines), np.ones(lines, int), np.zeros(lines),
                           np.full(lines, 1e-7), np.zeros(lines), np.zeros(lines))
    one = np.ones(DEPTHS)
    gpu_ctx.set_precision(prec)
    try:
        op = S.Synthe(gpu_ctx, tables).line_opacity(rec, dict(length=LENGTH), 500000.0,
                                                    np.full((DEPTHS, LENGTH), 1e-14, np.float32),
                                                    STRENGTH[:, None], np.full((DEPTHS, 1), 1e-5), one, one, one)
    finally:
        gpu_ctx.set_precision(_lib.PREC_MIXED)
    op = op[:, BINS - 1]
    assert np.all(op > 0)
    assert max(spread(o) for o in op) <= 2e-12


@pytest.mark.gpu
@pytest.mark.parametrize("lines", [1, 5000])
def test_infinite_wing_stays_inside_its_reach(gpu_ctx, tables, lines):
    """Lines of infinite strength: infinite up to their core's end, and nothing past
    MAXPROF bins, also where that lies within a sub-tile."""
    maxprof, far, core = 700, CENTRE + np.array([701, 740, 760, 5000]), CENTRE + np.array([0, 1, 49, 50])
    rec = S.make_lte_lines(np.full(lines, CENTRE), np.full(lines, np.inf), np.ones(lines, int), np.zeros(lines),
                           np.full(lines, 1e-7), np.zeros(lines), np.zeros(lines))
    one = np.ones(1)
    op = S.Synthe(gpu_ctx, tables).line_opacity(rec, dict(length=LENGTH), 500000.0,
                                                np.full((1, LENGTH), 1e-14, np.float32), np.ones((1, 1)),
                                                np.full((1, 1), 1e-5), one, one, one, maxprof=maxprof)[0]
    assert np.all(op[far - 1] == 0.0)
    assert np.all(np.isinf(op[core - 1]))
    assert np.all(np.isinf(op[2 * CENTRE - core - 1]))
