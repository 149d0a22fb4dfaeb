"""The staged wavelength loop of SYNTHE (k_spec_pre, the scattering systems,
k_spec_flux) at the sizes where its pieces end: depth counts around the warp
width and at the capacity, a single wavelength, the seam between two rounds
of wavelengths, and optically thick surfaces (which take the Eddington sweeps
instead of the 51-point grid), against the CPU oracle.

Tolerance 1e-9 relative: FP64 on both sides with the same steps; the forms
differ (Newton instead of A + (B + C v) v) and so do the roundings, which the
differences of neighbouring depths amplify by at most ~1e5 (tests of the RT
pass use the same bound for the same routines).
"""
import numpy as np
import pytest

from atlas12_b200 import surrogate, synthetic
from atlas12_b200 import synthe as S

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ross():
    return surrogate.RossTable(nt=48, np_=48, nwave=300)


def check(po, ops, gpu_ctx, tables, case, op, points):
    g = S.synthe_grid(case["wlbeg"], case["wlend"], case["resolu"])
    atm = case["atm"]
    flux, cont = S.Synthe(gpu_ctx, tables).spectrum(case["wledge"], case["contabs"], case["contscat"], atm["rhox"],
                                                    atm["hkt"], g, op)
    for iw in points:
        f, c = po.synthe_spectrum(ops, case["wledge"], case["contabs"], case["contscat"], atm["rhox"], atm["hkt"],
                                  g["wbegin"], g["ratio"], op, iw0=int(iw), iw1=int(iw))
        assert abs(flux[iw - 1] - f[0]) <= 1e-9 * abs(f[0]), (iw, flux[iw - 1], f[0])
        assert abs(cont[iw - 1] - c[0]) <= 1e-9 * abs(c[0]), (iw, cont[iw - 1], c[0])


@pytest.mark.parametrize("nrhox", [31, 32, 33, 64, 72, 96, 97, 100])
def test_spectrum_over_depth_counts(po, ops, gpu_ctx, tables, ross, nrhox):
    case = synthetic.synthe_case(nlines=1, wlbeg=500.0, wlend=500.05, nrhox=nrhox, ross=ross)
    n = S.synthe_grid(500.0, 500.05, 500000.0)["length"]
    # line opacity from none to optically thick at the first depth
    op = (np.logspace(-6, 8, n)[None, :] * np.ones((nrhox, 1))).astype(np.float32)
    op[:, 0] = 0.0
    check(po, ops, gpu_ctx, tables, case, op, np.unique(np.linspace(1, n, 12).astype(int)))


@pytest.mark.parametrize("wlend", [400.0009, 426.6, 432.0])
def test_spectrum_over_lengths(po, ops, gpu_ctx, tables, ross, wlend):
    """One wavelength, just under and just over one round (32,768 wavelengths)."""
    case = synthetic.synthe_case(nlines=1, wlbeg=400.0, wlend=wlend, ross=ross)
    n = S.synthe_grid(400.0, wlend, 500000.0)["length"]
    rng = np.random.default_rng(3)
    op = np.broadcast_to((10.0 ** rng.uniform(-4, 1, n)).astype(np.float32), (72, n)).copy()
    check(po, ops, gpu_ctx, tables, case, op, sorted({1, n, *[i for i in (32767, 32768, 32769, 32770) if i <= n]}))
