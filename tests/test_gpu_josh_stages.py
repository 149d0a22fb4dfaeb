"""JOSH's stages (prepare, the scattering systems, finish) at the sizes where
their pieces end, through the RT pass and the SYNTHE wavelength loop, against
the CPU oracle: depth counts around the warp width and at the capacity,
frequency counts around a group of eight systems, scattering from none to
nearly all of the opacity (series settled by norm, by residual, and
elimination), and the seam between two rounds of wavelengths.

Tolerances: the RT pass's sums 1e-9 relative, H(1) 1e-6 (FP64 on both sides;
the bounds of the RT-pass test).  Flux 1e-4, as the spectrum test: the line
opacity passes through a REAL(4) rounding on both sides.
"""
import numpy as np
import pytest

from atlas12_b200 import atlas, surrogate, synthetic
from atlas12_b200 import synthe as S

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ross():
    return surrogate.RossTable(nt=48, np_=48, nwave=300)


def rt_case(ross, nrhox, numnu, scatter, teff=5777.0, logg=4.44, seed=1):
    m = surrogate.grey_model(teff, logg, nrhox=nrhox, ross=ross)
    ws, rc = synthetic.geometric_waveset(90.0, 20000.0, numnu)
    ka, sg = surrogate.continuum_opacity(ws, m["t"], m["p"])
    rng = np.random.default_rng(seed)
    xl = ka * 10.0 ** rng.uniform(-3.0, 1.0, (numnu, 1))
    return m, ws, rc, ka, sg * scatter, xl, surrogate.HPLANCK / (surrogate.KBOL * m["t"])


@pytest.mark.parametrize("nrhox,numnu,scatter", [(33, 7, 1.0), (64, 8, 1.0e3),
                                                 (72, 9, 30.0), (72, 300, 0.0), (72, 300, 30.0), (72, 300, 1.0e3),
                                                 (96, 17, 30.0), (97, 15, 1.0e3), (100, 40, 1.0)])
def test_rt_pass_over_sizes_and_scattering(po, ops, gpu_ctx, tables, ross, nrhox, numnu, scatter):
    m, ws, rc, ka, sg, xl, hkt = rt_case(ross, nrhox, numnu, scatter)
    A = atlas.Atlas(gpu_ctx, tables)
    got, hs = A.rt_pass(ws, rc, ka, sg, xl, m["rhox"], m["t"], hkt, m["teff"])
    ref, rhs = po.atlas_rt_pass(ops, ws, rc, ka, sg, xl, m["rhox"], m["t"], hkt, m["teff"])
    for k in atlas.ACC_NAMES:
        scale = np.max(np.abs(ref[k]))
        assert np.max(np.abs(got[k] - ref[k])) <= 1e-9 * scale, k
    assert abs(got["pradk0"] - ref["pradk0"]) <= 1e-9 * abs(ref["pradk0"])
    np.testing.assert_allclose(hs, rhs, rtol=1e-6)


@pytest.mark.parametrize("wlend", [400.0009, 426.6, 432.0])
def test_spectrum_over_lengths(po, ops, gpu_ctx, tables, ross, wlend):
    """One wavelength, just under and just over one round (32,768 wavelengths)."""
    case = synthetic.synthe_case(nlines=1, wlbeg=400.0, wlend=wlend, ross=ross)
    g = S.synthe_grid(400.0, wlend, 500000.0)
    n, atm = g["length"], case["atm"]
    rng = np.random.default_rng(3)
    op = np.broadcast_to((10.0 ** rng.uniform(-4, 6, n)).astype(np.float32), (72, n)).copy()
    args = (case["wledge"], case["contabs"], case["contscat"], atm["rhox"], atm["hkt"])
    flux, cont = S.Synthe(gpu_ctx, tables).spectrum(*args, g, op)
    assert np.all(np.isfinite(flux)) and np.all(flux > 0)
    for iw in sorted({1, n, *[i for i in (1000, 32767, 32768, 32769, 32770) if i <= n]}):
        f, c = po.synthe_spectrum(ops, *args, g["wbegin"], g["ratio"], op, iw0=iw, iw1=iw)
        assert abs(flux[iw - 1] - f[0]) <= 1e-4 * abs(f[0]), iw
        assert abs(cont[iw - 1] - c[0]) <= 1e-4 * abs(c[0]), iw
