"""The work that a user has this framework do, as cases that can be timed.

A case names one public entry point (or the short chain of them that a
program calls together) with its sizes and options:

  batch      AtlasBatch: models loaded into slots, iterated, read back
  model      AtlasModel: one atmosphere iterated on the device
  driver     Atlas.linop1 + Atlas.rt_pass on host arrays, once per iteration
             of a driver that keeps the rest of ATLAS12 to itself
  kapp       Atlas.kapp + Atlas.hlinop: the continuum of one iteration
  select     SelectLines.select_dev: a line database filtered into LINEDATA
  synthe     Synthe.run: one spectrum, from line list to flux
  opacity    atlasgpu_synthe_line_opacity_dev at a molecular line density
  spectrum   atlasgpu_synthe_spectrum_dev: two JOSH solves per wavelength
  unit19     Synthe.nlte_opacity: hydrogen, Shore and merged-continuum records
  network    MLP.loss_grad + MLP.forward: training and use of the warm start

``prepare`` makes the inputs from the seed (atmospheres, line lists, tables)
and the handles a program keeps; ``run`` is one pass.  ``exact`` computes the
outputs in 64-bit numpy from the formulas alone where that is quick enough.
"""
import functools
import math

import numpy as np
import torch

from atlas12_b200 import _lib, atlas, linelists, operators, surrogate, synthetic, warmstart
from atlas12_b200 import synthe as synthe_mod
from atlas12_b200._lib import ptr

NSPEC = 270          # species of the ATLAS12 models
EXACT_PAIRS = 3.0e6  # largest (line, depth) count exact() walks
EXACT_SOLVES = 30000  # largest number of 51x51 systems exact() solves


def listed():
    return [
        # a grid of models on one GPU, the opacity-sampling workload of the benchmark
        dict(name="batch-32x30000", kind="batch", slots=32, numnu=30000, nlines=500000, iters=2, fp64=False, nrhox=72),
        # a small grid at the sizes of the tests
        dict(name="batch-8x5000", kind="batch", slots=8, numnu=5000, nlines=50000, iters=2, fp64=False, nrhox=72),
        # one model by itself, all FP64, two iterations from a given structure
        dict(name="model-30000-fp64", kind="model", numnu=30000, nlines=500000, iters=2, fp64=True, nrhox=72),
        # the two calls a Fortran driver makes per iteration, host arrays in and out
        dict(name="driver-3000", kind="driver", numnu=3000, nlines=20000, fp64=False, nrhox=72, kw=80),
        # the real continuum of one iteration: hydrogen, helium and H2 sources and the hydrogen lines
        dict(name="kapp-30000", kind="kapp", numnu=30000, nrhox=72),
        # a database of atomic lines filtered for one model
        dict(name="select-linerec-8M", kind="select", db=1, n=8000000),
        # the smallest spectrum (half a nanometre), where launches and copies count
        dict(name="synthe-0.5nm", kind="synthe", nlines=500, lo=400.0, width=0.5, mol=0.0, nrhox=72, fp64=False),
        # the 10 nm window with 20,000 lines
        dict(name="synthe-10nm", kind="synthe", nlines=20000, lo=400.0, width=10.0, mol=0.0, nrhox=72, fp64=False),
        # full-optical line density (20M lines over 300-1000 nm) on a 35 nm piece, 30 % molecular
        dict(name="opacity-1M", kind="opacity", nlines=1000000, lo=400.0, width=35.0, mol=0.3, nrhox=72, fp64=False),
        # the wavelength loop of the same piece
        dict(name="spectrum-35nm", kind="spectrum", nlines=2000, lo=400.0, width=35.0, mol=0.3, nrhox=72, fp64=False),
        # the Balmer lines around H-epsilon with 300 metal records of the unit-19 list
        dict(name="unit19-12nm", kind="unit19", n=300, lo=390.0, width=12.0, stehle=True, nrhox=72),
        # training step of the warm-start network
        dict(name="network-64", kind="network", n=64),
    ]


def draw(rng):
    def log(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    kind = rng.choice(["batch", "model", "driver", "kapp", "select", "synthe", "opacity", "spectrum", "unit19",
                       "network"])
    nrhox = rng.choice([72, 72, 72, 64, 56])
    fp64 = rng.random() < 0.3
    if kind == "batch":
        return dict(kind=kind, slots=log(1, 24), numnu=log(1000, 20000), nlines=log(2000, 300000), iters=2, fp64=fp64,
                    nrhox=nrhox)
    if kind == "model":
        return dict(kind=kind, numnu=log(1000, 30000), nlines=log(2000, 500000), iters=2, fp64=fp64, nrhox=nrhox)
    if kind == "driver":
        return dict(kind=kind, numnu=log(500, 12000), nlines=log(1000, 100000), fp64=fp64, nrhox=nrhox,
                    kw=rng.choice([72, 80, 99]))
    if kind == "kapp":
        return dict(kind=kind, numnu=log(500, 30000), nrhox=nrhox)
    if kind == "select":
        return dict(kind=kind, db=rng.choice([1, 2, 3, 4, 5, 6, 7]), n=log(20000, 6000000))
    if kind == "network":
        return dict(kind=kind, n=log(1, 4000))
    lo = round(rng.uniform(320.0, 900.0), 2)
    if kind == "synthe":
        width = round(math.exp(rng.uniform(math.log(0.5), math.log(12.0))), 2)
        return dict(kind=kind, nlines=log(300, 30000), lo=lo, width=width, mol=rng.choice([0.0, 0.3]), nrhox=nrhox,
                    fp64=fp64)
    if kind == "opacity":
        return dict(kind=kind, nlines=log(20000, 700000), lo=lo, width=round(rng.uniform(5.0, 40.0), 2), mol=0.3,
                    nrhox=nrhox, fp64=fp64)
    if kind == "spectrum":
        return dict(kind=kind, nlines=2000, lo=lo, width=round(rng.uniform(2.0, 40.0), 2), mol=0.3, nrhox=nrhox,
                    fp64=fp64)
    return dict(kind=kind, n=log(50, 1000), lo=round(rng.uniform(372.0, 480.0), 2),
                width=round(rng.uniform(4.0, 14.0), 2), stehle=rng.random() < 0.5, nrhox=nrhox)


# ---------------------------------------------------------------- inputs
@functools.lru_cache(maxsize=1)
def _ops():
    return operators.load()


@functools.lru_cache(maxsize=1)
def _ross():
    """A coarse Rosseland table: it only shapes the starting structures."""
    return surrogate.RossTable(nt=48, np_=48, nwave=300)


def _grey(teff, logg, nrhox):
    return surrogate.grey_model(teff, logg, nrhox=nrhox, ross=_ross())


def _context(case):
    return _lib.Context(0, _lib.PREC_FP64 if case.get("fp64") else _lib.PREC_MIXED)


def _star(seed):
    """A sun-like star, a few per cent off from seed to seed."""
    rng = np.random.default_rng(seed)
    return 5777.0 * rng.uniform(0.97, 1.03), 4.44 + rng.uniform(-0.1, 0.1)


def _synthe_case(case, seed):
    teff, logg = _star(seed)
    return synthetic.synthe_case(nlines=case["nlines"], wlbeg=case["lo"], wlend=case["lo"] + case["width"], seed=seed,
                                 teff=teff, logg=logg, mol_frac=case["mol"], nrhox=case["nrhox"], ross=_ross())


def _driver_inputs(case, seed):
    """The module arrays LINOP1 and RUN_RT_PASS read, of a sun-like model."""
    teff, logg = _star(seed)
    m = _grey(teff, logg, case["nrhox"])
    nr, kw = case["nrhox"], case["kw"]
    pop = surrogate.populations(m["t"], m["p"], 1.5, line_pop=surrogate.ATLAS_LINE_POP)
    d = pop["dopple"][:, :NSPEC]
    xnfdop, dopple = np.zeros((NSPEC, kw)), np.ones((NSPEC, kw))
    xnfdop[:, :nr] = np.where(d > 0, pop["xnfp"][:, :NSPEC] / np.maximum(d, 1e-300) / pop["rho"][:, None], 0.0).T
    dopple[:, :nr] = np.where(d > 0, d, 1.0).T
    hkt = surrogate.HPLANCK / (surrogate.KBOL * m["t"])
    ws, rc = synthetic.geometric_waveset(9.0, 160000.0, case["numnu"])
    cut = atlas.cutoff_grid()
    ka, sg = surrogate.continuum_opacity(cut, m["t"], m["p"], pop)
    tab = (ka + sg) * atlas.LINE_CUTOFF / (1.0 - np.exp(-(surrogate.CLIGHT_NMS / cut)[:, None] * hkt[None, :]))
    tabcont = np.zeros((cut.size + 1, kw))
    tabcont[:, :nr] = np.vstack([tab, tab[-1:]])
    acont, sigmac = np.zeros((ws.size, kw)), np.zeros((ws.size, kw))
    acont[:, :nr], sigmac[:, :nr] = surrogate.continuum_opacity(ws, m["t"], m["p"], pop)
    txnxn = (pop["nh"] * (1 - pop["xh"]) + 0.42 * 0.085 * pop["nh"]) * (m["t"] / 1e4) ** 0.3
    return dict(teff=teff, t=m["t"], rhox=m["rhox"], hkt=hkt, xnfdop=xnfdop, dopple=dopple, xne=pop["xne"],
                txnxn=txnxn, hckt=hkt * surrogate.CLIGHT, tabcont=tabcont, iwt=atlas.iwavetab(cut), ws=ws, rc=rc,
                acont=acont, sigmac=sigmac, lines=synthetic.atlas_lines(case["nlines"], ws[2], ws[-3], seed=seed))


def _kapp_inputs(case, seed):
    """Depth vectors KAPP and HLINOP read: hydrogen and helium populations of a warm dwarf."""
    rng = np.random.default_rng(seed)
    m = _grey(9000.0 * rng.uniform(0.9, 1.1), 4.0, case["nrhox"])
    t = m["t"]
    e = surrogate.eos(t, m["p"])
    nhe = 0.0851 * e["nh"]
    f1 = 1.0 / (1.0 + np.exp(-(t - 12000.0) / 1500.0))
    f2 = 1.0 / (1.0 + np.exp(-(t - 22000.0) / 2500.0))
    x4 = nhe * f1 * (1.0 - f2)
    ws, _ = synthetic.geometric_waveset(9.0, 160000.0, case["numnu"])
    return dict(ws=ws, t=t, xne=e["xne"], rho=e["rho"], h1=e["nh"] * (1 - e["xh"]) / 2, h2=e["nh"] * e["xh"],
                he1=nhe * (1.0 - f1), he2=x4 / 2.0, he3=nhe * f1 * f2, xnf4=x4)


def _unit19_inputs(case, seed):
    """Hydrogen and deuterium lines of the Balmer series with metal lines, Shore
    lines and merged-continuum edges, in a 9500 K atmosphere."""
    rng = np.random.default_rng(seed)
    lo, hi, n, nr = case["lo"], case["lo"] + case["width"], case["n"], case["nrhox"]
    g = synthe_mod.synthe_grid(lo, hi, 500000.0)
    m = _grey(9500.0 * rng.uniform(0.97, 1.03), 4.0, nr)
    atm = synthetic.synthe_atmosphere(m["teff"], 4.0, 2.0, nr, ross=_ross())
    wave = np.linspace(lo, hi, 200)
    ka, sg = surrogate.continuum_opacity(wave, m["t"], m["p"], atm["eos"])
    grid = g["wbegin"] * g["ratio"] ** np.arange(g["length"])
    cont = np.stack([np.interp(grid, wave, (ka + sg)[:, j]) for j in range(nr)]).astype(np.float32)
    L = synthetic.synthe_lines(n, lo, hi, seed=seed)
    r = np.zeros(n, _lib.NLTE_LINE)
    r["wlvac"], r["elo"], r["gf"], r["nelion"] = L["wlvac"], L["elo"], L["cgf"], L["nelion"]
    r["itype"] = rng.choice([0, 3, 1, 9, 30], n, p=[.8, .1, .06, .02, .02])
    for a, b in (("gammar", "gamrf"), ("gammas", "gamsf"), ("gammaw", "gamwf")):
        r[a] = L[b]
    f = r["itype"] == 1
    r["gammaw"][f] = 10.0 ** rng.uniform(4.0, 6.0, f.sum())
    r["gammas"][f] = r["gammaw"][f] * rng.uniform(-2.0, 2.0, f.sum())
    r["gammar"][f] = 10.0 ** rng.uniform(10.0, 12.0, f.sum())
    r["nbuff"] = np.floor(np.log(r["wlvac"]) / g["ratiolg"] + 0.5).astype(int) - g["ixwlbeg"] + 1
    recs = np.concatenate([synthetic.hydrogen_records(lo - 5.0, hi + 5.0, g["wbegin"], g["ratio"],
                                                      series=((2, 3, 20),)), r])
    recs = recs[np.argsort(recs["wlvac"], kind="stable")]
    nh1 = atm["eos"]["nh"] * (1.0 - atm["eos"]["xh"])
    hyd = dict(t=m["t"], xnfph1=nh1, xnfph2=atm["eos"]["nh"] * atm["eos"]["xh"], xnfhe1=0.085 * atm["eos"]["nh"],
               xnfh2=1e-5 * nh1 * np.exp(-m["t"] / 1500.0))
    return dict(recs=recs, grid=g, wlend=hi, cont=cont, atm=atm, contx=np.zeros((17, 26)), hyd=hyd,
                xnfpel=atm["xnfdop"] * atm["dopple"], base=np.zeros((nr, g["length"]), np.float32))


def _network_inputs(case, seed):
    rng = np.random.default_rng(seed)
    x = rng.uniform(-1.0, 1.0, (case["n"], warmstart.SHAPE[0])).astype(np.float32)
    t = rng.normal(size=(case["n"], warmstart.SHAPE[3])).astype(np.float32)
    i, h1, h2, o = warmstart.SHAPE
    p = [rng.normal(size=(b, a)) / math.sqrt(a) for a, b in ((i, h1), (h1, h2), (h2, o))]
    b = [0.1 * rng.normal(size=k) for k in (h1, h2, o)]
    return x, t, np.concatenate([v.ravel() for w, c in zip(p, b) for v in (w, c)]).astype(np.float32)


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def prepare(case, seed):
    k, ops = case["kind"], _ops()
    s = dict(case=case, kind=k)
    if k == "batch":
        ws, rc = synthetic.geometric_waveset(9.0, 160000.0, case["numnu"])
        s["ctx"] = _context(case)
        s["batch"] = atlas.AtlasBatch(s["ctx"], ops, nslots=case["slots"], waveset=ws, rcoset=rc, nrhox=case["nrhox"],
                                      linedata=synthetic.atlas_lines(case["nlines"], ws[2], ws[-3], seed=seed))
        s["params"] = warmstart.sample_params(case["slots"], seed)
        s["starts"] = [_grey(p[0], p[1], case["nrhox"]) for p in s["params"]]
    elif k == "model":
        ws, rc = synthetic.geometric_waveset(9.0, 160000.0, case["numnu"])
        s["ctx"] = _context(case)
        s["start"] = _grey(*_star(seed), case["nrhox"])
        s["model"] = atlas.AtlasModel(s["ctx"], ops, s["start"]["teff"], s["start"]["logg"], waveset=ws, rcoset=rc,
                                      nrhox=case["nrhox"], start=s["start"],
                                      linedata=synthetic.atlas_lines(case["nlines"], ws[2], ws[-3], seed=seed))
    elif k == "driver":
        s["in"] = _driver_inputs(case, seed)
        s["atlas"] = atlas.Atlas(_context(case), ops)
    elif k == "kapp":
        s["in"] = _kapp_inputs(case, seed)
        s["atlas"] = A = atlas.Atlas(_context(case), ops)
        A.set_kapp_tables(ops)
        A.set_kapp_h2_tables(ops)
        A.set_stehle_tables(synthetic.stehle_tables(seed=seed))
    elif k == "select":
        wt = ops["wavetab"]
        xn, hckt, tc = synthetic.selectlines_tables(wt, seed=seed)
        s["sel"] = linelists.SelectLines(_context(case), 72, xn, hckt, tc, atlas.iwavetab(wt), wt)
        recs = synthetic.selectlines_records(case["db"], case["n"], wt, seed=seed)
        s["in"] = _dev(np.ascontiguousarray(recs).view(np.uint8))
        s["out"] = torch.zeros((case["n"], 4), dtype=torch.int32, device="cuda")
        s["wavetab"] = wt
    elif k == "synthe":
        s["in"] = _synthe_case(case, seed)
        s["syn"] = synthe_mod.Synthe(_context(case), ops)
    elif k in ("opacity", "spectrum"):
        c = _synthe_case(case, seed)
        s["ctx"] = ctx = _context(case)
        syn = synthe_mod.Synthe(ctx, ops)
        s["grid"] = g = synthe_mod.synthe_grid(c["wlbeg"], c["wlend"], c["resolu"])
        L, atm = c["lines"], c["atm"]
        lines = synthe_mod.make_lte_lines(syn.bin_lines(L["wlvac"], g), L["cgf"], L["nelion"], L["elo"], L["gamrf"],
                                          L["gamsf"], L["gamwf"])
        cont = syn.continuum(c["wledge"], c["continall"], g)
        s["resolu"], s["nspec"] = c["resolu"], atm["xnfdop"].shape[1]
        if k == "opacity":
            s["lines"] = _dev(lines.view(np.uint8))
            s["cont"] = _dev(cont)
            s["vec"] = {n: _dev(atm[n]) for n in ("xnfdop", "dopple", "xne", "txnxn", "hckt")}
            s["out"] = torch.zeros(cont.shape, dtype=torch.float32, device="cuda")
        else:
            op = syn.line_opacity(lines, g, c["resolu"], cont, *(atm[n] for n in ("xnfdop", "dopple", "xne", "txnxn",
                                                                                 "hckt")))
            s["op"] = _dev(op)
            s["tab"] = [_dev(c[n]) for n in ("wledge", "contabs", "contscat")]
            s["vec"] = {n: _dev(atm[n]) for n in ("rhox", "hkt")}
            s["out"] = [torch.zeros(g["length"], dtype=torch.float64, device="cuda") for _ in range(2)]
    elif k == "unit19":
        s["in"] = _unit19_inputs(case, seed)
        s["syn"] = synthe_mod.Synthe(_context(case), ops)
        s["syn"].set_hydrogen_tables(ops, synthetic.stehle_tables(seed=seed) if case["stehle"] else None)
    else:
        s["x"], s["t"], p = _network_inputs(case, seed)
        s["mlp"] = warmstart.MLP(_context(case))
        s["mlp"].set_params(p)
    return s


# ---------------------------------------------------------------- one pass
def run(s):
    k, case = s["kind"], s["case"]
    if k == "batch":
        b = s["batch"]
        for i, (teff, logg, mh, vt) in enumerate(s["params"]):
            b.load(i, teff, logg, vt, mh, s["starts"][i], max_iter=30, tol_percent=0.1)
        b.step(case["iters"])
        status, iters, err, _ = b.poll()
        r = [b.structure(i) for i in range(case["slots"])]
        return dict({n: np.stack([x[n] for x in r]) for n in ("t", "rhox", "p", "xne", "flxerr", "hsurf")},
                    status=status, iters=iters, err=err)
    if k == "model":
        m, st = s["model"], s["start"]
        m.set_structure(st["t"], st["p"], st["rhox"])
        n, hist = m.iterate(max_iter=case["iters"], tol_percent=0.0, graph=True)
        return dict(m.structure(), hist=hist)
    if k == "driver":
        A, c = s["atlas"], s["in"]
        xl, used = A.linop1(c["lines"], case["nrhox"], c["xnfdop"], c["dopple"], c["xne"], c["txnxn"], c["hckt"],
                            c["tabcont"], c["iwt"], c["ws"])
        acc, hs = A.rt_pass(c["ws"], c["rc"], c["acont"], c["sigmac"], xl, c["rhox"], c["t"], c["hkt"], c["teff"])
        return dict(xlines=xl, used=used, acc=acc, hsurf=hs)
    if k == "kapp":
        A, c = s["atlas"], s["in"]
        ac, sg, sc = A.kapp(c["ws"], c["t"], c["xne"], c["rho"], c["h1"], c["h2"], c["he1"], c["he2"], c["he3"],
                            c["xnf4"], xnf3=c["he1"])
        ah, sh = A.hlinop(c["ws"], c["t"], c["xne"], c["rho"], c["h1"])
        return dict(acont=ac, sigmac=sg, scont=sc, ahline=ah, shline=sh)
    if k == "select":
        st = linelists.initial_state(s["wavetab"])
        m = s["sel"].select_dev(case["db"], s["in"], case["n"], st, s["out"], case["n"])
        return dict(lines=s["out"], count=m, nu=st["nu"], igr=st["igr"])
    if k == "synthe":
        wave, flux, cflux, op = s["syn"].run(s["in"])
        return dict(wave=wave, flux=flux, cflux=cflux, opacity=op)
    if k == "opacity":
        g, v = s["grid"], s["vec"]
        s["ctx"].call("atlasgpu_synthe_line_opacity_dev", ptr(s["lines"]), case["nlines"], g["length"], case["nrhox"],
                      s["resolu"], ptr(s["cont"]), ptr(v["xnfdop"]), ptr(v["dopple"]), s["nspec"], ptr(v["xne"]),
                      ptr(v["txnxn"]), ptr(v["hckt"]), synthe_mod.MAXPROF, ptr(s["out"]))
        return s["out"]
    if k == "spectrum":
        g, (we, ca, cs), v = s["grid"], s["tab"], s["vec"]
        s["ctx"].call("atlasgpu_synthe_spectrum_dev", ptr(we), we.numel(), ptr(ca), ptr(cs), ca.shape[1],
                      case["nrhox"], ptr(v["rhox"]), ptr(v["hkt"]), g["wbegin"], g["ratio"], g["length"], ptr(s["op"]),
                      ptr(s["out"][0]), ptr(s["out"][1]))
        return s["out"]
    if k == "unit19":
        c, a = s["in"], s["in"]["atm"]
        return s["syn"].nlte_opacity(c["recs"], c["grid"], c["wlend"], c["cont"], a["xnfdop"], a["dopple"], a["xne"],
                                     a["txnxn"], a["hckt"], c["contx"], c["base"], xnfpel=c["xnfpel"],
                                     hydrogen=c["hyd"])
    loss, grad = s["mlp"].loss_grad(s["x"], s["t"])
    return dict(loss=loss, grad=grad, y=s["mlp"].forward(s["x"]))


# ---------------------------------------------------------------- work
RT_FLOPS = 2.0 / 3.0 * 51 ** 3 + 8 * 51 ** 2  # scattering system and the J, H, K operators of one frequency


def work(case):
    k = case["kind"]
    if k in ("batch", "model", "driver"):
        n, nu, nr = case["nlines"], case["numnu"], case["nrhox"]
        models, iters = case.get("slots", 1), case.get("iters", 1)
        # two wings of about one point per depth and 4,000 frequencies' spacing, ten operations a point; the depth
        # vectors, ~110 operations per (frequency, depth)
        flops = 20.0 * n * nr * max(nu / 30000.0, 0.1) + nu * (RT_FLOPS + 110.0 * nr)
        if k == "driver":
            return dict(bytes=16.0 * n + 8.0 * nu * (3 * case["kw"] + 3), flops=flops)
        return dict(bytes=16.0 * n + 8.0 * models * (nu + 8 * nr), flops=flops * models * iters)
    if k == "kapp":
        e = float(case["numnu"]) * case["nrhox"]
        return dict(bytes=40.0 * e, flops=600.0 * e)
    if k == "select":
        size = {5: 32, 6: 8}.get(case["db"], 16)
        return dict(bytes=case["n"] * (size + 16 * 0.15), flops=20.0 * case["n"])
    if k == "network":
        i, a, b, o = warmstart.SHAPE
        p = i * a + a * b + b * o
        return dict(bytes=4.0 * (2 * p + case["n"] * (i + 2 * o)), flops=8.0 * p * case["n"])
    points = math.log(1.0 + case["width"] / case["lo"]) * 500000.0
    nr = case["nrhox"]
    solve = 2.0 * points * (2 * 18 * 51 ** 2 + 60.0 * nr)
    if k == "spectrum":
        return dict(bytes=4.0 * points * nr + 16.0 * points, flops=solve)
    if k == "unit19":
        return dict(bytes=68.0 * case["n"] + 12.0 * points * nr, flops=300.0 * points * nr)
    # a quarter of the (line, depth) pairs pass the gates, ~20 core points of ~200 operations each
    flops = 0.25 * case["nlines"] * nr * 20.0 * 200.0
    if k == "opacity":
        return dict(bytes=32.0 * case["nlines"] + 8.0 * points * nr, flops=flops)
    return dict(bytes=40.0 * case["nlines"] + 4.0 * points * nr + 16.0 * points, flops=flops + solve)


# ---------------------------------------------------------------- 64-bit values
def exact(case, seed):
    k, nr = case["kind"], case.get("nrhox", 72)
    if k == "network":
        return _exact_network(*_network_inputs(case, seed))
    if k == "driver":
        if case["nlines"] * nr > EXACT_PAIRS or case["numnu"] > 6000:
            return None
        c = _driver_inputs(case, seed)
        xl, used = _exact_linop(c, nr)
        acc, hs = _exact_rt(c, xl)
        return dict(xlines=xl, used=used, acc=acc, hsurf=hs)
    if k in ("synthe", "opacity"):
        if case["nlines"] * nr > EXACT_PAIRS:
            return None
        c = _synthe_case(case, seed)
        g = _exact_grid(c)
        cont = _exact_continuum(c, g)
        op = _exact_opacity(c, g, cont)
        if k == "opacity":
            return op
        flux = _exact_spectrum(c, g, op) if 2 * g["length"] <= EXACT_SOLVES else (None, None)
        return dict(wave=g["wave"] * 10.0, flux=flux[0], cflux=flux[1], opacity=op)
    if k == "spectrum":
        if case["nlines"] * nr > EXACT_PAIRS or 2.0 * math.log(1 + case["width"] / case["lo"]) * 5e5 > EXACT_SOLVES:
            return None
        c = _synthe_case(case, seed)
        g = _exact_grid(c)
        op = _exact_opacity(c, g, _exact_continuum(c, g)).astype(np.float32)
        return list(_exact_spectrum(c, g, op))
    return None  # whole numbers (select), or a model's own iteration and the continuum sources: no short formula


def _exact_network(x, t, p):
    x, t, p = (v.astype(np.float64) for v in (x, t, p))
    i, h1, h2, o = warmstart.SHAPE
    w, at = [], 0
    for a, b in ((i, h1), (h1, h2), (h2, o)):
        w.append((p[at:at + a * b].reshape(b, a), p[at + a * b:at + a * b + b]))
        at += a * b + b
    a1 = np.tanh(x @ w[0][0].T + w[0][1])
    a2 = np.tanh(a1 @ w[1][0].T + w[1][1])
    y = a2 @ w[2][0].T + w[2][1]
    d3 = 2.0 * (y - t) / y.size
    d2 = (d3 @ w[2][0]) * (1.0 - a2 ** 2)
    d1 = (d2 @ w[1][0]) * (1.0 - a1 ** 2)
    g = [v.ravel() for d, a in ((d1, x), (d2, a1), (d3, a2)) for v in (d.T @ a, d.sum(0))]
    return dict(loss=float(np.mean((y - t) ** 2)), grad=np.concatenate(g), y=y)


def _exact_linop(c, nr):
    """LINOP1 line by line in FP64: gates at every eighth depth, then at the
    depths of the blocks next to a passing one; both wings point by point,
    each value added before it is tested against TABCONT."""
    ld, ws = c["lines"], c["ws"]
    i16 = [((ld[:, k] >> sh) & 0xffff).astype(np.uint16).view(np.int16).astype(int) for k in (1, 2, 3) for sh in (0, 16)]
    ielion, ielo, igf, igr, igs, igw = i16
    tab = 10.0 ** ((np.arange(-32768, 32768) - 16384) * 0.001)
    wl = np.exp(ld[:, 0] * np.log(1.0 + 1.0 / 2000000.0))
    nel = np.abs((ielion / 10).astype(int))
    keep = (nel >= 1) & (nel <= c["xnfdop"].shape[0]) & (wl >= ws[0] - 1.0) & (wl <= ws[-1] + 1.0)
    wl, nel = wl[keep], nel[keep]
    cgf = 0.026538 / np.sqrt(np.pi) / 2.99792458e17 * wl * tab[igf[keep] + 32768]
    elo = tab[ielo[keep] + 32768]
    gr, gs, gw = (tab[q[keep] + 32768] * wl / (4.0 * np.pi * 2.99792458e17) for q in (igr, igs, igw))
    nu = np.minimum(np.searchsorted(ws, wl, side="right"), ws.size - 1)  # 0-based first point redward
    nc = np.searchsorted(c["iwt"][:-1], ld[keep, 0], side="right")
    h0, h1, h2 = _voigt_tables()
    xl = np.zeros((ws.size, c["tabcont"].shape[1]))
    tc = c["tabcont"][nc][:, :nr]
    strength = cgf[:, None] * c["xnfdop"][nel - 1][:, :nr]
    boltz = np.exp(-elo[:, None] * c["hckt"][None, :])
    ok = (strength >= tc) & (strength * boltz >= tc)
    nb = nr // 8
    coarse = ok[:, 7:8 * nb:8]
    near = coarse | np.concatenate([np.zeros((wl.size, 1), bool), coarse[:, :-1]], axis=1)
    walk = np.zeros_like(ok)
    walk[:, :8 * nb] = np.repeat(near, 8, axis=1) & ok[:, :8 * nb]
    walk[:, 7:8 * nb:8] = coarse
    used = int(np.count_nonzero(coarse.any(axis=1)))
    il, ij = np.nonzero(walk)
    center = (strength * boltz)[il, ij]
    dop = c["dopple"][nel[il] - 1, ij]
    a = (gr[il] + gs[il] * c["xne"][ij] + gw[il] * c["txnxn"][ij]) / dop
    limit = tc[il, ij]
    for side in (1, -1):
        act = np.arange(il.size)
        for step in range(0 if side > 0 else 1, 101):
            iw = nu[il[act]] + side * step
            on = (iw >= 0) & (iw < ws.size)
            act, iw = act[on], iw[on]
            if not act.size:
                break
            v = np.abs(ws[iw] - wl[il[act]]) / (dop[act] * wl[il[act]])
            cv = center[act] * _voigt_atlas(v, a[act], h0, h1, h2)
            np.add.at(xl, (iw, ij[act]), cv)
            act = act[cv >= limit[act]]
    return xl, used


@functools.lru_cache(maxsize=1)
def _voigt_tables():
    t = _ops()
    v = np.arange(2001) / 200.0
    h0 = np.exp(-v * v)
    h1 = _map1(np.asarray(t["tabvi"], float)[None, :], np.asarray(t["tabh1"], float)[None, :], v[None, :])[0][0]
    return h0, h1, h0 - 2.0 * v * v * h0


def _voigt_atlas(v, a, h0, h1, h2):
    iv = np.minimum((np.minimum(v, 10.0) * 200.0 + 1.5).astype(int), 2001) - 1
    out = np.where(v <= 10.0, (h2[iv] * a + h1[iv]) * a + h0[iv], a / (np.sqrt(np.pi) * np.maximum(v, 1e-30) ** 2))
    big = a > 0.2
    if big.any():
        iv = np.minimum((v * 200.0 + 1.5), 2001.0).astype(int) - 1
        vb, ab, i = v[big], a[big], iv[big]
        vv, aa = vb * vb, ab * ab
        q1 = h1[i] + h0[i] * 1.12838
        q2 = h2[i] + q1 * 1.12838 - h0[i]
        q3 = (1.0 - h2[i]) * 0.37613 - q1 * 0.66667 * vv + q2 * 1.12838
        q4 = (3.0 * q3 - q1) * 0.37613 + h0[i] * 0.66667 * vv * vv
        mid = ((((q4 * ab + q3) * ab + q2) * ab + q1) * ab + h0[i]) * \
            (((-.122727278 * ab + .532770573) * ab - .96284325) * ab + .979895032)
        u = (aa + vv) * 1.4142
        far = ab * 0.79788 / u
        au, vu = aa / u, vv / u
        far = np.where(ab <= 100.0, ((((au - 10.0 * vu) * au * 3.0 + 15.0 * vu * vu) + 3.0 * vv - aa) / (u * u) + 1.0)
                       * far, far)
        out[big] = np.where((ab <= 1.4) & (ab + vb <= 3.2), mid, far)
    return out


# JOSH on rows of frequencies: arrays are [row, depth]
def _parcoe(f, x):
    n = f.shape[1]
    d = np.diff(f, axis=1) / np.diff(x, axis=1)
    c = np.zeros_like(f)
    a, b = np.zeros_like(f), np.zeros_like(f)
    c[:, 1:-1] = (d[:, 1:] - d[:, :-1]) / (x[:, 2:] - x[:, :-2])
    b[:, 1:-1] = d[:, :-1] - (x[:, 1:-1] + x[:, :-2]) * c[:, 1:-1]
    a[:, 1:-1] = f[:, :-2] - x[:, :-2] * d[:, :-1] + x[:, 1:-1] * x[:, :-2] * c[:, 1:-1]
    for j, i in ((0, 0), (1, 1), (2, 2), (n - 1, n - 2)):
        c[:, j], b[:, j] = 0.0, d[:, i]
        a[:, j] = f[:, j] - x[:, j] * d[:, i]
    a0, b0, c0 = a.copy(), b.copy(), c.copy()
    with np.errstate(invalid="ignore", divide="ignore"):
        w = np.abs(c0[:, 2:]) / (np.abs(c0[:, 2:]) + np.abs(c0[:, 1:-1]))
    use = c0[:, 1:-1] != 0.0
    for q, q0 in ((a, a0), (b, b0), (c, c0)):
        q[:, 1:-1] = np.where(use, q0[:, 2:] + w * (q0[:, 1:-1] - q0[:, 2:]), q0[:, 1:-1])
        q[:, n - 2] = q[:, n - 1]
    return a, b, c


def _integ(x, f, start):
    a, b, c = _parcoe(f, x)
    lo, hi = x[:, :-1], x[:, 1:]
    term = (a[:, :-1] + b[:, :-1] * 0.5 * (hi + lo) + c[:, :-1] / 3.0 * ((hi + lo) * hi + lo * lo)) * (hi - lo)
    return np.concatenate([start[:, None], start[:, None] + np.cumsum(term, axis=1)], axis=1)


def _map1(xo, fo, xn):
    """MAP1 of rows (xo, fo) onto xn (rows broadcast); (values, MAP1's return value per row)."""
    rows, nold, nnew = fo.shape[0], fo.shape[1], xn.shape[1]
    xo, xn = np.broadcast_to(xo, (rows, nold)), np.broadcast_to(xn, (rows, nnew))
    L = np.clip((xo[:, :, None] <= xn[:, None, :]).sum(axis=1) + 1, 2, nold + 1)
    prev = np.zeros_like(L)
    for k in range(1, nnew):
        prev[:, k] = np.where(L[:, k] == L[:, k - 1], prev[:, k - 1], np.minimum(L[:, k - 1], nold))

    def at(v, i):
        return np.take_along_axis(v, np.clip(i - 1, 0, nold - 1), axis=1)

    def parabola(m):
        """Through the old points m-1, m, m+1."""
        x0, x1, x2, f0, f1, f2 = (at(v, m + q) for v in (xo, fo) for q in (-1, 0, 1))
        d = (f1 - f0) / (x1 - x0)
        c = ((f2 - f1) / (x2 - x1) - d) / (x2 - x0)
        return f0 - x0 * d + x0 * x1 * c, d - (x0 + x1) * c, c

    Lc = np.minimum(L, nold)
    lin = (L <= 3) | (L > nold)
    with np.errstate(all="ignore"):
        back = parabola(Lc - 1)  # L-2, L-1, L: the forward parabola of L-1 is the same one
        fore = parabola(Lc)
        w = np.where(np.abs(fore[2]) != 0.0, np.abs(fore[2]) / (np.abs(fore[2]) + np.abs(back[2])), 0.0)
        q = [np.where(Lc >= nold, b, f + w * (b - f)) for b, f in zip(back, fore)]
        slope = (at(fo, Lc) - at(fo, Lc - 1)) / (at(xo, Lc) - at(xo, Lc - 1))
        out = np.where(lin, at(fo, Lc) - at(xo, Lc) * slope + slope * xn, q[0] + (q[1] + q[2] * xn) * xn)
    return out, Lc[:, -1] - 1


def _deriv(x, f):
    d = np.diff(f, axis=1) / np.diff(x, axis=1)
    s = np.sign(x[:, 1:2] - x[:, :1])
    out = np.empty_like(f)
    out[:, 0], out[:, -1] = d[:, 0], d[:, -1]
    sc = np.maximum(np.maximum(np.abs(f[:, :-2]), np.abs(f[:, 1:-1])), np.abs(f[:, 2:])) / np.abs(x[:, 1:-1])
    sc = np.where(sc == 0.0, 1.0, sc)
    t = [q / sc / (s * np.sqrt(1.0 + (q / sc) ** 2) + 1.0) for q in (d[:, 1:], d[:, :-1])]
    out[:, 1:-1] = (t[0] + t[1]) / (1.0 - t[0] * t[1]) * sc
    return out


def _scatter(xa, xb, coefj):
    """XS of (1 - XALPHA) XSBAR + XALPHA (COEFJ XS) per row."""
    xs = np.empty_like(xb)
    for i in range(0, xb.shape[0], 2048):
        m = np.eye(51) - xa[i:i + 2048, :, None] * coefj[None, :, :]
        xs[i:i + 2048] = np.linalg.solve(m, ((1.0 - xa) * xb)[i:i + 2048, :, None])[:, :, 0]
    return np.where((xa.max(axis=1) > 0.0)[:, None], xs, xb)


def _josh_start(rhox, abtot, alpha, snubar):
    t = _ops()
    xtau, coefj = np.asarray(t["xtau8"], float), np.asarray(t["coefj"], float)
    x = np.broadcast_to(rhox, abtot.shape)
    tau = _integ(x, abtot, abtot[:, 0] * rhox[0])
    mapped = tau[:, 0] <= xtau[-1]
    xb, maxj = _map1(tau, snubar, xtau[None, :])
    xa, _ = _map1(tau, alpha, xtau[None, :])
    xa, xb = np.maximum(xa, 0.0), np.maximum(xb, 1e-38)
    top = xtau[None, :] < tau[:, :1]
    xb = np.where(top, np.maximum(snubar[:, :1], 1e-38), xb)
    xa = np.where(top, np.maximum(alpha[:, :1], 0.0), xa)
    xs = np.zeros_like(xb)
    xs[mapped] = np.maximum(_scatter(xa[mapped], xb[mapped], coefj), 1e-37)
    return tau, np.where(mapped, maxj, 1), mapped, xs


def _exact_rt(c, xl):
    """RUN_RT_PASS in FP64 over rows of frequencies."""
    t = _ops()
    xtau, coefj, coefh, ck = (np.asarray(t[k], float) for k in ("xtau8", "coefj", "coefh", "ck_j"))
    nr = c["t"].size
    freq = 2.99792458e17 / c["ws"]
    e = np.exp(-freq[:, None] * c["hkt"][None, :])
    stim = 1.0 - e
    bnu = 2.0 * surrogate.HPLANCK / surrogate.CLIGHT ** 2 * freq[:, None] ** 3 * e / stim
    ac, sg, al = c["acont"][:, :nr], c["sigmac"][:, :nr], xl[:, :nr] * stim
    ab = ac + al + sg
    alpha, snubar = sg / ab, (ac * bnu + al * bnu) / (ac + al)
    tau, maxj, mapped, xs = _josh_start(c["rhox"], ab, alpha, snubar)
    snu, hnu, jm, jn = (np.zeros_like(ab) for _ in range(4))
    knu = np.zeros(freq.size)
    for mj in np.unique(maxj):
        for r in (np.nonzero((maxj == mj) & mapped)[0], np.nonzero((maxj == mj) & ~mapped)[0]):
            if r.size:
                _josh_rows(r, int(mj), mapped[r[0]], nr, tau, xs, xtau, alpha, snubar, bnu, snu, hnu, jm, jn)
        r = np.nonzero(maxj == mj)[0]
        if mj == 1:
            knu[r] = jn[r, 0] / 3.0
            continue
        jm[r, :mj] = _map1(xtau[None, :], xs[r] @ coefj.T - xs[r], tau[r, :mj])[0]
        hnu[r, :mj] = _map1(xtau[None, :], xs[r] @ coefh.T, tau[r, :mj])[0]
        snu[r, :mj] = np.maximum(snu[r, :mj], 1e-38)
        jn[r, :mj] = np.maximum(jm[r, :mj] + snu[r, :mj], 1e-38)
        knu[r] = xs[r] @ ck
    neg = ((snu < 0) | (jn < 0) | (hnu < 0)).any(axis=1)
    for v in (snu, jn, hnu):
        v[neg] = np.maximum(v[neg], 1e-99)
    w = c["rc"][:, None]
    dab = _deriv(np.broadcast_to(c["rhox"], ab.shape), ab)
    d = np.maximum(1e-10, np.diff(tau, axis=1))
    d = np.concatenate([d, d[:, -1:]], axis=1)
    small = (0.922784335098467 - np.log(d)) * d / 4.0 + d * d / 12.0 - d ** 3 / 96.0 + d ** 4 / 720.0
    ex = np.where(d < 10.0, _e3(np.minimum(d, 10.0)), 0.0)
    if c["teff"] <= 4250.0:
        ex = np.where((d > 0.005) & (d < 0.02), 0.0, ex)
    term = np.where(d <= 0.01, small, 0.5 * (d + ex - 0.5) / d)
    diag = term.copy()
    diag[:, 1:] += term[:, :-1]
    dbdt = bnu * freq[:, None] * c["hkt"] / c["t"] / stim
    terms = dict(rjmins=ab * jm, rdabh=dab / ab * hnu, flxrad=hnu, raden=jn, h_total=hnu, accrad=ab * hnu,
                 rdiagj=ab * (diag - 1.0) / (1.0 - alpha * diag) * (1.0 - alpha) * dbdt, abross=dbdt / ab)
    acc = {k: (v * w).sum(axis=0) for k, v in terms.items()}
    acc["pradk0"] = float((knu * c["rc"]).sum())
    return acc, hnu[:, 0].copy()


def _josh_rows(r, mj, mapped, nr, tau, xs, xtau, alpha, snubar, bnu, snu, hnu, jm, jn):
    """SNU of rows r (all with MAXJ = mj) and the Eddington sweeps below it, each row until it has converged."""
    if mapped:
        snu[r, :mj] = _map1(xtau[None, :], xs[r], tau[r, :mj])[0]
    if mj == nr:
        return
    first, m = (0 if mj == 1 else mj), max(mj - 1, 1) - 1
    snu[r, first:] = snubar[r, first:]
    sb = snubar.copy()
    for _ in range(50):
        bad = (snu[r, m:] <= 0.0).any(axis=1)
        hit = r[bad]
        sb[hit, m:] = snu[hit, m:] = bnu[hit, m:]
        h = _deriv(tau[r, m:], snu[r, m:])
        low = (h <= 0.0).any(axis=1)
        hit = r[low]
        sb[hit, m:] = snu[hit, m:] = bnu[hit, m:]
        h[low] = _deriv(tau[hit, m:], snu[hit, m:]) if hit.size else h[low]
        hnu[r, m:] = h / 3.0
        j = _deriv(tau[r, mj - 1:], hnu[r, mj - 1:])
        jm[r, mj - 1:] = j
        jm[np.ix_(r[bad | low], np.arange(first, nr))] = 0.0
        jn[r, first:] = jm[r, first:] + snu[r, first:]
        new = (1.0 - alpha[r, first:]) * sb[r, first:] + alpha[r, first:] * jn[r, first:]
        err = (np.abs(new - snu[r, first:]) / new).sum(axis=1)
        snu[r, first:] = new
        r = r[~(err < 1e-5)]
        if not r.size:
            break


def _e3(x):
    """E3(x): 64-point Gauss-Legendre of x^2 int_x^inf e^-t / t^3 dt on t = x/u."""
    u, w = np.polynomial.legendre.leggauss(64)
    u, w = 0.5 * (u + 1.0), 0.5 * w
    return sum(wi * ui * np.exp(-x / ui) for ui, wi in zip(u, w))


def _exact_grid(c):
    ratio = 1.0 + 1.0 / c["resolu"]
    rl = math.log(ratio)
    beg = int(math.log(c["wlbeg"]) / rl)
    beg += math.exp(beg * rl) < c["wlbeg"]
    n = int(math.log(c["wlend"] / c["wlbeg"]) / rl)
    return dict(length=n, wave=math.exp(beg * rl) * ratio ** np.arange(n), ratiolg=rl, beg=beg)


def _edges(c, wave):
    """Interval of every wavelength and the three parabola weights on its table points."""
    we = c["wledge"]
    i = np.clip(np.searchsorted(we, wave, side="right") - 1, 0, we.size - 2)
    a, b = we[i], we[i + 1]
    h, dd = 0.5 * (a + b), 0.5 * (b - a) ** 2
    q = ((wave - h) * (wave - b) / dd, (a - wave) * (wave - b) * 2.0 / dd, (wave - a) * (wave - h) / dd)
    return lambda t: sum(q[k][None, :] * t[:, 3 * i + k] for k in range(3))


def _exact_continuum(c, g):
    v = _edges(c, g["wave"])(c["continall"]).astype(np.float32)
    return (10.0 ** np.maximum(v, np.float32(-15.0)).astype(np.float64)).astype(np.float32)


@functools.lru_cache(maxsize=1)
def _weideman():
    """Weideman's (1994) 32 coefficients and L."""
    n, m = 32, 128
    ell = math.sqrt(n / math.sqrt(2.0))
    theta = np.arange(-m + 1, m) * np.pi / m
    t = ell * np.tan(theta / 2.0)
    f = np.concatenate([[0.0], np.exp(-t * t) * (ell * ell + t * t)])
    a = np.real(np.fft.fft(np.fft.fftshift(f))) / (2 * m)
    return a[1:n + 1][::-1], ell


def _voigt_synthe(v, a):
    coef, ell = _weideman()
    z = np.abs(v) + 1j * a
    out = np.empty(z.shape)
    far = np.abs(v) + a > 15.0
    zf = z[far]
    out[far] = (1j * zf / (math.sqrt(math.pi) * (zf * zf - 0.5))).real
    zn = z[~far]
    d = ell - 1j * zn
    p = np.polyval(coef.astype(complex), (ell + 1j * zn) / d)
    out[~far] = (2.0 * p / d ** 2 + 1.0 / math.sqrt(math.pi) / d).real
    return out


def _exact_opacity(c, g, cont):
    """SYNTHE's LTE line loop in FP64: the centre, the core points up to ten
    Doppler widths or the first value below the cutoff, and x/n^2 beyond."""
    L, atm, n = c["lines"], c["atm"], g["length"]
    nb = (np.log(L["wlvac"]) / g["ratiolg"] + 0.5).astype(int) - g["beg"]  # 0-based
    el = L["nelion"] - 1
    out = np.zeros((atm["t"].size, n))
    for j in range(atm["t"].size):
        kmin = cont[j].astype(np.float64)[np.clip(nb, 0, n - 1)] * 1e-3
        k0 = L["cgf"].astype(np.float64) * atm["xnfdop"][j, el]
        kb = k0 * np.exp(-L["elo"].astype(np.float64) * atm["hckt"][j])
        s = np.nonzero((k0 >= kmin) & (kb >= kmin))[0]
        dop = atm["dopple"][j, el[s]]
        a = (L["gamrf"][s].astype(np.float64) + L["gamsf"][s].astype(np.float64) * atm["xne"][j] +
             L["gamwf"][s].astype(np.float64) * atm["txnxn"][j]) / dop
        n10 = (10.0 * dop * c["resolu"]).astype(int)
        dv = 1.0 / dop / c["resolu"]
        k, lim, mid = kb[s], kmin[s], nb[s]
        act = np.arange(s.size)
        acc = np.zeros(n)

        def add(at, v):
            on = (at >= 0) & (at < n)
            acc[:] += np.bincount(at[on], weights=v[on], minlength=n)

        step = 0
        while act.size:
            p = k[act] * _voigt_synthe(step * dv[act], a[act])
            add(mid[act] + step, p)
            if step:
                add(mid[act] - step, p)
                end = (p >= lim[act]) & (step == n10[act])
                for i, pv in zip(act[end], p[end]):
                    xw = pv * float(n10[i]) ** 2
                    m = int(min(math.sqrt(xw / lim[i]) + 1.0, 1000000.0))
                    for lo, hi in ((mid[i] + n10[i] + 1, mid[i] + m), (mid[i] - m, mid[i] - n10[i] - 1)):
                        lo, hi = max(lo, 0), min(hi, n - 1)
                        if lo <= hi:
                            acc[lo:hi + 1] += xw / (np.arange(lo, hi + 1) - mid[i]).astype(float) ** 2
                act = act[(p >= lim[act]) & (step < n10[act])]
            else:
                act = act[n10[act] >= 1]
            step += 1
        out[j] = acc
    return out


def _exact_spectrum(c, g, op):
    """Flux and continuum flux: H(1) of JOSH's 51-point solution with and without the lines."""
    atm, freq = c["atm"], 2.99792458e17 / g["wave"]
    w = _edges(c, g["wave"])
    ka, sg = (10.0 ** w(c[k]).T for k in ("contabs", "contscat"))
    e = np.exp(-freq[:, None] * atm["hkt"][None, :])
    bnu = 2.0 * surrogate.HPLANCK / surrogate.CLIGHT ** 2 * freq[:, None] ** 3 * e / (1.0 - e)
    ch = np.asarray(_ops()["ch_j"], float)
    got = []
    for line in (op.T.astype(np.float64) * (1.0 - e), np.zeros_like(ka)):
        ab = ka + sg + line
        tau, _, mapped, xs = _josh_start(atm["rhox"], ab, sg / ab, bnu)
        h = xs @ ch
        r = np.nonzero(~mapped)[0]
        if r.size:  # optically thick at the first depth: the Eddington sweeps' H(1)
            hnu = np.zeros_like(ab)
            _josh_rows(r, 1, False, ab.shape[1], tau, xs, None, sg / ab, bnu.copy(), bnu, np.zeros_like(ab), hnu,
                       np.zeros_like(ab), np.zeros_like(ab))
            h[r] = hnu[r, 0]
        got.append(h)
    return tuple(got)
