"""What a user of this framework has it do, as cases that can be timed and compared.

Every case is one pass through the public entry points on inputs that a seed makes: the model atmospheres
shipped with the package, line lists with the distributions of `fastspec_b200.workloads`, or a line opacity
spectrum of the same character.  The kinds:

  scalar   one spectrum of an atomic list through host arrays: line opacity, windows (and central line
           depths), then intensities and fluxes; mixed or FP64 precision
  dense    one spectrum of a molecular list that lies on the device, cool dwarf, wide grid
  batch    a grid of atmospheres that share one atomic list, replayed as one graph
  fit      flux, chi-square and gradients for log gf, abundances and microturbulence
  stokes   polarised spectrum of Zeeman lines: magnetic line opacity, then Stokes IQUV
  solve    formal solution alone for a given line opacity; plane-parallel or spherical
  broaden  disk integration with rotation, macroturbulence and an instrumental profile
"""
import math
import os

import numpy as np
import torch

import fastspec_b200 as F
from fastspec_b200 import adjoint as AD
from fastspec_b200 import workloads as W
from fastspec_b200.shard import GpuBackend

DEV = "cuda"
_DATA = os.path.join(os.path.dirname(os.path.abspath(F.__file__)), "data")
_STATE = ("rhox", "T", "xne", "xna", "rho", "fractionpf", "xamass", "potion", "ion", "frac_h1", "frac_he1")
_WSTART = {"solar": 5000.0, "cooldwarf": 5000.0, "magnetic": 6000.0}


def listed():
    return [
        # a short order or a single blend, as an abundance analysis asks for thousands of times: launches count
        dict(name="scalar_1k", kind="scalar", nlines=300, nwl=1001, dstep=0.01, nmu=7, prec="mixed", linstr=False),
        # the ordinary run: 200 A of a solar-type spectrum, with the central depths of its lines
        dict(name="scalar_40k", kind="scalar", nlines=20000, nwl=40001, dstep=0.005, nmu=7, prec="mixed", linstr=True),
        # the same spectrum in the plain FP64 path
        dict(name="scalar_40k_fp64", kind="scalar", nlines=20000, nwl=40001, dstep=0.005, nmu=7, prec="fp64",
             linstr=False),
        # a cut through a molecular list: a million lines, optical to K band
        dict(name="dense_1m", kind="dense", nlines=1000000, wend=25000.0, resol=300000.0, nmu=7),
        # ten million lines on the same grid: what most of a cool star's time goes into
        dict(name="dense_10m", kind="dense", nlines=10000000, wend=25000.0, resol=300000.0, nmu=7),
        # a grid of models for parameter determination
        dict(name="batch_24", kind="batch", natm=24, grid=W.SEED0 + 3, nlines=2000000, nmu=7),
        # one step of a fit to an observed spectrum: forward and backward
        dict(name="fit_100k", kind="fit", nlines=100000, span=500.0, dstep=0.005, nmu=7),
        # a magnetic star, field given in the observer's frame
        dict(name="stokes_50k", kind="stokes", nlines=5000, nwl=50001, dstep=0.002, nmu=9, bframe=1, prec="mixed"),
        # a line region of a magnetic star in FP64, field given in the star's frame
        dict(name="stokes_6k_fp64", kind="stokes", nlines=700, nwl=6001, dstep=0.004, nmu=5, bframe=0, prec="fp64"),
        # the solver alone, on an opacity spectrum that was kept: other angles or another source of opacity
        dict(name="solve_483k", kind="solve", atm="cooldwarf", nwl=482832, nmu=7, sphere=False),
        # a star whose limb matters: rays through a spherical model, the outermost ones grazing
        dict(name="solve_sphere_40k", kind="solve", atm="solar", nwl=40001, nmu=7, sphere=True),
        # a rotating star from kept intensities
        dict(name="broaden_200k", kind="broaden", nwl=200001, resol=300000.0, nmu=7, vsini=25.0, vmacro=4.0,
             vgau=65000.0),
    ]


def _log(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    kind = rng.choice(["scalar", "scalar", "dense", "batch", "fit", "stokes", "solve", "broaden"])
    if kind == "scalar":
        return dict(kind=kind, nlines=_log(rng, 30, 20000), nwl=_log(rng, 301, 40001),
                    dstep=rng.choice([0.0037, 0.005, 0.01, 0.02]), nmu=rng.randint(1, 9),
                    prec=rng.choice(["mixed", "fp64"]), linstr=rng.random() < 0.5)
    if kind == "dense":
        return dict(kind=kind, nlines=_log(rng, 20000, 4000000), wend=float(rng.randint(6000, 25000)),
                    resol=float(_log(rng, 40000, 300000)), nmu=rng.randint(1, 9))
    if kind == "batch":
        return dict(kind=kind, natm=rng.randint(2, 16), grid=rng.randint(1, 1 << 20), nlines=_log(rng, 100000, 2000000), nmu=rng.randint(3, 9))
    if kind == "fit":
        return dict(kind=kind, nlines=_log(rng, 500, 60000), span=float(_log(rng, 10, 400)),
                    dstep=rng.choice([0.005, 0.008, 0.015]), nmu=rng.randint(3, 7))
    if kind == "stokes":
        prec = rng.choice(["mixed", "fp64"])
        return dict(kind=kind, nlines=_log(rng, 50, 3000 if prec == "mixed" else 700),
                    nwl=_log(rng, 1001, 30001 if prec == "mixed" else 8001), dstep=rng.choice([0.002, 0.0031, 0.005]),
                    nmu=rng.randint(2, 9), bframe=rng.randint(0, 2), prec=prec)
    if kind == "solve":
        sphere = rng.random() < 0.4
        return dict(kind=kind, atm=rng.choice(["solar", "magnetic"] if sphere else ["solar", "cooldwarf", "magnetic"]),
                    nwl=_log(rng, 500, 100000 if sphere else 480000), nmu=rng.randint(1, 9), sphere=sphere)
    return dict(kind=kind, nwl=_log(rng, 2000, 200000), resol=float(_log(rng, 60000, 400000)), nmu=rng.randint(3, 9),
                vsini=rng.choice([0.0, rng.uniform(2.0, 40.0)]), vmacro=rng.uniform(0.5, 8.0),
                vgau=rng.choice([0.0, 48000.0, 90000.0]))


# ---- inputs --------------------------------------------------------------------------------------------

def _atmosphere(name):
    d = np.load(os.path.join(_DATA, "atm_%s.npz" % name))
    st = {k: d[k] for k in _STATE}
    st["frac_h2"] = d["frac_h2"] if "frac_h2" in d.files else np.zeros(len(d["T"]), np.float32)
    return st, {k: d[k] for k in ("cont_wave", "cont_opac", "vmicro", "molbrd", "species")}


def _contopac(meta, wave):
    """Continuum opacity [nwl][ntau] at absolute wavelengths, log-linear between the knots (on the device)."""
    x = torch.from_numpy(np.ascontiguousarray(meta["cont_wave"])).to(DEV)
    y = torch.from_numpy(np.log(meta["cont_opac"])).to(DEV)
    w = torch.from_numpy(np.ascontiguousarray(wave)).to(DEV).clamp(x[0], x[-1])
    i = torch.clamp(torch.searchsorted(x, w, right=True) - 1, 0, len(x) - 2)
    f = ((w - x[i]) / (x[i + 1] - x[i]))[:, None]
    return torch.exp(y[i] * (1.0 - f) + y[i + 1] * f).contiguous()


def _grid(case):
    """(wmode, wstart, wend, dstep) of a case: linear steps [A], or steps of c / R in ln lambda."""
    k = case["kind"]
    if k == "dense":
        return 1, 5000.0, case["wend"], 2.99792458e5 / case["resol"]
    if k == "fit":
        return 0, 4800.0, 4800.0 + case["span"], case["dstep"]
    if k == "solve":
        w0 = _WSTART[case["atm"]]
        if case["atm"] == "cooldwarf":
            return 1, w0, w0 * math.exp((case["nwl"] - 0.5) / 3e5), 2.99792458e5 / 3e5
        return 0, w0, w0 + (case["nwl"] - 0.5) * 0.002, 0.002
    if k == "broaden":
        return 1, 5000.0, 5000.0 * math.exp((case["nwl"] - 0.5) / case["resol"]), 2.99792458e5 / case["resol"]
    w0 = _WSTART["magnetic" if k == "stokes" else "solar"]
    return 0, w0, w0 + (case["nwl"] - 0.5) * case["dstep"], case["dstep"]


def _context(case, atm, grid, prec="mixed", **kw):
    st, meta = _atmosphere(atm)
    C = F.Context(precision=F.PREC_FP64 if prec == "fp64" else F.PREC_MIXED, vmicro=float(meta["vmicro"]),
                  molbrd=int(meta["molbrd"]), **kw)
    C.set_grid(*grid)
    C.set_atmosphere(st)
    co = _contopac(meta, C.wave + grid[1])
    torch.cuda.synchronize()
    C.set_contopac_dev(co.data_ptr())
    x, w, r = F.mu_quadrature(1, case["nmu"])
    C.set_mu(x, w)
    return C, st, meta, r


def _device_molecular(n, wmin, wmax, seed):
    """The cool-dwarf list's distributions (workloads.molecular_lines) drawn on the device, in wavelength order."""
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    f32 = dict(dtype=torch.float32, device=DEV)
    sig = torch.empty(n, dtype=torch.float64, device=DEV).uniform_(1e8 / wmax, 1e8 / wmin, generator=g)
    d = {"wl": torch.sort(1e8 / sig)[0]}
    d["spc"] = torch.randint(0, 4, (n,), generator=g, device=DEV, dtype=torch.int32)
    d["gf"] = torch.pow(10.0, torch.empty(n, **f32).normal_(-5.0, 1.5, generator=g))
    d["elo"] = torch.empty(n, **f32).exponential_(1.0, generator=g).clamp_(max=5.0)
    d["gvdw"] = torch.pow(10.0, torch.empty(n, **f32).uniform_(-8.0, -7.0, generator=g))
    d["grad"], d["gqst"] = torch.zeros(n, **f32), torch.zeros(n, **f32)
    d["ismol"] = torch.ones(n, dtype=torch.int32, device=DEV)
    return d


def _opacity(co, T, seed):
    """A line opacity spectrum [nwl][ntau] over the continuum co: three groups of lines, each a smoothed
    field of spikes with log-normal strengths, that change with depth as levels at 0, 2 and 5 eV do."""
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    n = co.shape[0]
    k = torch.arange(n, dtype=torch.float64, device=DEV)
    k = torch.minimum(k, n - k)
    Tt = torch.from_numpy(np.ascontiguousarray(T)).to(DEV)
    out = torch.zeros_like(co)
    for elow, width in ((0.0, 9.0), (2.0, 6.0), (5.0, 7.0)):
        spike = (torch.rand(n, generator=g, device=DEV, dtype=torch.float64) < 0.02) * \
            10.0 ** torch.empty(n, dtype=torch.float64, device=DEV).normal_(0.3, 1.3, generator=g)
        kern = torch.exp(-(k / width) ** 2) + 0.01 / (1.0 + (k / width) ** 2)
        s = torch.fft.irfft(torch.fft.rfft(spike) * torch.fft.rfft(kern), n=n).clamp_(min=1e-9)
        b = torch.exp(-elow * 11604.518 * (1.0 / Tt - 1.0 / 6000.0))
        out += s[:, None] * (b / (1.0 + b))[None, :]
    return (out * co).contiguous()


def _observed(arr, nwl, dstep, w0, seed):
    """An observed normalised spectrum of a list: absorption at its lines with signal to noise 300."""
    pix = np.clip(((arr["wl"] - w0) / dstep).astype(np.int64), 0, nwl - 1)
    s = np.bincount(pix, weights=np.minimum(arr["gf"].astype(np.float64) * 10.0 ** (-0.5 * arr["elo"]) * 3e2, 50.0),
                    minlength=nwl)
    k = np.minimum(np.arange(nwl), nwl - np.arange(nwl)) * dstep
    tau = np.fft.irfft(np.fft.rfft(s) * np.fft.rfft(np.exp(-(k / 0.03) ** 2)), n=nwl)
    noise = np.random.default_rng(seed + 1).normal(0.0, 1.0 / 300.0, nwl)
    return torch.from_numpy(0.1 + 0.9 * np.exp(-np.maximum(tau, 0.0)) + noise).to(DEV)


def _bfield(case):
    if case["bframe"] == 0:
        return np.array([1500.0, 400.0, -900.0])
    if case["bframe"] == 1:
        return np.array([2000.0, 60.0, 30.0])
    a = np.linspace(20.0, 70.0, case["nmu"])
    return np.concatenate([[1800.0], np.stack([a, 2.0 * a], 1).ravel()])


def _sphere(st):
    """(radius [cm], layer heights [cm]): a star of 250 times the model's own thickness."""
    h = W.model_heights(st["rhox"], st["rho"])
    return 250.0 * float(h[0] - h[-1]), h


def _tables(nwl, nmu):
    e = lambda *s: torch.empty(s, dtype=torch.float64, device=DEV)  # noqa: E731
    return dict(spl=e(nwl, nmu), spc=e(nwl, nmu), sfl=e(nwl), sfc=e(nwl))


def _batch_lines(case, seed):
    return W.atomic_lines(case["nlines"], 3000.0, 9000.0, seed, exact=False).arrays()


def prepare(case, seed):
    k, grid = case["kind"], None if case["kind"] == "batch" else _grid(case)
    if k == "scalar":
        C, _, _, _ = _context(case, "solar", grid, case["prec"])
        a = W.atomic_lines(case["nlines"], grid[1], grid[2], seed, exact=False).arrays()
        return dict(case=case, C=C, lines=F.LineList.from_arrays(a))
    if k == "dense":
        C, _, _, _ = _context(case, "cooldwarf", grid, limitram_gb=16.0)
        dt = _device_molecular(case["nlines"], grid[1], grid[2], seed)
        return dict(case=case, C=C, lines=GpuBackend(F, C, dt), out=_tables(C.nwl, case["nmu"]))
    if k == "batch":
        ctxs = []
        x, w, _ = F.mu_quadrature(1, case["nmu"])
        for m in W.batch_grid(case["natm"], case["grid"]):
            C = F.Context(vmicro=1.0)
            C.set_grid(**m["grid"])
            C.set_atmosphere(m["state"])
            C.set_contopac(_contopac(m["cont"], C.wave + m["grid"]["wstart"]).cpu().numpy())
            C.set_mu(x, w)
            ctxs.append(C)
        B = F.Batch(ctxs, F.LineList.from_arrays(_batch_lines(case, seed)))
        B.tune()
        return dict(case=case, B=B)
    if k == "fit":
        st, meta = _atmosphere("solar")
        a = W.atomic_lines(case["nlines"], grid[1], grid[2], seed, exact=False).arrays()
        wave = F.make_grid(*grid)
        M = AD.FluxModel(F, dict(wmode=grid[0], wstart=grid[1], wend=grid[2], dstep=grid[3]), st,
                         _contopac(meta, wave + grid[1]).cpu().numpy(), a, [str(s) for s in meta["species"]],
                         vmicro=float(meta["vmicro"]), nmu=case["nmu"])
        p = [torch.from_numpy(np.log10(a["gf"])).to(DEV), torch.zeros(len(AD.ELEMENTS), device=DEV),
             torch.tensor(float(meta["vmicro"]), device=DEV)]
        return dict(case=case, M=M, p=[v.requires_grad_(True) for v in p],
                    obs=_observed(a, len(wave), grid[3], grid[1], seed))
    if k == "stokes":
        C, _, _, _ = _context(case, "magnetic", grid, case["prec"])
        L = W.zeeman_lines(case["nlines"], grid[1], grid[2], seed)
        z = W.zeeman_components(L, F.zeeman_pattern)
        return dict(case=case, C=C, lines=F.LineList.from_arrays(L.arrays(), zeeman=z), bfield=_bfield(case))
    if k == "solve":
        C, st, meta, _ = _context(case, case["atm"], grid)
        if case["sphere"]:
            C.set_geometry(*_sphere(st))
        C.lineop_set(_opacity(_contopac(meta, C.wave + grid[1]), st["T"], seed).cpu().numpy())
        return dict(case=case, C=C, out=_tables(C.nwl, case["nmu"]))
    # broaden: intensities of a kept spectrum, limb-darkened
    C = F.Context()
    C.set_grid(*grid)
    x, w, r = F.mu_quadrature(1, case["nmu"])
    C.set_mu(x, w)
    spl, spc = _intensities(C.nwl, x, seed)
    return dict(case=case, C=C, r=r, spl=spl, spc=spc, sfl=torch.empty_like(spl[:, 0]), sfc=torch.empty_like(spl[:, 0]))


def _intensities(nwl, xmu, seed):
    mu = torch.from_numpy(xmu).to(DEV)
    one = torch.ones(nwl, 1, dtype=torch.float64, device=DEV)
    tau = _opacity(one, np.array([6000.0]), seed)[:, 0]
    spc = (1e6 * (0.4 + 0.6 * mu))[None, :] * (1.0 + 0.1 * torch.cos(torch.arange(nwl, device=DEV) * 1e-4))[:, None]
    spl = spc * (0.15 + 0.85 / (1.0 + tau[:, None] * (0.7 + 0.3 * mu)[None, :]))
    return spl.contiguous(), spc.contiguous()


# ---- one pass --------------------------------------------------------------------------------------------

def run(state):
    case = state["case"]
    k = case["kind"]
    if k == "scalar":
        C = state["C"]
        C.lineop_reset()
        r = C.lineop_calc(state["lines"], want_lineopac=False, want_linstr=case["linstr"])
        spl, spc, sfl, sfc = C.radtran()
        out = dict(spl=spl, spc=spc, sfl=sfl, sfc=sfc, flags=r["flags"], ileft=r["ileft"], iright=r["iright"])
        if case["linstr"]:
            out["linstr"] = r["linstr"]
        return out
    if k == "dense":
        C, o = state["C"], state["out"]
        C.lineop_reset()
        C.lineop_calc_dev(state["lines"].full)
        C.radtran_dev(*[o[q].data_ptr() for q in ("spl", "spc", "sfl", "sfc")])
        return o
    if k == "batch":
        state["B"].run()
        return [state["B"].flux(i) for i in range(case["natm"])]
    if k == "fit":
        p = state["p"]
        for v in p:
            v.grad = None
        f = AD.synth_flux(state["M"], *p)
        chi2 = (((f - state["obs"]) * 300.0) ** 2).sum()
        chi2.backward()
        return dict(flux=f.detach(), chi2=chi2.detach(), loggf=p[0].grad, abund=p[1].grad, vmicro=p[2].grad)
    if k == "stokes":
        C, b = state["C"], state["bfield"]
        F.lib().fsg_mag_lineop_reset(C.h)
        r = C.mag_lineop_calc(state["lines"], case["bframe"], b, want=False)
        spz, spc, sfl, sfc = C.mag_radtran(case["bframe"], b)
        return dict(spz=spz, spc=spc, sfl=sfl, sfc=sfc, flags=r["flags"], ileft=r["ileft"], iright=r["iright"])
    if k == "solve":
        o = state["out"]
        state["C"].radtran_dev(*[o[q].data_ptr() for q in ("spl", "spc", "sfl", "sfc")])
        return o
    state["C"].disk_integ_conv_dev(state["r"], case["vsini"], case["vmacro"], case["vgau"],
                                   *[state[q].data_ptr() for q in ("spl", "spc", "sfl", "sfc")])
    return dict(sfl=state["sfl"], sfc=state["sfc"])


# ---- the work of a pass ----------------------------------------------------------------------------------

def _window(atm, w0, w1):
    """Mean window [A] of a list's lines (rejected ones count 0) on a grid from w0 to w1, which cuts the widest ones
    short: measured on the lists of workloads.py; it hardly depends on the seed."""
    if atm == "cooldwarf":
        return min(w1 - w0, 0.0063 * 0.5 * (w0 + w1) * ((w1 - w0) / 20000.0) ** 0.4)
    return min(w1 - w0, (4.5 if atm == "magnetic" else 3.5) * ((w1 - w0) / 10.0) ** 0.55)


def work(case):
    """Bytes: lists, continuum opacity and results once each.  Flops: 12 for a line profile at a point, 60 for a
    step of the scalar solver, 900 for one of the polarised solver."""
    k, nmu = case["kind"], case["nmu"]
    if k == "batch":
        nwl, ntau, n = 1.0e4, 64, case["nlines"] * 110.0 / 6000.0
        ev = n * ntau * _window("solar", 6000.0, 6110.0) / 0.0115
        return dict(bytes=case["natm"] * (n * 36 + nwl * (ntau + 2) * 8),
                    flops=case["natm"] * (12 * ev + nwl * ntau * nmu * 2 * 60))
    wmode, w0, w1, step = _grid(case)
    nwl = int((w1 - w0) / step) + 1 if wmode == 0 else int(math.log(w1 / w0) * 2.99792458e5 / step) + 1
    if k == "broaden":
        taps = sum(1.0 + 2.0 * v / step for v in (case["vsini"] * 0.7, 7.0 * case["vmacro"])) * nmu
        return dict(bytes=nwl * (2 * nmu + 2) * 8, flops=nwl * taps * 4)
    atm = {"dense": "cooldwarf", "stokes": "magnetic"}.get(k, case.get("atm", "solar"))
    ntau = dict(solar=56, cooldwarf=71, magnetic=56)[atm]
    solve = nwl * ntau * nmu * 2 * 60.0 * (2.0 if case.get("sphere") else 1.0)
    if k == "solve":
        return dict(bytes=nwl * (2 * ntau + 2 * nmu + 2) * 8, flops=solve)
    pixel = 0.5 * (w0 + w1) * step / 2.99792458e5 if wmode else step
    n = case["nlines"]
    ev = n * ntau * max(1.0, _window(atm, w0, w1) / pixel)
    if k == "stokes":
        return dict(bytes=n * 300 + nwl * (ntau + 5 * nmu + 2) * 8, flops=9 * 20 * ev + nwl * ntau * nmu * 900.0)
    if k == "fit":
        return dict(bytes=n * 60 + nwl * (2 * ntau + 4) * 8, flops=(12 + 24) * ev + 3 * solve)
    return dict(bytes=n * 36 + nwl * (ntau + 2 * nmu + 2) * 8, flops=12 * ev + solve)


# ---- the same in 64 bits, in plain torch -------------------------------------------------------------------

_C, _H, _KB, _PI = 299792.458, 6.62607015e-27, 1.380649e-16, math.pi


def _t(a):
    return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float64)).to(DEV)


def _voigt_table():
    """H(a, v) on the table's nodes: v = 0.008 i, sqrt(a) = sqrt(8) j / 400, stored in single precision."""
    v = torch.arange(1002, dtype=torch.float64, device=DEV) * 0.008
    a = (torch.arange(402, dtype=torch.float64, device=DEV) * (math.sqrt(8.0) / 400)) ** 2
    z = torch.complex(v[None, :].expand(401, -1).contiguous(), a[1:, None].expand(-1, 1002).contiguous())
    s = 1.0 / z
    for n in range(1, 17):
        s = s + 2.0 * z * math.exp(-0.25 * n * n) / (z * z - 0.25 * n * n)
    w = 1j * s * (0.5 / _PI)
    pole = 2.0 * torch.exp(-z * z) / (1.0 - torch.exp(-4j * _PI * z))
    w = torch.where(z.imag < 6.0, w + pole, w)
    return torch.cat([torch.exp(-v * v)[None, :], w.real]).float(), a


def _hvoigt(tab, a, v):
    """H(a, v): the table inside a < 8, |v| < 8, two rational forms outside."""
    t, node = tab
    v = v.abs()
    a2, v2 = a * a, v * v
    s = v2 + a2
    far = a * (s + 0.5) / (s * s - v2 + a2 + 0.25)
    p, q = v2 - a2 - 1.5, 2.0 * v * a
    dr, di = v * p - a * q, v * q + a * p
    h = torch.where(s >= 196.0, far, ((p + 0.5) * di - q * dr) / (dr * dr + di * di)) / math.sqrt(_PI)
    m = (a < 8.0) & (v < 8.0)
    am, vm = a[m], v[m]
    ia = (torch.sqrt(am) * (400 / math.sqrt(8.0))).long()
    ua = (am - node[ia]) / (node[ia + 1] - node[ia])
    fv = vm * 125.0
    iv = fv.long()
    fv = fv - iv
    f = t.reshape(-1)
    lerp = lambda i: f[i].double() + fv * (f[i + 1] - f[i]).double()  # noqa: E731
    c0, c1 = lerp(ia * 1002 + iv), lerp((ia + 1) * 1002 + iv)
    h[m] = c0 + ua * (c1 - c0)
    return h


def _line_depths(st, a, wl, vmicro):
    """(LinCop, 1 / Doppler width, damping) [n][ntau] of atomic lines with Stark and van der Waals data."""
    T, xne, rho = (_t(st[k]) for k in ("T", "xne", "rho"))
    c = _C * 1e13
    spc = torch.from_numpy(np.asarray(a["spc"], np.int64)).to(DEV)
    col = lambda v: _t(v)[:, None]  # noqa: E731
    wl = wl[:, None]
    stim = 1.0 - torch.exp(-(c * _H / wl) / (_KB * T))
    exc = torch.exp(-col(a["elo"]) / (_KB * 1e-7 / 1.602176634e-19 * T))
    mass = 2.0 * _KB / (1.66053906660e-27 * 1e3) * 1e16 / c / c / _t(st["xamass"])[spc][:, None]
    dop = torch.sqrt(T * mass + 1e26 / c / c * vmicro * vmicro)
    z = math.sqrt(_PI) * 4.803204712e-10 ** 2 / (9.1093837139e-28 * _C ** 2) * 1e-18
    cop = z * exc * col(a["gf"]) * stim / (rho * dop / wl) * _t(st["fractionpf"]).T[spc]
    npb = _t(st["frac_h1"]) + 0.412265 * _t(st["frac_he1"])
    gam = col(a["grad"]) + col(a["gqst"]) * ((T / 1e4) ** (1.0 / 6.0) * xne) + col(a["gvdw"]) * ((T / 1e4) ** 0.3 * npb)
    return cop, 1.0 / (wl * dop), gam / (dop / wl * (4.0 * c * _PI))


def _wave_index(w, grid, nwl):
    wmode, w0, _, step = grid
    if wmode == 0:
        return (w / step).clamp(0.0, nwl - 2.0).long()
    return (torch.log((w / w0 + 1.0).clamp(min=1e-300)) / (step / _C)).clamp(0.0, nwl - 2.0).long()


def _ray(m, idx, x, y, start):
    """Emergent intensity along one ray: column mass m and layer idx of its points (outside in), opacity x and
    source function y by layer [nwl][ntau], start: whether the far end emits."""
    X, Y, n = x[:, idx], y[:, idx], len(m)

    def slope(dx, dx1, d0, d1):
        lam = (1.0 + dx1 / (dx + dx1)) / 3.0
        return torch.where(d0 * d1 > 0.0, d0 / (lam * d1 + (1.0 - lam) * d0) * d1, torch.zeros_like(d0))

    dm = m[1:] - m[:-1]
    dX = (X[:, 1:] - X[:, :-1]) / dm
    g = torch.cat([dX[:, :1], slope(dm[:-1], dm[1:], dX[:, :-1], dX[:, 1:])], 1)
    tau = dm * (X[:, 1:] + 2.0 * X[:, :-1] + dm / 2.0 * g) / 3.0
    dY = (Y[:, 1:] - Y[:, :-1]) / tau
    r = torch.cat([dY[:, :1], slope(tau[:, :-1], tau[:, 1:], dY[:, :-1], dY[:, 1:]), dY[:, -1:]], 1)
    u = 0.5 * (Y[:, :-1] + 0.5 * tau * r[:, :-1] + Y[:, 1:] - 0.5 * tau * r[:, 1:])
    inten = Y[:, n - 1].clone() if start else torch.zeros_like(Y[:, 0])
    for k in range(n - 2, -1, -1):
        d = tau[:, k]
        e = torch.exp(-d) * (d < 100.0)
        i2 = 1.0 / (d * d)
        thin = d < 5e-3
        d2 = d * d
        eps = torch.where(thin, 1.0 - d + 0.5 * d2 - d2 * d / 6.0 + d2 * d2 / 24.0, e)
        al = torch.where(thin, d / 3.0 - d2 / 12.0 + d2 * d / 60.0, (d2 - 2.0 * d + 2.0 - 2.0 * e) * i2)
        be = torch.where(thin, d / 3.0 - d2 * 0.25 + d2 * d * 0.1, (2.0 - (2.0 + 2.0 * d + d2) * e) * i2)
        ga = torch.where(thin, d / 3.0 - d2 / 6.0 + d2 * d * 0.05, (2.0 * d - 4.0 + (2.0 * d + 4.0) * e) * i2)
        inten = inten * eps + al * Y[:, k] + be * Y[:, k + 1] + ga * u[:, k]
    return inten


def _rays(rhox, xmu, sphere):
    """(column mass, layer, starts from the source function) of the ray of each angle."""
    n = len(rhox)
    out = []
    for mu in xmu:
        if sphere is None:
            out.append((_t(rhox / mu), torch.arange(n, device=DEV), True))
            continue
        r = sphere[0] + sphere[1]
        p = r[0] * math.sqrt((1.0 - mu) * (1.0 + mu))
        deep = n if p <= r[-1] else int(np.argmax(p >= r))
        z = np.sqrt((r[:deep] - p) * (r[:deep] + p))
        s = np.diff(rhox[:deep]) * (r[1:deep] + r[:deep - 1]) / (z[1:] + z[:-1])
        idx = np.arange(deep)
        if deep < n:
            chord = 2.0 * z[-1] * (rhox[deep] - rhox[deep - 1]) / (r[deep - 1] - r[deep])
            s, idx = np.concatenate([s, [chord], s[::-1]]), np.concatenate([idx, idx[::-1]])
        out.append((_t(np.concatenate([[0.0], np.cumsum(s)]) + rhox[0] / mu), torch.from_numpy(idx).to(DEV), deep == n))
    return out


def _planck(wl, T):
    return torch.exp(50.7649141 - 5.0 * torch.log(wl))[:, None] / \
        (torch.exp((_H * _C * 1e13 / _KB / wl)[:, None] / T) - 1.0)


def _spectrum(st, wave, co, lo, xmu, wmu, sphere=None):
    """Intensities and fluxes of opacities co and co + lo [nwl][ntau]."""
    y = _planck(_t(wave), _t(st["T"]))
    rays = _rays(np.asarray(st["rhox"], np.float64), xmu, sphere)
    sp = lambda x: torch.stack([_ray(m, i, x, y, s) for m, i, s in rays], 1)  # noqa: E731
    spl, spc = sp(co + lo), sp(co)
    w = _t(wmu)
    return dict(spl=spl, spc=spc, sfl=spl @ w, sfc=spc @ w)


def _line_opacity(st, meta, a, grid, wave, co, vmicro, eps=1e-4):
    """(LineOpac [nwl][ntau], retained lines, per-depth rows of the lines): every line over its window."""
    tab = _voigt_table()
    nwl = len(wave)
    off = _t(wave - grid[1])
    wc = _t(a["wl"]) - grid[1]
    cop, vv, av = _line_depths(st, a, wc + grid[1], vmicro)
    i = _wave_index(wc, grid, nwl)
    f = ((wc - off[i]) / (off[i + 1] - off[i]))[:, None]
    cc = co[i] * (1.0 - f) + co[i + 1] * f
    keep = ((cop / cc).amax(1) >= eps) & ((_hvoigt(tab, av, torch.zeros_like(av)) * cop / cc).amax(1) >= eps)
    r = cop / (eps * cc)
    half = torch.sqrt(torch.log(r.clamp(min=1.0)) + (av * (r / math.sqrt(_PI) - av)).clamp(min=0.0)) / vv
    half = torch.where(r > 1.0, half, torch.zeros_like(half)).amax(1)
    il = _wave_index(wc - half, grid, nwl)
    ir = (_wave_index(wc + half, grid, nwl) + 1).clamp(max=nwl - 1)
    lo = torch.zeros_like(co)
    sel = torch.nonzero(keep)[:, 0]
    ends = torch.cumsum(ir[sel] - il[sel] + 1, 0).cpu().numpy()
    most, at = 40000000 // co.shape[1], 0
    while at < len(sel):                      # lines whose windows have about `most` points together
        base = int(ends[at - 1]) if at else 0
        to = max(at + 1, int(np.searchsorted(ends, base + most)))
        s = sel[at:to]
        line = torch.repeat_interleave(s, ir[s] - il[s] + 1)
        pix = torch.arange(len(line), device=DEV) - \
            torch.repeat_interleave(_t(ends[at:to] - base).long() - (ir[s] - il[s] + 1), ir[s] - il[s] + 1) + il[line]
        for q in range(0, len(line), most):
            n, p = line[q:q + most], pix[q:q + most]
            lo.index_add_(0, p, _hvoigt(tab, av[n], (off[p] - wc[n])[:, None] * vv[n]) * cop[n])
        at = to
    return lo, keep, (cop, av, cc, tab, wc)


def _broadened(case, grid, xmu, wmu, r, spl, spc):
    """Rotation and macroturbulence of each annulus, their sum, then the instrumental profile."""
    nwl, dv = spl.shape[0], grid[3]
    area = lambda R, V: 0.5 * (np.clip(V, -R, R) * np.sqrt(np.maximum(0.0, R * R - np.clip(V, -R, R) ** 2)) +  # noqa: E731
                               R * R * np.arcsin(np.clip(V / R, -1.0, 1.0))) if R > 0.0 else 0.0 * V
    gauss = lambda s, j: np.exp(np.maximum(-20.0, -0.5 * (np.arange(-j, j + 1) / s) ** 2))  # noqa: E731

    def conv(f, k):
        k = _t(k / k.sum())
        p = (len(k) - 1) // 2
        f = torch.nn.functional.pad(f[:, None, :], (p, len(k) - 1 - p), mode="replicate")[:, 0, :]
        out = torch.zeros(2, nwl, dtype=torch.float64, device=DEV)
        for j in range(len(k)):
            out += f[:, j:j + nwl] * k[j]
        return out

    sig = case["vmacro"] / dv / math.sqrt(2.0)
    j = max(3, min(int(10.0 * sig), (nwl - 3) // 2))
    flux = torch.zeros(2, nwl, dtype=torch.float64, device=DEV)
    for m in range(len(xmu)):
        f = torch.stack([spl[:, m], spc[:, m]])
        r1, r2 = case["vsini"] * r[m], case["vsini"] * r[m + 1]
        if r2 > 0.5 * dv:
            n = 2 * int(r2 / dv) + 3
            v = np.abs(dv * (np.arange(n) - (n - 1) // 2))
            f = conv(f, area(r2, v + 0.5 * dv) - area(r2, v - 0.5 * dv) - area(r1, v + 0.5 * dv) + area(r1, v - 0.5 * dv))
        if case["vmacro"] > 0.0:
            k = [gauss(sig * q, j) if q > 0.0 else (np.arange(-j, j + 1) == 0) * 1.0
                 for q in (xmu[m], math.sqrt(1.0 - xmu[m] ** 2))]
            f = conv(f, 0.5 * k[0] / k[0].sum() + 0.5 * k[1] / k[1].sum())
        flux += f * float(wmu[m])
    if case["vgau"] > 0.0:
        s = (_C / case["vgau"] if case["vgau"] > 1000.0 else case["vgau"]) / dv / (2.0 * math.sqrt(2.0 * math.log(2.0)))
        flux = conv(flux, gauss(s, max(3, min(int(10.0 * s), int((nwl - 3.0) / 2.0)))))
    return dict(sfl=flux[0], sfc=flux[1])


def _wave(grid):
    wmode, w0, w1, step = grid
    n = int(((w1 - w0) / step if wmode == 0 else math.log(w1 / w0) / (step / _C)) + 1e-12) + 1
    i = np.arange(n, dtype=np.float64)
    return w0 + i * step if wmode == 0 else w0 * np.exp(i * (step / _C))


def _angles(n):
    """Cosines, flux weights and projected annulus radii of the Gauss-Legendre quadrature over the disk."""
    if n == 1:
        return np.array([1.0]), np.array([1.0]), np.array([0.0, 1.0])
    x, w = np.polynomial.legendre.leggauss(n)
    x, w = 0.5 * (x[::-1] + 1.0), w[::-1]
    return x, w * x, np.concatenate([[0.0], np.sqrt(np.cumsum(w * x)[:-1]), [1.0]])


def exact(case, seed):
    """The outputs in 64 bits.  None for line lists whose profiles take minutes this way (molecular lists, large
    grids of atmospheres), for gradients (their window edges have no plain form) and for polarised spectra (a
    search for every line's window, then minutes)."""
    k = case["kind"]
    if k == "scalar":
        grid = _grid(case)
        st, meta = _atmosphere("solar")
        wave = _wave(grid)
        co = _contopac(meta, wave)
        a = W.atomic_lines(case["nlines"], grid[1], grid[2], seed, exact=False).arrays()
        lo, keep, (cop, av, cc, tab, wc) = _line_opacity(st, meta, a, grid, wave, co, float(meta["vmicro"]))
        x, w, _ = _angles(case["nmu"])
        out = _spectrum(st, wave, co, lo, x, w)
        out.update(flags=None, ileft=None, iright=None)
        if case["linstr"]:
            s = _spectrum(st, (wc + grid[1]).cpu().numpy(), cc, _hvoigt(tab, av, torch.zeros_like(av)) * cop, x, w)
            d = 1.0 - (s["spl"][:, 0] / s["spc"][:, 0] if case["nmu"] == 1 else s["sfl"] / s["sfc"])
            out["linstr"] = torch.where(keep, d, torch.zeros_like(d))
        return out
    if k == "batch":
        if work(case)["flops"] > 2e11:
            return None
        out, (x, w, _), a = [], _angles(case["nmu"]), _batch_lines(case, seed)
        for m in W.batch_grid(case["natm"], case["grid"]):
            g = m["grid"]
            grid = (g["wmode"], g["wstart"], g["wend"], g["dstep"])
            wave = _wave(grid)
            co = _contopac(m["cont"], wave)
            i0, i1 = np.searchsorted(a["wl"], g["wstart"]), np.searchsorted(a["wl"], g["wend"], side="right")
            lo, _, _ = _line_opacity(m["state"], m["cont"], {q: v[i0:i1] for q, v in a.items()}, grid, wave, co, 1.0)
            s = _spectrum(m["state"], wave, co, lo, x, w)
            out.append((s["sfl"], s["sfc"]))
        return out
    if k == "solve":
        grid = _grid(case)
        st, meta = _atmosphere(case["atm"])
        wave = _wave(grid)
        co = _contopac(meta, wave)
        x, w, _ = _angles(case["nmu"])
        return _spectrum(st, wave, co, _opacity(co, st["T"], seed), x, w,
                         _sphere(st) if case["sphere"] else None)
    if k == "broaden":
        grid = _grid(case)
        x, w, r = _angles(case["nmu"])
        spl, spc = _intensities(len(_wave(grid)), x, seed)
        return _broadened(case, grid, x, w, r, spl, spc)
    return None
