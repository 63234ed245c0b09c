"""The work a user of the framework has it do, as timed cases.

Each case is one call (or the one chain of calls) that a redshift pipeline
makes through the public functions, on DESI-like spectra (cameras b/r/z at
0.8 A, 7958 pixels, 11-diagonal resolution, random masks) and the synthetic
GALAXY / QSO / STAR template set of redrock_b200.synth:

  scan      calc_zchi2_targets: chi2 of every target at every redshift of the
            templates, from host arrays to host arrays
  nmf       calc_zchi2 of a non-negative template
  build     DistTemplate: a template rebinned (and IGM-attenuated) onto the
            cameras at every redshift
  finegrid  rebin_template + transmission_Lyman + calc_zchi2_batch on a short
            redshift grid of one target: what redrock's own fitz calls after
            install()
  fitz      fitz_targets: refinement of the coarse minima of many targets
  zfind     zfind: scan, refinement and ranking
  grad      Chi2Scan: chi2 of (target, z) pairs and its backward pass to z and flux
  arch      Archetype.best_archetypes: archetype refits
  coadd     coadd_targets: exposures to one spectrum per camera

Targets of a pass are new Target objects (a pipeline fits each batch once),
templates are kept, as a program that fits batch after batch keeps them.
"""

import math
import random

import numpy as np
import scipy.sparse
import torch

from redrock_b200 import synth
from redrock_b200 import archetypes as A
from redrock_b200 import fitz as F
from redrock_b200 import rebin, zscan
from redrock_b200 import targets as T
from redrock_b200 import templates as TM
from redrock_b200.adjoint import Chi2Scan, PairContext
from redrock_b200.coadd import coadd_targets
from redrock_b200.igm import transmission_Lyman
from redrock_b200.zfind import zfind

NPIX = 7958           # pixels of the three cameras
NZ = {"GALAXY": 3311, "QSO": 3794, "STAR": 100, "NMF": 3311}
NB = {"GALAXY": 10, "QSO": 4, "STAR": 5, "NMF": 5}
NSTAR = 5


def listed():
    return [
        # one object looked at by hand, or a survey's last odd one: latency
        {"name": "scan 1", "op": "scan", "n": 1, "kinds": "all", "mask": 0.05, "drop": 0.0},
        # the targets of a small tile or of one fibre bundle
        {"name": "scan 37", "op": "scan", "n": 37, "kinds": "all", "mask": 0.05, "drop": 0.0},
        # a large batch with uneven masks and missing cameras: throughput
        {"name": "scan 800 uneven", "op": "scan", "n": 800, "kinds": "all", "mask": 0.4,
         "drop": 0.1},
        # NMF galaxy templates (redrock's second template method): bounded solves
        {"name": "scan nmf 7", "op": "nmf", "n": 7, "mask": 0.05},
        # start of a run: templates onto the cameras, without and with IGM
        {"name": "build galaxy", "op": "build", "kind": "GALAXY", "nz": 3311},
        {"name": "build qso", "op": "build", "kind": "QSO", "nz": 3794},
        # redrock's own fitz on the rebound functions: many such small calls per target
        {"name": "fine grid 15", "op": "finegrid", "kind": "GALAXY", "nz": 15, "mask": 0.05},
        # refinement of a batch's minima with one template
        {"name": "fitz 100", "op": "fitz", "n": 100, "kind": "GALAXY", "nminima": 3, "mask": 0.05},
        # the whole redshift fit of a batch
        {"name": "zfind 48", "op": "zfind", "n": 48, "nminima": 3, "mask": 0.05, "graph": False},
        # gradient of chi2 for continuous-z fits and flux sensitivities
        {"name": "grad 64x6", "op": "grad", "n": 64, "per": 6, "kind": "GALAXY", "mask": 0.05},
        # archetype refits of refined redshifts
        {"name": "arch 60x24", "op": "arch", "n": 60, "narch": 24, "mask": 0.05},
        # exposures of a night coadded with cosmic-ray rejection
        {"name": "coadd 24x3", "op": "coadd", "n": 24, "nexp": 3, "nsig": 4.0, "mask": 0.05},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["scan", "scan", "scan", "nmf", "build", "finegrid", "fitz", "zfind", "grad",
                     "arch", "coadd"])
    mask = round(rng.uniform(0.0, 0.4), 3)
    if op == "scan":
        kinds = rng.choice(["all", "all", "GALAXY", "QSO", "STAR"])
        n = _log_int(rng, 1, 700)
        return {"op": op, "n": n, "kinds": kinds, "mask": mask,
                "drop": 0.1 if n >= 400 else 0.0}
    if op == "nmf":
        return {"op": op, "n": _log_int(rng, 1, 24), "mask": mask}
    if op == "build":
        kind = rng.choice(["GALAXY", "QSO", "STAR"])
        return {"op": op, "kind": kind, "nz": _log_int(rng, 11, NZ[kind])}
    if op == "finegrid":
        return {"op": op, "kind": rng.choice(["GALAXY", "QSO", "STAR"]),
                "nz": rng.choice([1, 7, 15, 15, 31]), "mask": mask}
    if op == "fitz":
        return {"op": op, "n": _log_int(rng, 1, 150), "kind": rng.choice(["GALAXY", "QSO", "STAR"]),
                "nminima": rng.choice([1, 3, 5]), "mask": mask}
    if op == "zfind":
        return {"op": op, "n": _log_int(rng, 1, 100), "nminima": rng.choice([2, 3]), "mask": mask,
                "graph": rng.random() < 0.3}
    if op == "grad":
        return {"op": op, "n": _log_int(rng, 1, 100), "per": rng.randint(1, 8),
                "kind": rng.choice(["GALAXY", "QSO", "STAR"]), "mask": mask}
    if op == "arch":
        return {"op": op, "n": _log_int(rng, 1, 80), "narch": _log_int(rng, 5, 60), "mask": mask}
    return {"op": op, "n": _log_int(rng, 1, 40), "nexp": rng.randint(2, 5),
            "nsig": rng.choice([0.0, 2.5, 4.0]), "mask": mask}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
_KEEP = {}


def _specs():
    """The synthetic template set, and a non-negative galaxy set of five."""
    if "specs" not in _KEEP:
        s = synth.template_set()
        w = s[0].wave
        g = lambda c, sig: np.exp(-0.5 * ((w - c) / sig) ** 2)  # noqa: E731
        rip = lambda p: 0.3 * (1.0 + np.sin(2.0 * np.pi * w / p))  # noqa: E731
        old = (w / 5000.0) ** 0.5 / (1.0 + np.exp((4000.0 - w) / 40.0)) + 0.05
        nmf = [old * (1.0 - 0.4 * g(5175.0, 12.0)), (w / 4000.0) ** -2.0, (w / 6000.0) ** -0.6,
               rip(480.0) + g(3726.0, 2.0) + 1.3 * g(3728.8, 2.0) + 0.6 * g(4861.3, 2.0),
               rip(770.0) + g(4958.9, 2.0) + 3.0 * g(5006.8, 2.0) + 1.5 * g(6562.8, 2.5)]
        spec = synth.TemplateSpec("GALAXY", "", w, np.stack(nmf), s[0].redshifts, "Inoue14",
                                  method="NMF")
        _KEEP["specs"] = {"GALAXY": [s[0]], "QSO": [s[1]], "STAR": s[2:], "NMF": [spec],
                          "all": s}
    return _KEEP["specs"]


def _grids():
    if "grids" not in _KEEP:
        _KEEP["grids"] = synth.camera_grids()
    return _KEEP["grids"]


def _resolution(npix, sigma):
    """Gaussian 11-diagonal resolution, rows normalised, scipy DIA layout."""
    off = np.arange(-5, 6)
    kern = np.exp(-0.5 * (off / sigma) ** 2)
    rows = np.arange(npix)[None, :] - off[:, None]          # data[k, j] = R[j - off, j]
    ok = (rows >= 0) & (rows < npix)
    csum = np.concatenate([[0.0], np.cumsum(kern)])
    i = np.arange(npix)
    norm = csum[np.minimum(10, npix - 1 - i + 5) + 1] - csum[np.maximum(0, 5 - i)]
    return np.where(ok, kern[:, None] / norm[np.clip(rows, 0, npix - 1)], 0.0), off


def _spectra(case, seed, basis=None, positive=False, nexp=1):
    """[(spectra, true z)] of the case's targets, as plain host arrays in
    Spectrum objects."""
    rng = np.random.default_rng([int(seed), 77])
    spec = _specs()[basis or "GALAXY"][0]
    out = []
    for _ in range(case.get("n", 1)):
        z = rng.uniform(0.02, 1.4)
        c = rng.normal(size=spec.flux.shape[0])
        rest = (np.abs(c) if positive else c) @ spec.flux
        drop = int(rng.integers(3)) if rng.uniform() < case.get("drop", 0.0) else -1
        frac = case["mask"] if case["mask"] <= 0.1 else rng.uniform(0.0, case["mask"])
        sp = []
        for k, (band, wave) in enumerate(_grids().items()):
            n = len(wave)
            model = np.interp(wave / (1.0 + z), spec.wave, rest)
            for e in range(nexp):
                noise = rng.uniform(0.5, 2.0, size=n)
                ivar = 1.0 / noise ** 2
                ivar[rng.uniform(size=n) < frac] = 0.0
                flux = model + rng.normal(size=n) * noise
                if nexp > 1:
                    hit = rng.integers(n, size=4)
                    flux[hit] += rng.uniform(20.0, 200.0, size=4) * noise[hit]
                if k == drop:
                    continue
                data, off = _resolution(n, rng.uniform(0.8, 1.2))
                sp.append(T.Spectrum(wave, flux, ivar,
                                     scipy.sparse.dia_matrix((data, off), shape=(n, n)), band=band))
        out.append((sp, z))
    return out


def _targets(state):
    return [T.Target(1000 + i, sp) for i, sp in enumerate(state["spectra"])]


def _template(spec, nz=None):
    z = spec.redshifts
    if nz is not None and nz < len(z):
        z = z[np.linspace(0, len(z) - 1, nz).round().astype(int)]
    return TM.Template(spectype=spec.spectype, subtype=spec.subtype, redshifts=z, wave=spec.wave,
                       flux=spec.flux, method=spec.method, igm_model=spec.igm_model)


def _one(kind, seed):
    s = _specs()[kind]
    return s[int(seed) % len(s)]


def prepare(case, seed):
    op = case["op"]
    state = {"case": case, "seed": seed}
    if op == "build":
        # the redshift grid of another run: the same range, shifted a little
        t = _template(_one(case["kind"], seed), case["nz"])
        shift = 1e-6 * (int(seed) % 97)
        t._redshifts = t.redshifts + (shift if case["kind"] != "STAR" else 1e-3 * shift)
        state["template"] = t
        return state
    basis = "QSO" if case.get("kind") == "QSO" else "NMF" if op == "nmf" else "GALAXY"
    sp = _spectra(case, seed, basis if basis != "QSO" else "GALAXY", positive=op == "nmf",
                  nexp=case.get("nexp", 1))
    state["spectra"] = [s for s, _ in sp]
    state["z"] = np.array([z for _, z in sp])
    if op in ("scan", "nmf", "zfind"):
        kinds = "NMF" if op == "nmf" else case.get("kinds", "all")
        state["templates"] = [TM.DistTemplate(_template(s), _grids()) for s in _specs()[kinds]]
    elif op == "finegrid":
        state["template"] = _template(_one(case["kind"], seed))
        z0 = {"GALAXY": 0.05 + state["z"][0] * 0.9, "QSO": 1.0 + 2.0 * state["z"][0],
              "STAR": 1e-3 * (state["z"][0] - 0.7)}[case["kind"]]
        h = 1e-4 if case["kind"] == "STAR" else 3e-4 * (1.0 + z0)
        state["zgrid"] = np.linspace(z0 - h, z0 + h, case["nz"])
    elif op == "fitz":
        state["template"] = _template(_one(case["kind"], seed))
        dt = TM.DistTemplate(state["template"], _grids())
        tg = _targets(state)
        zc, _, pen = zscan.calc_zchi2([t.id for t in tg], tg, dt)
        state["chi2"] = [a.copy() for a in zc + pen]
        zscan.clear_caches()
    elif op == "grad":
        state["template"] = _template(_one(case["kind"], seed))
        state["ctx"] = PairContext(_targets(state), state["template"])
        rng = np.random.default_rng([int(seed), 78])
        lo, hi = {"GALAXY": (0.02, 1.5), "QSO": (0.3, 4.0), "STAR": (-1.5e-3, 1.5e-3)}[case["kind"]]
        n = case["n"] * case["per"]
        state["pair_t"] = np.repeat(np.arange(case["n"], dtype=np.int32), case["per"])
        state["pair_z"] = torch.tensor(rng.uniform(lo, hi, size=n), device="cuda")
        state["flux"] = state["ctx"].packed_flux()
        state["weight"] = torch.tensor(rng.uniform(0.5, 1.5, size=n), device="cuda")
    elif op == "arch":
        state["arch"] = A.Archetype.from_synth(synth.archetype_set(narch=case["narch"], seed=5))
        state["prior"] = F.prior_on_coeffs(1, 2, 0.1, 3)
    return state


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _whole(rows):
    """The array whose rows these are (results come as views of one array
    per template), or a stacked copy."""
    b = rows[0].base
    if isinstance(b, np.ndarray) and b.shape == (len(rows),) + rows[0].shape and \
            all(r.base is b for r in rows):
        return b
    return np.stack(rows)


def _filled(a, rows):
    """``a`` with its first axis filled up to ``rows`` (a target may have
    fewer minima than asked for): NaN, or -1 for whole numbers."""
    if len(a) >= rows:
        return a
    f = np.nan if a.dtype.kind == "f" else -1
    return np.concatenate([a, np.full((rows - len(a),) + a.shape[1:], f, dtype=a.dtype)])


def run(state):
    case = state["case"]
    op = case["op"]
    if op == "scan":
        tg = T.DistTargetsCopy(_targets(state))
        res = zscan.calc_zchi2_targets(tg, state["templates"])
        return {ft: {k: _whole([res[t.id][ft][k] for t in tg.local()])
                     for k in ("zchi2", "zcoeff", "penalty")}
                for ft in (d.template.full_type for d in state["templates"])}
    if op == "nmf":
        tg = _targets(state)
        zc, co, pen = zscan.calc_zchi2([t.id for t in tg], tg, state["templates"][0])
        return {"zchi2": zc, "zcoeff": co, "penalty": pen}
    if op == "build":
        d = TM.DistTemplate(state["template"], _grids())
        return d.basis.data_dict(as_numpy=False)
    if op == "finegrid":
        t, sp, z = state["template"], state["spectra"][0], state["zgrid"]
        w, f, wf = zscan.spectral_data(sp)
        dwave = {s.wavehash: s.wave for s in sp}
        binned = rebin.rebin_template(t, z, dwave=dwave, use_gpu=True)
        for hs, wave in dwave.items():
            tr = transmission_Lyman(z, wave, use_gpu=True, model=t.igm_model,
                                    always_return_array=False)
            if tr is not None:
                binned[hs] *= tr[:, :, None]
        zc, co = zscan.calc_zchi2_batch(sp, binned, w, f, wf, len(z), t.nbasis,
                                        t.solve_matrices_algorithm)
        return {"binned": binned, "zchi2": zc, "zcoeff": co}
    if op == "fitz":
        tg = _targets(state)
        res = F.fitz_targets(state["chi2"], state["template"].redshifts, tg, state["template"],
                             nminima=case["nminima"])
        return {k: np.concatenate([_filled(r[k], case["nminima"]) for r in res])
                for k in ("z", "zerr", "zwarn", "chi2", "zz", "zzchi2", "coeff", "npixels")}
    if op == "zfind":
        tg = T.DistTargetsCopy(_targets(state))
        _, zfit = zfind(tg, state["templates"], nminima=case["nminima"], graph=case["graph"])
        rows = case["n"] * case["nminima"] * 3           # at most, over the three spectral types
        return {k: _filled(v, rows) for k, v in zfit.items() if v.dtype.kind in "fiu"}
    if op == "grad":
        z = state["pair_z"].detach().requires_grad_(True)
        f = state["flux"].detach().requires_grad_(True)
        chi2, coeff = Chi2Scan.apply(z, f, state["ctx"], state["pair_t"])
        gz, gf = torch.autograd.grad(chi2, (z, f), state["weight"])
        return {"chi2": chi2.detach(), "coeff": coeff.detach(), "gz": gz, "gflux": gf}
    if op == "arch":
        tg = _targets(state)
        for t in tg:
            t.legendre(2)
        fits = state["arch"].best_archetypes([(t, float(z), None) for t, z in zip(tg, state["z"])],
                                             True, None, prior=state["prior"])
        return {"chi2": np.array([x[0] for x in fits]), "coeff": np.stack([x[1] for x in fits]),
                "index": np.array([int(x[2].rsplit("_", 1)[1]) for x in fits])}
    tg = _targets(state)
    coadd_targets(tg, cosmics_nsig=case["nsig"])
    sp = [s for t in tg for s in t.spectra]
    return {"flux": np.concatenate([s.flux for s in sp]),
            "ivar": np.concatenate([s.ivar for s in sp]),
            "rdata": np.concatenate([s.R.data.ravel() for s in sp])}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _eval_flops(n):
    """One chi2: 11-tap resolution of n bases, Gram, right-hand side, solve."""
    return NPIX * n * (22 + n + 3) + n ** 3 / 3 + 2 * n * n


def work(case):
    op = case["op"]
    target_bytes = NPIX * 8 * 13                       # resolution, flux, ivar
    if op in ("scan", "zfind", "nmf"):
        kinds = "NMF" if op == "nmf" else case.get("kinds", "all")
        sets = {"all": [("GALAXY", 1), ("QSO", 1), ("STAR", NSTAR)], "STAR": [("STAR", NSTAR)]}
        per_target, fl, basis = 0, 0.0, 0
        for k, m in sets.get(kinds, [(kinds, 1)]):
            per_target += m * NZ[k] * (NB[k] + 2) * 8
            basis += m * NZ[k] * NPIX * NB[k] * 8
            fl += m * NZ[k] * _eval_flops(NB[k])
            if op == "zfind":
                fl += m * case["nminima"] * 16 * (_eval_flops(NB[k]) + 20 * NPIX * NB[k])
        if op == "zfind":
            per_target = 2000
        return {"bytes": case["n"] * (target_bytes + per_target) + basis, "flops": case["n"] * fl}
    if op == "build":
        n = NB[case["kind"]]
        # about four samples to a bin: a product and a sum for each and basis
        return {"bytes": case["nz"] * NPIX * n * 8, "flops": case["nz"] * NPIX * n * 20}
    if op == "finegrid":
        n = NB[case["kind"]]
        return {"bytes": target_bytes + case["nz"] * NPIX * n * 8,
                "flops": case["nz"] * (_eval_flops(n) + 20 * NPIX * n)}
    if op == "fitz":
        n = NB[case["kind"]]
        ev = case["n"] * case["nminima"] * 16
        return {"bytes": case["n"] * (target_bytes + NZ[case["kind"]] * 8),
                "flops": ev * (_eval_flops(n) + 20 * NPIX * n)}
    if op == "grad":
        n = NB[case["kind"]]
        ev = case["n"] * case["per"]
        return {"bytes": case["n"] * (target_bytes + 2 * NPIX * 8),
                "flops": ev * (2 * _eval_flops(n) + 60 * NPIX * n)}
    if op == "arch":
        ev = case["n"] * case["narch"]
        return {"bytes": case["n"] * target_bytes, "flops": ev * NPIX * (20 + 22 + 2 * 9)}
    exp_bytes = case["n"] * case["nexp"] * NPIX * 8 * 13
    return {"bytes": exp_bytes + case["n"] * target_bytes,
            "flops": case["n"] * case["nexp"] * NPIX * 30}


# ---------------------------------------------------------------------------
# the same in plain 64-bit torch / numpy
# ---------------------------------------------------------------------------
def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _edges(w):
    e = np.empty(len(w) + 1)
    e[1:-1] = (w[:-1] + w[1:]) / 2
    e[0] = w[0] - (w[1] - e[1])
    e[-1] = w[-1] + (w[-1] - e[-2])
    return e


def _rebinned(wave, flux, z, grid):
    """(nz, nbin, nb): averages of the redshifted piecewise-linear flux over
    the grid's bins, from its running integral."""
    d = _dev()
    x = torch.tensor(np.asarray(wave), device=d)
    y = torch.tensor(np.ascontiguousarray(np.asarray(flux).T), device=d)
    cum = torch.zeros_like(y)
    cum[1:] = torch.cumsum(0.5 * (y[1:] + y[:-1]) * (x[1:] - x[:-1])[:, None], 0)
    zp1 = 1.0 + torch.tensor(np.asarray(z), device=d)
    e = torch.tensor(_edges(grid), device=d)[None, :] / zp1[:, None]
    j = (torch.searchsorted(x, e.contiguous(), right=True) - 1).clamp(0, len(x) - 2)
    t = e - x[j]
    slope = (y[j + 1] - y[j]) / (x[j + 1] - x[j])[..., None]
    c = cum[j] + t[..., None] * (y[j] + 0.5 * slope * t[..., None])
    return (c[:, 1:] - c[:, :-1]) / (e[:, 1:] - e[:, :-1])[..., None]


def _spread(sp, tz, wave_of):
    """R T of every spectrum, end to end: (nz, npix, nb)."""
    out = []
    for s in sp:
        t = tz[s.wavehash]
        data = torch.tensor(s.R.data, device=t.device)
        r = torch.zeros_like(t)
        n = t.shape[1]
        for k, off in enumerate(np.asarray(s.R.offsets)):
            lo, hi = max(0, -off), min(n, n - off)         # row i has R[i, i + off]
            r[:, lo:hi] += data[k, lo + off:hi + off, None] * t[:, lo + off:hi + off]
        out.append(r)
    return torch.cat(out, 1)


def _nnls(M, y):
    """min ||M c - y||, c >= 0, for a few columns: the best feasible subset."""
    nz, n = y.shape
    best = torch.full((nz,), math.inf, device=y.device, dtype=y.dtype)
    c = torch.zeros_like(y)
    for s in range(1 << n):
        cols = [i for i in range(n) if s >> i & 1]
        cc = torch.zeros_like(y)
        if cols:
            cc[:, cols] = torch.linalg.lstsq(M[:, :, cols], y[..., None]).solution[..., 0]
        r = ((M @ cc[..., None])[..., 0] - y).square().sum(1)
        use = (cc >= 0).all(1) & (r < best)
        best = torch.where(use, r, best)
        c = torch.where(use[:, None], cc, c)
    return c


def _fit(sp, tz, method="PCA"):
    """chi2 (nz,) and coefficients (nz, nb) of one target."""
    tb = _spread(sp, tz, None)
    w = torch.tensor(np.concatenate([s.ivar for s in sp]), device=tb.device)
    f = torch.tensor(np.concatenate([s.flux for s in sp]), device=tb.device)
    wt = tb * w[None, :, None]
    M = tb.transpose(1, 2) @ wt
    y = (wt * f[None, :, None]).sum(1)
    c = torch.linalg.solve(M, y) if method == "PCA" else _nnls(M, y)
    r = f[None] - (tb @ c[..., None])[..., 0]
    return (w[None] * r * r).sum(1), c


def _scan_exact(spectra, spec, method):
    z = spec.redshifts
    isoii = (3724 <= spec.wave) & (spec.wave <= 3733)
    oii = torch.tensor(spec.flux[:, isoii].sum(1), device=_dev())
    n, nb = len(spectra), spec.flux.shape[0]
    zc, co = np.zeros((n, len(z))), np.zeros((n, len(z), nb))
    pen = np.zeros((n, len(z)))
    for i0 in range(0, len(z), 128):
        tz = {h: _rebinned(spec.wave, spec.flux, z[i0:i0 + 128], w) for h, w in _grids().items()}
        for i, sp in enumerate(spectra):
            c2, c = _fit(sp, tz, method)
            zc[i, i0:i0 + 128], co[i, i0:i0 + 128] = c2.cpu(), c.cpu()
            if spec.spectype == "GALAXY" and method == "PCA":
                pen[i, i0:i0 + 128] = (-(c @ oii)).clamp(min=0).cpu()
    return {"zchi2": zc, "zcoeff": co, "penalty": pen}


def _cosmics(flux, ivar, wave, nsig):
    """redrock's rejection: outliers of the flux gradient across exposures."""
    out = ivar.copy()
    grad, gvar = [], []
    for f, v in zip(flux, ivar):
        good = v > 0
        f, v = f.copy(), v.copy()
        bad = v == 0
        f[bad] = np.interp(wave[bad], wave[good], f[good])
        v[bad] = np.interp(wave[bad], wave[good], v[good])
        var = 1.0 / v
        g, gv = f.copy(), var.copy()
        g[1:] = f[1:] - f[:-1]
        gv[1:] = var[1:] + var[:-1]
        g[0] = 0.0
        grad.append(g)
        gvar.append(gv)
    grad, giv = np.array(grad), 1.0 / np.array(gvar)
    mean = (giv * grad).sum(0) / giv.sum()
    d2 = giv * (grad - mean) ** 2
    chi2 = d2.sum(0) / (len(flux) - 1)
    for j in np.where(chi2 > nsig ** 2)[0]:
        out[np.argmax(d2[:, j]), j] = 0.0
    return out


def _coadd_exact(spectra, nsig):
    flux, ivar, rdata = [], [], []
    for sp in spectra:
        for band in dict.fromkeys(s.band for s in sp):
            g = [s for s in sp if s.band == band]
            f, v = np.array([s.flux for s in g]), np.array([s.ivar for s in g])
            vw = _cosmics(f, v, g[0].wave, nsig) if nsig > 0 and len(g) > 1 else v
            w = vw.sum(0)
            den = np.where(w == 0, 1.0, w)
            fl = np.where(w == 0, f.mean(0), (vw * f).sum(0) / den)
            rd = sum(s.R.data * s.ivar for s in g) / den
            n = len(w)
            rows = np.zeros(n)
            for k, off in enumerate(np.asarray(g[0].R.offsets)):
                i = np.arange(max(0, -off), min(n, n - off))
                rows[i] += rd[k, i + off]
            flux.append(fl)
            ivar.append(np.where(rows < 0.99, 0.0, w))
            rdata.append(rd.ravel())
    return {"flux": np.concatenate(flux), "ivar": np.concatenate(ivar),
            "rdata": np.concatenate(rdata)}


def exact(case, seed):
    op = case["op"]
    if op == "build":
        if case["kind"] == "QSO":
            return None                                  # the IGM tables are the framework's
        t = prepare(case, seed)["template"]
        return {h: torch.cat([_rebinned(t.wave, t.flux, t.redshifts[i:i + 256], w)
                              for i in range(0, len(t.redshifts), 256)])
                for h, w in _grids().items()}
    if op in ("fitz", "zfind", "arch"):
        return None                                      # chains of decisions
    if case.get("n", 1) > 100:
        return None
    basis = "NMF" if op == "nmf" else "GALAXY"
    spectra = [s for s, _ in _spectra(case, seed, basis, positive=op == "nmf",
                                      nexp=case.get("nexp", 1))]
    if op == "coadd":
        return _coadd_exact(spectra, case["nsig"])
    if op == "nmf":
        return _scan_exact(spectra, _specs()["NMF"][0], "NMF")
    if op == "scan":
        out = {}
        for s in _specs()[case["kinds"]]:
            ft = TM.make_fulltype(s.spectype, s.subtype)
            out[ft] = {"zchi2": None, "zcoeff": None, "penalty": None} \
                if s.spectype == "QSO" else _scan_exact(spectra, s, "PCA")
        return out
    if case["kind"] == "QSO":
        return None
    s = _one(case["kind"], seed)
    if op == "finegrid":
        st = prepare(case, seed)
        tz = {h: _rebinned(s.wave, s.flux, st["zgrid"], w) for h, w in _grids().items()}
        c2, c = _fit(st["spectra"][0], tz)
        return {"binned": tz, "zchi2": c2, "zcoeff": c}
    st = prepare(case, seed)                             # grad
    z, wt = st["pair_z"].cpu().numpy(), st["weight"]
    sp0 = st["spectra"]
    chi2, coeff = [], []
    off, npad = 0, []
    for w in _grids().values():
        npad.append((off, len(w)))
        off += st["ctx"].rows.batch.segs[len(npad) - 1].npix_pad
    gf = torch.zeros((case["n"], off), dtype=torch.float64, device=_dev())
    for i in range(len(z)):
        tz = {h: _rebinned(s.wave, s.flux, z[i:i + 1], w) for h, w in _grids().items()}
        k = int(st["pair_t"][i])
        c2, c = _fit(sp0[k], tz)
        tb = _spread(sp0[k], tz, None)
        w = torch.tensor(np.concatenate([q.ivar for q in sp0[k]]), device=_dev())
        f = torch.tensor(np.concatenate([q.flux for q in sp0[k]]), device=_dev())
        g = 2.0 * w * (f - (tb[0] @ c[0])) * wt[i]
        a = 0
        for o, n in npad:
            gf[k, o:o + n] += g[a:a + n]
            a += n
        chi2.append(c2)
        coeff.append(c)
    return {"chi2": torch.cat(chi2), "coeff": torch.cat(coeff), "gz": None, "gflux": gf}


if __name__ == "__main__":
    for c in listed() + [draw(random.Random(k)) for k in range(6)]:
        print(c, work(c))
