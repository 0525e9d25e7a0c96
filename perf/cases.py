"""What a user of the synthesis framework has it do, as measurable cases.

Each case goes through the package's public entry points (``korg_gb300.synthesize``,
``synthesize_prepared``, ``BatchSynthesis``, ``autograd.Synthesis``, ``loss_and_gradient``,
``line_absorption_``, ``radiative_transfer``, ``statmech.solve_layers``, ``postprocess.Rotation`` /
``LSF``, ``MolecularCrossSection``).  Sizes are those of the package's synthetic workloads, tests
and benchmark, and reductions of them.

kinds
  window         synthesis of one short window, a fit's inner call (host arrays in, flux out)
  whole          synthesize(): chemistry, continuum and the hot path of one atmosphere
  survey         synthesis of a wide spectrum: the full optical range, or a cool giant's molecular bands
  batch          many atmospheres on one grid through the batched engine, inputs uploaded each time
  gradient       forward and backward of the rectified least-squares loss through torch autograd (mixed)
  gradient_fp64  loss_and_gradient in its default precision
  opacity        line_absorption_ in its default precision (FP64)
  transfer       radiative_transfer of a shell atmosphere along rays
  chemistry      chemical equilibrium of every layer of several atmospheres
  broadening     rotation and line-spread function of a stack of spectra, and their reverse modes
  cross_section  precomputed molecular cross-section table in its default precision (FP64)
"""
import functools
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if os.path.join(_ROOT, "korg.jl_gb300") not in sys.path:
    sys.path.insert(0, os.path.join(_ROOT, "korg.jl_gb300"))

ATOMS = ["Fe I", "Fe II", "Ca I", "Ti I", "Ni I"]
# Teff, log g, [M/H] of the batch's and the chemistry's stars: the ranges of the batch workload
STARS = [(3500, 1.0, 0.0), (3900, 4.6, -0.5), (4300, 1.8, -1.0), (4700, 2.6, 0.3), (5100, 4.5, -0.2),
         (5500, 3.8, -2.0), (5777, 4.44, 0.0), (6000, 4.0, -1.5), (6300, 4.3, 0.2), (6600, 4.1, -0.8),
         (6900, 3.9, 0.0), (4000, 1.2, -2.3), (5300, 4.6, 0.4), (4900, 3.2, -1.2), (3700, 4.8, 0.1),
         (6100, 3.5, -0.4)]


def _synth(kind, name, star, L, lo, hi, step, n_lines, molecular):
    return {"name": name, "kind": kind, "star": star, "L": L, "lo": float(lo), "hi": float(hi), "step": step,
            "n_lines": n_lines, "molecular": molecular}


def listed():
    return [
        # a fit's window around a few lines: 20 A, 300 lines, 56 MARCS layers
        _synth("window", "window", 4, 56, 5100, 5120, 0.01, 300, False),
        # the whole call on the package's parity workload: 2,000 lines, 10,001 points
        _synth("whole", "whole call", 4, 56, 5000, 5100, 0.01, 2000, False),
        # the benchmark's full optical synthesis: 300,000 lines, 700,001 points
        _synth("survey", "full optical", 6, 56, 3000, 10000, 0.01, 300000, False),
        # a cool giant's molecular bands at the density of the 1M-line list, a 2000 A part of its range
        _synth("survey", "cool giant", 0, 80, 4000, 6000, 0.01, 286000, True),
        # the batched fit server: 8 atmospheres, 5k-50k lines each, a quarter of the infrared range
        {"name": "infrared batch", "kind": "batch", "n": 8, "L": 56, "lo": 15000.0, "hi": 15500.0, "step": 0.005,
         "n_min": 5000, "n_max": 50000},
        # the adjoint workload's gradient on a quarter of its range: 72 layers, 17,500 lines
        _synth("gradient", "infrared gradient", 3, 72, 15000, 15500, 0.005, 17500, True),
        # a window's loss and gradient in the default precision
        _synth("gradient_fp64", "window gradient FP64", 4, 56, 5100, 5120, 0.01, 400, False),
        # line_absorption! as it stands (FP64) on the parity workload
        _synth("opacity", "line opacity FP64", 4, 56, 5000, 5100, 0.01, 2000, False),
        # a giant's shell atmosphere along 20 rays (the reference's default mu grid), 200 A
        {"name": "shell transfer", "kind": "transfer", "star": 3, "L": 56, "nwl": 20001, "n_mu": 20,
         "I_scheme": "linear"},
        # every layer of 16 stars in one call
        {"name": "chemistry", "kind": "chemistry", "n": 16, "L": 56},
        # rotation and LSF of 16 spectra of 100,001 points onto a 0.2 A grid, forward and backward
        {"name": "broadening", "kind": "broadening", "n": 16, "lo": 15000.0, "hi": 15500.0, "step": 0.005,
         "vsini": 10.0, "R": 22500.0, "out_step": 0.2},
        # the table of one molecule on the default (vmic, T) grid: 11 x 51 x 10,001
        {"name": "cross section", "kind": "cross_section", "lo": 15000.0, "hi": 15100.0, "step": 0.01,
         "n_lines": 1000, "nv": 11, "nT": 51},
    ]


def _log(rng, a, b):
    return math.exp(rng.uniform(math.log(a), math.log(b)))


def draw(rng):
    kind = rng.choice(["window", "whole", "survey", "survey", "batch", "gradient", "gradient_fp64", "opacity",
                       "transfer", "chemistry", "broadening", "cross_section"])
    if kind == "batch":
        width = round(_log(rng, 20, 500), 2)
        n_max = int(width * rng.uniform(10, 100))
        return {"kind": kind, "n": rng.randint(2, 8), "L": rng.choice([56, 72]), "lo": 15000.0, "hi": 15000.0 + width,
                "step": rng.choice([0.005, 0.01]), "n_min": max(50, n_max // 10), "n_max": max(100, n_max)}
    if kind == "transfer":
        return {"kind": kind, "star": rng.randrange(16), "L": rng.choice([56, 72]), "nwl": int(_log(rng, 1001, 20001)),
                "n_mu": rng.randint(5, 20), "I_scheme": rng.choice(["linear", "linear", "linear_flux_only"])}
    if kind == "chemistry":
        return {"kind": kind, "n": rng.randint(1, 16), "L": rng.choice([56, 72])}
    if kind == "broadening":
        width = round(_log(rng, 20, 500), 2)
        return {"kind": kind, "n": rng.randint(1, 16), "lo": 15000.0, "hi": 15000.0 + width,
                "step": rng.choice([0.005, 0.01]), "vsini": round(rng.uniform(2, 15), 2),
                "R": round(rng.uniform(15000, 60000), 0), "out_step": rng.choice([0.1, 0.2])}
    if kind == "cross_section":
        width = round(_log(rng, 10, 100), 2)
        return {"kind": kind, "lo": 15000.0, "hi": 15000.0 + width, "step": 0.01,
                "n_lines": int(width * rng.uniform(3, 10)), "nv": rng.randint(3, 11), "nT": rng.choice([26, 51])}
    infrared = kind in ("survey", "gradient") and rng.random() < 0.5
    widths = {"window": (5, 60), "whole": (20, 300), "survey": (300, 2000), "gradient": (20, 400),
              "gradient_fp64": (5, 25), "opacity": (20, 120)}[kind]
    width = round(_log(rng, *widths), 2)
    lo = 15000.0 if infrared else round(rng.uniform(4000, 7000), 1) if kind in ("survey", "whole", "gradient") \
        else round(rng.uniform(5040, 6350 - width), 1)
    per_A = rng.uniform(10, 40) if kind in ("window", "whole", "gradient_fp64", "opacity") else rng.uniform(20, 100)
    molecular = kind in ("survey", "gradient") and rng.random() < 0.5
    c = _synth(kind, "", rng.randrange(16), rng.choice([56, 56, 72, 80]), lo, round(lo + width, 2),
               0.005 if infrared else 0.01, max(20, int(per_A * width)), molecular)
    del c["name"]
    return c


# ------------------------------------------------------------------------------ inputs
@functools.lru_cache(maxsize=64)
def _atmosphere(star, L):
    """The model atmosphere a user reads from disk."""
    from korg_gb300 import standin
    T, g, m = STARS[star]
    return standin.synthetic_atmosphere(float(T), float(g), float(m), L)


def _linelist(n, lo, hi, seed, molecular):
    from korg_gb300 import synthetic
    if not molecular:
        return synthetic.synthetic_linelist(n, lo, hi, seed=seed, species=ATOMS)
    infrared = lo > 10000  # the adjoint workload's mix, else the cool giant's
    na = int(n * (5 / 7 if infrared else 0.4))
    a = synthetic.synthetic_linelist(na, lo, hi, seed=seed, species=ATOMS)
    m = synthetic.synthetic_linelist(n - na, lo, hi, seed=seed + 1,
                                     species=["CO", "OH", "CN"] if infrared else ["TiO", "CO", "OH", "CN"],
                                     loggf=(-8.0, -2.0) if infrared else (-9.0, -1.0),
                                     E_lower=(0.0, 3.0 if infrared else 4.0), molecular=True)
    return a.concat(m).sorted()


def _prepared(star, L, lo, hi, step, ll):
    from korg_gb300 import prepare_synthesis
    atm, A_X = _atmosphere(star, L)
    return prepare_synthesis(atm, ll, A_X, (lo, hi, step), continuum="gpu", chemistry="gpu")


def _spectra(case, seed):
    """A stack of rectified absorption spectra on the case's grid (device, FP64)."""
    from korg_gb300 import Wavelengths
    g = Wavelengths((case["lo"], case["hi"], case["step"]))
    rng = np.random.default_rng(seed)
    w = torch.as_tensor(g.all_wls * 1e8, device="cuda")
    f = torch.ones((case["n"], len(g)), dtype=torch.float64, device="cuda")
    for k in range(case["n"]):
        n = int((case["hi"] - case["lo"]) * 0.4) + 1
        c = torch.as_tensor(rng.uniform(case["lo"], case["hi"], n), device="cuda")
        d = torch.as_tensor(rng.uniform(0.05, 0.8, n), device="cuda")
        s = torch.as_tensor(rng.uniform(0.08, 0.3, n), device="cuda")
        for i in range(0, n, 32):
            f[k] *= torch.prod(1 - d[i:i + 32, None] * torch.exp(-0.5 * ((w - c[i:i + 32, None]) / s[i:i + 32, None]) ** 2),
                               dim=0)
    out = np.arange(case["lo"] + 1, case["hi"] - 1, case["out_step"]) * 1e-8
    cot = torch.as_tensor(rng.standard_normal((case["n"], len(out))), device="cuda")
    return g, f, out, cot


def prepare(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng(seed)
    s = {"kind": kind, "case": case}
    if kind == "batch":
        from korg_gb300 import synthetic
        from korg_gb300.batch import BatchSynthesis
        lo, hi = case["lo"], case["hi"]
        master = _linelist(int(case["n_max"] * 2.5), lo, hi, seed, True)
        inputs = []
        for k in range(case["n"]):
            n = int(rng.integers(case["n_min"], case["n_max"] + 1))
            keep = np.sort(rng.choice(len(master), size=n, replace=False))
            inputs.append(_prepared((2 * k + 1) % 16, case["L"], lo, hi, case["step"], master.subset(keep)))
        s["batch"] = BatchSynthesis(inputs, precision="mixed")
    elif kind == "transfer":
        from korg_gb300 import continuum
        from korg_gb300.statmech import chemical_equilibrium
        atm, A_X = _atmosphere(case["star"], case["L"])
        ab = 10.0 ** (np.asarray(A_X) - 12)
        ne, nd = chemical_equilibrium(atm.T, atm.n_tot, atm.ne, ab / ab.sum())
        wl = np.linspace(5000.0, 5000.0 + 0.01 * (case["nwl"] - 1), case["nwl"]) * 1e-8
        knots = np.linspace(wl[0], wl[-1], 33)
        cn = np.ascontiguousarray(continuum.continuum_absorption(knots, atm.T, ne, nd).T)
        base = np.empty((len(wl), case["L"]))
        for l in range(case["L"]):
            base[:, l] = np.interp(wl, knots, cn[:, l])
        lines = 1 + 10.0 ** rng.uniform(-2, 2.5, (len(wl), 1)) * np.linspace(1.0, 0.3, case["L"])[None, :]
        x = 1.43877687750393 / (wl[:, None] * atm.T[None, :])
        S = 2 * 6.62607015e-27 * 2.99792458e10 ** 2 / wl[:, None] ** 5 / np.expm1(x)
        s.update(atm=atm, alpha=base * lines, S=S, ref=continuum.continuum_absorption(np.array([5e-5]), atm.T, ne, nd)[:, 0].copy(),
                 R=7e11)
    elif kind == "chemistry":
        T, nt, ne, ab, at = [], [], [], [], []
        for k in range(case["n"]):
            atm, A_X = _atmosphere(k, case["L"])
            a = 10.0 ** (np.asarray(A_X) - 12 + rng.uniform(-0.1, 0.1, 92) * (np.arange(92) > 1))
            T.append(atm.T * (1 + 0.002 * rng.uniform(-1, 1)))
            nt.append(atm.n_tot)
            ne.append(atm.ne)
            ab.append(a / a.sum())
            at.append(np.full(case["L"], k, np.int32))
        s.update(T=np.concatenate(T), n_tot=np.concatenate(nt), ne=np.concatenate(ne), ab=np.array(ab),
                 at=np.concatenate(at))
    elif kind == "broadening":
        g, f, out, cot = _spectra(case, seed)
        s.update(grid=g, flux=f, wls=torch.as_tensor(g.all_wls, device="cuda"), cot=cot,
                 out=torch.as_tensor(out, device="cuda"),
                 R=torch.tensor([case["R"]], dtype=torch.float64, device="cuda"))
    elif kind == "cross_section":
        from korg_gb300 import Wavelengths, synthetic
        s.update(ll=synthetic.synthetic_linelist(case["n_lines"], case["lo"], case["hi"], seed=seed, species=["CO"],
                                                 loggf=(-8.0, -2.0), E_lower=(0.0, 3.0), molecular=True),
                 wls=Wavelengths((case["lo"], case["hi"], case["step"])),
                 vmic=np.linspace(0.0, 4.0 + 4 / 3, case["nv"]), logT=np.linspace(3.0, 5.0, case["nT"]))
    else:
        ll = _linelist(case["n_lines"], case["lo"], case["hi"], seed, case["molecular"])
        if kind == "whole":
            s["atm"], s["A_X"] = _atmosphere(case["star"], case["L"])
            s["ll"], s["wls"] = ll, (case["lo"], case["hi"], case["step"])
            return s
        inp = s["inp"] = _prepared(case["star"], case["L"], case["lo"], case["hi"], case["step"], ll)
        nwl, L = len(inp.wls), case["L"]
        if kind == "gradient":
            from korg_gb300.autograd import Synthesis
            s["synth"] = Synthesis(inp, precision="mixed")
            s["x"] = {k: v.requires_grad_(True) for k, v in s["synth"].initial().items()}
            s["obs"] = torch.as_tensor(rng.uniform(0.5, 1.0, nwl), device="cuda")
        elif kind == "gradient_fp64":
            s["obs"] = rng.uniform(0.5, 1.0, nwl)
        elif kind == "opacity":
            a = np.empty((nwl, L))
            for l in range(L):
                a[:, l] = np.interp(inp.wls.all_wls, inp.cntm_knots, inp.cntm_vals[l])
            s["alpha0"] = a
    return s


# ------------------------------------------------------------------------------ one pass
def run(s):
    kind = s["kind"]
    if kind in ("window", "survey"):
        from korg_gb300 import synthesize_prepared
        r = synthesize_prepared(s["inp"], precision="mixed")
        return {"flux": r.flux, "cntm": r.cntm}
    if kind == "whole":
        from korg_gb300 import synthesize
        r = synthesize(s["atm"], s["ll"], s["A_X"], s["wls"])
        return {"flux": r.flux, "cntm": r.cntm}
    if kind == "batch":
        s["batch"].upload()
        flux, cntm = s["batch"].run()
        return {"flux": flux, "cntm": cntm}
    if kind == "gradient":
        x = s["x"]
        for v in x.values():
            v.grad = None
        flux, cntm = s["synth"](**x)
        loss = torch.sum((flux / cntm - s["obs"]) ** 2)
        loss.backward()
        return {"flux": flux.detach(), "cntm": cntm.detach(), "grad": {k: v.grad for k, v in x.items()}}
    if kind == "gradient_fp64":
        from korg_gb300.api import loss_and_gradient
        loss, g = loss_and_gradient(s["inp"], s["obs"])
        return {"loss": loss, "grad": g}
    if kind == "opacity":
        from korg_gb300 import line_absorption_
        from korg_gb300.api import ContinuumInterpolant
        from korg_gb300.data import default_partition_funcs
        inp, alpha = s["inp"], s["alpha0"].copy()
        line_absorption_(alpha, inp.linelist, inp.wls, inp.T, inp.ne, inp.number_densities, default_partition_funcs(),
                         inp.xi, ContinuumInterpolant(inp.cntm_knots, inp.cntm_vals))
        return {"alpha": alpha}
    if kind == "transfer":
        from korg_gb300 import radiative_transfer
        F, I, mu, w = radiative_transfer(s["atm"], s["alpha"], s["S"], s["case"]["n_mu"], alpha_ref=s["ref"],
                                         I_scheme=s["case"]["I_scheme"], R=s["R"])
        return {"F": F, "I": I}
    if kind == "chemistry":
        from korg_gb300.statmech import solve_layers
        dens, status, _ = solve_layers(s["T"], s["n_tot"], s["ne"], s["ab"], atm=s["at"])
        return {"densities": dens, "status": status}
    if kind == "broadening":
        from korg_gb300.postprocess import LSF, Rotation
        f = s["flux"].detach().requires_grad_(True)
        y = Rotation.apply(f, s["wls"], s["grid"], s["case"]["vsini"])
        z = LSF.apply(y, s["wls"], s["out"], s["R"])
        z.backward(s["cot"])
        return {"out": z.detach(), "grad": f.grad}
    if kind == "cross_section":
        from korg_gb300.molecular import MolecularCrossSection
        m = MolecularCrossSection(s["ll"], s["wls"], vmic_vals=s["vmic"], log_temp_vals=s["logT"])
        return {"table": m.table}
    raise ValueError(kind)


# ------------------------------------------------------------------------------ the path's own work
def work(case):
    """Inputs read once and outputs written once.  Operations: a line's profile (24 operations) over
    ten Doppler widths per layer (its wings can be had more cheaply), 35 per (layer, wavelength)
    and transfer; reverse modes twice their forward."""
    kind = case["kind"]
    core = lambda lo, step: 10 * lo * 6.7e-6 / step
    if kind == "chemistry":  # four Newton steps: LU of 93 unknowns
        n = case["n"] * case["L"]
        return {"bytes": n * 8.0 * (3 + 278 + 306) + case["n"] * 736.0, "flops": n * 4 * (2 / 3) * 93.0 ** 3}
    if kind == "transfer":  # 12 operations per (ray, layer, wavelength)
        n = float(case["nwl"]) * case["L"]
        return {"bytes": 16 * n + 8.0 * case["nwl"] * (case["n_mu"] + 1), "flops": 12 * n * case["n_mu"]}
    nwl = round((case["hi"] - case["lo"]) / case["step"]) + 1
    if kind == "broadening":
        m = (case["hi"] - case["lo"] - 2) / case["out_step"]
        win = 2 * case["lo"] * case["vsini"] / 299792.458 / case["step"]
        lsf = 8 * case["lo"] / case["R"] / 2.3548 / case["step"]
        return {"bytes": 16.0 * case["n"] * (nwl + m), "flops": 2 * case["n"] * 2 * (nwl * win + m * lsf) + 20.0 * nwl * win}
    if kind == "cross_section":
        t = float(case["nv"]) * case["nT"]
        return {"bytes": 8 * t * nwl + 72.0 * case["n_lines"] + 8.0 * nwl,
                "flops": 24 * t * case["n_lines"] * core(case["lo"], case["step"])}
    if kind == "batch":
        n, spectra = (case["n_min"] + case["n_max"]) / 2, case["n"]
    else:
        n, spectra = case["n_lines"], 1
    L = case["L"]
    lines = 24.0 * L * n * core(case["lo"], case["step"])
    if kind == "opacity":
        return {"bytes": 16.0 * L * nwl + 72.0 * n + 8.0 * nwl, "flops": lines}
    b = 72.0 * n + 8.0 * L * ((case["hi"] - case["lo"]) + 22) + 8.0 * nwl + 16.0 * nwl
    f = lines + 70.0 * L * nwl
    if kind in ("gradient", "gradient_fp64"):
        b, f = 2 * b + 8.0 * nwl, 3 * f
    return {"bytes": spectra * b, "flops": spectra * f}


# ------------------------------------------------------------------------------ the same in 64 bits
_k, _h, _c, _keV, _heV, _amu = 1.380649e-16, 6.62607015e-27, 2.99792458e10, 8.617333262145e-5, 4.135667696e-15, 1.6605402e-24


def _t(a):
    return torch.as_tensor(np.ascontiguousarray(a, np.float64), device="cuda")


def _hjerting(a, v):
    """Hunger's (1965) four-branch approximation of the Voigt function."""
    v2 = v * v
    H0 = torch.exp(-v2)
    p1 = -1.12470432 + (-0.15516677 + (3.288675912 + (-2.34357915 + 0.42139162 * v) * v) * v) * v
    p2 = -4.48480194 + (9.39456063 + (-6.61487486 + (1.98919585 - 0.22041650 * v) * v) * v) * v
    p3 = (0.554153432 + (0.278711796 + (-0.1883256872 + (0.042991293 - 0.003278278 * v) * v) * v) * v) / (v2 - 1.5)
    H1 = torch.where(v < 1.3, p1, torch.where(v < 2.4, p2, p3))
    H2 = (1 - 2 * v2) * H0
    c2, c23 = 2 / math.sqrt(math.pi), 2 / (3 * math.sqrt(math.pi))
    iv = 1 / v2
    wing = (a / math.sqrt(math.pi) * iv) * (1 + 1.5 * iv + 3.75 * iv * iv)
    near = H0 + (H1 + H2 * a) * a
    M1 = H1 + c2 * H0
    M2 = H2 - H0 + c2 * M1
    M3 = c23 * (1 - H2) - 2 / 3 * v2 * M1 + c2 * M2
    M4 = 2 / 3 * v2 * v2 * H0 - c23 * M1 + c2 * M3
    psi = 0.979895023 + (-0.962846325 + (0.532770573 - 0.122727278 * a) * a) * a
    mod = psi * (H0 + (M1 + (M2 + (M3 + M4 * a) * a) * a) * a)
    r2 = v2 / (a * a)
    u = 1 / math.sqrt(2) / ((r2 + 1) * a)
    u2 = u * u
    far = math.sqrt(2 / math.pi) * u * (1 + (3 * r2 - 1 + ((r2 - 2) * 15 * r2 + 2) * u2) * u2)
    return torch.where(a <= 0.2, torch.where(v >= 5, wing, near), torch.where((a <= 1.4) & (a + v < 3.2), mod, far))


def _add_lines(alpha, w, ll, T, ne, nv, xi, nU, knots, vals, cutoff):
    """alpha (nwl, L) += line opacity, every line over its window."""
    wl, El, m, grad, gst, v1, v2 = (_t(x)[:, None] for x in (ll.wl, ll.E_lower, ll.mass, ll.gamma_rad, ll.gamma_stark,
                                                             ll.vdW1, ll.vdW2))
    mol = torch.as_tensor(np.asarray(ll.is_mol) != 0, device="cuda")[:, None]
    T, ne, nv, xi = (_t(x)[None, :] for x in (T, ne, nv, xi))
    sigma = wl * torch.sqrt(_k * T / m + xi * xi / 2) / _c
    vbar = torch.sqrt(8 * _k * T / math.pi * (1 / (1.008 * _amu) + 1 / m))
    abo = 2 * (4 / math.pi) ** (v2 / 2) * torch.exp(torch.lgamma((4 - v2) / 2)) * 1e6 * v1 * (vbar / 1e6) ** (1 - v2)
    vdw = torch.where(v2 == -1, v1 * (T / 1e4) ** 0.3, abo)
    broad = ne * gst * (T / 1e4) ** (1 / 6) + nv * vdw
    gamma = (grad + torch.where(mol, torch.zeros_like(broad), broad)) * wl * wl / (_c * 4 * math.pi)
    beta = 1 / (_keV * T)
    sline = math.pi * 4.80320425e-10 ** 2 / 9.1093897e-28 / _c * (wl * wl / _c)
    amp = 10 ** _t(ll.log_gf)[:, None] * sline * (torch.exp(-beta * El) - torch.exp(-beta * (El + _c * _heV / wl)))
    amp = amp * _t(nU)[torch.as_tensor(np.asarray(ll.species_idx, np.int64), device="cuda")]
    vals = _t(vals)
    if len(knots) > 1:
        kn = _t(knots)
        i = (torch.searchsorted(kn, wl[:, 0], right=True) - 1).clamp(0, len(knots) - 2)
        t = ((wl[:, 0] - kn[i]) / (kn[i + 1] - kn[i]))[:, None]
        ac = vals.T[i] * (1 - t) + vals.T[i + 1] * t
    else:
        ac = vals.T.expand(len(ll.wl), -1)
    rho = ac * cutoff / amp
    s2 = math.sqrt(2 * math.pi)
    dw = torch.where(rho > 1 / (s2 * sigma), 0.0, sigma * torch.sqrt((-2 * torch.log(s2 * sigma * rho)).clamp(min=0)))
    lw = torch.where(rho > 1 / (math.pi * gamma), 0.0, torch.sqrt((gamma / (math.pi * rho) - gamma ** 2).clamp(min=0)))
    win = torch.sqrt(dw.amax(1) ** 2 + lw.amax(1) ** 2)
    lb = torch.searchsorted(w, wl[:, 0] - win)
    ub = torch.searchsorted(w, wl[:, 0] + win, right=True)
    lo, hi = lb.cpu().numpy(), ub.cpu().numpy()
    inv = 1 / (sigma * math.sqrt(2))
    a, scale = gamma * inv, inv / math.sqrt(math.pi) * amp
    order = np.flatnonzero(hi > lo)
    for c in range(0, len(order), 8):
        idx = order[c:c + 8]
        j0, j1 = lo[idx].min(), hi[idx].max()
        ix = torch.as_tensor(idx, device="cuda")
        x = (w[None, j0:j1] - wl[ix]).abs()
        j = torch.arange(int(j0), int(j1), device="cuda")[None]
        inside = (j >= lb[ix][:, None]) & (j < ub[ix][:, None])
        H = _hjerting(a[ix][:, None, :], x[:, :, None] * inv[ix][:, None, :]) * scale[ix][:, None, :]
        alpha[j0:j1] += torch.where(inside[:, :, None], H, 0.0).sum(0)


_E2 = [(2.5, 2.0, (0.037534261820486914, -0.04890051070806112, 0.033833820809153176, -0.016916910404576574,
                   0.007048712668573576, -0.0026785108140579598)),
       (3.5, 3.0, (0.010641925085272673, -0.013048381094197039, 0.008297844727977323, -0.003687930990212144,
                   0.0013061422257001345, -0.0003995258572729822)),
       (4.5, 4.0, (0.0031982292493385146, -0.0037793524098489054, 0.0022894548610917728, -0.0009539395254549051,
                   0.00031003034577284415, -8.466213288412284e-5)),
       (5.5, 5.0, (0.000996469042708825, -0.0011482955912753257, 0.0006737946999085467, -0.00026951787996341863,
                   8.310134632205409e-5, -2.1202073223788938e-5)),
       (6.5, 6.0, (0.0003182574636904001, -0.0003600824521626587, 0.00020656268138886323, -8.032993165122457e-5,
                   2.390771775334065e-5, -5.8334831318151185e-6)),
       (7.5, 7.0, (0.00010350984428214624, -0.00011548173161033826, 6.513442611103688e-5, -2.4813114708966427e-5,
                   7.200234178941151e-6, -1.7027366981408086e-6)),
       (9.0, 8.0, (3.413764515111217e-5, -3.76656228439249e-5, 2.096641424390699e-5, -7.862405341465122e-6,
                   2.2386015208338193e-6, -5.173353514609864e-7))]


def _expint2(x):
    """The reference's piecewise E2: series below 1.1, Taylor polynomials, asymptotic form from 9."""
    ix = 1 / x.clamp(min=1e-300)
    y = torch.exp(-x) * (1 + (-2 + (6 + (-24 + 120 * ix) * ix) * ix) * ix) * ix
    for end, at, c in reversed(_E2):
        d = x - at
        p = c[5]
        for q in c[4::-1]:
            p = q + p * d
        y = torch.where(x < end, p, y)
    s = 1 + ((torch.log(x.clamp(min=1e-300)) + 0.57721566490153286 - 1) + (-0.5 + (0.08333333333333333 + (
        -0.013888888888888888 + 0.0020833333333333333 * x) * x) * x) * x) * x
    return torch.where(x == 0, 1.0, torch.where(x < 1.1, s, y))


def _anchored_tau(alpha, fac, log_tau):
    ib = alpha * fac
    tau = torch.zeros_like(alpha)
    tau[:, 1:] = torch.cumsum(0.5 * (ib[:, 1:] + ib[:, :-1]) * (log_tau[1:] - log_tau[:-1]), 1)
    return tau


def _planar_flux(alpha, S, tau_ref, alpha_ref):
    lt = torch.log(tau_ref)
    tau = _anchored_tau(alpha, tau_ref / alpha_ref, lt)
    m = (S[:, 1:] - S[:, :-1]) / (tau[:, 1:] - tau[:, :-1])
    b = S[:, :-1] - m * tau[:, :-1]
    e2, ex = _expint2(tau), torch.exp(-tau)
    core = lambda t, e, x: (t * e * (3 * b + 2 * m * t) - x * (3 * b + 2 * m * (t + 1))) / 6
    return 2 * math.pi * (core(tau[:, 1:], e2[:, 1:], ex[:, 1:]) - core(tau[:, :-1], e2[:, :-1], ex[:, :-1])).sum(1)


def _exact_window(inp):
    w = _t(inp.wls.all_wls)
    i = (torch.searchsorted(_t(inp.cntm_knots), w, right=True) - 1).clamp(0, len(inp.cntm_knots) - 2)
    kn, v = _t(inp.cntm_knots), _t(inp.cntm_vals).T
    t = ((w - kn[i]) / (kn[i + 1] - kn[i]))[:, None]
    cn = v[i] * (1 - t) + v[i + 1] * t
    lay = (inp.T, inp.ne, inp.n_eff_vdW, inp.xi, inp.n_div_U)
    ref = _t(inp.alpha_ref_cntm)[None].clone()
    _add_lines(ref, _t([inp.ref_wl]), inp.linelist5, *lay, np.zeros(1), inp.alpha_ref_cntm[:, None], inp.cutoff_threshold)
    T = _t(inp.T)[None]
    S = 2 * _h * _c * _c / w[:, None] ** 5 / torch.expm1(_h * _c / (w[:, None] * _k * T))
    tr = _t(inp.tau_ref)
    cntm = _planar_flux(cn, S, tr, ref[0]) * 1e-8
    _add_lines(cn, w, inp.linelist, *lay, inp.cntm_knots, inp.cntm_vals, inp.cutoff_threshold)
    return {"flux": _planar_flux(cn, S, tr, ref[0]) * 1e-8, "cntm": cntm}


def _exact_shell(s):
    """Rays through a shell: the surface mu grid's impact parameters, anchored tau along each ray,
    the linear formal solution (or its flux-only form); a ray that misses the core starts at its
    deepest layer with what the inward ray brings there."""
    atm, L, n_mu = s["atm"], s["case"]["L"], s["case"]["n_mu"]
    r = s["R"] + atm.z
    mu, wt = np.polynomial.legendre.leggauss(n_mu)
    mu, wt = mu / 2 + 0.5, wt / 2
    alpha, S, ref = _t(s["alpha"]), _t(s["S"]), _t(s["ref"])
    F, out = torch.zeros(len(alpha), dtype=torch.float64, device="cuda"), []
    for m_u, w_u in zip(mu, wt):
        b = r[0] * math.sqrt(1 - m_u * m_u)
        if b < r[-1]:
            n = L
        else:
            k = int(np.argmin(np.abs(r - b)))
            n = (k - 1 if r[k] < b else k) + 1
        ss = np.sqrt(r[:n] ** 2 - b * b)
        fac, lt = _t(atm.tau_ref[:n]) / ref[:n] * _t(r[:n] / ss), _t(np.log(atm.tau_ref[:n]))

        def ray(al, Sc, f, l, start):
            tau = _anchored_tau(al, f, l)
            if s["case"]["I_scheme"] == "linear":
                I = start
                for q in range(n - 2, -1, -1):
                    d = tau[:, q + 1] - tau[:, q]
                    m = (Sc[:, q + 1] - Sc[:, q]) / d
                    I = (I - Sc[:, q] - m * (d + 1)) * torch.exp(-d) + m + Sc[:, q]
                return I, None
            I, e = start, torch.exp(-tau)
            for q in range(n - 1):
                d = tau[:, q + 1] - tau[:, q]
                m = (Sc[:, q + 1] - Sc[:, q]) / torch.where(d == 0, 1.0, d)
                I = I + (-e[:, q + 1] * (Sc[:, q + 1] + m) + e[:, q] * (Sc[:, q] + m))
            return I, e[:, n - 1]

        start = torch.zeros_like(F)
        if n < L:
            I, e = ray(alpha[:, :n].flip(1), S[:, :n].flip(1), fac.flip(0), -lt.flip(0), start)
            start = I if e is None else I * e
        I, _ = ray(alpha[:, :n], S[:, :n], fac, lt, start)
        out.append(I)
        F = F + I * w_u * m_u
    return {"F": 2 * math.pi * F * r[0] ** 2 / s["R"] ** 2, "I": torch.stack(out)}


def _exact_broadening(s):
    c, f, w = s["case"], s["flux"], s["wls"]
    n = len(w)
    step = float(s["grid"].ranges[0][1])
    eps, v = 0.6, c["vsini"] * 1e5 / _c
    c1, c2, c3 = 2 * (1 - eps), math.pi * eps / 2, math.pi * (1 - eps / 3)
    dl = w * v
    lb, ub = torch.searchsorted(w, w - dl), torch.searchsorted(w, w + dl, right=True) - 1
    W = int((ub - lb).max()) + 1
    q = torch.arange(W, device="cuda")

    def K(d, D):
        e = d.abs() >= D
        z = torch.where(e, 0.0, d)
        k = (0.5 * c1 * z * torch.sqrt(1 - z * z / (D * D)) + 0.5 * c1 * D * torch.asin(z / D) +
             c2 * (z - z ** 3 / (3 * D * D))) / (c3 * D)
        return torch.where(e, 0.5 * torch.sign(d), k)

    def rot_weights(i):
        D = dl[i][:, None]
        m = lb[i][:, None] + q
        d = ((m - i[:, None]).double() + 0.5) * step
        kn = torch.where(m < ub[i][:, None], K(d, D), 0.5)
        kp = torch.where(q == 0, -0.5, K(d - step, D))
        return torch.where(m <= ub[i][:, None], kn - kp, 0.0), m.clamp(max=n - 1)

    def lsf_weights():
        o = s["out"]
        sg = o / c["R"] / (2 * math.sqrt(2 * math.log(2)))
        a, b = torch.searchsorted(w, o - 4.0 * sg), torch.searchsorted(w, o + 4.0 * sg, right=True) - 1
        m = a[:, None] + torch.arange(int((b - a).max()) + 1, device="cuda")
        j = m.clamp(max=n - 1)
        p = torch.where(m <= b[:, None], torch.exp(-0.5 * ((w[j] - o[:, None]) / sg[:, None]) ** 2), 0.0)
        return p / p.sum(1, keepdim=True), j

    y, g = torch.empty_like(f), torch.zeros_like(f)
    pieces = [torch.arange(k, min(n, k + 8192), device="cuda") for k in range(0, n, 8192)]
    for i in pieces:
        wt, j = rot_weights(i)
        y[:, i] = torch.stack([(fk[j] * wt).sum(1) for fk in f])
    wl, jl = lsf_weights()
    z = torch.stack([(yk[jl] * wl).sum(1) for yk in y])
    gy = torch.zeros_like(f)
    for k in range(len(f)):
        gy[k].index_add_(0, jl.reshape(-1), (wl * s["cot"][k][:, None]).reshape(-1))
    for i in pieces:
        wt, j = rot_weights(i)
        for k in range(len(f)):
            g[k].index_add_(0, j.reshape(-1), (wt * gy[k][i][:, None]).reshape(-1))
    return {"out": z, "grad": g}


def exact(case, seed):
    """The same outputs from plain torch in 64 bits; None where that is too long (whole spectra with
    hydrogen lines, gradients) or iterative (chemical equilibrium)."""
    kind = case["kind"]
    if kind not in ("window", "opacity", "transfer", "broadening", "cross_section"):
        return None
    s = prepare(case, seed)
    if kind == "window":  # 5040-6400 A: outside every hydrogen line's window
        return _exact_window(s["inp"])
    if kind == "opacity":
        inp, a = s["inp"], _t(s["alpha0"])
        _add_lines(a, _t(inp.wls.all_wls), inp.linelist, inp.T, inp.ne, inp.n_eff_vdW, inp.xi, inp.n_div_U,
                   inp.cntm_knots, inp.cntm_vals, 3e-4)
        return {"alpha": a}
    if kind == "transfer":
        return _exact_shell(s)
    if kind == "broadening":
        return _exact_broadening(s)
    from korg_gb300.data import default_partition_funcs
    T = 10.0 ** s["logT"]
    ll, w = s["ll"], _t(s["wls"].all_wls)
    U = default_partition_funcs()[ll.species[0]](np.log(T))
    nU = np.zeros((len(ll.species), len(T)))
    nU[:] = 1 / (1e-32 * U)
    table = []
    for v in s["vmic"]:
        a = torch.zeros((len(w), len(T)), dtype=torch.float64, device="cuda")
        _add_lines(a, w, ll, T, np.zeros(len(T)), np.zeros(len(T)), np.full(len(T), v * 1e5), nU, np.zeros(1),
                   np.ones((len(T), 1)), 1.0)
        table.append(a * 1e-32)
    return {"table": torch.stack(table)}
