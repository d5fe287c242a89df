"""Timing cases of the viscoelastic time step and its companions.

Each case goes through the package's public entry points (fastearth3d_b200.lib)
the way a coupled climate / GIA program does: a handle is created once, the
reference state and the lateral viscosity are set once, and the timed pass is
one call sequence of the time loop. The kinds:

  sht       Gauss-grid analysis and synthesis of host fields: what a coupler
            does with a load or a topography outside the step (the smallest
            calls: two transfers and two short kernels each)
  response  the response operators of a host that runs its own sea-level
            solver: begin_step, apply, advance with a host load spectrum
  step      one interval of the interval driver: ice in (host array or device
            pointer), sub-steps with drift, sea-level equation and memory
            advance, and the coupling fields out (host arrays) or the
            device-resident rsl
  grad      the rsl misfit of a few intervals and its gradient with respect to
            the ice history and the lateral viscosity (inversion programs)
  batch     an ensemble of small models advanced together

Sizes are those of the repository's workloads (lmax 64 / 60 elements without
an ocean; lmax 128 / 100 elements with sea level and rotation; the same with
lateral viscosity; ensemble members of lmax 64-256) and odd ones between:
lmax need not be a power of two, the Gauss grid may have more rows and columns
than the transform needs, and 24 to 100 radial elements are in use.
"""
import math

import numpy as np
import torch

from fastearth3d_b200 import lib as vlib
from fastearth3d_b200 import synth
from fastearth3d_b200.abi import VG_RHEOL_MAXWELL, set_layers

PRECISION = {"fp64": 0, "split": 1, "exact": 2}  # visc3d_precision
N_ICE = 8  # ice fields of the history that passes cycle through


def _step(name, lmax, n_elem, **kw):
    c = {"name": name, "kind": "step", "lmax": lmax, "nlat": lmax + 1, "nphi": 2 * (lmax + 1), "n_elem": n_elem,
         "dt_yr": 50.0, "sle": True, "rotation": False, "trap": False, "visc3d": False, "precision": "fp64",
         "toroidal": False, "host": False}
    c.update(kw)
    return c


def listed():
    return [
        # one field in and out of spectral space at the smallest model size in use
        {"name": "sht_l32", "kind": "sht", "lmax": 32, "nlat": 33, "nphi": 66},
        # the largest ensemble size on an oversampled grid whose row length has a large odd factor
        {"name": "sht_l255_odd", "kind": "sht", "lmax": 255, "nlat": 259, "nphi": 518},
        # a host with its own sea-level solver, 1-D earth
        {"name": "response_l64", "kind": "response", "lmax": 64, "nlat": 65, "nphi": 130, "n_elem": 60, "visc3d": False,
         "precision": "fp64"},
        # the plain 1-D workload: no ocean, so a step is drift, load and memory advance (launches and latency count)
        _step("step_1d_l64", 64, 60, sle=False),
        # the 1-D production workload: sea level with migrating coastlines and rotation, ice from the host and the
        # coupling fields back to it
        _step("step_1d_sle_rot_l128", 128, 100, dt_yr=100.0, rotation=True, host=True),
        # the adaptive trapezoidal scheme at an in-between size
        _step("step_1d_trap_l85", 85, 48, trap=True),
        # lateral viscosity at the headline size, default (FP64) arithmetic
        _step("step_3d_fp64_l128", 128, 100, visc3d=True),
        # the same with the exact tensor-core products
        _step("step_3d_exact_l128", 128, 100, visc3d=True, precision="exact"),
        # toroidal channels at a small odd size on a larger grid, through host arrays
        _step("step_3d_tor_l47", 47, 37, visc3d=True, toroidal=True, nlat=50, nphi=100, host=True),
        # the largest ensemble member
        _step("step_3d_fp64_l256", 256, 100, visc3d=True),
        # gradient of a data misfit through the coupled 3-D step
        {"name": "grad_3d_l64", "kind": "grad", "lmax": 64, "nlat": 65, "nphi": 130, "n_elem": 60, "dt_yr": 50.0,
         "visc3d": True, "nsteps": 4, "ckpt": 2, "sites": 100},
        # a small ensemble on one GPU, every other member with lateral viscosity
        {"name": "batch_6", "kind": "batch", "members": 6, "lmax": 64, "n_elem": 40, "dt_yr": 50.0,
         "precision": "exact"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["sht", "sht", "response", "step", "step", "step", "step", "step", "grad", "batch"])
    lmax = _log_int(rng, 24, 240)
    n_elem = rng.randint(24, 100)
    nlat = lmax + 1 + rng.choice([0, 0, 1, 2, 5])
    nphi = 2 * (lmax + 1 + rng.choice([0, 0, 1, 3, 6]))
    if kind == "sht":
        return {"kind": kind, "lmax": lmax, "nlat": nlat, "nphi": nphi}
    if kind == "response":
        return {"kind": kind, "lmax": lmax, "nlat": nlat, "nphi": nphi, "n_elem": n_elem,
                "visc3d": rng.random() < 0.4, "precision": rng.choice(["fp64", "exact"])}
    if kind == "grad":
        lmax = _log_int(rng, 24, 80)
        return {"kind": kind, "lmax": lmax, "nlat": lmax + 1 + rng.choice([0, 2]),
                "nphi": 2 * (lmax + 1 + rng.choice([0, 3])), "n_elem": rng.randint(24, 60), "dt_yr": 50.0,
                "visc3d": rng.random() < 0.7, "nsteps": rng.randint(2, 4), "ckpt": rng.randint(1, 4),
                "sites": rng.randint(20, 200)}
    if kind == "batch":
        return {"kind": kind, "members": rng.randint(2, 6), "lmax": _log_int(rng, 24, 80),
                "n_elem": rng.randint(24, 60), "dt_yr": 50.0, "precision": rng.choice(["fp64", "exact"])}
    visc3d = rng.random() < 0.6
    toroidal = visc3d and rng.random() < 0.2
    trap = rng.random() < 0.15
    if toroidal or trap:
        lmax = _log_int(rng, 24, 100)
        nlat, nphi = lmax + 1 + rng.choice([0, 3]), 2 * (lmax + 1 + rng.choice([0, 2]))
    precision = "fp64"
    if visc3d:
        precision = rng.choice(["fp64", "fp64", "exact"] if toroidal else ["fp64", "fp64", "exact", "exact", "split"])
    c = _step("", lmax, n_elem, nlat=nlat, nphi=nphi, visc3d=visc3d, toroidal=toroidal, trap=trap, precision=precision,
              sle=rng.random() < 0.85, rotation=(not visc3d and not trap and rng.random() < 0.4),
              host=rng.random() < 0.4)
    del c["name"]
    return c


# ---------------------------------------------------------------- prepare


def _params(case):
    p = vlib.default_params()
    p.lmax, p.nlat, p.nphi = case["lmax"], case["nlat"], case["nphi"]
    set_layers(p, synth.EARTH4)
    for i, c in enumerate(synth.element_counts(case.get("n_elem", 24))):
        p.ne_layer[i] = max(1, c)
    p.rotation = 1 if case.get("rotation") else 0
    p.scheme = 2 if case.get("trap") else 0
    p.visc3d_precision = PRECISION[case.get("precision", "fp64")]
    p.toroidal = 1 if case.get("toroidal") else 0
    return p


def _field(seed, lmax, nlat, nphi, std, mean):
    lf = min(32, lmax)
    return synth.random_sh_field(seed, lf, lf, nlat, nphi, std, mean)


def _pert(p, f2d):
    """The lateral log10-viscosity pattern in every Maxwell element, bottom-up."""
    out = []
    for i in range(p.n_layer - 1, -1, -1):
        on = p.rheology[i] == VG_RHEOL_MAXWELL
        out += [f2d if on else np.zeros_like(f2d)] * p.ne_layer[i]
    return np.stack(out)


def _model(case, seed):
    """A model in the middle of a run: reference state, lateral viscosity, a few intervals of memory; with its ice
    history (N_ICE interval-end fields on the host)."""
    nlat, nphi = case["nlat"], case["nphi"]
    p = _params(case)
    m = vlib.Model(p)
    ice = synth.ice_caps(seed, 6, nlat, nphi).reshape(-1)
    topo = (_field(seed + 1, case["lmax"], nlat, nphi, 2500.0, -1500.0) if case.get("sle", True)
            else np.full((nlat, nphi), 1000.0)).reshape(-1)
    m.set_reference(topo, np.zeros(nlat * nphi), 0.4 * ice)
    if case["visc3d"]:
        m.enable_visc3d(_pert(p, np.clip(_field(seed + 2, case["lmax"], nlat, nphi, 0.4, 0.0), -1.0, 1.0)))
    ices = [(0.45 + 0.05 * math.sin(2 * math.pi * k / N_ICE)) * ice for k in range(N_ICE)]
    return m, topo, ices


def _spectra(rng, lmax, n):
    """Load spectra in kg/m^2, white up to degree 4 and falling as 1/l beyond, real at m = 0."""
    l = np.concatenate([np.arange(k, lmax + 1) for k in range(lmax + 1)])
    m = np.concatenate([np.full(lmax + 1 - k, k) for k in range(lmax + 1)])
    z = rng.standard_normal((n, l.size)) + 1j * rng.standard_normal((n, l.size)) * (m > 0)
    return 1e5 * z / np.maximum(l, 4)


def _members(case):
    sizes = [0, 8, -5, 16, 3, -8]
    out = []
    for i in range(case["members"]):
        lmax = max(20, case["lmax"] + sizes[i])
        out.append({"lmax": lmax, "nlat": lmax + 1, "nphi": 2 * (lmax + 1), "n_elem": case["n_elem"], "sle": True,
                    "visc3d": i % 2 == 0, "precision": case["precision"] if i % 2 == 0 else "fp64"})
    return out


class _Rsl:
    """The handle's device-resident rsl as a tensor (no copy); it holds the model, whose memory it is."""

    def __init__(self, m):
        self.m = m
        self.__cuda_array_interface__ = {"shape": (m.p.nlat, m.p.nphi), "typestr": "<f8", "version": 3,
                                         "data": (m.rsl_device_ptr(), False)}


def _rsl(m):
    return torch.as_tensor(_Rsl(m), device="cuda")


def _on_device(ices):
    return torch.from_numpy(np.stack(ices)).cuda()


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind, s = case["kind"], {"case": case, "k": 0}
    if kind == "sht":
        s["m"] = vlib.Model(_params(case))
        s["f"] = (synth.ice_caps(seed, 6, case["nlat"], case["nphi"])
                  + _field(seed + 1, case["lmax"], case["nlat"], case["nphi"], 2500.0, -1500.0)).reshape(-1)
        s["q"] = _spectra(rng, case["lmax"], 1)[0]
        return s
    if kind == "batch":
        s["ms"], s["ice"] = [], []
        for i, c in enumerate(_members(case)):
            m, _, ices = _model(c, seed + 100 * i)
            s["ms"].append(m)
            s["ice"].append(_on_device(ices))
        torch.cuda.synchronize()
        for _ in range(3):
            run(s)
        return s
    m, topo, ices = _model(case, seed)
    s["m"] = m
    if kind == "response":
        s["sigma"] = _spectra(rng, case["lmax"], 4)
        m.set_dt((15.0 if case["visc3d"] else 50.0) * synth.SEC_PER_YEAR)
        for _ in range(3):
            run(s)
        return s
    if kind == "grad":
        for k in range(2):
            m.update(ices[k], case["dt_yr"])
        s["ice"] = np.stack([ices[(2 + k) % N_ICE] for k in range(case["nsteps"])])
        land = np.flatnonzero(topo > 0.0)
        s["sites"] = rng.choice(land, min(case["sites"], land.size), replace=False).astype(np.int32)
        s["obs"] = rng.normal(0.0, 5.0, (case["nsteps"], s["sites"].size))
        return s
    s["ice"] = ices if case["host"] else _on_device(ices)
    torch.cuda.synchronize()
    for _ in range(3):
        run(s)
    return s


# ---------------------------------------------------------------- run


def run(s):
    case = s["case"]
    kind, k = case["kind"], s["k"]
    s["k"] = k + 1
    if kind == "sht":
        return {"q": s["m"].analysis(s["f"]), "f": s["m"].synthesis(s["q"])}
    if kind == "response":
        m, sigma = s["m"], s["sigma"][k % 4]
        m.begin_step()
        u, n = m.apply(sigma)
        m.advance(sigma)
        return {"u": u, "n": n}
    if kind == "grad":
        out = s["m"].sle_misfit_grad(s["ice"], case["dt_yr"], s["sites"], s["obs"], ckpt_every=case["ckpt"],
                                     want_pert=case["visc3d"])
        return list(out)
    if kind == "batch":
        vlib.update_batch(s["ms"], [t[k % N_ICE].data_ptr() for t in s["ice"]], case["dt_yr"], on_device=True)
        return [_rsl(m) for m in s["ms"]]
    m = s["m"]
    if case["host"]:
        m.update(s["ice"][k % N_ICE], case["dt_yr"])
        rsl, z_bed, c, sigma = m.fields()
        out = {"rsl": rsl, "z_bed": z_bed, "C": c, "sigma": sigma}
        return out if case["sle"] else {**out, "drift": m.drift()}
    m.update_device(s["ice"][k % N_ICE].data_ptr(), case["dt_yr"])
    if not case["sle"]:  # no ocean, so rsl stays zero: the result is the viscous surface displacement
        return {"drift": m.drift()}
    return {"rsl": _rsl(m)}


# ---------------------------------------------------------------- work


def _sub_steps(case):
    # Maxwell-CFL count of the synthetic earth: rate of the softest element, a decade below the layer's viscosity
    # with lateral viscosity
    rate = 0.9e11 / 5e20 * (10.0 if case["visc3d"] else 1.0)
    return max(1, math.ceil(rate * case["dt_yr"] * synth.SEC_PER_YEAR - 1e-9))


def _sht_work(c, fields):
    """One Gauss-grid transform of `fields` fields: the field and its spectrum once, an FFT per row, the Legendre sums
    with the equatorial symmetry."""
    nlm, ng = (c["lmax"] + 1) * (c["lmax"] + 2) // 2, c["nlat"] * c["nphi"]
    return fields * 8.0 * (ng + 2 * nlm), fields * (2.5 * ng * math.log2(c["nphi"]) + 2.0 * nlm * c["nlat"])


def _sub_step_work(c):
    """One sub-step: the memory read and written once, the band sweeps, eight sea-level iterations of an analysis and
    two syntheses, and with lateral viscosity the tensor transforms (products and quadratures, the rows by FFT)."""
    nk, ne = (c["lmax"] + 1) * (c["lmax"] + 2) // 2 - 1, c["n_elem"]
    chan = 6 if c.get("toroidal") else 4
    by = 2.0 * 8 * 6 * chan * ne * nk
    fl = 2.0 * nk * 4 * (ne + 1) * 2 * 19 + 6 * chan * ne * nk * 10.0
    if c.get("sle", True):
        fl += 8 * _sht_work(c, 3)[1]
    if c["visc3d"]:
        ne3d, npr = 0.54 * ne, 10 if c.get("toroidal") else 6
        fl += 2 * npr * 6 * ne3d * (nk * c["nlat"] * 1.0)
        fl += 2 * 2.5 * 18 * ne3d * c["nlat"] * c["nphi"] * math.log2(c["nphi"])
        by += 8.0 * ne3d * c["nlat"] * c["nphi"]
    return by, fl


def work(case):
    kind = case["kind"]
    if kind == "sht":
        by, fl = _sht_work(case, 2)
    elif kind == "response":
        by, fl = _sub_step_work({**case, "sle": False})
    elif kind == "batch":
        by = fl = 0.0
        for c in _members(case):
            c = {**c, "dt_yr": case["dt_yr"]}
            b, f = _sub_step_work(c)
            by, fl = by + _sub_steps(c) * b, fl + _sub_steps(c) * f
    else:
        n = _sub_steps(case) * (3 if case.get("trap") else 1)
        if kind == "grad":
            n *= 2 * case["nsteps"]
        by, fl = (n * v for v in _sub_step_work(case))
    return {"bytes": by, "flops": fl}


# ---------------------------------------------------------------- exact


def _legendre(lmax, x):
    """Orthonormal associated Legendre functions without the Condon-Shortley phase, [lm (m-major)][x]."""
    out, s = [], np.sqrt((1.0 - x) * (1.0 + x))
    pmm = np.full(x.size, math.sqrt(1.0 / (4.0 * math.pi)))
    for m in range(lmax + 1):
        if m:
            pmm = pmm * s * math.sqrt((2.0 * m + 1.0) / (2.0 * m))
        a, b = np.zeros_like(x), pmm
        out.append(b)
        for l in range(m + 1, lmax + 1):
            c = math.sqrt((2.0 * l + 1.0) / ((l - m) * (l + m)))
            d = math.sqrt((l + m - 1.0) * (l - m - 1.0) / (2.0 * l - 3.0)) if l > m + 1 else 0.0
            a, b = b, c * (math.sqrt(2.0 * l - 1.0) * x * b - d * a)
            out.append(b)
    return np.stack(out)


def exact(case, seed):
    """The transforms have a closed form; a time step's value is the model's own."""
    if case["kind"] != "sht":
        return None
    lmax, nlat, nphi = case["lmax"], case["nlat"], case["nphi"]
    rng = np.random.default_rng(seed)
    f = (synth.ice_caps(seed, 6, nlat, nphi) + _field(seed + 1, lmax, nlat, nphi, 2500.0, -1500.0))
    q = _spectra(rng, lmax, 1)[0]
    x, w = np.polynomial.legendre.leggauss(nlat)
    x, w = x[::-1], w[::-1]
    P = _legendre(lmax, x)
    beg = np.concatenate([[0], np.cumsum(lmax + 1 - np.arange(lmax + 1))])
    F = np.fft.rfft(f, axis=1)[:, : lmax + 1] * (2.0 * math.pi / nphi)
    qa = np.concatenate([P[beg[m]: beg[m + 1]] @ (w * F[:, m]) for m in range(lmax + 1)])
    G = np.zeros((nlat, nphi // 2 + 1), complex)
    for m in range(lmax + 1):
        G[:, m] = q[beg[m]: beg[m + 1]] @ P[beg[m]: beg[m + 1]]
    return {"q": qa, "f": (np.fft.irfft(G, nphi, axis=1) * nphi).reshape(-1)}
