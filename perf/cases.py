"""Measured cases of the GPU path: what one outer iteration of a 3D-PDR run asks of the library.

An outer iteration traces the columns and the UV field along the rays, evaluates the reaction
rates, integrates the chemistry of every cell, solves the level populations of the coolants from
their line optical depths, and closes with the heating, the thermal-balance update and the level
convergence check.  Each case is one of these steps through its public entry point, over the sizes
and forms it meets: a handful of cells (latency), an ordinary batch, a grid; the reduced and the
full network; the FP64 and the mixed form; device buffers and the host-buffer call of the Fortran
driver.  Inputs follow the distributions of the benchmark's configurations (workloads.py).

The rate constants and populations that a step takes as *inputs* are made here in plain torch, so
that they depend on the seed alone and not on another kernel of the library; exact() uses the same
plain evaluations.
"""
import csv
import math
import os
import sys

import numpy as np
import torch

PKG = os.path.join(os.getcwd(), "3d-pdr_gb300")
if PKG not in sys.path:
    sys.path.insert(0, PKG)
import pdrgpu as G  # noqa: E402
import workloads as W  # noqa: E402

F8 = torch.float64
KB, CL, HP = 1.38065040e-16, 2.99792458e+10, 6.62606896e-27
EV, AU, MP, PC = 1.60217646e-12, 1.66053878e-24, 1.67262164e-24, 3.08568025e+18
YEAR = 3.1556926e7
COOLANTS = ("CII", "CI", "OI", "CO")


def listed():
    return [
        # one small request (the 4^3 grid of the smallest configuration): a solve as long as its slowest cell
        {"name": "chem_reduced_mixed_64", "kind": "chem", "network": "reduced", "precision": "mixed", "ncell": 64},
        # an ordinary served batch, two waves of the persistent grid and a remainder
        {"name": "chem_reduced_mixed_5003", "kind": "chem", "network": "reduced", "precision": "mixed", "ncell": 5003},
        # a whole small grid (40^3), the work that dominates a run
        {"name": "chem_reduced_mixed_64000", "kind": "chem", "network": "reduced", "precision": "mixed", "ncell": 64000},
        # the Fortran driver's call: host buffers, FP64, copies included
        {"name": "chem_reduced_host_fp64_1500", "kind": "host", "network": "reduced", "precision": "fp64", "ncell": 1500},
        # the full network's block integrator, three cells deep on every SM slot
        {"name": "chem_full_mixed_900", "kind": "chem", "network": "full", "precision": "mixed", "ncell": 900},
        # the rate constants of a grid, reduced network
        {"name": "rates_reduced_100003", "kind": "rates", "network": "reduced", "ncell": 100003, "nrays": 12, "zeta": False},
        # the rate constants of a full-network batch, each cell with its own cosmic-ray rate
        {"name": "rates_full_8000", "kind": "rates", "network": "full", "ncell": 8000, "nrays": 12, "zeta": True},
        # CO level populations in the default form (the reference's elimination)
        {"name": "levpop_co_fp64_20011", "kind": "levpop", "coolant": "CO", "precision": "fp64", "ncell": 20011,
         "nrays": 12, "pseudo1d": False, "line": False},
        # CO level populations of a grid in the mixed form
        {"name": "levpop_co_mixed_64000", "kind": "levpop", "coolant": "CO", "precision": "mixed", "ncell": 64000,
         "nrays": 12, "pseudo1d": False, "line": False},
        # a fine-structure coolant of a grid, with the per-line emission
        {"name": "levpop_cii_fp64_100000", "kind": "levpop", "coolant": "CII", "precision": "fp64", "ncell": 100000,
         "nrays": 12, "pseudo1d": False, "line": True},
        # UV field, the columns the rates need and the CO optical depths along the rays of a lattice
        {"name": "rays_29", "kind": "rays", "coolant": "CO", "side": 29, "points": 12},
        # the end of an iteration: heating, thermal balance, level convergence of a grid
        {"name": "outer_100000", "kind": "outer", "ncell": 100000},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["chem", "chem", "chem", "host", "rates", "rates", "levpop", "levpop", "rays", "outer"])
    if kind == "chem":
        network = rng.choice(["reduced", "reduced", "full"])
        precision = rng.choice(["mixed", "mixed", "fp64"]) if network == "reduced" else "mixed"
        hi = 900 if network == "full" else (64000 if precision == "mixed" else 8000)
        return {"kind": kind, "network": network, "precision": precision, "ncell": _log_int(rng, 8, hi)}
    if kind == "host":
        return {"kind": kind, "network": "reduced", "precision": rng.choice(["fp64", "mixed"]), "ncell": _log_int(rng, 30, 6000)}
    if kind == "rates":
        network = rng.choice(["reduced", "full"])
        return {"kind": kind, "network": network, "ncell": _log_int(rng, 50, 100000 if network == "reduced" else 8000),
                "nrays": 12, "zeta": rng.random() < 0.5}
    if kind == "levpop":
        coolant = rng.choice(["CII", "CI", "OI", "CO", "CO"])
        precision = rng.choice(["fp64", "mixed"])
        return {"kind": kind, "coolant": coolant, "precision": precision, "ncell": _log_int(rng, 50, 64000 if coolant == "CO" else 100000),
                "nrays": 12, "pseudo1d": rng.random() < 0.25, "line": rng.random() < 0.5}
    if kind == "rays":
        return {"kind": kind, "coolant": rng.choice(["CII", "CI", "OI", "CO"]), "side": _log_int(rng, 4, 29), "points": rng.randint(5, 12)}
    return {"kind": kind, "ncell": _log_int(rng, 100, 100000)}


# ------------------------------------------------------------------ seeded draws

class _Draw:
    def __init__(self, seed):
        self.g = torch.Generator(device="cuda")
        self.g.manual_seed(int(seed))

    def u(self, lo, hi, *shape):
        return lo + (hi - lo) * torch.rand(shape, generator=self.g, device="cuda", dtype=F8)

    def logu(self, lo, hi, *shape):
        return 10.0 ** self.u(lo, hi, *shape)


def _cells(d, network, n, nrays=12):
    """Physical conditions of n cells, the distributions of workloads.chemistry()."""
    full = network == "full"
    c = {"n_H": d.logu(2.0, 5.0, n),
         "T": d.logu(1.0, math.log10(2000.0), n) if full else d.u(10.0, 300.0, n),
         "Td": d.u(10.0, 20.0, n)}
    G0 = d.logu(0.0, 5.0, n) if full else torch.full((n,), 10.0, dtype=F8, device="cuda")
    c["AV"] = d.u(0.0, 10.0, n, nrays)
    cols = torch.zeros((n, nrays, 5), dtype=F8, device="cuda")
    cols[..., 0] = d.logu(14.0, 22.0, n, nrays)
    for k in (2, 3, 4):
        cols[..., k] = d.logu(10.0, 18.0, n, nrays)
    c["column5"] = cols
    c["rad"] = (G0 / nrays)[:, None].repeat(1, nrays).contiguous()
    return c


# ------------------------------------------------------------------ plain evaluation of the network and its rates

_TABLES = {}


def _tables(name):
    """Species, reactions, branches and ODE slots of a network, parsed from its data files."""
    if name in _TABLES:
        return _TABLES[name]
    data = os.path.join(os.getcwd(), "data")

    def rows(f):
        return [[x.strip() for x in r] for r in csv.reader(open(os.path.join(data, f))) if any(x.strip() for x in r)]

    def num(s):
        return float(s) if s else 0.0
    spec = [r[1] for r in rows("species_%s.d" % name)]
    layout = rows("layout_%s.d" % name)
    slot = {r[2]: int(r[0]) - 1 for r in layout}
    slot[spec[-1]] = len(spec) - 1
    xe = [int(r[3]) for r in layout]
    R = []
    for f in rows("rates_%s.d" % name):
        r = {"re": f[1:4], "pr": f[4:8], "a": num(f[8]), "b": num(f[9]), "g": num(f[10]), "lo": num(f[12]), "hi": num(f[13]), "dup": 0}
        if R and R[-1]["re"] == r["re"] and R[-1]["pr"] == r["pr"]:
            R[-1]["dup"] = R[-1]["dup"] or 1
            r["dup"], r["lo"] = R[-1]["dup"] + 1, R[-1]["hi"]
        R.append(r)
    for r in R:
        (r1, r2, r3), p = r["re"], r["pr"]
        ion = lambda x: (p[0], p[1]) in ((x + "+", "e-"), ("e-", x + "+"))  # noqa: E731
        if r2 == "PHOTON":
            k = "PHOTO"
            if not r3:
                k = ("H2" if r1 == "H2" else "HD" if r1 == "HD" else "CO" if r1 == "CO" and "C" in p and "O" in p else
                     "CI" if r1 == "C" and ion("C") else "PHOTO")
        elif r2 in ("CRP", "CRPHOT", "FREEZE", "ELFRZE", "CRH", "PHOTD", "THERM"):
            k = r2
        elif r2.startswith("#"):
            k = "GRAIN"
        elif r2 in ("XRAY", "XRSEC", "XRLYA", "XRPHOT"):
            k = "XRAY"
        elif r1 == "H" and r2 == "H" and r3 in ("", "#") and p[0] == "H2" and p[1] in ("", "#"):
            k = "H2FORM"
        else:
            k = "PAH" if any(x in ("PAH", "PAH0", "PAH+", "PAH-") for x in r["re"]) else "THERMAL"
        r["kind"] = k
        one = r2 in ("PHOTON", "CRP", "CRPHOT", "", "FREEZE", "ELFRZE", "CRH", "PHOTD", "THERM") or r2.startswith("#")
        r["ode"] = "X" if k == "XRAY" else "G" if r3 == "#" else "U" if one else "B"
        r["sa"], r["sb"] = slot[r1], slot[r2] if r["ode"] == "B" else None
        r["sp"] = [slot[x] for x in p if x in slot and slot[x] < len(spec) - 1]
    _TABLES[name] = {"spec": spec, "xe": xe, "reac": R}
    return _TABLES[name]


LAM = [910., 950., 1000., 1050., 1110., 1180., 1250., 1390., 1490., 1600., 1700., 1800., 1900., 2000., 2100., 2190., 2300., 2400.,
       2500., 2740., 3440., 4000., 4400., 5500., 7000., 9000., 12500., 22000., 34000., 1.0e9]
XLAM = [5.76, 5.18, 4.65, 4.16, 3.73, 3.40, 3.11, 2.74, 2.63, 2.62, 2.54, 2.50, 2.58, 2.78, 3.01, 3.12, 2.86, 2.58, 2.35, 2.00,
        1.58, 1.42, 1.32, 1.00, 0.75, 0.48, 0.28, 0.12, 0.05, 0.00]
SCO = [[0.000, -1.408e-02, -1.099e-01, -4.400e-01, -1.154, -1.888, -2.760, -4.001],
       [-8.539e-02, -1.015e-01, -2.104e-01, -5.608e-01, -1.272, -1.973, -2.818, -4.055],
       [-1.451e-01, -1.612e-01, -2.708e-01, -6.273e-01, -1.355, -2.057, -2.902, -4.122],
       [-4.559e-01, -4.666e-01, -5.432e-01, -8.665e-01, -1.602, -2.303, -3.146, -4.421],
       [-1.303, -1.312, -1.367, -1.676, -2.305, -3.034, -3.758, -5.077],
       [-3.883, -3.888, -3.936, -4.197, -4.739, -5.165, -5.441, -6.446]]


def _natural(x, y):
    """Second derivatives of the natural cubic splines through y[..., i] at x[i]."""
    n = len(x)
    y2, u = [torch.zeros_like(y[..., 0]) for _ in range(n)], [torch.zeros_like(y[..., 0]) for _ in range(n)]
    for i in range(1, n - 1):
        sig = (x[i] - x[i - 1]) / (x[i + 1] - x[i - 1])
        p = sig * y2[i - 1] + 2.0
        y2[i] = (sig - 1.0) / p
        u[i] = (6.0 * ((y[..., i + 1] - y[..., i]) / (x[i + 1] - x[i]) - (y[..., i] - y[..., i - 1]) / (x[i] - x[i - 1]))
                / (x[i + 1] - x[i - 1]) - sig * u[i - 1]) / p
    y2[n - 1] = torch.zeros_like(y[..., 0])
    for i in range(n - 2, -1, -1):
        y2[i] = y2[i] * y2[i + 1] + u[i]
    return torch.stack(y2, -1)


def _spline(x, y, y2, at):
    """The splines y (one for all points, or one for each) at the points `at`."""
    xa = torch.tensor(x, dtype=F8, device=at.device)
    lo = torch.searchsorted(xa, at.contiguous()).clamp(1, len(x) - 1)

    def pick(v, i):
        return v[i] if v.dim() == 1 else v.gather(-1, i[..., None])[..., 0]
    h = xa[lo] - xa[lo - 1]
    A, B = (xa[lo] - at) / h, (at - xa[lo - 1]) / h
    return A * pick(y, lo - 1) + B * pick(y, lo) + ((A ** 3 - A) * pick(y2, lo - 1) + (B ** 3 - B) * pick(y2, lo)) * h * h / 6.0


def _scatter(av, lam):
    x = torch.tensor(XLAM, dtype=F8, device=av.device)
    tl = (av / 1.086) * _spline(LAM, x, _natural(LAM, x), lam)
    A, K = [1.000, 2.006, -1.438, 0.7364, -0.5076, -0.0592], [0.7514, 0.8490, 1.013, 1.282, 2.005, 5.832]
    far = sum(a * torch.where(k * tl < 100.0, torch.exp(-k * tl), torch.zeros_like(tl)) for a, k in zip(A[1:], K[1:]))
    return torch.where(tl < 1.0, A[0] * torch.exp(-K[0] * tl), far)


def _h2shield(n, dopw):
    td = n * 0.5 * 1.497358985e-2 * 1.0e-2 / dopw
    safe = td.clamp(min=1e-300)
    jd = torch.where(td < 2.0, torch.exp(-0.666666667 * td), torch.where(td < 10.0, 0.638 * safe ** -1.25,
                     torch.where(td < 100.0, 0.505 * safe ** -1.15, 0.344 * safe ** -1.0667)))
    r = 8.0e7 / (1.772453851 * dopw)
    t = 3.02 * (r * 1.0e3) ** -0.064
    u = torch.sqrt(td * r) / t
    return jd + r / (t * torch.sqrt(0.785398163 + u * u))


def _coshield(nco, nh2):
    x, z = [12.0 + i for i in range(8)], [18.0 + i for i in range(6)]
    a = torch.log10(nco + 1.0).clamp(x[0], x[-1])
    b = torch.log10(nh2 + 1.0).clamp(z[0], z[-1])
    s = torch.tensor(SCO, dtype=F8, device=a.device).T.contiguous()          # [nco][nh2]
    s2 = _natural(z, s)
    y = torch.stack([_spline(z, s[i], s2[i], b) for i in range(8)], -1)
    return 10.0 ** _spline(x, y, _natural(x, y), a)


def _h2_formation(T, Td):
    stick = 1.0 / (1.0 + 0.04 * torch.sqrt(T + Td) + 0.2 * T / 1e2 + 0.08 * (T / 1e2) ** 2)
    eff = []
    for es, eh2, ehp in ((110.0, 320.0, 450.0), (260.0, 520.0, 800.0)):
        sq = (1.0 + math.sqrt((3.0e4 - es) / (ehp - es))) ** 2
        f1 = 0.005 * 1e-10 / (2 * 3.0e12 * torch.exp(-eh2 / Td))
        f2 = sq / 4.0 * torch.exp(-es / Td)
        eps = 1.0 / (1.0 + 1.3e13 / 2e-10 * torch.exp(-1.5 * 3.0e4 / Td) * sq)
        eff.append(1.0 / (1.0 + f1 + f2) * eps)
    return 0.5 * 1.45e5 * torch.sqrt(T / 1e2) * (8.473e-22 * eff[0] + 7.908e-22 * eff[1]) * stick


PHYS = dict(zeta_s=5e-17, omega=0.42, grain_radius=1e-7, metallicity=1.0, g2d=100.0, v_turb_kms=1.0)


def _rate_constants(name, c, zeta=None):
    """The rate constants of every cell, (ncell, nreac), in plain torch."""
    T, Td, rad, AV, col = c["T"], c["Td"], c["rad"], c["AV"], c["column5"]
    z = zeta if zeta is not None else torch.full_like(T, PHYS["zeta_s"] / 1.3e-17)
    dopw = 1.0e5 / (1000.0 * 1.0e-8)
    R = _tables(name)["reac"]
    out = torch.zeros((len(T), len(R)), dtype=F8, device=T.device)
    nco, nh2 = col[..., 2], col[..., 0]
    u, w = torch.log10(nco + 1.0), torch.log10(nh2 + 1.0)
    lbar = ((5675.0 - 200.6 * w) - (571.6 - 24.09 * w) * u + (18.22 - 0.7664 * w) * u * u).clamp(913.6, 1076.1)
    sc1000 = _scatter(AV, torch.full_like(AV, 1000.0))
    for i, r in enumerate(R):
        a, b, g, k = r["a"], r["b"], r["g"], r["kind"]
        if k == "H2" or k == "HD":
            v = (a * rad * _h2shield(col[..., 0 if k == "H2" else 1], dopw) * sc1000 / 2.0).sum(1)
        elif k == "CO":
            v = (a * rad * _coshield(nco, nh2) * _scatter(AV, lbar) / 2.0).sum(1)
        elif k == "CI":
            tau = g * AV + 1.1e-17 * col[..., 3] + 0.9 * T[:, None] ** 0.27 * (nh2 / 1.59e21) ** 0.45
            v = (a * rad * torch.exp(-tau) / 2.0).sum(1)
        elif k == "PHOTO":
            v = (a * rad * torch.exp(-g * AV) / 2.0).sum(1)
        elif k == "PHOTD":
            y = torch.where(T < 50.0, 3.5e-3, torch.where(T < 85.0, 4.0e-3, torch.where(T < 100.0, 5.5e-3, 7.5e-3)))
            v = (1.7e8 * rad * torch.exp(-1.8 * AV) * 2.4e-22).sum(1) * y
        elif k == "H2FORM":
            v = _h2_formation(T, Td)
        elif k == "PAH":
            v = a * (T / 100.0) ** b * 0.4
        elif k == "THERMAL":
            v = a * (T / 300.0) ** b * torch.exp(-g / T)
            if g < -200.0:
                v = torch.where(T < r["lo"], 0.0, v)
        elif k == "CRP":
            v = a * z
        elif k == "CRPHOT":
            v = a * z * (T / 300.0) ** b * g / (1.0 - PHYS["omega"])
        elif k in ("FREEZE", "ELFRZE"):
            cion = 1.0 if b == 0.0 else (1.0 + 16.71e-4 / (PHYS["grain_radius"] * T) if b == 1.0 else 0.0)
            v = a * 4.57e4 * 2.4e-22 * torch.sqrt(T / g) * cion * 0.3
        elif k == "CRH":
            v = 2.06e-3 * z * 2.4e-22 * (1.0e5 if g <= 1210.0 else 0.0)
        elif k == "THERM":
            v = math.sqrt(2.0 * 1.5e15 * KB / (math.pi ** 2 * AU) * a / g) * torch.exp(-a / Td)
        else:
            v = torch.full_like(T, a if k == "GRAIN" else 0.0)
        if r["dup"] and k in ("THERMAL", "PHOTO", "CRP", "CRPHOT"):
            # the first member of the group whose range holds T, else its last
            head = i - (r["dup"] - 1)
            last = i
            while last + 1 < len(R) and R[last + 1]["dup"] > R[last]["dup"]:
                last += 1
            sel = torch.full_like(T, last, dtype=torch.long)
            for m in range(last, head - 1, -1):
                sel = torch.where(T <= R[m]["hi"], m, sel)
            v = torch.where(sel == i, v, 0.0)
        if not r["re"][0].startswith("G"):
            v = v.clamp(max=1.0)
        out[:, i] = torch.where(v < 1.0e-99, 0.0, v)
    return out


# ------------------------------------------------------------------ plain evaluation of a coolant

_COOL = {}


def _coolant(key):
    """A LAMDA file as the library reads it: levels, A, B, frequencies, collision tables."""
    if key in _COOL:
        return _COOL[key]
    fname, n, _ = G.COOLANTS[key]
    L = open(os.path.join(os.getcwd(), "data", fname)).read().split("\n")
    at = 7
    E, g = np.zeros(n), np.zeros(n)
    for k in range(n):
        f = L[at + k].split()
        E[k], g[k] = float(f[1]) * CL * HP, float(f[2])
    at += n + 1
    nlin = int(L[at].split()[0])
    at += 2
    A, B, F = np.zeros((n, n)), np.zeros((n, n)), np.zeros((n, n))
    lines = []
    for k in range(nlin):
        f = L[at + k].split()
        i, j = int(f[1]) - 1, int(f[2]) - 1
        F[i, j] = F[j, i] = float(f[4]) * 1e9
        A[i, j] = float(f[3])
        B[i, j] = A[i, j] / (2.0 * HP * F[i, j] ** 3 / CL ** 2)
        B[j, i] = B[i, j] * (g[i] / g[j])
        lines.append((i, j))
    F = np.where(F == 0.0, np.abs(E[:, None] - E[None, :]) / HP, F)
    at += nlin + 1
    npart = int(L[at].split()[0])
    at += 1
    part = {}
    for _ in range(npart):
        p = int(L[at + 1].split()[0])
        ncol, m = int(L[at + 3].split()[0]), int(L[at + 5].split()[0])
        at += 7
        t = []
        while len(t) < m:
            t += [float(x) for x in L[at].split()]
            at += 1
        at += 1
        C = np.zeros((m, n, n))
        for k in range(ncol):
            f = L[at + k].split()
            i, j = int(f[1]) - 1, int(f[2]) - 1
            v = np.array([float(x) for x in f[3:3 + m]])
            C[:, i, j] = v
            C[:, j, i] = np.where(v != 0.0, v * (g[i] / g[j]) * np.exp(-(E[i] - E[j]) / (KB * np.array(t[:m]))), 0.0)
        at += ncol
        part[p] = (np.array(t[:m]), C)
    d = lambda v: torch.tensor(v, dtype=F8, device="cuda")  # noqa: E731
    _COOL[key] = {"n": n, "lines": lines, "E": d(E), "g": d(g), "A": d(A), "B": d(B), "F": d(F),
                  "part": {p: (d(t), d(C)) for p, (t, C) in part.items()}}
    return _COOL[key]


def _lte(key, T, dens):
    c = _coolant(key)
    w = c["g"][None, :] * torch.exp(-c["E"][None, :] / KB / T[:, None])
    return dens[:, None] * w / w.sum(1, keepdim=True)


def _levpop_exact(s, case):
    """Populations, cooling and line emission: rates, escape probabilities, one dense solve per cell."""
    c = _coolant(case["coolant"])
    n, N = c["n"], case["ncell"]
    T, Td, rho = s["T"], s["Td"], s["n_H"]
    nH, nHp, ne, nHe, nH2 = s["partner5"].unbind(1)
    para = torch.where(nH2 > 0, 1.0 / (1.0 + 9.0 * torch.exp(-170.5 / T)), 0.0)
    ortho = torch.where(nH2 > 0, 1.0 - para, 0.0)
    R = torch.zeros((N, n, n), dtype=F8, device="cuda")
    for p, (t, C) in sorted(c["part"].items()):
        k = torch.searchsorted(t, T, right=True)          # first table temperature above T
        hi, lo = k.clamp(max=len(t) - 1), (k - 1).clamp(min=0)
        step = torch.where(hi == lo, 0.0, (T - t[lo]) / torch.where(hi == lo, 1.0, t[hi] - t[lo]))
        one = (k == 0) | (k == len(t))
        step = torch.where(one, 0.0, step)
        dens = {1: nH2, 2: nH2 * para, 3: nH2 * ortho, 4: ne, 5: nH, 6: nHe, 7: nHp}[p]
        R += (C[lo] + (C[hi] - C[lo]) * step[:, None, None]) * dens[:, None, None]
    line = torch.zeros((N, n, n), dtype=F8, device="cuda")
    ngrain = 2.0e-12 * rho
    f32 = lambda v: float(np.float32(v))  # noqa: E731
    for l, (i, j) in enumerate(c["lines"]):
        f, A = float(c["F"][i, j]), float(c["A"][i, j])
        t2 = 2.0 * HP * f ** 3 / CL ** 2
        cmb = t2 / (torch.exp(torch.tensor(HP * f / KB / 2.7, dtype=F8)) - 1.0).item()   # zero for the UV lines
        bb = cmb + t2 / (torch.exp(HP * f / KB / Td) - 1.0) * 2.0 * ngrain * f32(0.01) * (f32(1.3) * f / 3e11)
        ni, nj = s["spop"][:, i], s["spop"][:, j]
        tpop = nj * c["g"][i] / (ni * c["g"][j]) - 1.0
        flat = tpop.abs() < 1e-50
        S = torch.where(flat, HP * f * ni * A / 4.0 / math.pi, t2 / torch.where(flat, 1.0, tpop))
        tau = s["tau"][:, l, :]
        br = torch.where(tau.abs() < 1e-8, 1.0, -torch.expm1(-tau.clamp(min=-5.0)) / torch.where(tau == 0, 1.0, tau))
        br = torch.where(tau < -5.0, (1.0 - math.exp(5.0)) / -5.0, br)
        # pseudo-1D: every ray but the seventh is opaque, and the sum stands for the average
        beta = br[:, 6] + (case["nrays"] - 1) * 1e-50 if case["pseudo1d"] else br.mean(1)
        beta = torch.where(flat, 1.0, beta)
        none = ni == 0.0
        S, beta = torch.where(none, 0.0, S), torch.where(none, 1.0, beta)
        line[:, i, j] = torch.where(none, 0.0, A * HP * f * ni * beta * (S - bb) / torch.where(none, 1.0, S))
        field = (1.0 - beta) * S + beta * bb
        R[:, i, j] += A + c["B"][i, j] * field
        R[:, j, i] += c["B"][j, i] * field
    R = torch.where(R.abs() < 1e-50, 0.0, R)
    M = R.transpose(1, 2).clone()
    idx = torch.arange(n, device="cuda")
    M[:, idx, idx] = M[:, idx, idx] * 0 - (R.sum(2))
    scale = M.abs().amax(2, keepdim=True).clamp(min=1e-300)
    M = M / scale
    M[:, n - 1, :] = 1.0
    b = torch.zeros((N, n, 1), dtype=F8, device="cuda")
    b[:, n - 1, 0] = s["cdens"]
    pop = torch.linalg.solve(M, b)
    pop = (pop + torch.linalg.solve(M, b - M @ pop))[..., 0]
    return pop.clamp(min=0.0), line.sum((1, 2)), line


# ------------------------------------------------------------------ plain integration of the chemistry

def _integrate(name, k, n_H, x0, t_end):
    """The network from x0 to t_end: linearly implicit Euler with polynomial extrapolation over
    macro steps that grow by a constant ratio, every cell in step (numpy, 64 bits)."""
    tab = _tables(name)
    n = len(tab["spec"]) - 1
    N = len(n_H)
    one, el = n + 1, n
    a, b, use, nh = [], [], [], []
    nu = []
    for i, r in enumerate(tab["reac"]):
        if r["ode"] == "X":
            continue
        v = np.zeros(n)
        for p in r["sp"]:
            v[p] += 1.0
        for q in [r["sa"]] * (2 if r["ode"] == "G" else 1) + ([r["sb"]] if r["ode"] == "B" else []):
            if q < n:
                v[q] -= 1.0
        a.append(r["sa"])
        b.append(r["sb"] if r["ode"] == "B" else one)
        nh.append(r["ode"] in "BG")
        use.append(i)
        nu.append(v)
    a, b, nu, xe = np.array(a), np.array(b), np.array(nu), np.array(tab["xe"], dtype=np.float64)
    kn = k[:, use] * np.where(np.array(nh)[None, :], n_H[:, None], 1.0)
    pa, pb = np.zeros((len(a), n)), np.zeros((len(a), n))       # d(slot value)/dx
    for r in range(len(a)):
        for m, s in ((pa, a[r]), (pb, b[r])):
            if s < n:
                m[r, s] = 1.0
            elif s == el:
                m[r] = xe

    def parts(x):
        full = np.concatenate([x, (x @ xe)[:, None], np.ones((N, 1))], 1)
        fa, fb = kn * full[:, b], kn * full[:, a]
        return fa * full[:, a], fa, fb

    def f(x):
        return parts(x)[0] @ nu

    def jac(x):
        _, fa, fb = parts(x)
        w = fa[:, :, None] * pa[None] + fb[:, :, None] * pb[None]
        return np.einsum("ri,nrj->nij", nu, w)

    x, t, H = x0.copy(), 0.0, 1.0e-2
    eye = np.eye(n)[None]
    seq = (1, 2, 3, 4, 5, 6, 7, 8)
    while t < t_end:
        H = min(H, t_end - t)
        J = jac(x)
        rows = []
        for q, m in enumerate(seq):
            h = H / m
            inv = np.linalg.inv(eye - h * J)
            y = x
            for _ in range(m):
                y = y + (inv @ (h * f(y))[:, :, None])[:, :, 0]
            row = [y]
            for l in range(1, q + 1):
                row.append(row[l - 1] + (row[l - 1] - rows[q - 1][l - 1]) / (m / seq[q - l] - 1.0))
            rows.append(row)
        x = rows[-1][-1]
        t += H
        H = max(0.35 * t, 1.0e-2)
    return x


# ------------------------------------------------------------------ states

_HANDLES = {}


def _network(name):
    if name not in _HANDLES:
        _HANDLES[name] = G.Network(name)
    return _HANDLES[name]


def _cool(key):
    if key not in _HANDLES:
        _HANDLES[key] = G.Coolant(key)
    return _HANDLES[key]


def _chem_inputs(case, seed):
    name, n = case["network"], case["ncell"]
    c = _cells(_Draw(seed), name, n)
    c["rate"] = torch.cat([_rate_constants(name, {k: v[i:i + 16384] for k, v in c.items()}) for i in range(0, n, 16384)])
    x0 = W.initial_abundances(_tables(name)["spec"], s_plus=(name != "reduced"))
    c["ab0"] = torch.as_tensor(np.tile(x0, (n, 1)), device="cuda")
    return c


def _levpop_inputs(case, seed):
    d, n, key = _Draw(seed), case["ncell"], case["coolant"]
    n_H, T, xH2, xe = d.logu(2.0, 6.0, n), d.u(10.0, 2000.0, n), d.u(0.0, 0.5, n), d.logu(-8.0, -3.0, n)
    s = {"n_H": n_H, "T": T, "Td": d.u(10.0, 20.0, n), "cdens": n_H * W.COOLANT_X[key]}
    s["partner5"] = torch.stack([(1.0 - 2.0 * xH2).clamp(min=0.0) * n_H, xe * n_H, xe * n_H, 0.1 * n_H, xH2 * n_H], 1).contiguous()
    s["spop"] = _lte(key, T, s["cdens"])
    s["tau"] = d.logu(-3.0, 3.0, n, len(_coolant(key)["lines"]), case["nrays"])
    return s


def _rays_inputs(case, seed):
    """A lattice of cells with evaluation points along the 12 base directions (workloads.rays())."""
    d, n, m = _Draw(seed), case["side"], case["points"]
    step = 0.05
    v = torch.as_tensor(W.healpix_base_directions(), device="cuda")
    ax = torch.arange(n, device="cuda", dtype=F8)
    lat = torch.stack(torch.meshgrid(ax, ax, ax, indexing="ij"), -1).reshape(-1, 3)
    pos = lat[:, None, None, :] + torch.arange(m + 1, device="cuda", dtype=F8)[None, None, :, None] * v[None, :, None, :]
    inside = ((pos >= -0.5) & (pos <= n - 0.5)).all(-1)
    ncell = n ** 3
    s = {"epray": (inside.long().cumprod(-1).sum(-1) - 1).to(torch.int32).reshape(-1).contiguous(),
         "offset": torch.arange(ncell * 12, device="cuda", dtype=torch.int64) * (m + 1),
         "xyz": (pos * step).reshape(-1, 3).contiguous()}
    p = pos.round().clamp(0, n - 1).long()
    s["gridpoint"] = (p[..., 0] * n * n + p[..., 1] * n + p[..., 2]).to(torch.int32).reshape(-1).contiguous()
    s["rho"] = d.logu(2.0, 5.0, ncell)
    s["abundance"] = d.logu(-12.0, -2.0, ncell, 33)
    s["T"] = d.u(10.0, 300.0, ncell)
    key = case["coolant"]
    s["pop"] = _lte(key, s["T"], s["rho"] * W.COOLANT_X[key]) * d.u(0.5, 1.5, ncell, _coolant(key)["n"])
    return s


def _outer_inputs(case, seed):
    d, n = _Draw(seed), case["ncell"]
    c = _cells(d, "reduced", n)
    s = {"n_H": c["n_H"], "T": c["T"], "Td": c["Td"], "uv": d.logu(-2.0, 2.0, n), "abundance": d.logu(-12.0, -1.0, n, 33)}
    s["rate"] = torch.cat([_rate_constants("reduced", {k: v[i:i + 16384] for k, v in c.items()}) for i in range(0, n, 16384)])
    s["cooling"] = [d.logu(-25.0, -21.0, n) for _ in COOLANTS]
    sp = _tables("reduced")["spec"]
    s["species"] = [sp.index(x) for x in ("C+", "C", "O", "CO")]
    s["sol"], s["alt"], s["pop"] = [], [], []
    for k, key in zip(s["species"], COOLANTS):
        dens = s["abundance"][:, k] * s["n_H"]
        p = _lte(key, s["T"], dens)
        # a mature iteration: most levels moved by less than the check's 1 %, some by more
        s["sol"].append(p * (1.0 + 0.02 * d.u(-0.6, 0.6, *p.shape)))
        s["alt"].append(p)
        s["pop"].append(p.clone())
    return s


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("chem", "host"):
        s = _chem_inputs(case, seed)
        for k in ("AV", "column5", "rad"):
            s.pop(k)
        net = _network(case["network"])
        opts = G.chem_opts(case["precision"])
        if kind == "chem":
            # what a program that solves batches keeps: a solver instance with its own scratch
            return dict(s, kind=kind, ab=torch.empty_like(s["ab0"]), solver=G.Solver(net, case["ncell"], opts),
                        status=torch.empty(case["ncell"], dtype=torch.int32, device="cuda"))
        h = {k: np.ascontiguousarray(s[k].cpu().numpy()) for k in ("ab0", "rate", "n_H", "T")}
        return dict(h, kind=kind, net=net, opts=opts, ab=np.empty_like(h["ab0"]))
    if kind == "rates":
        d = _Draw(seed)
        c = _cells(d, case["network"], case["ncell"], case["nrays"])
        zeta = d.logu(-1.0, 2.0, case["ncell"]) if case["zeta"] else None
        return dict(c, kind=kind, net=_network(case["network"]), phys=G.phys(**PHYS), zeta=zeta)
    if kind == "levpop":
        return dict(_levpop_inputs(case, seed), kind=kind, cool=_cool(case["coolant"]), pseudo1d=case["pseudo1d"],
                    line=case["line"], precision=case["precision"])
    if kind == "rays":
        s = _rays_inputs(case, seed)
        n = case["side"] ** 3
        r = G.Rays(n, 12, n, n * 12 * (case["points"] + 1), s["epray"].data_ptr(), s["offset"].data_ptr(),
                   s["xyz"].data_ptr(), s["gridpoint"].data_ptr())
        return dict(s, kind=kind, rays=r, cool=_cool(case["coolant"]), vectors=W.healpix_base_directions())
    s = _outer_inputs(case, seed)
    return dict(s, kind=kind, net=_network("reduced"), phys=G.phys(**PHYS), tb=G.ThermalBalance(s["T"].clone()))


def run(s):
    kind = s["kind"]
    if kind == "chem":
        s["ab"].copy_(s["ab0"])                       # the integration is in place
        st = s["solver"].run(s["ab"], s["rate"], s["n_H"], status=s["status"])
        return {"abundance": s["ab"][:, :-1], "electron": s["ab"][:, -1], "status": st}
    if kind == "host":
        np.copyto(s["ab"], s["ab0"])
        st = G.calculate_abundances_host(s["net"], s["ab"], s["rate"], s["n_H"], s["T"], s["opts"])
        return {"abundance": s["ab"][:, :-1], "electron": s["ab"][:, -1], "status": st}
    if kind == "rates":
        rate, st = G.reaction_rates(s["net"], s["phys"], s["T"], s["Td"], s["rad"], s["AV"], s["column5"], zeta=s["zeta"])
        return {"rate": rate, "status": st}
    if kind == "levpop":
        pop, cooling, line, st = G.level_populations(s["cool"], s["n_H"], s["T"], s["Td"], s["partner5"], s["cdens"], s["spop"],
                                                     s["tau"], pseudo1d=s["pseudo1d"], precision=s["precision"], want_line=s["line"])
        return {"pop": pop, "cooling": cooling, "line": line, "ok": st == 1}
    if kind == "rays":
        col, av, rad, uv = G.uvfield(s["rays"], s["rho"], 0, (10.0, 0.0, 0.0), s["vectors"])
        sel = G.column_densities(s["rays"], s["rho"], s["abundance"], species=[5, 0, 17, 3, 9])
        tau = G.optical_depths(s["cool"], s["rays"], s["pop"], s["T"], 1.0e5)
        return {"column": col, "av": av, "rad": rad, "uv": uv, "column5": sel, "tau": tau}
    tb = s["tb"]
    heat = G.heating(s["net"], 0, s["phys"], s["n_H"], s["T"], s["Td"], s["uv"], s["abundance"], s["rate"])
    tb.T.copy_(s["T"])                                # the search starts from this iteration's temperatures
    tb.flags.zero_()
    nconv = tb.update(heat, s["cooling"], level_conv=True, first_time=True)
    s["sol"], s["alt"] = s["alt"], s["sol"]           # the solutions of one iteration after the other
    counts = tb.level_convergence(s["alt"], s["pop"], s["abundance"], s["species"])
    return {"heating": heat, "T": tb.T, "Fmean": tb.Fmean, "Fratio": tb.Fratio, "flags": tb.flags, "cooling": tb.total_cooling,
            "converged": nconv, "counts": counts, "pop": s["pop"]}


def work(case):
    kind = case["kind"]
    if kind in ("chem", "host"):
        full = case["network"] == "full"
        nspec, nreac, n = (215, 2926, 214) if full else (33, 329, 32)
        # counted on the configurations' cells: RHS calls, Jacobians, Newton iterations and steps per cell, with
        # the operation counts of the generated f() and Jacobian and of an n x n factorisation and solve
        nfe, nje, nni, nst = (2046, 196, 2042, 1794) if full else (1656, 187, 1652, 1358)
        frhs, fjac = (37547, 52409) if full else (3986, 5569)
        flops = nfe * frhs + nje * (fjac + 2 * n ** 3 / 3) + nni * (2 * n * n + 4 * n) + nst * 30 * n
        return {"bytes": case["ncell"] * 8.0 * (2 * nspec + nreac + 1), "flops": float(case["ncell"]) * flops}
    if kind == "rates":
        nreac = 2926 if case["network"] == "full" else 329
        R = _tables(case["network"])["reac"]
        photo = sum(r["kind"] in ("PHOTO", "H2", "HD", "CO", "CI", "PHOTD") for r in R)
        nr = case["nrays"]
        # an exponential and a power are taken as 20 operations each
        return {"bytes": case["ncell"] * 8.0 * (nreac + 3 + 7 * nr) + 4.0 * case["ncell"],
                "flops": case["ncell"] * (25.0 * photo * nr + 45.0 * (nreac - photo) + 300.0 * nr)}
    if kind == "levpop":
        c = _coolant(case["coolant"])
        n, L, nr = c["n"], len(c["lines"]), case["nrays"]
        out = n + 1 + (n * n if case["line"] else 0)
        return {"bytes": case["ncell"] * (8.0 * (9 + n + (L * nr) + out) + 4.0),
                "flops": case["ncell"] * (2.0 * n ** 3 / 3 + 6.0 * len(c["part"]) * n * n + 25.0 * L * nr + 60.0 * L)}
    if kind == "rays":
        c = _coolant(case["coolant"])
        n, L, m = case["side"], len(c["lines"]), case["points"]
        N = n ** 3
        # a ray holds about as many points as the lattice leaves it: half of `points` at small sides
        pts = N * 12.0 * max(1.0, m * min(1.0, n / (2.0 * m)))
        return {"bytes": pts * 28.0 + N * 12 * 12.0 + N * 8.0 * (1 + 5 + c["n"] + 1) + N * 8.0 * 12 * (3 + 5 + L) + N * 8.0,
                "flops": pts * (10.0 * 3 + 5 * 5 + 9.0 * L)}
    N = case["ncell"]
    lev = sum(_coolant(k)["n"] for k in COOLANTS)
    return {"bytes": N * (8.0 * (4 + 12 + 33 + 20) + 8.0 * (4 + 12 + 8 + 1) + 8.0 * 3 * lev + 4.0), "flops": N * (400.0 + 4.0 * lev)}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("chem", "host"):
        if case["network"] != "reduced" or case["ncell"] > 64:
            return None                               # minutes of plain integration
        s = _chem_inputs(case, seed)
        x = _integrate("reduced", s["rate"].cpu().numpy(), s["n_H"].cpu().numpy(), s["ab0"].cpu().numpy()[:, :-1], 1.0e7 * YEAR)
        # the electron entry is that of the integrator's last right-hand side, past the end time: no plain value
        return {"abundance": np.where(x < 1e-30, 0.0, x), "electron": None, "status": None}
    if kind == "rates":
        d = _Draw(seed)
        c = _cells(d, case["network"], case["ncell"], case["nrays"])
        zeta = d.logu(-1.0, 2.0, case["ncell"]) if case["zeta"] else None
        B = 16384
        out = [_rate_constants(case["network"], {k: v[i:i + B] for k, v in c.items()}, None if zeta is None else zeta[i:i + B])
               for i in range(0, case["ncell"], B)]
        return {"rate": torch.cat(out), "status": None}
    if kind == "levpop":
        s = _levpop_inputs(case, seed)
        got = [_levpop_exact({k: v[i:i + 4096] for k, v in s.items()}, dict(case, ncell=min(4096, case["ncell"] - i)))
               for i in range(0, case["ncell"], 4096)]
        pop, cooling, line = (torch.cat([g[k] for g in got]) for k in range(3))
        return {"pop": pop, "cooling": cooling, "line": line if case["line"] else None, "ok": None}
    if kind == "rays":
        s = _rays_inputs(case, seed)
        N, m = case["side"] ** 3, case["points"]
        ep = s["epray"].long().reshape(N, 12)
        xyz = s["xyz"].reshape(N, 12, m + 1, 3)
        gp = s["gridpoint"].long().reshape(N, 12, m + 1)
        h = (xyz[:, :, 1:] - xyz[:, :, :-1]).square().sum(-1).sqrt()
        h = torch.where(torch.arange(1, m + 1, device="cuda")[None, None] <= ep[..., None], h, 0.0)
        rho = s["rho"][gp]
        col = ((rho[..., 1:] + rho[..., :-1]) * 0.5 * h * PC).sum(-1)
        f32 = lambda v: float(np.float32(v))  # noqa: E731
        av = col * f32(6.289e-22)
        rad = torch.full_like(av, 10.0 / 12)
        uv = (rad * torch.exp(-av * f32(3.02))).sum(1)
        sel = torch.stack([((lambda q: (q[..., 1:] + q[..., :-1]) * 0.5 * h * PC)(rho * s["abundance"][:, k][gp])).sum(-1)
                           for k in (5, 0, 17, 3, 9)], -1)
        c = _coolant(case["coolant"])
        frac2 = 1.0 / torch.sqrt(8.0 * KB * s["T"] / math.pi / MP + 1.0e10)
        tau = torch.empty((N, len(c["lines"]), 12), dtype=F8, device="cuda")
        for l, (i, j) in enumerate(c["lines"]):
            f1 = float(c["A"][i, j]) * CL ** 3 / (8.0 * math.pi * float(c["F"][i, j]) ** 3)
            t = (s["pop"][:, j] * c["g"][i] - s["pop"][:, i] * c["g"][j])[gp]
            tau[:, l] = ((t[..., 1:] + t[..., :-1]) * 0.5 / c["g"][j] * h * PC).sum(-1) * f1 * frac2[:, None]
        return {"column": col, "av": av, "rad": rad, "uv": torch.where(uv < 1e-50, 0.0, uv), "column5": sel, "tau": tau}
    s = _outer_inputs(case, seed)
    heat = _heating_exact(s)
    cool = sum(s["cooling"])
    fm = heat[:, 11] - cool
    T = torch.where(fm > 0, 1.3 * s["T"], torch.where(fm < 0, (0.7 * s["T"]).clamp(min=2.7), s["T"]))
    return {"heating": heat, "T": T, "Fmean": fm, "Fratio": 2.0 * fm.abs() / (heat[:, 11] + cool).abs(), "flags": None, "cooling": cool,
            "converged": None, "counts": None, "pop": s["sol"]}


def _heating_exact(s):
    """The twelve heating terms of the reduced network, with the driver's single-precision literals."""
    r4 = lambda v: float(np.float32(v))  # noqa: E731
    sp = _tables("reduced")["spec"]
    nr = {r["kind"]: i for i, r in enumerate(_tables("reduced")["reac"]) if r["kind"] in ("H2FORM", "H2", "CI")}
    x = lambda *q: s["abundance"][:, next(sp.index(v) for v in q if v in sp)]  # noqa: E731
    R = lambda i: s["rate"][:, i - 1]  # noqa: E731
    n, T, Td, xe = s["n_H"], s["T"], s["Td"], s["abundance"][:, -1]
    hab = 1.68 * s["uv"]
    xk, xd = KB * T / (13.6 * EV), 6.0 / 13.6
    gam = 2.9e-4 * 0.1 * torch.sqrt(T) * hab / (xe * n)
    dl = xk - xd + gam
    q = torch.full_like(T, 0.5)
    done = torch.zeros_like(T, dtype=torch.bool)
    for _ in range(100):
        nq = q - (q ** 3 + dl * q * q - gam) / (3 * q * q + 2 * dl * q)
        stop = (nq - q).abs() < 1.0e-2
        q = torch.where(done, q, nq)
        done = done | stop
        if bool(done.all()):
            break
    pe = 2.7e-25 * 1.8 * n * 0.1 * hab * ((1.0 - q) ** 2 / q + xk * (q * q - 1.0) / (q * q))
    dlt = hab * torch.sqrt(T) / (xe * n)
    beta = 0.735 / T ** r4(0.068)
    eps = 4.87e-2 / (1.0 + 4.0e-3 * dlt ** r4(0.73)) + 3.65e-2 * (T / 1e4) ** r4(0.7) / (1.0 + 2.0e-4 * dlt)
    pah = 1.30e-24 * eps * hab * n - 4.65e-30 * T ** 0.944 * dlt ** beta * xe * n * n
    wd = 1.0e-26 * hab * n * (5.72 + 3.45e-2 * T ** 0.495) / (1.0 + 7.08e-3 * dlt ** 0.692 * (1.0 + 1.98e-2 * dlt ** 0.52))
    cion = EV * R(nr["CI"] + 1) * x("C") * n
    h2f = 1.5 * EV * R(nr["H2FORM"] + 1) * n * x("H") * n
    h2p = r4(0.4) * EV * R(nr["H2"] + 1) * x("H2") * n
    ncr = 1.0e6 / torch.sqrt(T) / (1.6 * x("H") * torch.exp(-((400.0 / T) ** 2)) + 1.4 * x("H2") * torch.exp(-(18100.0 / (T + 1200.0))))
    fuv = r4(2.2) * EV * 9.0 * R(nr["H2"] + 1) * x("H2") * n / (1.0 + ncr / n)
    cr = r4(9.4) * EV * PHYS["zeta_s"] * n * x("H2")
    turb = 3.5e-28 / 5.0 * n
    e = lambda v: r4(v) * EV  # noqa: E731
    chem = (x("H2+") * n * xe * R(216) * e(10.9) + x("H2+") * n * x("H") * R(155) * e(0.94) + x("HCO+") * n * xe * n * R(240) * e(7.51)
            + x("H3+") * n * xe * n * (R(217) * e(4.76) + R(218) * e(9.23))
            + x("H3O+") * n * xe * n * (R(236) * e(1.16) + R(237) * e(5.63) + R(238) * e(6.27))
            + x("He+", "HE+") * n * x("H2") * n * (R(50) + R(170)) * e(6.51)
            + x("He+", "HE+") * n * x("CO") * n * (R(89) + R(90) + R(91)) * e(2.22))
    acc = 0.35 * torch.exp(-torch.sqrt((Td + T) / 5.0e2)) + 0.1
    gg = 4.003e-12 * n * (1.998e-12 * n) * (math.pi * PHYS["grain_radius"] ** 2) * acc * torch.sqrt(T) * (Td - T)
    tot = pah + cion + h2f + h2p + fuv + cr + turb + chem + gg
    return torch.stack([pe, pah, wd, cion, h2f, h2p, fuv, cr, torch.full_like(pe, 0) + turb, chem, gg, tot], 1)
