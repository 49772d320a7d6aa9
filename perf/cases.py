"""Timed cases of the framework: what its users have it do, over the range of
sizes, precisions and closures they do it at.

Every case goes through the package's public entry points:

  residual, jacobian  one F(t) or J(t) dt on device tensors (the plug points of
                      another Newton driver), FP64 or FP32;
  solve               a solve from t = 0 and its observables on a kept context;
  solute              hnc3d_run_solute on host buffers, as a script calls it;
  pes                 one point of a scan: the context rebound to a moved
                      geometry, a warm-started solve, its free energy and g;
  gradient            dmu/d(q, sigma, eps, x) at a converged t (the backward
                      direction);
  batch               many solutes of uneven sizes in one call;
  solvent             the 3D solve of the pure solvent.

Solvent and thermodynamic state are those of the benchmark (PR-SPC/E water,
rho 0.0333295, beta 1.6889, chi from 1D DRISM at rmax 160 / nrad 4096).
`exact` is a plain torch FP64 restatement of the same equations.
"""
import functools
import math
import random

import numpy as np
import torch

from bgy3d_b200 import (RismContext, find_molecule, hnc3d_run_batch, hnc3d_run_solute, hnc3d_run_solvent,
                        rism_solvent, synthetic_solute)

BASE = {"rho": 0.0333295, "beta": 1.6889, "rmax": 160.0, "nrad": 4096, "dielectric": 78.4, "max-iter": 200}
WATER = "water, PR-SPC/E"
GRIDS = [n for n in range(32, 513, 2) if 2 ** 9 * 3 ** 6 % n == 0]  # even 2^a 3^b
BATCH_GRIDS = [64, 72, 96, 108, 128, 144, 162]


def listed():
    return [
        # one residual at the default grid and box: the smallest call, where launches and latency count
        {"name": "residual-64-f64", "kind": "residual", "nx": 64, "ny": 64, "nz": 64, "half": 10.0, "closure": "HNC",
         "sites": 3, "precision": "fp64"},
        # a Jacobian product of a many-solute grid that is no power of two, FP32
        {"name": "jacobian-108-f32", "kind": "jacobian", "nx": 108, "ny": 108, "nz": 108, "half": 20.0,
         "closure": "KH", "sites": 24, "precision": "fp32"},
        # the product that a plain FP64 solve of the benchmark's solute makes hundreds of
        {"name": "jacobian-256-f64", "kind": "jacobian", "nx": 256, "ny": 256, "nz": 256, "half": 24.0,
         "closure": "KH", "sites": 24, "precision": "fp64"},
        # the same in FP32 on the largest grid (a 150-site solute in a 96 A box)
        {"name": "jacobian-512-f32", "kind": "jacobian", "nx": 512, "ny": 512, "nz": 512, "half": 48.0,
         "closure": "KH", "sites": 150, "precision": "fp32"},
        # a script's call for a small molecule at the default grid and box, g back on the host
        {"name": "solute-64", "kind": "solute", "n": 64, "half": 10.0, "closure": "KH", "molecule": "methanol",
         "precision": "mixed", "tol": 1e-10, "restart": False},
        # water in water as the reference documents it (HNC, 96^3, 20 A box), plain FP64 arithmetic, t and g back
        {"name": "solute-96-hnc", "kind": "solute", "n": 96, "half": 10.0, "closure": "HNC", "molecule": WATER,
         "precision": "fp64", "tol": 1e-10, "restart": True},
        # the benchmark's solve: 24 sites, 256^3, mixed precision
        {"name": "solve-256", "kind": "solve", "n": 256, "half": 24.0, "closure": "KH", "sites": 24,
         "precision": "mixed", "tol": 1e-10},
        # a mid-sized solve on a grid with odd half rows
        {"name": "solve-162", "kind": "solve", "n": 162, "half": 20.0, "closure": "KH", "sites": 17,
         "precision": "mixed", "tol": 1e-10},
        # a point of a potential-energy scan
        {"name": "pes-128", "kind": "pes", "n": 128, "half": 18.0, "closure": "KH", "sites": 12,
         "precision": "mixed", "tol": 1e-10},
        # the adjoint gradient of a mid-sized solute
        {"name": "gradient-128", "kind": "gradient", "n": 128, "half": 18.0, "closure": "KH", "sites": 12,
         "precision": "mixed", "tol": 1e-10},
        # many small and mid-sized solutes at once
        {"name": "batch-10", "kind": "batch", "count": 10, "pick": 7, "closure": "KH", "precision": "mixed",
         "tol": 1e-10},
        # the pure solvent at the grid and box of the documented 3D solvent run
        {"name": "solvent-96", "kind": "solvent", "n": 96, "half": 10.0, "closure": "KH", "tol": 1e-12},
    ]


def _grid(rng, lo, hi):
    """An even 2^a 3^b size, near-uniform in its logarithm."""
    x = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min((n for n in GRIDS if lo <= n <= hi), key=lambda n: abs(math.log(n / x)))


def draw(rng):
    kind = rng.choice(["residual", "residual", "jacobian", "jacobian", "solve", "solve", "solute", "solute", "pes",
                       "gradient", "batch", "solvent"])
    closure = rng.choice(["KH", "KH", "PSE2", "PSE3", "HNC"])
    mixed = rng.choice(["mixed", "mixed", "fp64"])
    h = rng.uniform(0.1875, 0.4)
    if kind in ("residual", "jacobian"):
        nx = _grid(rng, 32, 432)
        ny, nz = (nx, nx) if rng.random() < 0.6 else (_grid(rng, max(32, nx // 2), min(432, 2 * nx)) for _ in "yz")
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "half": round(max(9.0, nx * h / 2), 2),
                "closure": closure, "sites": rng.randint(1, 60), "precision": rng.choice(["fp64", "fp32"])}
    if kind == "solute":
        return {"kind": kind, "n": _grid(rng, 48, 192), "half": round(rng.uniform(10.0, 16.0), 2), "closure": "KH",
                "molecule": rng.choice([WATER, "water", "hydrogen chloride", "carbon disulfide", "methanol",
                                        "butanoic acid", "hexane"]),
                "precision": mixed, "tol": 1e-10, "restart": rng.random() < 0.5}
    if kind == "batch":
        return {"kind": kind, "count": rng.randint(4, 10), "pick": rng.randrange(1 << 20), "closure": "KH",
                "precision": mixed, "tol": 1e-10}
    if kind == "solvent":
        return {"kind": kind, "n": _grid(rng, 48, 96), "half": round(rng.uniform(9.0, 12.0), 2),
                "closure": rng.choice(["KH", "PSE2"]), "tol": 1e-12}
    n = _grid(rng, 64, {"solve": 216, "pes": 162, "gradient": 128}[kind])
    if kind == "gradient" or n > 128:
        mixed = "mixed"
    return {"kind": kind, "n": n, "half": round(max(12.0, n * min(h, 0.3) / 2), 2), "closure": "KH",
            "sites": rng.randint(3, 40), "precision": mixed, "tol": 1e-10}


# ------------------------------------------------------------------ inputs
def _settings(c, n=None, half=None):
    precision = c.get("precision", "fp64")
    return dict(BASE, N=c["n"] if n is None else n, L=c["half"] if half is None else half, closure=c["closure"],
                **{"precision": "mixed" if precision == "fp32" else precision, "norm-tol": c.get("tol", 1e-10)})


@functools.lru_cache(maxsize=8)
def _chi(closure):
    """The solvent's susceptibility, tabulated once per closure as a program does (PSE: the KH table)."""
    closure = "HNC" if closure == "HNC" else "KH"
    return rism_solvent(find_molecule(WATER), dict(BASE, L=24.0, N=256, closure=closure, **{"norm-tol": 1e-12}))[
        "susceptibility"]


def _solute(c, seed, half, sites=None):
    """The case's solute: a molecule of the database, turned at random, or a synthetic one."""
    if "molecule" not in c:
        n = c["sites"] if sites is None else sites
        return synthetic_solute(n, radius=14.0 if n > 60 else min(6.0, 0.4 * half), seed=seed)
    rng = np.random.default_rng(seed)
    q, r = np.linalg.qr(rng.standard_normal((3, 3)))
    q = q * np.sign(np.diag(r))
    return [dict(s, x=tuple(float(v) for v in q @ np.array(s["x"]))) for s in find_molecule(c["molecule"])]


def _moved(solute, seed):
    """The next geometry of a scan: one site displaced by 0.05 A."""
    rng = np.random.default_rng(seed + 77)
    u, d = int(rng.integers(len(solute))), rng.standard_normal(3)
    d *= 0.05 / np.linalg.norm(d)
    out = [dict(s) for s in solute]
    out[u]["x"] = tuple(float(v) for v in np.array(out[u]["x"]) + d)
    return out


def _batch(c, seed):
    """Site counts and grids (from the case) and the solutes (from the seed)."""
    rng = random.Random(c["pick"])
    solutes, sets = [], []
    for i in range(c["count"]):
        n, grid = rng.randint(3, 40), rng.choice(BATCH_GRIDS)
        sol = synthetic_solute(n, radius=6.0, seed=seed * 64 + i)
        solutes.append(sol)
        sets.append(_settings(c, n=grid, half=22.0))
    return solutes, sets


def _fields(c, seed, device):
    """A mid-solve t (a few units around the solute, some noise) and a Newton direction, in the case's precision."""
    dtype = torch.float64 if c["precision"] == "fp64" else torch.float32
    g = torch.Generator(device=device).manual_seed(seed)
    solute = _solute(c, seed, c["half"])
    ax = [torch.arange(n, device=device, dtype=torch.float64) * (2 * c["half"] / n) - c["half"]
          for n in (c["nx"], c["ny"], c["nz"])]
    pos = torch.tensor([s["x"] for s in solute], device=device, dtype=torch.float64)
    e = [torch.exp(-0.25 * (a[None] - pos[:, d, None]) ** 2) for d, a in enumerate(ax)]
    shape = (3, c["nz"], c["ny"], c["nx"])
    T = torch.randn(shape, generator=g, device=device, dtype=dtype) * 0.05
    amp = torch.rand((3, len(solute)), generator=g, device=device, dtype=torch.float64) * 2.0 - 0.7
    for s in range(3):
        T[s] += torch.einsum("u,uz,uy,ux->zyx", amp[s], e[2], e[1], e[0]).clamp(-4.0, 4.0).to(dtype)
    dT = torch.randn(shape, generator=g, device=device, dtype=dtype) * 0.01
    return solute, T, dT


# --------------------------------------------------------------- the cases
def prepare(case, seed):
    c, kind = case, case["kind"]
    water = find_molecule(WATER)
    if kind == "solvent":
        # the solvent's own sites, one bond a little stretched by the seed
        rng = np.random.default_rng(seed)
        w = find_molecule("water")
        w = [dict(s, x=tuple(float(v) for v in np.array(s["x"]) * (1.0 + 0.01 * rng.random()))) for s in w]
        return {"case": c, "solvent": w, "settings": _settings(c)}
    chi = _chi(c["closure"])
    if kind in ("residual", "jacobian"):
        solute, T, dT = _fields(c, seed, "cuda")
        ctx = RismContext(solute, water, _settings(c, n=(c["nx"], c["ny"], c["nz"])), chi)
        return {"case": c, "ctx": ctx, "T": T, "dT": dT, "out": torch.empty_like(T)}
    if kind == "batch":
        solutes, sets = _batch(c, seed)
        return {"case": c, "solutes": solutes, "solvent": water, "settings": sets, "chi": chi}
    solute, s = _solute(c, seed, c["half"]), _settings(c)
    if kind == "solute":
        return {"case": c, "solute": solute, "solvent": water, "settings": s, "chi": chi}
    ctx = RismContext(solute, water, s, chi)
    state = {"case": c, "ctx": ctx, "T": ctx.zeros()}
    if kind in ("pes", "gradient"):
        state["T0"] = ctx.solve(ctx.zeros())[0]
    if kind == "pes":
        state["moved"] = _moved(solute, seed)
    return state


MU = ("free-energy", "mu-hnc", "mu-kh", "mu-gf", "partial-molar-volume-factor")


def run(state):
    kind = state["case"]["kind"]
    ctx = state.get("ctx")
    if kind == "residual":
        F, norms = ctx.iterate_t1(state["T"], out=state["out"])
        return {"F": F, "norms": list(norms)}
    if kind == "jacobian":
        return {"J": ctx.jacobian_t1(state["T"], state["dT"], out=state["out"])}
    if kind in ("solve", "pes"):
        T = state["T"]
        if kind == "solve":
            T.zero_()
        else:
            ctx.set_solute(state["moved"])
            T.copy_(state["T0"])
        ctx.solve(T)
        obs = ctx.observables(T, want_g=True)
        return {"T": T, "g": obs["GUV"], "mu": [obs[k] for k in MU]}
    if kind == "gradient":
        g = ctx.gradient(state["T0"])
        return {k: g[k] for k in ("charge", "sigma", "epsilon", "x")}
    if kind == "solute":
        keep = state["case"]["restart"]
        r = hnc3d_run_solute(state["solute"], state["solvent"], state["settings"], state["chi"], want_restart=keep)
        return {"g": r["GUV"], "T": r["RESTART"] if keep else None, "mu": [r[k] for k in MU]}
    if kind == "batch":
        rs = hnc3d_run_batch(state["solutes"], state["solvent"], state["settings"], state["chi"])
        return {"mu": [[r[k] for k in MU] for r in rs]}
    r = hnc3d_run_solvent(state["solvent"], state["settings"])
    return {"chi": r["susceptibility-3d"], "g": r["GVV"], "t": r["RESTART"],
            "mu": [r["free-energy"], r["compressibility"]]}


def work(case):
    """Bytes: each input field read and each result field written once.  Flops: the transforms (2.5 N log2 N per
    real field and direction), the closure and the k-space products of one evaluation, and the solute's field
    (about 40 per point, solvent site and solute site) where the call has to make it."""
    c, kind = case, case["kind"]

    def evaluation(n, m):
        return m * n * (5.0 * math.log2(n) + 30.0 + 4.0 * m)

    if kind in ("residual", "jacobian"):
        n, b = c["nx"] * c["ny"] * c["nz"], 8 if c["precision"] == "fp64" else 4
        return {"bytes": (3 if kind == "residual" else 4) * 3 * n * b, "flops": evaluation(n, 3)}
    if kind == "batch":
        rng = random.Random(c["pick"])
        total = {"bytes": 0, "flops": 0}
        for _ in range(c["count"]):
            sites, n = rng.randint(3, 40), rng.choice(BATCH_GRIDS) ** 3
            total["bytes"] += 3 * n * 8
            total["flops"] += evaluation(n, 3) + 40 * 3 * n * sites
        return total
    n = c["n"] ** 3
    if kind == "solvent":
        return {"bytes": 6 * n * 8 * 3, "flops": evaluation(n, 6)}
    sites = c["sites"] if "sites" in c else len(find_molecule(c["molecule"]))
    if kind == "gradient":
        return {"bytes": 2 * 3 * n * 8, "flops": 2 * evaluation(n, 3) + 60 * 3 * n * sites}
    fields = {"solve": 3, "pes": 3, "solute": 3 if c.get("restart") else 2}[kind]
    return {"bytes": fields * 3 * n * 8,
            "flops": evaluation(n, 3) + (40 * 3 * n * sites if kind in ("solute", "pes") else 0)}


# ------------------------------------------- the same equations in plain FP64
EPS0INV, G0, RCAP = 331.84164, 1.2, 0.2


def _cap(r, f, df):
    """f(r) with a parabola below RCAP (value and slope continuous)."""
    R = torch.tensor(RCAP, dtype=torch.float64, device=r.device)
    a, b = f(R), df(R) / (2 * R)
    inside = r < RCAP
    return torch.where(inside, a + b * (r * r - R * R), f(torch.where(inside, R, r)))


def _lj(r):
    return _cap(r, lambda x: 4 * (x ** -12 - x ** -6), lambda x: 4 * (6 * x ** -7 - 12 * x ** -13))


def _cs(r):
    k = 2 / math.sqrt(math.pi)
    return _cap(r, lambda x: torch.erfc(x) / x, lambda x: -(torch.erfc(x) + k * x * torch.exp(-x * x)) / (x * x))


def _cl(r):
    small = r < 0.02
    x, r2 = torch.where(small, torch.ones_like(r), r), r * r
    series = 2 / math.sqrt(math.pi) * (1 + r2 * (-1 / 3 + r2 * (1 / 10 - r2 / 42)))
    return torch.where(small, series, torch.erf(x) / x)


def _series(n, x):
    y, term = torch.zeros_like(x), torch.ones_like(x)
    for k in range(1, n + 1):
        term = term * x / k
        y = y + term
    return y


class Plain:
    """F(t) = (chi - 1) * c(t) - beta/eps0 tau - t on a grid, its Jacobian, solve and observables."""

    def __init__(self, n, half, closure, solute, chi):
        self.dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        self.n = tuple(n)
        h = [2.0 * half / k for k in n]
        self.h3, self.closure, self.beta, self.rho = h[0] * h[1] * h[2], closure, BASE["beta"], BASE["rho"]
        self.solvent = find_molecule(WATER)
        self.q = [s["charge"] for s in self.solvent]
        t = functools.partial(torch.tensor, device=self.dev, dtype=torch.float64)
        self.site = {k: t([s[k] for s in solute]) for k in ("charge", "sigma", "epsilon", "x")}
        self.ax = [torch.arange(k, device=self.dev, dtype=torch.float64) * hk - half for k, hk in zip(n, h)]
        dk = math.pi / half
        fr = [torch.arange(k, device=self.dev) for k in (n[0] // 2 + 1, n[1], n[2])]
        fr = [torch.where(i <= k // 2, i, i - k) for i, k in zip(fr, n)]
        self.sign = [1.0 - 2.0 * (i % 2).abs().double() for i in fr]
        self.k = [i.double() * dk for i in fr]
        kk = torch.sqrt((self.k[0][None, None, :] ** 2 + self.k[1][None, :, None] ** 2) + self.k[2][:, None, None] ** 2)
        nrad, dkr = chi.shape[-1], math.pi / BASE["rmax"]
        at = kk / torch.full_like(kk, dkr) - 0.5  # a true division: many |k| fall on the rule's ties
        i = torch.clamp((at + 0.5).long(), 0, nrad - 1)
        ip, im = torch.where(i < nrad - 2, i + 1, i), torch.where(i > 1, i - 1, i)
        frac = (at - i) / (ip - im)
        chi = t(chi)
        kr = (torch.arange(nrad, device=self.dev, dtype=torch.float64) + 0.5) * dkr
        lr = 4 * math.pi * torch.exp(-kr * kr / (4 * G0 * G0)) / (kr * kr)

        def radial(tab):
            return tab[i] + (tab[ip] - tab[im]) * frac

        self.K = {}
        for a in range(3):
            for b in range(a + 1):
                self.K[a, b] = self.K[b, a] = radial(chi[a, b] - (1.0 if a == b else 0.0))
        self.S = [radial(self.beta * EPS0INV * lr * sum(chi[j, a] * self.q[j] for j in range(3))) for a in range(3)]

    def potential(self, site=None):
        """The short-range field [3][...] and the long-range Coulomb field of the solute."""
        site = site or self.site
        v, uc = [0.0, 0.0, 0.0], 0.0
        for u in range(site["charge"].numel()):
            d2 = [(a - site["x"][u, d]) ** 2 for d, a in enumerate(self.ax)]
            r2 = d2[2][:, None, None] + d2[1][None, :, None] + d2[0][None, None, :]
            r = torch.sqrt(torch.clamp(r2, min=1e-24))
            cs = G0 * _cs(G0 * r)
            uc = uc + EPS0INV * site["charge"][u] * G0 * _cl(G0 * r)
            for s, a in enumerate(self.solvent):
                eps = torch.sqrt(a["epsilon"] * site["epsilon"][u])
                v[s] = v[s] + eps * _lj(r / (0.5 * (a["sigma"] + site["sigma"][u]))) + \
                    a["charge"] * EPS0INV * site["charge"][u] * cs
        return torch.stack(v), uc

    def form_factor(self, site=None):
        site = site or self.site
        f = 0.0
        for u in range(site["charge"].numel()):
            p = [torch.polar(torch.ones_like(k), -k * site["x"][u, d]) * s
                 for d, (k, s) in enumerate(zip(self.k, self.sign))]
            f = f + site["charge"][u] * p[2][:, None, None] * p[1][None, :, None] * p[0][None, None, :]
        return f / self.h3

    def closed(self, v, t):
        """c(t) and its slope."""
        x = t - self.beta * v
        if self.closure == "HNC":
            e = torch.expm1(x)
            return e - t, e
        n = 1 if self.closure == "KH" else int(self.closure[3:])
        e, pos = torch.expm1(torch.clamp(x, max=0.0)), torch.clamp(x, min=0.0)
        return torch.where(x < 0, e, _series(n, pos)) - t, torch.where(x < 0, e, _series(n - 1, pos))

    def back(self, f):
        """Complex to real; along x the imaginary parts of the first and last coefficient are not read."""
        f = torch.fft.ifftn(f, dim=(-3, -2))
        f = torch.cat((f[..., :1].real.to(f.dtype), f[..., 1:-1], f[..., -1:].real.to(f.dtype)), dim=-1)
        return torch.fft.irfft(f, n=self.n[0], dim=-1)

    def conv(self, c):
        f = torch.fft.rfftn(c, dim=(-3, -2, -1))
        return self.back(torch.stack([sum(self.K[a, b] * f[b] for b in range(3)) for a in range(3)]))

    def tau(self, site=None):
        f = self.form_factor(site)
        return self.back(torch.stack([s * f for s in self.S]))

    def F(self, v, tau, t):
        return self.conv(self.closed(v, t)[0]) - tau - t

    def J(self, d, u):
        return self.conv(d * u) - u

    def solve(self, v, tau, tol=1e-12):
        def residual(t):
            return self.F(v, tau, t)

        def jacobian(t):
            d = self.closed(v, t)[1]
            return lambda u: self.J(d, u)

        return _newton(residual, jacobian, torch.zeros_like(v), tol)

    def observables(self, v, uc, t, functional=None):
        """mu of a functional (default: the closure's), or all of MU."""
        c = self.closed(v, t)[0]
        h, x = c + t, t - self.beta * v
        cl = torch.stack([-self.beta * q * uc for q in self.q])
        base = -c - h * (c + cl) / 2
        f = self.rho * self.h3 / self.beta
        n = 2 if self.closure == "KH" else (0 if self.closure == "HNC" else int(self.closure[3:]) + 1)

        def mu(name):
            if name == "HNC":
                return f * (base + h * h / 2).sum()
            if name == "GF":
                return f * base.sum()
            extra = torch.zeros_like(h) if name == "KH" else h * h / 2 - x ** n / math.factorial(n)
            return f * (base + torch.where(h < 0, h * h / 2, extra)).sum()

        if functional:
            return mu(functional)
        return [float(mu(self.closure)), float(mu("HNC")), float(mu("KH")), float(mu("GF")),
                1.0 - float(self.rho * self.h3 * c.sum())], h + 1.0


def _gmres(A, b, rtol, restart=30, most=3000):
    x, r, its = torch.zeros_like(b), b, 0
    stop = rtol * float(b.norm())
    while its < most and float(r.norm()) > stop:
        beta = r.norm()
        V, H = [r / beta], torch.zeros(restart + 1, restart, dtype=torch.float64)
        for j in range(restart):
            w = A(V[j])
            its += 1
            for i in range(j + 1):
                H[i, j] = (V[i] * w).sum()
                w = w - H[i, j].item() * V[i]
            H[j + 1, j] = w.norm()
            e = torch.zeros(j + 2, dtype=torch.float64)
            e[0] = beta
            y = torch.linalg.lstsq(H[:j + 2, :j + 1], e[:, None]).solution[:, 0]
            left = float((H[:j + 2, :j + 1] @ y - e).norm())
            V.append(w / w.norm())
            if left <= stop or its >= most:
                break
        for i, yi in enumerate(y.tolist()):
            x = x + yi * V[i]
        r = b - A(x)
    return x


def _newton(F, jacobian, t, tol):
    r = F(t)
    for _ in range(60):
        if float(r.abs().max()) < tol:
            break
        dt = _gmres(jacobian(t), r, 1e-3 if float(r.abs().max()) > 1e-9 else 1e-2)
        lam = 1.0
        while True:
            trial = t - lam * dt
            rt = F(trial)
            if float(rt.norm()) < (1 - 1e-4 * lam) * float(r.norm()) or lam < 1e-3:
                break
            lam *= 0.5
        if lam < 1e-3:
            break  # the rounding floor
        t, r = trial, rt
    return t


def exact(case, seed):
    c, kind = case, case["kind"]
    with torch.no_grad():
        if kind == "solvent":
            return None  # a solver of its own (a matrix equation per k), not restated here
        if kind in ("residual", "jacobian"):
            dev = "cuda" if torch.cuda.is_available() else "cpu"
            solute, T, dT = _fields(c, seed, dev)
            P = Plain((c["nx"], c["ny"], c["nz"]), c["half"], c["closure"], solute, _chi(c["closure"]))
            v, _ = P.potential()
            if kind == "jacobian":
                return {"J": P.J(P.closed(v, T.double())[1], dT.double())}
            F = P.F(v, P.tau(), T.double())
            return {"F": F, "norms": [float(F.abs().max()), float(F.norm())]}
        if kind == "batch":
            mus = []
            for solute, s in zip(*_batch(c, seed)):
                P = Plain((s["N"],) * 3, s["L"], c["closure"], solute, _chi(c["closure"]))
                v, uc = P.potential()
                mus.append(P.observables(v, uc, P.solve(v, P.tau()))[0])
            return {"mu": mus}
        solute = _solute(c, seed, c["half"])
        if kind == "pes":
            solute = _moved(solute, seed)
        P = Plain((c["n"],) * 3, c["half"], c["closure"], solute, _chi(c["closure"]))
        v, uc = P.potential()
        t = P.solve(v, P.tau())
        if kind != "gradient":
            mu, g = P.observables(v, uc, t)
            return {"T": t, "g": g, "mu": mu} if kind != "solute" or c["restart"] else {"g": g, "T": None, "mu": mu}
    # dmu/dp = dmu/dp|_t - lambda . dF/dp|_t with J^T lambda = dmu/dt
    t.requires_grad_(True)
    b = torch.autograd.grad(P.observables(v, uc, t, c["closure"]), t)[0]
    t.requires_grad_(False)
    d = P.closed(v, t)[1]
    lam = d * _gmres(lambda u: P.J(d, u), P.conv(b), 1e-11) - b
    out = {k: torch.zeros_like(a) for k, a in P.site.items()}
    for u in range(len(solute)):  # one site at a time: the fields are sums over sites
        one = {k: a[u:u + 1].clone().requires_grad_(True) for k, a in P.site.items()}
        v1, uc1 = P.potential(one)
        fixed = {k: a[u:u + 1] for k, a in P.site.items()}
        with torch.no_grad():
            v0, uc0 = P.potential(fixed)
        vu, ucu = v - v0 + v1, uc - uc0 + uc1
        total = P.observables(vu, ucu, t, c["closure"]) - \
            (lam * (P.conv(P.closed(vu, t)[0]) - P.tau(one))).sum()
        for k, g in zip(out, torch.autograd.grad(total, [one[k] for k in out])):
            out[k][u] = g[0]
    return {k: out[k] for k in ("charge", "sigma", "epsilon", "x")}
