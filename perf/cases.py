"""Timed cases of the framework: what a laminarSMOKE run asks of it, through the Python binding of the C ABI.

Two families of calls.

``step``: the reaction step of one CFD time step (``ReactionStep.step_device`` / ``step_cv_device`` /
``step``, lsg_reaction_step*).  Every cell's reactor is integrated over dt; the fields are stepped on a
copy, as a solver with the compact Strang scheme does, so that a pass can be repeated.  From a handful of
cells (one rank's patch, an ignition delay study) to a million (a whole mesh on one GPU), device fields and
host fields (the OpenFOAM-facing call), constant pressure and constant volume, one dt for all or one per
cell (local time stepping), the packaged H2/CO, H2 and CH4 mechanisms and mechanisms of 121 to 501
components, FP64 (the default) and mixed precision (the documented setting).

``properties`` and ``steady``: what surrounds the step.  The property update after every step
(lsg_properties_device) and the steady solvers' linearised sources (lsg_steady_sources_sparse_device, the
default ``sparseJacobian true``).
"""
import functools
import os

import numpy as np
import torch

from laminarsmoke_b200 import cells, lsg, mech
from laminarsmoke_b200.mech import blob

R_GAS = 8314.4621
POOL = os.path.join("tests", "golden", "h2co_hot_pool.npz")   # near-equilibrium H2/CO mixtures

# Mean work of one cell's integration by the kind of state and mechanism: BDF steps, RHS calls, RHS calls of the
# finite-difference Jacobians, factorisations, linear solves (the solver's own counters).
COUNTS = {
    ("mixing", "h2co"): (205, 273, 73, 29, 271), ("uneven", "h2co"): (74, 87, 30, 17, 85),
    ("coflow", "h2co"): (143, 169, 51, 25, 167), ("mixing", "ch4"): (353, 421, 193, 49, 419),
    ("mixing", "h2"): (150, 200, 40, 25, 200), ("mixing", "padded"): (188, 267, 260, 27, 265),
    ("coflow", "syn120p"): (2712, 3710, 1176, 241, 3707),
}


def listed():
    def step(name, mechanism, n, states, **kw):
        c = {"name": name, "path": "step", "mech": mechanism, "cells": n, "states": states, "precision": "mixed",
             "fields": "device", "reactor": "p", "p": 101325.0, "dt": 1e-5, "lts": False}
        c.update(kw)
        return c

    return [
        # a whole mesh of uneven stiffness on one GPU: cold, igniting and near-equilibrium cells
        step("step_h2co_uneven_1m", "h2co", 1 << 20, "uneven"),
        # an ordinary laminar coflow mesh, 200 x 400 cells
        step("step_h2co_coflow_80k", "h2co", 80000, "coflow"),
        # one MPI rank's host fields with local time stepping, an odd number of cells
        step("step_h2co_host_lts_20k", "h2co", 20011, "mixing", fields="host", lts=True),
        # the smallest calls: latency and launches count
        step("step_h2co_67", "h2co", 67, "mixing"),
        # the default options (all FP64) on the CPU-runnable case of 4,096 mixtures
        step("step_h2co_fp64_4096", "h2co", 4096, "mixing", precision="fp64"),
        # a hydrocarbon skeletal mechanism (25 components), constant volume, odd size
        step("step_ch4_cv_4097", "ch4", 4097, "mixing", reactor="v", p=202650.0),
        # large mechanisms: 121 components, sparse chemistry, all FP64 ...
        step("step_121_fp64_592", "h2co+106", 592, "mixing", precision="fp64"),
        # ... 121 components, 800 reactions, a flame's cells ...
        step("step_syn120_fp64_96", "syn120p", 96, "coflow", precision="fp64", dt=1e-7),
        # ... and 501 components in mixed precision (tensor-core inverse)
        step("step_501_mixed_148", "h2co+486", 148, "mixing"),
        # the property update of a whole mesh, every field
        {"name": "properties_h2co_1m", "path": "properties", "mech": "h2co", "cells": 1 << 20, "soret": True,
         "lewis": False},
        # a ragged patch, CH4
        {"name": "properties_ch4_39999", "path": "properties", "mech": "ch4", "cells": 39999, "soret": False,
         "lewis": False},
        # the steady solvers' sources
        {"name": "steady_h2co_80k", "path": "steady", "mech": "h2co", "cells": 80000},
    ]


def _size(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(("step", "step", "step", "large", "properties", "steady"))
    if kind == "properties":
        return {"path": "properties", "mech": rng.choice(("h2co", "ch4", "h2")), "cells": _size(rng, 1, 1 << 20),
                "soret": rng.random() < 0.5, "lewis": rng.random() < 0.25}
    if kind == "steady":
        return {"path": "steady", "mech": rng.choice(("h2co", "ch4", "h2")), "cells": _size(rng, 1, 200000)}
    c = {"path": "step", "precision": rng.choice(("mixed", "fp64")), "fields": rng.choice(("device", "host")),
         "reactor": rng.choice(("p", "p", "v")), "p": round(101325.0 * rng.uniform(0.8, 5.0), 1),
         "dt": float("%.3g" % (10.0 ** rng.uniform(-6.0, -5.0))), "lts": rng.random() < 0.3}
    if kind == "large":
        k = _size(rng, 31, 486)
        c.update(mech="h2co+%d" % k, cells=_size(rng, 1, 600 if k < 114 else 148), states="mixing", dt=1e-5, reactor="p")
        return c
    m = rng.choice(("h2co", "h2co", "h2", "ch4"))
    most = {"h2co": 100000, "h2": 100000, "ch4": 16000}[m] // (4 if c["precision"] == "fp64" else 1)
    c.update(mech=m, cells=_size(rng, 1, most), states="mixing")
    if m == "h2co" and rng.random() < 0.4:
        c.update(states="uneven", cells=_size(rng, 1, 4 * most))
    return c


@functools.lru_cache(maxsize=None)
def _mechanism(name):
    data, species = mech.load(name)
    return data, species, blob.unpack(data)[0]


def _states(case, species, mw, seed):
    """Cell-major Y [cells, species] and T [cells]."""
    n, name = case["cells"], case["mech"]
    kind = case.get("states", "mixing")
    if kind == "uneven":
        return cells.h2co_uneven(species, mw, n, cells.pool_from_file(POOL), seed=seed)
    if kind == "coflow":
        Y, T = cells.coflow_fields(species, mw, seed=seed, fuel={"H2": 0.5, "CO": 0.5} if name == "h2co" else None)
        if n < T.size:   # an evenly strided part of the mesh, starting anywhere
            start = np.random.default_rng(seed).integers(0, T.size // n)
            pick = start + np.arange(n) * (T.size // n)
            Y, T = Y[pick], T[pick]
        return Y, T
    if name.startswith("h2co"):
        return cells.h2co_mixing(species, mw, n, seed=seed)
    if name == "ch4":
        return cells.synthetic_mixing(species, mw, n, seed, (800.0, 2400.0))
    rng = np.random.default_rng(seed)   # H2 / air with radicals
    yf, ya = cells.fuel_air_mass(species, mw, {"H2": 1.0}, {"O2": 0.21, "N2": 0.79})
    Z = rng.uniform(0.0, 0.3, n)[:, None]
    Y = Z * yf + (1.0 - Z) * ya
    minor = [i for i, s in enumerate(species) if s not in ("H2", "O2", "N2")]
    Y[:, minor] = 10.0 ** rng.uniform(-10.0, -4.0, (n, len(minor)))
    return Y / Y.sum(axis=1, keepdims=True), rng.uniform(900.0, 2200.0, n)


def _inputs(case, seed):
    """Host arrays of a case, from the seed alone: Y [species, cells], T, p, dt or None, rho or None, Lewis or None."""
    _, species, A = _mechanism(case["mech"])
    mw = A["mw"]
    Y, T = _states(case, species, mw, seed)
    n = T.size
    rng = np.random.default_rng([seed, 17])
    p = np.full(n, case["p"]) if "p" in case else 101325.0 * rng.uniform(0.5, 5.0, n)
    dt = case["dt"] * 10.0 ** rng.uniform(-1.0, 0.0, n) if case.get("lts") else None
    rho = p / (R_GAS * T * (Y / mw).sum(axis=1)) if case.get("reactor") == "v" else None
    lewis = 10.0 ** rng.uniform(-0.7, 0.3, len(species)) if case.get("lewis") else None
    return np.ascontiguousarray(Y.T), T, p, dt, rho, lewis


def prepare(case, seed):
    Y, T, p, dt, rho, lewis = _inputs(case, seed)
    data = _mechanism(case["mech"])[0]
    nc, n = Y.shape
    mixed = case.get("precision") == "mixed"
    ctx = lsg.ReactionStep(lsg.Mechanism(data),
                           precision=lsg.LSG_PRECISION_MIXED if mixed else lsg.LSG_PRECISION_FP64)
    s = {"case": case, "ctx": ctx}
    if case["path"] == "step" and case["fields"] == "host":
        s.update(Y0=Y, T0=T, Y=np.empty_like(Y), T=np.empty_like(T), dt=case["dt"] if dt is None else dt, rho=rho)
        return s

    def dev(x):
        return None if x is None else torch.from_numpy(np.ascontiguousarray(x)).to("cuda")

    s.update(Y0=dev(Y), T0=dev(T))
    if case["path"] == "step":
        s.update(Y=torch.empty_like(s["Y0"]), T=torch.empty_like(s["T0"]),
                 Q=torch.zeros(n, dtype=torch.float64, device="cuda"),
                 status=torch.zeros(n, dtype=torch.int32, device="cuda"),
                 dt=case["dt"] if dt is None else dev(dt), rho=dev(rho))
    else:
        s.update(p=dev(p), lewis=dev(lewis))
        if case["path"] == "steady":
            s.update(imp=torch.zeros(nc + 1, n, dtype=torch.float64, device="cuda"),
                     exp=torch.zeros(nc + 1, n, dtype=torch.float64, device="cuda"))
    return s


def run(state):
    s, c = state, state["case"]
    ctx = s["ctx"]
    if c["path"] == "properties":
        return ctx.properties_device(s["Y0"], s["T0"], s["p"], soret=c["soret"], lewis=s["lewis"])
    if c["path"] == "steady":
        ctx.steady_sources_sparse_device(s["Y0"], s["T0"], s["imp"], s["exp"], p=s["p"])
        return {"implicit": s["imp"], "explicit": s["exp"]}
    if c["fields"] == "host":
        np.copyto(s["Y"], s["Y0"])
        np.copyto(s["T"], s["T0"])
        if c["reactor"] == "v":
            Q, status, _ = ctx.step_cv(s["Y"], s["T"], s["rho"], s["dt"])
        else:
            Q, status, _ = ctx.step(s["Y"], s["T"], s["dt"], p=c["p"])
        return {"Y": s["Y"], "T": s["T"], "Q": Q, "status": status}
    s["Y"].copy_(s["Y0"])
    s["T"].copy_(s["T0"])
    if c["reactor"] == "v":
        ctx.step_cv_device(s["Y"], s["T"], s["rho"], s["dt"], Q=s["Q"], status=s["status"])
    else:
        ctx.step_device(s["Y"], s["T"], s["dt"], p=c["p"], Q=s["Q"], status=s["status"])
    return {"Y": s["Y"], "T": s["T"], "Q": s["Q"], "status": s["status"]}


def _rhs_flops(A):
    """FP64 operations of one right-hand side, 20 for each exponential or logarithm."""
    nc, nr = (int(v) for v in A["dims"])
    nnz = len(A["reac_species"]) + len(A["prod_species"])
    n_exp = nr + len(A["rev_thermo"]) + 5 * len(A["fo_rxn"]) + 2
    return 40 * nc + 12 * nr + 4 * nnz + 20 * n_exp


def work(case):
    A = _mechanism(case["mech"])[2]
    nc, n = int(A["dims"][0]), case["cells"]
    ne, rhs = nc + 1, _rhs_flops(A)
    if case["path"] == "properties":
        nt = len(A["tr_iteta"]) if case["soret"] else 0
        pairs = nc * (nc - 1) // 2
        per = nc * 100 + pairs * (14 + (0 if case["lewis"] else 32)) + nt * nc * 9
        return {"bytes": 8 * n * (nc + 2 + 3 * nc + 8 + nt), "flops": per * n}
    if case["path"] == "steady":
        return {"bytes": 8 * n * (nc + 2 + 2 * ne), "flops": n * (3 * rhs + 20 * len(A["reac_species"]))}
    kind = "padded" if "+" in case["mech"] else case["mech"]
    steps, calls, jac, fact, solve = COUNTS[(case["states"], kind)]
    per = ((calls + jac) * rhs + fact * (2.0 / 3.0 * ne ** 3 + ne * ne) + solve * 2.0 * ne * ne + steps * 30.0 * ne)
    return {"bytes": n * (8 * (2 * ne + 1) + 4 + 8 * bool(case["lts"])), "flops": float(per * n)}


def _at(A, key, width, T):
    """NASA coefficients [species, width, 1 or cells] of the range each cell's T lies in."""
    nc = int(A["dims"][0])
    hi, lo = (torch.from_numpy(A[key + e].reshape(nc, width, 1)).to(T) for e in ("_ht", "_lt"))
    return torch.where(T > torch.from_numpy(A["t_mid"]).to(T)[:, None, None], hi, lo)


def _nasa(A, T):
    """cp/R, h/RT and s/R of every species at T: [species, cells] each."""
    lT = torch.log(T)
    a, h, s = _at(A, "cp", 5, T), _at(A, "dh", 6, T), _at(A, "ds", 6, T)
    cp = a[:, 0] + T * a[:, 1] + T ** 2 * a[:, 2] + T ** 3 * a[:, 3] + T ** 4 * a[:, 4]
    hh = h[:, 0] + T * h[:, 1] + T ** 2 * h[:, 2] + T ** 3 * h[:, 3] + T ** 4 * h[:, 4] + h[:, 5] / T
    ss = s[:, 0] * lT + T * s[:, 1] + T ** 2 * s[:, 2] + T ** 3 * s[:, 3] + T ** 4 * s[:, 4] + s[:, 5]
    return cp, hh, ss


def _exact_properties(case, A, Y, T, p, lewis):
    col = lambda k: torch.from_numpy(A[k]).to(T)[:, None]
    mw = col("mw")
    nc = mw.shape[0]
    W = 1.0 / (Y / mw).sum(0)
    x = W * Y / mw
    cp, h, _ = _nasa(A, T)
    powers = torch.stack([torch.log(T) ** k for k in range(4)])
    fit = lambda k: torch.exp(torch.from_numpy(A[k].reshape(-1, 4)).to(T) @ powers)
    eta, lam = fit("tr_eta"), fit("tr_lambda")
    mu = torch.zeros_like(T)
    for k in range(nc):
        d = torch.sqrt(eta[k] / eta) * (mw / mw[k]) ** 0.25
        mu += x[k] * eta[k] / (x * (1.0 + d) ** 2 / torch.sqrt(8.0 * (1.0 + mw[k] / mw))).sum(0)
    cpm = R_GAS * (cp * x).sum(0)
    lm = 0.5 * ((x * lam).sum(0) + 1.0 / (x / lam).sum(0))
    psi = W / (R_GAS * T)
    out = {"X": x, "cTot": p / (R_GAS * T), "psi": psi, "mu": mu, "lambda": lm, "cp": cpm / W, "cv": (cpm - R_GAS) / W,
           "h": R_GAS * T * (h * x).sum(0) / W, "MWmix": W, "cp_species": cp * R_GAS / mw}
    if case["lewis"]:
        out["Dmix"] = lm / (p * psi * out["cp"]) / torch.from_numpy(lewis).to(T)[:, None]
    else:
        xs = (x + 1e-14) / (1.0 + 1e-14 * nc)
        Ws = (xs * mw).sum(0)
        pair = torch.zeros(nc, nc, dtype=torch.long)
        j, k = torch.triu_indices(nc, nc, 1)
        pair[j, k] = pair[k, j] = torch.arange(j.numel())
        gam = torch.from_numpy(A["tr_gamma"].reshape(-1, 4)).to(T)
        D = torch.empty_like(x)
        for k in range(nc):
            o = [j for j in range(nc) if j != k]
            inv = (p / 1e5) / torch.exp(gam[pair[k, o].to(T.device)] @ powers)
            D[k] = (Ws - xs[k] * mw[k]) / (Ws * (xs[o] * inv).sum(0))
        out["Dmix"] = D
    if case["soret"]:
        it = A["tr_iteta"]
        th = torch.from_numpy(A["tr_teta"].reshape(len(it), nc, 4)).to(T) @ torch.stack([T ** k for k in range(4)])
        it = torch.from_numpy(it).long().to(T.device)
        out["Dsoret"] = out["Dmix"][it] * (th * x[it][:, None] * x[None]).sum(1) * mw[it] / W
    return out


def _rows(A, ptr, sp, val, nr, nc, like):
    """Dense [rows, species] of a row-pointer list."""
    M = np.zeros((nr, nc))
    for r in range(nr):
        for q in range(A[ptr][r], A[ptr][r + 1]):
            M[r, A[sp][q]] += A[val][q]
    return torch.from_numpy(M).to(like)


def _fall_off(A, kArr, M, T):
    """k_inf (Pr / (1 + Pr)) F / k0 of every fall-off reaction: [slots, cells]."""
    c = {k: torch.from_numpy(A["fo_" + k]).to(T)[:, None] for k in ("lnA", "beta", "e_over_r", "a", "b", "c", "d", "e")}
    kInf = torch.exp(c["lnA"] + c["beta"] * torch.log(T) - c["e_over_r"] / T)
    Pr = kArr * M / kInf
    lPr = torch.log10(Pr)
    cent = (1.0 - c["a"]) * torch.exp(-T / c["b"]) + c["a"] * torch.exp(-T / c["c"])
    cent = torch.where(c["d"] != 0.0, cent + torch.exp(-c["d"] / T), cent)
    lF = torch.log10(cent)
    s = lPr - 0.4 - 0.67 * lF
    q = s / (0.75 - 1.27 * lF - 0.14 * s)
    troe = 10.0 ** (lF / (1.0 + q * q))
    sri = (c["a"] * torch.exp(-c["b"] / T) + torch.exp(-T / c["c"])) ** (1.0 / (1.0 + lPr ** 2)) * c["d"] * T ** c["e"]
    kind = torch.from_numpy(A["fo_type"]).to(T)[:, None]
    F = torch.where(kind == 1, troe, torch.where(kind == 2, sri, torch.ones_like(T)))
    return kInf * (Pr / (1.0 + Pr)) * F / kArr


class _Kinetics:
    """Rates of progress of a mechanism of elementary, third-body and fall-off reactions."""

    def __init__(self, A, T):
        nc, nr = (int(v) for v in A["dims"])
        self.A, self.nc, self.nr = A, nc, nr
        self.nr_ = _rows(A, "reac_ptr", "reac_species", "reac_nu", nr, nc, T)
        self.np_ = _rows(A, "prod_ptr", "prod_species", "prod_nu", nr, nc, T)
        self.tb, self.fo = (torch.from_numpy(A[k]).long().to(T.device) for k in ("tb_rxn", "fo_rxn"))
        self.te = 1.0 + _rows(A, "tb_ptr", "tb_species", "tb_eff_m1", len(A["tb_rxn"]), nc, T)
        self.fe = 1.0 + _rows(A, "fo_ptr", "fo_species", "fo_eff_m1", len(A["fo_rxn"]), nc, T)
        self.rev = torch.zeros(nr, 1, dtype=torch.float64, device=T.device)
        self.rev[torch.from_numpy(A["rev_thermo"]).long().to(T.device)] = 1.0

    def rates(self, c, cTot, T):
        """Forward and reverse rates [reactions, cells]; the fall-off correction and Arrhenius constants."""
        A = self.A
        col = lambda k: torch.from_numpy(A[k]).to(T)[:, None]
        _, h, s = _nasa(A, T)
        kArr = col("a_sign") * torch.exp(col("lnA") + col("beta") * torch.log(T) - col("e_over_r") / T)
        k = kArr.clone()
        Mt = cTot + (self.te - 1.0) @ c
        k[self.tb] *= Mt
        G = _fall_off(A, kArr[self.fo], cTot + (self.fe - 1.0) @ c, T)
        k[self.fo] *= G
        dn = self.np_ - self.nr_
        uK = self.rev * torch.exp(dn @ (h - s) - col("delta_nu") * torch.log(101325.0 / (R_GAS * T)))
        f, r = torch.ones_like(k), torch.ones_like(k)
        for i in range(self.nc):
            for v in (1.0, 2.0, 3.0):
                f[self.nr_[:, i] == v] *= c[i] ** v
                r[self.np_[:, i] == v] *= c[i] ** v
        return k * f, k * r * uK, h, Mt, G, kArr

    def sources(self, om, T, p):
        """R_i MW_i and the heat release of the mixture."""
        mw = torch.from_numpy(self.A["mw"]).to(T)[:, None]
        W = 1.0 / (om / mw).sum(0)
        cTot = p / (R_GAS * T)
        c = cTot * W * om / mw
        f, r, h, _, _, _ = self.rates(c, c.sum(0), T)
        R = (self.np_ - self.nr_).T @ (f - r)
        return R * mw, -R_GAS * T * (R * h).sum(0)


def _exact_steady(A, Y, T, p):
    K = _Kinetics(A, T)
    mw = torch.from_numpy(A["mw"]).to(T)[:, None]
    S, q = K.sources(Y.clamp_min(0.0), T, p)
    S = torch.cat([S, q[None]])
    dT = torch.minimum(torch.maximum(2.220446049250313e-16 ** 0.5 * T, 1e-12 + 1e-7 * T), 1e-3 + 1e-3 * T)
    JT = (K.sources(Y.clamp_min(0.0), T + dT, p)[1] - q) / dT
    om = Y.clamp_min(1e-13)
    cTot = p / (R_GAS * T)
    rho = cTot / (om / mw).sum(0)
    c = om * rho / mw
    f, r, _, Mt, G, kArr = K.rates(c, cTot, T)
    net = f - r
    dn = K.np_ - K.nr_
    J = torch.empty_like(Y)
    M = cTot + (K.fe - 1.0) @ c
    for k in range(K.nc):
        d = (K.nr_[:, k, None] * f - K.np_[:, k, None] * r) / om[k]
        d[K.tb] += net[K.tb] * c[k] / om[k] * (K.te[:, k, None] - 1.0) / Mt
        plus = M + (K.fe[:, k, None] - 1.0) * (1e-4 * rho / mw[k])
        dG = (_fall_off(A, kArr[K.fo], plus, T) - G) / 1e-4
        has = (K.fe[:, k, None] != 1.0).to(T)
        d[K.fo] += has * net[K.fo] * dG / G
        J[k] = (dn[:, k, None] * d).sum(0) * mw[k]
    J = torch.cat([J, JT[None]])
    return {"implicit": J, "explicit": S - J * torch.cat([Y, T[None]])}


def exact(case, seed):
    # An integration of every cell's stiff system to 64-bit accuracy takes far more than 20 seconds in torch or numpy.
    if case["path"] == "step":
        return None
    Y, T, p, _, _, lewis = _inputs(case, seed)
    A = _mechanism(case["mech"])[2]
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    parts = []
    for at in range(0, T.size, 1 << 17):
        y, t, q = (torch.from_numpy(np.ascontiguousarray(v[..., at:at + (1 << 17)])).to(dev) for v in (Y, T, p))
        parts.append(_exact_properties(case, A, y, t, q, lewis) if case["path"] == "properties" else _exact_steady(A, y, t, q))
    return {k: torch.cat([o[k] for o in parts], dim=-1) for k in parts[0]}
