"""Performance cases of the muon DCS framework, each one pass through its public entry points.

Energies follow the law of the repository's own workload and benchmark: K log-uniform in [1e-3, 1e6] GeV and
nu = q / K log-uniform in [1e-7, 1].  Elements are those of the batched workload (Z = 1 .. 82), particles the muon and
the tau.  `exact` restates the formulas in plain float64 torch.
"""
import math

import numpy as np
import torch

from noa_gb300 import dcs
from noa_gb300.batched import BatchPlan
from noa_gb300.elements import BATCH_Z, ELEMENTS, MUON_MASS, TAU_MASS
from noa_gb300.surrogate import GRID, Surrogate, init_params

PROCESSES = ("bremsstrahlung", "pair_production", "photonuclear", "ionisation")
MASS = {"muon": MUON_MASS, "tau": TAU_MASS}
XLOW = 0.05
# Floating operations of one evaluation averaged over the workload's law, early exits included, with a logarithm,
# exponential or power counted as 20 (the benchmark's convention).
FLOPS = {"bremsstrahlung": 156.3, "pair_production": 1192.5, "photonuclear": 949.7, "ionisation": 58.0}


def listed():
    return [
        # a stepping code or a notebook that asks for one short list of energies: all latency and launches
        {"name": "lookup", "kind": "dcs", "precision": "fp64", "n": 61, "Z": 11, "particle": "muon", "allocate": True},
        # a table of cross-sections of one element, ragged, heavy and for the tau: fills the chip once or twice
        {"name": "table", "kind": "dcs", "precision": "fp64", "n": 60_013, "Z": 82, "particle": "tau",
         "allocate": True},
        # the headline: bulk evaluation of the four processes in standard rock into kept buffers
        {"name": "bulk", "kind": "dcs", "precision": "fp64", "n": 30_000_000, "Z": 11, "particle": "muon",
         "allocate": False},
        # the FP32-compensated form at an ordinary size, hydrogen (its own branches in every process)
        {"name": "fp32c_table", "kind": "dcs", "precision": "fp32c", "n": 250_007, "Z": 1, "particle": "muon",
         "allocate": True},
        # and in bulk
        {"name": "fp32c_bulk", "kind": "dcs", "precision": "fp32c", "n": 20_000_000, "Z": 26, "particle": "muon",
         "allocate": False},
        # a composite material: ten elements with uneven counts in one replayed launch per process
        {"name": "material", "kind": "batched", "precision": "fp64", "n": 1_000_000, "elements": 10, "graph": True},
        # a caller with its energies in (page-locked) host memory, the end-to-end path
        {"name": "host", "kind": "host", "precision": "fp64", "n": 2_000_003, "Z": 11, "particle": "muon",
         "pinned": True},
        # the physics tables of one element: energy-loss integrals and soft scattering on a kinetic energy grid
        {"name": "losses_grid", "kind": "losses", "n": 146, "Z": 11, "min_points": 180},
        # the same for a fine grid
        {"name": "losses_fine", "kind": "losses", "n": 20_011, "Z": 26, "min_points": 180},
        # elastic scattering of a ten-element material on a kinetic energy grid, up to the hard-scattering cut-off
        {"name": "elastic", "kind": "elastic", "n": 5_003, "elements": 10},
        # the learned surrogate answering queries: network in the trusted cells, FP32C elsewhere
        {"name": "surrogate", "kind": "surrogate", "process": "photonuclear", "n": 5_000_000, "elements": 10},
        # and its training, forward and backward with Adam
        {"name": "training", "kind": "training", "process": "pair_production", "batch": 8192, "steps": 12},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["dcs", "dcs", "dcs", "batched", "host", "losses", "losses", "elastic", "surrogate",
                       "training"])
    precision = rng.choice(["fp64", "fp32c"])
    z = rng.choice(BATCH_Z)
    particle = rng.choice(["muon", "muon", "tau"])
    if kind == "dcs":
        return {"kind": kind, "precision": precision, "n": _log_int(rng, 1, 2e7), "Z": z, "particle": particle,
                "allocate": rng.random() < 0.5}
    if kind == "batched":
        return {"kind": kind, "precision": precision, "n": _log_int(rng, 1e3, 1e7), "elements": rng.randint(2, 10),
                "graph": rng.random() < 0.5}
    if kind == "host":
        return {"kind": kind, "precision": precision, "n": _log_int(rng, 1, 4e6), "Z": z, "particle": particle,
                "pinned": rng.random() < 0.5}
    if kind == "losses":
        return {"kind": kind, "n": _log_int(rng, 8, 2e4), "Z": z, "min_points": rng.choice([60, 100, 180, 300])}
    if kind == "elastic":
        return {"kind": kind, "n": _log_int(rng, 8, 5e4), "elements": rng.randint(1, 10)}
    if kind == "surrogate":
        return {"kind": kind, "process": rng.choice(["pair_production", "photonuclear"]),
                "n": _log_int(rng, 1e4, 1e7), "elements": rng.randint(2, 10)}
    return {"kind": kind, "process": rng.choice(["pair_production", "photonuclear"]),
            "batch": rng.choice([2048, 4096, 8192]), "steps": rng.randint(4, 24)}


# ---------------------------------------------------------------- inputs
def _rand(seed, n):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.rand(n, generator=g, dtype=torch.float64, device="cuda")


def _pairs(seed, n):
    K = 10.0 ** (9.0 * _rand(2 * seed, n) - 3.0)
    return K, K * 10.0 ** (7.0 * _rand(2 * seed + 1, n) - 7.0)


def _grid(seed, n):
    """A rising grid of kinetic energies."""
    return torch.sort(10.0 ** (9.0 * _rand(2 * seed, n) - 3.0)).values


def _counts(n, elements):
    """Uneven counts that add up to n: log-uniform shares over a factor of 3000, as in the batched workload."""
    w = [3000.0 ** (((7 * i + 3) % 10) / 9.0) for i in range(elements)]
    c = [int(n * x / sum(w)) for x in w]
    c[w.index(max(w))] += n - sum(c)
    return c


def _elements(case):
    return [ELEMENTS[z] for z in BATCH_Z[:case["elements"]]]


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind in ("dcs", "host"):
        s["element"], s["mass"] = ELEMENTS[case["Z"]], MASS[case["particle"]]
        s["K"], s["q"] = _pairs(seed, case["n"])
        if kind == "host":
            s["K"], s["q"] = s["K"].cpu(), s["q"].cpu()
            s["out"] = [torch.zeros_like(s["K"]) for _ in PROCESSES]
            if case["pinned"]:
                s["K"], s["q"] = s["K"].pin_memory(), s["q"].pin_memory()
                s["out"] = [o.pin_memory() for o in s["out"]]
        elif not case["allocate"]:
            s["out"] = [torch.zeros_like(s["K"]) for _ in PROCESSES]
    elif kind == "batched":
        s["K"], s["q"] = _pairs(seed, case["n"])
        s["out"] = [torch.zeros_like(s["K"]) for _ in PROCESSES]
        s["plans"] = [BatchPlan(p, _elements(case), _counts(case["n"], case["elements"]), MUON_MASS,
                                case["precision"]) for p in PROCESSES]
    elif kind == "losses":
        s["element"], s["K"] = ELEMENTS[case["Z"]], _grid(seed, case["n"])
        s["out"] = [torch.zeros_like(s["K"]) for _ in range(9)]
    elif kind == "elastic":
        n, nel = case["n"], case["elements"]
        s["elements"], s["K"] = _elements(case), _grid(seed, n)
        for name, shape in (("fCM", (nel, n, 2)), ("screening", (nel, n, 9)), ("fspin", (nel, n)),
                            ("invlambda", (nel, n)), ("G", (nel, n, 2)), ("mu0", (n,)), ("lb_h", (n,))):
            s[name] = torch.zeros(shape, dtype=torch.float64, device="cuda")
        s["mu"] = torch.ones(1, dtype=torch.float64, device="cuda")
    elif kind == "surrogate":
        s["K"], s["q"] = _pairs(seed, case["n"])
        s["out"] = torch.zeros_like(s["K"])
        s["counts"] = _counts(case["n"], case["elements"])
        model = Surrogate(case["process"], elements_z=BATCH_Z[:case["elements"]])
        # features scaled to [-1, 1] over the trained domain, a residual of small spread
        norm = np.array([3.45, -8.06, 0.4, 2.6, 0.1, 0.12, 2.4, 0.37, 0.0, 20.0], dtype=np.float32)
        model.set_params(init_params(seed % 1000), norm)
        # the share of cells that a trained model is trusted in: away from the kinematic edges, at random
        g = np.random.default_rng(seed)
        trust = g.random((case["elements"], *GRID)) < 0.3
        trust[:, :, -4:] = False
        s["model"], s["trust"] = model, trust.astype(np.uint8)
    else:
        n = 4 * case["batch"] * 4
        s["model"] = Surrogate(case["process"], batch=case["batch"])
        K, q = _pairs(seed, n)
        elem = torch.arange(n, device="cuda") % len(BATCH_Z)
        X, R, valid, _ = s["model"].prepare(K, q, elem)
        pick = torch.nonzero(valid).ravel()
        pick = pick[torch.arange(2 * case["batch"], device="cuda") % pick.numel()]
        s["model"].fit_norm(X[pick], R[pick])
        s["X"], s["T"] = s["model"].normalise(X[pick], R[pick])
        s["params"], s["norm"] = init_params(seed % 1000), s["model"].norm
    return s


# ---------------------------------------------------------------- one pass
def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "dcs":
        if case["allocate"]:
            return [dcs.map(p, s["K"], s["q"], s["element"], s["mass"], case["precision"]) for p in PROCESSES]
        return [dcs.vmap(p, o, s["K"], s["q"], s["element"], s["mass"], case["precision"])
                for p, o in zip(PROCESSES, s["out"])]
    if kind == "host":
        return [dcs.vmap_host(p, o, s["K"], s["q"], s["element"], s["mass"], case["precision"])
                for p, o in zip(PROCESSES, s["out"])]
    if kind == "batched":
        return [(plan.execute_graph if case["graph"] else plan.execute)(o, s["K"], s["q"])
                for plan, o in zip(s["plans"], s["out"])]
    if kind == "losses":
        for i, p in enumerate(PROCESSES):
            for moment in (0, 1):
                dcs.recoil_integral(p, moment, s["out"][2 * i + moment], s["K"], XLOW, s["element"], MUON_MASS,
                                    case["min_points"])
        dcs.soft_scattering(s["out"][8], s["K"], s["element"], MUON_MASS)
        return s["out"]
    if kind == "elastic":
        for i, el in enumerate(s["elements"]):
            dcs.coulomb_data(s["fCM"][i], s["screening"][i], s["fspin"][i], s["invlambda"][i], s["K"], el, MUON_MASS)
            dcs.coulomb_transport(s["G"][i], s["screening"][i], s["fspin"][i], s["mu"])
        dcs.hard_scattering(s["mu0"], s["lb_h"], s["G"], s["fCM"], s["screening"], s["invlambda"], s["fspin"])
        return {k: s[k] for k in ("fCM", "screening", "fspin", "invlambda", "G", "mu0", "lb_h")}
    if kind == "surrogate":
        return s["model"].infer(s["K"], s["q"], s["counts"], trust=s["trust"], out=s["out"])
    m = s["model"]
    m.set_params(s["params"], s["norm"])
    losses = m.fit(s["X"], s["T"], steps=case["steps"])
    params, adam_m, adam_v, _ = m.get_params()
    return {"losses": losses, "params": params, "adam_m": adam_m, "adam_v": adam_v}


def work(case):
    n, kind = case.get("n", 0), case["kind"]
    if kind in ("dcs", "host", "batched"):
        return {"bytes": 4 * 24.0 * n, "flops": sum(FLOPS.values()) * n}
    if kind == "losses":
        nodes = 6 * math.ceil(case["min_points"] / 6)
        return {"bytes": 9 * 16.0 * n, "flops": n * (2 * nodes * sum(FLOPS.values()) + 102 * FLOPS["photonuclear"])}
    if kind == "elastic":
        # about ten steps of the root search, two objectives each
        return {"bytes": 8.0 * n * (3 + 15 * case["elements"]), "flops": n * case["elements"] * (300.0 + 20 * 150)}
    if kind == "surrogate":
        return {"bytes": 24.0 * n, "flops": 0.25 * n * FLOPS[case["process"]]}
    return {"bytes": case["steps"] * (case["batch"] * 20.0 + 33793 * 28.0),
            "flops": case["steps"] * case["batch"] * 6.0 * 33793}


# ---------------------------------------------------------------- the same in plain 64 bits
ME, NA, PM, MPI = 0.510998910e-3, 6.02214076e23, 0.931494, 0.134977
GL6 = ((0.03376524, 0.16939531, 0.38069041, 0.61930959, 0.83060469, 0.96623476),
       (0.08566225, 0.18038079, 0.23395697, 0.23395697, 0.18038079, 0.08566225))
GL8 = ((0.01985507, 0.10166676, 0.2372338, 0.40828268, 0.59171732, 0.7627662, 0.89833324, 0.98014493),
       (0.05061427, 0.11119052, 0.15685332, 0.18134189, 0.18134189, 0.15685332, 0.11119052, 0.05061427))
GL9 = ((0.0, -0.8360311073266358, 0.8360311073266358, -0.9681602395076261, 0.9681602395076261, -0.3242534234038089,
        0.3242534234038089, -0.6133714327005904, 0.6133714327005904),
       (0.3302393550012598, 0.1806481606948574, 0.1806481606948574, 0.0812743883615744, 0.0812743883615744,
        0.3123470770400029, 0.3123470770400029, 0.2606106964029354, 0.2606106964029354))


def _select(closed, v):
    return torch.where(closed, torch.zeros_like(v), v)


def _bremsstrahlung(K, q, el, m):
    Z, A, se = el.Z, el.A, 1.648721271
    bn, be = (202.4, 446.0) if Z == 1 else (182.7 * Z ** (-1 / 3), 1429.0 * Z ** (-2 / 3))
    dn, rem, E = 1.54 * A ** 0.27, 5.63588e-13 * ME / m, K + m
    nu = q / E
    delta = 0.5 * m * m / E * nu / (1 - nu)
    phi_n = torch.log(bn * (m + delta * (dn * se - 2)) / (dn * (ME + delta * se * bn))).clamp(min=0)
    phi_e = torch.log(be * m / ((1 + delta * (m / (ME * ME * se))) * (ME + delta * se * be))).clamp(min=0)
    phi_e = _select(q >= E / (1 + 0.5 * m * m / (ME * E)), phi_e)
    d = 7.297182e-7 * rem * rem * Z * (Z * phi_n + phi_e) * (4 / 3 * (1 / nu - 1) + nu)
    return d.clamp(min=0) * 1e3 * NA / A


def _pair_production(K, q, el, m):
    Z, A, se = el.Z, el.A, 1.6487212707
    z13, r, E = Z ** (1 / 3), m / ME, K + m
    closed = (q <= 4 * ME) | (q >= K + m * (1 - 0.75 * se * z13))
    q = torch.where(closed, 0.1 * K, q)
    nu = q / E
    beta = 0.5 * nu * nu / (1 - nu)
    az = (202.4 if Z == 1 else 183.0) / z13
    gamma = 1 + K / m
    x0, x1 = 4 * ME / q, 6 / (gamma * (gamma - q / m))
    am = (x0 + 2 * (1 - x0) * x1) / (1 + (1 - x1) * torch.sqrt((1 - x0).clamp(min=0)))
    closed = closed | (am >= 1) | (am <= 0)
    tmin = torch.log(torch.where(closed, torch.full_like(am, 0.5), am))
    total = torch.zeros_like(K)
    for x, w in zip(*GL8):
        eps = torch.exp(x * tmin)
        rho2 = (1 - eps) ** 2
        s = eps * (2 - eps)
        xi = 0.5 * r * r * beta * s
        be = torch.where(xi >= 1e3, 0.5 / xi * ((3 - rho2) + 2 * beta * (1 + rho2)),
                         ((2 + rho2) * (1 + beta) + xi * (3 + rho2)) * torch.log(1 + 1 / xi) + (s - beta) / (1 + xi)
                         - 3 - rho2)
        ye = (5 - rho2 + 4 * beta * (1 + rho2)) / (2 * (1 + 3 * beta) * torch.log(3 + 1 / xi) - rho2
                                                    - 2 * beta * (2 - rho2))
        xe, cl = (1 + xi) * (1 + ye), 2 * se * ME * az / s
        le = torch.log(az * torch.sqrt(xe) * q / (q + cl * xe)) - 0.5 * torch.log(1 + 2.25 * z13 * z13 / (r * r) * xe)
        bmu = torch.where(xi <= 1e-3, 0.5 * xi * (5 - rho2 + beta * (3 + rho2)),
                          ((1 + rho2) * (1 + 1.5 * beta) - (1 + 2 * beta) * s / xi) * torch.log(1 + xi)
                          + xi * (s - beta) / (1 + xi) + (1 + 2 * beta) * s)
        ymu = (4 + rho2 + 3 * beta * (1 + rho2)) / ((1 + rho2) * (1.5 + 2 * beta) * torch.log(3 + xi) + 1 - 1.5 * rho2)
        lmu = torch.log(r * az * q / (1.5 * z13 * (q + cl * (1 + xi) * (1 + ymu))))
        total += w * ((be * le).clamp(min=0) + (bmu * lmu).clamp(min=0) / (r * r)) * eps
    total *= -tmin
    g1, g2 = (4.4e-5, 4.8e-5) if Z == 1 else (1.95e-5, 5.30e-5)
    zeta = (0.073 * torch.log(gamma / (1 + g1 * gamma * z13 * z13)) - 0.26).clamp(min=0)
    zeta = _select((gamma <= 35) | (zeta == 0), zeta / (0.058 * torch.log(gamma / (1 + g2 * gamma * z13)) - 0.14))
    d = 1.794664e-34 * Z * (Z + zeta) * (E - q) * total / (q * E)
    return _select(closed, d.clamp(min=0) * 1e3 * NA * E / A)


def _photonuclear(K, q, el, m):
    A, E = el.A, K + m
    closed = (q < 1) | (q < 2e-3 * K) | (q >= E - m) | (q <= MPI * (1 + 0.5 * MPI / PM))
    q = torch.where(closed, 0.5 * E, q)
    y = q / E
    lo, hi = m * m * y * y / (1 - y), 2 * PM * (q - MPI) - MPI * MPI
    closed = closed | (hi < lo)
    lo, hi = torch.where(closed, torch.ones_like(lo), lo), torch.where(closed, torch.full_like(hi, 2.0), hi)
    q = torch.where(closed, torch.full_like(q, 10.0), q)
    width, mid = torch.log(hi) - torch.log(lo), 0.5 * (torch.log(hi) + torch.log(lo))
    total = torch.zeros_like(K)
    for node, w in zip(*GL9):
        Q2 = torch.exp(mid + 0.5 * width * node)
        x = 0.5 * Q2 / (PM * q)
        w2 = Q2 * (1 / x - 1)
        lnt = torch.log(torch.log(torch.log((Q2 + 0.52544) / 0.06527) / math.log(0.52544 / 0.06527)))
        xp, xr = (Q2 + 49.457) / (Q2 + 49.457 + w2), (Q2 + 0.15052) / (Q2 + 0.15052 + w2)
        cp = 0.28067 + (0.28067 - 0.22291) * (1 / (1 + torch.exp(2.1979 * lnt)) - 1)
        ap = -0.0808 + (-0.0808 + 0.44812) * (1 / (1 + torch.exp(1.1709 * lnt)) - 1)
        bp = 0.36292 + 1.8917 * torch.exp(1.8439 * lnt)
        cr = 0.80107 + 0.97307 * torch.exp(3.4942 * lnt)
        ar = 0.58400 + 0.37888 * torch.exp(2.6063 * lnt)
        br = 0.01147 + 3.7582 * torch.exp(0.49338 * lnt)
        l1x = torch.log(1 - x)
        f2 = Q2 / (Q2 + 0.31985) * (cp * torch.exp(ap * torch.log(xp) + bp * l1x)
                                    + cr * torch.exp(ar * torch.log(xr) + br * l1x))
        a = torch.where(x < 0.0014, torch.full_like(x, A ** -0.1),
                        torch.where(x < 0.04, torch.exp((0.069 * torch.log10(x) + 0.097) * math.log(A)),
                                    torch.ones_like(x)))
        f2a = 0.5 * A * a * (2 + x * (-1.85 + x * (2.45 + x * (-2.35 + x)))) * f2
        q2 = Q2.clamp(min=0.3)
        theta = 1 + 12 * q2 / (1 + q2) * 0.015625 / (0.015625 + x * x)
        rw = 0.635 / torch.log(q2 / 0.04) * theta + 0.5747 / q2 - 0.3534 / (0.09 + q2 * q2)
        dds = ((1 - y + 0.5 * (1 - 2 * m * m / Q2) * (y * y + Q2 / (E * E)) / (1 + rw)) / (Q2 * Q2)
               - 0.25 / (E * E * Q2))
        total += w * 2.603096e-35 * f2a * dds / q * Q2
    return _select(closed, total.clamp(min=0) * 0.5 * width * 1e3 * NA * E / A)


def _ionisation(K, q, el, m):
    p2, E = K * (K + 2 * m), K + m
    wmax = 2 * ME * p2 / (m * m + ME * (ME + 2 * E))
    closed = (wmax < 0.05 * K) | (q > wmax) | (q <= 0.62 * el.I)
    cs = 1.535336e-5 * E * el.Z / el.A * (0.5 / p2 + 1 / q * (E * E / p2 / q - 1 / wmax))
    l1 = torch.log(1 + 2 * q / ME)
    delta = 1.16141e-3 * l1 * (torch.log(4 * E * (E - q).clamp(min=0) / (m * m)) - l1)
    return _select(closed, cs * (1 + _select(K < 0.5 * (m - ME) ** 2 / ME, delta)))


_FORMULA = dict(zip(PROCESSES, (_bremsstrahlung, _pair_production, _photonuclear, _ionisation)))


def _evaluate(process, K, q, el, m):
    step = 1 << 22
    return torch.cat([_FORMULA[process](K[i:i + step], q[i:i + step], el, m) for i in range(0, K.numel(), step)])


def _closed_form_ionisation(moment, K, el, m):
    p2, E = K * (K + 2 * m), K + m
    wmax = 2 * ME * p2 / (m * m + ME * (ME + 2 * E))
    wmin = (K * XLOW).clamp(min=0.62 * el.I)
    a0, a1, a2, lw = 0.5 / p2, -1 / wmax, E * E / p2, torch.log(wmax / wmin)
    if moment == 0:
        term = a0 * (wmax - wmin) + a1 * lw + a2 * (1 / wmin - 1 / wmax)
    else:
        term = 0.5 * a0 * (wmax * wmax - wmin * wmin) + a1 * (wmax - wmin) + a2 * lw
    return _select((wmax < 0.05 * K) | (wmax <= wmin), 1.535336e-5 * el.Z / el.A * term)


def _loss(process, moment, K, el, m, min_points):
    intervals = math.ceil(min_points / 6)
    lo = torch.log(K * XLOW)
    h = (torch.log(K) - lo) / intervals
    total = torch.zeros_like(K)
    for i in range(6 * intervals):
        q = torch.exp(lo + h * (i // 6 + GL6[0][i % 6]))
        total += _evaluate(process, K, q, el, m) * q ** (1 + moment) * h * GL6[1][i % 6]
    total /= K + m
    if process != "ionisation":
        return total
    return torch.where(K <= 0.5 * (m - ME) ** 2 / ME, _closed_form_ionisation(moment, K, el, m), total)


def _soft_scattering(K, el, m):
    p2, E = K * (K + 2 * m), K + m
    wmax, w0 = 2 * ME * p2 / (m * m + ME * (ME + 2 * E)), 2 * p2 / ME
    mu3, mu2 = torch.minimum(K * 0.05 / w0, wmax / w0), 0.62 * el.I / w0
    ion = 2 * 1.535336e-5 / el.A * el.Z * (0.25 * w0 / p2 * (mu3 * mu3 - mu2 * mu2) - (mu3 - mu2) / wmax
                                          + E * E / (w0 * p2) * torch.log(mu3 / mu2))
    total, lo = _select(mu2 >= mu3, ion), math.log(1e-6)
    for i in range(102):
        nu = 0.05 * math.exp(lo - lo / 17 * (i // 6 + GL6[0][i % 6]))
        q = nu * K
        q2, tmax = q * q, 1.876544 * q
        tmin = q2 * m * m / (E * (E - q))
        b1, c1 = 1 / (1 - q2 / 0.4), 1 / (1 - 0.4 / q2)
        l1, l2 = b1 * torch.log((q2 + tmax) / (q2 + tmin)), c1 * torch.log((0.4 + tmax) / (0.4 + tmin))
        i0, i1 = torch.log(tmax / tmin) - l1 - l2, l1 * q2 + l2 * 0.4
        i2 = (tmax - tmin) * (b1 * q2 + c1 * 0.4) - l1 * q2 * q2 - l2 * 0.16
        f = _photonuclear(K, q, el, m) * (i1 * tmax - i2) / ((i0 * tmax - i1) * K * (K + 2 * m)) * nu
        total += 2 * f * (-lo / 17) * GL6[1][i % 6]
    return total


def _coulomb(K, el, m):
    ma = el.A * 0.931494
    s = 1 / torch.sqrt((m + ma) ** 2 + 2 * ma * K)
    k0 = ((K * ma + m * (m + ma)) * s - m).clamp(min=1e-9)
    b2 = K * (K + 2 * m) / (K + m + ma) ** 2
    fcm = torch.stack([(K + m + ma) * s, torch.sqrt((m / ma) ** 2 * (1 - b2) + b2)], -1)
    e = k0 + m
    fspin, p2 = k0 * (e + m) / (e * e), k0 * (k0 + 2 * m)
    s1, s2 = 5.8406e-2 / p2 / (1.02934 * el.A ** (1 / 3) + 0.435) ** 2, 5.8406e-2 / p2 / 4
    z2 = 5.3251346e-5 * (el.Z * e) ** 2 / p2
    series = sum(z2 / (i * (i * i + z2)) for i in range(1, 11 + el.Z))
    ck = torch.exp(torch.where(z2 > 1, series, 1 - 1 / (1 + z2) + z2 * (0.2021 + z2 * (0.0083 * z2 - 0.0369))))
    r = (k0 / e) ** 2
    s0 = 5.179587126e-12 * el.Z ** (2 / 3) * (r * ck + (1 - r) * (1 + 3.34 * z2)) / p2
    d01, d02, d12 = 1 / (s0 - s1), 1 / (s0 - s2), 1 / (s1 - s2)
    f = [(d01 * d02) ** 2, (d01 * d12) ** 2, (d12 * d02) ** 2]
    screening = torch.stack([s0, s1, s2, 2 * f[0] * (d01 + d02), 2 * f[1] * (d12 - d01), -2 * f[2] * (d12 + d02),
                             *f], -1)
    dw = k0 * (k0 + 2 * m) / (el.Z * e)
    return fcm, screening, fspin, 1 / (el.A * 2.54910918e8 * s0 * (1 + s0) * dw * dw)


def _transport(screening, fspin):
    """Transport coefficients up to mu = 1."""
    c0, c1 = 0.0, 0.0
    for i in range(3):
        s = screening[..., i]
        r, ll = 1 / (1 + s), torch.log(1 + 1 / s)
        i1, j1, i2, j2 = ll - r, 1 - s * ll, 1 - 2 * s * ll + s * r, 0.5 + s * s * ll - s
        c0 = c0 + screening[..., 3 + i] * (ll - fspin * j1) + screening[..., 6 + i] * (r / s - fspin * i1)
        c1 = c1 + screening[..., 3 + i] * (j1 - fspin * j2) + screening[..., 6 + i] * (i1 - fspin * i2)
    s0, s1, s2 = screening[..., 0], screening[..., 1], screening[..., 2]
    k = s0 * (1 + s0) * s1 * s1 * s2 * s2
    return torch.stack([c0 * k, 2 * c1 * k], -1)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("dcs", "host"):
        K, q = _pairs(seed, case["n"])
        return [_evaluate(p, K, q, ELEMENTS[case["Z"]], MASS[case["particle"]]) for p in PROCESSES]
    if kind == "batched":
        K, q = _pairs(seed, case["n"])
        counts = _counts(case["n"], case["elements"])
        return [torch.cat([_evaluate(p, k, r, el, MUON_MASS) for k, r, el in
                           zip(K.split(counts), q.split(counts), _elements(case)) if k.numel()]) for p in PROCESSES]
    if kind == "losses":
        K, el = _grid(seed, case["n"]), ELEMENTS[case["Z"]]
        return [_loss(p, moment, K, el, MUON_MASS, case["min_points"]) for p in PROCESSES for moment in (0, 1)] + [
            _soft_scattering(K, el, MUON_MASS)]
    if kind == "elastic":
        fcm, screening, fspin, invlambda = (torch.stack(v) for v in zip(*(
            _coulomb(_grid(seed, case["n"]), el, MUON_MASS) for el in _elements(case))))
        # the cut-off is the end of a root search that stops at 1e-6: no 64-bit value of its own
        return {"fCM": fcm, "screening": screening, "fspin": fspin, "invlambda": invlambda,
                "G": _transport(screening, fspin), "mu0": None, "lb_h": None}
    # the surrogate's answers depend on a learned network in bfloat16
    return None
