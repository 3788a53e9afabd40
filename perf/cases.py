"""The work that a user of this framework has it do, as cases to be timed and compared.

A case is one call (or the calls of one step) through the public Python API:
source terms and Jacobians of batches of cells, the stiff reactor advance, the
surrogate + fallback advance, the tabulated (FLINT's own tables) chemistry of a
CFD step, and a stretch of surrogate training.  ``listed()`` holds the sizes
that stand for real use, ``draw()`` more of the same ranges.

All outputs are FP64 but the training's (FP32 weights), all inputs are made on
the GPU from the seed.  The reactor cases integrate at rtol 1e-10 .. 1e-11
instead of the default 1e-8: two builds that differ in the last bit of one rate
take different step-size decisions, so at 1e-8 their results differ by the
integrator's own tolerance, and the step counts differ too (they are control
decisions, not results, and are not returned).  At 1e-10 the results of any
correct build agree to about 1e-10.
"""
import json
import math
import os

import numpy as np
import torch

from flint_gb300.api import CELL_MAJOR, SPECIES_MAJOR, Chemistry
from flint_gb300.mech import Mechanism
from flint_gb300.surrogate import Surrogate, train
from flint_gb300.tables import Tables, generate

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_MECH = {
    "c1": "flint_gb300/data/mech_c1.json",                # 2-step CH4/air, 6 species, 2 reactions
    "c2": "flint_gb300/data/mech_c2.json",                # 31 species, 160 reactions
    "c5": "flint_gb300/data/mech_c5.json",                # 54 species, 320 reactions
    "tsr_rich_31": "tests/golden/mech_tsr_rich_31.json",  # a reduced CH4/air mechanism, 31 species
}
_CKPT = {"c2": "flint_gb300/data/surrogate_c3.bin"}
_ATM = 101325.0


def _path(rel):
    return os.path.join(_ROOT, rel)


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the source terms of one block of a CFD grid, called once per block and
        # stage: launch latency counts (the reference's chemistry_source)
        {"name": "source_c1_block", "kind": "source", "mech": "c1", "n": 4096},
        # the source terms with cp and h of a whole small grid, 2-step CH4/air
        {"name": "wdot_c1_64k", "kind": "wdot", "mech": "c1", "n": 65536, "thermo": True, "species_major": False},
        # the source terms with cp and h of a million cells, detailed mechanism
        {"name": "wdot_c2_1m", "kind": "wdot", "mech": "c2", "n": 1048576, "thermo": True, "species_major": False},
        # the larger mechanism, species-major storage (Fortran's (N, ns)), a ragged count
        {"name": "wdot_c5_ragged", "kind": "wdot", "mech": "c5", "n": 100003, "thermo": False, "species_major": True},
        # source terms + analytic Jacobian for an implicit solver
        {"name": "jac_c2_64k", "kind": "jac", "mech": "c2", "n": 65536, "species_major": False},
        {"name": "jac_c5_ragged", "kind": "jac", "mech": "c5", "n": 20011, "species_major": False},
        # the right-hand side of a few hundred cells, as an outer ODE solver asks for it
        {"name": "rhs_c2_small", "kind": "rhs", "mech": "c2", "n": 300},
        # the stiff 0D reactor advance, every cell over its own dt
        {"name": "reactor_c2", "kind": "reactor", "mech": "c2", "n": 8192, "rtol": 1e-10},
        {"name": "reactor_c5", "kind": "reactor", "mech": "c5", "n": 2048, "rtol": 1e-11},
        # the learned advance: networks, gate and FP64 fallback of a million cells
        {"name": "surrogate_c2_1m", "kind": "surrogate", "mech": "c2", "n": 1048576, "rtol": 1e-10},
        # a CFD step on FLINT's own tables: conserved to primitive variables, then the source terms
        {"name": "tables_c2_256k", "kind": "tables", "mech": "c2", "n": 262144, "ndim": 3},
        # a stretch of surrogate training: batches drawn, forward, backward, Adam
        {"name": "train_c2", "kind": "train", "mech": "c2", "steps": 20, "batch": 4096},
    ]


def _size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["source", "wdot", "wdot", "wdot", "jac", "jac", "rhs", "reactor", "surrogate", "tables", "train"])
    if kind == "source":
        return {"kind": kind, "mech": "c1", "n": _size(rng, 100, 400000)}
    if kind == "wdot":
        mech = rng.choice(["c1", "c2", "c5", "tsr_rich_31"])
        hi = {"c1": 2000000, "c2": 1048576, "c5": 400000, "tsr_rich_31": 1048576}[mech]
        return {"kind": kind, "mech": mech, "n": _size(rng, 500, hi), "thermo": rng.random() < 0.5,
                "species_major": rng.random() < 0.5}
    if kind == "jac":
        mech = rng.choice(["c2", "c5", "tsr_rich_31"])
        return {"kind": kind, "mech": mech, "n": _size(rng, 200, 20000 if mech == "c5" else 65536),
                "species_major": rng.random() < 0.5}
    if kind == "rhs":
        return {"kind": kind, "mech": rng.choice(["c2", "c5"]), "n": _size(rng, 50, 20000)}
    if kind == "reactor":
        mech = rng.choice(["c2", "c5"])
        return {"kind": kind, "mech": mech, "n": _size(rng, 200, 8000) if mech == "c2" else _size(rng, 100, 2000),
                "rtol": 10.0 ** rng.uniform(-10.5, -10.0) if mech == "c2" else 10.0 ** rng.uniform(-11.0, -10.7)}
    if kind == "surrogate":
        return {"kind": kind, "mech": "c2", "n": _size(rng, 20000, 1000000), "rtol": 10.0 ** rng.uniform(-10.5, -10.0)}
    if kind == "tables":
        return {"kind": kind, "mech": rng.choice(["c2", "tsr_rich_31"]), "n": _size(rng, 500, 260000),
                "ndim": rng.choice([1, 2, 3])}
    return {"kind": "train", "mech": "c2", "steps": rng.randint(5, 20), "batch": _size(rng, 512, 4096)}


# ------------------------------------------------------------------ the inputs
def _uniform(n, lo, hi):
    return lo + (hi - lo) * torch.rand(n, dtype=torch.float64, device="cuda")


def _names(m):
    return [s.name for s in m.species]


def _methane_air(m, n, phi_lo, phi_hi):
    """Mass fractions of CH4 + air at equivalence ratios phi_lo .. phi_hi."""
    names = _names(m)
    W = torch.tensor([s.mw for s in m.species], dtype=torch.float64, device="cuda")
    o2 = 2.0 / _uniform(n, phi_lo, phi_hi)
    X = torch.zeros(n, m.ns, dtype=torch.float64, device="cuda")
    X[:, names.index("CH4")] = 1.0
    X[:, names.index("O2")] = o2
    X[:, names.index("N2")] = 3.76 * o2
    Y = X * W
    return Y / Y.sum(1, keepdim=True)


def _partly_burnt(m, n):
    """2-step CH4/air: a mixture of unburnt and burnt gas with progress U(0, 1)."""
    names = _names(m)
    W = torch.tensor([s.mw for s in m.species], dtype=torch.float64, device="cuda")
    o2 = 2.0 / _uniform(n, 0.5, 2.0)
    Xu = torch.zeros(n, m.ns, dtype=torch.float64, device="cuda")
    Xb = torch.zeros_like(Xu)
    Xu[:, names.index("CH4")] = 1.0
    Xu[:, names.index("O2")] = o2
    x = torch.clamp(o2 / 1.5, max=1.0)                 # CH4 burnt to CO + 2 H2O
    y = torch.minimum(x, 2.0 * (o2 - 1.5 * x))         # CO burnt to CO2
    Xb[:, names.index("CH4")] = 1.0 - x
    Xb[:, names.index("CO")] = x - y
    Xb[:, names.index("CO2")] = y
    Xb[:, names.index("H2O")] = 2.0 * x
    Xb[:, names.index("O2")] = o2 - 1.5 * x - 0.5 * y
    Xu[:, names.index("N2")] = 3.76 * o2
    Xb[:, names.index("N2")] = 3.76 * o2
    c = _uniform(n, 0.0, 1.0)[:, None]
    Yu, Yb = Xu * W, Xb * W
    Y = (1.0 - c) * Yu / Yu.sum(1, keepdim=True) + c * Yb / Yb.sum(1, keepdim=True)
    return Y.clamp(min=0.0)


def _dirichlet(n, k, alpha=0.3):
    """Dirichlet(alpha) mass fractions: most species are traces, as in a flame."""
    g = torch._standard_gamma(torch.full((n, k), alpha, dtype=torch.float64, device="cuda")).clamp(min=1e-200)
    return g / g.sum(1, keepdim=True)


def _states(m, mech, n, seed):
    """T, p, Y of `n` cells for source terms."""
    torch.manual_seed(seed)
    if mech == "c1":
        T, p, Y = _uniform(n, 300.0, 2500.0), _uniform(n, 1.0, 20.0) * _ATM, _partly_burnt(m, n)
    else:
        T, p, Y = _uniform(n, 800.0, 2800.0), _uniform(n, 1.0, 40.0) * _ATM, _dirichlet(n, m.ns)
    return T, p, Y.contiguous()


def _reactor_states(m, mech, n, seed):
    """T, p, Y, dt of `n` cells for a reactor advance."""
    torch.manual_seed(seed)
    if mech == "c5":
        T, p, Y = _uniform(n, 900.0, 2000.0), _uniform(n, 1.0, 40.0) * _ATM, _methane_air(m, n, 0.4, 3.0)
        dt = 10.0 ** _uniform(n, -7.0, -4.0)
    else:
        T, p, Y = _uniform(n, 900.0, 1600.0), _uniform(n, 1.0, 20.0) * _ATM, _methane_air(m, n, 0.5, 2.0)
        dt = 10.0 ** _uniform(n, -6.0, -4.0)
    return T, p, Y.contiguous(), dt


def _load(mech):
    return Mechanism.load(_path(_MECH[mech]))


def _density(m, T, p, Y):
    W = torch.tensor([s.mw for s in m.species], dtype=torch.float64, device="cuda")
    return p / (m.r_eos * T * (Y / W).sum(1))


def _cfd_state(m, mech, n, ndim, seed):
    """Partial densities, conserved variables and a temperature guess of `n` cells."""
    T, p, Y = _states(m, mech, n, seed)
    roi = _density(m, T, p, Y)[:, None] * Y
    rho = roi.sum(1)
    u = torch.randn(n, ndim, dtype=torch.float64, device="cuda") * 100.0
    h = _mix_enthalpy(m, T, Y)
    energy = h - p / rho + 0.5 * (u * u).sum(1)
    cons = torch.cat([roi, rho[:, None] * u, (rho * energy)[:, None]], 1).contiguous()
    guess = T * (1.0 + 0.02 * torch.randn(n, dtype=torch.float64, device="cuda"))
    return roi.contiguous(), cons, guess.clamp(400.0, 2990.0), T


def _mix_enthalpy(m, T, Y):
    W = torch.tensor([s.mw for s in m.species], dtype=torch.float64, device="cuda")
    return ((_nasa(m, T)[1] * T[:, None] * m.r_thermo / W) * Y).sum(1)


def prepare(case, seed):
    kind, mech = case["kind"], case["mech"]
    m = _load(mech)
    if kind == "tables":
        roi, cons, guess, T = _cfd_state(m, mech, case["n"], case["ndim"], seed)
        return {"kind": kind, "tables": Tables(generate(m)), "roi": roi, "cons": cons, "guess": guess, "T": T}
    chem = Chemistry(m)
    s = {"kind": kind, "chem": chem}
    if kind in ("reactor", "surrogate"):
        T, p, Y, dt = _reactor_states(m, mech, case["n"], seed)
        s.update(T0=T, p=p, Y0=Y, dt=dt, T=T.clone(), Y=Y.clone(), rtol=case["rtol"], atol=case["rtol"] * 1e-6)
        s["status"] = torch.empty(case["n"], dtype=torch.int32, device="cuda")
        s["nsteps"] = torch.empty_like(s["status"])
        if kind == "surrogate":
            s["sur"] = Surrogate.load(chem, _path(_CKPT[mech]), weights_only=True)
        return s
    if kind == "train":
        # normalised features of reactor states, and targets near what the
        # trained network predicts for them (a training set in mid-training)
        sur = Surrogate.load(chem, _path(_CKPT[mech]))
        X = sur.features(*_reactor_states(m, mech, 65536, seed))
        Yt = sur.predict(X)
        Yt += 0.05 * torch.randn_like(Yt)
        s.update(sur=sur, X=X, Yt=Yt, steps=case["steps"], batch=case["batch"], seed=seed)
        return s
    T, p, Y = _states(m, mech, case["n"], seed)
    if kind == "source":
        s.update(roi=(_density(m, T, p, Y)[:, None] * Y).contiguous(), T=T)
        return s
    if case.get("species_major"):
        s.update(layout=SPECIES_MAJOR, Y=Y.t().contiguous())
    else:
        s.update(layout=CELL_MAJOR, Y=Y)
    s.update(T=T, p=p, thermo=case.get("thermo", False))
    return s


# ------------------------------------------------------------------ one pass
def run(s):
    kind, chem = s["kind"], s.get("chem")
    if kind == "source":
        return chem.chemistry_source(s["roi"], s["T"])
    if kind == "wdot":
        cp, h = (torch.empty_like(s["T"]), torch.empty_like(s["T"])) if s["thermo"] else (None, None)
        w, cp, h = chem.wdot(s["T"], s["p"], s["Y"], layout=s["layout"], cp=cp, h=h)
        return [w, cp, h] if s["thermo"] else [w]
    if kind == "jac":
        return list(chem.wdot_jac(s["T"], s["p"], s["Y"], layout=s["layout"], wdot=torch.empty_like(s["Y"])))
    if kind == "rhs":
        return chem.rhs(s["T"], s["p"], s["Y"])
    if kind in ("reactor", "surrogate"):
        # the states are advanced in place, so each pass starts from a fresh copy
        s["T"].copy_(s["T0"])
        s["Y"].copy_(s["Y0"])
        if kind == "reactor":
            chem.reactor_advance(s["T"], s["p"], s["Y"], s["dt"], rtol=s["rtol"], atol=s["atol"], max_steps=200000,
                                 status=s["status"], nsteps=s["nsteps"])
        else:
            s["sur"].advance(s["T"], s["p"], s["Y"], s["dt"], rtol=s["rtol"], atol=s["atol"], max_steps=200000,
                             status=s["status"], nsteps=s["nsteps"], wait=False)
        return [s["T"], s["Y"], s["status"]]
    if kind == "tables":
        prim, T = s["tables"].cons2prim(s["cons"], s["guess"])
        return [prim, T, s["tables"].chemistry_source(s["roi"], s["T"])]
    hist = train(s["sur"], s["X"], s["Yt"], s["steps"], batch=s["batch"], lr=1e-3, total=2000, seed=s["seed"] % 1000,
                 log_every=s["steps"])
    state, step = s["sur"].get_state()
    P = s["sur"].P
    return [float(hist[-1][1]), state[:P].copy(), state[P:2 * P].copy(), state[2 * P:].copy(), int(step)]


# ------------------------------------------------------------------ what a pass cannot do without
# FP64 operations of one evaluation, counted on the mechanism: two exponentials
# and a dozen products per reaction, a polynomial per species and property, one
# multiply-add per entry of the stoichiometric matrix; the Jacobian adds the
# products by slot and its assembly.
def _kinetics_flops(ns, nr, jac=False):
    f = 60.0 * nr + 40.0 * ns + 8.0 * nr
    return f + (60.0 * nr + 6.0 * (ns + 1) ** 2) if jac else f


def work(case):
    kind = case["kind"]
    ns, nr = {"c1": (6, 2), "c2": (31, 160), "c5": (54, 320), "tsr_rich_31": (31, 197)}[case["mech"]]
    nv = ns + 1
    if kind == "train":
        dims = [ns + 2, 256, 256, 256, 256, ns + 1]
        weights = sum(a * b + b for a, b in zip(dims, dims[1:]))
        rows = case["steps"] * case["batch"]
        return {"bytes": 4.0 * rows * (dims[0] + dims[-1]) + case["steps"] * 24.0 * weights,
                "flops": 6.0 * rows * weights}
    n = case["n"]
    if kind == "source":
        return {"bytes": 8.0 * n * (2 * ns + 1), "flops": n * _kinetics_flops(ns, nr)}
    if kind == "wdot":
        return {"bytes": 8.0 * n * (2 * ns + 2 + (2 if case["thermo"] else 0)), "flops": n * _kinetics_flops(ns, nr)}
    if kind == "jac":
        return {"bytes": 8.0 * n * (2 * ns + 2 + nv * nv), "flops": n * _kinetics_flops(ns, nr, True)}
    if kind == "rhs":
        return {"bytes": 8.0 * n * (ns + 2 + nv), "flops": n * _kinetics_flops(ns, nr)}
    if kind == "tables":
        nc = ns + 1 + case["ndim"]
        return {"bytes": 8.0 * n * (2 * nc + 3 + 2 * ns), "flops": n * (20.0 * nr + 30.0 * ns)}
    # reactor: about 900 steps per cell at these tolerances (650 on the larger
    # mechanism), two Newton iterations (a right-hand side and a solve) each and
    # a factorisation every sixth step; the surrogate integrates 0.3 % of its
    # cells and runs two networks over all of them
    steps = 650.0 if case["mech"] == "c5" else 900.0
    cell = steps * (2.0 * (_kinetics_flops(ns, nr) + 2.0 * nv * nv) + nv ** 3 / 9.0)
    if kind == "reactor":
        return {"bytes": 8.0 * n * (2 * ns + 4), "flops": n * cell}
    net = 2.0 * 2.0 * ((ns + 2) * 256 + 3 * 256 * 256 + 256 * (ns + 1))
    return {"bytes": 8.0 * n * (2 * ns + 4), "flops": n * (0.003 * cell + net + 100.0 * ns)}


# ------------------------------------------------------------------ the same in plain torch, 64 bits
def _t(x):
    return torch.tensor(np.asarray(x, dtype=np.float64), device="cuda")


def _nasa(m, T):
    """cp/R, h/RT, s/R of every species, (n, ns) each."""
    lo, hi, tmid = _t([s.low for s in m.species]), _t([s.high for s in m.species]), _t([s.tmid for s in m.species])
    T = T[:, None]
    a = [torch.where(T <= tmid, lo[:, j], hi[:, j]) for j in range(7)]
    cp = a[0] + T * (a[1] + T * (a[2] + T * (a[3] + T * a[4])))
    h = a[0] + T * (a[1] / 2 + T * (a[2] / 3 + T * (a[3] / 4 + T * a[4] / 5))) + a[5] / T
    s = a[0] * torch.log(T) + T * (a[1] + T * (a[2] / 2 + T * (a[3] / 3 + T * a[4] / 4))) + a[6]
    return cp, h, s


class _Plain:
    """The kinetics of one mechanism file, written out."""

    def __init__(self, mech):
        with open(_path(_MECH[mech])) as f:
            d = json.load(f)
        self.d, sp, rx = d, d["species"], d["reactions"]
        self.m = type("M", (), {"species": [type("S", (), x) for x in sp], "r_eos": d["r_eos"], "r_thermo": d["r_thermo"]})
        names = [x["name"] for x in sp]
        ns, nr = len(sp), len(rx)
        self.ns, self.nr = ns, nr
        self.W = _t([x["mw"] for x in sp])
        nu1, nu2, orders, eff = (np.zeros((nr, ns)) for _ in range(4))
        for j, r in enumerate(rx):
            for k, v in r["reactants"].items():
                nu1[j, names.index(k)] = v
                orders[j, names.index(k)] = v
            for k, v in (r["orders"] or {}).items():
                orders[j, names.index(k)] = v
            for k, v in r["products"].items():
                nu2[j, names.index(k)] = v
            if r["rtype"]:
                if r["collider"] is not None:
                    eff[j, names.index(r["collider"])] = 1.0
                else:
                    eff[j, :] = r["default_eff"]
                    for k, v in (r["efficiencies"] or {}).items():
                        eff[j, names.index(k)] = v
        self.nu1, self.nu2, self.orders, self.eff = nu1, nu2, orders, _t(eff)
        self.net = _t(nu2 - nu1)
        self.slots = [self._slots(orders), self._slots(nu2)]
        self.A, self.b, self.E = (_t([r[k] for r in rx]) for k in ("A", "b", "EaR"))
        self.A0, self.b0, self.E0 = (_t([r[k] for r in rx]) for k in ("A0", "b0", "EaR0"))
        self.type = np.array([r["rtype"] for r in rx])
        self.rev = _t([1.0 if r["reversible"] else 0.0 for r in rx])
        tr = np.array([(list(r["troe"]) + [0.0] * 4)[:4] if r["troe"] else [0.5, 1.0, 1.0, 0.0] for r in rx])
        self.troe = [_t(tr[:, i]) for i in range(4)]

    @staticmethod
    def _slots(o):
        """(species, power) by slot, (nr,) each; unused slots have power 0."""
        width = max(1, int((o != 0).sum(1).max()))
        idx, pw = np.zeros((width, o.shape[0]), dtype=np.int64), np.zeros((width, o.shape[0]))
        for j in range(o.shape[0]):
            for i, k in enumerate(np.nonzero(o[j])[0]):
                idx[i, j], pw[i, j] = k, o[j, k]
        return [(torch.tensor(idx[i], device="cuda"), _t(pw[i])) for i in range(width)]

    def _product(self, c, side):
        out = None
        for idx, pw in self.slots[side]:
            x = c[:, idx]
            x = torch.where(pw == 1.0, x, torch.where(pw == 2.0, x * x, torch.where(
                pw == 0.0, torch.ones_like(x), torch.where(x > 0, torch.exp(pw * torch.log(x.clamp(min=1e-300))), torch.zeros_like(x)))))
            out = x if out is None else out * x
        return out

    def rates(self, T, c):
        """Molar production rates (n, ns) at concentrations c."""
        m = self.m
        _, h, s = _nasa(m, T)
        lnT, T1 = torch.log(T)[:, None], T[:, None]
        kf = self.A * torch.exp(self.b * lnT - self.E / T1)
        lnC0 = torch.log(self.d["p_ref"] / (m.r_thermo * T1))
        inv_kc = torch.exp((h - s) @ self.net.t() - self.net.sum(1) * lnC0)
        fall, third = (_t(x) > 0 for x in (self.type >= 2, self.type == 1))
        k = kf
        if (self.type > 0).any():
            M = c @ self.eff.t()
            k = torch.where(third, kf * M, kf)
            if (self.type >= 2).any():
                pr = torch.where(fall, self.A0 * torch.exp(self.b0 * lnT - self.E0 / T1) / kf * M, torch.ones_like(kf))
                a, t3, t1, t2 = self.troe
                fc = (1 - a) * torch.exp(-T1 / t3) + a * torch.exp(-T1 / t1) + torch.where(
                    t2 != 0, torch.exp(-t2 / T1), torch.zeros_like(kf))
                lf = torch.log10(fc)
                x = torch.log10(pr.clamp(min=1e-300)) - 0.4 - 0.67 * lf
                f1 = x / (0.75 - 1.27 * lf - 0.14 * x)
                F = torch.where(_t(self.type == 3) > 0, 10.0 ** (lf / (1 + f1 * f1)), torch.ones_like(kf))
                k = torch.where(fall, kf * pr / (1 + pr) * F, k)
        q = k * self._product(c, 0) - k * self.rev * inv_kc * self._product(c, 1)
        return q @ self.net

    def conc(self, T, p, Y):
        sw = (Y / self.W).sum(1)
        rho = p / (self.m.r_eos * T * sw)
        return rho, rho[:, None] * Y / self.W

    def rhs(self, T, p, Y):
        rho, c = self.conc(T, p, Y)
        w = self.rates(T, c)
        cp, h, _ = _nasa(self.m, T)
        fT = -T * (h * w).sum(1) / (c * cp).sum(1)
        return torch.cat([self.W * w / rho[:, None], fT[:, None]], 1)


def _chunks(n, size):
    return [slice(i, min(n, i + size)) for i in range(0, n, size)]


def _exact_tables(case, P, roi, cons, guess, T):
    """cons2prim's Newton and the source terms on 1-K tables, in plain torch."""
    m, ns, ndim = P.m, P.ns, case["ndim"]
    ri = 8314.51 / P.W
    tmin, tmax = 1.0, 3000.0

    def at(T, col):
        T0 = torch.floor(T)
        i = T0.clamp(tmin, tmax - 1)
        cp0, h0, _ = _nasa(m, i)
        cp1, h1, _ = _nasa(m, i + 1)
        scale = m.r_thermo / P.W
        a, b = (cp0 * scale, cp1 * scale) if col == 0 else (h0 * i[:, None] * scale, h1 * (i[:, None] + 1) * scale)
        return a + (b - a) * (T - T0)[:, None]

    rho = roi.sum(1)
    R = (ri * roi).sum(1) / rho
    u = cons[:, ns:ns + ndim] / rho[:, None]
    energy = cons[:, -1] / rho - 0.5 * (u * u).sum(1)
    t, diff = guess.clone(), torch.full_like(guess, 1e3)
    for _ in range(20):
        go = (diff / energy).abs() >= 1e-6
        e = (at(t, 1) * roi).sum(1) / rho - R * t
        cv = (at(t, 0) * roi).sum(1) / rho - R
        diff = torch.where(go, (e - energy).abs(), diff)
        t = torch.where(go, t + (energy - e) / cv, t)
    prim = torch.cat([roi, u, (rho * R * t)[:, None]], 1)

    # the rate constants between the two rows of the tables
    c = roi / P.W
    i = torch.floor(T)
    d = (T - i)[:, None]

    def lerp(f):
        a, b = f(i[:, None]), f(i[:, None] + 1)
        return a + (b - a) * d

    def inv_kc(t):
        _, h, s = _nasa(m, t[:, 0])
        return torch.exp((h - s) @ P.net.t() - P.net.sum(1) * torch.log(P.d["p_ref"] / (m.r_thermo * t)))

    def kf(t):
        return P.A * torch.exp(P.b * torch.log(t) - P.E / t)

    fall, third = (_t(x) > 0 for x in (P.type >= 2, P.type == 1))
    M = c @ P.eff.t()
    k, kr = lerp(kf), lerp(lambda t: kf(t) * inv_kc(t) * P.rev)
    k, kr = torch.where(third, k * M, k), torch.where(third, kr * M, kr)
    if (P.type >= 2).any():
        a, t3, t1, t2 = P.troe
        fc = lerp(lambda t: (1 - a) * torch.exp(-t / t3) + a * torch.exp(-t / t1) + torch.where(
            t2 != 0, torch.exp(-t2 / t), torch.zeros_like(t * a)))
        pr = torch.where(fall, lerp(lambda t: P.A0 * torch.exp(P.b0 * torch.log(t) - P.E0 / t)) / lerp(kf) * M, torch.ones_like(M))
        lf = torch.log10(fc)
        x = torch.log10(pr) - 0.4 - 0.67 * lf
        f1 = x / (0.75 - 1.27 * lf - 0.14 * x)
        F = torch.where(_t(P.type == 3) > 0, 10.0 ** (lf / (1 + f1 * f1)), torch.ones_like(lf))
        kk = lerp(kf) * pr / (1 + pr) * F
        kc = lerp(lambda t: (1.0 / inv_kc(t)).clamp(max=1e300))
        k, kr = torch.where(fall, kk, k), torch.where(fall, P.rev * kk / kc, kr)

    def power(side):
        out = None
        for idx, pw in P._slots(P.nu1 if side == 0 else P.nu2):
            x = torch.where(pw == 0, torch.ones_like(c[:, idx]), torch.where(pw == 1, c[:, idx], c[:, idx] ** pw))
            out = x if out is None else out * x
        return out

    w = ((k * power(0) - kr * power(1)) @ P.net) * P.W
    return prim, t, w


def exact(case, seed):
    kind, mech = case["kind"], case["mech"]
    if kind in ("reactor", "surrogate", "train"):
        return None   # integrated trajectories and mixed-precision networks: no value in 64 bits within seconds
    m, P, n = _load(mech), _Plain(mech), case["n"]
    if kind == "tables":
        roi, cons, guess, T = _cfd_state(m, mech, n, case["ndim"], seed)
        parts = [_exact_tables(case, P, roi[s], cons[s], guess[s], T[s]) for s in _chunks(n, 65536)]
        return [torch.cat(x) for x in zip(*parts)]
    T, p, Y = _states(m, mech, n, seed)
    if kind == "source":
        c = (_density(m, T, p, Y)[:, None] * Y).clamp(min=0.0) / P.W
        return torch.cat([P.rates(T[s], c[s]) * P.W for s in _chunks(n, 65536)])
    if kind == "rhs":
        return P.rhs(T, p, Y)
    w = torch.cat([P.rates(T[s], P.conc(T[s], p[s], Y[s])[1]) * P.W for s in _chunks(n, 65536)])
    wl = w.t().contiguous() if case.get("species_major") else w
    if kind == "wdot":
        if not case["thermo"]:
            return [wl]
        out = []
        for col in (0, 1):
            f = [((_nasa(P.m, T[s])[col] * (T[s][:, None] if col else 1.0) * P.m.r_thermo / P.W) * Y[s]).sum(1)
                 for s in _chunks(n, 262144)]
            out.append(torch.cat(f))
        return [wl] + out
    nv = P.ns + 1
    J = torch.empty(n, nv, nv, dtype=torch.float64, device="cuda")
    for s in _chunks(n, 32768):
        for col in range(nv):
            dT, dY = torch.zeros_like(T[s]), torch.zeros_like(Y[s])
            (dT if col == P.ns else dY[:, col]).fill_(1.0)
            J[s, col] = torch.func.jvp(lambda t, y: P.rhs(t, p[s], y), (T[s], Y[s]), (dT, dY))[1]
    return [wl, J]
