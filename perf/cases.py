"""The work that users of this framework have it do, as cases that can be timed and checked.

Every case goes through a public entry point: the plugin's `computeRR` on host
arrays, the device-tensor `Solver.solve` (one mechanism, or several in one
launch), a gradient through `ChemistryStep`, and the plugin's per-cell side
paths (`jacobian`, `cell_rates`, `gather_states` / `scatter_rates` / `qdot`).
Mechanisms and batches are the seeded synthetic ones of
`gpufoam_b200.mechanism` (10, 53 and 100 species); sizes and temperature, time
step and pressure ranges are those of the benchmark and the tests.

`exact` restates the chemistry in plain torch, in 64 bits.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from gpufoam_b200 import adjoint as AD
from gpufoam_b200 import evaluator as E
from gpufoam_b200 import flops
from gpufoam_b200 import mechanism as M

ABS_TOL, REL_TOL, DTC0 = 1e-8, 1e-4, 1e-7
P_ATM = 101325.0
MECHS = {"h2": M.h2_size, "gri": M.gri_size, "large": M.large}
# mean attempted substeps per cell over the batches below (for work())
ATTEMPTS = {"h2": 39.0, "gri": 53.0, "large": 26.0}
# the launch form that the autotuner picks for the 53-species batches
TUNED = dict(kind=1, threads_per_cell=128, scratch_in_shared=1, register_budget=1, lu_panel=4, specialize=1)
# and the one for launches that mix mechanisms
WIDE = dict(kind=1, threads_per_cell=256, scratch_in_shared=1)


@functools.lru_cache(maxsize=None)
def raw_mechanism(name):
    return MECHS[name](0)


def listed():
    return [
        # a small case's flow step through the plugin's entry point: 1,024 cells of a hydrogen-size mechanism
        dict(name="rr-h2-1k", kind="rr", mech="h2", n=1024, solver=34, dT=1e-5, batch="hot"),
        # an MPI rank's share of a flame: 1,500 cells, 40 % of them cold, host arrays in and out
        dict(name="rr-gri-1500", kind="rr", mech="gri", n=1500, solver=34, dT=1e-6, batch="bimodal"),
        # the headline batch (cold and igniting cells of the 53-species mechanism), in the autotuner's form
        dict(name="solve-gri-64k", kind="solve", mech="gri", n=65536, solver=34, dT=1e-6, batch="bimodal", form="tuned"),
        # the same mechanism with Rosenbrock23, every cell reacting, as a user gets it without tuning
        dict(name="solve-gri-r23-6k", kind="solve", mech="gri", n=6007, solver=23, dT=1e-6, batch="hot", form="default"),
        # many cells of a small mechanism
        dict(name="solve-h2-100k", kind="solve", mech="h2", n=100003, solver=34, dT=1e-5, batch="hot", form="default"),
        # few cells of a large mechanism (100 species)
        dict(name="solve-large-701", kind="solve", mech="large", n=701, solver=34, dT=1e-6, batch="hot", form="default"),
        # three mechanisms in one launch, a time step and a pressure per cell
        dict(name="solve-mixed-2k", kind="mixed", mech="gri", n=2250, solver=34, dT=1e-5, batch="hot", form="wide"),
        # a gradient step of training on the small mechanism: integration, then the adjoint sweep
        dict(name="grad-h2-2k", kind="grad", mech="h2", n=2048, solver=34, dT=1e-5, batch="ignition"),
        # and on the 53-species mechanism (Rosenbrock34, through the first part of ignition)
        dict(name="grad-gri-600", kind="grad", mech="gri", n=600, solver=34, dT=1e-5, batch="ignition"),
        # the system's derivatives and Jacobian at given states (analysis, timescale and sensitivity tools)
        dict(name="jacobian-gri-4k", kind="jacobian", mech="gri", n=4096, batch="hot"),
        # the plugin's calculate() and tc() on a whole field
        dict(name="cell-rates-gri-60k", kind="cell_rates", mech="gri", n=60000, batch="bimodal"),
        # the copies around a flow step on device fields: states gathered, rates scattered, heat release
        dict(name="fields-gri-500k", kind="fields", mech="gri", n=500000, batch="hot"),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["rr", "solve", "solve", "solve", "mixed", "grad", "jacobian", "cell_rates", "fields"])
    mech = rng.choice(["h2", "gri", "gri", "large"])
    case = dict(kind=kind, mech=mech, n=1, batch=rng.choice(["hot", "bimodal"]))
    if kind in ("rr", "solve"):
        # bounded by the largest listed case's cost: a cell costs some 1 : 30 : 400
        lo, hi = {"h2": (100, 100003), "gri": (64, 20000), "large": (32, 1000)}[mech]
        solver = rng.choice([12, 23, 34, 34]) if mech == "h2" else rng.choice([23, 34, 34])
        # Rosenbrock12 takes some 15 times the steps
        case.update(n=_log_int(rng, lo, hi if solver != 12 else 6000), solver=solver, dT=1e-5 if mech == "h2" else 1e-6)
        if kind == "solve":
            case["form"] = rng.choice(["tuned", "default"]) if mech == "gri" else "default"
    elif kind == "mixed":
        case.update(mech="gri", n=_log_int(rng, 150, 2250), solver=34, dT=1e-5, batch="hot", form=rng.choice(["wide", "default"]))
    elif kind == "grad":
        case.update(mech=rng.choice(["h2", "gri"]), solver=rng.choice([23, 34, 34]), dT=1e-5, batch="ignition")
        case["n"] = _log_int(rng, 64, 4096) if case["mech"] == "h2" else _log_int(rng, 32, 600)
    elif kind == "jacobian":
        case["n"] = _log_int(rng, 100, {"h2": 60000, "gri": 4096, "large": 1200}[mech])
    elif kind == "cell_rates":
        case["n"] = _log_int(rng, 300, {"h2": 300000, "gri": 60000, "large": 30000}[mech])
    else:
        case["n"] = _log_int(rng, 5000, {"h2": 2000000, "gri": 500000, "large": 250000}[mech])
    return case


# ---------------------------------------------------------------- inputs

def cell_states(raw, n, batch, gen, p=None):
    """[n][nS + 2] states (Y, T, p) on the GPU: Y ~ Dirichlet(0.5), T over the
    batch's range; "bimodal": 40 % cold cells, nearly inert."""
    nS = raw.n_species
    rnd = lambda k: torch.rand(k, dtype=torch.float64, device="cuda", generator=gen)  # noqa: E731
    # a gamma(1/2) variate is half the square of a normal one
    Y = torch.randn((n, nS), dtype=torch.float64, device="cuda", generator=gen).square_().add_(1e-300)
    Y /= Y.sum(dim=1, keepdim=True)
    u = rnd(n)
    if batch == "bimodal":
        cold = rnd(n) < 0.4
        T = torch.where(cold, 300.0 + 400.0 * u, 1100.0 + 1300.0 * u)
        Y = torch.where(cold[:, None], Y * 1e-4, Y)
        Y[:, nS - 1] += torch.where(cold, 1.0 - 1e-4, 0.0)
    elif batch == "ignition":
        T = 1100.0 + 500.0 * u
    else:
        T = 1000.0 + 1500.0 * u
    out = torch.empty((n, nS + 2), dtype=torch.float64, device="cuda")
    out[:, :nS] = Y
    out[:, nS] = T
    out[:, nS + 1] = P_ATM if p is None else p
    return out


def mixed_shares(n):
    n_h2, n_large = max(1, n * 4 // 15), max(1, n // 15)
    return [("h2", n_h2), ("gri", n - n_h2 - n_large), ("large", n_large)]


def inputs(case, seed):
    """The case's tensors, from the seed alone."""
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    rnd = lambda k: torch.rand(k, dtype=torch.float64, device="cuda", generator=gen)  # noqa: E731
    n = case["n"]
    if case["kind"] == "mixed":
        shares = mixed_shares(n)
        ld = max(raw_mechanism(m).n_eqns for m, _ in shares)
        Y = torch.zeros((n, ld), dtype=torch.float64, device="cuda")
        mech_id = torch.empty(n, dtype=torch.int32, device="cuda")
        o = 0
        for k, (name, cnt) in enumerate(shares):
            raw = raw_mechanism(name)
            Y[o:o + cnt, :raw.n_eqns] = cell_states(raw, cnt, case["batch"], gen, P_ATM * (0.5 + 39.5 * rnd(cnt)))
            mech_id[o:o + cnt] = k
            o += cnt
        order = torch.randperm(n, device="cuda", generator=gen)
        dt = torch.exp(math.log(1e-7) + math.log(case["dT"] / 1e-7) * rnd(n))
        return dict(Y0=Y[order].contiguous(), mech_id=mech_id[order].contiguous(), deltaT_cell=dt,
                    dtc0=torch.full((n,), DTC0, dtype=torch.float64, device="cuda"))
    raw = raw_mechanism(case["mech"])
    out = dict(Y0=cell_states(raw, n, case["batch"], gen), rho=0.2 + rnd(n),
               dtc0=torch.full((n,), DTC0, dtype=torch.float64, device="cuda"))
    if case["kind"] == "grad":
        w = torch.randn((n, raw.n_eqns), dtype=torch.float64, device="cuda", generator=gen)
        w[:, raw.n_species] *= 1e-3  # kelvins against mass fractions
        w[:, raw.n_species + 1] = 0.0
        out["weights"] = w
    if case["kind"] == "fields":
        out["RR"] = torch.randn((n, raw.n_species), dtype=torch.float64, device="cuda", generator=gen)
    return out


def dtc_max(case):
    """The plugin's maxChemicalTimeStep: a tenth of the flow step (the largest one, where each cell has its own)."""
    return 0.1 * case["dT"]


def ode_inputs(case):
    return E.OdeInputs(f"Rosenbrock{case['solver']}", absTol=ABS_TOL, relTol=REL_TOL)


def prepare(case, seed):
    kind = case["kind"]
    x = inputs(case, seed)
    st = dict(case=case, **x)
    if kind == "mixed":
        st["mechs"] = [E.Mechanism(raw_mechanism(m)) for m, _ in mixed_shares(case["n"])]
    else:
        raw = raw_mechanism(case["mech"])
        if kind == "grad":
            st["solver"] = AD.AdjointSolver(raw, ode_inputs(case), traj_cap=512)
            st["theta"] = torch.tensor(st["solver"].parameters(), requires_grad=True)
            st["Y0"].requires_grad_(True)
            return st
        st["mechs"] = [E.Mechanism(raw)]
    if kind == "rr":
        # the plugin holds host arrays
        raw = raw_mechanism(case["mech"])
        st["evaluator"] = E.GpuKernelEvaluator(case["n"], raw.n_eqns, raw.n_species, st["mechs"][0], ode_inputs(case))
        st["host"] = [st[k].cpu().numpy() for k in ("rho", "dtc0", "Y0")]
    elif kind in ("solve", "mixed"):
        st["solver"] = E.Solver(st["mechs"], ode_inputs(case))
        if case["form"] != "default":
            st["solver"].set_launch(**(TUNED if case["form"] == "tuned" else WIDE))
    elif kind == "fields":
        raw = raw_mechanism(case["mech"])
        cols = st["Y0"].t().contiguous()
        st["fields"] = [cols[i] for i in range(raw.n_species)]
        st["T"], st["p"] = cols[raw.n_species], cols[raw.n_species + 1]
        out = torch.empty((raw.n_species, case["n"]), dtype=torch.float64, device="cuda")
        st["RR_fields"] = [out[i] for i in range(raw.n_species)]
        st["out"] = out
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "rr":
        rho, dtc, Y = st["host"]
        RR, dtn, mn = st["evaluator"].computeRR(case["dT"], dtc_max(case), rho, dtc, Y)
        return dict(RR=RR, deltaTChem=dtn, minDeltaT=mn)
    if kind == "solve":
        RR = torch.empty((case["n"], st["Y0"].shape[1] - 2), dtype=torch.float64, device="cuda")
        out = st["solver"].solve(st["Y0"], case["dT"], st["dtc0"].clone(), dtc_max(case), rho=st["rho"], RR=RR)
        return {k: out[k] for k in ("Ynew", "RR", "deltaTChem", "status", "counters")}
    if kind == "mixed":
        out = st["solver"].solve(st["Y0"], 0.0, st["dtc0"].clone(), dtc_max(case), deltaT_cell=st["deltaT_cell"],
                                 mech_id=st["mech_id"], Ynew=torch.zeros_like(st["Y0"]))
        return {k: out[k] for k in ("Ynew", "deltaTChem", "status", "counters")}
    if kind == "grad":
        Y1 = AD.ChemistryStep.apply(st["Y0"], st["theta"], st["solver"], case["dT"], DTC0)
        gY, gt = torch.autograd.grad((st["weights"] * Y1).sum(), [st["Y0"], st["theta"]])
        return dict(Ynew=Y1.detach(), dY0=gY, dtheta=gt)
    if kind == "jacobian":
        dfdx, J = E.jacobian(st["mechs"][0], st["Y0"])
        return dict(dfdx=dfdx, J=J)
    if kind == "cell_rates":
        RR, tc = E.cell_rates(st["mechs"][0], st["rho"], st["Y0"])
        return dict(RR=RR, tc=tc)
    y = E.gather_states(st["fields"], st["T"], st["p"])
    E.scatter_rates(st["RR"], st["RR_fields"])
    return dict(y=y, RR_fields=st["out"], Qdot=E.qdot(st["mechs"][0], st["RR"]))


def work(case):
    kind, n = case["kind"], case["n"]
    if kind == "mixed":
        parts = [work(dict(case, kind="solve", mech=m, n=k)) for m, k in mixed_shares(n)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    raw = raw_mechanism(case["mech"])
    nS, ne = raw.n_species, raw.n_eqns
    if kind in ("rr", "solve", "grad"):
        f_att, f_rhs = flops.model(raw, case["solver"])
        att = ATTEMPTS[case["mech"]] * {12: 15.0, 23: 1.7, 34: 1.0}[case["solver"]] * (0.64 if case["batch"] == "bimodal" else 1.0)
        # a gradient: the integration, the steps again, and twice a step's work for its reverse
        per = att * (f_att + f_rhs) * (4.0 if kind == "grad" else 1.0)
        return {"bytes": n * 8.0 * (2 * ne + nS + 4) * (2.0 if kind == "grad" else 1.0), "flops": n * per}
    if kind == "jacobian":
        f_att, f_rhs = flops.model(raw, 34)
        return {"bytes": n * 8.0 * (2 * ne + ne * ne), "flops": n * (f_att - 2.0 * ne ** 3 / 3.0 - 8.0 * ne * ne - 2 * f_rhs)}
    if kind == "cell_rates":
        return {"bytes": n * 8.0 * (ne + 1 + nS + 1), "flops": n * flops.model(raw, 34)[1]}
    # states gathered and rates scattered (read and written once each), heat release from the rates
    return {"bytes": n * 8.0 * (2 * ne + 2 * nS + nS + 1), "flops": n * 2.0 * nS}


# ---------------------------------------------------------------- the same in plain torch, 64 bits

RR_GAS, P_STD, SMALL = 6.02214e+26 * 1.38065e-23, 1e5, 2.220446049250313e-16
LN_K_MAX = 0.5 * math.log(1.7976931348623157e+308 / 10.0)


class Chemistry:
    """The mechanism's equations over a batch of states, from the raw mechanism."""

    def __init__(self, raw):
        self.raw = raw
        dev = dict(dtype=torch.float64, device="cuda")
        nS, nR = raw.n_species, raw.n_reactions
        self.nS, self.nR = nS, nR
        t = lambda a: torch.as_tensor(np.asarray(a, dtype=np.float64), **dev)  # noqa: E731
        self.W = t(raw.W)
        self.Rs = RR_GAS / self.W
        self.Tc = t(raw.Tcommon)
        self.lo, self.hi = t(raw.low_raw) * self.Rs[:, None], t(raw.high_raw) * self.Rs[:, None]
        rx = raw.reactions
        self.width = max(max(len(r.lhs), len(r.rhs)) for r in rx)
        idx = np.full((2, nR, self.width), nS, dtype=np.int64)  # nS: a concentration of 1
        ex = np.zeros((2, nR, self.width))
        nu = np.zeros((nR, nS))
        for q, r in enumerate(rx):
            for s, side in enumerate((r.lhs, r.rhs)):
                for e, (i, st, x) in enumerate(side):
                    idx[s, q, e], ex[s, q, e] = i, x
                    nu[q, i] += st if s else -st
        self.idx = torch.as_tensor(idx, device="cuda")
        self.ex, self.nu = t(ex), t(nu)
        self.theta = t(AD.parameters_of(raw))
        self.sign = t([np.sign(r.A) for r in rx])
        self.inf = t([[math.log(r.Ainf) if r.Ainf > 0 else 0.0, r.betainf, r.Tainf] for r in rx])
        self.troe = t([r.troe for r in rx])
        kind = np.array([r.rate_type for r in rx])
        self.is_tb, self.is_fall = (torch.as_tensor(v, device="cuda") for v in (kind == 1, kind >= 2))
        self.is_troe = torch.as_tensor(kind == 3, device="cuda")
        self.eff = t([r.efficiencies if r.efficiencies is not None else np.zeros(nS) for r in rx])
        self.rev = t([0.0 if r.irreversible else 1.0 for r in rx])

    def mixture(self, Y, T, p):
        Yp = Y.clamp_min(0.0)
        v = self.Rs * T[:, None] / p[:, None]  # 1 / rho_i
        rhoM = 1.0 / (Yp * v).sum(1)
        a = torch.where((T[:, None] < self.Tc)[:, :, None], self.lo, self.hi)
        t = T[:, None]
        Cp = (((a[..., 4] * t + a[..., 3]) * t + a[..., 2]) * t + a[..., 1]) * t + a[..., 0]
        Ha = ((((a[..., 4] / 5 * t + a[..., 3] / 4) * t + a[..., 2] / 3) * t + a[..., 1] / 2) * t + a[..., 0]) * t + a[..., 5]
        dCp = ((4 * a[..., 4] * t + 3 * a[..., 3]) * t + 2 * a[..., 2]) * t + a[..., 1]
        G = Ha - t * ((((a[..., 4] / 4 * t + a[..., 3] / 3) * t + a[..., 2] / 2) * t + a[..., 1]) * t
                      + a[..., 0] * t.log() + a[..., 6])
        return dict(Y=Yp, v=v, rhoM=rhoM, Cp=Cp, Ha=Ha, dCp=dCp, G=G, c=rhoM[:, None] * Yp / self.W, T=T)

    def powers(self, c, side):
        """c_e^x_e of a side's entries and x_e c_e^(x_e - 1), [n][nR][width]."""
        cp = torch.cat([c, torch.ones_like(c[:, :1])], 1)[:, self.idx[side]]
        x = self.ex[side]
        one = x == 1.0
        two = x == 2.0
        pw = torch.where(one, cp, torch.where(two, cp * cp, cp ** torch.where(one | two, 0.0, x)))
        d = torch.where(one, 1.0, torch.where(two, 2.0 * cp, x * cp ** torch.where(one | two, 1.0, x - 1.0)))
        return pw, d

    def rates(self, c, T, G, theta):
        """kf, kr, 1/Kc, dkf/dT (the reference's form) and the pure Arrhenius part, [n][nR]."""
        t, it, lt = T[:, None], 1.0 / T[:, None], T.log()[:, None]
        k0 = self.sign * torch.exp(theta[:, 0] + theta[:, 1] * lt - theta[:, 2] * it)
        dln0 = (theta[:, 1] + theta[:, 2] * it) * it
        Mc = c @ self.eff.T
        kI = torch.exp(self.inf[:, 0] + self.inf[:, 1] * lt - self.inf[:, 2] * it)
        dlnI = (self.inf[:, 1] + self.inf[:, 2] * it) * it
        Pr = k0 / kI * Mc
        al, t3, t1, t2 = self.troe.T
        Fc = (1 - al) * torch.exp(-t / t3) + al * torch.exp(-t / t1) + torch.exp(-t2 * it)
        lP, lF = torch.log10(Pr.clamp_min(SMALL)), torch.log10(Fc.clamp_min(SMALL))
        cc, n = -0.4 - 0.67 * lF, 0.75 - 1.27 * lF
        F = 10.0 ** (lF / (1 + ((lP + cc) / (n - 0.14 * (lP + cc))) ** 2))
        shape = Pr / (1 + Pr) * torch.where(self.is_troe, F, 1.0)
        kf = torch.where(self.is_fall, kI * shape, torch.where(self.is_tb, Mc * k0, k0))
        dk = torch.where(self.is_fall, kI * dlnI * shape, kf * dln0)
        dG = (G * self.W) @ self.nu.T
        arg = -dG * it / RR_GAS
        nm = self.nu.sum(1)
        lnKc = torch.where(arg < 600, arg, LN_K_MAX) + nm * torch.log(P_STD / (RR_GAS * t))
        iK = torch.exp(-lnKc)
        return kf, self.rev * kf * iK, iK, dk, k0

    def rhs(self, Y, T, p, theta=None):
        theta = self.theta if theta is None else theta
        m = self.mixture(Y, T, p)
        kf, kr, *_ = self.rates(m["c"], T, m["G"], theta)
        w = kf * self.powers(m["c"], 0)[0].prod(2) - kr * self.powers(m["c"], 1)[0].prod(2)
        dY = (w @ self.nu) * self.W / m["rhoM"][:, None]
        return torch.cat([dY, (-(dY * m["Ha"]).sum(1) / (m["Y"] * m["Cp"]).sum(1))[:, None]], 1)

    def jacobian(self, Y, T, p, theta=None):
        """f and the (nS + 1)^2 Jacobian as the reference defines it."""
        theta = self.theta if theta is None else theta
        nS, n = self.nS, Y.shape[0]
        m = self.mixture(Y, T, p)
        c, rhoM, W = m["c"], m["rhoM"][:, None], self.W
        kf, kr, iK, dk, k0 = self.rates(c, T, m["G"], theta)
        H = (m["Ha"] * W) @ self.nu.T  # reaction enthalpy: dlnKc/dT = H / (R T^2) - nm / T
        it = 1.0 / T[:, None]
        dlnK = H * it * it / RR_GAS - self.nu.sum(1) * it
        dkr = self.rev * (dk * iK - kr * dlnK)
        C = []
        terms, cols, rxn = [], [], []
        for side, k in ((0, kf), (1, -kr)):
            pw, d = self.powers(c, side)
            C.append(pw.prod(2))
            for j in range(self.width):
                prod = d[:, :, j]
                for i in range(self.width):
                    if i != j:
                        prod = prod * pw[:, :, i]
                real = self.idx[side, :, j] < nS
                terms.append((prod * k)[:, real])
                cols.append(self.idx[side, real, j])
                rxn.append(torch.nonzero(real)[:, 0])
        terms, cols, rxn = torch.cat(terms, 1), torch.cat(cols), torch.cat(rxn)
        # D[r][col] = d omega_r / d c_col, then raw = nu^T D
        D = torch.zeros((n, self.nR * nS), dtype=torch.float64, device="cuda").index_add(1, rxn * nS + cols, terms)
        D = D.view(n, self.nR, nS)
        phi = k0 * (C[0] - self.rev * C[1] * iK)
        D = D + torch.where(self.is_tb, phi, 0.0)[:, :, None] * self.eff
        raw = torch.einsum("rs,nrc->nsc", self.nu, D)
        rT = (C[0] * dk - C[1] * dkr) @ self.nu
        w = kf * C[0] - kr * C[1]
        dY = (w @ self.nu) * W / rhoM
        CpM = (m["Y"] * m["Cp"]).sum(1)
        dT = -(dY * m["Ha"]).sum(1) / CpM
        av = ((m["Y"] * m["v"]).sum(1) / T)[:, None] * rhoM
        Wr = (W / rhoM)[:, :, None]
        JYY = Wr * raw * (rhoM / W)[:, None, :] + (rhoM * m["v"])[:, None, :] * dY[:, :, None]
        JYT = (W / rhoM) * (rT - av * (raw * c[:, None, :]).sum(2)) + av * dY
        JTY = (-(JYY * m["Ha"][:, :, None]).sum(1) - m["Cp"] * dT[:, None]) / CpM[:, None]
        JTT = (-(dY * m["Cp"] + JYT * m["Ha"]).sum(1) - dT * (m["Y"] * m["dCp"]).sum(1)) / CpM
        J = torch.cat([torch.cat([JYY, JYT[:, :, None]], 2), torch.cat([JTY, JTT[:, None]], 1)[:, None, :]], 1)
        return torch.cat([dY, dT[:, None]], 1), J


def _method(solver):
    """gamma, a, c, b, e, d of Rosenbrock12, 23 and 34."""
    if solver == 12:
        g = 1.0 + 1.0 / 1.414213562373095
        return g, [[], [1 / g]], [[], [-2 / g]], [1.5 / g, 0.5 / g], [1.5 / g - 1 / g, 0.5 / g], [g, -g], [1]
    if solver == 23:
        g = 0.43586652150845899941601945119356
        return (g, [[], [1.0], [1.0, 0.0]],
                [[], [-1.0156171083877702091975600115545], [4.0759956452537699824805835358067, 9.2076794298330791242156818474003]],
                [1.0, 6.1697947043828245592553615689730, -0.4277225654321857332623837380651],
                [0.5, -2.9079558716805469821718236208017, 0.2235406989781156962736090927619],
                [g, 0.24291996454816804366592249683314, 2.1851380027664058511513169485832], [1])
    return (0.5, [[], [2.0], [48 / 25, 6 / 25]], [[], [-8.0], [372 / 25, 12 / 5], [-112 / 125, -54 / 125, -2 / 5]],
            [19 / 9, 0.5, 25 / 108, 125 / 108], [34 / 108, 7 / 36, 0.0, 125 / 108], [0.5, -1.5, 605 / 250, 29 / 250], [1, 2])


def _attempt(chem, y, p, h, solver, theta=None):
    g, a, c, b, e, d, fresh = _method(solver)
    nS = chem.nS
    dfdx, J = chem.jacobian(y[:, :nS], y[:, nS], p, theta)
    A = torch.eye(nS + 1, dtype=torch.float64, device="cuda") / (g * h)[:, None, None] - J
    f, ks = dfdx, []
    LU = torch.linalg.lu_factor(A)
    for i in range(len(b)):
        if i in fresh:
            z = y + sum(aij * k for aij, k in zip(a[i], ks))
            f = chem.rhs(z[:, :nS], z[:, nS], p, theta)
        r = f + (h * d[i])[:, None] * dfdx
        if i:
            r = r + sum(cij * k for cij, k in zip(c[i], ks)) / h[:, None]
        ks.append(torch.linalg.lu_solve(*LU, r[:, :, None])[:, :, 0])
    yn = y + sum(bi * k for bi, k in zip(b, ks))
    err = sum(ei * k for ei, k in zip(e, ks)).abs() / (ABS_TOL + REL_TOL * torch.maximum(y.abs(), yn.abs()))
    return yn, err.detach().amax(1)


def _integrate(chem, cells, dT, dtc0, solver, steps=None):
    """One flow step of every cell: (Ynew, deltaTChem, [accepted, attempts]); with
    `steps`, a list that receives each attempt's (cells, states, sizes) that was accepted."""
    nS, n = chem.nS, cells.shape[0]
    y, p = cells[:, :nS + 1].clone(), cells[:, nS + 1]
    x, dtc = torch.zeros_like(dT), dtc0.clone()
    step, h = dtc0.clone(), dtc0.clone()
    last = torch.zeros(n, dtype=torch.bool, device="cuda")
    count = torch.zeros((n, 2), dtype=torch.int32, device="cuda")
    fresh, live = torch.ones_like(last), torch.ones_like(last)
    before = step.clone()
    floor = (10.0 / 0.9) ** (-1.0 / 0.2)
    while bool(live.any()):
        start = live & fresh
        before = torch.where(start, step, before)
        cut = start & ((x + step - dT) * (x + step) > 0)
        last |= cut
        h = torch.where(cut, dT - x, torch.where(start, step, h))
        i = torch.nonzero(live)[:, 0]
        yn, err = _attempt(chem, y[i], p[i], h[i], solver)
        count[i, 1] += 1
        bad = err > 1
        h[i] = torch.where(bad, h[i] * torch.clamp_min(0.9 * err ** -0.25, 0.2), h[i])
        fresh[i] = ~bad
        j, ok = i[~bad], ~bad
        if steps is not None:
            steps.append((j, y[j].clone(), h[j].clone()))
        x[j] += h[j]
        y[j] = yn[ok]
        count[j, 0] += 1
        grow = torch.where(err[ok] > floor, (0.9 * err[ok].clamp_min(1e-300) ** -0.2).clamp(0.2, 10.0), 9.0)
        step[j] = grow * h[j]
        done = torch.zeros_like(live)
        done[j] = (x[j] - dT[j]) * dT[j] >= 0
        dtc = torch.where(done, torch.where(last & (count[:, 0] > 1), before, step), dtc)
        live &= ~done
    out = cells.clone()
    out[:, :nS] = y[:, :nS].clamp_min(0.0)
    out[:, nS] = y[:, nS]
    return out, dtc, count


def _gradient(chem, x, case):
    """The recorded steps in reverse, each differentiated by autograd."""
    nS, n = chem.nS, case["n"]
    cells, w = x["Y0"], x["weights"]
    steps = []
    dT = torch.full((n,), case["dT"], dtype=torch.float64, device="cuda")
    Y1, _, _ = _integrate(chem, cells, dT, x["dtc0"], case["solver"], steps)
    bar = torch.where((Y1[:, :nS + 1] > 0) | (torch.arange(nS + 1, device="cuda") == nS), w[:, :nS + 1], 0.0)
    theta_bar = torch.zeros_like(chem.theta)
    for j, y, h in reversed(steps):
        if j.numel() == 0:
            continue
        y = y.requires_grad_(True)
        th = chem.theta.clone().requires_grad_(True)
        yn, _ = _attempt(chem, y, cells[j, nS + 1], h, case["solver"], th)
        gy, gt = torch.autograd.grad((bar[j] * yn).sum(), [y, th])
        bar[j] = gy
        theta_bar += gt
    full = torch.zeros_like(cells)
    full[:, :nS + 1] = bar
    return dict(Ynew=Y1, dY0=full, dtheta=theta_bar)


def exact(case, seed):
    kind, n = case["kind"], case["n"]
    if kind == "mixed":
        return None  # cells that take 1 to some hundred substeps, three mechanisms: minutes
    raw = raw_mechanism(case["mech"])
    nS = raw.n_species
    # a lockstep integration in torch within some 20 seconds
    if kind in ("rr", "solve", "grad"):
        if n * (nS + 1) ** 2 > 6e6 * (0.3 if kind == "grad" else 1.0) or case["solver"] == 12:
            return None
    chem, x = Chemistry(raw), inputs(case, seed)
    Y0 = x["Y0"]
    if kind in ("rr", "solve"):
        dT = torch.full((n,), case["dT"], dtype=torch.float64, device="cuda")
        Yn, dtc, count = _integrate(chem, Y0, dT, x["dtc0"], case["solver"])
        RR = x["rho"][:, None] * (Yn[:, :nS] - Y0[:, :nS]) / case["dT"]
        if kind == "rr":
            return dict(RR=RR.reshape(-1), deltaTChem=dtc.clamp_max(dtc_max(case)), minDeltaT=float(dtc.min()))
        return dict(Ynew=Yn, RR=RR, deltaTChem=dtc.clamp_max(dtc_max(case)), status=torch.zeros(n, dtype=torch.int32), counters=count)
    if kind == "grad":
        return _gradient(chem, x, case)
    if kind == "jacobian":
        dfdx = torch.zeros((n, nS + 2), dtype=torch.float64, device="cuda")
        J = torch.zeros((n, nS + 2, nS + 2), dtype=torch.float64, device="cuda")
        for o in range(0, n, 1024):
            s = slice(o, min(n, o + 1024))
            dfdx[s, :nS + 1], J[s, :nS + 1, :nS + 1] = chem.jacobian(Y0[s, :nS], Y0[s, nS], Y0[s, nS + 1])
        return dict(dfdx=dfdx, J=J)
    if kind == "cell_rates":
        RR, tc = [], []
        for o in range(0, n, 8192):
            s = slice(o, min(n, o + 8192))
            c, T = x["rho"][s, None] * Y0[s, :nS] / chem.W, Y0[s, nS]
            kf, kr, *_ = chem.rates(c, T, chem.mixture(Y0[s, :nS], T, Y0[s, nS + 1])["G"], chem.theta)
            wf, wr = kf * chem.powers(c, 0)[0].prod(2), kr * chem.powers(c, 1)[0].prod(2)
            RR.append(((wf - wr) @ chem.nu) * chem.W)
            lhs = torch.tensor([sum(st for _, st, _ in r.lhs) for r in raw.reactions], dtype=torch.float64, device="cuda")
            rhs = torch.tensor([sum(st for _, st, _ in r.rhs) for r in raw.reactions], dtype=torch.float64, device="cuda")
            a, b = wf * rhs, wr * lhs
            tc.append((a + b).sum(1) / (a * a + b * b).sum(1) * c.sum(1))
        return dict(RR=torch.cat(RR), tc=torch.cat(tc))
    Ts = 298.15
    a = chem.lo
    hf = ((((a[:, 4] / 5 * Ts + a[:, 3] / 4) * Ts + a[:, 2] / 3) * Ts + a[:, 1] / 2) * Ts + a[:, 0]) * Ts + a[:, 5]
    return dict(y=Y0, RR_fields=x["RR"].t().contiguous(), Qdot=-(x["RR"] @ hf))
