"""Performance cases of the chemistry library: what a flow solver has it do.

A flow solver calls the batched integration once per CFD step (``fcs_integrate``
through ``fcs._lib.Context``), the source terms (``fcs_rates``) where the model
calls ``calculate()``/``Qdot()``, an implicit coupling the analytic Jacobian
(``fcs_jacobian``), and the surrogate its ensemble forward and its training
gradients.  The cases run those entry points on the mechanisms of the golden
fixtures (10 to 200 species), with two kinds of cell states:

* ``first``: the first CFD step from the workloads' seeded initial fields, far
  from equilibrium, initial sub-step 1e-7 (some hundred attempted steps a cell);
* ``next``: a later CFD step: the fixtures' states after one step with the
  sub-steps they ended with, each mixed with a little of another cell's state
  as transport does between two chemistry steps.

``exact`` restates rates, right-hand side, Jacobian (by automatic
differentiation), the Rodas34 step and the network in 64-bit torch.
"""
import functools
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "fastchemistrysolver-openfoam-10_gb300"))

from fcs import _lib  # noqa: E402
from fcs.mechanism import FlatMechanism  # noqa: E402

RU, PSTD = 8314.470066505449722171761095523834228515625, 1e5

# fixture, CFD step, Treact, and the measured mean attempted steps per cell of
# a first and of a later step (for work())
FAMILIES = {
    "ignition": ("ignition_10s_OptRodas34", 1e-5, 0.0, 80, 8),
    "falloff": ("falloff_16s_OptRodas34", 1e-5, 0.0, 140, 12),
    "counterflow": ("counterflow_53s_OptRodas34", 1e-6, 0.0, 256, 27),
    "uneven": ("uneven_111s_OptRodas34", 5e-6, 700.0, 230, 18),
    "large": ("large_200s_OptRodas34", 1e-5, 0.0, 250, 27),
}
MLP = {"width": 256, "depth": 4, "members": 4}


def listed():
    step = {"op": "step", "solver": "OptRodas34", "precision": "fp64", "arrays": "device", "graph": False, "lts": False}
    return [
        # the smallest call: a handful of reactor cells over host arrays, as the OpenFOAM plugin makes it
        {"name": "reactor", **step, "family": "ignition", "state": "first", "cells": 100, "arrays": "host"},
        # a large field of a small mechanism, the step as one graph
        {"name": "ignition field", **step, "family": "ignition", "state": "first", "cells": 65536, "graph": True},
        # a small mechanism with every fall-off kind, the extrapolation method
        {"name": "falloff seulex", **step, "family": "falloff", "state": "first", "cells": 513, "solver": "OptSeulex"},
        # start-up of a flame on one rank's share of the field
        {"name": "flame start", **step, "family": "counterflow", "state": "first", "cells": 1500},
        # a later step of the same flame: the common call of a long run
        {"name": "flame", **step, "family": "counterflow", "state": "next", "cells": 12001},
        # the same, local time stepping in mixed precision on a small share
        {"name": "flame mixed lts", **step, "family": "counterflow", "state": "next", "cells": 1000,
         "precision": "mixed", "lts": True},
        # a later step of a large field
        {"name": "flame field", **step, "family": "counterflow", "state": "next", "cells": 44801, "graph": True},
        # 111 species, two fifths of the cells below Treact
        {"name": "uneven", **step, "family": "uneven", "state": "next", "cells": 2000},
        # 200 species: a cell's working set exceeds shared memory
        {"name": "large", **step, "family": "large", "state": "next", "cells": 150},
        # source terms of a whole field
        {"name": "rates", "op": "rates", "family": "counterflow", "cells": 65536},
        # analytic Jacobians of 111 species
        {"name": "jacobian", "op": "jacobian", "family": "uneven", "cells": 2001},
        # the surrogate over a field (every member), and a training batch's gradients
        {"name": "surrogate", "op": "forward", "family": "counterflow", "cells": 65536},
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    op = rng.choice(["step", "step", "step", "step", "rates", "jacobian", "forward", "gradients"])
    if op == "forward":
        return {"op": op, "family": rng.choice(["ignition", "counterflow", "uneven"]), "cells": size(100, 65536)}
    if op == "gradients":
        return {"op": op, "family": rng.choice(["ignition", "counterflow", "uneven"]), "cells": 128 * size(1, 64)}
    if op == "rates":
        return {"op": op, "family": rng.choice(["ignition", "counterflow", "uneven"]), "cells": size(100, 65536)}
    if op == "jacobian":
        return {"op": op, "family": rng.choice(["ignition", "counterflow", "uneven"]), "cells": size(20, 2000)}
    family, state, lo, hi = rng.choice([
        ("ignition", "first", 64, 65536), ("ignition", "next", 1000, 65536), ("falloff", "first", 64, 2000),
        ("counterflow", "first", 50, 1500), ("counterflow", "next", 500, 24000), ("uneven", "next", 64, 2000),
        ("large", "next", 16, 150)])
    cells = size(lo, hi)
    # the other solvers and mixed precision on the sizes where one step stays under two seconds
    small = state == "first" and family != "counterflow" and cells <= 2000
    solver = rng.choice(["OptRodas34", "OptRosenbrock34", "OptRodas23", "OptSeulex"]) if small else "OptRodas34"
    precision = "mixed" if family == "counterflow" and state == "next" and cells < 8000 and rng.random() < 0.3 else "fp64"
    return {"op": "step", "solver": solver, "precision": precision, "arrays": rng.choice(["device", "device", "host"]),
            "graph": False, "lts": rng.random() < 0.25, "family": family, "state": state, "cells": cells}


# ------------------------------------------------------------------------
# inputs


@functools.lru_cache(maxsize=None)
def fixture(family):
    """The family's mechanism and its fixture's cell states after one step."""
    g = np.load(os.path.join(ROOT, "tests", "golden", FAMILIES[family][0] + ".npz"))
    arrays = {k: np.ascontiguousarray(g["mech_" + k]) for k in (
        "W", "T_low", "T_high", "T_common", "high_coeffs", "low_coeffs", "type", "reversible", "lhs_offset",
        "lhs_species", "rhs_offset", "rhs_species", "arrhenius", "arrhenius2", "efficiencies", "falloff_params",
        "plog_offset", "plog_table")}
    flat = FlatMechanism(int(arrays["W"].shape[0]), int(arrays["type"].shape[0]), **arrays)
    react = g["in_T"] > FAMILIES[family][2]
    after = {"T": g["T"][react], "Y": g["Y"][:, react], "p": g["in_p"][react], "subDt": g["subDt"][react]}
    return flat, after


def cells_of(family, state, n, seed):
    """Cell states (numpy, species-major Y): T, p, Y, rho0, subDt."""
    flat, after = fixture(family)
    ns = flat.n_species
    rng = np.random.default_rng(seed)
    if state == "first":
        subDt = np.full(n, 1e-7)
        if family == "ignition":
            T, p = rng.uniform(1000.0, 1500.0, n), np.full(n, 1e5)
            Y = rng.dirichlet(np.full(ns, 0.5), size=n).T
        elif family == "falloff":
            T, p = rng.uniform(900.0, 1800.0, n), 10.0 ** rng.uniform(4.0, 7.0, n)
            Y = rng.dirichlet(np.full(ns, 0.5), size=n).T
        elif family == "counterflow":
            x = rng.random(n)
            T = 300.0 + 1900.0 * 0.5 * (1.0 + np.tanh((x - 0.5) / 0.08))
            p = rng.uniform(1e5, 5e6, n)
            ends = np.random.default_rng(53).dirichlet(np.full(ns, 0.5), size=2)
            mix = rng.random(n)
            Y = np.outer(ends[0], 1.0 - mix) + np.outer(ends[1], mix)
        else:
            T, p = rng.uniform(1200.0, 2200.0, n), rng.uniform(1e5, 1e6, n)
            Y = rng.dirichlet(np.full(ns, 0.3), size=n).T
    else:
        m = after["T"].shape[0]
        a, b = rng.integers(0, m, n), rng.integers(0, m, n)
        w = rng.uniform(0.0, 0.00005, n)
        T = (after["T"][a] * (1 - w) + after["T"][b] * w) * rng.uniform(0.9998, 1.0002, n)
        Y = after["Y"][:, a] * (1 - w) + after["Y"][:, b] * w
        p = after["p"][a] * rng.uniform(0.999, 1.001, n)
        subDt = after["subDt"][a].copy()
        if FAMILIES[family][2] > 0:  # the cold part of the field does not react
            T = np.where(rng.random(n) < 0.4, rng.uniform(300.0, 700.0, n), T)
    Y = np.ascontiguousarray(Y)
    rho0 = p / (RU * T * (Y / flat.W[:, None]).sum(axis=0))
    return {"T": np.ascontiguousarray(T), "p": np.ascontiguousarray(p), "Y": Y, "rho0": rho0, "subDt": subDt}


def deltas_of(case, seed):
    """Per-cell time steps of a local-time-stepping call."""
    dt = FAMILIES[case["family"]][1]
    return dt * np.random.default_rng(seed + 77).uniform(0.5, 1.0, case["cells"])


def network_of(case, seed):
    """Parameters (per member) and normalisation of a surrogate of the family's size."""
    ns = fixture(case["family"])[0].n_species
    dims = [ns + 3] + [MLP["width"]] * MLP["depth"] + [ns + 2]
    rng = np.random.default_rng(seed + 5)
    members = []
    for _ in range(MLP["members"]):
        layers = []
        for i, o in zip(dims[:-1], dims[1:]):
            layers.append((rng.normal(0, math.sqrt(2.0 / i), (o, i)).astype(np.float32),
                           rng.normal(0, 0.1, o).astype(np.float32)))
        members.append(layers)
    return dims, members


def samples_of(case, seed):
    """Surrogate inputs (T, ln p, ln dt, Y) and target outputs in raw units."""
    family, n = case["family"], case["cells"]
    c = cells_of(family, "first", n, seed)
    x = np.empty((n, c["Y"].shape[0] + 3), np.float32)
    x[:, 0], x[:, 1], x[:, 2], x[:, 3:] = c["T"], np.log(c["p"]), math.log(FAMILIES[family][1]), c["Y"].T
    rng = np.random.default_rng(seed + 9)
    t = rng.normal(0, 1, (n, x.shape[1] - 1)).astype(np.float32)
    t[:, 0] *= 300.0
    t[:, 1:-1] *= 0.02
    return x, t, (x.mean(0), np.maximum(x.std(0), 1e-3), t.mean(0), np.maximum(t.std(0), 1e-6))


class State:
    pass


def prepare(case, seed):
    s = State()
    s.op = case["op"]
    if s.op in ("forward", "gradients"):
        dims, members = network_of(case, seed)
        x, t, norm = samples_of(case, seed)
        s.mlp = _lib.Mlp(dims[0], dims[-1], seed=1, **MLP)
        s.mlp.set_normalization(*norm)
        for m, layers in enumerate(members):
            s.mlp.set_params(m, np.concatenate([np.concatenate([w.ravel(), b]) for w, b in layers]))
        s.x, s.t = (torch.from_numpy(x).cuda(), None) if s.op == "forward" else (x, t)
        torch.cuda.synchronize()
        return s
    family, n = case["family"], case["cells"]
    flat, _ = fixture(family)
    s.n, s.dt = n, FAMILIES[family][1]
    s.ctx = _lib.Context(0)
    s.ctx.load_mechanism(flat)
    if s.op != "step":
        s.ctx.set_options(abs_tol=1e-8, rel_tol=1e-4)
        d = {k: torch.from_numpy(v).cuda() for k, v in cells_of(family, "first", n, seed).items()}
        s.p, s.T, s.rho, s.Y = d["p"], d["T"], d["rho0"], d["Y"]
        N = flat.n_species + 1
        new = functools.partial(torch.zeros, dtype=torch.float64, device="cuda")
        s.out = (new(flat.n_species, n), new(n), new(n)) if s.op == "rates" else (new(n, N, N), new(N, n))
        torch.cuda.synchronize()
        return s
    s.ctx.set_options(solver=case["solver"], precision=case["precision"], abs_tol=1e-8, rel_tol=1e-4,
                      treact=FAMILIES[family][2])
    c = cells_of(family, case["state"], n, seed)
    s.host = case["arrays"] == "host"
    s.flags = _lib.CUDA_GRAPH if case["graph"] else 0
    dtc = deltas_of(case, seed) if case["lts"] else None
    if s.host:
        s.p, s.rho0, s.start = c["p"], c["rho0"], (c["T"], c["Y"], c["subDt"])
        s.T, s.Y, s.sub, s.RR = c["T"].copy(), c["Y"].copy(), c["subDt"].copy(), np.zeros_like(c["Y"])
        s.status, s.dtc = np.zeros(n, np.int32), dtc
    else:
        d = {k: torch.from_numpy(v).cuda() for k, v in c.items()}
        s.p, s.rho0, s.start = d["p"], d["rho0"], (d["T"], d["Y"], d["subDt"])
        s.T, s.Y, s.sub, s.RR = d["T"].clone(), d["Y"].clone(), d["subDt"].clone(), torch.zeros_like(d["Y"])
        s.status = torch.zeros(n, dtype=torch.int32, device="cuda")
        s.dtc = None if dtc is None else torch.from_numpy(dtc).cuda()
        torch.cuda.synchronize()
    return s


def run(s):
    if s.op == "forward":
        torch.cuda.current_stream().synchronize()  # the library works on its own stream
        return [s.mlp.forward(m, s.x, device=True) for m in range(s.mlp.members)]
    if s.op == "gradients":
        return [s.mlp.gradients(m, s.x, s.t) for m in range(s.mlp.members)]
    if s.op == "step":
        if s.host:
            np.copyto(s.T, s.start[0]), np.copyto(s.Y, s.start[1]), np.copyto(s.sub, s.start[2])
        else:
            s.T.copy_(s.start[0]), s.Y.copy_(s.start[1]), s.sub.copy_(s.start[2])
            torch.cuda.current_stream().synchronize()
        _, stats, dmin = s.ctx.integrate_raw(s.n, s.dt, s.p, s.rho0, s.T, s.Y, s.sub, s.RR, s.status,
                                             device=not s.host, dt_per_cell=s.dtc, flags=s.flags)
        return {"T": s.T, "Y": s.Y, "subDt": s.sub, "RR": s.RR, "status": s.status, "deltaTMin": dmin,
                "cells": stats["cells_integrated"]}
    L, ptr = s.ctx.L, lambda a: a.data_ptr()
    if s.op == "rates":
        RR, Q, tc = s.out
        s.ctx._check(L.fcs_rates(s.ctx.h, s.n, ptr(s.p), ptr(s.T), ptr(s.rho), ptr(s.Y), ptr(RR), ptr(Q),
                                 _lib.PTR_DEVICE))
        s.ctx._check(L.fcs_tc(s.ctx.h, s.n, ptr(s.p), ptr(s.T), ptr(s.rho), ptr(s.Y), ptr(tc), _lib.PTR_DEVICE))
    else:
        J, f = s.out
        s.ctx._check(L.fcs_jacobian(s.ctx.h, s.n, ptr(s.p), ptr(s.T), ptr(s.Y), ptr(J), ptr(f), _lib.PTR_DEVICE))
    return list(s.out)


def work(case):
    n = case["cells"]
    flat, _ = fixture(case["family"])
    ns, nr = flat.n_species, flat.n_reactions
    N = ns + 1
    ntb = int(np.isin(flat.type, (1, 3, 4, 5, 7)).sum())
    rhs = 40 * ns + 12 * nr + 2 * ns * ntb
    jac = rhs + 40 * nr + 4 * ns * ntb + 10 * N * N
    if case["op"] in ("forward", "gradients"):
        dims = [ns + 3] + [MLP["width"]] * MLP["depth"] + [ns + 2]
        params = sum(i * o + o for i, o in zip(dims[:-1], dims[1:]))
        passes = 1 if case["op"] == "forward" else 3
        return {"bytes": MLP["members"] * (4.0 * n * (dims[0] + dims[-1]) + 4.0 * params * (1 if passes == 1 else 2)),
                "flops": MLP["members"] * passes * 2.0 * n * (params - sum(dims[1:]))}
    if case["op"] == "rates":
        return {"bytes": 8.0 * n * (2 * ns + 6), "flops": 2.0 * n * rhs}
    if case["op"] == "jacobian":
        return {"bytes": 8.0 * n * (ns + 2 + N + N * N), "flops": 1.0 * n * jac}
    _, _, treact, first, later = FAMILIES[case["family"]]
    attempts = n * (first if case["state"] == "first" else later) * (0.6 if treact > 0 else 1.0)
    attempt = jac + 2.0 / 3.0 * N ** 3 + 6 * 2 * N * N + 5 * rhs + 40 * N
    return {"bytes": 8.0 * n * (3 * ns + 7), "flops": attempts * attempt}


# ------------------------------------------------------------------------
# the same in 64-bit torch, without the library


class Chemistry:
    """Rates of the Arrhenius, third-body and PLOG kinds; states are [n], Y [n, ns]."""

    def __init__(self, flat):
        def t(a):
            return torch.as_tensor(np.asarray(a), device="cuda")
        self.ns, self.nr = flat.n_species, flat.n_reactions
        ns, nr = self.ns, self.nr
        self.W, self.Tcommon = t(flat.W), t(flat.T_common)
        self.Trange = float(flat.T_low.min()), float(flat.T_high.max())
        self.low, self.high = t(flat.low_coeffs.reshape(ns, 7)), t(flat.high_coeffs.reshape(ns, 7))
        self.arr = t(flat.arrhenius.reshape(nr, 3))
        self.type, self.rev = t(flat.type), t(flat.reversible) != 0

        def sides(off, sp):  # species ns stands for "none": concentration 1, Gibbs factor 0
            k = int(np.diff(off).max())
            idx = np.full((nr, k), ns)
            for r in range(nr):
                idx[r, :off[r + 1] - off[r]] = sp[off[r]:off[r + 1]]
            return t(idx), t(np.diff(off).astype(np.float64))
        self.lhs, self.nl = sides(flat.lhs_offset, flat.lhs_species)
        self.rhs, self.nrr = sides(flat.rhs_offset, flat.rhs_species)
        nu = np.zeros((nr, ns))
        for r in range(nr):
            for sp in flat.lhs_species[flat.lhs_offset[r]:flat.lhs_offset[r + 1]]:
                nu[r, sp] -= 1
            for sp in flat.rhs_species[flat.rhs_offset[r]:flat.rhs_offset[r + 1]]:
                nu[r, sp] += 1
        self.nu = t(nu)
        self.tb = t(np.nonzero(flat.type == 1)[0])
        self.eff = t(flat.efficiencies.reshape(nr, ns)[flat.type == 1])
        self.plog = [(r, flat.plog_table.reshape(-1, 4)[flat.plog_offset[r]:flat.plog_offset[r + 1]])
                     for r in np.nonzero(flat.type == 2)[0]]

    def coeffs(self, T):
        return torch.where((T[:, None] < self.Tcommon)[..., None], self.low, self.high).unbind(-1)

    def constants(self, T, p, C):
        """Kf with third bodies and 1/Kc before its clamp."""
        a0, a1, a2, a3, a4, a5, a6 = self.coeffs(T)
        t, lnT = T[:, None], T.log()[:, None]
        g = (a0 * (lnT - 1) + a6 - a5 / t + t * (a1 / 2 + t * (a2 / 6 + t * (a3 / 12 + t * a4 / 20))))
        A, beta, Ta = self.arr.unbind(1)
        k = A * torch.exp(beta * lnT - Ta / t)
        cols = list(k.unbind(1)) if self.plog else None
        for r, rows in self.plog:
            lp = np.log(rows[:, 0])
            at = torch.clamp(torch.searchsorted(torch.as_tensor(lp, device=T.device), p.log()) - 1, 0, len(lp) - 2)
            ln = torch.stack([math.log(A_) + b_ * lnT[:, 0] - ta_ / T for _, A_, b_, ta_ in rows], 1)
            lpt = torch.as_tensor(lp, device=T.device)
            f = torch.clamp((p.log() - lpt[at]) / (lpt[at + 1] - lpt[at]), 0.0, 1.0)
            lo, hi = ln.gather(1, at[:, None])[:, 0], ln.gather(1, at[:, None] + 1)[:, 0]
            cols[r] = torch.exp(lo + (hi - lo) * f)
        if self.plog:
            k = torch.stack(cols, 1)
        if len(self.tb):
            M = torch.ones_like(k).index_copy(1, self.tb, C @ self.eff.T)
            k = k * M
        gz = torch.cat([g, torch.zeros_like(g[:, :1])], 1)
        ln_invKc = gz[:, self.lhs].sum(-1) - gz[:, self.rhs].sum(-1) + (self.nrr - self.nl) * torch.log(RU * t / PSTD)
        return k, ln_invKc

    def products(self, C):
        Cz = torch.cat([C, torch.ones_like(C[:, :1])], 1)

        def prod(idx):
            v = Cz[:, idx[:, 0]]
            for q in range(1, idx.shape[1]):
                v = v * Cz[:, idx[:, q]]
            return v
        return prod(self.lhs), prod(self.rhs)

    def net(self, T, p, C):
        k, ln_invKc = self.constants(T, p, C)
        invKc = torch.exp(torch.clamp(ln_invKc, max=-math.log(1.4901171103413047e-8)))
        CF, CR = self.products(C)
        return torch.where(self.rev, k * (CF - invKc * CR), k * CF) @ self.nu

    def derivatives(self, p, T, Y, last=False):
        Y = torch.clamp(Y, min=0)
        x = Y / self.W
        v = RU * T / p * x.sum(1)
        C = x / v[:, None]
        Tc = torch.clamp(T, *self.Trange)  # a rejected attempt's stages may leave the range of the fits
        dY = self.W * v[:, None] * self.net(Tc, p, C)
        T = T if last else Tc
        a0, a1, a2, a3, a4, a5, _ = self.coeffs(Tc)
        t = T[:, None]
        cp = RU / self.W * (a0 + t * (a1 + t * (a2 + t * (a3 + t * a4))))
        ha = RU / self.W * (a5 + t * (a0 + t * (a1 / 2 + t * (a2 / 3 + t * (a3 / 4 + t * a4 / 5)))))
        return torch.cat([dY, -((ha * dY).sum(1) / (Y * cp).sum(1))[:, None]], 1)

    def jacobian(self, p, T, Y):
        y = torch.cat([Y, T[:, None]], 1).requires_grad_(True)
        f = self.derivatives(p, y[:, -1], y[:, :-1])
        rows = [torch.autograd.grad(f[:, i].sum(), y, retain_graph=True)[0] for i in range(self.ns + 1)]
        return torch.stack(rows, 1), f.detach()

    def source_terms(self, p, T, rho, Y):
        C = rho[:, None] * Y / self.W
        RR = self.net(T, p, C) * self.W
        t = torch.tensor(298.15, dtype=torch.float64, device=T.device)
        a0, a1, a2, a3, a4, a5, _ = torch.where((t < self.Tcommon)[:, None], self.low, self.high).unbind(-1)
        hf = RU / self.W * (a5 + t * (a0 + t * (a1 / 2 + t * (a2 / 3 + t * (a3 / 4 + t * a4 / 5)))))
        k, ln_invKc = self.constants(T, p, C)
        CF, CR = self.products(C)
        wf = self.nrr * k * CF
        wr = torch.where(self.rev, self.nl * k * CR * torch.exp(torch.clamp(ln_invKc, max=-math.log(1.49011611938476e-8))),
                         0.0)
        tc = (wf + wr).sum(1) / (wf * wf + wr * wr).sum(1) * C.sum(1)
        return RR, -(RR * hf).sum(1), tc

    # OptRodas34 with its step-size control (the constants of the method)
    A = ((), (1.544,), (0.9466785280815826, 0.2557011698983284),
         (3.314825187068521, 2.896124015972201, 0.9986419139977817),
         (1.221224509226641, 6.019134481288629, 12.53708332932087, -0.6878860361058950))
    C_ = ((), (-5.6688,), (-2.430093356833875, -0.2063599157091915),
          (-0.1073529058151375, -9.594562251022355, -20.47028614809616),
          (7.496443313967647, -10.24680431464352, -33.99990352819905, 11.70890893206160),
          (8.083246795921522, -7.981132988064893, -31.52159432874371, 16.31930543123136, -6.058818238834054))
    D = (0.25, -0.1043, 0.1035, -0.03620000000000023)

    def attempt(self, p, y, dx, abs_tol, rel_tol):
        J, f0 = self.jacobian(p, y[:, -1], y[:, :-1])
        h = dx[:, None]
        M = torch.diag_embed((4.0 / h).expand_as(y)) - J
        lu, piv = torch.linalg.lu_factor(M)
        ks = []
        for s in range(6):
            if s == 0:
                b = f0
            elif s < 5:
                z = y + sum(a * k for a, k in zip(self.A[s], ks))
                b = self.derivatives(p, z[:, -1], z[:, :-1])
            else:
                z = y + sum(a * k for a, k in zip(self.A[4], ks[:4])) + ks[4]
                b = self.derivatives(p, z[:, -1], z[:, :-1], last=True)
            if s < 4:
                b = b + h * self.D[s] * f0
            b = b + sum((c / h * k for c, k in zip(self.C_[s], ks)), torch.zeros_like(y))
            ks.append(torch.linalg.lu_solve(lu, piv, b[..., None])[..., 0])
        yn = y + sum(a * k for a, k in zip(self.A[4], ks[:4])) + ks[4] + ks[5]
        tol = abs_tol + rel_tol * torch.maximum(y.abs(), yn.abs())
        return yn, (ks[5].abs() / tol).amax(1)

    def step(self, p, T, Y, sub, dt, abs_tol, rel_tol):
        y = torch.cat([torch.clamp(Y, min=0), T[:, None]], 1)
        x, nxt, sub = torch.zeros_like(T), sub.clone(), sub.clone()
        dx, retry = sub.clone(), torch.zeros_like(T, dtype=torch.bool)
        last, steps = retry.clone(), torch.zeros_like(T)
        live = torch.arange(T.shape[0], device=T.device)
        while live.numel():
            fresh = live[~retry[live]]
            nxt[fresh] = sub[fresh]
            over = fresh[x[fresh] + sub[fresh] > dt[fresh]]
            last[over], sub[over] = True, dt[over] - x[over]
            dx[fresh] = sub[fresh]
            yn, err = self.attempt(p[live], y[live], dx[live], abs_tol, rel_tol)
            bad = err > 1
            no, yes, e = live[bad], live[~bad], err[~bad]
            dx[no] = dx[no] * torch.clamp(0.9 * err[bad] ** -0.25, min=0.2)
            retry[no], retry[yes] = True, False
            y[yes] = yn[~bad]
            x[yes] += dx[yes]
            sub[yes] = torch.where(e > (10 / 0.9) ** -5.0, torch.clamp(0.9 * e ** -0.2, 0.2, 10.0), 9.0) * dx[yes]
            done = yes[x[yes] >= dt[yes]]
            keep = done[(steps[done] > 0) & last[done]]
            sub[keep] = nxt[keep]
            steps[yes] += 1
            gone = torch.zeros_like(retry)
            gone[done] = True
            live = live[~gone[live]]
        return y[:, -1], torch.clamp(y[:, :-1], min=0), sub


def exact(case, seed):
    if case["op"] in ("forward", "gradients"):
        _, members = network_of(case, seed)
        x, t, norm = samples_of(case, seed)
        x, t = (torch.from_numpy(v).cuda().double() for v in (x, t))
        im, istd, om, ostd = (torch.from_numpy(np.asarray(v, np.float32)).cuda().double() for v in norm)
        out = []
        for layers in members:
            params = [torch.from_numpy(v).cuda().double().requires_grad_(True) for wb in layers for v in wb]
            h = (x - im) / istd
            for i in range(0, len(params), 2):
                h = h @ params[i].T + params[i + 1]
                if i < len(params) - 2:
                    h = torch.nn.functional.gelu(h)
            if case["op"] == "forward":
                out.append((h * ostd + om).detach())
            else:
                loss = ((h - (t - om) / ostd) ** 2).mean()
                g = torch.autograd.grad(loss, params)
                out.append((float(loss.detach()), torch.cat([v.reshape(-1) for v in g]).cpu().numpy()))
        return out
    family, n = case["family"], case["cells"]
    flat, _ = fixture(family)
    if case["op"] == "step":
        # one Rodas34 attempt differentiates every row: minutes beyond the small mechanisms and fields,
        # and the other methods, kinds and precisions are the library's own
        if family != "ignition" or case["solver"] != "OptRodas34" or case["precision"] != "fp64" or n > 2000:
            return None
        c = {k: torch.from_numpy(v).cuda() for k, v in cells_of(family, case["state"], n, seed).items()}
        dt = torch.from_numpy(deltas_of(case, seed)).cuda() if case["lts"] else torch.full_like(c["T"], FAMILIES[family][1])
        T, Y, sub = Chemistry(flat).step(c["p"], c["T"], c["Y"].T.contiguous(), c["subDt"], dt, 1e-8, 1e-4)
        Yn = Y.T.contiguous()
        # the next sub-step jumps with the last bit of the accepted steps' sum (whether it reaches the end exactly)
        return {"T": T, "Y": Yn, "subDt": None, "RR": (Yn - c["Y"]) * c["rho0"] / dt, "status": None,
                "deltaTMin": None, "cells": None}
    c = {k: torch.from_numpy(v).cuda() for k, v in cells_of(family, "first", n, seed).items()}
    chem, Y = Chemistry(flat), c["Y"].T.contiguous()
    if case["op"] == "rates":
        parts = [[v.detach() for v in chem.source_terms(c["p"][i:i + 8192], c["T"][i:i + 8192], c["rho0"][i:i + 8192],
                                                        Y[i:i + 8192])] for i in range(0, n, 8192)]
        RR, Q, tc = (torch.cat(v) for v in zip(*parts))
        return [RR.T.contiguous(), Q, tc]
    parts = [chem.jacobian(c["p"][i:i + 500], c["T"][i:i + 500], Y[i:i + 500]) for i in range(0, n, 500)]
    J, f = (torch.cat(v) for v in zip(*parts))
    return [J, f.T.contiguous()]
