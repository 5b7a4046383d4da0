"""Performance cases of the HSolve framework: what a program has it do, over
the range of sizes it is used at.

Every case steps HSolve cells through the public Python entry points and reads
the results back, as a driving script does between two outputs:

  cable    one FP64 drop-in HSolve: a soma and an unbranched HH cable
  dropin   one FP64 drop-in HSolve: a branched cell with HH Na/K, Ca(HVA),
           K(Ca) HHChannel2D, a CaConc per compartment and SynChans
  group    the HSolves of one clock tick, stepped together (Tick)
  batch    a population in one batch, FP64 or mixed precision, in the layout
           a new batch has or in the one the autotuner picks for large
           populations ("merged": one global-memory forest per CTA)
  cohort   a serving cohort: requests of different lengths, from reinit to the
           last one's end, with the output the serving loop polls
  cluster  one large cell, mixed precision, on a thread-block cluster

The time step is 25 us everywhere.  Except for `cohort`, which starts over,
each pass goes on from the state the pass before it left.
"""
import functools
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "moose-core_gb300"))

from moose_gb300 import models  # noqa: E402
from moose_gb300.abi import HS_PREC_FP64, HS_PREC_MIXED  # noqa: E402
from moose_gb300.batch import Batch  # noqa: E402
from moose_gb300.hsolve import HSolve, Tick  # noqa: E402

DT = 25e-6
T_EVENTS = 0.5          # s of synaptic input each cell comes with
STRIDE = 40             # dt steps between the soma samples of a cohort


def listed():
    return [
        # a script that looks at the cell after every step (a controller, a
        # Table on every tick): one step, then every compartment's Vm
        dict(name="cable_201_one_step", kind="cable", compartments=201, steps=1),
        # the single-cell workload: 10 ms of the 201-compartment squid cable
        dict(name="cable_201", kind="cable", compartments=201, steps=400),
        # one reconstructed-size neuron with synaptic input, 2.5 ms
        dict(name="dropin_500", kind="dropin", compartments=500, synapses=200, steps=100),
        # one very large neuron
        dict(name="dropin_4999", kind="dropin", compartments=4999, synapses=200, steps=40),
        # 256 cells, each its own HSolve, on one clock tick
        dict(name="group_256", kind="group", cells=256, lo=100, hi=1000, steps=40),
        # a small population, reference precision, synaptic input
        dict(name="batch_fp64_256", kind="batch", precision="fp64", cells=256, lo=50, hi=5000, synapses=200,
             steps=20, layout="default"),
        # a large population, reference precision, injected currents
        dict(name="batch_fp64_1024", kind="batch", precision="fp64", cells=1024, lo=50, hi=5000, synapses=0,
             steps=20, layout="default"),
        # one small request alone on the GPU: the step latency of the batch
        dict(name="batch_mixed_1", kind="batch", precision="mixed", cells=1, lo=203, hi=203, synapses=50,
             steps=400, layout="default"),
        # a large population, mixed precision, synaptic input, as created
        dict(name="batch_mixed_1024", kind="batch", precision="mixed", cells=1024, lo=50, hi=5000, synapses=200,
             steps=100, layout="default"),
        # the same in the layout the autotuner picks
        dict(name="batch_mixed_1024_merged", kind="batch", precision="mixed", cells=1024, lo=50, hi=5000,
             synapses=200, steps=100, layout="merged"),
        # one admission round of the serving loop
        dict(name="cohort_24", kind="cohort", cells=24, lo=100, hi=10000, steps=400),
        # the largest request with SMs to spare
        dict(name="cluster_9001", kind="cluster", compartments=9001, ctas=4, steps=100),
    ]


def draw(rng):
    def logint(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["cable", "dropin", "dropin", "group", "batch64", "batch64", "mixed", "mixed", "mixed",
                       "cohort", "cluster"])
    if kind == "cable":
        return dict(kind="cable", compartments=logint(20, 401), steps=logint(1, 200))
    if kind == "dropin":
        return dict(kind="dropin", compartments=logint(50, 4999), synapses=rng.choice([0, 13, 200]),
                    steps=logint(1, 40))
    if kind == "group":
        lo = logint(50, 400)
        return dict(kind="group", cells=logint(2, 256), lo=lo, hi=lo + logint(50, 600), steps=logint(1, 40))
    if kind == "cohort":
        return dict(kind="cohort", cells=logint(2, 24), lo=100, hi=logint(400, 10000), steps=STRIDE * rng.randint(2, 10))
    if kind == "cluster":
        return dict(kind="cluster", compartments=logint(2000, 9001), ctas=rng.choice([2, 4, 8]),
                    steps=logint(10, 100))
    prec = "fp64" if kind == "batch64" else "mixed"
    return dict(kind="batch", precision=prec, cells=logint(1, 1024), lo=50, hi=logint(200, 5000),
                synapses=rng.choice([0, 50, 200]), steps=logint(5, 20 if prec == "fp64" else 100),
                layout="default" if prec == "fp64" else rng.choice(["default", "merged"]))


# ---- the cells -----------------------------------------------------------------

@functools.lru_cache(maxsize=None)
def _kca_tables(divs):
    """The K(Ca) gate's 2-D tables: a constant of the channel library."""
    return models.kca_2d_tables(vdivs=divs, cadivs=divs)


def _branched(rnd, n, max_children):
    """A random dendritic tree of n compartments grown from the soma: each
    open tip gets one child, or with probability 1/2 a branch point."""
    parent = np.full(n, -1, np.int32)
    tips, count = [0], 1
    while count < n:
        k = int(rnd.random() * len(tips))
        tips[k], tips[-1] = tips[-1], tips[k]
        t = tips.pop()
        kids = rnd.randint(2, max_children) if rnd.random() < 0.5 else 1
        for _ in range(min(kids, n - count)):
            parent[count] = t
            tips.append(count)
            count += 1
    rng = np.random.default_rng(rnd.getrandbits(63))
    d = np.exp(rng.normal(math.log(1.5e-6), 0.4, n))
    length = rng.uniform(5e-6, 20e-6, n)
    d[0], length[0] = 20e-6, 20e-6
    return parent, d, length, rng


def _cell(rnd, n, synapses, max_children, divs):
    parent, d, length, rng = _branched(rnd, n, max_children)
    return models.active_cell(parent, d, length, inject=float(rng.uniform(0.1e-9, 1e-9)), n_syn=synapses, rng=rng,
                              t_end=T_EVENTS, kca_tables=_kca_tables(divs))


def _sizes(case):
    """Compartments of each cell: the case's, the same for every seed."""
    rnd = random.Random("%(cells)d %(lo)d %(hi)d" % case)
    if case["kind"] == "group":
        return [rnd.randint(case["lo"], case["hi"]) for _ in range(case["cells"])]
    lo, hi = math.log(case["lo"]), math.log(case["hi"])
    return [int(round(math.exp(rnd.uniform(lo, hi)))) for _ in range(case["cells"])]


def _models(case, seed):
    """The case's cells, and for a cohort each request's number of steps."""
    rnd = random.Random("%d %s" % (seed, case["kind"]))
    if case["kind"] == "cable":
        # a step current from the start, its amplitude the seed's
        return [models.config1_cell(n_cable=case["compartments"] - 1, inject=rnd.uniform(0.3e-9, 0.9e-9), t_on=0.0,
                                    t_off=1e4)], None
    if case["kind"] in ("dropin", "cluster"):
        return [_cell(rnd, case["compartments"], case.get("synapses", 200), 4,
                      300 if case["kind"] == "dropin" else 3000)], None
    if case["kind"] == "group":
        return [_cell(rnd, n, 0, 2, 300) for n in _sizes(case)], None
    sizes = _sizes(case)
    if case["kind"] == "cohort":
        steps = [rnd.randint(case["steps"] // 4, case["steps"]) for _ in sizes]
        steps[0] = case["steps"]
        # a step current, or synapses, with even odds
        return [_cell(rnd, n, rnd.choice([0, rnd.randint(50, 500)]), 4, 3000) for n in sizes], steps
    return [_cell(rnd, n, case["synapses"], 4, 3000) for n in sizes], None


# ---- passes ----------------------------------------------------------------------

def prepare(case, seed):
    cells, stops = _models(case, seed)
    kind, steps = case["kind"], case["steps"]
    if kind in ("cable", "dropin", "group"):
        solvers = []
        for m in cells:
            h = HSolve(m, dt=DT)
            h.target = m.seed
            h.reinit(DT)
            solvers.append(h)
        return dict(kind=kind, steps=steps, solvers=solvers, tick=Tick(solvers))
    if kind == "cohort":
        b = Batch(cells, DT, HS_PREC_MIXED, steps_per_launch=steps, max_ctas=len(cells))
        b.record(np.arange(len(cells)), np.zeros(len(cells), np.uint32), STRIDE, steps // STRIDE + 2)
        b.set_stop_steps(stops)
    elif kind == "cluster":
        b = Batch(cells, DT, HS_PREC_MIXED, max_ctas=case["ctas"], cluster_ctas=case["ctas"])
    elif case["precision"] == "fp64":
        b = Batch(cells, DT, HS_PREC_FP64)
    elif case["layout"] == "merged":
        b = Batch(cells, DT, HS_PREC_MIXED, forest_nodes=8, elim_warps=8)
    else:
        b = Batch(cells, DT, HS_PREC_MIXED)
    b.reinit(DT)
    return dict(kind=kind, steps=steps, batch=b)


def run(state):
    kind, steps = state["kind"], state["steps"]
    if kind in ("cable", "dropin"):
        h = state["solvers"][0]
        h.process(steps)
        return [h.vm(), h.ca()] if kind == "dropin" else [h.vm()]
    if kind == "group":
        state["tick"].process(steps)
        return [np.concatenate([h.vm() for h in state["solvers"]])]
    b = state["batch"]
    if kind == "cohort":
        b.reinit(DT)
        b.process(steps)
        return list(b.poll(0, steps // STRIDE + 1)) + [b.read_all("Vm")]
    b.process(steps)
    return [b.read_all("Vm"), b.read_all("Ca")]


def _expected_compartments(case):
    if "compartments" in case:
        return case["compartments"]
    if case["kind"] == "group":
        return case["cells"] * (case["lo"] + case["hi"]) / 2
    lo, hi = case["lo"], case["hi"]
    return case["cells"] * ((hi - lo) / math.log(hi / lo) if hi > lo else lo)


def work(case):
    """Per pass: state and parameters read once, state and results written
    once (a population's state could stay on the chip between steps), and the
    arithmetic of every step.  FP64 sizes per compartment: V 16 B, matrix row
    32 B, gates 16 B each, Gbar 8 B, pool 32 B, K(Ca) 24 B; SynChan 40 B."""
    mixed = case["kind"] in ("cohort", "cluster") or case.get("precision") == "mixed"
    n, s = _expected_compartments(case), 4 if mixed else 8
    steps = case["steps"] * (0.625 if case["kind"] == "cohort" else 1.0)
    if case["kind"] == "cable":
        state, out, flops = 48 + 3 * 2 * s + 2 * s, 8, 55
    else:
        state, out, flops = 48 + 5 * 2 * s + 3 * s + 4 * s + 3 * s, 16, 130
    syn = case.get("synapses", 200 if case["kind"] == "cluster" else 0) * case.get("cells", 1)
    return {"bytes": n * (state + out) + syn * 5 * s, "flops": n * steps * flops + syn * steps * 8}


# ---- the same in 64 bits, from the equations ---------------------------------------

class _Exact:
    """The cells of a case stepped together in plain torch, FP64: the HSolve
    equations (gates trapezoidal on the tabulated rates, implicit membrane
    step solved on the tree with every branch point as a massless node)."""

    def __init__(self, cells, stops):
        n_each = np.array([m.n_compt for m in cells])
        base = np.concatenate([[0], np.cumsum(n_each)])
        n = self.n = int(base[-1])
        self.dev = dev = torch.device("cuda" if n > 20000 and torch.cuda.is_available() else "cpu")
        cat = lambda k: np.concatenate([np.asarray(getattr(m, k), np.float64) for m in cells])  # noqa: E731
        t = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=dev)  # noqa: E731
        par = np.concatenate([np.where(m.parent >= 0, m.parent + b, -1) for m, b in zip(cells, base)]).astype(np.int64)
        Ra, Rm, Cm, Em = cat("Ra"), cat("Rm"), cat("Cm"), cat("Em")
        Ga = 2.0 / Ra
        kids = np.bincount(par[par >= 0], minlength=n)
        junction = np.full(n, -1, np.int64)
        fork = np.nonzero(kids >= 2)[0]
        junction[fork] = n + np.arange(len(fork))
        total = n + len(fork)
        diag, off, tp = np.zeros(total), np.zeros(total), np.full(total, -1, np.int64)
        diag[:n] = 2.0 * Cm / DT + 1.0 / Rm
        c = np.nonzero(par >= 0)[0]
        p = par[c]
        one = kids[p] == 1
        g = Ga[p] * Ga[c] / (Ga[p] + Ga[c])
        np.add.at(diag, c[one], g[one])
        np.add.at(diag, p[one], g[one])
        tp[c[one]], off[c[one]] = p[one], -g[one]
        b, q = c[~one], p[~one]
        np.add.at(diag, b, Ga[b])
        np.add.at(diag, junction[q], Ga[b])
        tp[b], off[b] = junction[q], -Ga[b]
        np.add.at(diag, fork, Ga[fork])
        np.add.at(diag, junction[fork], Ga[fork])
        tp[junction[fork]], off[junction[fork]] = fork, -Ga[fork]
        # nodes level by level from the roots
        order = np.argsort(tp, kind="stable")
        first = np.searchsorted(tp[order], np.arange(-1, total))
        last = np.searchsorted(tp[order], np.arange(-1, total), side="right")
        levels, cur = [], order[first[0]:last[0]]
        while len(cur):
            levels.append(cur)
            cnt = last[cur + 1] - first[cur + 1]
            start = np.repeat(first[cur + 1] - np.concatenate([[0], np.cumsum(cnt)[:-1]]), cnt)
            cur = order[start + np.arange(cnt.sum())]
        perm = np.concatenate(levels)
        at = np.empty(total, np.int64)
        at[perm] = np.arange(total)
        self.cut = np.concatenate([[0], np.cumsum([len(x) for x in levels])]).tolist()
        self.perm, self.at = t(perm), t(at[:n])
        self.par, self.off = t(np.where(tp[perm] >= 0, at[tp[perm]], 0)), t(off[perm])
        self.diag, self.total = t(diag), total
        self.cmdt, self.emrm = t(2.0 * Cm / DT), t(Em / Rm)
        self.V = t(cat("initVm"))
        self.inj = t(cat("inject"))
        self.cells, self.base, self.t = cells, base, t
        cell_of = np.repeat(np.arange(len(cells)), n_each)
        self.stop = None if stops is None else t(np.asarray(stops)[cell_of])
        # channels: the k-th of every compartment is of one kind
        m0 = cells[0]
        self.nch = len(m0.chan_compt) // m0.n_compt
        self.gates = [(mn, mx, t(A), t(B)) for mn, mx, A, B in m0.gates]
        self.chan = []
        for k in range(self.nch):
            gb = np.concatenate([m.chan_Gbar[k::self.nch] for m in cells])
            gi = [(int(g[k]), float(p[k])) for g, p in ((m0.chan_xgate, m0.chan_Xpower), (m0.chan_ygate, m0.chan_Ypower))
                  if p[k] > 0]
            state = []
            for g_, _ in gi:
                A, B = self.rates(g_, self.V)
                state.append(A / B)
            self.chan.append([t(gb), float(m0.chan_Ek[k]), gi, state])
        self.pool = len(m0.pool_compt) > 0
        if self.pool:
            tau, Bp = cat("pool_tau"), cat("pool_B")
            self.f1, self.f2 = t(4.0 / (2.0 + DT / tau) - 1.0), t(2.0 * Bp * DT / (2.0 + DT / tau))
            self.basal = t(cat("pool_CaBasal"))
            self.c, self.ca = torch.zeros_like(self.V), self.basal.clone()
            x0, x1, y0, y1, A, B = m0.gates2d[0]
            self.g2 = (x0, x1, y0, y1, A.shape[0], A.shape[1], t(A).reshape(-1), t(B).reshape(-1))
            self.kg, self.kx = t(cat("c2d_Gbar")), t(cat("c2d_X"))
            self.kek = float(m0.c2d_Ek[0])
        # synapses: dual exponential, events of each step added up
        ns = [len(m.syn_compt) for m in cells]
        sb = np.concatenate([[0], np.cumsum(ns)])
        self.ns = int(sb[-1])
        if self.ns:
            self.sn = t(np.concatenate([m.syn_compt.astype(np.int64) + b for m, b in zip(cells, base)]))
            a, b = 1e-3, 3e-3
            assert all((m.syn_tau1 == a).all() and (m.syn_tau2 == b).all() for m in cells)
            peak = a * b * math.log(a / b) / (a - b)
            self.norm = (a - b) / (a * b * (math.exp(-peak / a) - math.exp(-peak / b)))
            self.sx, self.sy = torch.zeros(self.ns, dtype=torch.float64, device=dev), None
            self.sy = self.sx.clone()
            self.ex = (a * -math.expm1(-DT / a), math.exp(-DT / a), b * -math.expm1(-DT / b), math.exp(-DT / b))
            es = np.concatenate([m.ev_syn.astype(np.int64) + b for m, b in zip(cells, sb)])
            et, ew = cat("ev_time"), cat("ev_weight")
            k = np.maximum(0, np.floor(et / DT).astype(np.int64) - 2)
            while True:
                late = DT * (k + 1).astype(np.float64) < et
                if not late.any():
                    break
                k[late] += 1
            self.ev = (k, es, ew)

    def rates(self, g, v):
        mn, mx, A, B = self.gates[g]
        n = A.numel() - 1
        dx = (mx - mn) / n
        x = (v.clamp(mn, mx) - mn) / dx
        i = x.long().clamp(max=n)
        f = x - i
        j = (i + 1).clamp(max=n)
        return A[i] + (A[j] - A[i]) * f, B[i] + (B[j] - B[i]) * f

    def rates2(self, v, ca):
        x0, x1, y0, y1, nx, ny, A, B = self.g2
        x = (v.clamp(x0, x1) - x0) * ((nx - 1) / (x1 - x0))
        y = (ca.clamp(y0, y1) - y0) * ((ny - 1) / (y1 - y0))
        xi, yi = x.long().clamp(max=nx - 1), y.long().clamp(max=ny - 1)
        xf, yf = x - xi, y - yi
        xj, yj = (xi + 1).clamp(max=nx - 1), (yi + 1).clamp(max=ny - 1)
        w = ((1 - xf) * (1 - yf), xf * (1 - yf), (1 - xf) * yf, xf * yf)
        k = (xi * ny + yi, xj * ny + yi, xi * ny + yj, xj * ny + yj)
        return sum(u * A[q] for u, q in zip(w, k)), sum(u * B[q] for u, q in zip(w, k))

    def step(self, s):
        V = self.V
        live = None if self.stop is None else s < self.stop
        keep = (lambda new, old: new) if live is None else (lambda new, old: torch.where(live, new, old))
        for m, b in zip(self.cells, self.base):
            for q in np.nonzero(m.stim_step == s)[0]:
                self.inj[int(b) + int(m.stim_compt[q])] = float(m.stim_value[q])
        G, GE = torch.zeros_like(V), torch.zeros_like(V)
        gca = None
        for k, ch in enumerate(self.chan):
            gb, ek, gi, st = ch
            fr = torch.ones_like(V)
            for j, (g, power) in enumerate(gi):
                A, B = self.rates(g, V)
                h = 1.0 + DT / 2.0 * B
                st[j] = keep((st[j] * (2.0 - h) + DT * A) / h, st[j])
                fr = fr * st[j] ** int(power)
            gk = gb * fr
            G, GE = G + gk, GE + gk * ek
            if k == 2:
                gca, eca = gk, ek
        if self.pool:
            A, B = self.rates2(V, self.ca)
            e = torch.exp(-B * DT)
            x = torch.where(B > 1e-10, self.kx * e + A / B * -torch.expm1(-B * DT), self.kx + A * DT)
            self.kx = keep(x, self.kx)
            gk = self.kg * self.kx
            G, GE = G + gk, GE + gk * self.kek
        if self.ns:
            act = np.zeros(self.ns)
            now = self.ev[0] == s
            np.add.at(act, self.ev[1][now], self.ev[2][now] / DT)
            self.sx = self.t(act) * self.ex[0] + self.sx * self.ex[1]
            self.sy = self.sx * self.ex[2] + self.sy * self.ex[3]
            G.index_add_(0, self.sn, self.sy * self.norm)          # reversal potential 0
        d = self.diag.clone()
        d[:self.n] += G
        r = torch.zeros(self.total, dtype=torch.float64, device=self.dev)
        r[:self.n] = V * self.cmdt + self.emrm + GE + self.inj
        d, r = d[self.perm], r[self.perm]
        cut = self.cut
        for L in range(len(cut) - 2, 0, -1):
            i = slice(cut[L], cut[L + 1])
            f = self.off[i] / d[i]
            d.index_add_(0, self.par[i], -f * self.off[i])
            r.index_add_(0, self.par[i], -f * r[i])
        x = r / d
        f = self.off / d
        for L in range(1, len(cut) - 1):
            i = slice(cut[L], cut[L + 1])
            x[i] -= f[i] * x[self.par[i]]
        mid = x[self.at]
        self.V = keep(2.0 * mid - V, V)
        if self.pool:
            c = self.f1 * self.c + self.f2 * (gca * (eca - mid))
            ca = self.basal + c
            low = ca < 0.0
            ca, c = torch.where(low, torch.zeros_like(ca), ca), torch.where(low, -self.basal, c)
            self.c, self.ca = keep(c, self.c), keep(ca, self.ca)


def exact(case, seed):
    cells, stops = _models(case, seed)
    sim = _Exact(cells, stops)
    if case["kind"] != "cohort":
        for s in range(case["steps"]):
            sim.step(s)
        vm = sim.V.cpu().numpy()
        if case["kind"] in ("cable", "group"):
            return [vm]
        return [vm, sim.ca.cpu().numpy()]
    n = case["steps"] // STRIDE + 1
    trace = np.zeros((n, len(cells)))       # a request has no samples after its end
    soma = torch.as_tensor(sim.base[:-1], device=sim.dev)
    trace[0] = sim.V[soma].cpu().numpy()
    for s in range(case["steps"]):
        sim.step(s)
        if (s + 1) % STRIDE == 0:
            on = np.asarray(stops) > s
            trace[(s + 1) // STRIDE][on] = sim.V[soma].cpu().numpy()[on]
    return [trace, None, None, sim.V.cpu().numpy()]
