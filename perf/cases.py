"""The work that users of braincell_gb300 have it do, as timed cases.

A case is a dict of plain values.  ``prepare`` builds what a program holds before the call (a plan, a Cell, a
network, a trainer), ``run`` is one pass through the public entry points, ``work`` what a pass cannot do without,
and ``exact`` the same result from a plain float64 restatement of the model in torch (dense per tree level, no
kernels of the package).  States are read back in the precision of the plan (float32 for FP32 plans).

Kinds
-----
single   a SingleCompartment population stepped in a closed loop: ``update(I_ext)`` with another input every step,
         then ``V`` is read: launches, copies and host work.
update   a multi-compartment ``Cell`` stepped one ``dt`` at a time through the solver registry (interactive use,
         coupling to other simulators): the smallest call.
cellrun  ``Cell.run(dt, duration)`` of a small cell with its probe traces: a latency-bound run.
batch    a ``Plan`` over many cells: reset, n fused steps, read V.  ``lo`` to ``hi`` compartments a cell; ``shape`` 1 is the launch shape of the benchmark, 0 the library's defaults.
large    cells of 10,000 to 20,000 compartments with dynamic calcium.
network  cells joined by event-driven synapses: ``Network`` lowering, delivery between launches.
ports    cells whose distal subtrees are GRU ports (the surrogate's reduced run).
gru      a training window of the surrogate network: forward and backward through time.
"""

from __future__ import annotations

import math
from dataclasses import replace
from functools import lru_cache

import numpy as np
import torch

import braincell_gb300
from braincell_gb300 import SingleCompartment, _abi, environ
from braincell_gb300 import surrogate as S
from braincell_gb300 import workloads as W
from braincell_gb300.gru import GRUTrainer, init_params
from braincell_gb300.mech import AllRegion, CableProperty, Channel, CurrentClamp, CVPerBranch, ExpSyn, RootLocation, StateProbe
from braincell_gb300.morph import Branch, Morphology
from braincell_gb300.network import Connection, Network, Population
from braincell_gb300.runtime import Plan

DT = 0.025
# the launch shape of the repository's benchmark
SHAPE = dict(tile_nodes=2500, threads_per_tile=512, threads_big=512)


def listed():
    return [
        # 20,000 point neurons in a closed loop, one neuron per thread
        {"name": "single_20k", "kind": "single", "n": 20_000},
        # the 16 x 113-compartment configuration, one step per call
        {"name": "cell_update", "kind": "update", "n": 16},
        # the same cells through Cell.run: 1,000 steps, a trace per cell
        {"name": "cell_run", "kind": "cellrun", "n": 16, "steps": 1000},
        # a study of 300 uneven cells with the library's default launch shape
        {"name": "uneven_300", "kind": "batch", "n": 300, "lo": 50, "hi": 2000, "shape": 0, "steps": 400,
         "precision": "f32"},
        # the 10,000-cell configuration in the benchmark's launch shape (10 ms of its 200 ms)
        {"name": "uneven_10k", "kind": "batch", "n": 10_000, "lo": 50, "hi": 2000, "shape": 1, "steps": 400,
         "precision": "f32"},
        # 20,000 small cells (3 to 60 compartments)
        {"name": "small_20k", "kind": "batch", "n": 20_000, "lo": 3, "hi": 60, "shape": 1, "steps": 401,
         "precision": "f32"},
        # a double-precision reference run
        {"name": "uneven_f64", "kind": "batch", "n": 250, "lo": 50, "hi": 2000, "shape": 1, "steps": 200,
         "precision": "f64"},
        # the large-cell configuration, and one such cell alone (a single detailed neuron)
        {"name": "large_256", "kind": "large", "n": 256, "steps": 100},
        {"name": "large_1", "kind": "large", "n": 1, "steps": 200},
        # 1,000 cells, 10 contacts each, 10 ms
        {"name": "network_1k", "kind": "network", "n": 1000, "steps": 400},
        # surrogate inference and training
        {"name": "ports_1500", "kind": "ports", "n": 1500, "steps": 400},
        {"name": "gru_512", "kind": "gru", "n": 512, "steps": 400},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["single", "update", "cellrun", "batch", "batch", "batch", "large", "network", "ports", "gru"])
    if kind == "single":
        return {"kind": kind, "n": _log(rng, 64, 100_000)}
    if kind == "update":
        return {"kind": kind, "n": _log(rng, 1, 64)}
    if kind == "cellrun":
        return {"kind": kind, "n": _log(rng, 1, 64), "steps": rng.randint(100, 1000)}
    if kind == "batch":
        lo, hi = rng.choice([(50, 2000), (3, 60), (20, 400), (500, 3000)])
        prec = rng.choice(["f32", "f32", "f32", "f64"])
        cv = 1.0 * (hi - lo) / math.log(hi / lo)
        most = (6.0e6 if prec == "f32" else 3.0e5) / cv
        return {"kind": kind, "n": _log(rng, 30, min(most, 20_000)), "lo": lo, "hi": hi, "shape": rng.randint(0, 1),
                "steps": rng.randint(50, 400 if prec == "f32" else 200), "precision": prec}
    if kind == "large":
        return {"kind": kind, "n": _log(rng, 1, 256), "steps": rng.randint(20, 100)}
    if kind == "network":
        return {"kind": kind, "n": _log(rng, 64, 2000), "steps": rng.randint(200, 400)}
    if kind == "ports":
        return {"kind": kind, "n": _log(rng, 50, 1500), "steps": rng.randint(100, 400)}
    return {"kind": kind, "n": _log(rng, 5, 512), "steps": rng.randint(20, 400)}


# ------------------------------------------------------------------------------------------------ inputs
_HH = dict(na=Channel("Na_HH1952"), k=Channel("K_HH1952"), leak=Channel("IL", g_max=0.3, E=-54.4))


def _single_inputs(case, seed):
    rng = np.random.default_rng([seed, 11])
    n = case["n"]
    v0 = -70.0 + rng.integers(0, 32, n) * (10.0 / 32.0)
    amps = rng.uniform(2e3, 2.5e4, (8, n))  # nA/cm^2, another row every step
    return v0, amps


def _small_cell(case, seed):
    rest = -70.0 + 10.0 * np.random.default_rng([seed, 23]).random()
    return W.desc_to_cell(W.small(1, seed=seed)[0], pop_size=case["n"], V_init=float(rest))


@lru_cache(maxsize=16)
def _cells(kind, n, lo, hi):
    """The cells of a study (the generators' own seeds); every seed of a case has other stimuli and resting voltages."""
    return W.large(n) if kind == "large" else W.uneven(n, n_range=(lo, hi))


def _batch_descs(case, seed):
    rng = np.random.default_rng([seed, 19])
    out = []
    for d in _cells(case["kind"], case["n"], case.get("lo", 50), case.get("hi", 2000)):
        f, rest = rng.uniform(0.7, 1.3), rng.uniform(-70.0, -62.0)
        out.append(replace(d, v_rest=float(rest), pulses=[(b, x, on, off, a * f) for b, x, on, off, a in d.pulses]))
    return out


def _neuron(pop, clamp):
    soma = Branch.from_lengths(lengths=[20.0], radii=[10.0, 10.0], type="soma")
    m = Morphology.from_root(soma, name="soma")
    for k in range(3):
        m.attach(parent="soma", parent_x=1.0, child_name=f"d{k}",
                 child_branch=Branch.from_lengths(lengths=[80.0], radii=[1.0, 0.6], type="basal_dendrite"))
    c = braincell_gb300.Cell(m, cv_policy=CVPerBranch(), pop_size=pop)
    c.paint(AllRegion(), CableProperty(), Channel("IL", g_max=0.3, E=-70.0), Channel("Na_Ba2002", g_max=120.0),
            Channel("KDR_Ba2002", g_max=36.0))
    if clamp:
        c.place(RootLocation(0.5), CurrentClamp(delay=1.0, durations=40.0, amplitudes=clamp))
    c.place(RootLocation(0.5), ExpSyn(tau=2.0, e=0.0, weight=0.05, name="ampa"))
    c.place(RootLocation(0.5), StateProbe())
    return c


def _network(case, seed):
    rng = np.random.default_rng([seed, 13])
    n = case["n"]
    nd = max(1, n // 8)
    ne = n - nd
    pops, cons = [], []
    # four driver groups with different clamps, then the driven cells
    sizes = [nd // 4 + (k < nd % 4) for k in range(4)]
    names = []
    for k, s in enumerate(sizes):
        if s:
            pops.append(Population(f"drv{k}", _neuron(s, 1.2 + 0.2 * k + float(rng.uniform(0.0, 0.1)))))
            names.append((f"drv{k}", s))
    pops.append(Population("exc", _neuron(ne, 0.0)))
    for name, s in names:
        m = max(1, 8 * ne // len(names))
        cons.append(Connection(name, "exc", rng.integers(0, s, m), rng.integers(0, ne, m), synapse="ampa",
                               weight=rng.uniform(0.02, 0.08, m), delay=rng.uniform(1.0, 6.0, m)))
    m = 2 * ne
    cons.append(Connection("exc", "exc", rng.integers(0, ne, m), rng.integers(0, ne, m), synapse="ampa",
                           weight=rng.uniform(0.0, 0.02, m), delay=rng.uniform(1.5, 8.0, m)))
    return Network(pops, cons)


def _port_inputs(case, seed):
    model = S.load_model(S.PACKAGED_MODEL)
    red, ports = [], []
    for d in _batch_descs(case, seed):
        r, p = S.reduce_desc(d, model.cut_depth)
        red.append(r)
        ports.append(p)
    return model, S.ports_to_batch(red, ports)


def _gru_inputs(case, seed):
    n, T = case["n"], case["steps"]
    rng = np.random.default_rng([seed, 17])
    x = rng.normal(size=(n, T, 4)).astype(np.float32)
    y = rng.normal(scale=0.5, size=(n, T)).astype(np.float32)
    return init_params(seed), x, y


# ------------------------------------------------------------------------------------------------ passes
def prepare(case, seed):
    kind = case["kind"]
    if kind == "single":
        v0, amps = _single_inputs(case, seed)
        sc = SingleCompartment(case["n"], V_initializer=v0, **_HH)
        sc.init_state()
        return {"kind": kind, "sc": sc, "amps": amps, "k": 0}
    if kind in ("update", "cellrun"):
        cell = _small_cell(case, seed)
        cell.init_state()
        return {"kind": kind, "cell": cell, "steps": case.get("steps", 1)}
    if kind in ("batch", "large"):
        batch = W.descs_to_batch(_batch_descs(case, seed))
        prec = case.get("precision", "f32")
        kw = SHAPE if case.get("shape", 1) else {}
        return {"kind": kind, "plan": Plan(batch, precision=prec, record_every=0, **kw), "steps": case["steps"],
                "dtype": np.float64 if prec == "f64" else np.float32}
    if kind == "network":
        net = _network(case, seed)
        net.init_state()
        return {"kind": kind, "net": net, "steps": case["steps"]}
    if kind == "ports":
        model, batch = _port_inputs(case, seed)
        plan = Plan(batch, record_every=0, tile_nodes=S.PORT_TILE_NODES, lane_nodes=S.PORT_LANE_NODES,
                    tile_order=S.PORT_TILE_ORDER, threads_per_tile=S.PORT_THREADS, threads_big=S.PORT_THREADS,
                    threads_global=S.PORT_THREADS)
        plan.set_surrogate(model.theta, model.norm())
        return {"kind": "batch", "plan": plan, "steps": case["steps"], "dtype": np.float32}
    theta, x, y = _gru_inputs(case, seed)
    tr = GRUTrainer(x, y, theta, batch=case["n"], window=case["steps"], seed=seed)
    tr._set_batch(np.arange(case["n"]))
    return {"kind": kind, "tr": tr, "n": case["n"], "steps": case["steps"]}


def run(state):
    kind = state["kind"]
    if kind == "single":
        sc = state["sc"]
        amps = state["amps"][state["k"] % 8]
        state["k"] += 1
        with environ.context(dt=DT):
            spike = sc.update(amps)
        return {"spike": spike, "V": sc.V.astype(np.float32)}
    if kind == "update":
        cell = state["cell"]
        with environ.context(dt=DT):
            spike = cell.update()
        return {"spike": spike, "V": cell.V.astype(np.float32)}
    if kind == "cellrun":
        cell = state["cell"]
        cell.reset_state()
        res = cell.run(dt=DT, duration=(state["steps"] - 0.5) * DT)
        return {"trace": [t.astype(np.float32) for t in res.traces.values()], "V": cell.V.astype(np.float32)}
    if kind in ("batch", "large"):
        plan = state["plan"]
        plan.reset()
        plan.run(state["steps"], DT)
        return {"V": plan.state("V").astype(state["dtype"], copy=False)}
    if kind == "network":
        net = state["net"]
        plan = net._plan
        plan.reset()
        net.run(dt=DT, duration=state["steps"] * DT)
        return {"V": plan.state("V").astype(np.float32), "g": net.synapse_g().astype(np.float32)}
    tr, n, T = state["tr"], state["n"], state["steps"]
    tr.h.zero_()
    tr.loss.zero_()
    tr.grads.zero_()
    tr.forward_window(n, 0, T)
    tr.backward_window(n, 0, T)
    return {"y": tr.yout, "grads": tr.grads, "h": tr.h, "loss": tr.loss.float()}


# ------------------------------------------------------------------------------------------------ work
def _mean_cv(lo, hi):
    return (hi - lo) / math.log(hi / lo)


def work(case):
    """Bytes: per compartment its voltage pair and gates once in and once out, its coefficients once, the result once.
    Operations: the steps' arithmetic, an exponential or a division counted as one operation (14 for the solve of a
    compartment, about 30 a gate, 20 for the currents)."""
    kind, n, steps = case["kind"], case["n"], case.get("steps", 1)
    if kind == "single":
        return {"bytes": n * (2 * (8 + 3 * 4) + 16 + 8 + 12), "flops": n * (3 * 45 + 30)}
    if kind in ("update", "cellrun"):
        cv = 113 * n
        return {"bytes": cv * (2 * (8 + 8) + 16 + 12) + (4 * n * steps if kind == "cellrun" else 0),
                "flops": cv * steps * 94}
    if kind == "batch":
        cv, r = n * _mean_cv(case["lo"], case["hi"]), 8 if case["precision"] == "f64" else 4
        return {"bytes": cv * r * (2 * (2 + 3) + 4 + 1), "flops": cv * steps * 124}
    if kind == "large":
        cv = 15_000 * n
        return {"bytes": cv * 4 * (2 * (2 + 7) + 4 + 1), "flops": cv * steps * 260}
    if kind == "network":
        cv = 4 * n
        return {"bytes": cv * 4 * (2 * (2 + 3) + 4 + 1) + 10 * n * 16 + n * 8, "flops": cv * steps * 170}
    if kind == "ports":
        cv, ports = 117 * n, 4.3 * n
        gru = 2 * (3 * 64 * 64 + 4 * 3 * 64) + 64 * 20
        return {"bytes": cv * 4 * (2 * (2 + 3) + 4 + 1) + ports * 2 * 64 * 4, "flops": steps * (cv * 124 + ports * gru)}
    fwd = 2 * (3 * 64 * 64 + 4 * 3 * 64) + 64 * 20
    return {"bytes": n * steps * (16 + 4 + 4) + 2 * 14_000 * 4, "flops": 3.0 * n * steps * fwd}


# ------------------------------------------------------------------------------------------------ float64
def _exprel(x):
    return torch.where(x == 0, torch.ones_like(x), torch.expm1(x) / torch.where(x == 0, torch.ones_like(x), x))


def _ab(a, b):
    s = torch.where(a + b > 0, a + b, torch.ones_like(a + b))  # 0 where the channel is absent
    return a / s, 1.0 / s


class _Channels:
    """Gates and currents of the nodes in one list, in torch float64 (NaN-free: absent channels have g = 0)."""

    def __init__(self, P, mech):
        p = lambda name: P[:, getattr(_abi, "BC_P_" + name)]  # noqa: E731
        has = lambda name: (mech & getattr(_abi, "BC_M_" + name)) != 0  # noqa: E731
        self.p, self.has = p, has
        self.on = {k: bool(has(k).any()) for k in ("IL", "KLEAK", "NA", "KDR", "CAL", "CAT", "HCN", "AHP", "CADET", "NAHH",
                                                   "KHH")}
        g = {}
        for k in ("NA", "KDR", "CAL", "CAT", "HCN", "AHP", "NAHH", "KHH"):
            g[k] = torch.where(has(k), p(k + "_G"), torch.zeros_like(p(k + "_G")))
        g["IL"] = torch.where(has("IL"), p("IL_G"), torch.zeros_like(p("IL_G")))
        g["KLEAK"] = torch.where(has("KLEAK"), p("KLEAK_G"), torch.zeros_like(p("IL_G")))
        self.g = g
        self.cadet = has("CADET")

    def rates(self, v, ci):
        """{gate: (steady state, time constant in ms)}."""
        p, on, e = self.p, self.on, torch.exp
        r = {}
        if on["NA"]:
            vp = v - p("NA_VSH")
            i, t = _ab(1.28 / _exprel(-(vp - 13) / 4), 1.4 / _exprel((vp - 40) / 5))
            r["NA_P"] = i, t / p("NA_PHI")
            i, t = _ab(0.128 * e(-(vp - 17) / 18), 4 / (1 + e(-(vp - 40) / 5)))
            r["NA_Q"] = i, t / p("NA_PHI")
        if on["KDR"]:
            vp = v - p("KDR_VSH")
            i, t = _ab(0.16 / _exprel(-(vp - 15) / 5), 0.5 * e(-(vp - 10) / 40))
            r["KDR_P"] = i, t / p("KDR_PHI")
        if on["NAHH"]:
            vp = v - p("NAHH_VSH")
            i, t = _ab(1 / _exprel(-(vp - 5) * 0.1), 4 * e(-(vp + 20) / 18))
            r["NAHH_P"] = i, t / p("NAHH_PHI")
            i, t = _ab(0.07 * e(-(vp + 20) * 0.05), 1 / (1 + e(-(vp - 10) * 0.1)))
            r["NAHH_Q"] = i, t / p("NAHH_PHI")
        if on["KHH"]:
            vp = v - p("KHH_VSH")
            i, t = _ab(0.1 / _exprel(-(vp + 10) * 0.1), 0.125 * e(-(vp + 20) / 80))
            r["KHH_P"] = i, t / p("KHH_PHI")
        if on["CAL"]:
            w = v - p("CAL_VSH")
            r["CAL_P"] = 1 / (1 + e(-(w + 10) / 4)), (0.4 + 0.35 / torch.cosh((w + 5) / 15)) / p("CAL_PHIP")
            r["CAL_Q"] = 1 / (1 + e((w + 25) / 2)), (300 + 50 / torch.cosh((w + 40) / 9.5)) / p("CAL_PHIQ")
        if on["CAT"]:
            w = v - p("CAT_VSH")
            r["CAT_P"] = (1 / (1 + e(-(w + 59) / 6.2)),
                          (1 / (e(-(w + 132) / 16.7) + e((w + 16.8) / 18.2)) + 0.612) / p("CAT_PHIP"))
            r["CAT_Q"] = (1 / (1 + e((w + 83) / 4)),
                          torch.where(w >= -80, e(-(w + 22) / 10.5) + 28, e((w + 467) / 66.6)) / p("CAT_PHIQ"))
        if on["HCN"]:
            r["HCN_P"] = (1 / (1 + e((v + 75) / 5.5)),
                          1 / (e(-0.086 * v - 14.59) + e(0.0701 * v - 1.87)) / p("HCN_PHI"))
        if on["AHP"]:
            i, t = _ab(p("AHP_ALPHA") * ci ** p("AHP_N"), p("AHP_BETA"))
            r["AHP_P"] = i, t / p("AHP_PHI")
        return r

    def start(self, v):
        self.ci = self.p("CA_CI0").clone()
        self.x = {k: i.clone() for k, (i, _) in self.rates(v, self.ci).items()}

    def e_ca(self):
        if not self.on["CADET"]:
            return self.p("ECA")
        nernst = 1e3 * 8.314462618 / (2 * 96485.33212) * self.p("CA_TEMP") * torch.log(self.p("CA_CO") / self.ci)
        return torch.where(self.cadet, nernst, self.p("ECA"))

    def currents(self, v):
        """(G, I) in mS/cm^2 and uA/cm^2, and the calcium current."""
        p, on, g, x = self.p, self.on, self.g, self.x
        G, cur = torch.zeros_like(v), torch.zeros_like(v)

        def add(gg, E):
            nonlocal G, cur
            G = G + gg
            cur = cur + gg * (E - v)

        add(g["IL"], p("IL_E"))
        add(g["KLEAK"], p("EK"))
        if on["NA"]:
            add(g["NA"] * x["NA_P"] ** 3 * x["NA_Q"], p("ENA"))
        if on["KDR"]:
            add(g["KDR"] * x["KDR_P"] ** 4, p("EK"))
        if on["NAHH"]:
            add(g["NAHH"] * x["NAHH_P"] ** 3 * x["NAHH_Q"], p("ENA"))
        if on["KHH"]:
            add(g["KHH"] * x["KHH_P"] ** 4, p("EK"))
        ica = torch.zeros_like(v)
        eca = self.e_ca()
        for k in ("CAL", "CAT"):
            if on[k]:
                gg = g[k] * x[k + "_P"] ** 2 * x[k + "_Q"]
                add(gg, eca)
                ica = ica + gg * (eca - v)
        if on["HCN"]:
            add(g["HCN"] * x["HCN_P"], p("HCN_E"))
        if on["AHP"]:
            add(g["AHP"] * x["AHP_P"] ** 2, p("EK"))
        return G, cur, ica

    def advance(self, v, ica, dt):
        """Calcium from the step-start calcium current, then every gate at the new voltage (exp-Euler)."""
        p = self.p
        if self.on["CADET"]:
            drive = torch.clamp(ica * (10 / (2 * 96485.33212)) / p("CA_D"), min=0.0)
            f = drive + (p("CA_CREST") - self.ci) / p("CA_TAU")
            new = self.ci - torch.expm1(-dt / p("CA_TAU")) * p("CA_TAU") * f
            self.ci.copy_(torch.where(self.cadet, new, self.ci))
        for k, (i, t) in self.rates(v, self.ci).items():
            self.x[k].copy_(self.x[k] - torch.expm1(-dt / t) * (i - self.x[k]))


def _tree(b):
    """Point tree of a batch with one frustum per branch, children at x = 1 of their parents: per compartment a node
    (first, in compartment order), then per branch its end point, then per cell its root point."""
    ncv = b.branch_ncv.astype(np.int64)
    nb, nc = ncv.size, b.n_cells
    cell_of_branch = np.repeat(np.arange(nc), np.diff(b.cell_branch_offsets))
    n_cv = int(ncv.sum())
    br = np.repeat(np.arange(nb), ncv)
    first = np.concatenate([[0], np.cumsum(ncv)[:-1]])
    k = np.arange(n_cv) - first[br]
    rp, rd, L = b.seg_r_prox, b.seg_r_dist, b.seg_length
    region = cell_of_branch * b.n_regions + b.branch_region
    ra = b.region_ra[region][br]

    def half(j):  # half-compartment j of 2 ncv: (lateral area um^2, axial resistance MOhm)
        m = 2 * ncv[br]
        r0 = rp[br] + (rd[br] - rp[br]) * (j / m)
        r1 = rp[br] + (rd[br] - rp[br]) * ((j + 1) / m)
        s = L[br] / m
        return np.pi * (r0 + r1) * np.sqrt(s ** 2 + (r1 - r0) ** 2), ra * s / (np.pi * r0 * r1) * 1e-2

    a0, r0 = half(2 * k)
    a1, r1 = half(2 * k + 1)
    area = a0 + a1
    end = n_cv + np.arange(nb)                       # end point of each branch
    root = n_cv + nb + np.arange(nc)                 # root point of each cell
    n = n_cv + nb + nc
    parent = np.full(n, -1, np.int64)
    g = np.zeros(n)                                  # uS to the parent
    par_b = b.branch_parent.astype(np.int64)
    par_g = np.where(par_b >= 0, par_b + b.cell_branch_offsets[:-1][cell_of_branch], -1)
    prox = np.where(par_g >= 0, end[par_g], root[cell_of_branch])
    head = k == 0
    parent[:n_cv] = np.where(head, prox[br], np.arange(n_cv) - 1)
    g[:n_cv] = np.where(head, 1 / r0, 1 / (np.roll(r1, 1) + r0))
    last = first + ncv - 1
    parent[end] = last
    g[end] = 1 / r1[last]
    depth = np.zeros(n, np.int64)                    # node depth, branch by branch (parents precede children)
    base = np.zeros(nb, np.int64)
    level = np.zeros(nb, np.int64)
    todo = par_g < 0
    while todo.any():                                # branches by generation
        base[todo] = np.where(par_g[todo] >= 0, base[par_g[todo]] + ncv[par_g[todo]] + 1, 0)
        level[todo] = 1
        todo = (level == 0) & (par_g >= 0) & (level[np.maximum(par_g, 0)] == 1)
    depth[:n_cv] = base[br] + k + 1
    depth[end] = base + ncv + 1
    return dict(n=n, n_cv=n_cv, parent=parent, g=g, depth=depth, area=area, region=region[br], first=first, ncv=ncv, end=end,
                branch0=b.cell_branch_offsets[:-1])


def _node_at(t, cell, branch, x):
    b = t["branch0"][cell] + branch
    k = np.minimum((x * t["ncv"][b]).astype(np.int64), t["ncv"][b] - 1)
    return np.where(x >= 1.0, t["end"][b], t["first"][b] + k)


def _first_step(t):
    return np.maximum(0, np.ceil(t / DT - 1e-9)).astype(np.int64)


def _dev(a):
    return torch.as_tensor(np.ascontiguousarray(a)).cuda()


def _simulate(b, steps, *, v0=None, amps=None, gru=None, probe=None):
    """float64 staggered steps of a batch: implicit voltage (linearised currents), calcium, gates; event-driven
    synapses and GRU ports where the batch has them.  Returns V, V before the last step, synapse g, probe traces."""
    t = _tree(b)
    n, n_cv = t["n"], t["n_cv"]
    order = np.argsort(t["depth"], kind="stable")
    pos = np.empty(n, np.int64)
    pos[order] = np.arange(n)
    par = np.where(t["parent"][order] >= 0, pos[np.maximum(t["parent"][order], 0)], 0)
    cut = np.concatenate([[0], np.cumsum(np.bincount(t["depth"]))])
    levels = [(int(cut[d]), int(cut[d + 1])) for d in range(len(cut) - 1)]
    f64 = torch.float64
    par_t, g_ax = _dev(par), _dev(t["g"][order] * 1e3)                    # nS
    mid = _dev(pos[:n_cv])
    area = _dev(t["area"])
    P = _dev(b.region_params.astype(np.float64))[_dev(t["region"])]
    ch = _Channels(P, _dev(b.region_mech.astype(np.int64))[_dev(t["region"])])
    cap = area * _dev(b.region_cm)[_dev(t["region"])] * 1e-2 / DT          # nS
    base = torch.zeros(n, dtype=f64, device="cuda")
    base.index_add_(0, par_t, g_ax)               # roots carry g = 0
    base += g_ax
    v = P[:, _abi.BC_P_VREST].clone() if v0 is None else _dev(np.asarray(v0, np.float64))
    ch.start(v)
    x = torch.zeros(n, dtype=f64, device="cuda")
    x[mid] = v
    v_old = v.clone()
    step = torch.zeros((), dtype=torch.int64, device="cuda")
    npulse = b.pulse_cell.size
    if npulse:
        p_node = _dev(pos[_node_at(t, b.pulse_cell, b.pulse_branch, b.pulse_x)])
        p_on, p_off = _dev(_first_step(b.pulse_t_on)), _dev(_first_step(b.pulse_t_off))
        p_amp = _dev(b.pulse_amp if amps is None else np.asarray(amps, np.float64)) * 1e3
    nsyn = b.syn_cell.size
    if nsyn:
        s_cv = _dev(_node_at(t, b.syn_cell, b.syn_branch, b.syn_x))
        s_e, s_tau = _dev(b.syn_e), _dev(b.syn_tau)
        s_g = torch.zeros(nsyn, dtype=f64, device="cuda")
        raw = b.conn_delay / DT
        delay = np.maximum(np.where(np.abs(raw - np.rint(raw)) <= 1e-7, np.rint(raw), np.ceil(raw - 1e-12)), 1)
        ring = int(delay.max()) + 1 if delay.size else 1
        due = torch.zeros((ring, nsyn), dtype=f64, device="cuda")
        c_pre, c_post = _dev(b.conn_pre.astype(np.int64)), _dev(b.conn_post)
        c_w, c_d = _dev(b.conn_weight), _dev(delay.astype(np.int64))
        cv_cell = _dev(np.repeat(np.arange(b.n_cells), b.cell_ncv()))
    if gru is not None:
        th, norm = gru
        H = 64
        th = _dev(th.astype(np.float64))
        o = [0, 3 * H * H, 3 * H * H + 12 * H, 3 * H * H + 15 * H, 3 * H * H + 18 * H, 3 * H * H + 19 * H]
        Wh, Wx = th[o[0]:o[1]].view(3 * H, H), th[o[1]:o[2]].view(3 * H, 4)
        bx, bh, wo, bo = th[o[2]:o[3]], th[o[3]:o[4]], th[o[4]:o[5]], th[o[5]]
        q_end = _dev(pos[_node_at(t, b.port_cell, b.port_branch, np.ones(b.port_cell.size))])
        q_br = t["branch0"][b.port_cell] + b.port_branch
        q_att = _dev(t["first"][q_br] + t["ncv"][q_br] - 1)
        q_g, q_e, q_f = _dev(b.port_g) * 1e3, _dev(b.port_e), _dev(b.port_feat)
        h = torch.zeros((b.port_cell.size, H), dtype=f64, device="cuda")
    pr = None if probe is None else _dev(_node_at(t, b.probe_cell, b.probe_branch, b.probe_x))

    def one():
        if nsyn:
            s_g.add_(due.index_select(0, (step % ring).view(1))[0])
            due.index_fill_(0, (step % ring).view(1), 0.0)
        G, cur, ica = ch.currents(v)
        D, R = base.clone(), torch.zeros(n, dtype=f64, device="cuda")
        D.index_add_(0, mid, cap + area * G * 1e-2)
        R.index_add_(0, mid, cap * v + area * (cur + G * v) * 1e-2)
        if npulse:
            R.index_add_(0, p_node, torch.where((step >= p_on) & (step < p_off), p_amp, torch.zeros_like(p_amp)))
        if nsyn:
            D.index_add_(0, mid[s_cv], s_g * 1e3)
            R.index_add_(0, mid[s_cv], s_g * s_e * 1e3)
        if gru is not None:
            xin = torch.stack([(v[q_att] - q_e) / norm[0], torch.zeros_like(q_e), q_f[:, 0], q_f[:, 1]], 1)
            ax, ah = xin @ Wx.T + bx, h @ Wh.T + bh
            r = torch.sigmoid(ax[:, :H] + ah[:, :H])
            z = torch.sigmoid(ax[:, H:2 * H] + ah[:, H:2 * H])
            nn = torch.tanh(ax[:, 2 * H:] + r * ah[:, 2 * H:])
            h.copy_((1 - z) * nn + z * h)
            D.index_add_(0, q_end, q_g)
            R.index_add_(0, q_end, q_g * (q_e + norm[1] * (h @ wo + bo)))
        for lo, hi in reversed(levels[1:]):
            w = g_ax[lo:hi] / D[lo:hi]
            D.index_add_(0, par_t[lo:hi], w * g_ax[lo:hi], alpha=-1.0)
            R.index_add_(0, par_t[lo:hi], w * R[lo:hi])
        lo, hi = levels[0]
        x[lo:hi] = R[lo:hi] / D[lo:hi]
        for lo, hi in levels[1:]:
            x[lo:hi] = (R[lo:hi] + g_ax[lo:hi] * x[par_t[lo:hi]]) / D[lo:hi]
        v_old.copy_(v)
        v.copy_(x[mid])
        ch.advance(v, ica, DT)
        if nsyn:
            s_g.mul_(torch.exp(-DT / s_tau))
            fired = torch.zeros(b.n_cells, dtype=f64, device="cuda")
            fired.index_add_(0, cv_cell, ((v_old < 0) & (v >= 0)).to(f64))
            due.view(-1).index_add_(0, ((step + c_d) % ring) * nsyn + c_post, c_w * (fired[c_pre] > 0).to(f64))
        step.add_(1)

    traces = []
    # the step is recorded once as a CUDA graph (thousands of small tree-level operations) and replayed; the first
    # step runs eagerly as its warm-up
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    graph = None
    with torch.cuda.stream(side):
        for k in range(steps):
            if k == 0:
                one()
            else:
                if graph is None:
                    torch.cuda.synchronize()
                    graph = torch.cuda.CUDAGraph()
                    with torch.cuda.graph(graph, stream=side):
                        one()
                graph.replay()
            if pr is not None:
                traces.append(v[pr].clone())
    torch.cuda.synchronize()
    del graph
    return dict(V=v.cpu().numpy(), V_old=v_old.cpu().numpy(), g=s_g.cpu().numpy() if nsyn else None,
                trace=torch.stack(traces, 1).cpu().numpy() if traces else None)


def _exact_gru(case, seed):
    theta, x, y = _gru_inputs(case, seed)
    n, T, H = case["n"], case["steps"], 64
    th = torch.tensor(theta, dtype=torch.float64, device="cuda", requires_grad=True)
    xs, ys = torch.tensor(x, dtype=torch.float64, device="cuda"), torch.tensor(y, dtype=torch.float64, device="cuda")
    cut = np.cumsum([0, 3 * H * H, 12 * H, 3 * H, 3 * H, H, 1])
    Wh, Wx, bx, bh, wo, bo = (th[a:b] for a, b in zip(cut[:-1], cut[1:]))
    Wh, Wx = Wh.view(3 * H, H), Wx.view(3 * H, 4)
    h = torch.zeros((n, H), dtype=torch.float64, device="cuda")
    out = []
    ax = xs @ Wx.T + bx
    for t in range(T):
        a, c = ax[:, t], h @ Wh.T + bh
        r, z = torch.sigmoid(a[:, :H] + c[:, :H]), torch.sigmoid(a[:, H:2 * H] + c[:, H:2 * H])
        nn = torch.tanh(a[:, 2 * H:] + r * c[:, 2 * H:])
        h = (1 - z) * nn + z * h
        out.append(h @ wo + bo)
    yo = torch.stack(out, 1)
    err = ((yo - ys) ** 2).sum()
    (err / (n * T)).backward()
    return {"y": yo.detach(), "grads": th.grad, "h": h.detach(), "loss": err.detach().reshape(1)}


def exact(case, seed):
    kind = case["kind"]
    if kind == "gru":
        return _exact_gru(case, seed)
    if kind == "single":
        v0, amps = _single_inputs(case, seed)
        sc = SingleCompartment(case["n"], V_initializer=v0, **_HH)
        r = _simulate(sc.batch(v0), 1, v0=v0, amps=amps[0] * (sc.area * 1e-8))
        return {"spike": ((r["V_old"] < 0) & (r["V"] >= 0)).astype(np.float64), "V": r["V"]}
    if kind in ("update", "cellrun"):
        cell = _small_cell(case, seed)
        r = _simulate(cell.batch(), case.get("steps", 1), probe=True if kind == "cellrun" else None)
        shape = (case["n"], -1)
        if kind == "update":
            return {"spike": ((r["V_old"] < 0) & (r["V"] >= 0)).astype(np.float64).reshape(shape), "V": r["V"].reshape(shape)}
        return {"trace": [r["trace"]], "V": r["V"].reshape(shape)}
    if kind in ("batch", "large"):
        return {"V": _simulate(W.descs_to_batch(_batch_descs(case, seed)), case["steps"])["V"]}
    if kind == "network":
        r = _simulate(_network(case, seed).batch(), case["steps"])
        return {"V": r["V"], "g": r["g"]}
    model, batch = _port_inputs(case, seed)
    return {"V": _simulate(batch, case["steps"], gru=(model.theta, [float(q) for q in model.norm()]))["V"]}
