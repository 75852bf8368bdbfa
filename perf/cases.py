"""The work a program does with this package, as cases that can be measured.

Each case is one call, or the short sequence of calls, that a user's program
makes through the public entry points:

  count     ops.count_SEIRP over device columns: the per-node tally that a
            report or a component outside the engine asks for each tick.
  adjoint   one evaluation of an ops.IncidencePlan, the inner step of a
            calibration.  mode "target": loss and gradient against a target
            curve, as calibrate.fit_incidence asks for them; "vjp": lam and
            the gradients of sum(g * lam), the network's among them;
            "torch": lam as an autograd node, a torch loss, its gradients.
  table     SEIR_ABM(pars) with the five components: the agent table drawn
            on the device and the network built.
  run       the same, then run(): a whole simulation from its parameters to
            its results and final table.
  step      a simulation whose table is already on the device, through the
            handle: create, bind, start, every tick, results and columns.
  batch     engine.run_replicates: the replicates of one calibration trial.

Sizes are those of the package's own workloads (synthetic.py): Zamfara-like
(14 nodes, 1e6 agents, 365 days), Nigeria-like (774 nodes, 2.2e8 agents) and
continental (4000 nodes), and small ones.
"""

from __future__ import annotations

import math

import numpy as np
import torch

import laser_polio_gb300 as lp
from laser_polio_gb300 import _lib
from laser_polio_gb300 import engine
from laser_polio_gb300 import ops
from laser_polio_gb300 import synthetic

COMPONENTS = (lp.VitalDynamics_ABM, lp.DiseaseState_ABM, lp.RI_ABM, lp.SIA_ABM, lp.Transmission_ABM)
SCALARS = ("R", "amp", "peak", "k", "a", "b", "c")
BATCH_NODES = (14, 44, 120, 300)


def listed():
    return [
        # the tally of a small test population: launches and latency
        {"name": "count_14n_20k", "kind": "count", "nodes": 14, "agents": 20011, "strains": 3},
        # the tally of the Nigeria-scale table: every column read once
        {"name": "count_774n_220m", "kind": "count", "nodes": 774, "agents": 220_000_003, "strains": 3},
        # one L-BFGS evaluation for a province over a year
        {"name": "adjoint_14n_365d", "kind": "adjoint", "nodes": 14, "ticks": 365, "strains": 1, "mode": "target"},
        # the same through torch.autograd for a region, an odd window
        {"name": "adjoint_torch_300n_181d", "kind": "adjoint", "nodes": 300, "ticks": 181, "strains": 2,
         "mode": "torch"},
        # one L-BFGS evaluation at the Nigeria scale, a year, three strains
        {"name": "adjoint_774n_365d", "kind": "adjoint", "nodes": 774, "ticks": 365, "strains": 3, "mode": "target"},
        # the same at the continental scale over a quarter
        {"name": "adjoint_4000n_90d", "kind": "adjoint", "nodes": 4000, "ticks": 90, "strains": 3, "mode": "target"},
        # a Zamfara-like model built
        {"name": "table_14n_1m", "kind": "table", "nodes": 14, "agents": 1_000_000, "days": 365},
        # a Nigeria-scale model built
        {"name": "table_774n_220m", "kind": "table", "nodes": 774, "agents": 220_000_000, "days": 365},
        # a Zamfara-like year, parameters to results
        {"name": "run_14n_1m_365d", "kind": "run", "nodes": 14, "agents": 1_000_000, "days": 365},
        # a Nigeria-scale year with births, RI, campaigns and a growing epidemic
        {"name": "step_774n_220m_365d", "kind": "step", "nodes": 774, "agents": 220_000_000, "days": 365},
        # continental node count, a widespread epidemic: the mixing and the selection at their largest
        {"name": "step_4000n_200m_120d", "kind": "step", "nodes": 4000, "agents": 200_000_000, "days": 120},
        # the replicates of a calibration trial, node counts and sizes uneven
        {"name": "batch_12x_365d", "kind": "batch", "replicates": 12, "agents": 18_000_000, "days": 365},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["count", "count", "adjoint", "adjoint", "adjoint", "table", "run", "step", "step", "batch"])
    if kind == "count":
        return {"kind": kind, "nodes": _log_int(rng, 1, 4000), "agents": _log_int(rng, 5_000, 220_000_000),
                "strains": rng.randint(1, 4)}
    if kind == "adjoint":
        nodes = _log_int(rng, 5, 2500)
        return {"kind": kind, "nodes": nodes, "ticks": _log_int(rng, 20, 365 if nodes < 1000 else 120),
                "strains": rng.randint(1, 3), "mode": rng.choice(["target", "target", "vjp", "torch"])}
    if kind == "batch":
        return {"kind": kind, "replicates": rng.randint(2, 12), "agents": _log_int(rng, 500_000, 18_000_000),
                "days": rng.randint(60, 365)}
    nodes = _log_int(rng, 3, 2000)
    agents = _log_int(rng, max(20_000, 200 * nodes), 120_000_000 if kind != "run" else 40_000_000)
    return {"kind": kind, "nodes": nodes, "agents": agents, "days": rng.randint(40, 365 if agents < 30_000_000 else 120)}


# -- inputs ----------------------------------------------------------------------
def _count_state(case, seed):
    """Columns as a run leaves them: node-contiguous agents, a few per cent
    infected, the dead among them, newborns of all nodes at the end."""
    n, nodes = int(case["agents"]), int(case["nodes"])
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    u = torch.rand(n, generator=g, device="cuda")
    state = torch.full((n,), 3, dtype=torch.int8, device="cuda")
    state[u < 0.30] = 0
    state[u < 0.04] = 2
    state[u < 0.01] = 1
    state[u > 0.97] = -1
    del u
    old = n - n // 20
    node = torch.empty(n, dtype=torch.int16, device="cuda")
    weight = torch.rand(nodes, generator=g, device="cuda", dtype=torch.float64) + 0.2
    edge = (torch.cumsum(weight, 0) / weight.sum() * old).to(torch.int64)
    edge[-1] = old
    sizes = torch.diff(edge, prepend=torch.zeros(1, dtype=torch.int64, device="cuda"))
    node[:old] = torch.repeat_interleave(torch.arange(nodes, dtype=torch.int16, device="cuda"), sizes)
    node[old:] = torch.randint(0, nodes, (n - old,), generator=g, device="cuda", dtype=torch.int16)
    strain = torch.randint(0, int(case["strains"]), (n,), generator=g, device="cuda", dtype=torch.int8)
    pp = torch.full((n,), -1, dtype=torch.int8, device="cuda")
    pp[state >= 2] = torch.randint(0, 2, (n,), generator=g, device="cuda", dtype=torch.int8)[state >= 2]
    par = torch.zeros(n, dtype=torch.int8, device="cuda")
    par[(pp == 1) & (state == 3)] = 1
    return {"cols": (node, state, strain, pp, par), "nodes": nodes, "strains": int(case["strains"]), "n": n}


def _adjoint_inputs(case, seed):
    """Replayed aggregates of the shape a forward run records, the
    parameters, a target curve and an upstream gradient."""
    T, G, S = int(case["ticks"]), int(case["nodes"]), int(case["strains"])
    rng = np.random.default_rng(int(seed))
    pops = np.maximum(np.round(rng.lognormal(np.log(2.8e5), 0.7, G)), 1.0)
    xy = rng.uniform(0.0, 1000.0, (G, 2))
    dist = np.sqrt((xy[:, None, 0] - xy[None, :, 0]) ** 2 + (xy[:, None, 1] - xy[None, :, 1]) ** 2)
    dist[dist == 0] = 1.0
    np.fill_diagonal(dist, 0.0)
    pop = pops[None, :] * (1.0 + 27.0 / 365000.0) ** np.arange(T)[:, None]
    srisk = pop * rng.uniform(0.05, 0.3, G)[None, :] * rng.lognormal(-0.005, 0.1, (T, G))
    scal = np.array([1.0, 0.25, 0.125])[:S]
    infected = rng.gamma(2.0, 150.0, (T, G, S)) * (rng.uniform(size=(T, G, S)) > 0.3)
    beta = 0.6 * infected * scal[None, None, :]
    inp = {"srisk": srisk, "beta": beta, "pop": pop, "doy": (np.arange(T) % 365 + 1).astype(np.float64),
           "year": np.full(T, 365.0), "pops": pops, "dist": dist}
    par = {"R": 1.0, "amp": 0.4, "peak": 180.0, "k": 0.5, "a": 1.0, "b": 1.0, "c": 2.0, "max_frac": 0.2,
           "r0s": rng.lognormal(0.0, 0.3, G)}
    target = srisk * 1e-3 * rng.lognormal(0.0, 1.0, (T, G))
    g = rng.normal(0.0, 1.0, (T, G))
    return inp, par, target, g


def _adjoint_state(case, seed):
    inp, par, target, g = _adjoint_inputs(case, seed)
    mode = case["mode"]
    state = {"mode": mode, "plan": ops.IncidencePlan(inp, target if mode == "target" else None), "par": par, "g": g}
    if mode == "torch":
        leaf = {n: torch.tensor(par[n], dtype=torch.float64, requires_grad=True) for n in (*SCALARS, "r0s")}
        state["leaf"], state["target"] = leaf, torch.as_tensor(np.log1p(target))
    return state


def _pars(nodes, agents, days, seed):
    """Parameters of a Nigeria-like model (synthetic.nigeria_like_pars) with
    per-node immunity and a few infections in a tenth of the nodes."""
    pars, immun, rng = synthetic.nigeria_like_pars(agents, nodes, days, seed)
    prev = np.zeros(nodes, np.int64)
    prev[rng.choice(nodes, size=max(1, nodes // 10), replace=False)] = 20
    pars.update({"init_immun": list(immun), "init_prev": list(prev), "age_pyramid_path": None})
    return pars


def _build(pars):
    sim = lp.SEIR_ABM(lp.PropertySet(pars))
    sim.components = list(COMPONENTS)
    return sim


def _step_state(case, seed):
    sim = _build(_pars(case["nodes"], case["agents"], case["days"], seed))
    spec = engine.build_sim_spec(sim)
    out = {name: torch.zeros_like(t) for name, t in spec.columns.items()}
    return {"sim": sim, "spec": spec, "out": out, "res": spec.results}


def _batch_pars(case, seed):
    rng = np.random.default_rng(int(seed))
    n = int(case["replicates"])
    share = 2.0 ** (3.0 * (5 * np.arange(n) % n) / n)  # the largest replicate about eight times the smallest
    agents = np.maximum((share / share.sum() * case["agents"]).astype(np.int64), 20_000)
    out = []
    for r in range(n):
        nodes = BATCH_NODES[r % len(BATCH_NODES)]
        p = _pars(nodes, int(agents[r]), int(case["days"]), int(seed) * 1000 + r)
        p.update({"r0": float(rng.uniform(8, 20)), "seasonal_amplitude": float(rng.uniform(0.1, 0.6)),
                  "seasonal_peak_doy": int(rng.integers(0, 365)), "gravity_k": float(rng.lognormal(np.log(0.5), 0.5))})
        out.append(p)
    return out


def prepare(case, seed):
    kind = case["kind"]
    if kind == "count":
        state = _count_state(case, seed)
    elif kind == "adjoint":
        state = _adjoint_state(case, seed)
    elif kind == "step":
        state = _step_state(case, seed)
    elif kind == "batch":
        state = {"pars": _batch_pars(case, seed)}
    else:
        state = {"pars": _pars(case["nodes"], case["agents"], case["days"], seed)}
    state["kind"] = kind
    return state


# -- one pass ----------------------------------------------------------------------
def _results(sim):
    return {k: v for k, v in vars(sim.results).items() if isinstance(v, np.ndarray) and v.dtype == np.int32}


def _run_table(state):
    sim = _build(state["pars"])
    out = {"columns": sim.people.device_columns(), "network": sim.instances[-1].network}
    sim.components = []  # the model and its parts refer to each other: let go of it now
    return out


def _run_run(state):
    sim = _build(state["pars"])
    sim.run()
    out = {"results": _results(sim), "columns": sim.people.device_columns(), "count": sim.people.count}
    sim.components = []  # gives the engine's memory back
    return out


def _run_step(state):
    spec = state["spec"]
    h = _lib.Handle([spec.desc])
    h.bind_columns(0, spec.columns)
    h.start()
    h.step(spec.desc.nt - 1)
    h.sync()
    h.read_results(0, state["res"])
    h.read_columns(0, state["out"])
    h.close()
    return {"results": state["res"], "columns": state["out"]}


def _run_batch(state):
    sims = [_build(p) for p in state["pars"]]
    errors = engine.run_replicates(sims)
    if any(e is not None for e in errors):
        raise RuntimeError(f"a replicate failed: {errors}")
    out = []
    for s in sims:
        res = _results(s)
        out.append((np.concatenate([res[k].reshape(-1) for k in sorted(res)]),
                    s.people.device_columns()["disease_state"]))
        s.components = []
    return out


def _run_adjoint(state):
    plan, par = state["plan"], state["par"]
    if state["mode"] == "target":
        return plan.evaluate(par, network_grad=False)
    if state["mode"] == "vjp":
        return plan.evaluate(par, state["g"], lam=True)
    leaf = state["leaf"]
    lam = ops.expected_incidence_torch(plan, {**leaf, "max_frac": par["max_frac"]})
    loss = ((torch.log1p(lam) - state["target"]) ** 2).sum()
    grads = torch.autograd.grad(loss, list(leaf.values()))
    return {"lam": lam.detach(), "loss": loss.detach(), "grad": dict(zip(leaf, grads))}


def run(state):
    kind = state["kind"]
    if kind == "count":
        return list(ops.count_SEIRP(*state["cols"], state["nodes"], state["strains"], state["n"]))
    return {"adjoint": _run_adjoint, "table": _run_table, "run": _run_run, "step": _run_step,
            "batch": _run_batch}[kind](state)


# -- the work a pass cannot do without -------------------------------------------
SLOT_BYTES = 29  # the fifteen columns of one agent
RESULTS = 28     # int32 results per node and day, strains counted one by one (three strains)


def work(case):
    kind = case["kind"]
    if kind == "count":
        return {"bytes": 6.0 * case["agents"] + 4.0 * case["nodes"] * (6 + 2 * case["strains"]), "flops": 0.0}
    if kind == "adjoint":
        T, G, S = case["ticks"], case["nodes"], case["strains"]
        out = G if case["mode"] == "target" else T * G + G + (G * G if case["mode"] == "vjp" else 0)
        return {"bytes": 8.0 * (T * G * (2 + S) + G * G + 3 * G + out), "flops": 4.0 * T * S * G * G}
    if kind == "batch":
        days = case["days"] + 1
        return {"bytes": 2.0 * SLOT_BYTES * case["agents"] + 4.0 * RESULTS * 120 * days * case["replicates"],
                "flops": 0.0}
    slots, nodes = float(case["agents"]), float(case["nodes"])
    if kind == "table":
        return {"bytes": SLOT_BYTES * slots + 16.0 * nodes * nodes, "flops": 0.0}
    bytes_ = 8.0 * nodes * nodes + 4.0 * RESULTS * nodes * (case["days"] + 1)
    # a run writes its table; a step reads the one it is given and writes the final one
    return {"bytes": bytes_ + (2.0 if kind == "step" else 1.0) * SLOT_BYTES * slots, "flops": 0.0}


# -- the adjoint in plain numpy, 64 bits -----------------------------------------
def exact(case, seed):
    """lam, loss and gradients of an adjoint case; the other kinds return
    integers and draws, which have no value but the package's own."""
    if case["kind"] != "adjoint":
        return None
    inp, par, target, g = _adjoint_inputs(case, seed)
    beta, pops, srisk = inp["beta"], inp["pops"], inp["srisk"]
    T, G, S = beta.shape
    total = pops.sum()
    with np.errstate(divide="ignore"):
        flow = par["k"] * (pops[:, None] ** par["a"]) * (pops[None, :] ** par["b"]) / inp["dist"] ** par["c"]
    flow /= total ** par["c"]
    np.fill_diagonal(flow, 0.0)
    row = flow.sum(axis=1)
    cap = row > par["max_frac"]
    scale = np.where(cap, par["max_frac"] / np.where(cap, row, 1.0), 1.0)
    net = flow * scale[:, None]
    b2 = np.ascontiguousarray(beta.transpose(0, 2, 1)).reshape(T * S, G)
    u = (b2 * (1.0 - net.sum(axis=1))[None, :] + b2 @ net).reshape(T, S, G)
    angle = 2.0 * np.pi * (inp["doy"] - par["peak"]) / inp["year"]
    seas = 1.0 + par["amp"] * np.cos(angle)
    popc = np.maximum(inp["pop"], 1.0)
    q = seas[:, None] * par["r0s"][None, :] * par["R"] / popc
    e = np.exp(-u * q[:, None, :])
    lam = srisk * (1.0 - e).sum(axis=1)
    resid = np.log1p(lam) - np.log1p(target)
    loss = float((resid**2).sum())
    up = g if case["mode"] == "vjp" else 2.0 * resid / (1.0 + lam)
    gr = (up * srisk)[:, None, :] * e
    gu = (gr * q[:, None, :]).reshape(T * S, G)
    gq = (gr * u).sum(axis=1)
    gs = (gq * par["r0s"][None, :] * par["R"] / popc).sum(axis=1)
    gnet = b2.T @ gu - (b2 * gu).sum(axis=0)[:, None]
    np.fill_diagonal(gnet, 0.0)
    inner = np.where(cap, (gnet * flow).sum(axis=1) / np.where(cap, row, 1.0), 0.0)
    w = scale[:, None] * (gnet - inner[:, None]) * flow
    with np.errstate(divide="ignore"):
        logd = np.log(inp["dist"])
    np.fill_diagonal(logd, 0.0)
    grad = {"R": float((gq * seas[:, None] * par["r0s"][None, :] / popc).sum()),
            "amp": float((gs * np.cos(angle)).sum()),
            "peak": float((gs * par["amp"] * np.sin(angle) * 2.0 * np.pi / inp["year"]).sum()),
            "k": float(w.sum() / par["k"]),
            "a": float((w * np.log(pops)[:, None]).sum()),
            "b": float((w * np.log(pops)[None, :]).sum()),
            "c": float((w * (-logd - math.log(total))).sum()),
            "r0s": (gq * seas[:, None] * par["R"] / popc).sum(axis=0)}
    if case["mode"] == "target":
        return {"loss": loss, "grad": grad}
    if case["mode"] == "vjp":
        return {"lam": lam, "grad": {**grad, "network": gnet}}
    as64 = {n: torch.as_tensor(np.asarray(v, np.float64)) for n, v in grad.items()}
    return {"lam": torch.as_tensor(lam), "loss": torch.tensor(loss, dtype=torch.float64), "grad": as64}
