"""The planning work this library is used for, as timed cases.

Four kinds, each through the public Python entry points (the C ABI underneath):

  propagate  `propagate_samples`: parent states and draws in, end states,
             verdicts and region ids out -- the inner layer of every plan, and
             the entry of a program that keeps its own tree
  plan       `KGMT.plan`: one query planned alone, its tree left on the device
             and its path on the host, as the reference's callers use it
  batch      `BatchPlanner.plan`: many independent queries in one call, the
             path of every solved query read back
  served     `Server`: a burst of queries submitted, stepped until all are done

Sizes come from the repository's configurations (kgmt_gb300/config.py) and
workloads (kgmt_gb300/workloads.py).  Scenes are seeded and synthetic.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from kgmt_gb300.config import (DI_RULE_REFERENCE, MAX_SAMPLE_DIM, MODEL_DOUBLE_INTEGRATOR, MODEL_DUBINS_AIRPLANE,
                               MODEL_QUADROTOR, MODEL_UNICYCLE, double_integrator_batched,
                               double_integrator_single, dubins_airplane, quadrotor_large, unicycle)
from kgmt_gb300.planner import KGMT, BatchPlanner, Server, pack_configs, propagate_samples
from kgmt_gb300._abi import KgmtResult

DEV = "cuda"
MODELS = {"unicycle": (MODEL_UNICYCLE, unicycle), "di": (MODEL_DOUBLE_INTEGRATOR, double_integrator_single),
          "dubins": (MODEL_DUBINS_AIRPLANE, dubins_airplane), "quad": (MODEL_QUADROTOR, quadrotor_large)}


def listed():
    return [
        # -- the propagation layer, one case per model, smallest to largest --
        # a handful of candidate edges checked against a sparse scene: the smallest call there is
        {"name": "propagate_di_1000", "kind": "propagate", "model": "di", "n": 1000, "obstacles": 10, "rule": 0},
        # one node past a power of two, planar workspace and planar boxes
        {"name": "propagate_unicycle_8193", "kind": "propagate", "model": "unicycle", "n": 8193, "obstacles": 10, "rule": 0},
        # an ordinary frontier expansion in a scene of the batched workload's density
        {"name": "propagate_dubins_49999", "kind": "propagate", "model": "dubins", "n": 49999, "obstacles": 50, "rule": 0},
        # a late iteration of the large quadrotor plan (2M-node tree, 200 boxes)
        {"name": "propagate_quad_1m", "kind": "propagate", "model": "quad", "n": 1 << 20, "obstacles": 200, "rule": 0},
        # -- one query planned alone: each model with its own configuration --
        # the planar car: a few small iterations, all latency
        {"name": "plan_unicycle", "kind": "plan", "model": "unicycle", "obstacles": 10, "capacity": 100_000, "spn": 4, "coarse": 8, "fine": 4},
        # the double integrator, T = 100k: the plain form of the benchmark
        {"name": "plan_di", "kind": "plan", "model": "di", "obstacles": 10, "capacity": 100_000, "spn": 4, "coarse": 8, "fine": 2},
        # the Dubins airplane, T = 200k
        {"name": "plan_dubins", "kind": "plan", "model": "dubins", "obstacles": 10, "capacity": 200_000, "spn": 4, "coarse": 8, "fine": 2},
        # the large quadrotor query: T = 2M, 200 boxes, 8 samples a node
        {"name": "plan_quad_2m", "kind": "plan", "model": "quad", "obstacles": 200, "capacity": 2_000_000, "spn": 8, "coarse": 16, "fine": 4},
        # -- many queries in one call --
        # the benchmark's batch: 256 double-integrator queries, 50 boxes each, T = 50k
        {"name": "batch_di_256", "kind": "batch", "mix": "di", "queries": 256, "obstacles": 50, "capacity": 50_000},
        # a small odd-sized batch of all four models
        {"name": "batch_models_61", "kind": "batch", "mix": "models", "queries": 61, "obstacles": 50, "capacity": 20_000},
        # the heterogeneous batch: half double integrator, half quadrotor, 5..1000 boxes,
        # grids 8^3..32^3, T 10k..500k
        {"name": "batch_mixed_256", "kind": "batch", "mix": "mixed", "queries": 256, "obstacles": 1000, "capacity": 500_000},
        # -- continuous batching --
        # a burst of the heterogeneous set through a server with fewer slots than queries
        {"name": "served_mixed_120", "kind": "served", "mix": "mixed", "queries": 120, "slots": 96, "obstacles": 1000, "capacity": 200_000},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["propagate", "propagate", "plan", "plan", "batch", "served"])
    if kind == "propagate":
        model = rng.choice(sorted(MODELS))
        return {"kind": kind, "model": model, "n": _log(rng, 100, 1 << 20), "obstacles": _log(rng, 1, 200),
                "rule": rng.choice([0, 0, 1]) if model == "di" else 0}
    if kind == "plan":
        model = rng.choice(sorted(MODELS))
        cap = _log(rng, 10_000, 2_000_000 if model == "quad" else 200_000)
        return {"kind": kind, "model": model, "obstacles": _log(rng, 3, 200), "capacity": cap,
                "spn": rng.choice([2, 4, 8]), "coarse": rng.choice([8, 16]), "fine": rng.choice([2, 4])}
    mix = rng.choice(["di", "models", "mixed"])
    if kind == "batch":
        return {"kind": kind, "mix": mix, "queries": _log(rng, 2, 256), "obstacles": _log(rng, 10, 100 if mix != "mixed" else 1000),
                "capacity": _log(rng, 10_000, 50_000 if mix != "mixed" else 500_000)}
    n = _log(rng, 8, 120)
    return {"kind": kind, "mix": mix, "queries": n, "slots": max(4, int(n * rng.uniform(0.3, 1.2))),
            "obstacles": _log(rng, 10, 100 if mix != "mixed" else 1000), "capacity": _log(rng, 10_000, 50_000 if mix != "mixed" else 200_000)}


# ---------------------------------------------------------------------------
# scenes
# ---------------------------------------------------------------------------
def _rng(seed, salt):
    return np.random.Generator(np.random.Philox(key=(seed * 1_000_003 + salt) & 0xFFFFFFFFFFFFFFFF))


def _boxes(rng, n, start, goal, radius, dims=3):
    """n boxes in the unit workspace (rows of min xyz, max xyz), edges U[0.5, 1.5]
    of a length that keeps the filled volume near 5 % and at most 0.1, none over
    the start or the goal ball."""
    edge = min(0.1, (0.05 / n) ** (1.0 / 3.0))
    out = np.zeros((0, 6), np.float32)
    start, goal = np.asarray(start[:dims], np.float64), np.asarray(goal[:dims], np.float64)
    while len(out) < n:
        c, e = rng.uniform(0.1, 0.9, (2 * n + 8, dims)), rng.uniform(0.5, 1.5, (2 * n + 8, dims)) * edge
        lo, hi = c - e / 2, c + e / 2
        over_start = ((start >= lo - 0.01) & (start <= hi + 0.01)).all(1)
        near_goal = np.linalg.norm(np.clip(goal, lo, hi) - goal, axis=1) <= radius + 0.01
        keep = ~(over_start | near_goal)
        rows = np.zeros((int(keep.sum()), 6), np.float32)
        rows[:, 5] = 1.0  # a planar box stands for all heights
        rows[:, :dims], rows[:, 3:3 + dims] = lo[keep], hi[keep]
        out = np.concatenate([out, rows])
    return np.ascontiguousarray(out[:n])


def _start_row(model, pos):
    x = np.zeros(MAX_SAMPLE_DIM, np.float32)
    if model == MODEL_UNICYCLE:
        x[:4] = [pos[0], pos[1], math.pi / 4, 0.1]
    elif model == MODEL_DUBINS_AIRPLANE:
        x[:6] = [pos[0], pos[1], pos[2], math.pi / 4, 0.4, 0.15]
    else:
        x[:3] = pos
    return x


def _goal_row(model, pos):
    x = np.zeros(MAX_SAMPLE_DIM, np.float32)
    d = 2 if model == MODEL_UNICYCLE else 3
    x[:d] = pos[:d]
    return x


def _queries(case, seed):
    """The batch's queries: configs, start and goal rows, boxes."""
    rng = _rng(seed, 7)
    cfgs, inits, goals, boxes = [], [], [], []
    for i in range(case["queries"]):
        qseed = seed * 1_000_003 + i
        n_obs, cap = case["obstacles"], case["capacity"]
        if case["mix"] == "di":
            cfg = double_integrator_batched(qseed).replace(tree_capacity=cap)
        elif case["mix"] == "models":
            name = ("unicycle", "di", "dubins", "quad")[i % 4]
            cfg = MODELS[name][1](qseed).replace(tree_capacity=cap)
            if name == "quad":
                cfg = cfg.replace(coarse_len=8, fine_len=2)
        else:
            n_obs = max(5, int(round(math.exp(rng.uniform(math.log(5), math.log(max(6, n_obs)))))))
            coarse = int(rng.choice([8, 16, 32]))
            cap = int(round(math.exp(rng.uniform(math.log(10_000), math.log(max(10_001, cap))))))
            cfg = (quadrotor_large if i % 2 else double_integrator_single)(qseed)
            cfg = cfg.replace(tree_capacity=cap, coarse_len=coarse, fine_len=2 if coarse == 32 else int(rng.choice([2, 4])))
        start, goal = rng.uniform(0.03, 0.2, 3).astype(np.float32), rng.uniform(0.8, 0.97, 3).astype(np.float32)
        cfgs.append(cfg)
        inits.append(_start_row(cfg.model, start))
        goals.append(_goal_row(cfg.model, goal))
        boxes.append(_boxes(rng, n_obs, start, goal, cfg.goal_radius, cfg.ws_dims))
    return cfgs, np.stack(inits), np.stack(goals), boxes


def _propagate_config(case, seed):
    cfg = MODELS[case["model"]][1](seed)
    return cfg.replace(di_rule=DI_RULE_REFERENCE) if case["rule"] else cfg


def _propagate_inputs(case, seed):
    """Parent rows as a tree holds them (inside the workspace and the bounds),
    eight uniforms in (0, 1] a sample, boxes in the model's layout."""
    cfg, n = _propagate_config(case, seed), case["n"]
    g = torch.Generator(device=DEV)
    g.manual_seed(seed * 7919 + 5)
    uni = lambda lo, hi, k: lo + (hi - lo) * torch.rand((n, k), generator=g, device=DEV)  # noqa: E731
    x0 = torch.zeros((n, cfg.sample_dim), device=DEV)
    x0[:, :cfg.ws_dims] = uni(0.03, 0.97, cfg.ws_dims)
    if cfg.model == MODEL_UNICYCLE:
        x0[:, 2:3], x0[:, 3:4] = uni(-math.pi, math.pi, 1), uni(0.0, 0.3, 1)
    elif cfg.model == MODEL_DUBINS_AIRPLANE:
        x0[:, 3:4], x0[:, 4:5], x0[:, 5:6] = uni(-math.pi, math.pi, 1), uni(-0.9, 0.9, 1), uni(0.0, 0.3, 1)
    elif cfg.model == MODEL_QUADROTOR:
        x0[:, 3:6], x0[:, 6:9], x0[:, 9:12] = uni(-0.6, 0.6, 3), uni(-0.25, 0.25, 3), uni(-1.5, 1.5, 3)
    else:
        x0[:, 3:6] = uni(-0.25, 0.25, 3)
    u = 1.0 - torch.rand((n, 8), generator=g, device=DEV)
    if cfg.model == MODEL_UNICYCLE:  # steering short of +-pi/2, where its tangent has no digits left
        u[:, 1] = 0.05 + 0.9 * u[:, 1]
    rows = _boxes(_rng(seed, 11), case["obstacles"], np.float32([0.05] * 3), np.float32([0.95] * 3), cfg.goal_radius, cfg.ws_dims)
    if cfg.ws_dims == 2:
        rows = np.ascontiguousarray(rows[:, [0, 1, 3, 4]])
    return cfg, x0, u, torch.from_numpy(rows).to(DEV)


# ---------------------------------------------------------------------------
# prepare / run
# ---------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    if kind == "propagate":
        cfg, x0, u, obs = _propagate_inputs(case, seed)
        n = case["n"]
        return {"kind": kind, "cfg": cfg, "x0": x0, "u": u, "obs": obs, "n": n,
                "x1": torch.zeros((n, cfg.sample_dim), device=DEV), "valid": torch.zeros(n, dtype=torch.uint8, device=DEV),
                "r1": torch.zeros(n, dtype=torch.int32, device=DEV), "r2": torch.zeros(n, dtype=torch.int32, device=DEV)}
    if kind == "plan":
        cfg = MODELS[case["model"]][1](seed).replace(tree_capacity=case["capacity"], samples_per_node=case["spn"],
                                                     coarse_len=case["coarse"], fine_len=case["fine"])
        start, goal = np.float32([0.05] * 3), np.float32([0.95] * 3)
        rows = _boxes(_rng(seed, 13), case["obstacles"], start, goal, cfg.goal_radius, cfg.ws_dims)
        if cfg.ws_dims == 2:
            rows = np.ascontiguousarray(rows[:, [0, 1, 3, 4]])
        t, d = cfg.tree_capacity, cfg.sample_dim
        return {"kind": kind, "planner": KGMT(cfg), "init": _start_row(cfg.model, start)[:d], "goal": _goal_row(cfg.model, goal)[:d],
                "obs": torch.from_numpy(rows).to(DEV), "n_obs": len(rows), "views": None,
                "samples": torch.zeros((t, d), device=DEV), "parents": torch.zeros(t, dtype=torch.int32, device=DEV),
                "costs": torch.zeros(t, device=DEV), "path": np.zeros((cfg.max_iterations + 2, d), np.float32)}
    cfgs, inits, goals, boxes = _queries(case, seed)
    if kind == "batch":
        counts = np.array([len(b) for b in boxes], np.uint32)
        offsets = (np.cumsum(counts) - counts).astype(np.uint32)
        return {"kind": kind, "planner": BatchPlanner(len(cfgs)), "cfgs": cfgs, "carr": pack_configs(cfgs), "res": (KgmtResult * len(cfgs))(),
                "inits": inits, "goals": goals, "boxes": np.concatenate(boxes), "offsets": offsets, "counts": counts,
                "paths": np.zeros((len(cfgs), max(c.max_iterations for c in cfgs) + 2, MAX_SAMPLE_DIM), np.float32)}
    return {"kind": kind, "server": Server(max_slots=case["slots"], memory_budget=4 << 30, iters_per_step=2),
            "queries": list(zip(cfgs, inits, goals, boxes))}


class _DeviceRows:
    """A planner's device array as torch sees it."""

    def __init__(self, address, shape, kind):
        self.__cuda_array_interface__ = {"shape": shape, "typestr": kind, "data": (address, False), "version": 2}


def _tree_views(p):
    """The planner's tree (samples, parents, costs) as torch tensors of its whole capacity."""
    t, d = p.config.tree_capacity, p.config.sample_dim
    at = p.d_treeSamples_ptr_, p.d_treeSamplesParentIdxs_ptr_, p.d_treeSampleCosts_ptr_
    rows = [(at[0], (t, d), "<f4"), (at[1], (t,), "<i4"), (at[2], (t,), "<f4")]
    return at[0], [torch.as_tensor(_DeviceRows(*r), device=DEV) for r in rows]


def _whole_results(rows):
    return {k: np.array([r[k] for r in rows], np.int64) for k in ("status", "iterations", "tree_size", "goal_index", "samples_drawn")}


def run(state):
    kind = state["kind"]
    if kind == "propagate":
        s = state
        propagate_samples(s["cfg"], s["x0"], s["u"], s["obs"], s["obs"].shape[0], s["n"], s["x1"], s["valid"], s["r1"], s["r2"])
        return {"x1": s["x1"], "valid": s["valid"], "r1": s["r1"], "r2": s["r2"]}
    if kind == "plan":
        s, p = state, state["planner"]
        r = p.plan(s["init"], s["goal"], s["obs"], s["n_obs"])
        # the program keeps the tree and the path: the planner's next plan overwrites its own
        if s["views"] is None or s["views"][0] != p.d_treeSamples_ptr_:
            s["views"] = _tree_views(p)
        n, k = p.h_treeSize_, len(p.h_controlPathToGoal_)
        for name, rows in zip(("samples", "parents", "costs"), s["views"][1]):
            s[name][:n].copy_(rows[:n])
        s["path"][:k] = p.h_controlPathToGoal_
        out = {name: r[name] for name in ("status", "iterations", "tree_size", "goal_index", "path_len", "samples_drawn", "goal_cost")}
        return out | {name: s[name] for name in ("samples", "parents", "costs", "path")}
    if kind == "batch":
        s, p = state, state["planner"]
        p.plan(s["cfgs"], s["inits"], s["goals"], s["boxes"], s["offsets"], s["counts"], carr=s["carr"], res=s["res"])
        f = np.ctypeslib.as_array(s["res"])
        out = {k: f[k].astype(np.int64) for k in ("status", "iterations", "tree_size", "goal_index", "path_len", "samples_drawn")}
        for i in np.flatnonzero(out["path_len"]):
            rows = p.copy_path(int(i))
            s["paths"][i, :rows.shape[0], :rows.shape[1]] = rows
        return out | {"goal_cost": f["goal_cost"].copy(), "paths": s["paths"]}
    srv, done = state["server"], []
    tickets = [srv.submit(*q) for q in state["queries"]]
    while len(done) < len(tickets):
        srv.step()
        done += srv.poll()
    done.sort(key=lambda r: r["ticket"])
    return _whole_results(done)


# ---------------------------------------------------------------------------
# the work a pass cannot do without
# ---------------------------------------------------------------------------
# operations of one integration step (a multiply, add, compare each one), and
# the mean steps of a sample whose step count is uniform over the model's range
STEP_OPS = {"unicycle": 44, "di": 81, "dubins": 148, "quad": 662}
STEPS = {"unicycle": 5.5, "di": 3.5, "dubins": 5.5, "quad": 9.0}
DIM = {"unicycle": 7, "di": 10, "dubins": 10, "quad": 17}
# samples a query draws and nodes it keeps before it ends, typical of these
# configurations (a query of a small tree ends when the tree is full)
SAMPLES = {"unicycle": 14_000, "di": 200_000, "dubins": 130_000, "quad": 8_850_000}
NODES = {"unicycle": 3_600, "di": 23_000, "dubins": 21_000, "quad": 1_850_000}


def _query_work(model, capacity, boxes):
    nodes = min(NODES[model], capacity)
    samples = SAMPLES[model] * nodes / NODES[model]
    return {"bytes": nodes * (4 * DIM[model] + 8) + 24 * boxes, "flops": samples * STEPS[model] * STEP_OPS[model]}


def work(case):
    if case["kind"] == "propagate":
        n, m = case["n"], case["model"]
        return {"bytes": n * (4 * 2 * DIM[m] + 32 + 9) + case["obstacles"] * 24, "flops": n * STEPS[m] * STEP_OPS[m]}
    if case["kind"] == "plan":
        return _query_work(case["model"], case["capacity"], case["obstacles"])
    total = {"bytes": 0.0, "flops": 0.0}
    names = {"di": ["di"], "models": ["unicycle", "di", "dubins", "quad"], "mixed": ["di", "quad"]}[case["mix"]]
    cap, obs = case["capacity"], case["obstacles"]
    if case["mix"] == "mixed":  # the mean of a log-uniform range
        cap = (cap - 10_000) / math.log(cap / 10_000) if cap > 10_000 else cap
        obs = (obs - 5) / math.log(obs / 5) if obs > 5 else obs
    for m in names:
        w = _query_work(m, cap, obs)
        for k in total:
            total[k] += w[k] * case["queries"] / len(names)
    return total


# ---------------------------------------------------------------------------
# the propagation layer in 64 bits
# ---------------------------------------------------------------------------
def _f(v):
    """A configuration value as the planner holds it (32 bits), in 64 bits."""
    return float(np.float32(v))


def _quad_ode(c, s, u):
    phi, th, psi, uu, vv, ww, p, q, r = s[3:12]
    sp, cp, st, ct, ss, cs = phi.sin(), phi.cos(), th.sin(), th.cos(), psi.sin(), psi.cos()
    g, im, ix, iy, iz = _f(c.gravity), _f(c.mass_inv), _f(c.ix), _f(c.iy), _f(c.iz)
    drag = -_f(c.nu) * (uu * uu + vv * vv + ww * ww).sqrt()
    spin = -_f(c.mu) * (p * p + q * q + r * r).sqrt()
    return [ct * cs * uu + (sp * st * cs - cp * ss) * vv + (cp * st * cs + sp * ss) * ww,
            ct * ss * uu + (sp * st * ss + cp * cs) * vv + (cp * st * ss - sp * cs) * ww,
            -st * uu + sp * ct * vv + cp * ct * ww,
            p + (q * sp + r * cp) * st / ct, q * cp - r * sp, (q * sp + r * cp) / ct,
            r * vv - q * ww - g * st + im * drag * uu, p * ww - r * uu + g * ct * sp + im * drag * vv,
            q * uu - p * vv + g * ct * cp + im * drag * ww + im * u[0],
            (iy - iz) / ix * q * r + (u[1] + spin * p) / ix, (iz - ix) / iy * p * r + (u[2] + spin * q) / iy,
            (ix - iy) / iz * p * q + (u[3] + spin * r) / iz]


def _ode(c, s, u):
    if c.model == MODEL_QUADROTOR:
        return _quad_ode(c, s, u)
    if c.model == MODEL_DOUBLE_INTEGRATOR:
        return [s[3], s[4], s[5], u[0], u[1], u[2]]
    if c.model == MODEL_DUBINS_AIRPLANE:
        v, cp = s[5], s[4].cos()
        return [v * cp * s[3].cos(), v * cp * s[3].sin(), v * s[4].sin(), u[1], u[2], u[0]]
    return [s[3] * s[2].cos(), s[3] * s[2].sin(), s[3] / _f(c.wheelbase) * u[1].tan(), u[0]]


def _step(c, s, u, h):
    if c.model == MODEL_UNICYCLE:  # explicit Euler
        return [a + h * d for a, d in zip(s, _ode(c, s, u))]
    k1 = _ode(c, s, u)
    k2 = _ode(c, [a + 0.5 * h * d for a, d in zip(s, k1)], u)
    k3 = _ode(c, [a + 0.5 * h * d for a, d in zip(s, k2)], u)
    k4 = _ode(c, [a + h * d for a, d in zip(s, k3)], u)
    out = [a + h / 6 * (d1 + 2 * d2 + 2 * d3 + d4) for a, d1, d2, d3, d4 in zip(s, k1, k2, k3, k4)]
    if c.model == MODEL_DOUBLE_INTEGRATOR and c.di_rule == DI_RULE_REFERENCE:  # the reference's own position formula
        out[:3] = [s[j] + h / 6 * (5 * s[3 + j] + 2 * u[j] * h) for j in range(3)]
    return out


def exact(case, seed):
    """End states of the propagation layer in 64 bits, each sample stopped at
    its first step outside a bound or in a box.  A plan's tree has no such
    value: it grows by accept and reject decisions on 32-bit states, and the
    tree that 64-bit states would grow is another tree."""
    if case["kind"] != "propagate":
        return None
    c, x0, u32, obs = _propagate_inputs(case, seed)
    w, h = c.ws_dims, _f(c.step_size)
    n_state = {MODEL_UNICYCLE: 4, MODEL_QUADROTOR: 12}.get(c.model, 6)
    n_ctrl = 4 if c.model == MODEL_QUADROTOR else 3
    s = [x0[:, j].double() for j in range(n_state)]
    lo, hi = np.float32(c.u_min), np.float32(c.u_max)
    ctrl = [float(lo[j]) + u32[:, j].double() * float(hi[j] - lo[j]) for j in range(n_ctrl)]
    # the step count is a whole number that the 32-bit product decides
    k = (c.min_steps + (u32[:, n_ctrl] * float(c.max_steps - c.min_steps + 1)).int()).clamp(max=c.max_steps)
    box = obs.double()
    alive = torch.ones(case["n"], dtype=torch.bool, device=DEV)
    for i in range(c.max_steps):
        run_ = alive & (k > i)
        new = _step(c, s, ctrl, h)
        q = s[:w]
        s = [torch.where(run_, a, b) for a, b in zip(new, s)]
        ok = torch.ones_like(alive)
        for j in range(w):
            ok &= (s[j] >= _f(c.ws_min)) & (s[j] <= _f(c.ws_max))
        speeds = {MODEL_UNICYCLE: [], MODEL_DOUBLE_INTEGRATOR: [3, 4, 5], MODEL_DUBINS_AIRPLANE: [5], MODEL_QUADROTOR: [6, 7, 8]}[c.model]
        for j in speeds:
            ok &= (s[j] >= _f(c.v_min)) & (s[j] <= _f(c.v_max))
        if c.model == MODEL_DUBINS_AIRPLANE:
            ok &= (s[4] >= _f(c.pitch_min)) & (s[4] <= _f(c.pitch_max))
        bb = [(torch.minimum(q[j], s[j]), torch.maximum(q[j], s[j])) for j in range(w)]
        for o in range(box.shape[0]):
            hit = torch.ones_like(alive)
            for j in range(w):
                hit &= (bb[j][1] > box[o, j]) & (box[o, w + j] > bb[j][0])
            ok &= ~hit
        alive &= ~run_ | ok
    cols = {MODEL_UNICYCLE: [0, 1, 2], MODEL_DOUBLE_INTEGRATOR: [0, 1, 2], MODEL_DUBINS_AIRPLANE: [1, 2, 0], MODEL_QUADROTOR: [0, 1, 2, 3]}[c.model]
    rows = s + [ctrl[j] for j in cols]
    if c.model != MODEL_UNICYCLE:
        rows.append(h * k.double())
    return {"x1": torch.stack(rows, 1), "valid": None, "r1": None, "r2": None}
