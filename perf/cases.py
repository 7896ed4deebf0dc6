"""The work that users of this framework have it do, as cases that can be timed.

Three kinds of program use it: one that steps or runs a flood solver (a single
call per step from Python, whole adaptive runs of surface-only and coupled
cities in both surface schemes), one that runs many storms together (ragged
batches, members of one city), and one that trains the learned surrogate or
screens storms with it.  Every case goes through the calls such a program
makes.  Meshes, networks and storms are the seeded synthetic ones of
``floodgb.synthetic``; initial states, storms and network inputs come from the
seed that ``prepare`` is given.

``listed`` has the named cases, ``draw`` more of the same ranges, ``prepare``
what the program holds before the call, ``run`` one pass, ``work`` the bytes
and operations a pass cannot do without, ``exact`` the outputs of a pass in 64
bits from plain torch.
"""

from __future__ import annotations

import functools
import math
import sys
from pathlib import Path

import numpy as np
import torch

ROOT = Path(__file__).resolve().parents[1]
sys.path.insert(0, str(ROOT / "gpu-urban-flood-cupy-jax_gb300"))

from floodgb import backend  # noqa: E402
from floodgb.batch import BatchSolver, Member  # noqa: E402
from floodgb.config import load_config  # noqa: E402
from floodgb.rainfall import uniform_rainfall  # noqa: E402
from floodgb.solver import members_for_city, solver_for_city  # noqa: E402
from floodgb.surrogate import ops  # noqa: E402
from floodgb.surrogate.experiment import load as load_networks  # noqa: E402
from floodgb.surrogate.model import FIN, FOUT, H, MPNN  # noqa: E402
from floodgb.surrogate.pipeline import MeshFeatures, ensemble_rollouts, rain_window, windows  # noqa: E402
from floodgb.synthetic import make_coupled_city, make_grid_city, production_workload, storm_hyetograph  # noqa: E402
from floodgb.topology import TriangularSurfaceForcing, TriangularSurfaceState  # noqa: E402

DEV = "cuda"
WEIGHTS = ROOT / "gpu-urban-flood-cupy-jax_gb300" / "floodgb" / "surrogate" / "weights" / "mpnn_grid224.npz"
PRODUCTION_TRIANGLES = 981_880
ENSEMBLE_GRIDS = (71, 158, 224, 354)  # squares per side of the ensemble's meshes: 10,082 .. 250,632 triangles
NODE_IN = 12  # network inputs per cell that are not padding
LEARNING_RATE = 1e-4


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # a program that drives the solver from Python, one step per call, on host arrays: the CFL
        # step and the surface step of the small 20,000-triangle workload
        {"name": "step_call_20k", "kind": "step", "grid": 100, "per_cell": False},
        # the small workload's adaptive run, surface only: launches and latency
        {"name": "run_grid_20k", "kind": "run", "city": "grid", "size": 100, "seconds": 300, "mode": "full_swe",
         "rule": "orifice"},
        # a small coupled city (the size that the coupled tests use)
        {"name": "run_coupled_8k", "kind": "run", "city": "coupled", "size": 8000, "seconds": 300,
         "mode": "full_swe", "rule": "orifice"},
        # the production-shaped coupled city, part of its hour: 981,880 triangles, 118,768 nodes
        {"name": "run_coupled_1m", "kind": "run", "city": "coupled", "size": PRODUCTION_TRIANGLES, "seconds": 180,
         "mode": "full_swe", "rule": "orifice"},
        # the same city with the fast routing scheme
        {"name": "run_inertial_1m", "kind": "run", "city": "coupled", "size": PRODUCTION_TRIANGLES, "seconds": 120,
         "mode": "local_inertial", "rule": "orifice"},
        # a ragged ensemble of surface-only storms: members of all four ensemble meshes in one batch
        {"name": "batch_ragged_16", "kind": "batch", "grids": "71,158,224,354", "per_size": 4, "seconds": 300},
        # storms over one coupled city as members of one solver
        {"name": "members_32k_x4", "kind": "members", "size": 32000, "members": 4, "seconds": 120},
        # one dense layer of the network: the message MLP's first product, rows gathered at both
        # ends of every dual edge of the 100,352-triangle mesh
        {"name": "edge_layer_100k", "kind": "dense", "cells": 100352, "fan": 3, "segments": 3, "n": 128, "f32": False,
         "relu": True, "residual": False},
        # one window of one storm through the network on the small mesh: latency
        {"name": "forward_20k", "kind": "forward", "grid": 100, "copies": 1, "layers": 8},
        # one window of 19 storms together on the screening mesh (1.9 M cells, 5.7 M dual edges)
        {"name": "forward_100k_x19", "kind": "forward", "grid": 224, "copies": 19, "layers": 8},
        # an optimizer step on one window of the screening mesh
        {"name": "train_100k", "kind": "train", "grid": 224, "layers": 8},
        # screening: hourly rollouts of a few storms by the two shipped networks, results on the host
        {"name": "rollouts_100k_x6", "kind": "rollouts", "grid": 224, "storms": 6, "hours": 3},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "run", "run", "batch", "members", "dense", "forward", "forward", "train", "rollouts"])
    if kind == "step":
        return {"kind": kind, "grid": _log_int(rng, 16, 354), "per_cell": rng.random() < 0.4}
    if kind == "run":
        mode = "full_swe" if rng.random() < 0.7 else "local_inertial"
        rule = rng.choice(["orifice", "weir_orifice", "capacity", "head_limited_capacity"])
        if rng.random() < 0.5:
            return {"kind": kind, "city": "grid", "size": _log_int(rng, 24, 500), "seconds": rng.randint(60, 240),
                    "mode": mode, "rule": "orifice"}
        return {"kind": kind, "city": "coupled", "size": _log_int(rng, 3000, 120000), "seconds": rng.randint(60, 240),
                "mode": mode, "rule": rule}
    if kind == "batch":
        grids = sorted(_log_int(rng, 30, 300) for _ in range(rng.randint(1, 4)))
        return {"kind": kind, "grids": ",".join(map(str, grids)), "per_size": rng.randint(1, 5),
                "seconds": rng.randint(60, 240)}
    if kind == "members":
        return {"kind": kind, "size": _log_int(rng, 3000, 48000), "members": rng.randint(2, 8),
                "seconds": rng.randint(40, 120)}
    if kind == "dense":
        f32 = rng.random() < 0.5
        return {"kind": kind, "cells": _log_int(rng, 700, 300000), "fan": rng.choice([1, 3]),
                "segments": rng.randint(1, 3), "n": rng.choice([64, 128]), "f32": f32,
                "relu": rng.random() < 0.5, "residual": f32 and rng.random() < 0.5}
    if kind == "forward":
        grid = _log_int(rng, 16, 300)
        copies = _log_int(rng, 1, max(1, min(40, 1_800_000 // (2 * grid * grid))))
        return {"kind": kind, "grid": grid, "copies": copies, "layers": rng.randint(2, 8)}
    if kind == "train":
        return {"kind": kind, "grid": _log_int(rng, 16, 224), "layers": rng.randint(2, 8)}
    return {"kind": kind, "grid": _log_int(rng, 40, 224), "storms": rng.randint(1, 6), "hours": rng.randint(1, 3)}


# ------------------------------------------------------------------ what a program keeps
def _cpu(x):
    return np.asarray(x)


@functools.lru_cache(maxsize=6)
def _grid_scenario(n, mesh_seed):
    return make_grid_city(n=n, size_m=10.0 * n, seed=mesh_seed)


@functools.lru_cache(maxsize=2)
def _coupled_scenario(size):
    if size == PRODUCTION_TRIANGLES:
        return production_workload()
    boundary = int(180 * math.sqrt(size / 4000.0))
    boundary += (3 * size + boundary) % 2
    return make_coupled_city(
        n_triangles=size, n_edges=(3 * size + boundary) // 2, n_active=int(0.83 * size), n_nodes=int(0.12 * size),
        n_links=int(0.1412 * size), n_inlets=int(0.0625 * size), n_outfalls=4, area_km2=0.0003 * size, seed=3)


def _scenario(case):
    return _grid_scenario(case["size"], 5) if case["city"] == "grid" else _coupled_scenario(case["size"])


def _run_config(case, sc):
    return load_config(None, dict(sc.overrides, **{
        "solver.duration_min": case["seconds"] / 60.0, "solver.surface_step_mode": case.get("mode", "full_swe"),
        "physics.inlet_capture_rule": case.get("rule", "orifice")}))


@functools.lru_cache(maxsize=1)
def _kept_solver(city, size, seconds, mode, rule):
    """The solver a program keeps for one city: many initial states are run with it."""

    case = {"city": city, "size": size, "seconds": seconds, "mode": mode, "rule": rule}
    sc = _scenario(case)
    return sc, solver_for_city(sc.city, sc.rainfall, _run_config(case, sc))


@functools.lru_cache(maxsize=1)
def _kept_members(size, members, seconds):
    sc = _coupled_scenario(size)
    cfg = _run_config({"seconds": seconds}, sc)
    storms = [uniform_rainfall(20.0 + 15.0 * m, 60.0) for m in range(members)]
    return sc, members_for_city(sc.city, storms, cfg)


@functools.lru_cache(maxsize=2)
def _kept_mesh(grid, copies):
    mf = MeshFeatures(make_grid_city(n=grid, size_m=1000.0, seed=11).city.topologies.surface_topology)
    return mf, (mf.graph if copies == 1 else mf.graph.replicate(copies))


@functools.lru_cache(maxsize=1)
def _kept_network(layers, grid, copies):  # (its activation buffers are kept per graph)
    return MPNN(n_layers=layers, seed=7)


@functools.lru_cache(maxsize=1)
def _shipped_networks(grid):
    return load_networks(WEIGHTS)[0]


def _generator(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def _waves(xy, gen, count=8):
    """A smooth field of unit scale on points xy [n, 2] (relative coordinates)."""

    k = torch.randn(count, 2, generator=gen, device=DEV) * 14.0
    p = torch.rand(count, generator=gen, device=DEV) * 6.2832
    return torch.sin(xy @ k.T + p).sum(1) * math.sqrt(2.0 / count)


def _wet_state(city, seed):
    """A mid-storm state in cell order: about half of the cells dry, sheets and ponds of a few
    centimetres to decimetres on the others, moving at up to a few decimetres a second."""

    gen = _generator(seed)
    topo = city.topologies.surface_topology
    xy = torch.as_tensor(_cpu(city.mesh.centroids_xy), device=DEV, dtype=torch.float32)
    xy = (xy - xy.mean(0)) / (xy.max() - xy.min())
    act = torch.ones(xy.shape[0], device=DEV)
    if topo.active_mask is not None:
        act = (torch.as_tensor(_cpu(topo.active_mask), device=DEV) > 0.5).float()
    h = 0.05 * torch.relu(_waves(xy, gen)) + 0.1 * torch.relu(_waves(xy, gen) - 1.0)
    h = h * (0.5 + torch.rand(h.shape, generator=gen, device=DEV)) * act
    hu = 0.2 * h * _waves(xy, gen)
    hv = 0.2 * h * _waves(xy, gen)
    return [t.contiguous() for t in (h, hu, hv)]


def _wet_nodes(city, seed):
    gen = _generator(seed + 1)
    cp, pp = city.topologies.coupling_topology, city.topologies.pipe_topology
    full = torch.as_tensor(_cpu(cp.node_storage_area_m2) * _cpu(cp.node_max_depth_m), device=DEV).double()
    v = full * 0.8 * torch.rand(full.shape, generator=gen, device=DEV).double()
    q = 0.05 * torch.randn(pp.link_count, generator=gen, device=DEV).double()
    return v.contiguous(), q.contiguous()


# ------------------------------------------------------------------ prepare
def prepare(case, seed):
    return globals()["_prepare_" + case["kind"]](case, int(seed))


def run(state):
    return globals()["_run_" + state["kind"]](state)


def work(case):
    b, f = globals()["_work_" + case["kind"]](case)
    return {"bytes": float(b), "flops": float(f)}


def exact(case, seed):
    return globals()["_exact_" + case["kind"]](case, int(seed))


# -- one step per call, host arrays
def _prepare_step(case, seed):
    sc = _grid_scenario(case["grid"], 5)
    h, hu, hv = (t.cpu().numpy() for t in _wet_state(sc.city, seed))
    rain, infil = np.float32(1.4e-5), np.float32(2.0e-6)
    if case["per_cell"]:
        r = np.random.default_rng(seed)
        rain = (rain * r.uniform(0.5, 1.5, h.size)).astype(np.float32)
        infil = (infil * r.uniform(0.0, 2.0, h.size)).astype(np.float32)
    return {"kind": "step", "topo": sc.city.topologies.surface_topology, "state": TriangularSurfaceState(h, hu, hv),
            "forcing": TriangularSurfaceForcing(rainfall_rate_mps=rain, infiltration_capacity_mps=infil)}


def _run_step(s):
    dt = backend.stable_triangular_timestep_s(s["topo"], s["state"], cfl=0.85)
    new, _ = backend.step_triangular_surface(s["state"], s["topo"], s["forcing"], dt)
    return {"dt": np.float32(dt), "h": new.h_m, "hu": new.hu_m2ps, "hv": new.hv_m2ps}


def _work_step(case):
    c = 2 * case["grid"] ** 2
    # state in and out, the cell and edge tables once; the CFL pass reads state and cell length
    return c * (24 + 20 + 16 + (8 if case["per_cell"] else 0)) + 1.5 * c * 24, c * 250


def _exact_step(case, seed):
    s = _prepare_step(case, seed)
    ex = _Flow(s["topo"])
    st = [torch.as_tensor(a, device=DEV).double() for a in (s["state"].h_m, s["state"].hu_m2ps, s["state"].hv_m2ps)]
    dt = ex.stable_dt(st, 0.85)
    f = lambda a: torch.as_tensor(a, device=DEV).double()  # noqa: E731
    h, hu, hv = ex.surface_step(st, dt, f(s["forcing"].rainfall_rate_mps), f(s["forcing"].infiltration_capacity_mps))
    return {"dt": dt, "h": h, "hu": hu, "hv": hv}


# -- adaptive runs
def _prepare_run(case, seed):
    sc, solver = _kept_solver(case["city"], case["size"], case["seconds"], case["mode"], case["rule"])
    st = _wet_state(sc.city, seed)
    v, q = _wet_nodes(sc.city, seed) if solver.node_count else (None, None)
    wet = None
    if solver.kind == 1:
        wet = 1800.0 * torch.rand(st[0].shape, generator=_generator(seed + 2), device=DEV)
    out = [torch.empty_like(t) for t in st] + [torch.empty_like(t) for t in (v, q) if t is not None]
    return {"kind": "run", "city": sc.city, "solver": solver, "in": st, "nodes": (v, q), "wet": wet, "out": out}


def _run_run(s):
    solver = s["solver"]
    solver.reset_clock()
    solver.set_state(*s["in"], *s["nodes"], s["wet"])
    solver.run()
    solver.get_state_device(*s["out"])
    return s["out"]


def _step_work(cells, active, nodes, links, inlets, per_cell, steps):
    per = cells * (44 + (24 if per_cell else 0)) + 1.5 * cells * 24 + links * 68 + nodes * 48 + inlets * 16
    return per * steps, (active * 250 + links * 120 + nodes * 60) * steps


def _work_run(case):
    coupled = case["city"] == "coupled"
    cells = case["size"] if coupled else 2 * case["size"] ** 2
    steps = case["seconds"]  # about one step a second at the least (the step is at most a second)
    n = cells if coupled else 0
    return _step_work(cells, (0.83 if coupled else 1.0) * cells, 0.12 * n, 0.1412 * n, 0.0625 * n, coupled, steps)


def _exact_run(case, seed):
    s = _prepare_run(case, seed)
    sc = _scenario(case)
    fields = sc.city.infiltration_fields if s["solver"].kind == 1 else None
    ex = _Flow(sc.city.topologies.surface_topology, sc.city.topologies if s["solver"].node_count else None,
               rule=case["rule"], fields=fields, inertial=case["mode"] == "local_inertial")
    return ex.run([t.double() for t in s["in"]], s["nodes"], s["wet"], sc.rainfall, float(case["seconds"]))


# -- ragged batches
def _prepare_batch(case, seed):
    rng = np.random.default_rng(seed)
    members, states = [], []
    for n in map(int, case["grids"].split(",")):
        for _ in range(case["per_size"]):
            sc = _grid_scenario(n, 5)
            storm = uniform_rainfall(float(rng.uniform(20.0, 120.0)), 60.0)
            members.append(Member(sc.city, storm, _run_config(case, sc), float(case["seconds"])))
            states.append([t.cpu().numpy() for t in _wet_state(sc.city, int(rng.integers(1 << 20)))])
    batch = BatchSolver(members)
    for k, st in enumerate(states):
        batch.set_state(k, *st)
    return {"kind": "batch", "batch": batch, "members": members, "states": states}


def _run_batch(s):
    s["batch"].run()
    return [list(s["batch"].state(k)) for k in range(s["batch"].n)]


def _work_batch(case):
    cells = sum(2 * int(n) ** 2 for n in case["grids"].split(",")) * case["per_size"]
    return _step_work(cells, cells, 0, 0, 0, False, case["seconds"])


def _exact_batch(case, seed):
    s = _prepare_batch(case, seed)
    out = []
    for m, st in zip(s["members"], s["states"]):
        ex = _Flow(m.city.topologies.surface_topology)
        out.append(ex.run([torch.as_tensor(a, device=DEV).double() for a in st], (None, None), None, m.rainfall,
                          float(case["seconds"])))
    return out


# -- storms over one coupled city
def _prepare_members(case, seed):
    sc, solver = _kept_members(case["size"], case["members"], case["seconds"])
    per = []
    for m in range(case["members"]):
        st = _wet_state(sc.city, seed * 16 + m)
        v, q = _wet_nodes(sc.city, seed * 16 + m)
        wet = 1800.0 * torch.rand(st[0].shape, generator=_generator(seed * 16 + m + 2), device=DEV)
        per.append({"in": st, "nodes": (v, q), "wet": wet,
                    "out": [torch.empty_like(t) for t in st] + [torch.empty_like(v), torch.empty_like(q)]})
    return {"kind": "members", "solver": solver, "members": per}


def _run_members(s):
    solver = s["solver"]
    solver.reset_clock()
    for m, p in enumerate(s["members"]):
        solver.select(m).set_state(*p["in"], *p["nodes"], p["wet"])
    solver.run()
    for m, p in enumerate(s["members"]):
        solver.select(m).get_state_device(*p["out"])
    return [p["out"] for p in s["members"]]


def _work_members(case):
    c = case["size"] * case["members"]
    return _step_work(c, 0.83 * c, 0.12 * c, 0.1412 * c, 0.0625 * c, True, case["seconds"])


def _exact_members(case, seed):
    s = _prepare_members(case, seed)
    sc = _coupled_scenario(case["size"])
    ex = _Flow(sc.city.topologies.surface_topology, sc.city.topologies, fields=sc.city.infiltration_fields)
    return [ex.run([t.double() for t in p["in"]], p["nodes"], p["wet"], uniform_rainfall(20.0 + 15.0 * m, 60.0),
                   float(case["seconds"])) for m, p in enumerate(s["members"])]


# -- one dense layer
def _prepare_dense(case, seed):
    gen = _generator(seed)
    c, rows = case["cells"], case["cells"] * case["fan"]
    bf = lambda *s: torch.randn(*s, generator=gen, device=DEV).to(torch.bfloat16)  # noqa: E731
    x = bf(c, H)
    gathered = case["fan"] > 1
    # senders lie near their receiver, as in a mesh
    dst = torch.arange(rows, device=DEV, dtype=torch.int32) // case["fan"]
    src = (dst + torch.randint(-300, 301, (rows,), generator=gen, device=DEV, dtype=torch.int32)).clamp_(0, c - 1)
    segs = [(x, dst if gathered else None, H)]
    if case["segments"] > 1:
        segs.append((x, src, H) if gathered else (bf(rows, H), None, H))
    if case["segments"] > 2:
        segs.append((bf(rows, H), None, H))
    k = H * case["segments"]
    w = (torch.randn(case["n"], k, generator=gen, device=DEV) / math.sqrt(k)).to(torch.bfloat16)
    bias = torch.randn(case["n"], generator=gen, device=DEV) * 0.1
    res = torch.randn(rows, case["n"], generator=gen, device=DEV) if case["residual"] else None
    out = torch.empty(rows, case["n"], device=DEV, dtype=torch.float32 if case["f32"] else torch.bfloat16)
    return {"kind": "dense", "segs": segs, "w": w, "bias": bias, "res": res, "out": out, "relu": case["relu"]}


def _run_dense(s):
    f32 = s["out"].dtype == torch.float32
    ops.gemm(s["segs"], s["w"], bias=s["bias"], residual=s["res"], out_f32=s["out"] if f32 else None,
             out_bf16=None if f32 else s["out"], relu=s["relu"])
    return s["out"]


def _work_dense(case):
    c, rows, n = case["cells"], case["cells"] * case["fan"], case["n"]
    gathered = min(2 if case["fan"] > 1 else 0, case["segments"])
    b = rows * H * 2 * (case["segments"] - gathered) + (c * H * 2 + rows * 4 * gathered if gathered else 0)
    b += rows * n * ((4 if case["f32"] else 2) + (4 if case["residual"] else 0))
    return b, 2.0 * rows * n * H * case["segments"]


def _exact_dense(case, seed):
    s = _prepare_dense(case, seed)
    a = torch.cat([(t if r is None else t[r.long()]).double() for t, r, _ in s["segs"]], 1)
    y = a @ s["w"].double().T + s["bias"].double()
    y = torch.relu(y) if s["relu"] else y
    return y if s["res"] is None else y + s["res"].double()


# -- the network: one window forward
def _window_inputs(mf, copies, seed):
    """Inputs of one hourly window of `copies` storms (bf16 [copies * cells, 64])."""

    gen, rng, xs = _generator(seed), np.random.default_rng(seed), []
    for k in range(copies):
        h = torch.relu(torch.randn(mf.C, generator=gen, device=DEV)) * 0.04
        hu = 0.05 * h * torch.randn(mf.C, generator=gen, device=DEV)
        hv = 0.05 * h * torch.randn(mf.C, generator=gen, device=DEV)
        mm, peak, prev = rng.uniform(5, 60), rng.uniform(10, 120), rng.uniform(0, 60)
        xs.append(mf.inputs(h, hu, hv, h * 1.2, mm, peak, prev, 1.0))
    return torch.cat(xs)


def _prepare_forward(case, seed):
    mf, g = _kept_mesh(case["grid"], case["copies"])
    net = _kept_network(case["layers"], case["grid"], case["copies"])
    return {"kind": "forward", "net": net, "graph": g, "x": _window_inputs(mf, case["copies"], seed)}


def _run_forward(s):
    return s["net"].forward(s["graph"], s["x"], train=False)


def _network_work(cells, layers, weights_bytes=0):
    """Bytes and operations of one window through the network: inputs and outputs once (the dual
    graph's features and indices among the inputs); three directed dual edges per cell."""

    e = 3.0 * cells
    b = cells * (FIN * 2 + FOUT * 4 + 4) + e * (FIN * 2 + 8)
    f = 2.0 * cells * (FIN * H + H * H + H * H + H * FOUT) + 2.0 * e * (FIN * H + H * H)
    f += layers * (2.0 * e * (3 * H * H + H * H) + 2.0 * cells * (2 * H * H + H * H))
    return b, f


def _work_forward(case):
    return _network_work(2.0 * case["grid"] ** 2 * case["copies"], case["layers"])


def _weights64(net):
    return [(d.w.double(), d.b.double()) for d in net.layers()]


def _network64(wb, layers, g, x, ef):
    """The network in 64 bits; wb: its layers' weights in the order of MPNN.layers()."""

    lin = lambda p, v: v @ p[0].T + p[1]  # noqa: E731
    mlp = lambda p, q, v: lin(q, torch.relu(lin(p, v)))  # noqa: E731
    src, dst = g.src.long(), g.dst.long()
    h = mlp(wb[0], wb[1], x)
    e = mlp(wb[2], wb[3], ef)
    for k in range(layers):
        e1, e2, n1, n2 = wb[6 + 4 * k:10 + 4 * k]
        w1, b1 = e1
        # [h_i, h_j, e_ij] W^T as three products, the first two per cell
        z = (h @ w1[:, :H].T)[dst] + (h @ w1[:, H:2 * H].T)[src] + e @ w1[:, 2 * H:].T + b1
        m = lin(e2, torch.relu(z))
        a = torch.zeros_like(h).index_add(0, dst, m)
        h = h + mlp(n1, n2, torch.cat([h, a], 1))
    return mlp(wb[4], wb[5], h)


def _exact_forward(case, seed):
    s = _prepare_forward(case, seed)
    mf, _ = _kept_mesh(case["grid"], case["copies"])
    wb = _weights64(s["net"])
    with torch.no_grad():
        return torch.cat([_network64(wb, case["layers"], mf.graph, x.double(), mf.graph.ef_bf.double())
                          for x in s["x"].split(mf.C)])


# -- the network: one optimizer step
def _prepare_train(case, seed):
    mf, g = _kept_mesh(case["grid"], 1)
    gen = _generator(seed + 3)
    net = MPNN(n_layers=case["layers"], seed=seed)
    net.t = 200  # training in progress: the optimizer's moments are warm
    for d in net.layers():
        for m1, m2 in ((d.m1w, d.m2w), (d.m1b, d.m2b)):
            m1.copy_(1e-4 * torch.randn(m1.shape, generator=gen, device=DEV))
            m2.copy_(1e-6 * (0.5 + torch.rand(m2.shape, generator=gen, device=DEV)))
    yt = 0.3 * torch.randn(mf.C, 4, generator=gen, device=DEV)
    wts = (1.0 + 3.0 * torch.rand(mf.C, 4, generator=gen, device=DEV)) * mf.active_dev[:, None].float()
    return {"kind": "train", "net": net, "graph": g, "x": _window_inputs(mf, 1, seed), "target": yt, "weights": wts,
            "norm": wts.sum(), "dy": torch.zeros(mf.C, FOUT, device=DEV)}


def _flat(tensors):
    return torch.cat([t.reshape(-1) for t in tensors])


def _run_train(s):
    net, g, dy = s["net"], s["graph"], s["dy"]
    y = net.forward(g, s["x"])
    diff = y[:, :4] - s["target"]
    loss = (s["weights"] * diff * diff).sum() / s["norm"]
    dy[:, :4] = s["weights"] * diff * (2.0 / s["norm"])
    net.zero_grad()
    net.backward(g, s["x"], dy)
    net.step(LEARNING_RATE)
    layers = net.layers()
    return {"loss": loss, "y": y, "grad_w": _flat(d.gw for d in layers), "grad_b": _flat(d.gb for d in layers),
            "w": _flat(d.w for d in layers), "b": _flat(d.b for d in layers)}


def _work_train(case):
    cells = 2.0 * case["grid"] ** 2
    b, f = _network_work(cells, case["layers"])
    params = 65_000 + case["layers"] * 115_000
    return b + cells * (4 * 8 + FOUT * 4) + params * 28, 3.0 * f


def _exact_train(case, seed):
    s = _prepare_train(case, seed)
    net, g = s["net"], s["graph"]
    wb = [(w.requires_grad_(), b.requires_grad_()) for w, b in _weights64(net)]
    y = _network64(wb, case["layers"], g, s["x"].double(), g.ef_bf.double())
    diff = y[:, :4] - s["target"].double()
    loss = (s["weights"].double() * diff * diff).sum() / s["norm"].double()
    loss.backward()
    t, new_w, new_b = net.t + 1, [], []
    with torch.no_grad():
        for d, (w, b) in zip(net.layers(), wb):
            for p, m1, m2, to in ((w, d.m1w, d.m2w, new_w), (b, d.m1b, d.m2b, new_b)):
                g_ = p.grad.reshape(m1.shape)
                a = (0.9 * m1.double() + 0.1 * g_) / (1.0 - 0.9 ** t)
                v = (0.999 * m2.double() + 0.001 * g_ * g_) / (1.0 - 0.999 ** t)
                to.append(p.reshape(m1.shape) - LEARNING_RATE * a / (v.sqrt() + 1e-8))
    return {"loss": loss.detach(), "y": y.detach(), "grad_w": _flat(w.grad for w, _ in wb),
            "grad_b": _flat(b.grad for _, b in wb), "w": _flat(new_w), "b": _flat(new_b)}


# -- screening rollouts
def _prepare_rollouts(case, seed):
    mf, _ = _kept_mesh(case["grid"], 1)
    rng = np.random.default_rng(seed)
    storms = [storm_hyetograph(rng) for _ in range(case["storms"])]
    hours = [case["hours"] - 0.25 * (k % 4) for k in range(case["storms"])]  # (ragged ends, as storms have)
    return {"kind": "rollouts", "mf": mf, "nets": _shipped_networks(case["grid"]), "storms": storms,
            "seconds": [3600.0 * v for v in hours]}


def _run_rollouts(s):
    preds, spread = ensemble_rollouts(s["nets"], s["mf"], s["storms"], s["seconds"], copies=len(s["storms"]))
    return {"h": [p[1] for p in preds], "hmax": [p[2] for p in preds], "spread": np.float32(spread)}


def _work_rollouts(case):
    b, f = _network_work(2.0 * case["grid"] ** 2 * case["storms"], 8)
    return 2 * case["hours"] * b, 2 * case["hours"] * f


def _exact_rollouts(case, seed):
    s = _prepare_rollouts(case, seed)
    mf = s["mf"]
    ef, act = mf.graph.ef_bf.double(), mf.active_dev
    hs, hms, spread = [], [], []
    with torch.no_grad():
        for storm, seconds in zip(s["storms"], s["seconds"]):
            per = []
            for net in s["nets"]:
                wb = _weights64(net)
                z = torch.zeros(mf.C, device=DEV, dtype=torch.float64)
                h, hu, hv, hm, prev, got = z, z, z, z, 0.0, []
                for t0, t1 in windows(seconds):
                    depth, peak = rain_window(storm, t0, t1)
                    x = mf.static.double().clone()
                    x[:, 0], x[:, 1], x[:, 2], x[:, 3] = 10 * h, 10 * hu, 10 * hv, 10 * hm
                    x[:, 8], x[:, 9], x[:, 10], x[:, 11] = depth / 100, prev / 100, peak / 100, (t1 - t0) / 3600
                    y = _network64(wb, 8, mf.graph, x, ef)
                    hn = torch.clamp(h + y[:, 0] / 10, min=0.0) * act
                    hm = torch.maximum(hn + torch.clamp(y[:, 1], min=0.0) / 10, torch.maximum(h, hn)) * act
                    wet = (hn > 1.0e-4) & act
                    hu, hv = (torch.where(wet, y[:, k] / 10, z) for k in (2, 3))
                    h, prev = hn, depth
                    got.append(torch.stack([h, hm]))
                per.append(torch.stack(got))
            mean = sum(per) / len(per)
            hs.append(mean[:, 0])
            hms.append(mean[:, 1])
            d2 = sum(((p[:, 1] - mean[:, 1]) ** 2).sum() for p in per)
            spread.append(float(torch.sqrt(d2 / (len(per) * mean.shape[0] * max(int(act.sum()), 1)))))
    return {"h": hs, "hmax": hms, "spread": np.asarray(spread)}


# ------------------------------------------------------------------ the flood step in 64 bits
class _Flow:
    """The flood step and its adaptive loop in 64 bits: hydrostatic reconstruction with HLL
    fluxes or the local-inertial scheme, Manning friction, rain and infiltration, the velocity
    clamp, and the drainage network (inlets, links, outfalls, overflow)."""

    G, MD = 9.80665, 1.0e-5

    def __init__(self, topo, drainage=None, rule="orifice", fields=None, inertial=False):
        f = lambda a: torch.as_tensor(_cpu(a), device=DEV).double()  # noqa: E731
        i = lambda a: torch.as_tensor(_cpu(a), device=DEV).long()  # noqa: E731
        self.bed, self.n, self.area = f(topo.bed_elevation_m), f(topo.manning_n), f(topo.cell_area_m2)
        self.length = f(topo.characteristic_length_m)
        self.L, r = i(topo.edge_left_cell), i(topo.edge_right_cell)
        self.nx, self.ny, self.len = f(topo.edge_normal_x), f(topo.edge_normal_y), f(topo.edge_length_m)
        self.act = torch.ones_like(self.bed, dtype=torch.bool)
        if topo.active_mask is not None:
            self.act = f(topo.active_mask) > 0.5
        self.inner = r >= 0
        self.R = torch.where(self.inner, r, self.L)
        self.la, self.ra = self.act[self.L], self.act[self.R]
        self.ai = self.inner & self.la & self.ra
        code = i(topo.boundary_code)
        self.code = torch.where(self.inner & self.la & ~self.ra, torch.zeros_like(code), code)
        self.fields, self.inertial, self.drainage, self.rule = fields, inertial, None, rule
        if fields is not None:
            self.mult, self.f0, self.fc, self.k = map(f, (fields.rainfall_multiplier, fields.horton_f0_mps,
                                                          fields.horton_fc_mps, fields.horton_k_per_s))
        if drainage is not None:
            cp, pp = drainage.coupling_topology, drainage.pipe_topology
            self.drainage = True
            self.icell, self.inode, self.ncell = map(i, (cp.inlet_cell_index, cp.inlet_node_index,
                                                         cp.node_surface_cell_index))
            self.inv, self.sto, self.full = map(f, (cp.node_invert_elevation_m, cp.node_storage_area_m2,
                                                    cp.node_max_depth_m))
            self.full = self.full * self.sto
            self.icap, self.isur = f(cp.inlet_capture_capacity_m3ps), f(cp.inlet_surcharge_capacity_m3ps)
            self.lf, self.lt = i(pp.link_from_node_index), i(pp.link_to_node_index)
            self.llen, self.ln, self.lcap = f(pp.link_length_m), f(pp.link_manning_n), f(pp.link_flow_capacity_m3ps)
            self.dia, self.minor = f(pp.link_diameter_m), f(pp.link_minor_loss_coefficient)
            self.oarea, self.ocoef, self.otail = map(f, (pp.outfall_area_m2, pp.outfall_coefficient,
                                                         pp.outfall_tailwater_head_m))
            self.wave = float(pp.pressurized_wave_speed_mps)

    def stable_dt(self, st, cfl):
        hs = torch.clamp(st[0], min=self.MD)
        c = torch.sqrt(self.G * hs)
        if not self.inertial:
            c = torch.hypot(st[1] / hs, st[2] / hs) + c
        return float((cfl * self.length / torch.clamp(c, min=1e-12)).min())

    def _ghost(self, hl, ul, vl):
        m = ul * self.nx + vl * self.ny
        wall = (self.code == 0) | (self.code == 2)
        return (torch.where(wall, ul - 2 * m * self.nx, ul), torch.where(wall, vl - 2 * m * self.ny, vl))

    def surface_step(self, st, dt, rain, infil):
        g, md, L, R, nx, ny = self.G, self.MD, self.L, self.R, self.nx, self.ny
        z = torch.zeros((), device=DEV, dtype=torch.float64)
        hl, ul, vl = (torch.where(self.la, v[L], z) for v in st)
        gu, gv = self._ghost(hl, ul, vl)
        hr, ur, vr = (torch.where(self.ai, v[R], w) for v, w in zip(st, (hl, gu, gv)))
        zl, zr = self.bed[L], torch.where(self.ai, self.bed[R], self.bed[L])
        hl, hr, zs = torch.clamp(hl, min=0), torch.clamp(hr, min=0), torch.maximum(zl, zr)
        hls, hrs = torch.clamp(hl + zl - zs, min=0), torch.clamp(hr + zr - zs, min=0)
        side = []
        for h, a, b, hs in ((hl, ul, vl, hls), (hr, ur, vr, hrs)):
            u, v = torch.where(h > md, a / h, z), torch.where(h > md, b / h, z)
            un = torch.where(hs > md, u * nx + v * ny, z)
            p = 0.5 * g * hs * hs
            q = torch.stack([hs, u * hs, v * hs])
            side.append((un, torch.sqrt(g * hs), q, torch.stack([hs * un, q[1] * un + p * nx, q[2] * un + p * ny])))
        (unl, cl, ql, fl), (unr, cr, qr, fr) = side
        sl = torch.clamp(torch.minimum(unl - cl, unr - cr), max=0)
        sr = torch.clamp(torch.maximum(unl + cl, unr + cr), min=0)
        d = sr - sl
        ok = (d > 1e-12) & ((hls > md) | (hrs > md))
        f = torch.where(ok, (sr * fl - sl * fr + sl * sr * (qr - ql)) / torch.where(ok, d, z + 1), z)
        pl, pr = 0.5 * g * (hl * hl - hls * hls), 0.5 * g * (hr * hr - hrs * hrs)
        left = torch.stack([f[0], f[1] + pl * nx, f[2] + pl * ny]) * self.len
        right = torch.stack([f[0], f[1] + pr * nx, f[2] + pr * ny]) * self.len
        left = torch.where(~self.inner & (self.code == 4) & (left[0] < 0), z, left)
        left, right = torch.where(self.la, left, z), torch.where(self.ai, right, z)
        acc = torch.zeros(3, self.bed.numel(), device=DEV, dtype=torch.float64)
        acc.index_add_(1, L, -left)
        acc.index_add_(1, R, right)
        h = torch.clamp(st[0] + dt * acc[0] / self.area, min=0)
        u, v = st[1] + dt * acc[1] / self.area, st[2] + dt * acc[2] / self.area
        hs = torch.clamp(h, min=md)
        damp = 1 + dt * g * self.n ** 2 * torch.hypot(u, v) * hs ** (-7.0 / 3.0)
        u, v = torch.where(h > md, u / damp, z), torch.where(h > md, v / damp, z)
        return self._sources(h, u, v, dt, rain, infil)

    def inertial_step(self, st, dt, rain, infil):
        g, md, L, R, nx, ny = self.G, self.MD, self.L, self.R, self.nx, self.ny
        z = torch.zeros((), device=DEV, dtype=torch.float64)
        hl, ul, vl = (torch.where(self.la, v[L], z) for v in st)
        hr, ur, vr = (torch.where(self.ra, v[R], z) for v in st)
        bl, br = self.bed[L], self.bed[R]
        el = bl + hl
        er = torch.where(self.ai, br + hr, bl)
        flow = torch.clamp(torch.maximum(el, er) - torch.where(self.ai, torch.maximum(bl, br), bl), min=0)
        dist = torch.clamp(0.5 * (self.length[L] + self.length[R]), min=1e-6)
        man = torch.where(self.ai, 0.5 * (self.n[L] + self.n[R]), self.n[L])
        nl, nr = ul * nx + vl * ny, ur * nx + vr * ny
        old = torch.where(self.ai, 0.5 * (nl + nr), nl) * self.len
        a = torch.clamp(flow * self.len, min=1e-8)
        rad = torch.clamp(flow, min=1e-6) ** (4.0 / 3.0)
        q = (old - g * a * dt * (er - el) / dist) / (1 + g * dt * man ** 2 * old.abs() / (rad * a))
        edge = ~self.inner & self.la & ((self.code == 1) | (self.code == 4))
        q = torch.where(self.ai | edge, q, z)
        q = torch.where(edge, torch.clamp(q, min=0), q)
        zc = torch.zeros_like(self.bed)
        donor = torch.where(q >= 0, L, R)
        req = zc.index_add(0, donor, torch.where(self.ai, q.abs() * dt, z))
        vol = torch.clamp(st[0], min=0) * self.area
        scale = torch.where(req > 1e-12, torch.clamp(vol / torch.where(req > 1e-12, req, z + 1), max=1), z + 1)
        lim = torch.where(self.ai, q * scale[donor], q) * dt
        dv = zc.index_add(0, L, -lim).index_add(0, R, torch.where(self.ai, lim, z))
        inner_q = torch.where(self.inner, q, z)
        qx = zc.index_add(0, L, q * nx).index_add(0, R, inner_q * nx)
        qy = zc.index_add(0, L, q * ny).index_add(0, R, inner_q * ny)
        h = torch.clamp(st[0] + dv / self.area, min=0)
        per = torch.clamp(2 * self.area / torch.clamp(self.length, min=1e-12), min=1e-12)
        u, v = torch.where(h > md, qx / per, z), torch.where(h > md, qy / per, z)
        return self._sources(h, u, v, dt, rain, infil)

    def _sources(self, h, u, v, dt, rain, infil):
        z = torch.zeros((), device=DEV, dtype=torch.float64)
        h1 = h + torch.clamp(rain, min=0) * dt
        h2 = h1 - torch.minimum(h1, torch.clamp(infil, min=0) * dt)
        s = torch.where(h1 > self.MD, h2 / torch.clamp(h1, min=self.MD), z)
        wet = (h2 > self.MD) & self.act
        return torch.where(self.act, h2, z), torch.where(wet, u * s, z), torch.where(wet, v * s, z)

    def _requests(self, h, v):
        """Capture and surcharge rates wanted by each inlet (m^3/s)."""

        g2, z = 2 * self.G, torch.zeros_like(self.icap)
        hc = h[self.icell]
        dh = self.bed[self.icell] + hc - self.inv[self.inode] - (torch.clamp(v, min=0) / self.sto)[self.inode]
        if self.rule == "capacity":
            return self.icap, z
        if self.rule == "head_limited_capacity":
            return torch.where(dh > 0, self.icap, z), torch.where(dh < 0, self.isur, z)
        q = 0.62 * 0.04 * torch.sqrt(g2 * dh.abs()) * torch.sign(dh)
        take = torch.clamp(q, min=0)
        if self.rule == "weir_orifice":
            dep = torch.clamp(hc, min=0)
            take = torch.minimum(take, 0.45 * 0.0 * dep * torch.sqrt(g2 * dep))
        return torch.minimum(take, self.icap), torch.minimum(torch.clamp(-q, min=0), self.isur)

    def drainage_step(self, h, v, q, dt):
        g = self.G
        zn, zc = torch.zeros_like(v), torch.zeros_like(h)
        v = torch.clamp(v, min=0)
        cap, sur = (r * dt for r in self._requests(h, v))
        cf = torch.clamp(torch.clamp(h, min=0) * self.area / torch.clamp(zc.index_add(0, self.icell, cap), min=1e-12), max=1)
        sf = torch.clamp(v / torch.clamp(zn.index_add(0, self.inode, sur), min=1e-12), max=1)
        cap, sur = cap * cf[self.icell], sur * sf[self.inode]
        v = v.index_add(0, self.inode, cap - sur)
        h = h.index_add(0, self.icell, (sur - cap) / self.area[self.icell])
        # links
        d = torch.clamp(v, min=0) / self.sto
        f, t = self.lf, self.lt
        inv = torch.minimum(self.inv[f], self.inv[t])
        dep = torch.clamp(0.5 * (d[f] + d[t] + self.inv[f] + self.inv[t]) - inv, min=0)
        dia = self.dia
        rg, od = 0.5 * dia, torch.minimum(dep, dia)
        th = 2 * torch.acos(torch.clamp((rg - od) / rg, -1, 1))
        fa = 0.25 * math.pi * dia * dia
        wet = dep >= dia
        ca = torch.where(wet, fa, 0.5 * rg * rg * (th - torch.sin(th)))
        cp = torch.where(wet, math.pi * dia, rg * th)
        a = torch.clamp(ca + g * fa / self.wave ** 2 * torch.clamp(dep - dia, min=0), min=1e-12)
        rad = torch.clamp(ca / torch.clamp(cp, min=1e-12), min=1e-12)
        slope = (self.inv[f] + d[f] - self.inv[t] - d[t]) / self.llen
        fric = g * self.ln ** 2 * q.abs() / (rad ** (4.0 / 3.0) * a) + self.minor * q.abs() / (2 * self.llen * a)
        up = (q + g * a * dt * slope) / (1 + dt * fric)
        tr = torch.maximum(torch.minimum(up, self.lcap), -self.lcap) * dt
        donor = torch.where(tr >= 0, f, t)
        fac = torch.clamp(torch.clamp(v, min=0) / torch.clamp(zn.index_add(0, donor, tr.abs()), min=1e-12), max=1)
        tr = tr * fac[donor]
        v = torch.clamp(torch.clamp(v, min=0).index_add(0, f, -tr).index_add(0, t, tr), min=0)
        # outfalls, then the overflow back to the surface
        dh = self.inv + v / self.sto - self.otail
        out = self.ocoef * self.oarea * torch.sqrt(2 * g * torch.clamp(dh, min=0))
        v = v - torch.minimum(v, out * dt)
        over = torch.clamp(v - self.full, min=0) * (self.ncell >= 0)
        cell = torch.clamp(self.ncell, min=0)
        return h.index_add(0, cell, over / self.area[cell]), v - over, tr / dt

    def run(self, st, nodes, wet, rainfall, seconds):
        """The adaptive loop from t = 0: the CFL step every 32 steps (x 0.85) and 0.8 of it between,
        at most a second; returns [h, hu, hv] and, coupled, the node volumes and no link flows: the
        flow of a nearly level pipe swings with the last bits of its end volumes, so after some
        steps it has no value that rounding does not decide."""

        v, q = nodes
        v, q = (None, None) if v is None else (v.clone(), q.clone())
        wt = None if wet is None else wet.double()
        t, step, cached = 0.0, 0, 0.0
        one = torch.ones((), device=DEV, dtype=torch.float64)
        starts, ends = _cpu(rainfall.start_min) * 60.0, _cpu(rainfall.end_min) * 60.0
        rates = _cpu(rainfall.intensity_mmhr) / 3.6e6
        while t < seconds:
            if step % 32 == 0:
                cached = self.stable_dt(st, 0.85)
            dt = max(min(cached if step % 32 == 0 else 0.8 * cached, 1.0, seconds - t), 1e-3)
            now = (starts <= t) & (t < ends)
            rate = one * float(rates[now][0] if now.any() else 0.0)
            rain, infil = rate, 0.0 * one
            if self.fields is not None:
                rain, infil = rate * self.mult, self.fc + (self.f0 - self.fc) * torch.exp(-self.k * wt)
            st = (self.inertial_step if self.inertial else self.surface_step)(st, dt, rain, infil)
            h, hu, hv = st
            hm = torch.clamp(h, min=1e-8)
            lim = torch.clamp(5.0 / torch.clamp(torch.hypot(hu, hv) / hm, min=1e-12), max=1.0)
            hu, hv = hu * lim, hv * lim
            if v is not None:
                h, v, q = self.drainage_step(h, v, q, dt)
            st = (h, hu, hv)
            if wt is not None:
                wt = wt + dt * (h > self.MD)
            t, step = t + dt, step + 1
        return [*st] + ([] if v is None else [v, None])
