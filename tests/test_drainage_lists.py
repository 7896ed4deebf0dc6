"""The drainage passes keep the first entries of each item's list in registers
(four inlets or links of a node, two inlets of a cell) and read the rest as
they come: networks with lists below, at and above those lengths against the
oracle's float64 step."""

import numpy as np
import pytest

import oracle
from floodgb import native
from floodgb.config import load_config
from floodgb.solver import solver_for_city
from floodgb.synthetic import coupled_test_city


def _city(inlets_per_node, nodes_per_cell, hub_links, seed):
    """A small city whose node 0 has `inlets_per_node` inlets (all in one cell) and `hub_links`
    extra links, and whose first `nodes_per_cell` nodes overflow into one cell."""

    import dataclasses

    sc = coupled_test_city(scale=1, seed=seed, duration_min=2.0)
    topo = sc.city.topologies
    cp, pp = topo.coupling_topology, topo.pipe_topology
    cell, node = cp.inlet_cell_index.copy(), cp.inlet_node_index.copy()
    home = int(cp.node_surface_cell_index[0])
    cell[:inlets_per_node] = home
    node[:inlets_per_node] = 0
    surf = cp.node_surface_cell_index.copy()
    surf[:nodes_per_cell] = home
    frm, to = pp.link_from_node_index.copy(), pp.link_to_node_index.copy()
    inv = np.asarray(cp.node_invert_elevation_m)
    for k in range(hub_links):
        other = 20 + k
        frm[k], to[k] = (0, other) if inv[0] >= inv[other] else (other, 0)
    topo.coupling_topology = dataclasses.replace(cp, inlet_cell_index=cell, inlet_node_index=node,
                                                 node_surface_cell_index=surf)
    topo.pipe_topology = dataclasses.replace(pp, link_from_node_index=frm, link_to_node_index=to)
    h = np.zeros(sc.cell_count, np.float32)
    rng = np.random.default_rng(seed)
    act = np.asarray(topo.surface_topology.active_mask) > 0.5
    h[act] = rng.uniform(0.0, 0.3, int(act.sum()))
    topo.surface_state = dataclasses.replace(topo.surface_state, h_m=h)
    vol = np.asarray(cp.node_storage_area_m2, np.float64) * np.asarray(cp.node_max_depth_m) * rng.uniform(0, 1.1, cp.node_count)
    topo.pipe_state = dataclasses.replace(topo.pipe_state, node_volume_m3=vol)
    sc.overrides["solver.snapshot_interval_min"] = 1.0
    return sc


@pytest.mark.gpu
@pytest.mark.parametrize("inlets,nodes,links", [(1, 1, 0), (2, 2, 2), (4, 3, 4), (5, 4, 5), (11, 6, 9)])
def test_list_lengths_around_the_registers_match_the_oracle(inlets, nodes, links):
    from floodgb.build import build_library

    build_library()
    native.load()
    if native.device_count() < 1:
        pytest.skip("no CUDA device")
    sc = _city(inlets, nodes, links, seed=11 + inlets)
    cfg = load_config(None, sc.overrides)
    ref = oracle.run(sc, cfg, max_steps=10_000)
    s = solver_for_city(sc.city, sc.rainfall, cfg)
    try:
        s.run()
        prog = s.progress()
        _, depth, _, _, volume = s.snapshots()
    finally:
        s.close()
    # the run gates of the coupled tests: equal step counts within 2, depth RMSE 1e-4 m
    assert prog.error == 0 and abs(prog.step_count - ref.step_count) <= 2
    d = depth[-1].astype(np.float64) - ref.depth[-1]
    assert float(np.sqrt(np.mean(d * d))) <= 1.0e-4
    assert np.isfinite(volume).all()
