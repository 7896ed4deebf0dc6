"""One drainage step of the networks of test_drainage_lists (lists below, at and above
what the passes keep in registers) against the oracle's float64 step, entry by
entry: node volumes, link flows, depths and the exchange totals.  The tolerances are
those of the reference's golden pipe steps."""

import dataclasses

import numpy as np
import pytest

import oracle
from floodgb import backend, native
from floodgb.topology import TriangularPipeNetworkState
from test_drainage_lists import _city

LISTS = [(1, 1, 0), (2, 2, 2), (4, 3, 4), (5, 4, 5), (11, 6, 9)]
DT = 0.5
V_TOL = dict(rtol=1.0e-5, atol=1.0e-5)


def _case(inlets, nodes, links):
    t = _city(inlets, nodes, links, seed=11 + inlets).city.topologies
    rng = np.random.default_rng(inlets)
    flow = rng.uniform(-0.02, 0.02, len(t.pipe_topology.link_from_node_index))
    cp, V = t.coupling_topology, np.array(t.pipe_state.node_volume_m3, np.float64)
    V[0] = 0.5 * float(cp.node_storage_area_m2[0]) * float(cp.node_max_depth_m[0])  # neither full nor empty after the step
    return t, np.asarray(t.surface_state.h_m), V, flow


def _without_inlet(cp, k):
    keep = np.arange(len(cp.inlet_cell_index)) != k
    per_inlet = {f.name: np.asarray(getattr(cp, f.name))[keep] for f in dataclasses.fields(cp)
                 if f.name.startswith("inlet_") and np.ndim(getattr(cp, f.name)) == 1
                 and len(getattr(cp, f.name)) == len(keep)}
    return dataclasses.replace(cp, **per_inlet)


@pytest.mark.parametrize("inlets,nodes,links", LISTS)
def test_an_entry_left_out_shows(inlets, nodes, links):
    """The oracle without the altered node's last inlet, or with its last link's ends
    joined (it carries nothing): the node's volume leaves the tolerance."""

    t, h, V, Q = _case(inlets, nodes, links)
    cp, pp = t.coupling_topology, t.pipe_topology
    whole = oracle.pipe_step(t.surface_topology, cp, pp, h, V, Q, DT)[1][0]
    off = [oracle.pipe_step(t.surface_topology, _without_inlet(cp, inlets - 1), pp, h, V, Q, DT)[1][0]]
    if links:
        frm, to = pp.link_from_node_index.copy(), pp.link_to_node_index.copy()
        frm[links - 1] = to[links - 1] = 50
        off.append(oracle.pipe_step(t.surface_topology, cp, dataclasses.replace(pp, link_from_node_index=frm, link_to_node_index=to),
                                    h, V, Q, DT)[1][0])
    for v in off:
        assert abs(v - whole) > 20 * (V_TOL["atol"] + V_TOL["rtol"] * abs(whole))


@pytest.mark.gpu
@pytest.mark.parametrize("inlets,nodes,links", LISTS)
def test_a_step_matches_the_oracle_entry_by_entry(inlets, nodes, links):
    from floodgb.build import build_library

    build_library()
    native.load()
    if native.device_count() < 1:
        pytest.skip("no CUDA device")
    t, h, V, Q = _case(inlets, nodes, links)
    want_h, want_v, want_q, want_diag = oracle.pipe_step(t.surface_topology, t.coupling_topology, t.pipe_topology, h, V, Q, DT)
    got_h, state, diag = backend.step_triangular_dynamic_pipe_network(
        h, t.surface_topology, t.coupling_topology, t.pipe_topology, TriangularPipeNetworkState(V, Q), DT)
    np.testing.assert_allclose(state.node_volume_m3, want_v, **V_TOL)
    np.testing.assert_allclose(state.link_flow_m3ps, want_q, rtol=1.0e-4, atol=1.0e-5)
    home = int(t.coupling_topology.node_surface_cell_index[0])
    np.testing.assert_allclose(got_h, want_h, rtol=1.0e-5, atol=1.0e-6)
    assert abs(float(got_h[home]) - float(want_h[home])) <= 1.0e-5 * float(want_h[home]) + 1.0e-6
    got = [diag.surface_capture_m3, diag.surface_surcharge_m3, diag.link_abs_flow_m3, diag.outfall_discharge_m3,
           diag.overflow_surcharge_m3, diag.unreturned_overflow_m3, diag.final_node_volume_m3]
    np.testing.assert_allclose(got, want_diag, rtol=1.0e-5, atol=1.0e-4)
