"""Runs of the surface alone: the steps between two CFL evaluations go in one
cooperative launch where every tile's block fits the device.  The same run
advanced a step at a time (each call starts inside a CFL interval and takes one
launch a step, or stops the long launch after its first step) gives the same
bits."""

import numpy as np
import pytest

from floodgb import native
from floodgb.config import load_config
from floodgb.domain import ProductionInfiltrationFields
from floodgb.exceptions import SimulationError
from floodgb.rainfall import rainfall_event
from floodgb.solver import FloodSolver
from floodgb.synthetic import make_grid_city


def _solver(n, per_cell, max_snapshots=None, rain=None, mode="full_swe"):
    sc = make_grid_city(n=n, size_m=10.0 * n, seed=n, duration_min=3.0)
    cfg = load_config(None, dict(sc.overrides, **{"solver.snapshot_interval_min": 1.0, "solver.surface_step_mode": mode,
                                               "solver.finite_check_interval_steps": 20}))
    topo = sc.city.topologies.surface_topology
    rng = np.random.default_rng(n)
    C = topo.cell_count
    fields = None
    if per_cell:
        f = [rng.uniform(lo, hi, C).astype(np.float32) for lo, hi in ((0.5, 1.0), (1e-5, 2e-5), (1e-6, 2e-6), (1e-3, 2e-3))]
        fields = ProductionInfiltrationFields(
            rainfall_multiplier=f[0], horton_f0_mps=f[1], horton_fc_mps=f[2], horton_k_per_s=f[3],
            open_fraction=np.ones_like(f[0]), active_mask=np.ones(C, bool))
    s = FloodSolver(topo, rainfall=rain or sc.rainfall, cfg=cfg, infiltration_fields=fields, infiltration_mps=1.0e-6,
                    centroids=sc.city.mesh.centroids_xy, duration_s=150.0, max_snapshots=max_snapshots)
    h = rng.uniform(0.0, 0.5, C).astype(np.float32)
    s.set_state(h, np.zeros_like(h), np.zeros_like(h))
    s.reset_clock()
    return s


# 32 cells (one partial tile), 512 (two whole tiles), 3,200 (13 tiles, a remainder),
# 33,800 (133 tiles), 160,178 (626 tiles: more than fit, a launch a step both ways);
# the local-inertial tiles read two rings of neighbours
@pytest.mark.gpu
@pytest.mark.parametrize("n", [4, 16, 40, 130, 283])
@pytest.mark.parametrize("per_cell", [False, True])
@pytest.mark.parametrize("mode", ["full_swe", "local_inertial"])
def test_a_run_equals_the_same_run_step_by_step(n, per_cell, mode):
    from floodgb.build import build_library

    build_library()
    native.load()
    if native.device_count() < 1:
        pytest.skip("no CUDA device")
    out = []
    for single in (False, True):
        s = _solver(n, per_cell, mode=mode)
        try:
            if single:
                for _ in range(70):  # past two CFL evaluations
                    s.run(s.progress().t_s + 1.0e-9)
                assert s.progress().step_count == 70
            s.run()
            out.append((s.progress(), s.get_state(wet_time=True), s.snapshots(), s.ledger()))
        finally:
            s.close()
    (p, state, snaps, led), (q, state1, snaps1, led1) = out
    assert p.error == 0 and p.step_count > 96 and p.snapshot_count >= 2
    assert (p.step_count, p.t_s, p.last_dt_s, p.cfl_eval_count) == (q.step_count, q.t_s, q.last_dt_s, q.cfl_eval_count)
    for a, b in zip((*state, *snaps), (*state1, *snaps1)):
        np.testing.assert_array_equal(a, b)
    assert led == led1


@pytest.mark.gpu
def test_an_error_of_the_planner_stops_the_long_launch():
    from floodgb.build import build_library

    build_library()
    native.load()
    if native.device_count() < 1:
        pytest.skip("no CUDA device")
    a, b = _solver(16, False, max_snapshots=1), _solver(16, False)
    try:
        h, hu, hv = a.get_state()[:3]
        with pytest.raises(SimulationError, match="snapshots"):
            a.run()  # the snapshot at 60 s, after the one of the start
        assert a.progress().error != 0
        with pytest.raises(SimulationError, match="snapshots"):
            a.run()
        a.set_state(h, hu, hv)
        a.reset_clock()
        a.run(50.0)  # the solver stays usable
        b.run(50.0)
        assert a.progress().error == 0 and a.progress().step_count == b.progress().step_count
        for x, y in zip(a.get_state(), b.get_state()):
            np.testing.assert_array_equal(x, y)
    finally:
        a.close()
        b.close()


@pytest.mark.gpu
@pytest.mark.parametrize("single", [False, True])
def test_a_non_finite_depth_is_reported_at_its_step(single):
    from floodgb.build import build_library

    build_library()
    native.load()
    if native.device_count() < 1:
        pytest.skip("no CUDA device")
    # beyond float32: an infinite rain depth from the first step, checked at step 20
    s = _solver(16, False, rain=rainfall_event(np.array([0.0]), np.array([60.0]), np.array([1.0e46])))
    try:
        with pytest.raises(SimulationError, match="Non-finite depth detected at step 20 "):
            if single:
                for _ in range(40):
                    s.run(s.progress().t_s + 1.0e-9)
            s.run()
        p = s.progress()
        assert p.error != 0 and p.error_step == 20
        with pytest.raises(SimulationError):
            s.run()
    finally:
        s.close()
