"""A finite check that fails inside a run of one launch stops the run as a launch a
step does: the step after the checked one was planned already and is done, no
other.  Clock, states and snapshots are those of a run capped at that step."""

import numpy as np
import pytest

from floodgb import native
from floodgb.config import load_config
from floodgb.domain import ProductionInfiltrationFields
from floodgb.exceptions import SimulationError
from floodgb.solver import FloodSolver
from floodgb.synthetic import make_grid_city

INTERVAL = 32


def _solver(n, mode, finite):
    sc = make_grid_city(n=n, size_m=10.0 * n, seed=n, duration_min=3.0)
    cfg = load_config(None, dict(sc.overrides, **{
        "solver.snapshot_interval_min": 0.1, "solver.surface_step_mode": mode, "solver.finite_check_interval_steps": finite,
        "solver.cfl_update_interval_steps": INTERVAL}))
    topo = sc.city.topologies.surface_topology
    C = topo.cell_count
    ones = np.ones(C, np.float32)
    mult = ones.copy()
    mult[C // 2] = np.inf  # one cell's rain depth, from the first step
    fields = ProductionInfiltrationFields(rainfall_multiplier=mult, horton_f0_mps=1e-5 * ones, horton_fc_mps=1e-6 * ones,
                                          horton_k_per_s=1e-3 * ones, open_fraction=ones, active_mask=np.ones(C, bool))
    s = FloodSolver(topo, rainfall=sc.rainfall, cfg=cfg, infiltration_fields=fields, centroids=sc.city.mesh.centroids_xy,
                    duration_s=150.0)
    h = np.random.default_rng(n).uniform(0.0, 0.5, C).astype(np.float32)
    s.set_state(h, np.zeros_like(h), np.zeros_like(h))
    s.reset_clock()
    return s


def _run(s, **kw):
    with pytest.raises(SimulationError) as e:
        s.run(**kw)
    return str(e.value), s.progress(), s.get_state(wet_time=True), s.snapshots()


# checks on every step, inside an interval, on its last two steps (no step, or one, is planned
# beyond them before the next evaluation), on the first and second of the next one; 2 and 13 tiles
@pytest.mark.gpu
@pytest.mark.parametrize("finite,done", [(1, 3), (20, 22), (30, 32), (31, 32), (32, 34), (33, 35)])
@pytest.mark.parametrize("n", [16, 40])
@pytest.mark.parametrize("mode", ["full_swe", "local_inertial"])
def test_a_failed_check_ends_the_run_a_step_later(finite, done, n, mode):
    from floodgb.build import build_library

    build_library()
    native.load()
    if native.device_count() < 1:
        pytest.skip("no CUDA device")
    s, capped = _solver(n, mode, finite), _solver(n, mode, 10**6)
    try:
        msg, p, state, snaps = _run(s)
        assert f"Non-finite depth detected at step {finite} " in msg
        assert (p.error_step, p.step_count) == (finite, done)
        msg, q, state1, snaps1 = _run(capped, max_steps=done)
        assert "step cap" in msg
        assert (p.t_s, p.last_dt_s, p.snapshot_count, p.cfl_eval_count) == (q.t_s, q.last_dt_s, q.snapshot_count, q.cfl_eval_count)
        for a, b in zip((*state, *snaps), (*state1, *snaps1)):
            np.testing.assert_array_equal(a, b)
        # the solver stays usable: the same run again
        C = s.cell_count
        h = np.random.default_rng(n).uniform(0.0, 0.5, C).astype(np.float32)
        s.set_state(h, np.zeros_like(h), np.zeros_like(h))
        s.reset_clock()
        _, p2, state2, _ = _run(s)
        assert (p2.error_step, p2.step_count, p2.t_s) == (p.error_step, p.step_count, p.t_s)
        for a, b in zip(state, state2):
            np.testing.assert_array_equal(a, b)
    finally:
        s.close()
        capped.close()


# checks that pass, on every step: the run is that without checks
@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["full_swe", "local_inertial"])
def test_passed_checks_change_nothing(mode):
    from floodgb.build import build_library

    build_library()
    native.load()
    if native.device_count() < 1:
        pytest.skip("no CUDA device")
    sc = make_grid_city(n=40, size_m=400.0, seed=3, duration_min=3.0)
    out = []
    for finite in (1, 7, 0):
        cfg = load_config(None, dict(sc.overrides, **{"solver.surface_step_mode": mode, "solver.finite_check_interval_steps": finite}))
        s = FloodSolver(sc.city.topologies.surface_topology, rainfall=sc.rainfall, cfg=cfg, centroids=sc.city.mesh.centroids_xy,
                        duration_s=150.0)
        try:
            h = np.random.default_rng(5).uniform(0.0, 0.5, sc.cell_count).astype(np.float32)
            s.set_state(h, np.zeros_like(h), np.zeros_like(h))
            s.reset_clock()
            s.run()
            out.append((s.progress(), s.get_state(), s.ledger()))
        finally:
            s.close()
    assert out[0][0].error == 0 and out[0][0].step_count > 64
    for p, state, led in out[1:]:
        assert p == out[0][0] and led == out[0][2]
        for a, b in zip(state, out[0][1]):
            np.testing.assert_array_equal(a, b)
