"""A scenario of a batch whose finite check fails ends with the checked step, planned
beside the surface kernel or not: clock, state, snapshots and ledger are those of a
batch with a planning launch a step, and the other scenarios run on."""

import dataclasses

import numpy as np
import pytest

from floodgb import native
from floodgb.batch import BatchSolver, Member
from floodgb.config import load_config
from floodgb.domain import ProductionInfiltrationFields
from floodgb.exceptions import SimulationError
from floodgb.rainfall import rainfall_event
from floodgb.synthetic import make_grid_city


def _member(n, seed, interval, finite, failing=False):
    rain = rainfall_event([0.0, 120.0], [120.0, 3600.0], [60.0, 20.0])
    sc = make_grid_city(n=n, size_m=200.0, seed=seed, hyetograph=rain, duration_min=4.0)
    city, over = sc.city, {"solver.snapshot_interval_min": 0.05, "solver.cfl_update_interval_steps": interval,
                           "solver.finite_check_interval_steps": finite}
    if failing:  # one cell's rain depth is infinite from the first step
        ones = np.ones(sc.cell_count, np.float32)
        mult = ones.copy()
        mult[sc.cell_count // 2] = np.inf
        city = dataclasses.replace(city, infiltration_fields=ProductionInfiltrationFields(
            rainfall_multiplier=mult, horton_f0_mps=1e-5 * ones, horton_fc_mps=1e-6 * ones, horton_k_per_s=1e-3 * ones,
            open_fraction=ones, active_mask=ones > 0))
        over["physics.infiltration_mode"] = "production_horton"
    return Member(city, sc.rainfall, load_config(None, dict(sc.overrides, **over)), 240.0)


# checks on every step, inside an interval, on its last two steps, on the first two of the
# next one; tiles on few CTAs (the next launch sets up early) and on every slot of the device
@pytest.mark.gpu
@pytest.mark.parametrize("finite", [1, 5, 10, 30, 31, 32, 33])
@pytest.mark.parametrize("tile", [128, 256])
@pytest.mark.parametrize("others", [3, 20])
def test_a_failed_check_ends_its_scenario(finite, tile, others):
    from floodgb.build import build_library

    build_library()
    native.load()
    if native.device_count() < 1:
        pytest.skip("no CUDA device")
    bad = others // 2
    out = []
    for extra in ([], [_member(9, 99, 20, 7)]):  # (20 steps: a planning launch a step)
        members = [_member(90 if others > 3 else 14, k, 32, finite) for k in range(others)]
        members[bad] = _member(14, 50, 32, finite, failing=True)
        with BatchSolver(members + extra, shape={"tile_cells": tile}) as b:
            with pytest.raises(SimulationError, match=f"scenario {bad}: non-finite depth detected at step {finite}$"):
                b.run()
            out.append([(b.progress(k), b.state(k), b.snapshots(k), b.ledger(k)) for k in range(others)])
    p = out[0][bad][0]
    assert (p.error_step, p.step_count) == (finite, finite + 1)
    for k, ((p, state, snaps, led), (q, state1, snaps1, led1)) in enumerate(zip(*out)):
        assert p == q and (p.error != 0) == (k == bad)
        for a, c in zip((*state, *snaps), (*state1, *snaps1)):
            np.testing.assert_array_equal(a, c)
        np.testing.assert_equal(led, led1)  # (the failed scenario's has infinities)
