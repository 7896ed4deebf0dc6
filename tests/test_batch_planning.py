"""Batches whose scenarios evaluate the CFL minimum on the same steps plan the
steps in between beside the surface kernel; with one scenario of another
interval every step has its planning launch.  Both give every scenario the
same steps, states, snapshots and ledger, bit for bit."""

import numpy as np
import pytest

from floodgb import native
from floodgb.batch import BatchSolver, Member
from floodgb.config import load_config
from floodgb.exceptions import SimulationError
from floodgb.rainfall import rainfall_event
from floodgb.synthetic import make_grid_city


def _member(n, seed, interval, minutes, mmhr=60.0):
    rain = rainfall_event([0.0, minutes / 2], [minutes / 2, 60.0], [mmhr, mmhr / 3])
    sc = make_grid_city(n=n, size_m=200.0, seed=seed, hyetograph=rain, duration_min=minutes)
    cfg = load_config(None, dict(sc.overrides, **{"solver.snapshot_interval_min": 2.0, "solver.cfl_update_interval_steps": interval,
                                                  "solver.finite_check_interval_steps": 20}))
    return Member(sc.city, sc.rainfall, cfg, minutes * 60.0)


def _skip_without_device():
    from floodgb.build import build_library

    build_library()
    native.load()
    if native.device_count() < 1:
        pytest.skip("no CUDA device")


# 1 scenario, 9 and 17 (one more than the planning warps of a CTA's, of two CTAs'), 1 to 64 tiles each, ending apart
@pytest.mark.gpu
@pytest.mark.parametrize("count", [1, 9, 17])
@pytest.mark.parametrize("tile", [128, 256])
@pytest.mark.parametrize("interval", [2, 16])
def test_planning_beside_the_step_gives_the_same_bits(count, tile, interval):
    _skip_without_device()
    sizes = [9, 90, 22, 40, 14]
    members = [_member(sizes[k % 5], k, interval, 4.0 + 0.5 * (k % 4)) for k in range(count)]
    out = []
    for extra in ([], [_member(9, 99, 20, 5.0)]):  # 20 steps: not a divisor of a chunk, nor the others' interval
        with BatchSolver(members + extra, shape={"tile_cells": tile}) as b:
            b.run()
            out.append([(b.progress(k), b.state(k), b.snapshots(k), b.ledger(k)) for k in range(count)])
    assert len({o[0].step_count for o in out[0]}) > 1 or count == 1
    for (p, state, snaps, led), (q, state1, snaps1, led1) in zip(*out):
        assert p.error == 0 and p == q
        for a, c in zip((*state, *snaps), (*state1, *snaps1)):
            np.testing.assert_array_equal(a, c)
        assert led == led1


@pytest.mark.gpu
@pytest.mark.parametrize("other", [32, 20])
def test_a_non_finite_depth_names_its_scenario_and_step(other):
    _skip_without_device()
    members = [_member(14, 1, 32, 5.0), _member(14, 2, 32, 5.0, mmhr=1.0e46), _member(9, 3, other, 5.0)]
    with BatchSolver(members) as b:
        with pytest.raises(SimulationError, match="scenario 1: non-finite depth detected at step 20$"):
            b.run()
