"""Runs of the surface alone in one cooperative launch where several CTAs share an
SM, and the meshes between: tiles with wide halos (cells in the caller's order)
leave k_surface fewer CTAs than tiles, while the run kernel, with half its shared
memory, would still fit.  Those take a launch a step.  Either way the run equals
the same run step by step, ledger included."""

import numpy as np
import pytest

from floodgb import native
from floodgb.config import load_config
from floodgb.domain import ProductionInfiltrationFields
from floodgb.solver import FloodSolver
from floodgb.synthetic import make_grid_city

DURATION_S, RAIN_MMHR = 120.0, 50.0


def _device_sms():
    from floodgb.build import build_library

    build_library()
    native.load()
    if native.device_count() < 1:
        pytest.skip("no CUDA device")
    import torch

    return torch.cuda.get_device_properties(0).multi_processor_count


def _city(tiles):
    n = int(np.sqrt(tiles * 256 / 2))  # 2 n^2 triangles
    return make_grid_city(n=n, size_m=10.0 * n, seed=n, rain_mmhr=RAIN_MMHR, duration_min=3.0)


def _solver(sc, centroids, mode):
    cfg = load_config(None, dict(sc.overrides, **{"solver.snapshot_interval_min": 1.0, "solver.surface_step_mode": mode}))
    topo = sc.city.topologies.surface_topology
    rng = np.random.default_rng(7)
    C = topo.cell_count
    mult = rng.uniform(0.5, 1.0, C).astype(np.float32)
    f = [rng.uniform(lo, hi, C).astype(np.float32) for lo, hi in ((1e-5, 2e-5), (1e-6, 2e-6), (1e-3, 2e-3))]
    fields = ProductionInfiltrationFields(rainfall_multiplier=mult, horton_f0_mps=f[0], horton_fc_mps=f[1], horton_k_per_s=f[2],
                                          open_fraction=np.ones_like(mult), active_mask=np.ones(C, bool))
    s = FloodSolver(topo, rainfall=sc.rainfall, cfg=cfg, infiltration_fields=fields,
                    centroids=sc.city.mesh.centroids_xy if centroids else None, duration_s=DURATION_S)
    h = rng.uniform(0.0, 0.5, C).astype(np.float32)
    s.set_state(h, np.zeros_like(h), np.zeros_like(h))
    s.reset_clock()
    rain_m3 = RAIN_MMHR * 1.0e-3 / 3600.0 * DURATION_S * float((mult.astype(np.float64) * topo.cell_area_m2).sum())
    return s, rain_m3


# tiles per SM: two, three and four CTAs of the run kernel an SM, then between k_surface's
# three CTAs an SM and the run kernel's four
@pytest.mark.gpu
@pytest.mark.parametrize("per_sm,centroids,mode", [(1.6, True, "full_swe"), (2.6, True, "full_swe"), (3.9, True, "full_swe"),
                                                   (3.48, False, "full_swe"), (1.6, True, "local_inertial")])
def test_run_equals_single_steps_with_several_tiles_an_sm(per_sm, centroids, mode):
    sms = _device_sms()
    sc = _city(int(per_sm * sms))
    lib, out = native.load(), []
    for single in (False, True):
        s, rain_m3 = _solver(sc, centroids, mode)
        try:
            if single:
                for _ in range(40):  # past a CFL evaluation
                    s.run(s.progress().t_s + 1.0e-9)
            before = lib.fl_launch_count()
            s.run()
            launches = lib.fl_launch_count() - before
            out.append((s.progress(), s.get_state(wet_time=True), s.snapshots(), s.ledger()))
            if not single:
                one_launch = launches < s.progress().step_count
        finally:
            s.close()
    assert one_launch == centroids
    (p, state, snaps, led), (q, state1, snaps1, led1) = out
    assert p.error == 0 and p.step_count > 64 and p.snapshot_count >= 2
    assert (p.step_count, p.t_s, p.last_dt_s, p.cfl_eval_count) == (q.step_count, q.t_s, q.last_dt_s, q.cfl_eval_count)
    for a, b in zip((*state, *snaps), (*state1, *snaps1)):
        np.testing.assert_array_equal(a, b)
    assert led == led1
    # every tile's rain is in the ledger (float32 terms, at most some 1e-7 each)
    assert abs(led["rainfall_input_m3"] - rain_m3) <= 1.0e-5 * rain_m3
