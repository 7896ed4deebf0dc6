"""Solvers and batches alive at the same time keep working whichever was made
last: launch limits belong to a kernel, so a later solver with smaller tiles
must not lower them below what an earlier one needs."""

import numpy as np
import pytest

from floodgb import native
from floodgb.config import load_config
from floodgb.solver import FloodSolver, solver_for_city
from floodgb.synthetic import make_grid_city


@pytest.mark.gpu
def test_a_later_solver_with_smaller_tiles_leaves_an_earlier_one_running():
    from floodgb.build import build_library

    build_library()
    native.load()
    if native.device_count() < 1:
        pytest.skip("no CUDA device")
    sc = make_grid_city(n=60, size_m=600.0, seed=2, duration_min=1.0)
    cfg = load_config(None, sc.overrides)
    # without centroids the cells keep the caller's order (here shuffled rows apart): larger halos, larger tiles
    first = FloodSolver(sc.city.topologies.surface_topology, rainfall=sc.rainfall, cfg=cfg)
    later = solver_for_city(sc.city, sc.rainfall, cfg)
    try:
        h = np.random.default_rng(0).uniform(0.0, 0.2, sc.cell_count).astype(np.float32)
        z = np.zeros_like(h)
        for s in (first, later, first):
            s.set_state(h, z, z)
            s.reset_clock()
            s.step(0.1, native.FL_PHASE_SURFACE | native.FL_PHASE_CLAMP, 1.0e-5)
        a, b = first.get_state(), later.get_state()
        for x, y in zip(a[:3], b[:3]):
            assert np.abs(x - y).max() <= 1.0e-6  # another tiling, the same step
    finally:
        first.close()
        later.close()
