"""Timing the drainage kernels leaves the ledger as it was: a timed launch does not
fetch the slots that the launch before it still adds to."""

import pytest

from floodgb import native
from floodgb.config import load_config
from floodgb.solver import solver_for_city
from floodgb.synthetic import coupled_test_city

DRAINAGE = ["surface_capture_m3", "surface_surcharge_m3", "outfall_discharge_m3", "overflow_surcharge_m3",
            "unreturned_overflow_m3", "link_abs_flow_m3"]


# one launch, part of a chain, several chains
@pytest.mark.gpu
@pytest.mark.parametrize("reps", [1, 7, 70])
def test_timing_the_drainage_kernels_leaves_their_ledger_terms(reps):
    from floodgb.build import build_library

    build_library()
    native.load()
    if native.device_count() < 1:
        pytest.skip("no CUDA device")
    sc = coupled_test_city(scale=1, seed=5, duration_min=2.0)
    s = solver_for_city(sc.city, sc.rainfall, load_config(None, sc.overrides))
    try:
        s.run()
        before = s.ledger()
        assert before["surface_capture_m3"] > 0.0 and before["link_abs_flow_m3"] > 0.0
        for kernel in (1, 2, 4, 5):
            assert 0.0 < s.time_kernel(kernel, reps=reps) < 10.0
        after = s.ledger()
        assert [after[k] for k in DRAINAGE] == [before[k] for k in DRAINAGE]
    finally:
        s.close()
