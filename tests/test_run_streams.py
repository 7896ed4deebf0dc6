"""Runs in one cooperative launch beside other work: two solvers on streams and
threads of their own, each of which needs most CTA slots of the device for its
tiles, and a solver beside the surrogate's persistent kernels, which take whole SMs.
A launch must not start in part and wait for CTAs that the other one keeps out:
every run ends without a time-out, with the bits of the run alone."""

import threading

import numpy as np
import pytest

from floodgb import native
from floodgb.config import load_config
from floodgb.solver import FloodSolver
from floodgb.synthetic import make_grid_city

torch = pytest.importorskip("torch")


def _sms():
    from floodgb.build import build_library

    build_library()
    native.load()
    if native.device_count() < 1:
        pytest.skip("no CUDA device")
    return torch.cuda.get_device_properties(0).multi_processor_count


def _solver(n, mode):
    sc = make_grid_city(n=n, size_m=10.0 * n, seed=n, duration_min=3.0)
    cfg = load_config(None, dict(sc.overrides, **{"solver.surface_step_mode": mode}))
    s = FloodSolver(sc.city.topologies.surface_topology, rainfall=sc.rainfall, cfg=cfg, infiltration_mps=1.0e-6,
                    centroids=sc.city.mesh.centroids_xy, duration_s=150.0)
    h = np.random.default_rng(n).uniform(0.0, 0.5, sc.cell_count).astype(np.float32)
    return s, h


def _run(s, h, stream=None):
    z = np.zeros_like(h)
    s.set_state(h, z, z, stream=stream)
    s.reset_clock(stream=stream)
    s.run(stream=stream)
    return s.get_state(stream=stream), s.progress(stream=stream), s.ledger(stream=stream)


def _same(a, b):
    for x, y in zip(a[0], b[0]):
        np.testing.assert_array_equal(x, y)
    assert a[1] == b[1] and a[2] == b[2]


def _threads(jobs):
    errors = []

    def guarded(job):
        try:
            job()
        except BaseException as e:  # noqa: BLE001
            errors.append(e)

    ts = [threading.Thread(target=guarded, args=(j,)) for j in jobs]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    if errors:
        raise errors[0]


# tiles per SM of the two solvers: both fit at once; each fits alone only
@pytest.mark.gpu
@pytest.mark.parametrize("per_sm", [(0.3, 0.4), (2.6, 3.9)])
@pytest.mark.parametrize("mode", ["full_swe", "local_inertial"])
def test_two_solvers_on_two_threads_and_streams(per_sm, mode):
    sms = _sms()
    scale = 1.0 if mode == "full_swe" else 0.5  # (the local-inertial tiles take more of an SM)
    pairs = [_solver(int(np.sqrt(f * scale * sms * 128)), mode) for f in per_sm]
    try:
        want = [_run(*p) for p in pairs]
        streams = [torch.cuda.Stream() for _ in pairs]

        def job(k):
            for _ in range(5):
                _same(_run(*pairs[k], stream=streams[k].cuda_stream), want[k])

        _threads([lambda k=k: job(k) for k in range(2)])
    finally:
        for s, _ in pairs:
            s.close()


@pytest.mark.gpu
def test_a_solver_beside_the_surrogate():
    from floodgb.surrogate.model import FIN, MPNN, DualGraph

    sms = _sms()
    s, h = _solver(int(np.sqrt(3.9 * sms * 128)), "full_swe")
    g = DualGraph(make_grid_city(n=101, size_m=1010.0, seed=4).city.topologies.surface_topology)
    net = MPNN(n_layers=8, seed=3)
    x = torch.randn(g.C, FIN, device="cuda").to(torch.bfloat16)
    y_alone = net.forward(g, x, train=False).clone()
    torch.cuda.synchronize()
    try:
        want = _run(s, h)
        side, main, done = torch.cuda.Stream(), torch.cuda.Stream(), threading.Event()

        def solve():
            try:
                for _ in range(5):
                    _same(_run(s, h, stream=main.cuda_stream), want)
            finally:
                done.set()

        def infer():
            with torch.cuda.stream(side):
                while not done.is_set():
                    for _ in range(20):
                        y = net.forward(g, x, train=False)
                    side.synchronize()
                assert torch.equal(y, y_alone)

        _threads([solve, infer])
    finally:
        s.close()
