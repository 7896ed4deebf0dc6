"""The network's fused blocks against the same network run product by product
(the path of graphs with more than three edges into a cell), which the oracle
tests pin: the blocks keep every rounding point and the order of every sum, so
the results are the same bits."""

import copy

import numpy as np
import pytest

# cells: 2 (one partial tile), 128 (one full tile), 162 and 20,402 (a remainder; more tiles than SMs)
GRIDS = [1, 8, 9, 101]


def _case(n, layers, copies=1):
    torch = pytest.importorskip("torch")
    from floodgb import native
    from floodgb.build import build_library
    from floodgb.surrogate.model import FIN, MPNN, DualGraph
    from floodgb.synthetic import make_grid_city

    build_library()
    native.load()
    if native.device_count() < 1:
        pytest.skip("no CUDA device")
    g = DualGraph(make_grid_city(n=n, size_m=10.0 * n, seed=4).city.topologies.surface_topology)
    if copies > 1:
        g = g.replicate(copies)
    assert g.max_in <= 3
    plain = copy.copy(g)
    assert g.max_out <= 3
    plain.max_in = 99  # product by product
    net, ref = MPNN(n_layers=layers, seed=3), MPNN(n_layers=layers, seed=3)
    rng = np.random.default_rng(n)
    for d, r in zip(net.layers(), ref.layers()):
        b = torch.as_tensor(rng.normal(0, 0.1, d.n_out).astype(np.float32), device="cuda")
        d.b.copy_(b)
        r.b.copy_(b)
    wide = torch.as_tensor(rng.normal(size=(g.C, FIN + 8)).astype(np.float32), device="cuda").to(torch.bfloat16)
    return torch, g, plain, net, ref, wide[:, 8:]


@pytest.mark.gpu
@pytest.mark.parametrize("n", GRIDS)
@pytest.mark.parametrize("train", [False, True])
def test_forward_blocks_give_the_products_bits(n, train):
    torch, g, plain, net, ref, x = _case(n, 3, copies=2 if n == 9 else 1)
    y = net.forward(g, x, train=train).clone()
    want = ref.forward(plain, x, train=train)
    assert bool(torch.isfinite(want).all()) and float(want.abs().max()) > 0
    assert torch.equal(y, want)
    if train:
        a, b = net.ws, ref.ws
        for k in ("zn", "ze", "e_bf", "zd"):
            assert torch.equal(getattr(a, k), getattr(b, k)), k
        for k in ("z1e", "agg_bf", "z1n", "h_bf"):
            for p, q in zip(getattr(a, k), getattr(b, k)):
                assert torch.equal(p, q), k


@pytest.mark.gpu
@pytest.mark.parametrize("n", GRIDS)
@pytest.mark.parametrize("layers", [0, 1, 3])
def test_backward_blocks_give_the_products_gradients(n, layers):
    """The blocks keep the order of every sum, those over rows included: the same bits."""

    torch, g, plain, net, ref, x = _case(n, layers)
    rng = np.random.default_rng(n + 50)
    dy = torch.as_tensor(rng.normal(size=(g.C, 64)).astype(np.float32), device="cuda")
    wide = torch.zeros(g.C, 68, device="cuda")
    wide[:, 3:67] = dy
    for model, graph, grad in ((net, g, wide[:, 3:67] if n == 9 else dy), (ref, plain, dy)):
        model.forward(graph, x)
        model.zero_grad()
        for d in model.layers():
            d.gb.add_(1.0)  # gradients are added to
        model.backward(graph, x, grad)
    for k, (d, r) in enumerate(zip(net.layers(), ref.layers())):
        for a, b in ((d.gw, r.gw), (d.gb, r.gb)):
            assert torch.equal(a, b), (k, tuple(a.shape), float((a - b).abs().max()))
    net.step(1e-3, weight_decay=0.01)
    for d in ref.layers():
        d.gw.copy_(net.layers()[ref.layers().index(d)].gw)
        d.gb.copy_(net.layers()[ref.layers().index(d)].gb)
        d.step(1e-3, 1, 0.01)
    for d, r in zip(net.layers(), ref.layers()):  # the same arithmetic tensor by tensor
        for a in ("w", "b", "m1w", "m2w", "m1b", "m2b", "w_bf", "wt_bf"):
            assert torch.equal(getattr(d, a), getattr(r, a)), a


@pytest.mark.gpu
def test_forward_rejects_inputs_of_another_shape():
    torch, g, _, net, _, x = _case(8, 1)
    with pytest.raises(ValueError):
        net.forward(g, x[:-1], train=False)
    with pytest.raises(ValueError):
        net.forward(g, x.float(), train=False)


def test_union_of_copies_on_the_device_matches_the_shifted_host_arrays():
    """The union's index arrays and its host copies (no GPU needed: torch on the CPU)."""

    pytest.importorskip("torch")
    from floodgb.surrogate.model import DualGraph
    from floodgb.synthetic import make_grid_city

    g = DualGraph(make_grid_city(n=5, size_m=50.0, seed=2).city.topologies.surface_topology, device="cpu")
    k = 3
    u = g.replicate(k)
    assert (u.C, u.E, u.max_in, u.max_out) == (k * g.C, k * g.E, g.max_in, g.max_out)
    for name, step in (("src", g.C), ("dst", g.C), ("send_order", g.E)):
        want = np.concatenate([getattr(g, name).numpy() + j * step for j in range(k)])
        np.testing.assert_array_equal(getattr(u, name).numpy(), want)
    for name in ("recv_start", "send_start"):
        a = getattr(g, name).numpy()
        want = np.concatenate([a[:-1] + j * g.E for j in range(k)] + [[k * g.E]])
        np.testing.assert_array_equal(getattr(u, name).numpy(), want)
    np.testing.assert_array_equal(u.row_start.numpy(), np.arange(k * g.E + 1))
    np.testing.assert_array_equal(u.src_h, u.src.numpy())
    np.testing.assert_array_equal(u.dst_h, u.dst.numpy())
    np.testing.assert_array_equal(u.indeg_h, u.indeg.numpy())
    np.testing.assert_array_equal(u.edge_features_h, np.tile(g.edge_features_h, (k, 1)))
    assert u.ef_bf.shape == (k * g.E, 64) and all(t.is_contiguous() for t in (u.src, u.ef_bf, u.recv_start))
    with pytest.raises(AttributeError):
        u.no_such_array
