"""What the fused passes' wrappers hand to the library, and what they refuse: the
library is a stand-in that reads the matrices through the pointers and leading
dimensions it is given (host memory: no GPU needed)."""

import ctypes as C
from types import SimpleNamespace

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from floodgb.surrogate import ops  # noqa: E402
from floodgb.surrogate.model import FIN, FOUT, MPNN, DualGraph  # noqa: E402
from floodgb.synthetic import make_grid_city  # noqa: E402


def _matrix(ptr, ld, rows, cols, ctype):
    flat = np.ctypeslib.as_array(C.cast(ptr, C.POINTER(ctype)), ((rows - 1) * ld + cols,))
    return np.stack([flat[r * ld:r * ld + cols] for r in range(rows)])


@pytest.fixture()
def case(monkeypatch):
    seen = {}

    def forward(desc, stream):
        d = desc._obj
        seen["x"] = _matrix(d.x, d.ldx, d.cells, FIN, C.c_int16)
        return 0

    def backward(desc, stream):
        d = desc._obj
        seen["x"] = _matrix(d.x, d.ldx, d.cells, FIN, C.c_int16)
        seen["dy"] = _matrix(d.dy, d.ldy, d.cells, FOUT, C.c_float)
        assert d.ldy >= FOUT and d.ldy % 8 == 0
        return 0

    lib = SimpleNamespace(fl_mpnn_forward=forward, fl_mpnn_backward=backward, fl_mpnn_backward_scratch=lambda *a: 0)
    monkeypatch.setattr(ops.N, "load", lambda: lib)
    monkeypatch.setattr(ops, "_stream", lambda: C.c_void_p(0))
    g = DualGraph(make_grid_city(n=5, size_m=50.0, seed=2).city.topologies.surface_topology, device="cpu")
    net = MPNN(n_layers=2, seed=1, device="cpu")
    gen = torch.Generator().manual_seed(3)
    x = torch.randn(g.C, FIN, generator=gen).to(torch.bfloat16)
    dy = torch.randn(g.C, FOUT, generator=gen)
    return g, net, x, dy, seen


def _views(t):
    """The matrix t in other layouts."""

    rows, cols = t.shape
    wide = torch.zeros(rows, 2 * cols + 8, dtype=t.dtype)
    wide[:, 8:8 + cols] = t
    tall = torch.zeros(rows + 3, cols, dtype=t.dtype)
    tall[:rows] = t
    return {"plain": t, "columns of a wider one": wide[:, 8:8 + cols], "rows of a taller one": tall[:rows],
            "narrow view of padded rows": t[:, :12]}


@pytest.mark.parametrize("layout", ["plain", "columns of a wider one", "rows of a taller one", "narrow view of padded rows"])
def test_forward_reads_the_inputs_in_their_layout(case, layout):
    g, net, x, _, seen = case
    net.forward(g, _views(x)[layout], train=False)
    np.testing.assert_array_equal(seen["x"], x.view(torch.int16).numpy())


@pytest.mark.parametrize("layout", ["plain", "columns of a wider one", "rows of a taller one", "narrow view of padded rows",
                                    "one row for all", "column-major", "unaligned", "more rows"])
def test_backward_reads_the_gradient_in_its_layout(case, layout):
    g, net, x, dy, seen = case
    views = _views(dy)
    want = dy.clone()
    if layout == "one row for all":
        given = dy[:1].expand(g.C, FOUT)
        want = given.clone()
    elif layout == "column-major":
        given = dy.t().contiguous().t()
    elif layout == "unaligned":
        given = torch.zeros(g.C * FOUT + 3)[3:].view(g.C, FOUT)
        given.copy_(dy)
    elif layout == "more rows":
        given = torch.cat([dy, dy])
    else:
        given = views[layout]
    net.forward(g, x)
    net.backward(g, _views(x)["columns of a wider one"], given)
    np.testing.assert_array_equal(seen["dy"], want.numpy())
    np.testing.assert_array_equal(seen["x"], x.view(torch.int16).numpy())


def test_backward_refuses_what_it_would_misread(case):
    g, net, x, dy, seen = case
    net.forward(g, x)
    seen.clear()
    for bad in (dy.to(torch.bfloat16), dy.double(), dy[:-1], dy[:, :32].clone(), dy.reshape(-1),
                torch.empty(g.C, FOUT, device="meta")):
        with pytest.raises(ValueError):
            net.backward(g, x, bad)
    for bad in (x.float(), x[:-1], x[:, :32].clone(), x.t().contiguous().t(), x.reshape(-1), torch.cat([x, x]), x.to("meta")):
        with pytest.raises(ValueError):
            net.backward(g, bad, dy)
        with pytest.raises(ValueError):
            net.forward(g, bad)
    assert not seen


def test_products_path_refuses_the_same_gradients(case):
    """A graph with more edges into a cell runs product by product."""

    g, net, x, dy, _ = case
    net.forward(g, x)
    g.max_in = 99
    for bad in (dy.to(torch.bfloat16), dy[:-1], dy.reshape(-1), dy.to("meta")):
        with pytest.raises(ValueError):
            net.backward(g, x, bad)
