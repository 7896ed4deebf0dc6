"""Thin wrappers of libfloodgb's surrogate kernels over CUDA tensors.

Every wrapper checks shapes, dtypes and strides on the host and calls one
C-ABI entry point; there is no fallback path.
"""

from __future__ import annotations

import ctypes as C

from .. import native as N


def _stream():
    import torch

    return C.c_void_p(torch.cuda.current_stream().cuda_stream)


def _ptr(t):
    return C.c_void_p(t.data_ptr()) if t is not None else None


def gemm(segments, b, *, bias=None, residual=None, out_f32=None, out_bf16=None, relu=False, k_splits=1,
         force_tiled=False):
    """out = act(cat_k(seg_rows) . b^T + bias) (+ residual) on the tensor cores.

    segments: list of (tensor bf16 [rows, >= width], row_index int32 [m] or None, width);
    b: bf16 [n, K]; outputs [m, >= n] (f32 and/or bf16).  With k_splits > 1,
    out_f32 is [k_splits, m, ldo] and receives one partial product per slice.
    """

    import torch

    lib = N.load()
    d = N.FlGemmDesc()
    if not 1 <= len(segments) <= 3:
        raise ValueError("1..3 A segments")
    m = None
    for i, (t, rows, width) in enumerate(segments):
        if t.dtype != torch.bfloat16 or t.dim() != 2 or t.stride(1) != 1:
            raise ValueError("A segments must be row-major bf16 matrices")
        if rows is not None:
            if rows.dtype != torch.int32:
                raise ValueError("row maps are int32")
            mi = rows.numel()
        else:
            mi = t.shape[0]
        m = mi if m is None else m
        if mi != m:
            raise ValueError("segments disagree on the number of rows")
        d.a[i] = N.FlGemmSegment(C.c_void_p(t.data_ptr()), _ptr(rows), t.stride(0), int(width))
    if b.dtype != torch.bfloat16 or b.stride(1) != 1:
        raise ValueError("B must be row-major bf16")
    out = out_f32 if out_f32 is not None else out_bf16
    d.n_seg = len(segments)
    d.m = int(m)
    d.n = int(b.shape[0])
    d.b = C.c_void_p(b.data_ptr())
    d.ldb = b.stride(0)
    d.bias = _ptr(bias)
    d.residual = _ptr(residual)
    d.ldr = residual.stride(0) if residual is not None else 0
    d.out_f32 = _ptr(out_f32)
    d.out_bf16 = _ptr(out_bf16)
    d.ldo = out.stride(-2)
    d.relu = int(bool(relu))
    d.k_splits = int(k_splits)
    d.force_tiled = int(bool(force_tiled))
    N.check(lib.fl_gemm_bf16(C.byref(d), _stream()), "fl_gemm_bf16")


def _dense_refs(layers):
    arr = (N.FlDenseRef * max(len(layers), 1))()
    for r, d in zip(arr, layers):
        r.w, r.ldw, r.b = d.w_bf.data_ptr(), d.w_bf.stride(0), d.b.data_ptr()
    return arr


def _pointers(tensors, n):
    """n pointers, cycling through the tensors (None: NULL pointers)."""

    ts = [t.data_ptr() for t in tensors] if tensors else [None]
    return (C.c_void_p * max(n, 1))(*[ts[k % len(ts)] for k in range(n)])


def _padded_rows(t, rows, cols, dtype, device, name):
    """t as `cols` wide rows in memory: a narrower view of rows that are (the
    padding belongs to its storage) is widened.  Anything else is refused."""

    if t.dtype != dtype or t.dim() != 2:
        raise ValueError(f"{name} must be a matrix of {dtype}, got {t.dtype} with {t.dim()} dimensions")
    if t.device != device:
        raise ValueError(f"{name} are on {t.device}, expected {device}")
    if t.shape[0] == rows and t.shape[1] < cols and t.stride(1) == 1 and t.stride(0) >= cols:
        held = t.untyped_storage().nbytes() // t.element_size() - t.storage_offset()
        if (rows - 1) * t.stride(0) + cols <= held:
            return t.as_strided((rows, cols), t.stride())
    if t.shape[0] < rows or t.shape[1] < cols:
        raise ValueError(f"{name} have shape {tuple(t.shape)}, expected ({rows}, {cols})")
    return t[:rows, :cols]


def node_inputs(x, g, device):
    """x checked as bf16 node inputs of graph g."""

    import torch

    if x.dtype != torch.bfloat16 or x.dim() != 2 or x.stride(1) != 1:
        raise ValueError("A segments must be row-major bf16 matrices")
    if x.shape == (g.C, 64) and x.device == device:
        return x
    if x.shape[0] != g.C:
        raise ValueError(f"inputs have shape {tuple(x.shape)}, expected ({g.C}, 64)")
    return _padded_rows(x, g.C, 64, torch.bfloat16, device, "inputs")


def output_gradients(dy, g, device):
    """dy checked as fp32 gradients of graph g's outputs."""

    import torch

    if dy.dtype == torch.float32 and dy.shape == (g.C, 64) and dy.device == device:
        return dy
    return _padded_rows(dy, g.C, 64, torch.float32, device, "output gradients")


def mpnn_forward(net, g, x, ws):
    """The network's forward pass over graph g (at most three edges into a
    cell) into workspace ws; hidden activations are kept where ws has them."""

    x = node_inputs(x, g, ws.y.device)
    L = net.n_layers
    d = N.FlMpnnForwardDesc()
    d.cells, d.edges, d.layers = g.C, g.E, L
    d.src, d.recv_start = _ptr(g.src), _ptr(g.recv_start)
    d.x, d.ldx = _ptr(x), x.stride(0)
    d.ef, d.lde = _ptr(g.ef_bf), g.ef_bf.stride(0)
    d.enc_n, d.enc_e, d.dec = _dense_refs(net.enc_n), _dense_refs(net.enc_e), _dense_refs(net.dec)
    d.edge = _dense_refs([m for pair in net.edge for m in pair])
    d.node = _dense_refs([m for pair in net.node for m in pair])
    d.zn, d.ze, d.e, d.zd = _ptr(ws.zn), _ptr(ws.ze), _ptr(ws.e_bf), _ptr(ws.zd)
    d.h_bf = _pointers(ws.h_bf, L + 1)
    d.agg, d.z1e, d.z1n = _pointers(ws.agg_bf, L), _pointers(ws.z1e, L), _pointers(ws.z1n, L)
    d.h_f32[0], d.h_f32[1] = ws.h_f32[0].data_ptr(), ws.h_f32[1].data_ptr()
    d.y = _ptr(ws.y)
    N.check(N.load().fl_mpnn_forward(C.byref(d), _stream()), "fl_mpnn_forward")


def backward_scratch(cells: int, edges: int, layers: int) -> int:
    """Floats of scratch that mpnn_backward needs on the current device."""

    n = C.c_int64()
    N.check(N.load().fl_mpnn_backward_scratch(cells, edges, layers, C.byref(n)), "fl_mpnn_backward_scratch")
    return n.value


def _dense_grads(layers):
    arr = (N.FlDenseGrad * max(len(layers), 1))()
    for r, d in zip(arr, layers):
        r.wt, r.ldwt = d.wt_bf.data_ptr(), d.wt_bf.stride(0)
        r.gw, r.gb = d.gw.data_ptr(), d.gb.data_ptr()
    return arr


def mpnn_backward(net, g, x, dy, ws):
    """Add the parameter gradients for the output gradient dy (fp32 [C, 64])
    of the forward pass whose activations ws holds (x, dy: checked by the caller)."""

    if dy.stride(1) != 1 or dy.stride(0) < 64 or dy.stride(0) % 8 or dy.data_ptr() % 32:
        ws.dy_f32.copy_(dy)
        dy = ws.dy_f32
    L = net.n_layers
    d = N.FlMpnnBackwardDesc()
    d.cells, d.edges, d.layers = g.C, g.E, L
    d.src, d.dst, d.recv_start = _ptr(g.src), _ptr(g.dst), _ptr(g.recv_start)
    d.send_start, d.send_order = _ptr(g.send_start), _ptr(g.send_order)
    d.x, d.ldx = _ptr(x), x.stride(0)
    d.ef, d.lde = _ptr(g.ef_bf), g.ef_bf.stride(0)
    d.enc_n, d.enc_e, d.dec = _dense_grads(net.enc_n), _dense_grads(net.enc_e), _dense_grads(net.dec)
    d.edge = _dense_grads([m for pair in net.edge for m in pair])
    d.node = _dense_grads([m for pair in net.node for m in pair])
    d.zn, d.ze, d.e, d.zd = _ptr(ws.zn), _ptr(ws.ze), _ptr(ws.e_bf), _ptr(ws.zd)
    d.h_bf, d.agg = _pointers(ws.h_bf, L + 1), _pointers(ws.agg_bf, L)
    d.z1e, d.z1n, d.dze = _pointers(ws.z1e, L), _pointers(ws.z1n, L), _pointers(ws.dze, L)
    d.dy, d.ldy = _ptr(dy), dy.stride(0)
    d.dh[0], d.dh[1] = ws.dh[0].data_ptr(), ws.dh[1].data_ptr()
    d.dz2c, d.dz1c, d.dagg, d.dyb = _ptr(ws.dz2_c), _ptr(ws.dz1_c), _ptr(ws.dagg_bf), _ptr(ws.dy_bf)
    d.dz2e, d.dz1f, d.gf, d.ef32 = _ptr(ws.dz2_e), _ptr(ws.dz1_f32), _ptr(ws.g_f32), _ptr(ws.e_f32)
    d.bits = _ptr(ws.bits)
    d.daggf = _pointers(ws.dagg_f32, L)
    d.scratch, d.scratch_floats = _ptr(ws.scratch), ws.scratch.numel()
    N.check(N.load().fl_mpnn_backward(C.byref(d), _stream()), "fl_mpnn_backward")


def adam_all(layers, lr, step, weight_decay=0.0, b1=0.9, b2=0.999, eps=1e-8):
    """One Adam step on every layer's weights (decayed) and biases."""

    n = len(layers)
    # biases are not decayed: their tensors go in a second call where the weights are
    for decay, part in (((weight_decay, "w"), (0.0, "b")) if weight_decay else ((0.0, "wb"),)):
        arr = (N.FlAdamTensor * (n * len(part)))()
        k = 0
        for d in layers:
            if "w" in part:
                a = arr[k]
                a.w, a.m1, a.m2, a.g = d.w.data_ptr(), d.m1w.data_ptr(), d.m2w.data_ptr(), d.gw.data_ptr()
                a.w_bf16, a.wt_bf16 = d.w_bf.data_ptr(), d.wt_bf.data_ptr()
                a.rows, a.cols, a.ldt = d.n_out, d.n_in, d.wt_bf.stride(0)
                k += 1
            if "b" in part:
                a = arr[k]
                a.w, a.m1, a.m2, a.g = d.b.data_ptr(), d.m1b.data_ptr(), d.m2b.data_ptr(), d.gb.data_ptr()
                a.rows, a.cols = 1, d.n_out
                k += 1
        N.check(N.load().fl_adam_all(arr, k, float(lr), float(b1), float(b2), float(eps), int(step), float(decay),
                                     _stream()), "fl_adam_all")


def status():
    N.check(N.load().fl_gemm_status(_stream()), "fl_gemm_status")


def _seg_array(segments):
    arr = (N.FlGemmSegment * 3)()
    for i, (t, rows, width) in enumerate(segments):
        arr[i] = N.FlGemmSegment(C.c_void_p(t.data_ptr()), _ptr(rows), t.stride(0), int(width))
    return arr


def transpose(segments, m, dst):
    """dst[k, r] = cat_k(segments)[r, k]; dst columns m.. zeroed."""

    N.check(N.load().fl_transpose_bf16(_seg_array(segments), len(segments), int(m), C.c_void_p(dst.data_ptr()),
                                       dst.stride(0), _stream()), "fl_transpose_bf16")


def segment_sum(src, col0, start, order, n_out, width, dst, dst_bf16=None, accumulate=False):
    """Fixed-order row sums; dst None (with dst_bf16, no accumulation) writes the bf16 copy only."""
    N.check(N.load().fl_segment_sum(C.c_void_p(src.data_ptr()), src.stride(0), int(col0), C.c_void_p(start.data_ptr()),
                                    _ptr(order), int(n_out), int(width), _ptr(dst), dst.stride(0) if dst is not None else 4,
                                    _ptr(dst_bf16), dst_bf16.stride(0) if dst_bf16 is not None else 0,
                                    int(bool(accumulate)), _stream()), "fl_segment_sum")


def relu_bwd(dx, z, out_bf16, out_f32=None):
    m, n = dx.shape[0], out_bf16.shape[1]
    N.check(N.load().fl_relu_bwd(C.c_void_p(dx.data_ptr()), dx.stride(0), _ptr(z), z.stride(0) if z is not None else 0,
                                 int(m), int(n), C.c_void_p(out_bf16.data_ptr()), out_bf16.stride(0), _ptr(out_f32),
                                 out_f32.stride(0) if out_f32 is not None else 0, _stream()), "fl_relu_bwd")


def colsum(x, m, n, scratch, out, accumulate=False):
    N.check(N.load().fl_colsum(C.c_void_p(x.data_ptr()), x.stride(0), int(m), int(n), C.c_void_p(scratch.data_ptr()),
                               C.c_void_p(out.data_ptr()), int(bool(accumulate)), _stream()), "fl_colsum")


def adam(w, m1, m2, g, lr, step, b1=0.9, b2=0.999, eps=1e-8, weight_decay=0.0, w_bf16=None, wt_bf16=None):
    rows, cols = w.shape
    N.check(N.load().fl_adam(C.c_void_p(w.data_ptr()), C.c_void_p(m1.data_ptr()), C.c_void_p(m2.data_ptr()),
                             C.c_void_p(g.data_ptr()), int(rows), int(cols), float(lr), float(b1), float(b2),
                             float(eps), int(step), float(weight_decay), _ptr(w_bf16), _ptr(wt_bf16),
                             wt_bf16.stride(0) if wt_bf16 is not None else 0, _stream()), "fl_adam")


def cast_bf16(src, dst):
    m, n = dst.shape
    N.check(N.load().fl_cast_bf16(C.c_void_p(src.data_ptr()), src.stride(0), int(m), int(n),
                                  C.c_void_p(dst.data_ptr()), dst.stride(0), _stream()), "fl_cast_bf16")
