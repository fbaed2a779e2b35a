"""The MLP kernels over the input forms that the network itself does not use: widths of 64 and
128 in any order, one to three segments, either output width, aggregation in any place, with
and without a residual; and a row map beside an aggregation, which is not read.  Against plain
PyTorch in 64 bits on the rounded operands.

Tolerances: forward and data gradients 1e-2 relative L2 a tile, as for single MLPs against the
oracle (the hidden rows are bf16, and the fp32 order of the sums flips some of their roundings);
weight gradients 1e-3, as their operands are exact in bf16 and only fp32 sums differ."""
import ctypes as C

import pytest

from storm_b200 import gnn

pytestmark = pytest.mark.gpu

ROWS = 128 * 149  # one tile more than SMs
# segments: i identity, m map, a aggregation; width / 64
FORMS = ["i1", "m2", "a1", "i1i1", "i1m2", "m1a2", "a1m1", "i1i1i1", "a1i2m1", "m2m1i2", "i2a2a1", "m1i2a2"]


def _ptr(t):
    return None if t is None else t.data_ptr()


def _inputs(form, seed):
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed)
    rnd = lambda *n: torch.randn(*n, generator=g, device="cuda")  # noqa: E731
    segs, parts, keep = [], [], []
    for kind, w in zip(form[::2], form[1::2]):
        q, width = gnn.Seg(), 64 * int(w)
        q.width = width
        src = rnd(3 * ROWS if kind == "a" else ROWS, width).bfloat16()
        q.src = src.data_ptr()
        x = src.double()
        if kind == "m":
            idx = torch.randint(-1, ROWS, (ROWS,), generator=g, device="cuda", dtype=torch.int32)
            q.idx = idx.data_ptr()
            x = torch.where((idx >= 0)[:, None], x[idx.clamp(min=0).long()], 0.0)
            keep.append(idx)
        elif kind == "a":
            nbr = torch.randint(-1, 3, (3, ROWS), generator=g, device="cuda", dtype=torch.int32)
            short = torch.zeros(4, dtype=torch.int32, device="cuda")
            q.idx, q.agg, q.agg_stride, q.nbr = short.data_ptr(), 1, ROWS, nbr.data_ptr()
            x = (x.reshape(3, ROWS, width) * (nbr[:, :, None] >= 0)).sum(0).float().bfloat16().double()
            keep += [nbr, short]
        segs.append(q)
        parts.append(x)
        keep.append(src)
    return rnd, segs, torch.cat(parts, dim=1), keep


def _close(got, ref, tol=1e-2):
    d = (got.double() - ref).reshape(ROWS // 128, -1).norm(dim=1)
    assert (d < tol * ref.reshape(ROWS // 128, -1).norm(dim=1)).all()


def _fill(a, segs, k_in, n_out):
    a.rows, a.nseg, a.k_in, a.n_out = ROWS, len(segs), k_in, n_out
    if not isinstance(a, gnn.MlpBwdData):
        for i, q in enumerate(segs):
            a.seg[i] = q
    return a


@pytest.mark.parametrize("n_out", [64, 128])
@pytest.mark.parametrize("form", FORMS)
def test_forward(form, n_out, storm_lib):
    import torch
    rnd, segs, A, keep = _inputs(form, 3)
    k_in = A.shape[1]
    w1, w2 = (rnd(128, k_in) / k_in ** 0.5).bfloat16(), (rnd(n_out, 128) / 11.0).bfloat16()
    b1, b2, res = rnd(128), rnd(n_out), rnd(ROWS, n_out).bfloat16()
    out, f32 = torch.empty((ROWS, n_out), dtype=torch.bfloat16, device="cuda"), torch.empty((ROWS, n_out), device="cuda")
    hid, err = torch.empty((ROWS, 128), dtype=torch.bfloat16, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    for save, with_res in ((None, None), (hid, res), (hid, None), (None, res)):
        a = _fill(gnn.MlpFwd(), segs, k_in, n_out)
        a.w1, a.b1, a.w2, a.b2 = _ptr(w1), _ptr(b1), _ptr(w2), _ptr(b2)
        a.res, a.out, a.out_f32, a.a1_save = _ptr(with_res), _ptr(out), _ptr(f32), _ptr(save)
        gnn._chk(gnn.lib().storm_gnn_mlp_forward(C.byref(a), _ptr(err), gnn._stream()))
        h = torch.relu(A @ w1.double().T + b1.double())
        y = h.float().bfloat16().double() @ w2.double().T + b2.double() + (0.0 if with_res is None else res.double())
        _close(out, y)
        _close(f32, y)
        if save is not None:
            _close(hid, h)
    assert int(err.item()) == 0


@pytest.mark.parametrize("n_out", [64, 128])
@pytest.mark.parametrize("form", FORMS)
def test_backward(form, n_out, storm_lib):
    import torch
    rnd, segs, A, keep = _inputs(form, 4)
    k_in = A.shape[1]
    w1, w2 = (rnd(128, k_in) / k_in ** 0.5).bfloat16(), (rnd(n_out, 128) / 11.0).bfloat16()
    dy, a1 = rnd(ROWS, n_out), torch.relu(rnd(ROWS, 128)).bfloat16()
    dz1, err = torch.empty((ROWS, 128), dtype=torch.bfloat16, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    widths = [q.width for q in segs]
    add = [rnd(ROWS, w) if i % 2 == 0 else None for i, w in enumerate(widths)]
    dseg = [torch.empty((ROWS, w), device="cuda") for w in widths]
    a = _fill(gnn.MlpBwdData(), segs, k_in, n_out)
    a.dy, a.a1, a.w1, a.w2, a.dz1_save = _ptr(dy), _ptr(a1), _ptr(w1), _ptr(w2), _ptr(dz1)
    for i, w in enumerate(widths):
        a.seg_width[i], a.dseg[i], a.dseg_add[i] = w, _ptr(dseg[i]), _ptr(add[i])
    gnn._chk(gnn.lib().storm_gnn_mlp_backward_data(C.byref(a), _ptr(err), gnn._stream()))
    dyb = dy.bfloat16().double()
    _close(dz1, (dyb @ w2.double()) * (a1 > 0))
    dA = torch.split(dz1.double() @ w1.double(), widths, dim=1)
    for o, ref, p in zip(dseg, dA, add):
        _close(o, ref if p is None else ref + p.double())

    b = _fill(gnn.MlpBwdWeight(), segs, k_in, n_out)
    b.dy, b.a1, b.dz1 = _ptr(dy), _ptr(a1), _ptr(dz1)
    n = int(gnn.lib().storm_gnn_weight_scratch_bytes(k_in, n_out))
    grad, scratch = torch.empty(gnn.lib().storm_gnn_grad_size(k_in, n_out), device="cuda"), torch.empty(n // 4, device="cuda")
    gnn._chk(gnn.lib().storm_gnn_mlp_backward_weight(C.byref(b), _ptr(grad), _ptr(scratch), n, _ptr(err), gnn._stream()))
    at = 0
    for ref in (dz1.double().T @ A, dz1.double().sum(0), dyb.T @ a1.double(), dy.double().sum(0)):
        g = grad[at:at + ref.numel()].double().reshape(ref.shape)
        assert (g - ref).norm() < 1e-3 * ref.norm()
        at += ref.numel()
    assert at == grad.numel() and int(err.item()) == 0
