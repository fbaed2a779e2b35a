"""The forward MLP kernel with several 128-row tiles per CTA: its ring of input blocks is
filled by two roles (TMA for rows that follow one another, per-row copies for maps and
aggregation), so the cases mix both from tile to tile, from one tile in all to a ragged
last wave.

Tolerance: as for single MLPs against the oracle (1e-2 relative L2, bf16 roundings flipped
by the fp32 summation order), held by every tile by itself and by every row's
largest error: a quarter of the row's largest value (64 bf16 roundings at its size), where
a block from another tile is off by its whole size."""
import numpy as np
import pytest

from oracle.gnn_oracle import GnnOracle, to_bf16
from storm_b200 import gnn

pytestmark = pytest.mark.gpu

SMS = 148


def _close(got, ref):
    got, ref = np.asarray(got, np.float64), np.asarray(ref, np.float64)
    d = (got - ref).reshape(-1, 128 * ref.shape[1])
    r = ref.reshape(d.shape)
    assert np.all(np.linalg.norm(d, axis=1) < 1e-2 * np.linalg.norm(r, axis=1))
    assert np.all(np.abs(got - ref).max(1) < 64 * 2.0 ** -8 * np.abs(ref).max(1))


def _map(rng, kind, rows, n):
    """A row map into n rows: runs of 128, scattered rows with gaps, or both by tile."""
    tiles = rows // 128
    start = rng.integers(0, n - 127, size=tiles)
    run = (start[:, None] + np.arange(128)).ravel()
    any_ = rng.integers(-1, n, size=rows)
    near = run.copy()
    near[127::128] = -1  # a run but for its last row
    if kind == "run":
        out = run
    elif kind == "scatter":
        out = any_
    else:
        pick = np.repeat(rng.integers(0, 3, size=tiles), 128)
        out = np.choose(pick, [run, any_, near])
    return out.astype(np.int32)


@pytest.mark.parametrize("tiles", [1, SMS - 1, SMS + 1, 3 * SMS + 5])
@pytest.mark.parametrize("layer,kinds", [("edge0", ("run", "scatter")), ("edge0", ("mixed", "mixed")), ("node0", ()),
                                         ("enc_edge", ()), ("dec", ())])
def test_forward_many_tiles(storm_lib, tiles, layer, kinds):
    import torch
    net = gnn.WarmStartNet(seed=11)
    dev = net.device
    rng = np.random.default_rng(tiles)
    rows, n = 128 * tiles, 128 * 40

    def mat(r, w):
        a = to_bf16(rng.normal(size=(r, w)))
        return a, torch.tensor(a, dtype=torch.bfloat16, device=dev)

    res = res_t = a1 = f32 = None
    n_out = 64 if layer == "dec" else 128
    orc = GnnOracle(net.specs, net.params_numpy(), net.n_layers)
    if layer == "edge0":
        res, res_t = mat(rows, 128)
        h, h_t = mat(n, 128)
        idx = [_map(rng, k, rows, n) for k in kinds]
        idx_t = [torch.tensor(i, device=dev) for i in idx]
        segs = [net._seg(res_t)] + [net._seg(h_t, idx=i) for i in idx_t]
        A = np.concatenate([res] + [GnnOracle.gather(h, i) for i in idx], axis=1)
        a1 = torch.empty((rows, 128), dtype=torch.bfloat16, device=dev)
    elif layer == "node0":
        res, res_t = mat(rows, 128)
        e, e_t = mat(3 * rows, 128)
        nbr = rng.integers(-1, 3, size=(3, rows)).astype(np.int32)
        nbr_t = torch.tensor(nbr, device=dev)
        segs = [net._seg(res_t), net._seg(e_t, agg=True, stride=rows, nbr=nbr_t)]
        A = np.concatenate([res, orc.agg(e, nbr, rows)], axis=1)
    else:
        A, x_t = mat(rows, 64 if layer == "enc_edge" else 128)
        segs = [net._seg(x_t, A.shape[1])]
        if layer == "dec":
            f32 = torch.empty((rows, 64), dtype=torch.float32, device=dev)
        else:
            a1 = torch.empty((rows, 128), dtype=torch.bfloat16, device=dev)
    out = torch.empty((rows, n_out), dtype=torch.bfloat16, device=dev)
    net._fwd(layer, rows, segs, out, res=res_t, out_f32=f32, a1_save=a1)
    torch.cuda.synchronize()
    net._check_err()
    _, ref, ref_a1 = orc.mlp(layer, A, res=res)  # (the result before and after its rounding)
    _close(out.float().cpu().numpy(), ref)
    if a1 is not None:
        _close(a1.float().cpu().numpy(), ref_a1)
    if f32 is not None:
        _close(f32.cpu().numpy(), ref)


@pytest.mark.parametrize("tiles", [1, SMS + 1, 3 * SMS + 5])
@pytest.mark.parametrize("kind", ["run", "scatter", "mixed"])
def test_forward_does_not_depend_on_saving(storm_lib, tiles, kind):
    """Saving the hidden rows takes a stage from the ring and changes no bit of the output."""
    import torch
    net = gnn.WarmStartNet(seed=14)
    dev = net.device
    rng = np.random.default_rng(tiles)
    rows, n = 128 * tiles, 128 * 40
    x = torch.randn((rows, 128), device=dev).bfloat16()
    h = torch.randn((n, 128), device=dev).bfloat16()
    idx = [torch.tensor(_map(rng, k, rows, n), device=dev) for k in (kind, "run")]
    segs = [net._seg(x)] + [net._seg(h, idx=i) for i in idx]
    out = [torch.empty((rows, 128), dtype=torch.bfloat16, device=dev) for _ in range(2)]
    net._fwd("edge0", rows, segs, out[0], res=x, a1_save=torch.empty_like(out[0]))
    net._fwd("edge0", rows, segs, out[1], res=x)
    torch.cuda.synchronize()
    net._check_err()
    assert torch.equal(out[0].view(torch.int16), out[1].view(torch.int16))


@pytest.mark.parametrize("tiles", [1, SMS + 1, 3 * SMS + 5])
@pytest.mark.parametrize("layer,outs", [("edge0", "axx"), ("edge0", "x0a"), ("node0", "ax"), ("node0", "00"),
                                        ("enc_edge", "0"), ("enc_edge", "a"), ("dec", "x")])
def test_backward_data_many_tiles(storm_lib, tiles, layer, outs):
    """`outs`, a letter a segment: no gradient (0), one (x), one with an addend (a)."""
    import torch
    net = gnn.WarmStartNet(seed=12)
    dev = net.device
    rng = np.random.default_rng(tiles)
    s = net.by_name[layer]
    rows, widths = 128 * tiles, [min(s.k_in, 128)] * len(outs)
    dy = rng.normal(size=(rows, s.n_out)).astype(np.float32)
    a1 = to_bf16(np.maximum(rng.normal(size=(rows, 128)), 0.0))
    add = [rng.normal(size=(rows, w)).astype(np.float32) if o == "a" else None for o, w in zip(outs, widths)]
    dy_t, a1_t = torch.tensor(dy, device=dev), torch.tensor(a1, dtype=torch.bfloat16, device=dev)
    add_t = [None if a is None else torch.tensor(a, device=dev) for a in add]
    out_t = [None if o == "0" else torch.empty((rows, w), dtype=torch.float32, device=dev) for o, w in zip(outs, widths)]
    dz_t = torch.empty((rows, 128), dtype=torch.bfloat16, device=dev)
    net._bwd_data(layer, rows, widths, dy_t, a1_t, dz_t, out_t, add_t)
    torch.cuda.synchronize()
    net._check_err()
    orc = GnnOracle(net.specs, net.params_numpy(), net.n_layers)
    _, w1, _, w2, _ = orc.weights(layer)
    dz = to_bf16((to_bf16(dy) @ w2) * (a1 > 0))
    _close(dz_t.float().cpu().numpy(), dz)
    da = np.asarray(dz, np.float64) @ w1
    for i, (o, a) in enumerate(zip(out_t, add)):
        if o is not None:
            ref = da[:, 128 * i:128 * i + widths[i]]
            _close(o.cpu().numpy(), ref if a is None else ref + a)


@pytest.mark.parametrize("tiles", [1, SMS + 1, 3 * SMS + 5])
@pytest.mark.parametrize("layer,kinds", [("edge0", ("run", "scatter")), ("edge0", ("mixed", "mixed")), ("node0", ()),
                                         ("enc_edge", ()), ("dec", ())])
def test_backward_weight_many_tiles(storm_lib, tiles, layer, kinds):
    """Operands are bf16 on both sides, so only the fp32 sums differ: at most 57,000 random
    terms, about 2^-24 sqrt(n) = 1.4e-5 of a sum; 1e-3 leaves room for the tensor cores'
    own rounding, while one 64-row stage lost or doubled shifts the sums by 3 % or more."""
    import torch
    net = gnn.WarmStartNet(seed=13)
    dev = net.device
    rng = np.random.default_rng(tiles)
    s = net.by_name[layer]
    rows, n = 128 * tiles, 128 * 40

    def mat(r, w):
        a = to_bf16(rng.normal(size=(r, w)))
        return a, torch.tensor(a, dtype=torch.bfloat16, device=dev)

    x, x_t = mat(rows, min(s.k_in, 128))
    segs, A = [net._seg(x_t, x.shape[1])], [x]
    h, h_t = mat(n, 128)
    idx = [_map(rng, k, rows, n) for k in kinds]
    idx_t = [torch.tensor(i, device=dev) for i in idx]
    segs += [net._seg(h_t, idx=i) for i in idx_t]
    A += [GnnOracle.gather(h, i) for i in idx]
    orc = GnnOracle(net.specs, net.params_numpy(), net.n_layers)
    if layer == "node0":
        e, e_t = mat(3 * rows, 128)
        nbr = rng.integers(-1, 3, size=(3, rows)).astype(np.int32)
        nbr_t = torch.tensor(nbr, device=dev)
        segs.append(net._seg(e_t, agg=True, stride=rows, nbr=nbr_t))
        A.append(orc.agg(e, nbr, rows))
    A = np.concatenate(A, axis=1)
    (dz, dz_t), (a1, a1_t) = mat(rows, 128), mat(rows, 128)
    dy = rng.normal(size=(rows, s.n_out)).astype(np.float32)
    dy_t = torch.tensor(dy, device=dev)
    net.grad.zero_()
    net._bwd_weight(layer, rows, segs, dy_t, a1_t, dz_t)
    torch.cuda.synchronize()
    net._check_err()
    got = net.grad.cpu().numpy()[s.offset:s.offset + s.size]
    f = np.float64
    parts = [dz.T.astype(f) @ A.astype(f), dz.sum(0, dtype=f), to_bf16(dy).T.astype(f) @ a1.astype(f), dy.sum(0, dtype=f)]
    o = 0
    for ref in parts:
        g = got[o:o + ref.size].astype(f).reshape(ref.shape)
        assert np.linalg.norm(g - ref) < 1e-3 * np.linalg.norm(ref)
        o += ref.size
    assert o == s.size
