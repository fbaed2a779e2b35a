"""Timed workloads of the framework, through its public entry points.

Each case is a dict of plain values; ``prepare`` makes what a program holds before the
call (mesh, solver handle, initial state, weights), ``run`` makes one pass and returns
its outputs.  Three kinds of work: the FVT time step on single meshes (``fvt``) and on
ensembles (``batch``), the CFL reduction for callers with their own device arrays
(``cfl``), and the warm-start network: one MLP block (``block``) or all of it (``net``).

The meshes are kept per case, as a program keeps them; the seed decides the state, the
features and the gradients.
"""
import ctypes
import functools
import math

import numpy as np
import torch

from storm_b200 import abi, fvt, gnn, scenarios

FLUX = {"roe": abi.FLUX_ROE, "hll": abi.FLUX_HLL, "rusanov": abi.FLUX_RUSANOV}


def listed():
    return [
        # a host program that couples to the solver every iteration on a small mesh
        # (reads the statistics after each call): launches and latency are all of it
        {"name": "channel_1k_single_steps", "kind": "fvt", "mesh": "channel", "cells": 1200, "flux": "roe",
         "mixed": False, "limiter": 2, "rk": 3, "slip": False, "steps": 20, "per_call": 1, "output": False},
        # the 8,000-cell steady channel marched in pseudo time (HLL, LSQ + BJ, SSP-RK3)
        {"name": "channel_8k_steady", "kind": "fvt", "mesh": "channel", "cells": 8000, "flux": "hll",
         "mixed": False, "limiter": 2, "rk": 3, "slip": False, "steps": 100, "per_call": 100, "output": False},
        # a mid-size transient run that writes vertex output, cell count no round number
        {"name": "meander_131k_output", "kind": "fvt", "mesh": "meander", "cells": 131070, "flux": "roe",
         "mixed": False, "limiter": 2, "rk": 3, "slip": False, "steps": 50, "per_call": 50, "output": True},
        # the transient meander on half a million cells in mixed precision
        {"name": "meander_500k_mixed", "kind": "fvt", "mesh": "meander", "cells": 500000, "flux": "roe",
         "mixed": True, "limiter": 2, "rk": 3, "slip": False, "steps": 60, "per_call": 60, "output": False},
        # wet/dry dam break between walls, Rusanov flux, a million cells
        {"name": "basin_1m_dambreak", "kind": "fvt", "mesh": "basin", "cells": 1000000, "flux": "rusanov",
         "mixed": False, "limiter": 2, "rk": 3, "slip": False, "steps": 60, "per_call": 60, "output": False},
        # the benchmark's size: the transient meander on two million cells, FP64
        {"name": "meander_2m", "kind": "fvt", "mesh": "meander", "cells": 2000000, "flux": "roe",
         "mixed": False, "limiter": 2, "rk": 3, "slip": False, "steps": 100, "per_call": 100, "output": False},
        # the steady ensemble: channels of 2k-8k cells advanced together, first order, mixed
        {"name": "batch_48_steady_mixed", "kind": "batch", "members": 48, "lo": 2000, "hi": 8000, "mixed": True,
         "limiter": 0, "steps": 150},
        # the CFL time step on the caller's own device arrays
        {"name": "cfl_dt_300k", "kind": "cfl", "cells": 300001},
        # the network's edge update (gathered rows, 384 -> 128 -> 128), inference
        {"name": "edge_block_fwd_100k", "kind": "block", "layer": "edge", "cells": 100000, "direction": "forward"},
        # its gradients, data and weights
        {"name": "edge_block_bwd_60k", "kind": "block", "layer": "edge", "cells": 60000, "direction": "backward"},
        # the whole network: a prediction for an ensemble of about 40k cells in all
        {"name": "net_predict_40k", "kind": "net", "cells": 40000, "train": False},
        # forward, loss and gradients of one training batch
        {"name": "net_train_25k", "kind": "net", "cells": 25000, "train": True},
    ]


def _size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["fvt", "fvt", "fvt", "fvt", "batch", "cfl", "block", "block", "net"])
    if kind == "fvt":
        cells = _size(rng, 1000, 600000)
        steps = max(10, min(100, 20000000 // cells))
        return {"kind": "fvt", "mesh": rng.choice(["channel", "meander", "meander", "basin"]), "cells": cells,
                "flux": rng.choice(["roe", "hll", "rusanov"]), "mixed": rng.random() < 0.3,
                "limiter": rng.choice([0, 1, 2, 2, 2]), "rk": rng.choice([2, 3, 3]), "slip": rng.random() < 0.3,
                "steps": steps, "per_call": rng.choice([1, steps, steps]), "output": rng.random() < 0.3}
    if kind == "batch":
        lo = _size(rng, 1000, 6000)
        return {"kind": "batch", "members": rng.randint(3, 40), "lo": lo, "hi": 3 * lo, "mixed": rng.random() < 0.6,
                "limiter": rng.choice([0, 0, 2]), "steps": rng.randint(40, 150)}
    if kind == "cfl":
        return {"kind": "cfl", "cells": _size(rng, 500, 1048576)}
    if kind == "block":
        return {"kind": "block", "layer": rng.choice(["edge", "edge", "node", "encoder", "decoder"]),
                "cells": _size(rng, 200, 60000), "direction": rng.choice(["forward", "backward"])}
    return {"kind": "net", "cells": _size(rng, 200, 30000), "train": rng.random() < 0.5}


# ---- meshes -----------------------------------------------------------------------

def _lattice(nx, ny, lx, ly, rng):
    """Jittered lattice of nx x ny quads (boundary nodes in place), each quad split along
    a diagonal drawn at random, so that the nodes have four to eight cells around them."""
    i, j = np.meshgrid(np.arange(nx + 1), np.arange(ny + 1), indexing="ij")
    inner = ((i > 0) & (i < nx) & (j > 0) & (j < ny)).reshape(-1)
    x = (i.reshape(-1) + inner * rng.uniform(-0.2, 0.2, inner.size)) * (lx / nx)
    y = (j.reshape(-1) + inner * rng.uniform(-0.2, 0.2, inner.size)) * (ly / ny) - ly / 2
    a = (i[:-1, :-1] * (ny + 1) + j[:-1, :-1]).reshape(-1)
    b, c, d = a + ny + 1, a + ny + 2, a + 1
    flip = rng.random(a.size) < 0.5
    tri = np.empty((2 * a.size, 3), dtype=np.int32)
    tri[0::2] = np.stack([a, b, np.where(flip, d, c)], axis=1) + 1
    tri[1::2] = np.stack([np.where(flip, b, a), c, d], axis=1) + 1
    return x, y, tri


def _waves(x, y, length, amp, rng, modes=12):
    """A smooth random field: plane waves of about `length`."""
    k = rng.normal(0.0, 1.0 / length, size=(modes, 2))
    p = rng.uniform(0.0, 2 * np.pi, size=modes)
    out = np.zeros_like(x)
    for m in range(modes):
        out += np.cos(x * k[m, 0] + y * k[m, 1] + p[m])
    return out * (amp * math.sqrt(2.0 / modes))


@functools.lru_cache(maxsize=2)
def _mesh(mesh, cells):
    """(prepared mesh, centroids, bed at the centroids, level, option defaults, output boundary)"""
    rng = np.random.default_rng(1000 + cells)
    if mesh == "channel":
        ny = max(2, int(round(math.sqrt(cells / 20.0))))
        nx = max(4, int(round(cells / (2 * ny))))
        sc = scenarios.channel(nx=nx, ny=ny, length=0.5 * nx, width=0.5 * ny, q=0.5 * ny)
        prob, level = sc.problem, None
        opt = dict(steady=1, stop_cr=1, rstop=1e-12, h_dry=1e-3, h_wet=1e-3)
    elif mesh == "meander":  # sine channel incised into a floodplain of 20:1, 30% dry
        ny = max(3, int(round(math.sqrt(cells / 40.0))))
        nx = max(6, int(round(cells / (2 * ny))))
        x, y, tri = _lattice(nx, ny, 4000.0, 200.0, rng)
        d = np.abs(y - 60.0 * np.sin(2 * np.pi * x / 400.0)) / 20.0
        zb = 0.0005 * (4000.0 - x) + _waves(x, y, 20.0, 0.5, rng) - 2.0 * np.clip(1.0 - d * d, 0.0, None)
        t = tri - 1
        rel = (zb - 0.0005 * (4000.0 - x))[t].mean(axis=1)
        level = float(np.quantile(rel, 0.7))
        ends = lambda col: np.arange(ny + 1) + col * (ny + 1) + 1  # noqa: E731
        prob = abi.ProblemHolder(x, y, tri, zb, rng.uniform(0.02, 0.06, len(tri)),
                                 inflow=[{"type": 1, "nodes": ends(0), "value": 200.0}],
                                 outflow=[{"type": 1, "nodes": ends(nx), "value": level}])
        opt = dict(steady=0, dt_op=1, h_dry=1e-4, h_wet=1e-4)
    else:  # a square basin of walls with mounds
        n = max(3, int(round(math.sqrt(cells / 2.0))))
        x, y, tri = _lattice(n, n, 1000.0, 1000.0, rng)
        x = x - 500.0
        zb = np.clip(_waves(x, y, 60.0, 0.6, rng), 0.0, None)
        prob, level = abi.ProblemHolder(x, y, tri, zb, np.full(len(tri), 0.025)), None
        opt = dict(steady=0, dt_op=1, h_dry=1e-3, h_wet=1e-3)
    pm = fvt.build_mesh(prob)
    t = prob.tri.reshape(-1, 3) - 1
    out = abi.OutputBoundaryHolder(prob, pm.numpy()) if prob.problem.n_elems < 200000 else None
    return pm, prob.x[t].mean(axis=1), prob.y[t].mean(axis=1), prob.zb[t].mean(axis=1), level, opt, out


def _state(mesh, xc, yc, zc, level, rng):
    """Depth and velocities to start from: a wavy surface over the bed with a smooth
    current where it is wet."""
    if mesh == "channel":
        h = np.maximum(rng.uniform(0.8, 1.2) + _waves(xc, yc, 5.0, 0.03, rng), 0.05)
    elif mesh == "meander":
        h = np.maximum(0.0005 * (4000.0 - xc) + level + _waves(xc, yc, 40.0, 0.03, rng) - zc, 0.0)
    else:
        r = rng.uniform(180.0, 300.0)
        h = np.where(np.hypot(xc - rng.uniform(-50, 50), yc) < r, rng.uniform(6.0, 12.0), 0.0)
    h[h < 1e-4] = 0.0
    u = np.where(h > 0.05, _waves(xc, yc, 50.0, 0.2, rng) + 0.2, 0.0)
    v = np.where(h > 0.05, _waves(xc, yc, 50.0, 0.1, rng), 0.0)
    return h, u, v


@functools.lru_cache(maxsize=2)
def _ensemble(members, lo, hi):
    scs = scenarios.batch_channels(members, lo, hi, seed=lo + members)
    return scs, [fvt.build_mesh(s.problem) for s in scs]


@functools.lru_cache(maxsize=2)
def _neighbours(cells):
    """Neighbour tables of channel meshes of `cells` cells in all."""
    tables, left, k = [], cells, 0
    while left > 0:
        n = min(left, 24000 if left > 30000 else left)
        ny = max(2, int(round(math.sqrt(n / 20.0))))
        sc = scenarios.channel(nx=max(3, n // (2 * ny)), ny=ny, seed=k)
        tables.append(gnn.neighbour_table(fvt.build_mesh(sc.problem).numpy()))
        left, k = left - n, k + 1
    return tables


# ---- prepare ----------------------------------------------------------------------

def prepare(case, seed):
    return {"fvt": _prepare_fvt, "batch": _prepare_batch, "cfl": _prepare_cfl, "block": _prepare_block,
            "net": _prepare_net}[case["kind"]](case, seed)


def _prepare_fvt(case, seed):
    pm, xc, yc, zc, level, opt, out = _mesh(case["mesh"], case["cells"])
    o = dict(opt, rkorder=case["rk"], opt_limiter=case["limiter"], flux=FLUX[case["flux"]], cfl=0.9,
             btype=int(case["slip"]), precision=abi.PREC_MIXED if case["mixed"] else abi.PREC_FP64)
    solver = fvt.Solver(pm, fvt.default_options(**o), keep=pm)
    h, u, v = _state(case["mesh"], xc, yc, zc, level, np.random.default_rng(seed))
    return {"case": case, "solver": solver, "start": (h, u, v), "out": out if case["output"] else None}


def _prepare_batch(case, seed):
    scs, meshes = _ensemble(case["members"], case["lo"], case["hi"])
    o = dict(rkorder=3, opt_limiter=case["limiter"], flux=abi.FLUX_HLL, cfl=0.9, steady=1, stop_cr=1, rstop=1e-12,
             h_dry=1e-3, h_wet=1e-3, precision=abi.PREC_MIXED if case["mixed"] else abi.PREC_FP64)
    solver = fvt.BatchSolver(meshes, fvt.default_options(**o), keep=meshes)
    rng = np.random.default_rng(seed)
    start = []
    for s in scs:
        h = s.h0 * rng.uniform(0.95, 1.1)
        start.append((h, np.where(h > 0.05, rng.uniform(0.0, 0.3), 0.0), np.zeros_like(h)))
    return {"case": case, "solver": solver, "start": start}


def _cfl_inputs(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    n = case["cells"]
    r = lambda lo, hi: torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * (hi - lo) + lo  # noqa: E731
    h = torch.clamp(r(-1.0, 3.0), min=0.0)  # a quarter of the cells dry
    return h, r(-1.0, 1.0) * (h > 0), r(-1.0, 1.0) * (h > 0), r(0.1, 0.4), r(1.2, 2.4)


def _prepare_cfl(case, seed):
    return {"case": case, "in": _cfl_inputs(case, seed), "dt": torch.zeros(1, device="cuda", dtype=torch.float64)}


_BLOCKS = {"edge": "edge0", "node": "node0", "encoder": "enc_edge", "decoder": "dec"}


def _block_inputs(case, seed):
    """Weights, input rows and row maps of one MLP block; the 64-bit check reads them too."""
    net = gnn.WarmStartNet(seed=seed)
    s, w1, b1, w2, b2 = net._wv(_BLOCKS[case["layer"]])
    g = torch.Generator(device="cuda").manual_seed(seed)
    rnd = lambda *n: torch.randn(*n, generator=g, device="cuda")  # noqa: E731
    b1[:gnn.HID].copy_(0.1 * rnd(gnn.HID))
    b2[:s.n_out].copy_(0.1 * rnd(s.n_out))
    nbr_l = _neighbours(case["cells"])
    T = sum(t.shape[1] for t in nbr_l)
    Tp = (T + 127) // 128 * 128
    off = np.cumsum([0] + [t.shape[1] for t in nbr_l])
    nbr = np.full((3, Tp), -1, dtype=np.int32)
    for o, t in zip(off, nbr_l):
        nbr[:, o:o + t.shape[1]] = np.where(t >= 0, t + o, -1)
    dst = np.tile(np.where(np.arange(Tp) < T, np.arange(Tp), -1).astype(np.int32), 3)
    st = {"case": case, "net": net, "spec": s, "w": (w1, b1, w2, b2), "Tp": Tp,
          "nbr": torch.from_numpy(nbr.reshape(-1)).cuda(), "dst": torch.from_numpy(dst).cuda()}
    edges = case["layer"] in ("edge", "encoder")
    st["rows"] = rows = 3 * Tp if edges else Tp
    st["x"] = rnd(rows, 64 if case["layer"] == "encoder" else gnn.HID).bfloat16()
    st["other"] = rnd(3 * Tp if case["layer"] == "node" else Tp, gnn.HID).bfloat16()
    st["dy"] = 1e-3 * rnd(rows, s.n_out)
    st["add"] = 1e-3 * rnd(rows, s.n_out)
    st["a1"] = torch.relu(rnd(rows, gnn.HID)).bfloat16()
    return st


def _segments(st):
    """[(matrix, row map, aggregated)] of the block's input."""
    layer, x, other = st["case"]["layer"], st["x"], st["other"]
    if layer == "edge":
        return [(x, None, False), (other, st["nbr"], False), (other, st["dst"], False)]
    if layer == "node":
        return [(x, None, False), (other, None, True)]
    return [(x, None, False)]


def _prepare_block(case, seed):
    st = _block_inputs(case, seed)
    net, s, rows, Tp = st["net"], st["spec"], st["rows"], st["Tp"]
    segs = []
    for m, idx, agg in _segments(st):
        q = gnn.Seg()
        q.src, q.width = m.data_ptr(), m.shape[1]
        q.idx = idx.data_ptr() if idx is not None else None
        if agg:
            q.agg, q.agg_stride, q.nbr = 1, Tp, st["nbr"].data_ptr()
        segs.append(q)
    w1, b1, w2, b2 = (t.data_ptr() for t in st["w"])
    dev = {"device": "cuda"}
    st["err"] = torch.zeros(1, dtype=torch.int32, **dev)
    res = case["layer"] in ("edge", "node")
    if case["direction"] == "forward":
        st["out"] = torch.empty((rows, s.n_out), dtype=torch.bfloat16, **dev)
        a = gnn.MlpFwd()
        a.w1, a.b1, a.w2, a.b2, a.out = w1, b1, w2, b2, st["out"].data_ptr()
        a.res = st["x"].data_ptr() if res else None
        st["calls"] = [a]
    else:
        st["dz1"] = torch.empty((rows, gnn.HID), dtype=torch.bfloat16, **dev)
        st["grad"] = torch.empty(s.size, dtype=torch.float32, **dev)
        st["scratch"] = torch.empty(int(gnn.lib().storm_gnn_weight_scratch_bytes(s.k_in, s.n_out)) // 4 + 1,
                                    dtype=torch.float32, **dev)
        a, b = gnn.MlpBwdData(), gnn.MlpBwdWeight()
        a.w1, a.w2, a.dz1_save = w1, w2, st["dz1"].data_ptr()
        a.dy = b.dy = st["dy"].data_ptr()
        a.a1 = b.a1 = st["a1"].data_ptr()
        b.dz1 = st["dz1"].data_ptr()
        st["dseg"] = []
        for i, q in enumerate(segs):
            a.seg_width[i] = q.width
            if case["layer"] != "encoder":  # nothing before the encoder wants its gradient
                st["dseg"].append(torch.empty((rows, q.width), dtype=torch.float32, **dev))
                a.dseg[i] = st["dseg"][-1].data_ptr()
                a.dseg_add[i] = st["add"].data_ptr() if res and i == 0 else None
        st["calls"] = [a, b]
    for a in st["calls"]:
        a.rows, a.nseg, a.k_in, a.n_out = rows, len(segs), s.k_in, s.n_out
        if not isinstance(a, gnn.MlpBwdData):
            for i, q in enumerate(segs):
                a.seg[i] = q
    st["keep"] = segs
    return st


def _prepare_net(case, seed):
    tables = _neighbours(case["cells"])
    rng = np.random.default_rng(seed)
    n = [t.shape[1] for t in tables]
    xn = [rng.standard_normal((k, gnn.IN_NODE), dtype=np.float32) for k in n]
    xe = [rng.standard_normal((3, k, gnn.IN_EDGE), dtype=np.float32) for k in n]
    g = gnn.build_graph_fast(tables, xn, xe)
    net = gnn.WarmStartNet(seed=seed)
    st = {"case": case, "net": net, "graph": gnn.DeviceGraph(g, net.device), "cells": g.T}
    if case["train"]:
        st["target"] = torch.from_numpy(rng.standard_normal((g.Tp, 3), dtype=np.float32)).cuda()
        st["mask"] = torch.from_numpy((np.arange(g.Tp) < g.T).astype(np.float32)).cuda()
    return st


# ---- run --------------------------------------------------------------------------

def run(state):
    return {"fvt": _run_fvt, "batch": _run_batch, "cfl": _run_cfl, "block": _run_block,
            "net": _run_net}[state["case"]["kind"]](state)


_STATS = ("iter", "ttime", "stime", "delt", "rmax", "rms_dh", "tmass")


def _run_fvt(st):
    """From a given state: so many iterations, then the state (and vertex output) back."""
    s, case = st["solver"], st["case"]
    s.set_state(*st["start"])
    for _ in range(case["steps"] // case["per_call"]):
        stats = s.step(case["per_call"])
    out = {k: stats[k] for k in _STATS}
    if st["out"] is not None:
        out["vertices"] = s.output_vertices(st["out"])
    out.update(s.state(("h", "u", "v", "hvtx")))
    return out


def _run_batch(st):
    s = st["solver"]
    for i, (h, u, v) in enumerate(st["start"]):
        s.set_scenario_state(i, h, u, v)
    s.step(st["case"]["steps"])
    got = [s.scenario_state(i) for i in range(s.n)]
    out = {k: np.concatenate([g[k] for g in got]) for k in ("h", "u", "v", "hvtx")}
    out["rms_dh"] = np.array([s.scenario_stats(i)["rms_dh"] for i in range(s.n)])
    return out


def _run_cfl(st):
    h, u, v, area, perim = st["in"]
    rc = fvt.lib().storm_fvt_cfl_dt_noalloc(h.data_ptr(), u.data_ptr(), v.data_ptr(), area.data_ptr(), perim.data_ptr(),
                                            h.numel(), 0.9, 1e-3, 1e-3, st["dt"].data_ptr(),
                                            torch.cuda.current_stream().cuda_stream)
    if rc:
        raise RuntimeError(fvt.lib().storm_fvt_last_error().decode())
    return st["dt"]


def _run_block(st):
    L, err = gnn.lib(), st["err"].data_ptr()
    stream = torch.cuda.current_stream().cuda_stream
    if len(st["calls"]) == 1:
        rc = L.storm_gnn_mlp_forward(ctypes.byref(st["calls"][0]), err, stream)
        out = {"out": st["out"]}
    else:
        a, b = st["calls"]
        rc = L.storm_gnn_mlp_backward_data(ctypes.byref(a), err, stream) or L.storm_gnn_mlp_backward_weight(
            ctypes.byref(b), st["grad"].data_ptr(), st["scratch"].data_ptr(), 4 * st["scratch"].numel(), err, stream)
        out = {"dz1": st["dz1"], "dseg": st["dseg"], "grad": st["grad"]}
    if rc:
        raise RuntimeError(fvt.lib().storm_fvt_last_error().decode())
    return out


def _run_net(st):
    net, case = st["net"], st["case"]
    y = net.forward(st["graph"], save=case["train"])
    if not case["train"]:
        return {"y": y}
    dy, parts = net.mse(y, st["target"], st["mask"], 3.0 * st["cells"])
    net.backward(dy)
    return {"y": y, "loss": parts, "grad": net.grad}


# ---- work and 64-bit values ---------------------------------------------------------

_MLP_NET = [("enc_node", 64, 128), ("enc_edge", 64, 128)] + [("edge", 384, 128), ("node", 256, 128)] * gnn.N_LAYERS + [
    ("dec", 128, 64)]


def _mlp_work(layer, cells, k_in, n_out, backward):
    rows = 3 * cells if layer in ("edge", "enc_edge", "encoder") else cells
    macs = k_in * gnn.HID + gnn.HID * n_out
    # matrices read, 2 bytes a value: own rows, the gathered cells once, the messages
    read = {"edge": 3 + 1, "node": 1 + 3, "enc_node": 0.5, "enc_edge": 1.5, "encoder": 1.5}.get(layer, 1) * cells * 256
    if not backward:
        return read + 2.0 * rows * n_out, 2.0 * rows * macs
    dseg = 0 if layer in ("enc_node", "enc_edge", "encoder") else 4 * k_in
    add = 4 * gnn.HID if layer in ("edge", "node") else 0
    return (read + rows * (4.0 * n_out + 2 * 2 * gnn.HID + dseg + add),
            2.0 * rows * (macs + gnn.HID * n_out + (gnn.HID * k_in if dseg else 0)))


def work(case):
    kind = case["kind"]
    if kind == "cfl":
        return {"bytes": 40.0 * case["cells"], "flops": 12.0 * case["cells"]}
    if kind == "block":
        k_in, n_out = {"edge": (384, 128), "node": (256, 128), "encoder": (64, 128), "decoder": (128, 64)}[case["layer"]]
        b, f = _mlp_work(case["layer"], case["cells"], k_in, n_out, case["direction"] == "backward")
        return {"bytes": b, "flops": f}
    if kind == "net":
        b = f = 0.0
        for name, k_in, n_out in _MLP_NET:
            for back in (False, True)[:2 if case["train"] else 1]:
                x, y = _mlp_work(name, case["cells"], k_in, n_out, back)
                b, f = b + x, f + y
        return {"bytes": b, "flops": f}
    if kind == "batch":
        cells = sum(p["n_cells"] for p in scenarios.batch_channel_params(case["members"], case["lo"], case["hi"],
                                                                         case["lo"] + case["members"]))
    else:
        cells = case["cells"]
    # one fused stage reads and writes each array of the scheme once (FP32 geometry and
    # gradients on the mixed path); a stage makes about 600 operations per cell
    per = scenarios.algorithmic_bytes_per_cell_stage(cells, 1.5 * cells, 0.5 * cells)
    if case["mixed"]:
        per *= 0.72
    stages = case.get("rk", 3) * case["steps"]
    return {"bytes": per * cells * stages + 48.0 * cells, "flops": 600.0 * cells * stages}


def exact(case, seed):
    """The 64-bit values of the CFL step and of one MLP block.  A time step has none short
    of a second solver, and the whole network's are those of its blocks."""
    if case["kind"] == "cfl":
        h, u, v, area, perim = _cfl_inputs(case, seed)
        wet = h >= 1e-3
        speed = torch.where(wet, torch.sqrt(u * u + v * v) + torch.sqrt(9.81 * h), torch.zeros_like(h))
        return (0.9 * area / ((speed + float(np.float32(1e-9))) * perim)).min().reshape(1)
    if case["kind"] != "block":
        return None
    st = _block_inputs(case, seed)
    s, Tp, rows = st["spec"], st["Tp"], st["rows"]
    w1, b1, w2, b2 = st["w"]
    w1 = w1[:gnn.HID * s.k_in].double().reshape(gnn.HID, s.k_in)
    w2 = w2[:s.n_out * gnn.HID].double().reshape(s.n_out, gnn.HID)
    b1, b2 = b1[:gnn.HID].double(), b2[:s.n_out].double()
    parts = []
    for m, idx, agg in _segments(st):
        m = m.double()
        if agg:
            m = (m.reshape(3, Tp, -1) * (st["nbr"].reshape(3, Tp, 1) >= 0)).sum(0)
        elif idx is not None:
            m = torch.where((idx >= 0)[:, None], m[idx.clamp(min=0).long()], torch.zeros((), dtype=m.dtype, device=m.device))
        parts.append(m)
    A = torch.cat(parts, dim=1)
    res = case["layer"] in ("edge", "node")
    if case["direction"] == "forward":
        y = torch.relu(A @ w1.T + b1) @ w2.T + b2
        return {"out": y + st["x"].double() if res else y}
    dy, a1 = st["dy"].double(), st["a1"].double()
    dz1 = (dy @ w2) * (a1 > 0)
    dA = dz1 @ w1
    widths = [m.shape[1] for m in parts]
    dseg = list(torch.split(dA, widths, dim=1)) if case["layer"] != "encoder" else []
    if res:
        dseg[0] = dseg[0] + st["add"].double()
    grad = torch.cat([(dz1.T @ A).reshape(-1), dz1.sum(0), (dy.T @ a1).reshape(-1), dy.sum(0)])
    return {"dz1": dz1, "dseg": dseg, "grad": grad}
