"""Meshes whose kernels need shared memory around the 48 KB that a launch may take without
being given more, which the kernel's static variables share with the dynamic part: the cell
kernel on stretched lattices (many edges between its blocks of 256 cells) in either block
size, and the boundary kernels on a boundary of 980 to 984 edges.  Bit for bit against the
oracle, each in a process of its own: a limit raised for an earlier handle stays raised."""
import multiprocessing as mp

import numpy as np
import pytest

from storm_b200 import abi, fvt, scenarios
from test_gpu_cell_blocks import _compare

pytestmark = pytest.mark.gpu

DEFAULT = 48 * 1024


def _spread(x):
    for s, m in ((8, 0x00FF00FF), (4, 0x0F0F0F0F), (2, 0x33333333), (1, 0x55555555)):
        x = (x | (x << s)) & m
    return x


def _cell_smem(sc):
    """The cell kernel's dynamic shared memory (FP64): 36,352 bytes of columns and 24 for each
    edge and wall of the fullest blocks of 256 cells in Morton order."""
    m = fvt.build_mesh(sc.problem).numpy()
    x, y = m["tri_xc"], m["tri_yc"]
    s = max(np.ptp(x), np.ptp(y))
    key = [_spread(np.minimum(65535, np.floor((a - a.min()) / s * 65535.0)).astype(np.uint32)) for a in (x, y)]
    blk = np.empty(m["n_elems"], dtype=np.int64)
    blk[np.argsort(key[0] | (key[1] << 1), kind="stable")] = np.arange(m["n_elems"]) // 256
    e = m["edge_e"].reshape(-1, 2)
    a, b = blk[e[m["flowedg1"][:m["flow_edges1"]] - 1] - 1].T
    n = np.bincount(a, minlength=blk.max() + 1) + np.bincount(b[a != b], minlength=blk.max() + 1)
    w = e[m["walledg1"][:m["wall_edges1"]] - 1].max(axis=1) - 1
    return 36352 + 24 * (int(n.max()) + int(np.bincount(blk[w]).max()))


def _child(kw, steps, out):
    try:
        from oracle import oracle
        _compare(scenarios.channel(**kw), oracle, steps)
        out.put("")
    except BaseException as e:  # as text: not every exception survives the way back
        out.put(repr(e))


def _alone(kw, steps):
    ctx = mp.get_context("spawn")
    out = ctx.Queue()
    p = ctx.Process(target=_child, args=(kw, steps, out), daemon=True)
    p.start()
    assert out.get(timeout=120) == ""
    p.join(timeout=60)


# aspect of the cells, quads along and across; static bytes of the block size they take
@pytest.mark.parametrize("aspect,nx,ny,static", [(18, 60, 70, 768), (15, 65, 130, 768), (22, 60, 300, 768),
                                                 (15, 260, 100, 384), (22, 150, 150, 384)])
def test_stretched_lattices(aspect, nx, ny, static, storm_lib, oracle_mod):
    kw = dict(nx=nx, ny=ny, length=0.5 * aspect * nx, width=0.5 * ny, flux=abi.FLUX_ROE)
    sc = scenarios.channel(**kw)
    assert (sc.n_elems <= 148 * 256) == (static == 768)
    assert DEFAULT - static < _cell_smem(sc) <= DEFAULT
    _alone(kw, 6)


@pytest.mark.parametrize("ny", [980, 981, 982, 983, 984])
def test_long_boundaries(ny, storm_lib, oracle_mod):
    # 48 bytes and two flags an edge, in whole doubles: 983 edges take 48 KB to the byte, and
    # up to 980 leave room for the 128 bytes of static variables
    assert (48 * 983 + (2 * 983 + 7) // 8 * 8) == DEFAULT
    _alone(dict(nx=9, ny=ny, length=4.5, width=0.5 * ny, q=0.5 * ny), 6)
