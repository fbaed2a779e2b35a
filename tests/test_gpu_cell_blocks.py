"""The phase path's block shapes against the oracle, bit for bit: cell counts around the
256-slot blocks of the cell kernel and around the count (148 blocks) where it changes its
block size, with dry cells, walls of both kinds, every flux and the limiter's ties (equal
ratios at two faces, which the gradient kernel hands to its careful path)."""
import numpy as np
import pytest

from storm_b200 import abi, fvt, scenarios

pytestmark = pytest.mark.gpu


def _compare(sc, oracle_mod, steps):
    sc.problem.cd[:] = 0.0  # no pow(): every value is then the oracle's, bit for bit
    o = oracle_mod.Oracle(sc.problem, sc.options, threads=8)
    pm = fvt.build_mesh(sc.problem)
    with fvt.Solver(pm, sc.options, keep=pm) as g:
        for s in (o, g):
            s.set_state(sc.h0, sc.u0, sc.v0)
        o.step(steps)
        g.step(steps)
        a, b = o.state(), g.state()
        for k in ("h", "u", "v", "rkh", "rku", "rkv", "hvtx"):
            assert np.array_equal(a[k].view(np.uint64), b[k].view(np.uint64)), k


@pytest.mark.parametrize("nx,ny", [(3, 2), (16, 8), (43, 3), (32, 12), (127, 3)])
@pytest.mark.parametrize("flux,btype", [(abi.FLUX_ROE, 0), (abi.FLUX_HLL, 1), (abi.FLUX_RUSANOV, 0)])
def test_block_edges(nx, ny, flux, btype, storm_lib, oracle_mod):
    sc = scenarios.channel(nx=nx, ny=ny, flux=flux, btype=btype)
    x = sc.problem.x[sc.problem.tri.reshape(-1, 3) - 1].mean(axis=1)
    sc.h0 = np.where(x > 0.7 * x.max(), 0.0, sc.h0)  # a front over a dry bed
    _compare(sc, oracle_mod, 20)  # (without friction the scheme itself blows up on the longest at 23)


@pytest.mark.parametrize("n_target", [37_000, 38_400])
def test_either_block_size(n_target, storm_lib, oracle_mod):
    _compare(scenarios.meander(n_target=n_target, seed=9), oracle_mod, 12)


@pytest.mark.parametrize("limiter", [1, 2])
def test_equal_ratios(limiter, storm_lib, oracle_mod):
    """Symmetric cells with one velocity behind both of two faces: the limiter's ratios tie."""
    sc = scenarios.channel(nx=24, ny=8, noise=0.0, opt_limiter=limiter)
    rng = np.random.default_rng(3)
    n = sc.n_elems
    sc.u0 = np.where(rng.random(n) < 0.5, 0.0, 0.0625)
    sc.v0 = np.where(rng.random(n) < 0.5, 0.0, 0.03125)
    _compare(sc, oracle_mod, 20)


@pytest.mark.parametrize("ny", [2, 15, 16, 17, 33])
@pytest.mark.parametrize("flux,btype,steady", [(abi.FLUX_ROE, 0, 1), (abi.FLUX_HLL, 1, 0), (abi.FLUX_RUSANOV, 1, 1)])
def test_boundary_cells(ny, flux, btype, steady, storm_lib, oracle_mod):
    """The cells with an open-boundary face (2 ny here, those in the corners with a wall too)
    around the 32 that a block of k_flux_bc updates."""
    over = {"steady": steady} if steady else {"steady": 0, "dt_op": 1}
    _compare(scenarios.channel(nx=9, ny=ny, flux=flux, btype=btype, **over), oracle_mod, 10)
