"""The state read back by every route the library has for it (whole records up to 16,384 cells,
dry flags up to 8,192; columns written by a kernel beyond), on both sides of the limits."""
import numpy as np
import pytest

from storm_b200 import fvt, scenarios

pytestmark = pytest.mark.gpu


def _state(n, seed):
    rng = np.random.default_rng(seed)
    h = np.where(rng.random(n) < 0.3, rng.uniform(0.0, 2e-3, n), rng.uniform(0.5, 2.0, n))
    u, v = (np.where(rng.random(n) < 0.5, 0.0, rng.normal(size=n)) for _ in range(2))
    return h, u, v


def _check(got, h, u, v):
    for k, x in (("h", h), ("u", u), ("v", v), ("rkh", h), ("rku", h * u), ("rkv", h * v)):
        if k in got:
            assert np.array_equal(got[k].view(np.uint64), x.view(np.uint64)), k


@pytest.mark.parametrize("nx,ny", [(2, 1), (64, 64), (241, 17), (64, 128), (121, 68), (150, 150)])
def test_read_back(nx, ny, storm_lib):
    sc = scenarios.channel(nx=nx, ny=ny, h_dry=1e-3, h_wet=1.5e-3)
    h, u, v = _state(sc.n_elems, nx)
    pm = fvt.build_mesh(sc.problem)
    with fvt.Solver(pm, sc.options, keep=pm) as s:
        s.set_state(h, u, v)
        for keys in (("h", "u", "v"), ("h",), ("u", "v"), ("v",), ("h", "u", "v", "rkh", "rku", "rkv")):
            _check(s.state(keys), h, u, v)
        dry = (h < 1e-3) | ((h < 1.5e-3) & (u * u + v * v == 0.0))
        assert np.array_equal(np.asarray(s.drycell()) != 0, dry)


def test_read_back_batch(storm_lib):
    scs = [scenarios.channel(nx=nx, ny=ny) for nx, ny in ((30, 7), (150, 60), (20, 20))]
    pms = [fvt.build_mesh(sc.problem) for sc in scs]
    with fvt.BatchSolver(pms, scs[0].options, keep=pms) as s:
        st = [_state(sc.n_elems, i) for i, sc in enumerate(scs)]
        for i, x in enumerate(st):
            s.set_scenario_state(i, *x)
        for i, x in reversed(list(enumerate(st))):
            _check(s.scenario_state(i), *x)
