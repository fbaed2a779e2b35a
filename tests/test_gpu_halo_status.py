"""Values that are not finite are reported by the part that owns the cell, not by the parts that
hold a copy of it (which leave copies out of all their sums as well)."""
import numpy as np
import pytest

from storm_b200 import abi, fvt, partition, scenarios

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("path", [fvt.STAGE_PHASES, fvt.STAGE_FUSED])
@pytest.mark.parametrize("elem", [1, 101])  # with an open-boundary face, and within
def test_halo_copy_not_finite(elem, path, storm_lib):
    import torch
    sc = scenarios.channel(nx=30, ny=6, flux=abi.FLUX_ROE, steady=0, dt_op=1)
    part = partition.GpuPartEngine(sc.problem, sc.options, 0.0, stage_path=path)
    try:
        for halo in (True, False):
            part.set_exchange([], [elem] if halo else [elem + 1])
            part.set_state(sc.h0, sc.u0, sc.v0)
            dt = part.iter_begin()
            part.iter_set_dt(dt)
            for s in (1, 2, 3):
                part.iter_stage(s)
            if not halo:  # the same value, in a cell of the part's own
                part.set_exchange([], [elem])
            part.unpack(3, False, torch.full((6,), float("nan"), dtype=torch.float64, device="cuda"))
            if not halo:
                part.set_exchange([], [elem + 1])
            sums = part.iter_fric(dt, None)
            st = part.iter_finish(sums)
            assert np.isfinite(sums).all() == halo
            assert st["device_status"] == (0 if halo else 1)
    finally:
        part.close()
