"""Grids whose bricks interpolate their far field (8 points per thread, spacings
up to about 0.2 A): every point against the FP64 grid with the default mode's
bounds, on cells that leave bricks cut by the grid's end, skewed, or nearly
empty; and the same bits from a single call, the explicit variant and a batch."""
import numpy as np
import pytest

import emptyroom_b200 as er
from emptyroom_b200 import synth

pytestmark = pytest.mark.gpu

CUBIC, SKEWED = (90.0, 90.0, 90.0), (62.0, 117.0, 74.0)


@pytest.mark.parametrize("abc, angles, n, dims", [
    ((9.0, 8.5, 9.5), CUBIC, 18, (129, 65, 97)),        # one line past whole bricks along each axis
    ((14.0, 11.0, 12.0), SKEWED, 60, (111, 100, 118)),
    ((11.0, 12.0, 10.0), SKEWED, 130, (136, 95, 120)),  # dense, 0.08 A along the first axis
    ((16.0, 9.0, 15.0), CUBIC, 40, (96, 72, 83)),       # 0.18 A: a thin far shell
    ((20.0, 8.0, 9.0), CUBIC, 3, (160, 64, 72)),        # almost no atoms
])
def test_far_field_against_fp64(ctx, abc, angles, n, dims):
    import torch
    f = synth.make_framework(300 + n, abc, angles, n, probe="CH4")
    fw = ctx.upload(f.particles(), f.t_matrix, f.rep, f.rc2)
    e = ctx.grid(fw, dims, precision=er.ER_TILE_P8)
    ref = ctx.grid(fw, dims, precision=er.ER_PREC_FP64, f64=True)
    cap = ref >= er.ER_ENERGY_CAP
    assert np.array_equal(e >= np.float32(er.ER_ENERGY_CAP), cap)
    d = np.abs(e.astype(np.float64) - ref)
    deep, high = ref < -10.0, (ref > 1e3) & ~cap
    assert (deep | high).sum() > 100  # the skewed cells are too dense for pores
    assert np.all(d[deep] <= 1e-5 * np.abs(ref[deep]))
    assert np.all(d[high] <= 1e-4 * ref[high])
    out = torch.empty(dims, dtype=torch.float32, device="cuda")
    plan = ctx.batch_plan([(fw, dims, out.data_ptr())], er.ER_BATCH_PERSISTENT)
    plan.run()
    ctx.synchronize()
    same = e if plan.tile(0) == 8 else ctx.grid(fw, dims)
    assert np.array_equal(out.cpu().numpy(), same)
    assert np.array_equal(ctx.grid(fw, dims), same)
    plan.close()
    fw.release()
