"""Which kernels a call launches, where the choice is the point: read from the CUDA
activity that torch's profiler records."""
import numpy as np
import pytest

import emptyroom_b200 as er
from emptyroom_b200 import synth

pytestmark = pytest.mark.gpu


def _kernels(ctx, call):
    """Names of the library's kernels that `call` launches."""
    import torch
    torch.cuda.init()
    activities = [torch.profiler.ProfilerActivity.CUDA]
    with torch.profiler.profile(activities=activities, acc_events=True) as p:
        call()
        ctx.synchronize()
    return [e.name for e in p.events() if "er::" in e.name]


@pytest.mark.parametrize("n, points", [(999_999, 4), (1_000_000, 8), (1_500_000, 8)])
def test_widom_warps_of_long_runs(ctx, n, points):
    """From 10^6 insertions on a warp takes 256 of them: with 128 its box has fewer
    atoms near enough for FP64 terms, and the energies are less accurate."""
    f = synth.make_framework(3, (16.0, 16.0, 16.0), (90.0, 90.0, 90.0), 24)
    fw = ctx.upload(f.particles(), f.t_matrix, f.rep, f.rc2)
    names = [k for k in _kernels(ctx, lambda: ctx.henry(fw, 298.0, n, seed=1)) if "henry_energy" in k]
    fw.release()
    assert len(names) == 1 and f"henry_energy_kernel<{points}, 1>" in names[0]


def _variants(names):
    """(points per thread, CTAs per brick) of the grid kernels among `names`."""
    return {tuple(int(x) for x in k.split("grid_kernel<")[1].split(">")[0].split(",")[1:])
            for k in names if "grid_kernel<" in k}


@pytest.mark.parametrize("n, split", [(32, 4), (50, 2), (80, 1)])
def test_autotuner_times_what_the_plan_runs(n, split):
    """A batch in one launch never divides its bricks, a launch of its own does where
    they are few: the tuner times the one or the other."""
    import torch
    f = synth.config1(0)
    out = torch.empty((n,) * 3, dtype=torch.float32, device="cuda")
    for mode, division in ((er.ER_BATCH_PERSISTENT, 1), (er.ER_BATCH_PLAIN, split)):
        with er.Context(0) as ctx:  # nothing tuned yet
            fw = ctx.upload(f.particles(), f.t_matrix, f.rep, f.rc2)
            plans = []
            names = _kernels(ctx, lambda: plans.append(ctx.batch_plan(
                [(fw, out.shape, out.data_ptr())], mode | er.ER_BATCH_AUTOTUNE | er.ER_BATCH_COMP)))
            plans[0].close()
            fw.release()
        assert _variants(names) == {(4, division), (8, 1)}


@pytest.mark.parametrize("edge, n, sigma, dims, kernel", [
    (25.8, 424, 3.5, 65, "acc_mark_kernel"), (12.0, 259, 3.7, 65, "acc_mark_kernel"),
    (8.0, 76, 3.7, 65, "acc_points_kernel"), (6.0, 32, 7.0, 33, "acc_points_kernel"),
    (6.0, 4, 3.7, 65, "acc_points_kernel")])
def test_accessibility_of_many_overlaps_goes_by_points(ctx, edge, n, sigma, dims, kernel):
    """Where every point lies in dozens of boxes, testing it against the images until
    one covers it is faster than marking every box."""
    t = np.diag([edge] * 3)
    frac = np.random.default_rng(1).random((n, 3))
    fw = ctx.upload(er.particles(frac, 50.0, sigma ** 2), t, er.replication_factors(t, 12.5), 12.5 ** 2)
    names = _kernels(ctx, lambda: ctx.accessibility(fw, (dims,) * 3))
    fw.release()
    assert [k for k in ("acc_mark_kernel", "acc_points_kernel") if any(k in x for x in names)] == [kernel]


@pytest.mark.parametrize("dims, tile", [((94, 200, 47), 4),    # 450 bricks of P = 8 on 444 CTA slots
                                        ((94, 200, 94), 8),    # twice as many
                                        ((80, 80, 80), 8)])    # 250: two on most SMs, 500 of P = 4
def test_larger_bricks_where_their_launch_ends_well(ctx, dims, tile):
    """A far field is worth P = 8 unless its few bricks leave most of the last wave
    idle (the spacing is 0.13 A in each case)."""
    import torch
    abc = tuple(0.13 * (d - 1) for d in dims)
    f = synth.make_framework(31, abc, (90.0, 90.0, 90.0), int(0.03 * np.prod(abc)))
    fw = ctx.upload(f.particles(), f.t_matrix, f.rep, f.rc2)
    out = torch.empty(dims, dtype=torch.float32, device="cuda")
    plan = ctx.batch_plan([(fw, dims, out.data_ptr())], er.ER_BATCH_PERSISTENT)
    got = plan.tile(0)
    plan.close()
    fw.release()
    assert got == tile


def test_a_small_job_is_not_tuned_by_a_large_one(ctx):
    """Two jobs of one density and spacing: the large one may run 8 points per thread,
    the small one on its own, whose bricks would halve to 20, may not."""
    import torch
    f = synth.make_framework(32, (32.0, 32.0, 32.0), (90.0, 90.0, 90.0), 810)
    with er.Context(0) as own:  # nothing tuned yet
        fw = own.upload(f.particles(), f.t_matrix, f.rep, f.rc2)
        out = torch.empty((160,) * 3, dtype=torch.float32, device="cuda")
        tiles = []
        for dims in ((160, 160, 160), (160, 16, 16)):
            plan = own.batch_plan([(fw, dims, out.data_ptr())],
                                  er.ER_BATCH_PERSISTENT | er.ER_BATCH_AUTOTUNE | er.ER_BATCH_COMP)
            tiles.append(plan.tile(0))
            plan.close()
        fw.release()
    assert tiles[0] in (4, 8) and tiles[1] == 4
