"""Grids of few bricks run on several CTAs per brick (2 or 4): every energy equals,
bit for bit, the one of the undivided bricks that a batch runs. (Widom runs whose
CTAs are divided are held to the oracle by the Henry tests, from 1 insertion on.)"""
import numpy as np
import pytest

import emptyroom_b200 as er
from emptyroom_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(2, 2, 2), (9, 8, 16), (8, 9, 17), (32, 32, 32), (40, 39, 41), (70, 33, 66)])
@pytest.mark.parametrize("comp", [False, True])
def test_split_bricks_keep_the_bits(ctx, dims, comp):
    import torch
    f = synth.make_framework(6, (17.0, 21.0, 19.0), (70.0, 101.0, 95.0), 400)
    fw = ctx.upload(f.particles(), f.t_matrix, f.rep, f.rc2)
    single = ctx.grid(fw, dims, precision=er.ER_PREC_COMP if comp else er.ER_PREC_NEAR64)
    out = torch.empty(dims, dtype=torch.float32, device="cuda")
    ctx.grid_batch([(fw, dims, out.data_ptr())], er.ER_BATCH_COMP if comp else er.ER_BATCH_PERSISTENT)
    assert np.array_equal(single, out.cpu().numpy())
    fw.release()



@pytest.mark.parametrize("n_jobs, dims", [(1, (86, 67, 35)), (3, (19, 40, 33)), (5, (2, 3, 2)), (2, (60, 64, 66))])
def test_small_plans_replay(ctx, n_jobs, dims):
    """Launches whose bricks all fit on the GPU are handed out by a counter that each
    replay leaves as it found it: every replay writes every point (the last case has
    too many bricks for that)."""
    import torch
    f = synth.make_framework(7, (17.0, 21.0, 19.0), (70.0, 101.0, 95.0), 200)
    fw = ctx.upload(f.particles(), f.t_matrix, f.rep, f.rc2)
    single = ctx.grid(fw, dims)
    outs = [torch.empty(dims, dtype=torch.float32, device="cuda") for _ in range(n_jobs)]
    plan = ctx.batch_plan([(fw, dims, o.data_ptr()) for o in outs], er.ER_BATCH_PERSISTENT)
    for _ in range(3):
        for o in outs:
            o.fill_(float("nan"))
        torch.cuda.synchronize()
        plan.run()
        ctx.synchronize()
        assert all(np.array_equal(o.cpu().numpy(), single) for o in outs)
    plan.close()
    fw.release()
