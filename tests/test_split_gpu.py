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

