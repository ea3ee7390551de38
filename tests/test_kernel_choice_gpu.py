"""Which kernels a call launches, where the choice is the point: read from the CUDA
activity that torch's profiler records."""
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
