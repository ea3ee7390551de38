"""FP64 grids at the edges of the staged atom lists: fewer than 32 atoms in reach,
several stages, several flushes of the candidate list, divided and whole bricks.
Bound as for the FP64 mode elsewhere: a few ulps of the sum of |terms|."""
import numpy as np
import pytest

import emptyroom_b200 as er
import oracle
from emptyroom_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("atoms, dims", [(1, (5, 4, 3)), (3, (17, 9, 18)), (60, (2, 2, 2)), (500, (33, 25, 34)),
                                         (900, (12, 11, 10))])
@pytest.mark.parametrize("flags", [0, er.ER_TILE_P8])
def test_fp64_lists_match_oracle(ctx, atoms, dims, flags):
    f = synth.make_framework(40 + atoms, (19.0, 18.0, 20.0), (95.0, 84.0, 103.0), atoms, probe="Xe")
    P = f.particles()
    fw = ctx.upload(P, f.t_matrix, f.rep, f.rc2)
    e = ctx.grid(fw, dims, precision=er.ER_PREC_FP64 | flags, f64=True)
    fw.release()
    ref = oracle.grid(P, f.t_matrix, f.rep, f.rc2, dims)
    S = oracle.grid_abs(P, f.t_matrix, f.rep, f.rc2, dims)
    cap = ref >= er.ER_ENERGY_CAP
    assert np.array_equal(e >= er.ER_ENERGY_CAP, cap)
    assert np.all(np.abs(e[~cap] - ref[~cap]) <= 1e-12 * S[~cap] + 1e-9)
