"""Widom runs where the layout of the insertions changes its kernels (one-CTA and
tiled scan of the bin counts, one or two placement passes, one or several
reduction blocks, 4 or 8 insertions per thread), with and without a pocket mask: K_H against the oracle."""
import numpy as np
import pytest

import oracle
from emptyroom_b200 import synth

pytestmark = pytest.mark.gpu

T = 310.0


@pytest.mark.parametrize("n", [2048, 2049, 1 << 18, (1 << 18) + 1, (3 << 19) - 1, 3 << 19])
@pytest.mark.parametrize("masked", [False, True])
def test_widom_layout_paths(ctx, n, masked):
    f = synth.config1(12)
    P = f.particles()
    fw = ctx.upload(P, f.t_matrix, f.rep, f.rc2)
    mask = (np.random.default_rng(n).random((17, 15, 19)) < 0.02).astype(np.uint8) if masked else None
    r = ctx.henry(fw, T, n, seed=77, block_mask=mask)
    again = ctx.henry(fw, T, n, seed=77, block_mask=mask)
    fw.release()
    assert r == again
    # the cell-list form (equal to the image loop) for the long runs
    sums = oracle.henry if n < 10**6 else oracle.henry_cells
    o = sums(P, f.t_matrix, f.rep, f.rc2, T, 77, n, mask=mask)
    assert r["n_blocked"] == o["n_blocked"] and r["n_insertions"] == n
    assert abs(r["sum_w"] - o["sum_w"]) <= 1e-6 * o["sum_w"]


@pytest.mark.parametrize("dims", [(2, 2, 2), (2, 3, 32), (3, 2, 33), (4, 5, 34), (3, 4, 64), (5, 3, 65),
                                  (2, 2, 66), (65, 33, 2), (40, 2, 97)])
def test_widom_mask_rows(ctx, dims):
    """Mask rows around the 32 cells that a warp takes at a time, and its last
    grid point blocked: the same insertions are blocked as in the oracle."""
    f = synth.config1(12)
    P = f.particles()
    fw = ctx.upload(P, f.t_matrix, f.rep, f.rc2)
    mask = (np.random.default_rng(dims[2]).random(dims) < 0.03).astype(np.uint8)
    mask[-1, -1, -1] = 1
    r = ctx.henry(fw, T, 4096, seed=78, block_mask=mask, want_energies=True)
    fw.release()
    o = oracle.henry(P, f.t_matrix, f.rep, f.rc2, T, 78, 4096, mask=mask, want_energies=True)
    assert r["n_blocked"] == o["n_blocked"] > 0
    assert np.array_equal(np.isinf(r["energies"]), np.isinf(o["energies"]))


@pytest.mark.parametrize("n", [999_999, 10**6])
def test_widom_at_the_line_between_warp_sizes(ctx, n):
    f = synth.make_framework(13, (17.0, 15.0, 19.0), (75.0, 102.0, 96.0), 80, probe="Xe")
    P = f.particles()
    fw = ctx.upload(P, f.t_matrix, f.rep, f.rc2)
    r = ctx.henry(fw, T, n, seed=79)
    fw.release()
    o = oracle.henry_cells(P, f.t_matrix, f.rep, f.rc2, T, 79, n)
    assert abs(r["sum_w"] - o["sum_w"]) <= 1e-6 * o["sum_w"]
