"""Pocket blocking at the edges of the labelling tiles (4 x 8 x 32 points) and of
the link read-back: counts, blocked grids, segment numbers and the device mask
against the oracle's flood fill, exactly."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

T = 250.0


def _check(ctx, E):
    import torch
    ob, on, oseg = oracle.block_pockets(E, T)
    blocked, n, seg = ctx.block_pockets(E, T, want_segments=True)
    assert n == on and np.array_equal(blocked, ob) and np.array_equal(seg, oseg)
    assert ctx.block_pockets(E, T)[1] == on
    grid = torch.from_numpy(E.astype(np.float32)).cuda()
    mask = torch.empty(E.shape, dtype=torch.uint8, device="cuda")
    assert ctx.block_pockets_device(grid.data_ptr(), E.shape, T, mask.data_ptr()) == on
    assert np.array_equal(mask.cpu().numpy() != 0, ob != E)


@pytest.mark.parametrize("dims", [(2, 2, 2), (4, 8, 32), (3, 7, 31), (5, 9, 33), (8, 16, 64), (9, 17, 97),
                                  (13, 2, 65)])
@pytest.mark.parametrize("open_share", [0.3, 0.6, 0.95])
def test_tile_edges(ctx, dims, open_share):
    rng = np.random.default_rng(sum(dims))
    _check(ctx, np.where(rng.random(dims) < open_share, -T, 16 * T))


@pytest.mark.parametrize("axis", [0, 1, 2])
def test_sheets_along_each_axis(ctx, axis):
    """Parallel sheets one point thick: stretches that run through every tile face."""
    E = np.full((9, 17, 66), 16 * T)
    cut = [slice(None)] * 3
    cut[axis] = slice(0, None, 2)
    E[tuple(cut)] = -T
    _check(ctx, E)


def test_more_links_than_the_first_copy(ctx):
    """A checkerboard: isolated points, more than 2048 distinct face links."""
    i, j, k = np.indices((3, 71, 71))
    _check(ctx, np.where((i + j + k) % 2 == 0, -T, 16 * T))


@pytest.mark.parametrize("open_share", [0.25, 0.31, 0.34])
def test_many_links_between_few_roots(ctx, open_share):
    """About where the open points percolate: thousands of links, of roots that have
    one and of roots that have hundreds, channels and pockets among them."""
    rng = np.random.default_rng(7)
    _check(ctx, np.where(rng.random((66, 64, 65)) < open_share, -T, 16 * T))
