"""Hard-sphere accessibility masks at the edges of the box marking kernel: bit for
bit the oracle's brute force over the 27 images of every atom."""
import numpy as np
import pytest

import emptyroom_b200 as er
import oracle

pytestmark = pytest.mark.gpu

CUBIC = (9.0, 9.0, 9.0, 90.0, 90.0, 90.0)
SKEWED = (8.5, 11.0, 14.0, 64.0, 118.0, 75.0)
TINY = (2.5, 3.0, 40.0, 90.0, 95.0, 100.0)  # narrower than the spheres along a and b


@pytest.mark.parametrize("cell, dims, n", [
    (CUBIC, (2, 2, 2), 5),          # the smallest grid: only face points
    (CUBIC, (17, 33, 16), 1),       # one atom: its boxes shared among blocks
    (SKEWED, (31, 29, 40), 60),
    (TINY, (11, 9, 64), 12),        # boxes cut on both sides of the cell
    (SKEWED, (2000, 3, 5), 7),      # a box longer than the on-chip axis table
    (CUBIC, (12, 13, 14), 0),       # no atoms
])
def test_accessibility_boxes_match_brute_force(ctx, cell, dims, n):
    rng = np.random.default_rng(n + dims[0])
    t, _, _ = er.cell_matrices(*cell)
    frac = rng.random((n, 3))
    if n > 2:
        frac[0] = 0.0                    # on the corner of the cell
        frac[1] = (0.999999, 0.5, -0.2)  # outside it
    sig2 = rng.uniform(1.0, 16.0, size=n)
    if n > 3:
        sig2[2] = 0.0                    # covers nothing
        sig2[3] = 36.0
    p = er.particles(frac, 50.0, sig2)
    fw = ctx.upload(p, t, er.replication_factors(t, 12.5), 12.5 ** 2)
    got = ctx.accessibility(fw, dims)
    fw.release()
    assert np.array_equal(got, oracle.accessibility(p, t, dims))


DENSE = (7.5, 8.0, 8.5, 80.0, 97.0, 104.0)


@pytest.mark.parametrize("cell, dims, n, spread, sigma", [
    (DENSE, (47, 49, 46), 70, 1.0, 3.7),              # c^2 / n on the points' side of the line
    (DENSE, (33, 30, 31), 80, 1.0, 6.0),              # few points
    ((12.0, 13.0, 12.5, 90.0, 90.0, 90.0), (50, 47, 48), 400, 0.2, 4.0),  # clustered: open points
    (TINY, (51, 60, 64), 37, 1.0, 5.0),               # 999 images: a last tile that is not full
    ((20.0, 6.0, 5.0, 100.0, 90.0, 70.0), (2, 3, 40000), 19, 1.0, 5.0),   # 513 images
])
def test_accessibility_of_many_overlaps_matches_brute_force(ctx, cell, dims, n, spread, sigma):
    """Spheres that overlap so often that the points test the images, not the images
    their boxes."""
    rng = np.random.default_rng(n + dims[0])
    t, _, _ = er.cell_matrices(*cell)
    frac = 0.1 + spread * rng.random((n, 3))
    sig2 = rng.uniform(0.9, 1.1, size=n) * sigma ** 2
    sig2[0] = 0.0
    p = er.particles(frac, 50.0, sig2)
    fw = ctx.upload(p, t, er.replication_factors(t, 12.5), 12.5 ** 2)
    got = ctx.accessibility(fw, dims)
    fw.release()
    assert np.array_equal(got, oracle.accessibility(p, t, dims))
    assert got.any() == (spread < 1.0)
