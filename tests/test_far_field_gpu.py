"""Grids whose bricks interpolate their far field (8 points per thread, spacings
up to about 0.2 A): every point against the FP64 grid with the default mode's
bounds, on cells that leave bricks cut by the grid's end, skewed, or nearly
empty; and the same bits from a single call, the explicit variant and a batch."""
import numpy as np
import pytest

import emptyroom_b200 as er
import oracle
from conftest import grid_errors, rotated_cell
from emptyroom_b200 import serve, synth

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


def _pore(sigma, edge, seed, density=0.08):
    """A wall of atoms of one mixed sigma around an empty sphere that the probe fits into."""
    f = np.random.default_rng(seed).random((int(density * edge ** 3), 3))
    return f[np.linalg.norm((f - 0.5) * edge, axis=1) > sigma + 3.2]


@pytest.mark.parametrize("sigma, spacing", [(5.0, 0.12), (5.0, 0.10), (6.0, 0.12), (8.0, 0.15)])
def test_far_field_of_large_sigma(ctx, sigma, spacing):
    """Bulky probes: the steep terms reach further, and so must the atoms summed one by
    one. Every other point of the grid is a point of the grid of twice the spacing,
    which is too coarse for a far field: what its energies are off by is the rounding
    of the FP32 terms, somewhat less of it (its larger warp boxes take more atoms to
    FP64: a factor of 1.7 between 0.07 and 0.18 A). The interpolation may not add to
    that: root mean square error at most twice the coarse grid's."""
    import torch
    edge = 2.0 * (sigma + 3.2) + 4.0
    frac = _pore(sigma, edge, int(100 * sigma))
    m = int(edge / spacing / 2) + 1
    t = np.diag([edge] * 3)
    fw = ctx.upload(er.particles(frac, np.full(len(frac), 94.0), np.full(len(frac), sigma * sigma)),
                    t, er.replication_factors(t, 12.5), 12.5 ** 2)
    rms, ok = [], None
    for n in (m, 2 * m - 1):
        e = torch.empty((n,) * 3, dtype=torch.float32, device="cuda")
        ref = torch.empty((n,) * 3, dtype=torch.float64, device="cuda")
        ctx.grid_device(fw, (n,) * 3, e.data_ptr())
        ctx.grid_device(fw, (n,) * 3, ref.data_ptr(), precision=er.ER_PREC_FP64, f64=True)
        ctx.synchronize()
        step = 1 if n == m else 2
        e, ref = (x[::step, ::step, ::step] for x in (e, ref))
        ok = ref.abs() < 1e3 if ok is None else ok
        rms.append(float((e.double() - ref)[ok].pow(2).mean().sqrt()))
    fw.release()
    assert int(ok.sum()) > 500
    assert rms[1] <= 2.0 * rms[0]


@pytest.mark.parametrize("abc, angles, n, dims, rotation", [
    ((14.0, 11.0, 12.0), SKEWED, 25, (111, 100, 118), None),
    ((14.0, 11.0, 12.0), SKEWED, 25, (111, 100, 118), 3),
    ((16.0, 14.0, 15.0), CUBIC, 60, (129, 113, 121), 5),
])
def test_far_field_at_moderate_energies(ctx, abc, angles, n, dims, rotation):
    """The energies between the deep and the steep ones too, and cell matrices that
    are not upper triangular: the grid tolerances of the parity tests, on points of
    every kind (the FP64 grid as reference)."""
    import torch
    f = synth.make_framework(700 + n, abc, angles, n, probe="Xe")
    P = f.particles()
    t = f.t_matrix if rotation is None else rotated_cell(f.t_matrix, rotation)
    fw = ctx.upload(P, t, f.rep, f.rc2)
    out = torch.empty(dims, dtype=torch.float32, device="cuda")
    plan = ctx.batch_plan([(fw, dims, out.data_ptr())], er.ER_BATCH_PERSISTENT)
    assert plan.tile(0) == 8  # chosen only where there is a far field
    plan.close()
    e = ctx.grid(fw, dims)
    ref = ctx.grid(fw, dims, precision=er.ER_PREC_FP64, f64=True)
    fw.release()
    rng = np.random.default_rng(8)
    moderate = np.flatnonzero(((ref >= -10.0) & (ref <= 1e3)).ravel())
    assert len(moderate) > 2000
    pick = np.concatenate([rng.choice(moderate, 2000, replace=False), rng.integers(0, ref.size, 3000)])
    pts = np.stack(np.unravel_index(pick, dims), axis=1) / (np.array(dims) - 1.0)
    S = oracle.points_abs(P, t, f.rep, f.rc2, pts)
    st = grid_errors(e.ravel()[pick], ref.ravel()[pick], S)
    assert st["neg_ok"] and st["pos_ok"] and st["cap_ok"], st


def test_far_field_through_every_entry_point(ctx):
    """A fine grid has the same bits from a single call, a batch copied to the host,
    the server and the blocking grid of a Widom batch."""
    import torch
    dims, T = (129, 65, 97), 298.0
    fs = [synth.make_framework(720 + k, (9.0, 8.5, 9.5), (85.0, 97.0, 90.0), 16 + 3 * k, probe="Kr")
          for k in range(3)]
    fws = [ctx.upload(f.particles(), f.t_matrix, f.rep, f.rc2) for f in fs]
    single = [ctx.grid(w, dims) for w in fws]
    out = torch.empty(dims, dtype=torch.float32, device="cuda")
    plan = ctx.batch_plan([(fws[0], dims, out.data_ptr())], er.ER_BATCH_PERSISTENT)
    assert plan.tile(0) == 8
    plan.close()

    hosts = [torch.empty(dims, dtype=torch.float32, pin_memory=True) for _ in fws]
    ctx.grid_batch([(w, dims, h.data_ptr()) for w, h in zip(fws, hosts)],
                   er.ER_BATCH_PERSISTENT | er.ER_BATCH_HOST_OUT)
    for h, s in zip(hosts, single):
        assert np.array_equal(h.numpy(), s)
        h.zero_()

    descs = [serve.framework_desc(f.particles(), f.t_matrix, f.rep, f.rc2) for f in fs]
    with serve.Server(ctx, 4 << 30, slots=3) as srv:
        tickets = [srv.submit_grid(k, d, dims, h.data_ptr()) for k, (d, h) in enumerate(zip(descs, hosts))]
        assert all(srv.wait(t)["status"] == 0 for t in tickets)
    for h, s in zip(hosts, single):
        assert np.array_equal(h.numpy(), s)

    got, pockets = ctx.henry_batch(fws, T, 20000, [1, 2, 3], block_dims=dims)
    for k, (w, s) in enumerate(zip(fws, single)):
        grid = torch.from_numpy(s).cuda()
        mask = torch.empty(dims, dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        assert ctx.block_pockets_device(grid.data_ptr(), dims, T, mask.data_ptr()) == pockets[k]
        assert ctx.henry_device_mask(w, T, 20000, k + 1, mask.data_ptr(), dims) == got[k]
        w.release()
