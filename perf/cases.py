"""Performance cases: the work that programs have this library do, at the sizes they have it do it.

A case is a dict of plain values; its "kind" names the call:

  grid        one probe-framework energy grid (the grid behind `writegrid`), left on the device or
              copied to the host, in one of the precision modes
  batch       a screening batch of triclinic frameworks, one work queue kept as a plan
  batch_small a screening batch of many coarse grids, one one-shot call
  henry       Widom insertions of one framework (the sum behind `henry`), with or without a pocket mask
  henry_batch a Widom screening batch: blocking grid, pocket mask and insertions per framework
  pockets     the pocket mask of an energy grid on the device
  interp      GCMC guest energies looked up in an energy grid
  access      the hard-sphere accessibility mask of a framework

prepare() builds what a program holds before the call (uploaded frameworks, plans, grids, guest
positions), run() is one call of the public entry points, exact() is the same result in FP64 from
plain torch, and work() counts the operations and bytes that the result cannot do without.

Frameworks are synthetic, as in the tests and the benchmark: atoms on randomly chosen, displaced
sites of a fine lattice, atom types with epsilon in [20, 100] K and sigma in [2.5, 3.8] A, probes
CH4 / Xe / Kr, cutoff 12.5 A.
"""
import math
import random

import numpy as np
import torch

import emptyroom_b200 as er

RC = 12.5
PROBES = {"CH4": (148.0, 3.73), "Xe": (221.0, 4.10), "Kr": (166.4, 3.636)}
MAX_DENSITY = 0.16  # atoms / A^3
CAP = 1.0e30        # energies at and above it are written as it
# FP32-pipe operations of one in-cutoff pair term: r^2 (3 sub, 1 mul, 2 fma), 1 rcp, u^3 (2 mul),
# C12 u^3 - C6 and the accumulation (2 fma); an fma counts twice
PAIR_FLOPS = 15

CUBIC = dict(a=25.8, b=25.8, c=25.8, alpha=90.0, beta=90.0, gamma=90.0, atoms=424, types=4)


def listed():
    return [
        # the coarse grid of a quick look at one material: the smallest call of the library
        dict(CUBIC, name="grid_32", kind="grid", probe="CH4", nx=32, ny=32, nz=32, prec="near64", host=False),
        # the usual grid: a 25.8 A cell at 0.2 A, kept on the device for what follows
        dict(CUBIC, name="grid_129", kind="grid", probe="Xe", nx=129, ny=129, nz=129, prec="near64", host=False),
        # a dense triclinic cell at 0.12 A: the largest single grid
        dict(name="grid_256_dense", kind="grid", a=30.1, b=32.4, c=28.7, alpha=85.0, beta=95.0, gamma=110.0,
             atoms=4096, types=4, probe="CH4", nx=256, ny=256, nz=256, prec="near64", host=False),
        # FP64 throughout, in host memory: the grid as the original program's arithmetic gives it; odd sizes
        dict(CUBIC, name="grid_fp64_host", kind="grid", probe="Kr", nx=65, ny=63, nz=61, prec="fp64", host=True),
        # materials screening: triclinic cells of 8-40 A at 0.1-0.2 A, the plan replayed
        dict(name="batch_screen", kind="batch", frameworks=8, cells=1000, lo=8.0, hi=40.0),
        # screening with coarse grids: many jobs that each fill a fraction of the GPU, one call
        dict(name="batch_small", kind="batch_small", frameworks=64, atoms=424, n=32),
        # the first estimate of a Henry coefficient: 64 x 256 x 2 insertions
        dict(CUBIC, name="henry_32k", kind="henry", probe="CH4", n_ins=32768, temperature=298.0, mask=0,
             energies=False),
        # the converged one: 10^7 insertions behind the pocket mask of a 0.2 A grid
        dict(CUBIC, name="henry_10m_mask", kind="henry", probe="Xe", n_ins=10000000, temperature=298.0, mask=129,
             energies=False),
        # Widom screening: per framework a 0.4 A blocking grid, its pocket mask, 10^6 insertions
        dict(name="henry_screen", kind="henry_batch", frameworks=6, atoms=424, probe="Xe", n_ins=1000000,
             temperature=298.0, block=65),
        # pocket blocking of the usual grid
        dict(CUBIC, name="pockets_129", kind="pockets", probe="CH4", n=129, temperature=298.0),
        # guest energies of a GCMC sweep, looked up in the usual grid
        dict(CUBIC, name="interp_1m", kind="interp", probe="CH4", n=129, points=1000000, f64=False),
        # hard-sphere accessibility of the usual cell at 0.4 A
        dict(CUBIC, name="access_65", kind="access", probe="CH4", nx=65, ny=63, nz=64),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _cell(rng, lo=8.0, hi=40.0):
    """A cell of the screening range that is neither flat nor degenerate."""
    while True:
        abc = [rng.uniform(lo, hi) for _ in range(3)]
        ang = [rng.uniform(60.0, 120.0) for _ in range(3)]
        c = [math.cos(math.radians(x)) for x in ang]
        s = 1.0 - sum(x * x for x in c) + 2.0 * c[0] * c[1] * c[2]
        if s > 0.1:
            return dict(zip(("a", "b", "c", "alpha", "beta", "gamma"), abc + ang))


def draw(rng):
    kind = rng.choice(["grid", "grid", "grid", "henry", "henry", "batch", "batch_small", "henry_batch", "pockets",
                       "interp", "access"])
    probe = rng.choice(sorted(PROBES))
    if kind == "grid":
        case = _cell(rng)
        prec = rng.choice(["near64", "near64", "near64", "comp", "fp32", "fp64"])
        top = 56 if prec == "fp64" else 192
        case.update(atoms=_log(rng, 50, 5000), types=rng.randint(2, 8), probe=probe, prec=prec, nx=_log(rng, 12, top),
                    ny=_log(rng, 12, top), nz=_log(rng, 12, top), host=rng.random() < 0.3)
    elif kind == "batch":
        case = dict(frameworks=rng.randint(2, 6), cells=rng.randint(1, 10**6), lo=8.0, hi=30.0)
    elif kind == "batch_small":
        case = dict(frameworks=rng.randint(5, 64), atoms=_log(rng, 50, 1000), n=rng.randint(16, 36))
    elif kind == "henry":
        case = _cell(rng)
        case.update(atoms=_log(rng, 50, 2000), types=rng.randint(2, 8), probe=probe, n_ins=_log(rng, 10000, 5000000),
                    temperature=rng.uniform(200.0, 500.0), mask=rng.choice([0, rng.randint(20, 130)]))
        # some programs look at the distribution of the insertion energies
        case["energies"] = not case["mask"] and case["n_ins"] < 500000
    elif kind == "henry_batch":
        case = dict(frameworks=rng.randint(2, 6), atoms=_log(rng, 50, 1000), probe=probe,
                    n_ins=_log(rng, 50000, 1000000), temperature=rng.uniform(250.0, 400.0), block=rng.randint(24, 66))
    elif kind == "pockets":
        case = _cell(rng, 15.0, 35.0)
        case.update(atoms=_log(rng, 100, 1000), types=4, probe=probe, n=rng.randint(30, 150),
                    temperature=rng.uniform(200.0, 400.0))
    elif kind == "interp":
        case = _cell(rng, 15.0, 35.0)
        case.update(atoms=_log(rng, 100, 1000), types=4, probe=probe, n=rng.randint(20, 130),
                    points=_log(rng, 1000, 5000000), f64=rng.random() < 0.3)
    else:
        case = _cell(rng, 12.0, 40.0)
        case.update(atoms=_log(rng, 50, 1000), types=4, probe=probe, nx=rng.randint(12, 72), ny=rng.randint(12, 72),
                    nz=rng.randint(12, 72))
    case["kind"] = kind
    if "a" in case:
        case["atoms"] = max(1, min(case["atoms"], int(MAX_DENSITY * _volume(case))))
    return case


# ------------------------------------------------------------------ frameworks
def _matrix(c):
    """Cell matrix (fractional to Cartesian), the first axis along x and the second in the xy plane."""
    ca, cb, cg = (math.cos(math.radians(c[k])) for k in ("alpha", "beta", "gamma"))
    sg = math.sin(math.radians(c["gamma"]))
    unit = math.sqrt(1.0 - ca * ca - cb * cb - cg * cg + 2.0 * ca * cb * cg)
    if c["alpha"] == c["beta"] == c["gamma"] == 90.0:
        return np.diag([c["a"], c["b"], c["c"]]).astype(np.float64)
    return np.array([[c["a"], c["b"] * cg, c["c"] * cb],
                     [0.0, c["b"] * sg, c["c"] * (ca - cb * cg) / sg],
                     [0.0, 0.0, c["c"] * unit / sg]])


def _volume(c):
    return float(abs(np.linalg.det(_matrix(c))))


class _Framework:
    """Atoms of one framework mixed with its probe: what a program has read from its files."""

    def __init__(self, cell, atoms, types, probe, seed):
        rng = np.random.default_rng([seed, 17])
        self.t = _matrix(cell)
        volume = float(abs(np.linalg.det(self.t)))
        lengths = np.linalg.norm(self.t, axis=0)
        edge = min(1.7, (volume / atoms / 1.6) ** (1.0 / 3.0))
        n = np.maximum(1, np.ceil(lengths / edge)).astype(int)
        while n.prod() < atoms:
            n += 1
        site = rng.choice(int(n.prod()), size=atoms, replace=False)
        ijk = np.stack(np.unravel_index(site, tuple(n)), axis=1)
        room = np.maximum(0.05, 1.0 - 1.2 * n / lengths)  # of a site's width, so that atoms stay about 1.2 A apart
        self.frac = ((ijk + 0.5 + (rng.random((atoms, 3)) - 0.5) * room) / n) % 1.0
        kind = rng.integers(0, types, size=atoms)
        eps_g, sig_g = PROBES[probe]
        self.eps = np.sqrt(eps_g * rng.uniform(20.0, 100.0, size=types)[kind])
        self.sig2 = ((sig_g + rng.uniform(2.5, 3.8, size=types)[kind]) / 2.0) ** 2

    def upload_args(self):
        return (er.particles(self.frac, self.eps, self.sig2), self.t, er.replication_factors(self.t, RC), RC * RC)


def _one(case, seed):
    return _Framework(case, case["atoms"], case["types"], case["probe"], seed)


def _screen_cells(case):
    """Cells, atom counts, probes and grid sizes of a screening batch."""
    rng = random.Random(case["cells"])
    jobs = []
    for _ in range(case["frameworks"]):
        c = _cell(rng, case["lo"], case["hi"])
        atoms = max(1, min(_log(rng, 100, 5000), int(MAX_DENSITY * _volume(c))))
        spacing = rng.uniform(0.1, 0.2)
        jobs.append((c, atoms, rng.choice(sorted(PROBES)), tuple(math.ceil(c[k] / spacing) for k in "abc")))
    return jobs


def _frameworks(case, seed):
    """The frameworks of a batch case and their grid sizes."""
    if case["kind"] == "batch":
        return [(_Framework(c, n, 8, probe, seed * 1000 + k), dims)
                for k, (c, n, probe, dims) in enumerate(_screen_cells(case))]
    if case["kind"] == "batch_small":
        probes = sorted(PROBES)
        return [(_Framework(CUBIC, case["atoms"], 4, probes[k % 3], seed * 1000 + k), (case["n"],) * 3)
                for k in range(case["frameworks"])]
    return [(_Framework(CUBIC, case["atoms"], 4, case["probe"], seed * 1000 + k), (case["block"],) * 3)
            for k in range(case["frameworks"])]


def _pocket_mask(case, seed):
    """A mask of blocked spheres, as pocket blocking leaves it on a case["mask"]^3 grid."""
    n = case["mask"]
    rng = np.random.default_rng([seed, 23])
    axis = np.arange(n) / (n - 1)
    mask = np.zeros((n, n, n), dtype=np.uint8)
    lengths = np.linalg.norm(_matrix(case), axis=0)
    for _ in range(8):
        centre, radius = rng.random(3), rng.uniform(1.0, 2.5)
        d2 = sum((((axis - centre[k] + 0.5) % 1.0 - 0.5).reshape([-1 if d == k else 1 for d in range(3)]) * lengths[k])
                 ** 2 for k in range(3))
        mask |= (d2 < radius * radius).astype(np.uint8)
    return mask


def _guest_points(case, seed):
    """Positions of trial moves: in the cell, or a little outside it."""
    return np.random.default_rng([seed, 29]).uniform(-0.1, 1.1, size=(case["points"], 3))


# ------------------------------------------------------------------ the calls
_context = None


def _ctx():
    """The program's one context."""
    global _context
    if _context is None:
        _context = er.Context(torch.cuda.current_device())
    return _context


class _State:
    """What a program holds between calls; frameworks and plans are given back with it."""

    def __init__(self, case):
        self.case, self.fws, self.plan, self.call = case, [], None, None

    def __del__(self):
        if self.plan is not None:
            self.plan.close()
        for f in self.fws:
            f.release()


PREC = {"near64": er.ER_PREC_NEAR64, "comp": er.ER_PREC_COMP, "fp32": er.ER_PREC_FP32, "fp64": er.ER_PREC_FP64}


def prepare(case, seed):
    ctx, st, kind = _ctx(), _State(case), case["kind"]
    if kind in ("batch", "batch_small", "henry_batch"):
        items = _frameworks(case, seed)
        st.fws = ctx.upload_many([f.upload_args() for f, _ in items])
    elif kind not in ("pockets", "interp"):
        st.fws = [ctx.upload(*_one(case, seed).upload_args())]
    if kind == "grid":
        dims, f64 = (case["nx"], case["ny"], case["nz"]), case["prec"] == "fp64"
        if case["host"]:
            st.call = lambda: ctx.grid(st.fws[0], dims, precision=PREC[case["prec"]], f64=f64)
        else:
            out = torch.empty(dims, dtype=torch.float64 if f64 else torch.float32, device="cuda")

            def grid():
                ctx.grid_device(st.fws[0], dims, out.data_ptr(), precision=PREC[case["prec"]], f64=f64)
                return out
            st.call = grid
    elif kind in ("batch", "batch_small"):
        outs = [torch.empty(dims, dtype=torch.float32, device="cuda") for _, dims in items]
        jobs = [(fw, dims, o.data_ptr()) for fw, (_, dims), o in zip(st.fws, items, outs)]
        if kind == "batch":
            st.plan = ctx.batch_plan(jobs, er.ER_BATCH_PERSISTENT | er.ER_BATCH_AUTOTUNE)

            def replay():
                st.plan.run()
                return outs
            st.call = replay
        else:
            def batch():
                ctx.grid_batch(jobs)
                return outs
            st.call = batch
    elif kind == "henry":
        args = (st.fws[0], case["temperature"], case["n_ins"], seed)
        if case["mask"]:
            mask = torch.from_numpy(_pocket_mask(case, seed)).cuda()
            st.call = lambda: ctx.henry_device_mask(*args, mask.data_ptr(), mask.shape)
        else:
            st.call = lambda: ctx.henry(*args, want_energies=case["energies"])
    elif kind == "henry_batch":
        seeds = [seed * 1000 + k for k in range(len(st.fws))]
        st.call = lambda: ctx.henry_batch(st.fws, case["temperature"], case["n_ins"], seeds, items[0][1])
    elif kind == "pockets":
        dims = (case["n"],) * 3
        grid = _energies(_one(case, seed), _axes(dims)).float().cuda()
        mask = torch.empty(dims, dtype=torch.uint8, device="cuda")
        st.call = lambda: (ctx.block_pockets_device(grid.data_ptr(), dims, case["temperature"], mask.data_ptr()), mask)
    elif kind == "interp":
        dims = (case["n"],) * 3
        grid = _interp_grid(case, seed).cuda()
        pts = torch.from_numpy(_guest_points(case, seed)).cuda()
        out = torch.empty(len(pts), dtype=torch.float64, device="cuda")

        def interp():
            ctx.grid_interp_device(grid.data_ptr(), dims, pts.data_ptr(), len(pts), out.data_ptr(), f64=case["f64"])
            return out
        st.call = interp
    else:
        st.call = lambda: ctx.accessibility(st.fws[0], (case["nx"], case["ny"], case["nz"]))
    torch.cuda.synchronize()  # the library works on a stream of its own
    return st


def run(state):
    return state.call()


# ------------------------------------------------------------------ the same in FP64
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


class _Images:
    """Every atom image within the cutoff of the cell, in Cartesian coordinates."""

    def __init__(self, f):
        dev = _device()
        self.t = torch.tensor(f.t, dtype=torch.float64, device=dev)
        width = 1.0 / np.linalg.norm(np.linalg.inv(f.t), axis=1)  # between opposite faces
        reach = np.floor(RC / width).astype(int) + 1
        shift = torch.cartesian_prod(*[torch.arange(-int(r), int(r) + 1, dtype=torch.float64, device=dev)
                                       for r in reach])
        frac = torch.tensor(f.frac, device=dev)
        q = (shift[:, None, :] + frac[None, :, :]).reshape(-1, 3)
        over = torch.clamp(torch.maximum(-q, q - 1.0), min=0.0) * torch.tensor(width, device=dev)
        keep = (over < RC + 1e-6).all(dim=1)
        atom = torch.arange(len(frac), device=dev).repeat(len(shift))[keep]
        self.xyz = q[keep] @ self.t.T
        self.eps4 = 4.0 * torch.tensor(f.eps, device=dev)[atom]
        self.sig2 = torch.tensor(f.sig2, device=dev)[atom]

    def energy(self, p):
        """Energies at fractional points p (m, 3) that lie close together."""
        x = p @ self.t.T
        lo, hi = x.min(dim=0).values - RC - 1e-6, x.max(dim=0).values + RC + 1e-6
        near = torch.clamp(torch.maximum(lo + RC - self.xyz, self.xyz - hi + RC), min=0.0).square().sum(1) < RC * RC
        a, eps4, sig2 = self.xyz[near], self.eps4[near], self.sig2[near]
        out = torch.empty(len(x), dtype=torch.float64, device=x.device)
        rows = max(1, 8000000 // max(1, len(a)))
        for i in range(0, len(x), rows):
            y = x[i:i + rows]
            d = y[:, 0, None] - a[None, :, 0]
            r2 = d * d
            for k in (1, 2):
                d = y[:, k, None] - a[None, :, k]
                r2.addcmul_(d, d)
            s6 = (sig2 / r2).pow_(3)
            e = (s6 * s6).sub_(s6).mul_(eps4)
            out[i:i + rows] = torch.where(r2 < RC * RC, e, 0.0).sum(dim=1)
        return torch.clamp(out, max=CAP)


def _axes(dims):
    return [torch.arange(n, dtype=torch.float64, device=_device()) / (n - 1) for n in dims]


def _energies(f, axes):
    """Energies on the lattice of three axes of fractional coordinates."""
    images = _Images(f)
    length = np.linalg.norm(f.t, axis=0)
    out = torch.empty([len(a) for a in axes], dtype=torch.float64, device=_device())
    step = [max(1, int(round(2.0 / L * (len(a) - 1)))) for a, L in zip(axes, length)]  # blocks of about 2 A
    for i in range(0, len(axes[0]), step[0]):
        for j in range(0, len(axes[1]), step[1]):
            for k in range(0, len(axes[2]), step[2]):
                cut = [a[s:s + n] for a, s, n in zip(axes, (i, j, k), step)]
                p = torch.cartesian_prod(*cut).reshape(-1, 3)
                out[i:i + step[0], j:j + step[1], k:k + step[2]] = images.energy(p).reshape([len(c) for c in cut])
    return out


def _interp_grid(case, seed):
    g = _energies(_one(case, seed), _axes((case["n"],) * 3))
    return g if case["f64"] else g.float()


def _philox(c, key):
    """Philox4x32-10 (Salmon et al., SC'11) of counter words c (a list of four int64 tensors)."""
    low = 0xFFFFFFFF
    k0, k1 = key
    for _ in range(10):
        p, q = c[0] * 0xD2511F53, c[2] * 0xCD9E8D57  # modulo 2^64
        c = [((q >> 32) & low) ^ c[1] ^ k0, q & low, ((p >> 32) & low) ^ c[3] ^ k1, p & low]
        k0, k1 = (k0 + 0x9E3779B9) & low, (k1 + 0xBB67AE85) & low
    return c


def _insertions(seed, n):
    """The n insertion points of a stream: 53-bit uniforms of counters (i, 0, 0, 0) and (i, 0, 1, 0)."""
    i = torch.arange(n, dtype=torch.int64, device=_device())
    zero = torch.zeros_like(i)
    key = (seed & 0xFFFFFFFF, seed >> 32)
    r, s = _philox([i, zero, zero, zero], key), _philox([i, zero, zero + 1, zero], key)
    u = [((a >> 5).double() * 67108864.0 + (b >> 6).double()) / 9007199254740992.0
         for a, b in ((r[0], r[1]), (r[2], r[3]), (s[0], s[1]))]
    return torch.stack(u, dim=1)


def _henry(case, seed):
    f, n, t = _one(case, seed), case["n_ins"], case["temperature"]
    p = _insertions(seed, n)
    if case["mask"]:
        m = case["mask"]
        mask = torch.from_numpy(_pocket_mask(case, seed)).to(p.device).bool()
        c = torch.clamp(torch.floor(p / (1.0 / (m - 1))).long(), max=m - 2)
        blocked = torch.zeros(n, dtype=torch.bool, device=p.device)
        for d in range(8):
            blocked |= mask[c[:, 0] + (d >> 2), c[:, 1] + ((d >> 1) & 1), c[:, 2] + (d & 1)]
        p = p[~blocked]
    images = _Images(f)
    bins = torch.tensor(np.maximum(1, np.round(np.linalg.norm(f.t, axis=0) / 2.0)), device=p.device)
    b = (p * bins).long()
    key = (b[:, 0] * int(bins[1]) + b[:, 1]) * int(bins[2]) + b[:, 2]
    key, order = torch.sort(key)
    p = p[order]
    ends = torch.cumsum(torch.bincount(key), 0).tolist()
    e = torch.cat([images.energy(p[i:j]) for i, j in zip([0] + ends[:-1], ends) if j > i])
    x = -e / t
    top = float(x.max())
    w = torch.exp(x - top)
    s, se = float(w.sum()), float((w * e).sum())
    out = {"sum_w": s * math.exp(top), "sum_ew": se * math.exp(top), "log_scale": top, "sum_w_scaled": s,
           "sum_ew_scaled": se, "n_insertions": float(n), "n_blocked": float(n - len(p)), "mean_energy": se / s,
           "kh_mol_m3_pa": s * math.exp(top) / n / t / 8.314}
    if case["energies"]:
        out["energies"] = torch.empty_like(e)
        out["energies"][order] = e
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "grid":
        return _energies(_one(case, seed), _axes((case["nx"], case["ny"], case["nz"])))
    if kind in ("batch", "batch_small"):
        return [_energies(f, _axes(dims)) for f, dims in _frameworks(case, seed)]
    if kind == "henry":
        return _henry(case, seed)
    if kind == "interp":
        n = case["n"]
        g = _interp_grid(case, seed).double()
        p = torch.from_numpy(_guest_points(case, seed)).to(g.device)
        p = p - torch.floor(p)
        c = torch.clamp(torch.floor(p / (1.0 / (n - 1))).long(), max=n - 2)
        d = (p - c * (1.0 / (n - 1))) / (1.0 / (n - 1))
        out = torch.zeros(len(p), dtype=torch.float64, device=g.device)
        for i in (0, 1):
            for j in (0, 1):
                for k in (0, 1):
                    w = [d[:, q] if on else 1.0 - d[:, q] for q, on in enumerate((i, j, k))]
                    out += w[0] * w[1] * w[2] * g[c[:, 0] + i, c[:, 1] + j, c[:, 2] + k]
        return out
    return None  # masks and counts are whole numbers; a Widom batch follows its pocket masks


# ------------------------------------------------------------------ what a pass cannot do without
def work(case):
    kind = case["kind"]
    sphere = 4.0 / 3.0 * math.pi * RC ** 3

    def pairs(points, atoms, volume):  # in-cutoff pair terms, on average
        return points * atoms * sphere / volume

    if kind == "grid":
        n = case["nx"] * case["ny"] * case["nz"]
        return {"bytes": n * (8 if case["prec"] == "fp64" else 4) + 40 * case["atoms"],
                "flops": PAIR_FLOPS * pairs(n, case["atoms"], _volume(case))}
    if kind == "batch":
        total = {"bytes": 0, "flops": 0}
        for c, atoms, _, dims in _screen_cells(case):
            n = math.prod(dims)
            total["bytes"] += 4 * n + 40 * atoms
            total["flops"] += PAIR_FLOPS * pairs(n, atoms, _volume(c))
        return total
    if kind == "batch_small":
        n = case["frameworks"] * case["n"] ** 3
        return {"bytes": 4 * n + 40 * case["frameworks"] * case["atoms"],
                "flops": PAIR_FLOPS * pairs(n, case["atoms"], _volume(CUBIC))}
    if kind == "henry":
        return {"bytes": 40 * case["atoms"] + case["mask"] ** 3,
                "flops": PAIR_FLOPS * pairs(case["n_ins"], case["atoms"], _volume(case))}
    if kind == "henry_batch":
        n = case["frameworks"] * (case["n_ins"] + case["block"] ** 3)
        return {"bytes": 40 * case["frameworks"] * case["atoms"],
                "flops": PAIR_FLOPS * pairs(n, case["atoms"], _volume(CUBIC))}
    if kind == "pockets":
        return {"bytes": 5 * case["n"] ** 3, "flops": 0}
    if kind == "interp":
        size = 8 if case["f64"] else 4
        return {"bytes": 32 * case["points"] + size * min(case["n"] ** 3, 8 * case["points"]),
                "flops": 30 * case["points"]}
    n = case["nx"] * case["ny"] * case["nz"]
    # the images that can overlap a point lie within the largest mixed sigma, about 4 A
    return {"bytes": n + 40 * case["atoms"], "flops": 9 * n * case["atoms"] * 4.0 / 3.0 * math.pi * 64 / _volume(case)}
