"""Performance cases of the FLIP-on-MSBG framework: the calls a user's program makes, through the
public Python binding, over the sizes the framework is used at.

A case is a dict of plain values.  `kind` says which call is measured:

  particles  the drop-in particle calls in the reference's order: aw_p2g, aw_backup_grid_velocity,
             gravity and walls, aw_g2p, aw_advect on the caller's arrays.  The step's start positions
             are copied in first (the caller keeps them), so that every pass moves the same particles.
  project    aw_project of a free-surface velocity field: divergence, multigrid solve, gradient.
  vcycle     one aw_vcycle_run (the reference's VCycleSolver::runCycle) from a zero guess.
  poisson    aw_solve on a closed box with a 32-sphere level map, from a zero pressure.
  flip       aw_flip_step on library-owned particles; `frame`: the particles are read back every step,
             as a program that writes frames does; `two_phase`: the sphere is a second liquid.
  rollout    forward and gradient of the differentiable rollout.

Liquid scenes are a column in the box's low corner plus (`sphere`) a falling sphere, 8 jittered
particles per finest cell, as in the framework's own scenes.  Grids have bx x by x bz blocks of 8^3
finest cells, as in its configurations, and level thresholds of 1, 3 and 7 blocks.  `shuffled` hands
the particles over in random order (an external source); otherwise they come in cell order, as after
an earlier step.
"""
from __future__ import annotations

import numpy as np
import torch

import anitowave_adaptive_b200 as aw
from anitowave_adaptive_b200 import scenes

GRAVITY = -9.81
ALPHA = 0.95
COLUMN = (0.4, 0.6, 1.0)                 # the dam, as a fraction of the domain
SPHERE = ((0.7, 0.8, 0.5), 0.12, -1.0)   # centre and radius (fractions of the x extent), velocity
PRECISION = {"fp32": aw.PRECISION_FP32, "mixed": aw.PRECISION_MIXED, "fp32_pcg": aw.PRECISION_FP32_PCG}


def _cube(N, base_res=8):
    return {"bx": N // base_res, "by": N // base_res, "bz": N // base_res, "base_res": base_res}


def listed():
    return [
        # a toy scene: a first try or a unit test of a user's program; launches and latency are all of it
        dict(name="particles_16", kind="particles", **_cube(16), levels=2, sphere=False, shuffled=False),
        # the 2-level dam break (64^3, 0.5M particles) fed by an external source in random order
        dict(name="particles_64_shuffled", kind="particles", **_cube(64), levels=2, sphere=False, shuffled=True),
        # a long tank: odd block counts on every axis, off-origin domain, 3 levels
        dict(name="particles_ragged", kind="particles", bx=19, by=9, bz=7, base_res=8, levels=3, sphere=True,
             shuffled=False),
        # the benchmark's transfers (128^3 effective, 3 levels, 4.1M particles)
        dict(name="particles_128", kind="particles", **_cube(128), levels=3, sphere=True, shuffled=False),
        # one projection of a program with its own particle code, plain FP32 V-cycle iteration (its FP32
        # residual stalls near 1e-5 here)
        dict(name="project_96_fp32", kind="project", **_cube(96), levels=2, sphere=True, precision="fp32",
             tolerance=3e-4),
        # the multigrid cycle as a building block (a user's own Krylov loop calls it)
        dict(name="vcycle_64", kind="vcycle", **_cube(64), levels=3, precision="fp32"),
        # the Poisson benchmark: 256^3 effective, 4 levels, 4.7M cells, mixed precision to 1e-6
        dict(name="poisson_256", kind="poisson", **_cube(256), levels=4, precision="mixed", tolerance=1e-6),
        # an interactive toy simulation whose particles are shown every step
        dict(name="flip_16_frame", kind="flip", **_cube(16), levels=2, sphere=False, two_phase=False, frame=True),
        # two liquids of density 1 and 3 on the 2-level 64^3 layout
        dict(name="flip_64_two_phase", kind="flip", **_cube(64), levels=2, sphere=True, two_phase=True, frame=False),
        # the benchmark's FLIP step
        dict(name="flip_128", kind="flip", **_cube(128), levels=3, sphere=True, two_phase=False, frame=False),
        # production size: 256^3 effective, 4 levels, 33M particles
        dict(name="flip_256", kind="flip", **_cube(256), levels=4, sphere=True, two_phase=False, frame=False),
        # gradient of an inverse problem: 4 steps, checkpoints every 2, forward and backward
        dict(name="rollout_32", kind="rollout", **_cube(32), levels=2, sphere=False, steps=4),
    ]


def draw(rng):
    kind = rng.choice(["particles", "particles", "project", "vcycle", "poisson", "flip", "flip", "rollout"])
    base = 8
    if kind in ("particles", "flip"):
        # domains of 16^3 to 192^3 finest cells, each axis its own odd or even block count
        n = 2 ** rng.uniform(4.0, 7.4)
        dims = [max(2, round(n * rng.uniform(0.7, 1.3) / base)) for _ in range(3)]
    elif kind == "rollout":
        n = 2 ** rng.uniform(4.0, 6.0)
        dims = [max(2, round(n / base))] * 3
    else:
        # the multigrid hierarchy ends in uniform levels when every block count is even
        n = 2 ** rng.uniform(4.5, 7.6)
        dims = [2 * max(1, round(n * rng.uniform(0.7, 1.3) / (2 * base))) for _ in range(3)]
    c = dict(kind=kind, bx=dims[0], by=dims[1], bz=dims[2], base_res=base, levels=rng.choice([2, 3]))
    if kind == "particles":
        c.update(sphere=rng.random() < 0.7, shuffled=rng.random() < 0.3)
    elif kind == "project":
        prec = rng.choice(["fp32", "mixed", "fp32_pcg"])
        c.update(sphere=rng.random() < 0.7, precision=prec, tolerance=1e-6 if prec == "mixed" else 3e-4)
    elif kind == "vcycle":
        c.update(precision=rng.choice(["fp32", "mixed"]))
    elif kind == "poisson":
        c.update(precision="mixed", tolerance=rng.choice([1e-5, 1e-6]))
    elif kind == "flip":
        c.update(sphere=True, two_phase=rng.random() < 0.3, frame=False)
    else:
        c.update(sphere=False, steps=rng.choice([2, 3, 4]))
    return c


# ------------------------------------------------------------------------------------------------
# scenes
# ------------------------------------------------------------------------------------------------
def _blocks(case):
    return case["bx"], case["by"], case["bz"]


def _cells(case):
    return tuple(b * case["base_res"] for b in _blocks(case))


def _spacing(case):
    """Finest cell size: the x extent of the domain is 1."""
    return 1.0 / _cells(case)[0]


def _domain_min(case):
    return (-0.25, 0.5, 0.125) if len(set(_blocks(case))) > 1 else (0.0, 0.0, 0.0)


def _thresholds(case):
    return [case["base_res"] * k for k in (1, 3, 7)[:case["levels"] - 1]]


def _time_step(case):
    n = max(_cells(case))
    return 1.0 / 960 if n <= 64 else (1.0 / 1920 if n <= 128 else 1.0 / 3840)


def _inside(case):
    """(liquid, sphere) masks over the finest cells, [z, y, x]."""
    nx, ny, nz = _cells(case)
    ax = [(torch.arange(n, device="cuda", dtype=torch.float64) + 0.5) / n for n in (nx, ny, nz)]
    x, y, z = ax[0][None, None, :], ax[1][None, :, None], ax[2][:, None, None]
    liquid = (x < COLUMN[0]) & (y < COLUMN[1]) & (z < COLUMN[2])
    if not case["sphere"]:
        return liquid, torch.zeros_like(liquid)
    (cx, cy, cz), r, _ = SPHERE
    ball = ((x - cx) ** 2 + ((y - cy) * ny / nx) ** 2 + ((z - cz) * nz / nx) ** 2) < r * r
    return liquid | ball, ball & ~liquid


def _particles(case, seed):
    """Float32 positions and velocities (n, 3) and the sphere label of every particle."""
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    mask, ball = _inside(case)
    cell = mask.nonzero()  # (z, y, x), x fastest: cell order
    n = cell.shape[0]
    sub = torch.arange(8, device="cuda")
    h = _spacing(case)
    pos = torch.empty((n, 8, 3), dtype=torch.float32, device="cuda")
    for a in range(3):
        jitter = torch.rand((n, 8), generator=gen, device="cuda", dtype=torch.float32)
        corner = ((sub >> a) & 1).float()[None, :]
        pos[:, :, a] = (cell[:, 2 - a].float()[:, None] + (corner + jitter) * 0.5) * h + _domain_min(case)[a]
    pos = pos.reshape(-1, 3)
    label = ball[cell[:, 0], cell[:, 1], cell[:, 2]].repeat_interleave(8)
    # a gentle swirl of a random phase and a little noise; the sphere falls
    phase = 6.2831853 * torch.rand(3, generator=gen, device="cuda")
    vel = 0.05 * torch.sin(6.0 * pos[:, [1, 2, 0]] + phase)
    vel += 0.01 * torch.randn(vel.shape, generator=gen, device="cuda")
    vel[:, 1] += label.float() * SPHERE[2]
    if case.get("shuffled"):
        p = torch.randperm(pos.shape[0], generator=gen, device="cuda")
        pos, vel, label = pos[p], vel[p], label[p]
    return pos.contiguous(), vel.contiguous(), label


def _grid(case, points):
    g = aw.MSBG(_blocks(case), _spacing(case) * case["base_res"], _domain_min(case), case["base_res"], case["levels"])
    g.levels_from_particles(points, _thresholds(case))
    g.enforce_grading()
    g.allocate()
    return g


def _held(view, owner):
    """A view of library memory that keeps the handle owning that memory alive."""
    view.owner = owner
    return view


def _channel(g, channel):
    return _held(g.channel(channel), g)


def _triplet(g, channel):
    return [_channel(g, channel + a) for a in range(3)]


def _waves(X, gen, terms=8):
    """A smooth random scalar field at the points X (n, 3) float32, in 64 bits."""
    k = 2.0 + 10.0 * torch.rand((terms, 3), generator=gen, device="cuda", dtype=torch.float64)
    ph = 6.2831853 * torch.rand(terms, generator=gen, device="cuda", dtype=torch.float64)
    out = torch.zeros(X.shape[0], dtype=torch.float64, device="cuda")
    Xd = X.double()
    for t in range(terms):
        out += torch.sin(Xd @ k[t] + ph[t])
    return out / terms


# ------------------------------------------------------------------------------------------------
# prepare / run
# ------------------------------------------------------------------------------------------------
def _closed_box(case, seed):
    """Grid refined around 32 fixed spheres and a smooth zero-mean right-hand side."""
    nx, ny, nz = _cells(case)
    c, r = scenes.poisson_spheres()
    dmin, h = _domain_min(case), _spacing(case)
    ax = [(torch.arange(n, device="cuda", dtype=torch.float64) + 0.5) / n for n in (nx, ny, nz)]
    mask = torch.zeros((nz, ny, nx), dtype=torch.bool, device="cuda")
    for s in range(c.shape[0]):
        mask |= ((ax[0][None, None, :] - c[s, 0]) ** 2 + (ax[1][None, :, None] - c[s, 1]) ** 2
                 + (ax[2][:, None, None] - c[s, 2]) ** 2) < r[s] ** 2
    cell = mask.nonzero()
    pts = torch.stack([(cell[:, 2 - a].double() + 0.5) * h + dmin[a] for a in range(3)], -1).float().contiguous()
    g = _grid(case, pts)
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    lv = torch.as_tensor(g.refinement_map().astype(np.int64), device="cuda")
    res = case["base_res"] >> lv
    H = (h * case["base_res"] / res.double()).repeat_interleave(res ** 3)
    f = _waves(g.face_positions(3), gen)
    f -= (f * H ** 3).sum() / (H ** 3).sum()
    return g, (f * H ** 3).float().contiguous()


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("vcycle", "poisson"):
        g, b = _closed_box(case, seed)
        sv = aw.Solver(g, precision=PRECISION[case["precision"]], tolerance=case.get("tolerance", 1e-6), max_cycles=100)
        sv.setup(None)
        s = dict(case=case, grid=g, solver=sv, b=b)
        if kind == "vcycle":
            sv.level_array(0, 1).copy_(b)
            s["x"] = _held(sv.level_array(0, 0), sv)
        else:
            s["p"] = torch.zeros(b.numel(), dtype=torch.float64 if case["precision"] == "mixed" else torch.float32,
                                 device="cuda")
        return s
    pos, vel, label = _particles(case, seed)
    g = _grid(case, pos)
    dt = _time_step(case)
    s = dict(case=case, grid=g, dt=dt)
    if kind == "particles":
        s.update(pos0=pos, pos=pos.clone(), vel=vel, u=_triplet(g, aw.VELOCITY_X), uo=_triplet(g, aw.VELOCITY_OLD_X),
                 m=_triplet(g, aw.MASS_DENSITY_X), count=_channel(g, aw.CELL_TYPE))
    elif kind == "project":
        gen = torch.Generator(device="cuda").manual_seed(int(seed) + 1)
        g.p2g(pos, vel)
        s["fluid"] = (g.channel(aw.CELL_TYPE) > 0).to(torch.uint8)
        s["u"] = _triplet(g, aw.VELOCITY_X)
        s["u0"] = [(0.2 * _waves(g.face_positions(a), gen)).float() for a in range(3)]
        s["u0"][1] += dt * GRAVITY
        s["solver"] = aw.Solver(g, precision=PRECISION[case["precision"]], tolerance=case["tolerance"], max_cycles=100)
    elif kind == "flip":
        F = aw.Flip(g, pos.cpu().numpy(), vel.cpu().numpy(), dt, ALPHA, (0, GRAVITY, 0), precision=aw.PRECISION_MIXED,
                    tolerance=1e-6, max_cycles=100)
        if case["two_phase"]:
            F.set_phase(label.float().cpu().numpy(), 1.0, 3.0)
        s.update(flip=F, u=_triplet(g, aw.VELOCITY_X), pressure=_channel(g, aw.PRESSURE),
                 count=_channel(g, aw.CELL_TYPE))
    else:
        gen = torch.Generator(device="cuda").manual_seed(int(seed) + 1)
        s["rollout"] = aw.Rollout(g, pos.cpu().numpy(), case["steps"], dt, ALPHA, (0, GRAVITY, 0),
                                  precision=aw.PRECISION_MIXED, tolerance=1e-8, checkpoint_every=2)
        s["u0"] = torch.cat([(0.2 * _waves(g.face_positions(a), gen)).float() for a in range(3)])
        s["target"] = pos + 0.02 * torch.randn(pos.shape, generator=gen, device="cuda")
    return s


def run(s):
    case, g = s["case"], s["grid"]
    kind = case["kind"]
    if kind == "particles":
        s["pos"].copy_(s["pos0"])
        g.p2g(s["pos"], s["vel"])
        g.backup_grid_velocity()
        g.add_gravity((0.0, GRAVITY, 0.0), s["dt"])
        g.wall_bc(aw.VELOCITY_X)
        g.g2p(s["vel"], s["pos"], ALPHA)
        g.advect(s["pos"], s["dt"])
        return {"pos": s["pos"], "vel": s["vel"], "u": s["u"], "u_old": s["uo"], "m": s["m"], "count": s["count"]}
    if kind == "project":
        for a in range(3):
            s["u"][a].copy_(s["u0"][a])
        g.project(s["solver"], s["fluid"], s["dt"])
        return {"u": s["u"]}
    if kind == "vcycle":
        s["x"].zero_()
        s["solver"].vcycle()
        return {"x": s["x"]}
    if kind == "poisson":
        s["p"].zero_()
        s["solver"].solve(s["b"], s["p"])
        return {"p": s["p"]}
    if kind == "flip":
        s["flip"].step()
        out = {"u": s["u"], "pressure": s["pressure"], "count": s["count"]}
        if case["frame"]:
            out["pos"], out["vel"] = s["flip"].particles()
        return out
    s["rollout"].forward(s["u0"], s["target"])
    pos = s["rollout"].final_positions()
    return {"pos": pos, "grad": s["rollout"].vjp()}


# ------------------------------------------------------------------------------------------------
# plain 64-bit layout, P2G, G2P and RK3
# ------------------------------------------------------------------------------------------------
def _levels(case):
    """Level of every block [z, y, x]: distance to the free surface in blocks, then 2:1 grading."""
    if case["kind"] in ("vcycle", "poisson"):
        return None
    R = case["base_res"]
    bx, by, bz = _blocks(case)
    occ, _ = _inside(case)
    surf = torch.zeros_like(occ)
    for d in range(3):
        n = occ.shape[d]
        lo, hi = occ.narrow(d, 0, n - 1), occ.narrow(d, 1, n - 1)
        surf.narrow(d, 0, n - 1).logical_or_(lo & ~hi)
        surf.narrow(d, 1, n - 1).logical_or_(hi & ~lo)
    bs = surf.view(bz, R, by, R, bx, R).any(5).any(3).any(1).float()[None, None]
    lv = torch.full((bz, by, bx), case["levels"] - 1, dtype=torch.int64, device="cuda")
    for k in range(case["levels"] - 2, -1, -1):
        K = _thresholds(case)[k] // R
        near = torch.nn.functional.max_pool3d(bs, 2 * K + 1, 1, K)[0, 0] > 0
        lv[near] = k
    while True:
        low = -torch.nn.functional.max_pool3d(-lv[None, None].float(), 3, 1, 1)[0, 0]
        new = torch.minimum(lv, low.long() + 1)
        if torch.equal(new, lv):
            return lv
        lv = new


class _Plain:
    """The block grid in plain torch: offsets, face lattices and MAC samples in 64 bits."""

    def __init__(self, case):
        self.case = case
        self.lv = _levels(case).reshape(-1)
        self.D = _blocks(case)
        self.res = case["base_res"] >> self.lv
        # single-precision geometry, as the grid stores it
        f = np.float32
        self.bs = float(f(_spacing(case) * case["base_res"]))
        self.dmin = [float(f(v)) for v in _domain_min(case)]
        r = self.res
        nf = (r + 1) * r * r
        self.foff = torch.cumsum(nf, 0) - nf
        self.coff = torch.cumsum(r ** 3, 0) - r ** 3
        self.nfaces, self.ncells = int(nf.sum()), int((r ** 3).sum())

    def coords(self, b):
        return [b % self.D[0], (b // self.D[0]) % self.D[1], b // (self.D[0] * self.D[1])]

    @staticmethod
    def face(a, f, r):
        return (f[0] + (r + 1) * (f[1] + r * f[2]) if a == 0 else
                f[0] + r * (f[1] + (r + 1) * f[2]) if a == 1 else f[0] + r * (f[1] + r * f[2]))

    def block_of(self, X):
        c = [((X[:, k] - self.dmin[k]) / self.bs).floor().long().clamp(0, self.D[k] - 1) for k in range(3)]
        return c, c[0] + self.D[0] * (c[1] + self.D[1] * c[2])

    def gather_faces(self, a, lattices):
        """Block-ordered face array from one dense lattice per level."""
        out = torch.zeros(self.nfaces, dtype=torch.float64, device="cuda")
        for l, lat in lattices.items():
            r = self.case["base_res"] >> l
            b = (self.lv == l).nonzero()[:, 0]
            n = [r + (k == a) for k in range(3)]
            i = torch.arange(n[0] * n[1] * n[2], device="cuda")
            f = [i % n[0], (i // n[0]) % n[1], i // (n[0] * n[1])]
            c = self.coords(b)
            g = [c[k][:, None] * r + f[k][None, :] for k in range(3)]
            out[self.foff[b][:, None] + i[None, :]] = lat[g[2], g[1], g[0]]
        return out

    def p2g(self, X, V):
        """(u, m) per axis: every face sums (1 - d^2/h^2)^3 over the particles within its cell size."""
        u, m = [], []
        for a in range(3):
            mass, mom = {}, {}
            for l in range(self.case["levels"]):
                if not bool((self.lv == l).any()):
                    continue
                r = self.case["base_res"] >> l
                n = [self.D[k] * r + (k == a) for k in range(3)]
                q = [(X[:, k] - self.dmin[k]) * (r / self.bs) - (0.0 if k == a else 0.5) for k in range(3)]
                i0 = [v.floor().long() for v in q]
                M = torch.zeros(n[0] * n[1] * n[2], dtype=torch.float64, device="cuda")
                P = torch.zeros_like(M)
                for e in range(8):
                    i = [i0[k] + ((e >> k) & 1) for k in range(3)]
                    w = (1.0 - sum((q[k] - i[k]) ** 2 for k in range(3))).clamp(min=0.0) ** 3
                    for k in range(3):
                        w = w * ((i[k] >= 0) & (i[k] < n[k]))
                        i[k] = i[k].clamp(0, n[k] - 1)
                    at = i[0] + n[0] * (i[1] + n[1] * i[2])
                    M.index_add_(0, at, w)
                    P.index_add_(0, at, w * V[:, a])
                mass[l], mom[l] = M.view(n[2], n[1], n[0]), P.view(n[2], n[1], n[0])
            m.append(self.gather_faces(a, mass))
            mo = self.gather_faces(a, mom)
            u.append(torch.where(m[a] > 1e-6, mo / m[a], torch.zeros_like(mo)))
        return u, m

    def counts(self, X):
        c, b = self.block_of(X)
        r = self.res[b]
        q = [((X[:, k] - self.dmin[k] - c[k] * self.bs) * r / self.bs).floor().long().clamp(min=0) for k in range(3)]
        q = [torch.minimum(v, r - 1) for v in q]
        at = self.coff[b] + q[0] + r * (q[1] + r * q[2])
        return torch.bincount(at, minlength=self.ncells).double()

    def walls(self, u):
        """Zero the domain's boundary faces."""
        for a in range(3):
            b = torch.arange(self.lv.numel(), device="cuda")
            c = self.coords(b)
            for l in range(self.case["levels"]):
                r = self.case["base_res"] >> l
                i = torch.arange(r * r, device="cuda")
                for side in (0, 1):
                    s = b[(self.lv == l) & (c[a] == (self.D[a] - 1 if side else 0))]
                    f = [None] * 3
                    f[a] = torch.full_like(i, r if side else 0)
                    f[(a + 1) % 3], f[(a + 2) % 3] = i % r, i // r
                    u[a][self.foff[s][:, None] + self.face(a, f, r)[None, :]] = 0.0

    def sample(self, u, a, X):
        """Trilinear MAC sample in the particle's block; ghost rows read the nearest face of the same
        axis in the neighbouring block, clamped back into the block at the domain's sides."""
        c, b = self.block_of(X)
        r = self.res[b]
        i0, fr = [], []
        for k in range(3):
            s = (X[:, k] - self.dmin[k] - c[k] * self.bs) * r / self.bs
            lo = 0
            if k != a:
                s, lo = s - 0.5, -1
            s = torch.minimum(s.clamp(min=float(lo)), r.double())
            i = torch.minimum(s.floor().long().clamp(min=lo), r - 1)
            i0.append(i)
            fr.append(s - i)
        t = [k for k in range(3) if k != a]
        out = torch.zeros(X.shape[0], dtype=torch.float64, device="cuda")
        for e in range(8):
            w = torch.ones_like(out)
            f = []
            for k in range(3):
                d = (e >> k) & 1
                f.append(i0[k] + d)
                w = w * (fr[k] if d else 1.0 - fr[k])
            o = {k: (f[k] >= r).long() - (f[k] < 0).long() for k in t}
            nc = [c[k] + o[k] if k in o else c[k] for k in range(3)]
            ok = torch.ones_like(b, dtype=torch.bool)
            for k in range(3):
                ok &= (nc[k] >= 0) & (nc[k] < self.D[k])
            nb = torch.where(ok, nc[0] + self.D[0] * (nc[1] + self.D[1] * nc[2]), b)
            rn = self.res[nb]
            q = [None] * 3
            q[a] = (2 * f[a] * rn + r) // (2 * r)
            for k in t:
                rel = torch.where(ok, 2 * f[k] + 1 - o[k] * 2 * r, 2 * torch.minimum(f[k].clamp(min=0), r - 1) + 1)
                q[k] = torch.minimum(((rel * rn) // (2 * r)).clamp(min=0), rn - 1)
            out += w * u[a][self.foff[nb] + self.face(a, q, rn)]
        return out

    def advect(self, u, X, dt):
        """Ralston RK3, clamped 0.01 finest cells inside the domain."""
        h0 = self.bs / self.case["base_res"]

        def vel(Y):
            return torch.stack([self.sample(u, a, Y) for a in range(3)], -1)
        k1 = vel(X)
        k2 = vel(X + 0.5 * dt * k1)
        k3 = vel(X + 0.75 * dt * k2)
        Y = X + dt * (2 * k1 + 3 * k2 + 4 * k3) / 9
        for k in range(3):
            Y[:, k] = Y[:, k].clamp(self.dmin[k] + 0.01 * h0, self.dmin[k] + self.D[k] * self.bs - 0.01 * h0)
        return Y


def exact(case, seed):
    """The particle calls have exact values.  A solve ends at the tolerance asked for, and so does every
    whole step, so those have none."""
    if case["kind"] != "particles":
        return None
    pos, vel, _ = _particles(case, seed)
    X, V = pos.double(), vel.double()
    G = _Plain(case)
    dt = float(np.float32(_time_step(case)))
    uo, m = G.p2g(X, V)
    u = [v.clone() for v in uo]
    u[1] += dt * float(np.float32(GRAVITY))
    G.walls(u)
    al = float(np.float32(ALPHA))
    un = torch.stack([G.sample(u, a, X) for a in range(3)], -1)
    old = torch.stack([G.sample(uo, a, X) for a in range(3)], -1)
    return {"pos": G.advect(u, X, dt), "vel": al * (V + un - old) + (1.0 - al) * un, "u": u, "u_old": uo, "m": m,
            "count": G.counts(X)}


# ------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ------------------------------------------------------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind in ("vcycle", "poisson"):
        g, b = _closed_box(case, 0)
        cells = b.numel()
        wide = 8 if case["precision"] == "mixed" else 4
        # right-hand side read, pressure written; one V(2,2)-cycle is about 60 operations per cell, and a
        # solve needs at least one
        return {"bytes": cells * (4 + wide), "flops": cells * 60}
    G = _Plain(case)
    n = 8 * int(_inside(case)[0].sum())
    faces, cells = 3 * G.nfaces, G.ncells
    if kind == "particles":
        # positions and velocities read and written; u, u_old, m and the counts written
        return {"bytes": n * 48 + faces * 12 + cells * 4, "flops": n * 600}
    if kind == "project":
        return {"bytes": faces * 8 + cells, "flops": cells * 80}
    # a step: particle state read and written; velocity, pressure and counts written
    step = {"bytes": n * 48 + faces * 4 + cells * 8, "flops": n * 600 + cells * 80}
    if kind == "flip":
        return step
    # forward, recomputation and adjoint of every step (at least one pass over the state each)
    return {k: 3 * case["steps"] * v for k, v in step.items()}
