"""The register-resident multigrid kernels for blocks with uniform coefficients against the staged
ones (AW_NO_UNIFORM).  The FP32 and FP16 arithmetic of a cell is the same operation by operation, so
FP32 solves agree bit for bit; the mixed form sums its FP64 dot products in another order, a relative
change of a few 1e-16 per scalar (bar 1e-9, the scalars' effect on a solve to 1e-9)."""
import os

import numpy as np
import pytest

torch = pytest.importorskip("torch")

import anitowave_adaptive_b200 as aw  # noqa: E402

pytestmark = pytest.mark.gpu


def _solver(g, uniform, **kw):
    if not uniform:
        os.environ["AW_NO_UNIFORM"] = "1"
    try:
        return aw.Solver(g, **kw)
    finally:
        os.environ.pop("AW_NO_UNIFORM", None)


def _grid(dims, levels, R0=8, num_levels=4):
    g = aw.MSBG(dims, 1.0, (0.0, 0.0, 0.0), R0, num_levels)
    g.set_refinement_map(np.asarray(levels, np.uint32))
    g.enforce_grading()
    g.allocate()
    return g


def _solve(g, uniform, precision, fluid, b, tol, p0=None, **kw):
    sv = _solver(g, uniform, precision=precision, tolerance=tol, **kw)
    sv.setup(fluid)
    dt = torch.float64 if precision == aw.PRECISION_MIXED else torch.float32
    p = torch.zeros(b.numel(), dtype=dt, device="cuda") if p0 is None else p0.to(dt).clone()
    out = [sv.solve(b, p, raise_on_error=False)[:2] + (p.cpu().clone(),)]
    # again from the result: nothing of the first solve may leak into the second
    out.append(sv.solve(b, p, raise_on_error=False)[:2] + (p.cpu(),))
    torch.cuda.synchronize()
    sv.close()
    return out


def _same(a, b):
    """Equal values, NaN where the other is NaN (a closed box of one block has a singular coarsest cell)."""
    return torch.equal(a.isnan(), b.isnan()) and torch.equal(a.nan_to_num(), b.nan_to_num())


# block maps with every neighbour kind (same, coarser, finer, wall, absent), block sizes 8..1, odd block
# counts (one-cell blocks shift the cell offsets to odd values: unpaired loads), a single block
MAPS = {
    "one": ((1, 1, 1), [0]),
    "row": ((4, 2, 2), [x for z in range(2) for y in range(2) for x in range(4)]),
    "odd": ((5, 3, 3), [min(3, abs(x - 2) + (y == 2)) for z in range(3) for y in range(3) for x in range(5)]),
    "hole": ((4, 4, 4), [4 if (x, y, z) == (2, 2, 1) else min(3, max(x, y, z)) for z in range(4) for y in range(4)
                         for x in range(4)]),
    "coarse": ((6, 6, 6), [3] * 216),
}


# (the mixed form with a free surface only: a closed box leaves the mean of p free, here at 1e10 times the
# rest of p, and the order of the FP64 sums moves it)
@pytest.mark.parametrize("name", list(MAPS))
@pytest.mark.parametrize("surface,precision", [(False, aw.PRECISION_FP32), (True, aw.PRECISION_FP32),
                                               (False, aw.PRECISION_FP32_PCG), (True, aw.PRECISION_FP32_PCG),
                                               (True, aw.PRECISION_MIXED)])
def test_uniform_matches_staged(name, surface, precision):
    dims, lv = MAPS[name]
    g = _grid(dims, lv)
    n = g.totals()[0]
    gen = torch.Generator(device="cuda").manual_seed(7)
    X = g.face_positions(3)
    fluid = torch.ones(n, dtype=torch.uint8, device="cuda")
    if surface:  # a slanted free surface, so that blocks are full, cut and empty
        fluid = (X[:, 0] + 0.7 * X[:, 1] < 0.55 * dims[0]).to(torch.uint8)
    b = torch.randn(n, generator=gen, device="cuda") * fluid
    if not surface:
        b -= b.mean()
    p0 = 0.01 * torch.randn(n, generator=gen, device="cuda") * fluid if precision == aw.PRECISION_FP32 else None
    tol = 1e-9 if precision == aw.PRECISION_MIXED else 1e-30
    cyc = 60 if precision == aw.PRECISION_MIXED else 3
    a = _solve(g, True, precision, fluid, b, tol, p0, max_cycles=cyc)
    s = _solve(g, False, precision, fluid, b, tol, p0, max_cycles=cyc)
    for (c1, r1, p1), (c0, r0, q0) in zip(a, s):
        assert c1 == c0
        if precision == aw.PRECISION_MIXED:
            assert (p1 - q0).norm() <= 1e-9 * q0.norm(), ((p1 - q0).norm(), q0.norm())
        else:
            assert _same(p1, q0)
            assert not r0 == r0 or abs(r1 - r0) <= 1e-12 * max(r0, 1e-30)
    g.close()


@pytest.mark.parametrize("pre,post,local", [(1, 1, 1), (0, 2, 2), (2, 0, 2), (3, 1, 2)])
def test_uniform_smoothing_schedules(pre, post, local):
    dims, lv = MAPS["odd"]
    g = _grid(dims, lv)
    gen = torch.Generator(device="cuda").manual_seed(3)
    n = g.totals()[0]
    fluid = (g.face_positions(3)[:, 2] < 2.3).to(torch.uint8)
    b = torch.randn(n, generator=gen, device="cuda") * fluid
    kw = dict(max_cycles=2, pre_smooth=pre, post_smooth=post, block_iterations=local)
    a = _solve(g, True, aw.PRECISION_FP32, fluid, b, 1e-30, **kw)
    s = _solve(g, False, aw.PRECISION_FP32, fluid, b, 1e-30, **kw)
    assert all(_same(x[2], y[2]) for x, y in zip(a, s))
    g.close()


def test_non_uniform_coefficients_take_the_staged_form():
    """One face of one block differs: the whole solve must see it (and see it go away again)."""
    dims, lv = MAPS["row"]
    g = _grid(dims, lv)
    gen = torch.Generator(device="cuda").manual_seed(5)
    n = g.totals()[0]
    b = torch.randn(n, generator=gen, device="cuda")
    b -= b.mean()
    beta = g.channel(aw.BETA_COEFF_X)
    for value in (0.5, 1.0):
        beta[1] = value  # a face between two cells of the first block
        a = _solve(g, True, aw.PRECISION_FP32, None, b, 1e-30, max_cycles=2)
        s = _solve(g, False, aw.PRECISION_FP32, None, b, 1e-30, max_cycles=2)
        assert all(_same(x[2], y[2]) for x, y in zip(a, s))
    g.close()


def test_fluid_flags_change_between_solves():
    """Cells that leave the liquid keep nothing of the earlier solve."""
    dims, lv = MAPS["hole"]
    g = _grid(dims, lv)
    gen = torch.Generator(device="cuda").manual_seed(9)
    n = g.totals()[0]
    X = g.face_positions(3)
    b = torch.randn(n, generator=gen, device="cuda")
    sv = aw.Solver(g, precision=aw.PRECISION_MIXED, tolerance=1e-9, max_cycles=60)
    for cut in (3.5, 1.2, 2.6):
        fluid = (X[:, 1] < cut).to(torch.uint8)
        sv.setup(fluid)
        p = torch.zeros(n, dtype=torch.float64, device="cuda")
        sv.solve(b * fluid, p)
        ref = _solve(g, True, aw.PRECISION_MIXED, fluid, b * fluid, 1e-9, max_cycles=60)[0][2]
        assert torch.equal(p.cpu(), ref)
        assert not p[fluid == 0].any()
    sv.close()
    g.close()


@pytest.mark.parametrize("name", ["row", "odd", "hole"])
@pytest.mark.parametrize("precision", [aw.PRECISION_FP32, aw.PRECISION_FP32_PCG])
def test_varying_coefficients(name, precision):
    """Every face its own 1/rho (a stirred two-phase interface): every block reads its weights."""
    dims, lv = MAPS[name]
    g = _grid(dims, lv)
    gen = torch.Generator(device="cuda").manual_seed(2)
    n = g.totals()[0]
    for a in range(3):
        beta = g.channel(aw.BETA_COEFF_X + a)
        beta.copy_(0.3 + 0.7 * torch.rand(beta.numel(), generator=gen, device="cuda"))
    fluid = (g.face_positions(3)[:, 0] < 0.7 * dims[0]).to(torch.uint8)
    b = torch.randn(n, generator=gen, device="cuda") * fluid
    a = _solve(g, True, precision, fluid, b, 1e-30, max_cycles=2)
    s = _solve(g, False, precision, fluid, b, 1e-30, max_cycles=2)
    assert all(_same(x[2], y[2]) for x, y in zip(a, s))
    g.close()


@pytest.mark.parametrize("precision", [aw.PRECISION_FP32, aw.PRECISION_MIXED])
def test_vcycle_call(precision):
    """aw_vcycle_run from a given x: register-resident against staged, launched, replayed and captured."""
    dims, lv = MAPS["odd"]
    g = _grid(dims, lv)
    gen = torch.Generator(device="cuda").manual_seed(4)
    n = g.totals()[0]
    fluid = (g.face_positions(3)[:, 1] < 2.2).to(torch.uint8)
    b = torch.randn(n, generator=gen, device="cuda") * fluid
    x0 = torch.randn(n, generator=gen, device="cuda")  # air cells too: their values are the neighbours' ghosts

    def cycles(uniform, capture):
        sv = _solver(g, uniform, precision=precision)
        sv.setup(fluid)
        x, bb = sv.level_array(0, 0), sv.level_array(0, 1)
        x.copy_(x0)
        bb.copy_(b)
        torch.cuda.synchronize()
        if capture:
            s = torch.cuda.Stream()
            with torch.cuda.stream(s):
                sv.vcycle()
                s.synchronize()
                x.copy_(x0)
                G = torch.cuda.CUDAGraph()
                with torch.cuda.graph(G, stream=s):
                    sv.vcycle(stream=torch.cuda.current_stream().cuda_stream)
                G.replay()
                G.replay()
                s.synchronize()
            del G
        else:
            sv.vcycle()
            sv.vcycle()
        torch.cuda.synchronize()
        out = x.cpu().clone()
        sv.close()
        return out

    ref = cycles(False, False)
    assert torch.equal(cycles(True, False), ref)
    assert torch.equal(cycles(True, True), ref)
    g.close()


# block grids around the limits of the one-launch form: a CTA (16 warps), clusters of 2 to 8 CTAs, and more (levels
# with launches of their own), 128 and more coarsest cells (two legs around the coarsest solve)
@pytest.mark.parametrize("dims", [(2, 1, 1), (2, 2, 2), (4, 4, 2), (5, 7, 1), (8, 4, 4), (43, 3, 1), (8, 8, 2), (3, 3, 3), (5, 5, 5), (8, 8, 8), (13, 11, 8)])
@pytest.mark.parametrize("spread", [1, 4])
@pytest.mark.parametrize("precision", [aw.PRECISION_FP32, aw.PRECISION_MIXED])
def test_small_levels_in_one_launch(dims, spread, precision):
    """The same bodies in one launch and in a launch per step: equal bits, the mixed form's FP64 sums too."""
    nb = int(np.prod(dims))
    lv = np.arange(nb) * 7919 % spread
    g = _grid(dims, lv)
    gen = torch.Generator(device="cuda").manual_seed(nb)
    n = g.totals()[0]
    X = g.face_positions(3)
    fluid = (X[:, 0] + 0.4 * X[:, 1] < 0.8 * dims[0]).to(torch.uint8)
    b = torch.randn(n, generator=gen, device="cuda") * fluid
    for varying in (False, True):
        if varying:
            beta = g.channel(aw.BETA_COEFF_Y)
            beta.copy_(0.3 + 0.7 * torch.rand(beta.numel(), generator=gen, device="cuda"))
        a = _solve(g, True, precision, fluid, b, 1e-30, max_cycles=4)
        os.environ["AW_NO_UNIFORM_LOW"] = "1"
        try:
            s = _solve(g, True, precision, fluid, b, 1e-30, max_cycles=4)
        finally:
            os.environ.pop("AW_NO_UNIFORM_LOW", None)
        for (c1, r1, p1), (c0, r0, q0) in zip(a, s):
            assert c1 == c0 and _same(p1, q0) and (r1 == r0 or r0 != r0)
    g.close()
