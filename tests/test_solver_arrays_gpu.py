"""Which arrays the solver takes and what it leaves in its own."""
import ctypes as C
import os
import statistics
import time

import numpy as np
import pytest

torch = pytest.importorskip("torch")

import anitowave_adaptive_b200 as aw  # noqa: E402

pytestmark = pytest.mark.gpu

ALL = (aw.PRECISION_FP32, aw.PRECISION_MIXED, aw.PRECISION_FP32_PCG)


def _grid(R0=8, dims=(5, 3, 3)):
    """Blocks of every size beside one another, an inactive one among them."""
    lv = [min(3, abs(x - 2) + (y == 2)) for z in range(dims[2]) for y in range(dims[1]) for x in range(dims[0])]
    lv[-1] = 4
    g = aw.MSBG(dims, 1.0, (0.0, 0.0, 0.0), R0, 4)
    g.set_refinement_map(np.asarray(lv, np.uint32))
    g.enforce_grading()
    g.allocate()
    return g


def _problem(g, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    n = g.totals()[0]
    fluid = (g.face_positions(3)[:, 0] < 3.3).to(torch.uint8)  # full, cut and empty blocks
    return n, fluid, torch.randn(n, generator=gen, device="cuda") * fluid


@pytest.mark.parametrize("precision", ALL)
@pytest.mark.parametrize("R0", [8, 16])
def test_arrays_that_start_at_any_element(R0, precision):
    """Views at odd elements of b and p give the bits of arrays of their own, and nothing beside them is touched."""
    g = _grid(R0)
    n, fluid, b0 = _problem(g, 1)
    dt = torch.float64 if precision == aw.PRECISION_MIXED else torch.float32
    sv = aw.Solver(g, precision=precision, tolerance=1e-30, max_cycles=3)
    sv.setup(fluid)
    ref = torch.zeros(n, dtype=dt, device="cuda")
    cyc, rel, st = sv.solve(b0, ref, raise_on_error=False)
    for ob, op in [(1, 0), (0, 1), (1, 1), (2, 3), (3, 2), (4, 4)]:
        bb = torch.full((n + 8,), 7.0, device="cuda")
        pp = torch.full((n + 8,), 7.0, dtype=dt, device="cuda")
        b, p = bb[ob:ob + n], pp[op:op + n]
        b.copy_(b0)
        p.zero_()
        torch.cuda.synchronize()
        assert sv.solve(b, p, raise_on_error=False) == (cyc, rel, st)
        assert torch.equal(p, ref) and torch.equal(b, b0)
        assert (pp[:op] == 7).all() and (pp[op + n:] == 7).all()
    sv.close()
    g.close()


def _solver(g, env=(), **kw):
    for k in env:
        os.environ[k] = "1"
    try:
        return aw.Solver(g, **kw)
    finally:
        for k in env:
            os.environ.pop(k, None)


@pytest.mark.parametrize("pre", [2, 0])
@pytest.mark.parametrize("form", ["launched", "replayed", "captured"])
def test_vcycle_sees_the_flags_and_coefficients_of_its_call(form, pre):
    """Fluid flags and 1/rho change between two V-cycles: the kernels right behind the check of the blocks read
    the new weights and masks, launched one by one, from the solver's graph and in a graph of the caller's."""
    g = _grid()
    n, _, b0 = _problem(g, 2)
    gen = torch.Generator(device="cuda").manual_seed(6)
    X = g.face_positions(3)
    steps = []
    for k in range(6):
        fluid = (X[:, k % 3] + 0.3 * X[:, (k + 1) % 3] < (3.0, 1.6, 2.5)[k % 3]).to(torch.uint8)
        steps.append((fluid, None if k % 2 else 0.3 + 0.7 * torch.rand(g.channel(aw.BETA_COEFF_Y).numel(), generator=gen,
                                                                      device="cuda")))
    env = {"launched": ("AW_NO_GRAPH",), "staged": ("AW_NO_UNIFORM",)}

    def run(form):
        sv = _solver(g, env.get(form, ()), pre_smooth=pre)
        x, b = sv.level_array(0, 0), sv.level_array(0, 1)
        out, G = [], None
        s = torch.cuda.Stream()
        with torch.cuda.stream(s):
            if form == "captured":
                G = torch.cuda.CUDAGraph()
                with torch.cuda.graph(G, stream=s):
                    sv.vcycle(stream=s.cuda_stream)
            for fluid, beta in steps:
                ch = g.channel(aw.BETA_COEFF_Y)
                ch.fill_(1.0) if beta is None else ch.copy_(beta)
                sv.update_coefficients(stream=s.cuda_stream)
                sv.setup(fluid, stream=s.cuda_stream)
                x.zero_()
                b.copy_(b0 * fluid)
                G.replay() if G else sv.vcycle(stream=s.cuda_stream)
                out.append(x.clone())
            s.synchronize()
        del G
        sv.close()
        return out

    for a, r in zip(run(form), run("staged")):
        assert torch.equal(a, r)
    g.close()


STAGED = ("AW_NO_UNIFORM", "AW_NO_UNIFORM_LOW", "AW_NO_DENSE_TAIL")
GRIDS = {  # one-cell blocks: 45 (odd), 256 (the tail's top), 32768 (uniform levels of 4096 cells and below)
    "odd": lambda: _grid(),
    "tail": lambda: _grid(8, (8, 8, 4)),
    "uniform": lambda: _even(2, (32, 32, 32)),
}


def _even(R0, dims):
    g = aw.MSBG(dims, 1.0, (0.0, 0.0, 0.0), R0, 2)
    g.set_refinement_map(np.asarray([(i // 7) % 2 for i in range(int(np.prod(dims)))], np.uint32))
    g.enforce_grading()
    g.allocate()
    return g


def _levels(sv, precision):
    """x, b, r and fluid flags of every level (r not on the coarsest; FP16 x without its scales)."""
    out, nl = {}, sv.num_levels()
    for m in range(nl):
        try:
            res = int(sv.level_array(m, 11).max())
        except aw.AWError:  # a uniform level
            res = 1
        for which in (0, 1, 2, 6):
            if which == 2 and m + 1 == nl:
                continue
            if which == 0 and precision == aw.PRECISION_MIXED and m > 0 and res > 1:
                p, n = C.c_void_p(), C.c_uint32()
                aw.check(aw.lib().aw_solver_level_array(sv.h, m, 0, C.byref(p), C.byref(n)))
                out[m, which] = aw._tensor_from_ptr(p.value, n.value, torch.float16).clone()
            else:
                out[m, which] = sv.level_array(m, which).clone()
    torch.cuda.synchronize()
    return out


def _cut(X, cut):
    return (X[:, 0] + 0.3 * X[:, 1] < cut * float(X[:, 0].max())).to(torch.uint8)


@pytest.mark.parametrize("name", list(GRIDS))
@pytest.mark.parametrize("precision", [aw.PRECISION_FP32, aw.PRECISION_MIXED])
def test_vcycle_leaves_every_levels_arrays(name, precision):
    """x, b and r of all levels after aw_vcycle_run: the register-resident, one-launch forms leave the bits of the
    staged ones, in blocks that lose their fluid from one call to the next too."""
    g = GRIDS[name]()
    n, _, b0 = _problem(g, 3)
    X = g.face_positions(3)
    got = []
    for env in (), STAGED:
        sv = _solver(g, env, precision=precision)
        x, b = sv.level_array(0, 0), sv.level_array(0, 1)
        for cut in (0.9, 0.6, 0.25):
            fluid = _cut(X, cut)
            sv.setup(fluid)
            x.zero_()
            b.copy_(b0 * fluid)
            torch.cuda.synchronize()
            sv.vcycle()
            torch.cuda.synchronize()
            got.append(_levels(sv, precision))
        sv.close()
    for a, r in zip(got[:3], got[3:]):
        assert a.keys() == r.keys()
        for k in a:
            assert torch.equal(a[k], r[k]), k
    g.close()


@pytest.mark.parametrize("name", list(GRIDS))
@pytest.mark.parametrize("precision", ALL)
def test_solve_leaves_every_levels_arrays(name, precision):
    """... and after aw_solve those of its last cycle, r in the FP32 form.  The mixed form's FP64 sums have another order: a relative
    change of some 1e-16 a scalar, at most an FP32 rounding here (bar 1e-5 of an array's largest value, FP16 x left
    out), and exact zeros without fluid."""
    g = GRIDS[name]()
    n, _, b0 = _problem(g, 4)
    X = g.face_positions(3)
    got = []
    for env in (), STAGED:
        sv = _solver(g, env, precision=precision, tolerance=1e-30, max_cycles=2)
        for cut in (0.9, 0.4):
            fluid = _cut(X, cut)
            sv.setup(fluid)
            p = torch.zeros(n, dtype=torch.float64 if precision == aw.PRECISION_MIXED else torch.float32, device="cuda")
            sv.solve(b0 * fluid, p, raise_on_error=False)
            got.append(_levels(sv, precision))
        sv.close()
    for a, r in zip(got[:2], got[2:]):
        for k in a:
            if precision != aw.PRECISION_FP32 and k[1] == 2:
                continue
            if precision != aw.PRECISION_MIXED or k[1] == 6:
                assert torch.equal(a[k], r[k]), k
            elif a[k].dtype == torch.float32:
                d = (a[k] - r[k]).abs().max()
                assert d <= 1e-5 * r[k].abs().max(), (k, d)
                air = a[k[0], 6] == 0
                assert not a[k][air].any() and not r[k][air].any(), k
    g.close()


@pytest.mark.parametrize("env", [(), ("AW_NO_UNIFORM",)])
def test_vcycle_after_a_solve_leaves_every_levels_arrays(env):
    """A mixed solve's cycles do not store r; a call after it does, in the tail's levels too."""
    g = GRIDS["tail"]()
    n, fluid, b0 = _problem(g, 5)
    got = []
    for e in env, STAGED:
        sv = _solver(g, e, precision=aw.PRECISION_MIXED, tolerance=1e-30, max_cycles=1)
        sv.setup(fluid)
        sv.solve(b0, torch.zeros(n, dtype=torch.float64, device="cuda"), raise_on_error=False)
        sv.level_array(0, 0).zero_()
        sv.level_array(0, 1).copy_(b0)
        torch.cuda.synchronize()
        sv.vcycle()
        torch.cuda.synchronize()
        got.append(_levels(sv, aw.PRECISION_MIXED))
        sv.close()
    assert all(torch.equal(got[0][k], got[1][k]) for k in got[1])
    g.close()


def test_solves_and_vcycles_by_turns_capture_nothing_again():
    """A V-cycle solve and aw_vcycle_run called in turn take about as long as each on its own (medians; capturing and
    instantiating the cycle's graph in every call made the pair take several times that)."""
    g = _grid(8, (8, 8, 4))
    n, fluid, b0 = _problem(g, 8)
    sv = aw.Solver(g, precision=aw.PRECISION_FP32, tolerance=1e-30, max_cycles=2)
    sv.setup(fluid)
    p = torch.zeros(n, device="cuda")
    sv.level_array(0, 1).copy_(b0)

    def solve():
        sv.solve(b0, p, raise_on_error=False)

    def seconds(*calls):
        t = []
        for _ in range(60):
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            for c in calls:
                c()
            torch.cuda.synchronize()
            t.append(time.perf_counter() - t0)
        return statistics.median(t[10:])

    alone = seconds(solve) + seconds(sv.vcycle)
    assert seconds(solve, sv.vcycle) <= 1.5 * alone
    sv.close()
    g.close()


@pytest.mark.parametrize("R0", [8, 1])
def test_reference_operator_iterates_on_air_cells_too(R0):
    """The reference's operator has a row on every cell, flagged or not: after one mixed CG iteration the V-cycle's
    next input (level-0 b) is b - A p on air cells as on fluid ones.  R0 = 1: an odd number of cells."""
    g = aw.MSBG((3, 3, 3), 1.0, (0.0, 0.0, 0.0), R0, 1)
    g.init_refinement_map(0)
    g.allocate()
    n = g.totals()[0]
    gen = torch.Generator(device="cuda").manual_seed(9)
    b = torch.randn(n, generator=gen, device="cuda")
    fluid = (torch.rand(n, generator=gen, device="cuda") < 0.6).to(torch.uint8)
    fluid[-1], fluid[-2], fluid[-3] = 0, 1, 0
    sv = aw.Solver(g, operator_mode=aw.OPERATOR_REFERENCE, precision=aw.PRECISION_MIXED, tolerance=1e-30, max_cycles=1)
    sv.setup(fluid)
    p = torch.zeros(n, dtype=torch.float64, device="cuda")
    sv.solve(b, p, raise_on_error=False)
    got = sv.level_array(0, 1).clone()
    sv.level_array(0, 1).copy_(b)
    sv.level_array(0, 0).copy_(p.float())
    torch.cuda.synchronize()
    sv.residual(0)
    torch.cuda.synchronize()
    want = sv.level_array(0, 2).clone()
    # FP32 residual: p rounded once, at most 13 rounded products and sums of values up to 12 |w| |p|
    w = max(float(sv.level_array(0, 3 + a).abs().max()) for a in range(3))
    tol = 16 * 2.0 ** -24 * (float(b.abs().max()) + 12 * w * float(p.abs().max()))
    assert float((got - want).abs().max()) <= tol
    assert float((want - b)[fluid == 0].abs().max()) > 100 * tol
    sv.close()
    g.close()


@pytest.mark.parametrize("precision", [aw.PRECISION_FP32, aw.PRECISION_MIXED])
def test_operators_by_turns_capture_nothing_again(precision):
    """Solves of one density and of a varying one in turn take about as long as each on its own (medians): the graphs
    of both forms are kept."""
    g = _grid(8, (8, 8, 4))
    n, fluid, b0 = _problem(g, 8)
    gen = torch.Generator(device="cuda").manual_seed(3)
    sv = aw.Solver(g, precision=precision, tolerance=1e-30, max_cycles=2)
    p = torch.zeros(n, dtype=torch.float64 if precision == aw.PRECISION_MIXED else torch.float32, device="cuda")
    beta = [g.channel(aw.BETA_COEFF_X + a) for a in range(3)]
    varied = [0.3 + 0.7 * torch.rand(t.numel(), generator=gen, device="cuda") for t in beta]
    plain = [torch.ones_like(t) for t in beta]

    def solve(values):
        for t, v in zip(beta, values):
            t.copy_(v)
        sv.update_coefficients()
        sv.setup(fluid)
        p.zero_()
        sv.solve(b0, p, raise_on_error=False)
        return p.clone()

    def seconds(*calls):
        t = []
        for _ in range(60):
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            for c in calls:
                solve(c)
            torch.cuda.synchronize()
            t.append(time.perf_counter() - t0)
        return statistics.median(t[10:])

    ref = [solve(plain), solve(varied)]
    assert not torch.equal(*ref)
    alone = seconds(plain) + seconds(varied)
    pair = seconds(plain, varied)
    for _ in range(2):
        assert torch.equal(solve(plain), ref[0]) and torch.equal(solve(varied), ref[1])
    assert pair < 1.3 * alone, (pair, alone)
    sv.close()
    g.close()
