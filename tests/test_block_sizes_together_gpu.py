"""Grids and solvers of different block sizes in one process: what a later, smaller one needs of a kernel's shared
memory does not take away what an earlier, larger one launches it with."""
import threading

import numpy as np
import pytest

torch = pytest.importorskip("torch")

import anitowave_adaptive_b200 as aw  # noqa: E402

pytestmark = pytest.mark.gpu


def _grid(R0, dims=(3, 2, 2)):
    g = aw.MSBG(dims, 1.0, (0.0, 0.0, 0.0), R0, 2)
    g.set_refinement_map((np.arange(int(np.prod(dims))) % 2).astype(np.uint32))
    g.enforce_grading()
    g.allocate()
    return g


def _problem(g):
    gen = torch.Generator(device="cuda").manual_seed(1)
    n = g.totals()[0]
    fluid = (g.face_positions(3)[:, 0] < 2.3).to(torch.uint8)
    return n, fluid, torch.randn(n, generator=gen, device="cuda") * fluid


def _solve(sv, b, mixed):
    p = torch.zeros(b.numel(), dtype=torch.float64 if mixed else torch.float32, device="cuda")
    sv.solve(b, p, raise_on_error=False)
    torch.cuda.synchronize()
    return p


def _level_calls(sv, b):
    """The level calls of one two-grid cycle, from x = 0."""
    sv.level_array(0, 0).zero_()
    sv.level_array(0, 1).copy_(b)
    sv.level_array(1, 0).zero_()
    sv.smooth(0, 2)
    sv.residual(0)
    sv.restrict(0)
    sv.smooth(1, 2)
    sv.prolongate(0)
    sv.residual(0)
    torch.cuda.synchronize()
    return sv.level_array(0, 0).clone(), sv.level_array(0, 2).clone()


@pytest.mark.parametrize("R0", [16, 8])
@pytest.mark.parametrize("precision", [aw.PRECISION_FP32, aw.PRECISION_MIXED, aw.PRECISION_FP32_PCG])
def test_a_smaller_solver_leaves_a_larger_one_working(R0, precision):
    mixed = precision == aw.PRECISION_MIXED
    g = _grid(R0)
    n, fluid, b = _problem(g)
    sv = aw.Solver(g, precision=precision, tolerance=1e-30, max_cycles=2)
    sv.setup(fluid)
    p, lev = _solve(sv, b, mixed), None if mixed else _level_calls(sv, b)
    small = [_grid(r, (2, 1, 1)) for r in (4, 2)]
    others = [aw.Solver(s, precision=precision) for s in small]
    assert torch.equal(_solve(sv, b, mixed), p)
    if not mixed:
        for a, r in zip(_level_calls(sv, b), lev):
            assert torch.equal(a, r)
    for o in others:
        o.close()
    sv.close()


@pytest.mark.parametrize("threads", [False, True])
def test_smaller_transfers_leave_larger_ones_working(threads):
    """P2G, G2P and advection of grids of every block size by turns, and by several host threads at once."""
    grids = {r: _grid(r) for r in (16, 8, 4)}
    gen = torch.Generator(device="cuda").manual_seed(2)
    n = 20_000
    pos = torch.rand((n, 3), generator=gen, device="cuda") * torch.tensor([3.0, 2.0, 2.0], device="cuda")
    vel = torch.randn((n, 3), generator=gen, device="cuda")
    torch.cuda.synchronize()
    bad = []

    def steps(r, k):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                s = torch.cuda.current_stream().cuda_stream
                for _ in range(k):
                    x, v = pos.clone(), vel.clone()
                    grids[r].p2g(x, v, stream=s)
                    grids[r].backup_grid_velocity(stream=s)
                    grids[r].g2p(v, x, 0.95, stream=s)
                    grids[r].advect(x, 0.01, stream=s)
                    torch.cuda.current_stream().synchronize()
        except Exception as e:  # noqa: BLE001
            bad.append(e)

    if threads:
        T = [threading.Thread(target=steps, args=(r, 40)) for r in grids]
        for t in T:
            t.start()
        for t in T:
            t.join()
    else:
        for r in (16, 8, 4, 16, 4, 8):
            steps(r, 1)
    assert not bad, bad
    for g in grids.values():
        g.close()
