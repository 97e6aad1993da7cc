"""P2G in blocks of crowded and of unequal cells: the sums of two phases against 64 bits, and the time beside that of
equal cells."""
import statistics

import numpy as np
import pytest

torch = pytest.importorskip("torch")

import anitowave_adaptive_b200 as aw  # noqa: E402

pytestmark = pytest.mark.gpu

EPS = float(np.finfo(np.float32).eps)


@pytest.mark.parametrize("counts", [[1], [15, 16, 17], [62, 63, 64, 65, 71, 72], [1000, 1, 0, 63], [16383, 16385, 3]])
@pytest.mark.parametrize("fill", [4, 40, 1024])  # cells that hold particles: a few, some, all
def test_phase_sums(counts, fill):
    dims, R = (2, 1, 1), 8
    if max(counts) * fill > 100_000:
        fill = 100
    g = aw.MSBG(dims, 1.0, (0.0, 0.0, 0.0), R, 1)
    g.set_refinement_map(np.zeros(2, np.uint32))
    g.allocate()
    rs = np.random.RandomState(len(counts) + fill)
    pos = []
    for k, c in enumerate(rs.permutation(2 * R ** 3)[:fill]):
        o = np.array([c % (2 * R), (c // (2 * R)) % R, c // (2 * R * R)])
        pos.append((o + rs.uniform(0.001, 0.999, (counts[k % len(counts)], 3))) / R)
    pos = np.concatenate(pos)
    pos = torch.tensor(pos[rs.permutation(len(pos))], dtype=torch.float32, device="cuda")
    vel = torch.randn(pos.shape, generator=torch.Generator(device="cuda").manual_seed(1), device="cuda")
    ph = torch.tensor(rs.choice([0.0, 0.3, 1.0], len(pos)), dtype=torch.float32, device="cuda")
    g.p2g_phase(pos, vel, ph, 1.0, 3.0)
    x = pos.double()
    for a in range(3):
        f = g.face_positions(a).double()
        q = torch.zeros(len(f), dtype=torch.float64, device="cuda")
        m, near = q.clone(), q.clone()
        for i in range(0, len(x), 4096):
            w = (1 - ((f[:, None, :] - x[None, i:i + 4096, :]) * R).square().sum(-1)).clamp_min(0) ** 3
            m += w.sum(1)
            q += w @ ph[i:i + 4096].double()
            near += (w > 0).sum(1)
        # a weight is off by 3 times its argument's error: positions of up to 16 cells, rounded three times
        # an axis, times a slope of 2; then a rounding for every term of a sum, and phi = Phi / m of both sums
        e = (3 * 3 * 2 * 3 * 16 * EPS + near * EPS) * near
        gm, gphi = g.channel(aw.MASS_DENSITY_X + a).double(), g.channel(aw.PHASE_FIELD_X + a).double()
        assert bool(((gm - m).abs() <= e + 1e-30).all())
        on = m > 1e-2
        assert bool(((gphi - q / m).abs()[on] <= (2 * e / m + 2 * EPS)[on]).all())
    g.close()


@pytest.mark.parametrize("phases", [False, True])
def test_unequal_crowded_cells_cost_what_equal_ones_do(phases):
    """300,000 particles of one block in 27 full and 37 part-filled cells against 64 equal ones: the same number of
    particles and tasks.  With every cell of 63 and more in one bin the former took 1.6 (1.3) times the latter."""
    g = aw.MSBG((4, 4, 4), 1.0, (0.0, 0.0, 0.0), 8, 1)
    g.init_refinement_map(0)
    g.allocate()
    gen = torch.Generator(device="cuda").manual_seed(5)
    n = 300_000
    ph = torch.ones(n, device="cuda")
    vel = torch.randn(n, 3, generator=gen, device="cuda")

    def timed(width):
        pos = torch.rand(n, 3, generator=gen, device="cuda") * width + 1.0
        ts = []
        for k in range(12):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            g.p2g_phase(pos, vel, ph, 1.0, 3.0) if phases else g.p2g(pos, vel)
            b.record()
            torch.cuda.synchronize()
            ts.append(a.elapsed_time(b))
        return statistics.median(ts[3:])

    unequal, equal = timed(0.4), timed(0.5)
    assert unequal < 1.25 * equal, (unequal, equal)
    g.close()
