"""P2G with cells of very different particle counts (the order of a block's cells by count, its last bin, the
slices of crowded cells), against the sums in 64 bits."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import anitowave_adaptive_b200 as aw  # noqa: E402

pytestmark = pytest.mark.gpu

EPS = float(np.finfo(np.float32).eps)


@pytest.mark.parametrize("counts", [[1], [15, 16, 17], [32, 33], [62, 63, 64, 65], [1000, 1, 0, 63], [3000]])
@pytest.mark.parametrize("fill", [4, 1024])  # cells that hold particles: a few, all
def test_p2g_sums(counts, fill):
    dims, R = (2, 1, 1), 8
    if max(counts) * fill > 100_000:
        fill = 40
    g = aw.MSBG(dims, 1.0, (0.0, 0.0, 0.0), R, 1)
    g.set_refinement_map(np.zeros(2, np.uint32))
    g.allocate()
    rs = np.random.RandomState(len(counts) + fill)
    cells = rs.permutation(2 * R ** 3)[:fill]
    pos = []
    for k, c in enumerate(cells):
        n = counts[k % len(counts)]
        o = np.array([c % (2 * R), (c // (2 * R)) % R, c // (2 * R * R)])
        pos.append((o + rs.uniform(0.001, 0.999, (n, 3))) / R)
    pos = torch.tensor(np.concatenate(pos)[rs.permutation(sum(len(p) for p in pos))], dtype=torch.float32, device="cuda")
    vel = torch.randn(pos.shape, generator=torch.Generator(device="cuda").manual_seed(1), device="cuda")
    g.p2g(pos, vel)
    x = pos.double()
    for a in range(3):
        f = g.face_positions(a).double()
        m = torch.zeros(len(f), dtype=torch.float64, device="cuda")
        p, near, size = m.clone(), m.clone(), m.clone()
        for i in range(0, len(x), 4096):
            d2 = ((f[:, None, :] - x[None, i:i + 4096, :]) * R).square().sum(-1)
            w = (1 - d2).clamp_min(0) ** 3
            v = vel[i:i + 4096, a].double()
            m += w.sum(1)
            p += w @ v
            near += (w > 0).sum(1)
            size += (w > 0).double() @ v.abs()
        # a weight is off by 3 times its argument's error: positions of up to 16 cells, rounded three times
        # an axis, times a slope of 2; then a rounding for every term of a sum
        e = 3 * 3 * 2 * 3 * 16 * EPS
        gm, gp = g.channel(aw.MASS_DENSITY_X + a).double(), g.channel(aw.MOMENTUM_X + a).double()
        assert bool(((gm - m).abs() <= (e + near * EPS) * near + 1e-30).all())
        assert bool(((gp - p).abs() <= (e + near * EPS) * size + 1e-30).all())
    g.close()
