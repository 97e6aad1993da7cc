"""Drop-in G2P and advection after a P2G of the same arrays (the order of the sort is used again when the
arrays' content hashes still match) against the same calls on copies at other addresses (no order to use):
particle counts around the four-particle hash step, arrays on and off a 16-byte boundary, inactive blocks,
and arrays that changed after the P2G."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import anitowave_adaptive_b200 as aw  # noqa: E402

pytestmark = pytest.mark.gpu

EPS = float(np.finfo(np.float32).eps)


def _grid(dims, base_res, seed):
    g = aw.MSBG(dims, 1.0 / max(dims), (0.0, 0.0, 0.0), base_res, 3 if base_res > 2 else 1)
    lv = np.random.RandomState(seed).randint(0, 4 if base_res > 2 else 1, int(np.prod(dims)))  # level 3: inactive
    lv[0] = 0
    g.set_refinement_map(lv.astype(np.uint32))
    g.enforce_grading()
    g.allocate()
    return g


def _at(x, off):
    """A copy of x whose first element lies `off` floats after a 16-byte boundary."""
    buf = torch.empty(x.numel() + 4, device="cuda")
    out = buf[off:off + x.numel()].view(x.shape)
    out.copy_(x)
    return out


@pytest.mark.parametrize("n", [1, 3, 4, 5, 1023, 1025, 70_001, 303_105, 1_250_000])  # 303104 = 148 x 8 CTAs of 256
@pytest.mark.parametrize("off", [0, 1])
@pytest.mark.parametrize("change", [None, "first", "last"])
def test_drop_in_calls(n, off, change):
    g = _grid((5, 4, 3), 8, 3)
    gen = torch.Generator(device="cuda").manual_seed(n)
    ext = torch.tensor([1.0, 0.8, 0.6], device="cuda")
    pos = _at(torch.rand((n, 3), generator=gen, device="cuda") * ext, off)
    vel = _at(torch.randn((n, 3), generator=gen, device="cuda"), off)
    at = {None: None, "first": 0, "last": -1}[change]
    alpha, dt, h = 0.95, 0.01, 0.2 / 8
    g.p2g(pos, vel)
    g.backup_grid_velocity()
    if change:
        vel[at, 1] += 0.5
    pos2, vel2 = _at(pos, 2), _at(vel, 2)
    before = vel.clone()
    g.g2p(vel, pos, alpha)
    g.g2p(vel2, pos2, alpha)
    # either side: 27 products a component and time level at most, each rounded twice
    umax = float(before.abs().max()) + 1
    assert float((vel - vel2).abs().max()) <= 108 * EPS * umax
    g.p2g(pos, vel)
    if change:
        pos[at, 2] *= 0.5
    pos2 = _at(pos, 2)
    g.advect(pos, dt)
    g.advect(pos2, dt)
    # three samples; a difference in position moves the next sample by the velocity's slope, 2 umax / h at most
    tol = 8 * EPS + dt * 3 * 108 * EPS * umax * (1 + 2 * dt * umax / h) ** 2
    assert float((pos - pos2).abs().max()) <= tol
    g.close()


def test_small_blocks_do_not_change_later_steps():
    """A FLIP step on 8-cell blocks after an advection of a grid of 4-cell blocks (smaller shared tiles)."""
    def step():
        g = _grid((2, 2, 2), 8, 1)
        g.set_refinement_map(np.zeros(8, np.uint32))
        g.allocate()
        gen = torch.Generator(device="cuda").manual_seed(1)
        pos = torch.rand((2000, 3), generator=gen, device="cuda") * torch.tensor([0.9, 0.4, 0.9], device="cuda") + 0.02
        vel = torch.randn((2000, 3), generator=gen, device="cuda") * 0.1
        sim = aw.Flip(g, pos.cpu().numpy(), vel.cpu().numpy(), 0.01)
        sim.step()
        out = sim.particles()[0]
        sim.close()
        g.close()
        return out

    h = _grid((2, 2, 2), 4, 1)
    p = torch.rand((100, 3), device="cuda")
    v = torch.zeros_like(p)
    h.p2g(p, v)
    h.advect(p, 0.01)
    h.close()
    out = step()
    assert bool(np.isfinite(np.asarray(out)).all())
