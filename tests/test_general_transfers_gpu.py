"""Drop-in G2P and advection of arrays that changed after the P2G, at the particle count where a thread of the
general kernels starts to take four: against copies at other addresses (a particle a thread, no sorted path)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import anitowave_adaptive_b200 as aw  # noqa: E402

pytestmark = pytest.mark.gpu

EPS = float(np.finfo(np.float32).eps)
LONG = 148 * 16 * 256


@pytest.mark.parametrize("n", [255, 257, LONG - 1, LONG, LONG + 1, LONG + 1023, LONG + 1025])
def test_changed_arrays(n):
    g = aw.MSBG((5, 4, 3), 0.2, (0.0, 0.0, 0.0), 8, 3)
    g.set_refinement_map(np.random.RandomState(1).randint(0, 4, 60).astype(np.uint32))  # level 3: inactive
    g.enforce_grading()
    g.allocate()
    gen = torch.Generator(device="cuda").manual_seed(n)
    pos = torch.rand((n, 3), generator=gen, device="cuda") * torch.tensor([1.0, 0.8, 0.6], device="cuda")
    vel = torch.randn((n, 3), generator=gen, device="cuda")
    g.p2g(pos, vel)
    g.backup_grid_velocity()
    vel[-1, 1] += 0.5
    umax = float(vel.abs().max()) + 1
    pos2, vel2 = pos.clone(), vel.clone()
    g.g2p(vel, pos, 0.95)
    g.g2p(vel2, pos2, 0.95)
    # 27 products a component and time level at most on either side, each rounded twice
    assert float((vel - vel2).abs().max()) <= 108 * EPS * umax
    g.p2g(pos, vel)
    pos[-1, 2] *= 0.5
    pos2 = pos.clone()
    g.advect(pos, 0.01)
    g.advect(pos2, 0.01)
    # three stages of such samples, dt times their sum, and the positions' own rounding; a stage point that
    # falls on the other side of a cell face moves the sample by the same order
    assert float((pos - pos2).abs().max()) <= 0.01 * 3 * 108 * EPS * umax + 4 * EPS
    g.close()
