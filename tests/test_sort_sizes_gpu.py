"""The particle sort at the sizes where its tiling changes: warps, 1024-key tiles, 4096-key steps, the tile
cap, one and several digits, random and crowded keys, against a stable torch sort of the same keys."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import anitowave_adaptive_b200 as aw  # noqa: E402

pytestmark = pytest.mark.gpu


def _grid(dims, seed):
    g = aw.MSBG(dims, 1.0 / max(dims), (0.0, 0.0, 0.0), 8, 3)
    lv = np.random.RandomState(seed).randint(0, 4, int(np.prod(dims)))  # level 3: inactive blocks
    g.set_refinement_map(lv.astype(np.uint32))
    g.enforce_grading()
    g.allocate()
    return g


# (3, 2, 1): one digit; 16^3 blocks: two
@pytest.mark.parametrize("dims", [(3, 2, 1), (16, 16, 16)])
@pytest.mark.parametrize("n", [1, 31, 33, 1023, 1025, 4095, 4097, 100_003, 592 * 1024, 592 * 1024 + 1, 5_000_001])
@pytest.mark.parametrize("crowded", [False, True])
def test_sort_is_stable(dims, n, crowded):
    g = _grid(dims, 1)
    gen = torch.Generator(device="cuda").manual_seed(n)
    pos = torch.rand((n, 3), generator=gen, device="cuda")
    if crowded:  # runs of one cell, half of the particles
        pos[n // 4:n // 4 + n // 2] = 0.3
    keys, perm = g.sort_particles(pos)
    torch.cuda.synchronize()
    k = torch.empty(n, dtype=torch.int64, device="cuda")
    k[perm.long()] = keys.long()
    ref = torch.sort(k, stable=True)
    assert torch.equal(ref.indices, perm.long())
    assert torch.equal(ref.values, keys.long())
    g.close()
