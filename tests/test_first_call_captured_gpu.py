"""The first P2G and sort of a grid inside a stream capture: its buffers are allocated while the work is only
recorded, so a direct call that comes before the first replay must not count on anything the capture would have
initialised.  (Freed device memory of all ones is left behind, so that fresh buffers are not zero by luck.)"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import anitowave_adaptive_b200 as aw  # noqa: E402

pytestmark = pytest.mark.gpu


def _grid():
    g = aw.MSBG((5, 4, 3), 0.2, (0.0, 0.0, 0.0), 8, 3)
    g.set_refinement_map((np.arange(60) % 3).astype(np.uint32))
    g.enforce_grading()
    g.allocate()
    return g


@pytest.mark.parametrize("n", [1, 5000, 300_000])
@pytest.mark.parametrize("call", ["p2g", "sort"])
def test_first_call_captured(n, call):
    gen = torch.Generator(device="cuda").manual_seed(n)
    pos = torch.rand((n, 3), generator=gen, device="cuda") * torch.tensor([1.0, 0.8, 0.6], device="cuda")
    vel = torch.randn((n, 3), generator=gen, device="cuda")
    keys, perm = (torch.empty(n, dtype=torch.int32, device="cuda") for _ in range(2))

    def run(g, stream=None):
        if call == "p2g":
            g.p2g(pos, vel, stream=stream)
        else:
            aw.check(aw.lib().aw_sort_particles(g.h, pos.data_ptr(), n, keys.data_ptr(), perm.data_ptr(), stream))

    def result(g):
        torch.cuda.synchronize()
        if call == "sort":
            return [keys.clone(), perm.clone()]
        return [g.channel(c + a).clone() for c in (aw.VELOCITY_X, aw.MASS_DENSITY_X) for a in range(3)] + [
            g.channel(aw.CELL_TYPE).clone()]

    ref_grid = _grid()
    run(ref_grid)
    ref = result(ref_grid)

    def same(got):
        for a, r in zip(got, ref):
            if a.dtype == torch.int32 or (a is got[-1]):
                assert torch.equal(a, r)
            else:  # float sums in an order of their own: at most some 1000 particles reach a face, so k eps is
                # 1.2e-4 of the largest value in mass and momentum each, and u is their quotient
                assert float((a - r).abs().max()) <= 1e-3 * float(r.abs().max())

    dirt = [torch.full((k,), -1, dtype=torch.int32, device="cuda") for k in [2 ** e for e in range(10, 24)] * 2]
    torch.cuda.synchronize()
    del dirt
    torch.cuda.empty_cache()
    g = _grid()
    s = torch.cuda.Stream()
    G = torch.cuda.CUDAGraph()
    with torch.cuda.graph(G, stream=s, capture_error_mode="relaxed"):
        run(g, s.cuda_stream)
    for go in (lambda: run(g), G.replay, lambda: run(g)):
        keys.zero_()
        perm.zero_()
        torch.cuda.synchronize()
        go()
        same(result(g))
    del G
    g.close()
    ref_grid.close()
