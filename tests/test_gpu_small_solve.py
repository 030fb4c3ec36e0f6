"""Solves of systems that fit one CTA (one launch) at the edges of that rule: the smallest grid, an
elongated one whose cells do not fill the threads, the largest, the first that does not fit, and
hierarchies whose bottom level has more than a few unknowns -- against the oracle's solve, and
against the kernels launched one by one (no CUDA graph)."""
import numpy as np
import pytest

from lica_boiling1d_b200.inputs import bubble_poisson_case
from oracle import oracle

pytestmark = pytest.mark.gpu


def _t(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


# 32 x 96: bottom level 2 x 6; 96 x 32: 3 x 1 levels end at 6 x 2; 64 x 96 does not fit
@pytest.mark.parametrize("nx,ny,nlevels,ncoarse", [(32, 32, 2, 1), (32, 96, 2, 2), (96, 32, 2, 1), (64, 64, 3, 1),
                                                   (64, 64, 2, 2), (128, 32, 2, 1), (64, 96, 2, 1)])
def test_small_solve(nx, ny, nlevels, ncoarse):
    import torch
    from lica_boiling1d_b200 import poisson
    c = bubble_poisson_case(nx, ny=ny, nbubbles=6, rmin=2.0, rmax=6.0)
    ref, it_ref, _, _, st_ref = oracle.mg_solve(c.f, c.bx, c.by, c.hx, c.hy, nlevels=nlevels, ncoarse=ncoarse, sym=5,
                                                method="pcg", rtol=1e-10, max_cycles=100)
    assert st_ref == 0
    got = {}
    for graph in (True, False):
        s = poisson.MultigridPoisson(nx, ny, c.hx, c.hy, nlevels=nlevels, ncoarse=ncoarse, use_graph=graph)
        for _ in range(2):      # the second solve from a fresh start, the context's own state left by the first
            p = torch.zeros((ny, nx), dtype=torch.float64, device="cuda")
            it, rel, st = s.solve(p, _t(c.f), _t(c.bx), _t(c.by), rtol=1e-10, max_iters=100)
        assert st == 0 and rel <= 1e-10 and abs(it - it_ref) <= 1, (graph, it, it_ref, rel, st)
        got[graph] = p.cpu().numpy()
        # an iteration cap is honoured and reported
        p.zero_()
        it, rel, st = s.solve(p, _t(c.f), _t(c.bx), _t(c.by), rtol=1e-10, max_iters=2)
        assert (it, st) == (2, 1) and rel > 1e-10
        # nothing to do: the start is the answer
        p.copy_(_t(got[graph]))
        it, rel, st = s.solve(p, _t(c.f), _t(c.bx), _t(c.by), rtol=1e-9, max_iters=100)
        assert (it, st) == (0, 0)
        np.testing.assert_array_equal(p.cpu().numpy(), got[graph])
        s.close()
    for g in got.values():
        assert np.linalg.norm(g - ref) <= 1e-10 * np.linalg.norm(ref)
