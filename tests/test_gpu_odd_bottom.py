"""Grids whose coarsening ends at an odd number of columns (3 x 2 to 3 x 13 cells, 5 x 2, 3 x 1), where
a row of the bottom level's colour-split arrays holds one cell more of one colour than of the other,
and a bottom level of more unknowns than a warp has lanes: the preconditioner against the oracle's bit
for bit, FP64 and mixed, and solves in the oracle's iterations."""
import numpy as np
import pytest

from lica_boiling1d_b200.inputs import bubble_poisson_case
from oracle import oracle

pytestmark = pytest.mark.gpu


def _t(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _case(nx, ny):
    return bubble_poisson_case(nx, ny=ny, nbubbles=6, rmin=2.0, rmax=6.0)


# bottom levels 3x2, 3x2, 5x2, 3x3, 3x4, 2x18, 3x13, and with the last outer level the bottom 3x2, 3x1
GRIDS = [(96, 64, 3), (192, 128, 4), (160, 64, 3), (96, 96, 3), (96, 128, 3), (32, 288, 2), (96, 416, 3),
         (96, 64, 6), (96, 32, 6)]


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("nx,ny,nlevels", GRIDS)
def test_preconditioner_bitwise(nx, ny, nlevels, precision):
    import torch
    from lica_boiling1d_b200 import poisson
    c = _case(nx, ny)
    ref = oracle.mg_precond(c.f, c.bx, c.by, c.hx, c.hy, nlevels=nlevels, ncoarse=2, sym=5,
                            mixed=(precision == "mixed"))
    s = poisson.MultigridPoisson(nx, ny, c.hx, c.hy, nlevels=nlevels, ncoarse=2, precision=precision)
    z = torch.empty((ny, nx), dtype=torch.float64, device="cuda")
    s.precond(z, _t(c.f), _t(c.bx), _t(c.by))
    s.close()
    np.testing.assert_array_equal(z.cpu().numpy(), ref)


# 96 x 32 is one launch with the graph, and the kernels one by one without it
@pytest.mark.parametrize("nx,ny,nlevels", GRIDS)
def test_solve_iterations(nx, ny, nlevels):
    import torch
    from lica_boiling1d_b200 import poisson
    c = _case(nx, ny)
    ref, it_ref, _, _, st_ref = oracle.mg_solve(c.f, c.bx, c.by, c.hx, c.hy, nlevels=nlevels, ncoarse=2, sym=5,
                                                method="pcg", rtol=1e-10, max_cycles=100)
    assert st_ref == 0
    for graph in (True, False):
        s = poisson.MultigridPoisson(nx, ny, c.hx, c.hy, nlevels=nlevels, ncoarse=2, use_graph=graph)
        p = torch.zeros((ny, nx), dtype=torch.float64, device="cuda")
        it, rel, st = s.solve(p, _t(c.f), _t(c.bx), _t(c.by), rtol=1e-10, max_iters=100)
        s.close()
        assert st == 0 and rel <= 1e-10 and it == it_ref, (graph, it, it_ref, rel, st)
        got = p.cpu().numpy()
        assert np.linalg.norm(got - ref) <= 1e-10 * np.linalg.norm(ref)
