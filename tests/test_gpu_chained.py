"""The multigrid kernels launched as a chain, each started before the one ahead of it has ended: the
weights are read ahead of the wait, so they are changed from one call to the next here, with no
synchronisation between the preconditioner's calls, on hierarchies with one tile shape, two, and none
above the single-CTA level.  The results are those of a context that is used once, bit for bit."""
import numpy as np
import pytest

from lica_boiling1d_b200.inputs import bubble_poisson_case

pytestmark = pytest.mark.gpu


def _case(nx, ny, k):
    import torch
    c = bubble_poisson_case(nx, ny=ny, nbubbles=5 + 3 * k, rmin=2.0, rmax=6.0 + 2 * k)
    return c, [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (c.f, c.bx, c.by)]


@pytest.mark.parametrize("nx,ny,opt", [(64, 96, dict(nlevels=2)), (128, 256, dict(nlevels=4, nu1=3, nu2=3)),
                                       (256, 128, dict(nlevels=4, precision="mixed")), (512, 512, dict(nlevels=5)),
                                       (64, 128, dict(nlevels=4, smoother="yline"))])
def test_chain(nx, ny, opt):
    import torch
    from lica_boiling1d_b200 import poisson
    cases = [_case(nx, ny, k) for k in range(2)]
    c0 = cases[0][0]

    def solver(graph):
        return poisson.MultigridPoisson(nx, ny, c0.hx, c0.hy, use_graph=graph, **opt)

    want, wantz = [], []
    for _, (f, bx, by) in cases:
        s = solver(False)
        p = torch.zeros_like(f)
        it, _, st = s.solve(p, f, bx, by, rtol=1e-8, max_iters=60)
        assert st == 0 and it > 1
        want.append((it, p))
        s.close()
        s = solver(False)
        z = torch.empty_like(f)
        s.precond(z, f, bx, by)
        torch.cuda.synchronize()
        wantz.append(z)
        s.close()
    for graph in (True, False):
        s = solver(graph)
        for rep in range(6):
            _, (f, bx, by) = cases[rep % 2]
            p = torch.zeros_like(f)
            it, _, st = s.solve(p, f, bx, by, rtol=1e-8, max_iters=60)
            assert st == 0 and it == want[rep % 2][0]
            assert torch.equal(p, want[rep % 2][1])
        zs = [torch.empty_like(f) for _ in range(12)]
        for rep, z in enumerate(zs):
            _, (f, bx, by) = cases[rep % 2]
            s.precond(z, f, bx, by)
        torch.cuda.synchronize()
        for rep, z in enumerate(zs):
            assert torch.equal(z, wantz[rep % 2])
        s.close()
