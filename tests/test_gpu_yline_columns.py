"""The y-line half-sweep's columns at the edges of its kernels: rows that do not fill its blocks of
eight, and columns too long for a CTA's shared memory -- one V-cycle against the oracle's, bit
for bit."""
import numpy as np
import pytest

from oracle import grid as OG
from oracle import oracle as O

pytestmark = pytest.mark.gpu


# 96 x 160: levels of 80, 40, 20, 10, 5 rows; 512 x 4352: level 0 keeps one thread per column
@pytest.mark.parametrize("nx,ny,nlevels", [(96, 160, 2), (512, 4352, 6)])
def test_yline_columns_bitwise(nx, ny, nlevels):
    import torch
    from lica_boiling1d_b200 import poisson as PP
    y = OG.section(3, 0.0, 1.0, 1, ny + 1, 2.0, 1.0, np.zeros(ny + 1))
    rng = np.random.default_rng(nx)
    rho = np.where(rng.random((ny, nx)) < 0.2, 1.0, 40.0)
    bx = 1.0 / (0.5 * (rho + np.roll(rho, 1, axis=1)))
    by = np.ones((ny + 1, nx))
    by[1:ny] = 1.0 / (0.5 * (rho[1:] + rho[:-1]))
    by[0], by[ny] = 1.0 / rho[0], 1.0 / rho[ny - 1]
    bxs, bys, fs = PP.stretched_system(y, bx, by, rng.standard_normal((ny, nx)))
    ref = O.mg_precond(fs, bxs, bys, 1.0 / nx, 1.0, nlevels=nlevels, ncoarse=1, sym=13)
    mg = PP.MultigridPoisson(nx, ny, 1.0 / nx, 1.0, nlevels=nlevels, ncoarse=1, smoother="yline")
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    z = torch.empty((ny, nx), dtype=torch.float64, device="cuda")
    mg.precond(z, t(fs), t(bxs), t(bys))
    mg.close()
    np.testing.assert_array_equal(z.cpu().numpy(), ref)


# a smoothing's first half-sweep from zero, from the coarse correction and from the iterate: the second
# coarse cycle starts from the first's result; one, two and three sweeps
@pytest.mark.parametrize("nx,ny,nu", [(64, 64, 1), (32, 96, 2), (96, 64, 3)])
def test_yline_start_of_smoothing(nx, ny, nu):
    import torch
    from lica_boiling1d_b200 import poisson as PP
    rng = np.random.default_rng(nx + nu)
    rho = np.where(rng.random((ny, nx)) < 0.2, 1.0, 40.0)
    bx = 1.0 / (0.5 * (rho + np.roll(rho, 1, axis=1)))
    by = np.ones((ny + 1, nx))
    by[1:ny] = 1.0 / (0.5 * (rho[1:] + rho[:-1]))
    by[0], by[ny] = 1.0 / rho[0], 1.0 / rho[ny - 1]
    f = rng.standard_normal((ny, nx))
    ref = O.mg_precond(f, bx, by, 1.0 / nx, 1.0 / ny, nlevels=2, nu1=nu, nu2=nu, ncoarse=2, sym=13)
    mg = PP.MultigridPoisson(nx, ny, 1.0 / nx, 1.0 / ny, nlevels=2, nu1=nu, nu2=nu, ncoarse=2, smoother="yline")
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    z = torch.full((ny, nx), float("nan"), dtype=torch.float64, device="cuda")
    for _ in range(2):
        mg.precond(z, t(f), t(bx), t(by))
    mg.close()
    np.testing.assert_array_equal(z.cpu().numpy(), ref)


# where the levels of the one-CTA kernel begin: above the coarsest outer level, at it, inside the inner
# cycle (its coarsest outer level too large), and odd row counts below it
@pytest.mark.parametrize("nx,ny,nlevels,ncoarse", [(128, 64, 5, 2), (64, 64, 2, 1), (96, 128, 2, 2), (32, 160, 4, 1)])
def test_yline_coarse_levels(nx, ny, nlevels, ncoarse):
    import torch
    from lica_boiling1d_b200 import poisson as PP
    rng = np.random.default_rng(nx * ny + nlevels)
    bx, by, f = rng.uniform(0.1, 40.0, (ny, nx)), rng.uniform(0.1, 40.0, (ny + 1, nx)), rng.standard_normal((ny, nx))
    ref = O.mg_precond(f, bx, by, 1.0 / nx, 0.2 / ny, nlevels=nlevels, ncoarse=ncoarse, sym=13)
    mg = PP.MultigridPoisson(nx, ny, 1.0 / nx, 0.2 / ny, nlevels=nlevels, ncoarse=ncoarse, smoother="yline")
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    z = torch.empty((ny, nx), dtype=torch.float64, device="cuda")
    mg.precond(z, t(f), t(bx), t(by))
    mg.close()
    np.testing.assert_array_equal(z.cpu().numpy(), ref)
