"""The column step's tridiagonal lines at the sizes where their pieces, segments and panels
end: whole steps and PRESSURE_CORRECTION against the oracle's serial Thomas algorithm, bit for
bit, in every CTA width; and lines whose pivots leave the range the fast forms take."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _steps(n, props, steps, threads):
    import torch
    from lica_boiling1d_b200.column import Columns
    dev = Columns.film(n, 1.0, [0.31], props).to("cuda")
    status = dev.steps(steps, props, threads=threads)
    torch.cuda.synchronize()
    ref = O.col_init(n, 1.0, 0.31, props)
    for _ in range(steps):
        assert O.col_step(ref, n, 1.0, props) == 0
    assert int(status.abs().max()) == 0
    host = dev.to(None)
    for k, v in ref.items():
        np.testing.assert_array_equal(host.arrays[k][0], v, err_msg=k)


# pieces of 1..17 rows; one, two and three segments of at most 512; panels of 64 and a remainder
@pytest.mark.parametrize("n", [16, 33, 63, 64, 65, 511, 512, 513, 1025])
@pytest.mark.parametrize("threads", [32, 64, 256])
def test_step_at_line_sizes(n, threads):
    from lica_boiling1d_b200.column import ColumnProps
    _steps(n, ColumnProps(denr=1000.0, visr=20.0, tcr=25.0), 2, threads)


@pytest.mark.parametrize("n", [33, 513])
def test_extreme_pivots(n):
    """Diffusion numbers near 1e120: the pivots of LHSPS and LHSW take the plain chain."""
    from lica_boiling1d_b200.column import ColumnProps
    _steps(n, ColumnProps(denr=1000.0, visr=20.0, tcr=25.0, re=1e-125), 1, 64)


# density jumps of 1e12 amplify a pivot's rounding beyond what the seeds allow: the plain chain
@pytest.mark.parametrize("n", [16, 63, 64, 65, 128, 300, 1025])
@pytest.mark.parametrize("ratio", [1e3, 1e12])
def test_pressure_line(n, ratio):
    import torch
    from lica_boiling1d_b200 import routines
    from lica_boiling1d_b200.column import ColumnProps
    rng = np.random.default_rng(n)
    props = ColumnProps(denr=1000.0)
    denf_zi = 1.0 / np.where(rng.random((3, n + 2)) < 0.3, ratio, 1.0 + rng.random((3, n + 2)))
    w, p = rng.standard_normal((3, n + 2)), rng.standard_normal((3, n + 2))
    sfgas = np.where(rng.random((3, 2 * n + 2)) < 0.02, rng.standard_normal((3, 2 * n + 2)), 0.0)
    rw, rp = w.copy(), p.copy()
    for c in range(3):
        O.col_pressure_correction(n, 1.0, props, 1e-5, rw[c], rp[c], denf_zi[c], sfgas[c])
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    gw, gp = t(w), t(p)
    routines.pressure_correction(n, 1.0, props, 1e-5, gw, gp, t(denf_zi), t(sfgas))
    torch.cuda.synchronize()
    np.testing.assert_array_equal(gw.cpu().numpy(), rw)
    np.testing.assert_array_equal(gp.cpu().numpy(), rp)
