"""The learned guess and its gradient on every GPU of the process: the kernels' shared-memory limits
are each device's own."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_guess_and_gradient_on_each_device():
    import torch
    from lica_boiling1d_b200 import train_guess
    from lica_boiling1d_b200.unet import LearnedGuess
    rng = np.random.default_rng(3)
    rho = train_guess.problem(rng, 64, 64)[0][None]
    f = rng.standard_normal((1, 64, 64))
    first = None
    for d in range(torch.cuda.device_count()):
        with torch.cuda.device(d):
            t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
            net = LearnedGuess(1, 64, 64, seed=11)
            x = net.guess(t(rho), t(f), 1.0 / 64 ** 2).cpu().numpy()
            g = net.grad(t(rho), t(f), 1.0 / 64 ** 2, t(1.0 / rho))
            net.close()
        assert np.isfinite(x).all() and np.isfinite(g).all() and np.any(g)
        first = first or (x, g)
        np.testing.assert_array_equal(x, first[0])
        np.testing.assert_array_equal(g, first[1])
