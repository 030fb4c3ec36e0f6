"""The weight gradients on the tensor cores at the sizes where their work splits: one image with
fewer pixel tiles than CTAs (two at the coarsest level), and image counts and shapes whose tiles
do not divide among the CTAs.  Every layer's weights and bias against the oracle's hand-written
backward pass, with the bar of the whole network's gradient test (1% relative L2: BF16 rounding
points of the activations and gradients, which the oracle shares, and FP32 against FP64 sums)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,h,w", [(1, 64, 64), (3, 64, 192), (1, 192, 128)])
def test_parameter_gradients_by_layer(n, h, w):
    import torch
    from lica_boiling1d_b200 import train_guess
    from lica_boiling1d_b200.unet import LearnedGuess
    from oracle import unet_ref as U
    rng = np.random.default_rng(h + w)
    rho = np.stack([train_guess.problem(rng, w, h)[0] for _ in range(n)])
    f = rng.standard_normal((n, h, w))
    yy, xx = np.meshgrid(np.arange(h) / h, np.arange(w) / w, indexing="ij")
    gx0 = 1e3 * (1.0 + 0.5 * np.sin(2 * np.pi * xx) * np.cos(2 * np.pi * yy))[None] / rho
    hsq = 1.0 / w ** 2
    net = LearnedGuess(n, h, w, seed=11)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    g = net.grad(t(rho), t(f), hsq, t(gx0))
    again = net.grad(t(rho), t(f), hsq, t(gx0))
    params = net.get_params().astype(np.float64)
    net.close()
    np.testing.assert_array_equal(g, again)     # fixed order of every sum
    _, cache = U.forward(params, rho, f, hsq)
    ref = U.backward(cache, gx0, hsq)
    o = 0
    for l, (c0, c1, co, _) in enumerate(U.LAYERS):
        for name, k in (("W", co * 9 * (c0 + c1)), ("b", co)):
            a, b = g[o:o + k].astype(np.float64), ref[o:o + k]
            assert np.linalg.norm(a - b) <= 1e-2 * np.linalg.norm(b), (l, name, np.linalg.norm(a - b) / np.linalg.norm(b))
            o += k
