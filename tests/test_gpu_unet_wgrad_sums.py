"""Rounding of the weight gradients' sums over many pixels.  Every image's gradient is exact up to its
own few hundred pixels, so a batch's is compared with the FP64 sum of its images' gradients, each
from a context of one 64 x 64 image (one or two pixel tiles a CTA).  The activations are the same
bits in both, so only the sums differ.

The bar: a weight of the batch passes through at most 8 additions in the tensor core (truncated, two
units of 2^-24 each), one addition a tile of the CTA (8192 tiles over 49 CTAs, 168) and 22 over the
CTAs, 206 units of 2^-24 = 1.3e-5 if all of them went one way."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_sums_do_not_drift_with_the_batch():
    import torch
    from lica_boiling1d_b200 import train_guess
    from lica_boiling1d_b200.unet import LearnedGuess
    from oracle import unet_ref as U
    size, distinct, times = 64, 8, 32
    rng = np.random.default_rng(5)
    rho = np.stack([train_guess.problem(rng, size, size)[0] for _ in range(distinct)])
    f = rng.standard_normal((distinct, size, size))
    yy, xx = np.meshgrid(np.arange(size) / size, np.arange(size) / size, indexing="ij")
    gx0 = 1e3 * (1.0 + 0.5 * np.sin(2 * np.pi * xx) * np.cos(2 * np.pi * yy))[None] / rho
    hsq = 1.0 / size ** 2
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    one = LearnedGuess(1, size, size, seed=11)
    ref = sum(one.grad(t(rho[k:k + 1]), t(f[k:k + 1]), hsq, t(gx0[k:k + 1])).astype(np.float64)
              for k in range(distinct)) * times
    one.close()
    net = LearnedGuess(distinct * times, size, size, seed=11)
    g = net.grad(*(t(np.tile(a, (times, 1, 1))) for a in (rho, f)), hsq, t(np.tile(gx0, (times, 1, 1))))
    net.close()
    o = 0
    for l, (c0, c1, co, _) in enumerate(U.LAYERS):
        for name, k in (("W", co * 9 * (c0 + c1)), ("b", co)):
            err = np.linalg.norm(g[o:o + k] - ref[o:o + k]) / np.linalg.norm(ref[o:o + k])
            assert err <= 1.3e-5, (l, name, err)
            o += k
