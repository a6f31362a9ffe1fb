"""Batch statistics from the epilogue of the convolutions by pairs of SMs: means that are large against the spread, and a first image unlike the others;
bounded by the variance, so that a sum of squares that cancels does not pass."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# one to four image rows a tile, a warp with few rows and with many, one accumulator and two taps beside each other
@pytest.mark.parametrize("n,cin,cout,hw", [(40, 64, 64, 32), (20, 64, 128, 56), (60, 128, 128, 16), (33, 128, 96, 28), (150, 96, 64, 9)])
@pytest.mark.parametrize("ratio", [0.0, 10.0, 1000.0])  # mean / standard deviation
@pytest.mark.parametrize("bias", [False, True])
def test_variance_and_mean(n, cin, cout, hw, ratio, bias):
    import gpu_util as g
    from test_gpu_pair_convolutions import _pairs

    assert _pairs(n, cin, cout, hw, hw)[0]
    rng = np.random.default_rng(n + cin + cout)
    x = rng.standard_normal((n, cin, hw, hw)).astype(np.float32)
    w = np.zeros((cout, cin, 3, 3), np.float32)  # the middle tap alone: the same mean at the edges of an image
    w[:, :, 1, 1] = rng.uniform(0.5, 1.0, (cout, cin))
    x += np.float32(ratio * np.sqrt((w[0] ** 2).sum()) / w[0].sum())
    b = g.dev(rng.uniform(-3, 3, cout).astype(np.float32)) if bias else None
    y = g.op("conv2d")(g.dev(x), g.dev(w), b, (1, 1), (1, 1), bn_stats=True)
    assert hasattr(y, "_bn_partials")
    _bounded(g, y)


def test_first_image_unlike_the_others():
    import gpu_util as g

    rng = np.random.default_rng(5)
    x, w = rng.standard_normal((300, 64, 16, 16)).astype(np.float32), rng.standard_normal((64, 64, 3, 3)).astype(np.float32)
    x[0] += 500
    y = g.op("conv2d")(g.dev(x), g.dev(w), None, (1, 1), (1, 1), bn_stats=True)
    assert hasattr(y, "_bn_partials")
    _bounded(g, y)


def _bounded(g, y):
    _, mean, var = g.op("batch_norm2d")(y, None, None, 1e-5, True, 0.1, None, None)
    y64 = g.host(y).astype(np.float64)
    mu, v = y64.mean((0, 2, 3)), y64.var((0, 2, 3))
    eps, large = 2.0 ** -24, np.abs(mu) + np.sqrt(v)
    # A handful of roundings of each value's distance from a running mean and of the sums, at most 64 in a row that all fall the same way; and each partial
    # mean is rounded to `eps` of its size, which the distances between them see once.  Cancelling sums of squares would be off by eps * large^2.
    assert (np.abs(g.host(mean) - mu) <= 8 * eps * large).all()
    assert (np.abs(g.host(var) - v) <= 64 * eps * v + 8 * eps * large * np.sqrt(v)).all()
