"""More column tiles than SMs: the epilogues that keep a CTA on one column tile (batch statistics, BatchNorm) have no grid
for that, and the convolution runs without them."""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu


def test_more_column_tiles_than_ctas():
    import gpu_util as g

    rng = np.random.default_rng(0)
    cout, s = 18976, 8  # 297 tiles of 64 columns over 16 pixels
    x, w = rng.standard_normal((1, 32, 32, 32)).astype(np.float32), rng.standard_normal((cout, 32, 1, 1)).astype(np.float32)
    xt, wt = g.dev(x), g.dev(w)
    want = np.einsum("nchw,oc->nohw", x[:, :, ::s, ::s].astype(np.float64), w[:, :, 0, 0])
    y = g.op("conv2d")(xt, wt, None, (s, s), (0, 0), bn_stats=True)
    assert rel_err(g.host(y), want) < 5e-3  # TF32 operands
    vec = lambda lo, hi: g.dev(rng.uniform(lo, hi, cout).astype(np.float32))
    gamma, beta, mean, var = vec(0.5, 1.5), vec(-1, 1), vec(-1, 1), vec(0.5, 2)
    plain = g.op("batch_norm2d")(y, gamma, beta, 1e-5, False, 0.1, mean, var)[0]
    res = g.dev(rng.standard_normal(y.shape).astype(np.float32))
    fused = lambda relu, res=None: g.op("conv2d_batch_norm")(xt, wt, None, (s, s), (0, 0), gamma, beta, mean, var, 1e-5, relu, res)
    assert np.array_equal(g.host(fused(False)), g.host(plain))
    assert np.array_equal(g.host(fused(True)), g.host(g.op("relu")(plain)))
    assert np.array_equal(g.host(fused(True, res)), g.host(g.op("add_relu")(plain, res)))
    trained = g.op("batch_norm2d")(y, gamma, beta, 1e-5, True, 0.1, mean, var)[0]
    yh = g.host(y).astype(np.float64)
    stats = yh.mean((0, 2, 3), keepdims=True), yh.var((0, 2, 3), keepdims=True)
    want = (yh - stats[0]) / np.sqrt(stats[1] + 1e-5) * g.host(gamma)[None, :, None, None] + g.host(beta)[None, :, None, None]
    assert rel_err(g.host(trained), want) < 1e-5
