"""The CUDA-core matrix product at the edges of its tiles, its vector widths and its reduction slices.

FP32 throughout: with K terms of unit variance the rounding of a sum is about 6e-8 * sqrt(K) of the largest
result, below 1e-5 for every K here."""
import numpy as np
import pytest

from conftest import rel_err
from oracle import ops as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("trans_a,trans_b", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (1, 10, 2001), (31, 33, 15), (65, 95, 17), (129, 97, 16), (257, 129, 33), (31, 64, 4099), (16, 128, 64),
                                   (1501, 1203, 130)])
def test_matrix_product(m, n, k, trans_a, trans_b, monkeypatch):
    import gpu_util as g
    from mytorch_b200.backends.cuda.env import CudaEnv

    env = CudaEnv.instance()
    rng = np.random.default_rng(m * 7 + n)
    a, b = rng.standard_normal((m, k)).astype(np.float32), rng.standard_normal((k, n)).astype(np.float32)
    at, bt = g.dev(a.T if trans_a else a), g.dev(b.T if trans_b else b)
    bias, c = rng.standard_normal(n).astype(np.float32), g.dev(np.full((m, n), 9.0, np.float32))
    args = (m, n, k, at._native_array, trans_a, bt._native_array, trans_b)
    monkeypatch.setenv("MTB_DISABLE_TC", "1")
    bias_t = g.dev(bias)
    env.lib.gemm_f32(*args, bias_t._native_array, 1, c._native_array, env.stream())
    want = np.maximum(a.astype(np.float64) @ b + bias, 0)
    assert np.max(np.abs(g.host(c) - want)) < 1e-5 * max(np.abs(a.astype(np.float64) @ b).max(), np.abs(want).max(), 1e-3)


@pytest.mark.parametrize("n,cin,cout,h,w,kh,kw,stride,pad", [
    (1, 1, 1, 1, 1, 1, 1, (1, 1), (0, 0)), (2, 3, 5, 9, 7, 3, 3, (1, 1), (1, 1)), (1, 17, 130, 12, 11, 3, 2, (1, 2), (0, 1)),
    (3, 20, 96, 13, 14, 5, 5, (2, 2), (2, 2)), (2, 36, 65, 8, 8, 1, 1, (2, 2), (0, 0)), (2, 6, 10, 23, 21, 2, 3, (5, 5), (1, 2)),
    (9, 48, 82, 15, 17, 3, 3, (1, 1), (1, 1)), (70, 4, 8, 31, 29, 3, 3, (3, 1), (1, 0)), (1, 128, 32, 7, 7, 3, 3, (1, 1), (1, 1))])
def test_convolution(n, cin, cout, h, w, kh, kw, stride, pad, monkeypatch):
    import gpu_util as g

    monkeypatch.setenv("MTB_DISABLE_TC", "1")
    rng = np.random.default_rng(cin * 100 + cout)
    x, wt = rng.standard_normal((n, cin, h, w)).astype(np.float32), rng.standard_normal((cout, cin, kh, kw)).astype(np.float32)
    b = rng.standard_normal(cout).astype(np.float32)
    want = O.conv2d_forward(x, wt, b, stride, pad)
    dy = rng.standard_normal(want.shape).astype(np.float32)
    xt, wtt, bt = g.dev(x, True), g.dev(wt, True), g.dev(b, True)
    y = g.op("conv2d")(xt, wtt, bt, stride, pad)
    dx, dw, db = g.op("conv2d_backward")(g.dev(dy), xt, wtt, bt, stride, pad)
    rdx, rdw, rdb = O.conv2d_backward(dy, x, wt, True, stride, pad)
    for got, ref in ((y, want), (dx, rdx), (dw, rdw), (db, rdb)):
        assert rel_err(g.host(got), ref) < 1e-5
