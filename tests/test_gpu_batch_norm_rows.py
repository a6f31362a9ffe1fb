"""BatchNorm (with ReLU, with addition and ReLU) forward and backward where the rows end inside a group of iterations, a CTA has no group, channels
are no fours and fill several column blocks; against the same formulas in 64 bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,c,h,w", [(1, 64, 3, 5), (7, 64, 3, 3), (2, 1028, 7, 9), (1, 3, 1, 2), (65, 128, 5, 7), (33, 64, 31, 31), (3, 7, 17, 19), (2, 16, 1, 1)])
@pytest.mark.parametrize("form", ["plain", "relu", "add_relu"])
def test_rows_of_any_count(n, c, h, w, form):
    import gpu_util as g

    rng = np.random.default_rng(n + c + w)
    f32 = lambda *s: rng.standard_normal(s).astype(np.float32)
    x, dy, res = f32(n, c, h, w) * 2 + 0.5, f32(n, c, h, w), f32(n, c, h, w)
    gamma, beta, eps = rng.uniform(0.5, 1.5, c).astype(np.float32), f32(c), 1e-3
    col = lambda v: v[None, :, None, None]
    xt, gt, bt, rt, dyt = g.dev(x, True), g.dev(gamma, True), g.dev(beta, True), g.dev(res, True), g.dev(dy)
    if form == "add_relu":
        y, mean, var = g.op("batch_norm2d_add_relu")(xt, rt, gt, bt, eps, True, 0.1, None, None)
        dx, dres, dg, db = g.op("batch_norm2d_add_relu_backward")(dyt, mean, var, xt, rt, gt, bt, eps)
    else:
        kind = "batch_norm2d" if form == "plain" else "batch_norm2d_relu"
        y, mean, var = g.op(kind)(xt, gt, bt, eps, True, 0.1, None, None)
        dx, dg, db = g.op(kind + "_backward")(dyt, mean, var, xt, gt, bt, eps)
    mu, v = x.astype(np.float64).mean((0, 2, 3)), x.astype(np.float64).var((0, 2, 3))
    hat = (x - col(mu)) / np.sqrt(col(v) + eps)
    t = hat * col(gamma) + col(beta) + (res if form == "add_relu" else 0)
    got = g.host(y)
    # a value is the result of a handful of roundings of numbers no larger than what is added up, the statistics of rows x 2^-23 at most
    unit = (np.abs(hat) + 2) * col(gamma) + np.abs(col(beta)) + np.abs(res)
    rounding = (n * h * w + 16) * 2.0 ** -23
    assert (np.abs(got - (t if form == "plain" else np.maximum(t, 0))) <= rounding * unit).all()
    # the ReLU's decision is the forward's own: where it cannot be told from 64 bits it is taken from the stored result
    upstream = dy.astype(np.float64) * (1 if form == "plain" else np.where(np.abs(t) > rounding * unit, t > 0, got > 0))
    m = n * h * w
    s0, s1 = upstream.sum((0, 2, 3)), (upstream * hat).sum((0, 2, 3))
    a0, a1 = np.abs(upstream).sum((0, 2, 3)), np.abs(upstream * hat).sum((0, 2, 3))
    assert (np.abs(g.host(db) - s0) <= rounding * (a0 + 1)).all() and (np.abs(g.host(dg) - s1) <= rounding * (a1 + a0 + 1)).all()
    want = col(gamma) / np.sqrt(col(v) + eps) * (upstream - col(s0) / m - hat * col(s1) / m)
    size = col(gamma) / np.sqrt(col(v) + eps) * (np.abs(upstream) + (col(a0) + 1) / m * (1 + np.abs(hat)) + (np.abs(hat) + 1) * (col(a1) + 1) / m)
    assert (np.abs(g.host(dx) - want) <= 2 * rounding * size).all()
    if form == "add_relu":
        assert np.array_equal(g.host(dres), upstream.astype(np.float32))
