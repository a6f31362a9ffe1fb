"""BatchNorm over more than 64 MB, where the passes walk the tensor together in groups of rows and the backward's sums start at its end: row counts that end inside a
group, one and several column blocks; with gradients of small whole numbers, whose sum is exact, so that a row that is left out or taken twice shows."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(85, 64, 57, 55), (41, 128, 57, 57), (17, 1028, 31, 33)]
EPS = 2.0 ** -24


def _operands(g, n, c, h, w, form):
    assert n * c * h * w * 4 > 64 << 20
    rng = np.random.default_rng(c + h)
    x = rng.standard_normal((n, c, h, w), dtype=np.float32) * 2 + np.float32(0.5)
    res = rng.standard_normal((n, c, h, w), dtype=np.float32) if form == "add_relu" else None
    dy = (rng.integers(1, 4, (n, c, h, w)) * rng.choice([-1, 1], (n, c, h, w))).astype(np.float32)
    return x, res, dy, rng.uniform(0.5, 1.5, c).astype(np.float32), rng.standard_normal(c).astype(np.float32)


@pytest.mark.parametrize("form", ["plain", "relu", "add_relu"])
@pytest.mark.parametrize("shape", SHAPES)
def test_every_row_once(shape, form):
    import gpu_util as g

    x, res, dy, gamma, beta = _operands(g, *shape, form)
    col = lambda v: v[None, :, None, None]
    xt, gt, bt, dyt = g.dev(x, True), g.dev(gamma, True), g.dev(beta, True), g.dev(dy)
    if form == "add_relu":
        rt = g.dev(res, True)
        y, mean, var = g.op("batch_norm2d_add_relu")(xt, rt, gt, bt, 1e-3, True, 0.1, None, None)
        dx, dres, dg, db = g.op("batch_norm2d_add_relu_backward")(dyt, mean, var, xt, rt, gt, bt, 1e-3)
    else:
        kind = "batch_norm2d" if form == "plain" else "batch_norm2d_relu"
        y, mean, var = g.op(kind)(xt, gt, bt, 1e-3, True, 0.1, None, None)
        dx, dg, db = g.op(kind + "_backward")(dyt, mean, var, xt, gt, bt, 1e-3)
    y, mean, var, dx, dg, db = (g.host(t).astype(np.float64) for t in (y, mean, var, dx, dg, db))
    count = x[:, 0].size
    mu, v = x.mean((0, 2, 3), dtype=np.float64), np.square(x - x.mean((0, 2, 3), dtype=np.float64).astype(np.float32)[None, :, None, None]).mean((0, 2, 3), dtype=np.float64)
    assert (np.abs(mean - mu) <= 64 * EPS * (np.abs(mu) + np.sqrt(v))).all() and (np.abs(var - v) <= 64 * EPS * v).all()  # at most 64 roundings in a row
    # from here on with the statistics that the kernel used: a value is a handful of roundings
    hat = (x - col(mean)) / np.sqrt(col(var) + 1e-3)
    t = hat * col(gamma) + col(beta) + (res if res is not None else 0)
    unit = (np.abs(hat) + 1) * col(gamma) + col(np.abs(beta)) + (np.abs(res) if res is not None else 0)
    assert (np.abs(y - (t if form == "plain" else np.maximum(t, 0))) <= 8 * EPS * unit).all()
    # the ReLU's decision is the forward's own; a result of exactly 0 does not tell on which side it fell
    passed = np.ones(x.shape, bool) if form == "plain" else y > 0
    unsure = np.zeros(x.shape, bool) if form == "plain" else (y == 0) & (np.abs(t) <= 8 * EPS * unit)
    up = dy * passed
    unsure = (np.abs(dy) * unsure).sum((0, 2, 3))
    s0, s1, a1 = up.sum((0, 2, 3), dtype=np.float64), (up * hat).sum((0, 2, 3)), np.abs(up * hat).sum((0, 2, 3))
    assert unsure.max() < 50 and (unsure == 0).mean() > 0.5
    assert (np.abs(db - s0) <= unsure).all()  # whole numbers below 2^24: exact
    assert (np.abs(dg - s1) <= 64 * EPS * a1 + 8 * unsure * np.abs(hat).max()).all()
    scale = col(gamma) / np.sqrt(col(var) + 1e-3)
    want, size = scale * (up - col(db) / count - hat * col(dg) / count), scale * (np.abs(dy) + 1 + np.abs(hat))
    wrong = np.abs(dx - want) > 16 * EPS * size
    assert not (wrong & (np.abs(t) > 8 * EPS * unit) if form != "plain" else wrong).any()
    if form == "add_relu":
        dres = g.host(dres)
        assert ((dres == up) | (np.abs(t) <= 8 * EPS * unit)).all()


@pytest.mark.parametrize("shape", SHAPES)
def test_pool_behind_it(shape):
    """The sums' and dx's form that takes the gradient through a 2x2 pool: the bits of the operators one by one."""
    import gpu_util as g

    x, _, _, gamma, beta = _operands(g, *shape, "relu")
    n, c, h, w = shape
    dy = np.random.default_rng(3).standard_normal((n, c, h // 2, w // 2), dtype=np.float32)
    xt, gt, bt, dyt = g.dev(x, True), g.dev(gamma, True), g.dev(beta, True), g.dev(dy)
    y, mean, var = g.op("batch_norm2d_relu_halved")(xt, gt, bt, 1e-3, True, 0.1, None, None)
    got = g.op("batch_norm2d_relu_halved_backward")(dyt, mean, var, xt, gt, bt, 1e-3)
    a, mean0, var0 = g.op("batch_norm2d_relu")(xt, gt, bt, 1e-3, True, 0.1, None, None)
    y0 = g.op("max_pool2d")(a, (2, 2), (2, 2), (0, 0))
    da, = g.op("max_pool2d_backward")(dyt, y0, a, (2, 2), (2, 2), (0, 0))
    want = g.op("batch_norm2d_relu_backward")(da, mean0, var0, xt, gt, bt, 1e-3)
    for u, v in zip((y, mean, var, *got), (y0, mean0, var0, *want)):
        assert np.array_equal(g.host(u), g.host(v))
