"""Short reductions whose results (and what is added to them) move through shared memory in blocks of 32 x 32: rows and
columns that end inside a tile, a block or a warp's share, several tiles a CTA, against the oracle on operands as the copy
engine rounds them, and statistics against the stored results."""
import numpy as np
import pytest

from oracle import ops as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,cin,cout,h,w", [
    (1, 32, 64, 32, 33), (3, 64, 96, 19, 23), (1, 32, 36, 45, 31), (2, 256, 260, 17, 9), (5, 96, 320, 41, 37), (9, 64, 132, 64, 61), (40, 64, 256, 33, 31),
    # either side of where results are stored from registers: few and many reduction blocks, a wave of tiles and more
    (40, 96, 64, 33, 31), (40, 64, 512, 33, 31), (20, 256, 480, 31, 33), (20, 256, 512, 31, 33), (2, 512, 992, 17, 15), (2, 512, 1024, 17, 15)])
def test_pointwise_convolution(n, cin, cout, h, w):
    import gpu_util as g

    rng = np.random.default_rng(n + cin + cout)
    f32 = lambda *s: rng.standard_normal(s).astype(np.float32)
    x, wt, b, dy, add = f32(n, cin, h, w), f32(cout, cin, 1, 1), f32(cout), f32(n, cout, h, w), f32(n, cin, h, w)
    xt, wtt, bt = g.dev(x, True), g.dev(wt), g.dev(b)
    s, p = (1, 1), (0, 0)
    y = g.op("conv2d")(xt, wtt, bt, s, p, bn_stats=True)
    norm = g.op("batch_norm2d")(y, None, None, 1e-5, True, 0.1, None, None)
    rx, rw, rdy = (O.round_tf32(t).astype(np.float64) for t in (x, wt[:, :, 0, 0], dy))

    def check(got, want, magnitude, terms):  # products of TF32 operands are exact in FP32: what is left is the sum's rounding
        assert (np.abs(got - want) <= (terms + 2) * 2.0 ** -23 * magnitude).all()

    yh = g.host(y)
    check(yh, np.einsum("nchw,oc->nohw", rx, rw) + b[None, :, None, None],
          np.einsum("nchw,oc->nohw", abs(rx), abs(rw)) + abs(b)[None, :, None, None], cin)
    assert np.array_equal(yh, g.host(g.op("conv2d")(xt, wtt, bt, s, p)))
    y64 = yh.astype(np.float64)
    rows = yh[:, 0].size
    assert (np.abs(g.host(norm[1]) - y64.mean((0, 2, 3))) <= rows * 2.0 ** -23 * np.abs(y64).mean((0, 2, 3))).all()
    assert (np.abs(g.host(norm[2]) - y64.var((0, 2, 3))) <= rows * 2.0 ** -23 * (y64 ** 2).mean((0, 2, 3))).all()
    if cout % 32:
        return  # the data gradient then is none of this kernel's
    want, magnitude = np.einsum("nohw,oc->nchw", rdy, rw), np.einsum("nohw,oc->nchw", abs(rdy), abs(rw))
    check(g.host(g.op("conv2d_backward")(g.dev(dy), xt, wtt, None, s, p)[0]), want, magnitude, cout)
    plus = g.op("conv2d_backward")(g.dev(dy), xt, wtt, None, s, p, accumulate_dx=g.dev(add))[0]
    check(g.host(plus), want + add, magnitude + abs(add), cout)


@pytest.mark.parametrize("m,n,k,bias", [(128, 64, 32, True), (129, 100, 64, True), (1000, 500, 92, False), (4099, 260, 480, True), (70, 64, 500, True)])
def test_linear(m, n, k, bias):
    import gpu_util as g

    rng = np.random.default_rng(m + n + k)
    f32 = lambda *s: rng.standard_normal(s).astype(np.float32)
    x, wt, b = f32(m, k), f32(n, k), f32(n)
    rx, rw = O.round_tf32(x).astype(np.float64), O.round_tf32(wt).astype(np.float64)
    y = g.host(g.op("linear")(g.dev(x), g.dev(wt), g.dev(b) if bias else None))
    want, magnitude = rx @ rw.T + (b if bias else 0), abs(rx) @ abs(rw).T + (abs(b) if bias else 0)
    assert (np.abs(y - want) <= (k + 2) * 2.0 ** -23 * magnitude).all()
