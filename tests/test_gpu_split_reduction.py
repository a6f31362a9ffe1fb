"""Convolutions whose reduction is split over a cluster, against the same kernels without the split: whole and ragged tiles of
64, 128 and 256 columns, 2 to 8 units a tile, last units with fewer blocks, strided residue classes, batch statistics."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,cin,cout,h,w,k,stride,pad", [
    (64, 512, 512, 4, 4, 3, 1, 1), (100, 512, 512, 4, 4, 3, 1, 1), (128, 256, 256, 8, 8, 3, 1, 1), (1, 512, 32, 8, 8, 3, 1, 1), (5, 256, 100, 9, 9, 3, 1, 1),
    (3, 288, 256, 11, 7, 3, 1, 1), (64, 256, 512, 8, 8, 3, 2, 1), (128, 256, 512, 8, 8, 3, 2, 1), (9, 2080, 160, 4, 4, 1, 1, 0), (2, 160, 288, 16, 16, 5, 1, 2)])
def test_split_against_unsplit(n, cin, cout, h, w, k, stride, pad, monkeypatch):
    import gpu_util as g

    rng = np.random.default_rng(cin + cout + n)
    x, wt = rng.standard_normal((n, cin, h, w)).astype(np.float32), rng.standard_normal((cout, cin, k, k)).astype(np.float32)
    b = rng.standard_normal(cout).astype(np.float32)
    s, p = (stride, stride), (pad, pad)
    dy = rng.standard_normal((n, cout, (h + 2 * pad - k) // stride + 1, (w + 2 * pad - k) // stride + 1)).astype(np.float32)

    def run(x, wt, b, dy):
        xt, wtt = g.dev(x, True), g.dev(wt)
        y = g.op("conv2d")(xt, wtt, g.dev(b), s, p, bn_stats=True)
        norm = g.op("batch_norm2d")(y, None, None, 1e-5, True, 0.1, None, None)
        return [g.host(t) for t in (y, g.op("conv2d_backward")(g.dev(dy), xt, wtt, None, s, p)[0], *norm[1:])]

    y, dx, mean, var = run(x, wt, b, dy)
    again = run(x, wt, b, dy)
    assert all(np.array_equal(u, v) for u, v in zip((y, dx, mean, var), again))
    monkeypatch.setenv("MTB_DISABLE_SPLITK", "1")
    y0, dx0, _, _ = run(x, wt, b, dy)
    ya, dxa, _, _ = run(abs(x), abs(wt), abs(b), abs(dy))
    # the same products, added in another order: each side's rounding is at most terms x 2^-23 of the sum of magnitudes
    assert (np.abs(y - y0) <= 2 * (cin * k * k + 8) * 2.0 ** -23 * ya).all()
    assert (np.abs(dx - dx0) <= 2 * (cout * k * k + 8) * 2.0 ** -23 * dxa).all()
    y64 = y.astype(np.float64)
    rows = y[:, 0].size
    mag = np.abs(y64).mean((0, 2, 3))
    assert (np.abs(mean - y64.mean((0, 2, 3))) <= rows * 2.0 ** -23 * mag).all()
    # two passes or pivoted sums in FP32: rows x 2^-23 of the second moment about zero bounds both
    assert (np.abs(var - y64.var((0, 2, 3))) <= rows * 2.0 ** -23 * (y64 ** 2).mean((0, 2, 3))).all()
