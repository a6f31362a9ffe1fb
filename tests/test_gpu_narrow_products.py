"""Products with few outputs and long reductions in tiles of 64 x 32 and 32 x 16: rows, columns and blocks that are not full."""
import numpy as np
import pytest

from oracle import ops as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k,bias", [(64, 128, 9216, True), (33, 40, 2052, True), (32, 16, 4096, False), (100, 70, 3000, True), (300, 128, 1184, True),
                                        (65, 8, 900, False), (97, 17, 132, True),
                                        (64, 128, 288, True), (64, 96, 1024, False), (40, 10, 92, True)])
def test_linear(m, n, k, bias):
    import gpu_util as g

    rng = np.random.default_rng(m + n + k)
    f32 = lambda *s: rng.standard_normal(s).astype(np.float32)
    x, wt, b = f32(m, k), f32(n, k), f32(n)
    rx, rw = O.round_tf32(x).astype(np.float64), O.round_tf32(wt).astype(np.float64)
    xt, wtt, bt = g.dev(x), g.dev(wt), g.dev(b) if bias else None
    y = g.host(g.op("linear")(xt, wtt, bt))
    want, magnitude = rx @ rw.T + (b if bias else 0), abs(rx) @ abs(rw).T + (abs(b) if bias else 0)
    assert (np.abs(y - want) <= (k + 2) * 2.0 ** -23 * magnitude).all()
    # an output's sum does not depend on the tile it is in: the same rows in a product too large for these tiles
    tall = g.host(g.op("linear")(g.dev(np.tile(x, (1 + 8192 // m, 1))), wtt, bt))
    assert np.array_equal(tall[:m], y) and np.array_equal(tall[m:2 * m], y)
