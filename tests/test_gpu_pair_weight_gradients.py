"""Weight gradients of 64 channels by pairs of SMs: image rows that are a multiple of 1, 2, 4 and 8 positions, last stages that end behind the last
image, ranges of one stage and of odd and even counts, output channels that end inside a block; against 64-bit sums over operands as
the copy engine rounds them."""
import ctypes

import numpy as np
import pytest

from oracle import ops as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,cout,h,w", [(70, 64, 32, 32), (131, 64, 32, 32), (24, 64, 56, 56), (40, 36, 45, 38), (100, 48, 29, 27), (9, 64, 100, 110), (33, 60, 50, 46),
                                        (20, 64, 70, 62), (1000, 64, 7, 9)])
def test_weight_gradient(n, cout, h, w):
    import gpu_util as g

    rng = np.random.default_rng(n + cout + w)
    x, dy = rng.standard_normal((n, 64, h, w)).astype(np.float32), rng.standard_normal((n, cout, h, w)).astype(np.float32)
    wt = g.dev(rng.standard_normal((cout, 64, 3, 3)).astype(np.float32), True)
    xt, dyt = g.dev(x), g.dev(dy)
    dw = g.host(g.op("conv2d_backward")(dyt, xt, wt, None, (1, 1), (1, 1))[1])
    assert np.array_equal(dw, g.host(g.op("conv2d_backward")(dyt, xt, wt, None, (1, 1), (1, 1))[1]))

    def sums(x, dy):
        xp = np.pad(x, ((0, 0), (0, 0), (1, 1), (1, 1)))
        d = dy.transpose(1, 0, 2, 3).reshape(cout, -1)
        return np.stack([np.stack([d @ xp[:, :, a:a + h, b:b + w].transpose(0, 2, 3, 1).reshape(-1, 64) for b in range(3)], -1) for a in range(3)], -2)

    rx, rdy = O.round_tf32(x).astype(np.float64), O.round_tf32(dy).astype(np.float64)
    # products of TF32 operands are exact in FP32; a sum loses at most its number of terms x 2^-23 of the sum of magnitudes
    assert (np.abs(dw - sums(rx, rdy)) <= n * h * w * 2.0 ** -23 * sums(abs(rx), abs(rdy))).all()
    assert np.linalg.norm(dw - sums(rx, rdy)) <= 5e-5 * np.linalg.norm(dw)


@pytest.mark.parametrize("n,cout,h,w", [(70, 64, 32, 32), (131, 64, 32, 32), (24, 64, 56, 56), (40, 36, 45, 38), (100, 48, 29, 27), (9, 64, 100, 110), (33, 60, 50, 46),
                                        (20, 64, 70, 62), (1000, 64, 7, 9)])
def test_shapes_above_run_by_pairs(n, cout, h, w):
    import gpu_util as g
    import mytorch_b200 as mt
    from mytorch_b200.backends.cuda.ops import _env

    out = (ctypes.c_int * 7)()
    _env(mt.tensor(np.zeros(4, np.float32), device=g.DEV)).lib.conv2d_pair_choice_f32(n, 64, h, w, 3, 3, 1, 1, 1, 1, cout, out)
    assert out[6] == 1
