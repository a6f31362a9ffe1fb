"""3x3 convolutions by pairs of SMs: tiles of whole image rows and tiles that start anywhere, image counts that leave the second CTA of a
pair without work, one to four blocks of reduction channels, column tiles that end inside a tile, every epilogue, and what is added on
boundaries of 4, 16 and 32 bytes; against 64-bit sums over operands as the copy engine rounds them."""
import ctypes

import numpy as np
import pytest

from oracle import ops as O

pytestmark = pytest.mark.gpu


def _product(x, w):
    """Products of TF32 operands summed in 64 bits, and the same of the magnitudes."""
    xp = np.pad(x, ((0, 0), (0, 0), (1, 1), (1, 1)))
    h, wd = x.shape[2:]
    return sum(np.einsum("nchw,oc->nohw", xp[:, :, a:a + h, b:b + wd], w[:, :, a, b], optimize=True) for a in range(3) for b in range(3))


@pytest.mark.parametrize("n,cin,cout,h,w", [
    (20, 64, 64, 32, 32), (9, 64, 64, 19, 28), (5, 64, 80, 41, 56), (16, 96, 96, 30, 30), (17, 128, 128, 16, 16), (5, 128, 192, 28, 28),
    (3, 64, 96, 64, 64), (200, 64, 64, 5, 4), (30, 128, 64, 13, 22), (2, 64, 112, 90, 81), (150, 96, 160, 8, 9)])
def test_forward_and_data_gradient(n, cin, cout, h, w):
    import gpu_util as g

    from mytorch_b200.backends.cuda.env import CudaMemory, CudaMemoryView

    rng = np.random.default_rng(n + cin + cout + w)
    f32 = lambda *s: rng.standard_normal(s).astype(np.float32)
    x, wt, b, dy, add = f32(n, cin, h, w), f32(cout, cin, 3, 3), f32(cout), f32(n, cout, h, w), f32(n, cin, h, w)
    rx, rw, rdy = (O.round_tf32(t).astype(np.float64) for t in (x, wt, dy))
    xt, wtt, bt, s, p = g.dev(x, True), g.dev(wt), g.dev(b), (1, 1), (1, 1)

    def check(got, want, magnitude, terms):  # products of TF32 operands are exact in FP32: what is left is the sum's rounding
        assert (np.abs(got - want) <= (terms + 3) * 2.0 ** -23 * magnitude).all()

    y = g.op("conv2d")(xt, wtt, bt, s, p)
    yh = g.host(y)
    check(yh, _product(rx, rw) + b[:, None, None], _product(abs(rx), abs(rw)) + abs(b)[:, None, None], 9 * cin)
    # the same bits with statistics, and in the inference form
    ys = g.op("conv2d")(xt, wtt, bt, s, p, bn_stats=True)
    assert np.array_equal(g.host(ys), yh)
    _, mean, var = g.op("batch_norm2d")(ys, None, None, 1e-5, True, 0.1, None, None)
    y64, rows = yh.astype(np.float64), yh[:, 0].size
    assert (np.abs(g.host(mean) - y64.mean((0, 2, 3))) <= rows * 2.0 ** -23 * np.abs(y64).mean((0, 2, 3))).all()
    assert (np.abs(g.host(var) - y64.var((0, 2, 3))) <= rows * 2.0 ** -23 * (y64 ** 2).mean((0, 2, 3))).all()
    res = g.dev(f32(*yh.shape))
    vec = lambda lo, hi: g.dev(rng.uniform(lo, hi, cout).astype(np.float32))
    gamma, beta, m, v = vec(0.5, 1.5), vec(-1, 1), vec(-1, 1), vec(0.5, 2)
    plain = g.op("batch_norm2d")(y, gamma, beta, 1e-5, False, 0.1, m, v)[0]
    assert np.array_equal(g.host(g.op("conv2d_batch_norm")(xt, wtt, bt, s, p, gamma, beta, m, v, 1e-5, True, res)), g.host(g.op("add_relu")(plain, res)))
    if cout % 32:
        return  # the data gradient then is none of this kernel's
    turned = rw[:, :, ::-1, ::-1].transpose(1, 0, 2, 3)
    dx = g.host(g.op("conv2d_backward")(g.dev(dy), xt, wtt, None, s, p)[0])
    check(dx, _product(rdy, turned), _product(abs(rdy), abs(turned)), 9 * cout)
    for start in (0, 16, 4):  # bytes past a boundary of 32
        at = g.dev(add)
        block = CudaMemory(0, at._native_array.nbytes + 32)
        window = CudaMemoryView(block, start, at._native_array.nbytes, 0)
        window.copy_from(at._native_array, window.nbytes)
        at._native_array = window
        assert np.array_equal(g.host(g.op("conv2d_backward")(g.dev(dy), xt, wtt, None, s, p, accumulate_dx=at)[0]), dx + add)


# 64 -> 64 on rows of 48 pixels: BatchNorm's coefficients leave the row-staged kernel no room for its whole filter, which must not decide between the kernels
@pytest.mark.parametrize("n,h", [(1, 48), (2, 48), (4, 40), (4, 11)])
def test_epilogue_does_not_choose_the_kernel(n, h):
    import gpu_util as g

    rng = np.random.default_rng(n + h)
    f32 = lambda *s: rng.standard_normal(s).astype(np.float32)
    xt, wt, s, p = g.dev(f32(n, 64, h, 48)), g.dev(f32(64, 64, 3, 3)), (1, 1), (1, 1)
    vec = lambda lo, hi: g.dev(rng.uniform(lo, hi, 64).astype(np.float32))
    gamma, beta, m, v = vec(0.5, 1.5), vec(-1, 1), vec(-1, 1), vec(0.5, 2)
    want = g.op("batch_norm2d")(g.op("conv2d")(xt, wt, None, s, p), gamma, beta, 1e-5, False, 0.1, m, v)[0]
    assert np.array_equal(g.host(g.op("conv2d_batch_norm")(xt, wt, None, s, p, gamma, beta, m, v, 1e-5, False)), g.host(want))


def _pairs(*shape):
    """Whether (forward, data gradient) of n, cin, cout, h, w run by pairs of SMs."""
    import gpu_util as g
    import mytorch_b200 as mt
    from mytorch_b200.backends.cuda.ops import _env

    n, cin, cout, h, w = shape
    out = (ctypes.c_int * 7)()
    _env(mt.tensor(np.zeros(4, np.float32), device=g.DEV)).lib.conv2d_pair_choice_f32(n, cin, h, w, 3, 3, 1, 1, 1, 1, cout, out)
    return bool(out[0]), bool(out[3])


@pytest.mark.parametrize("shape", [
    (20, 64, 64, 32, 32), (40, 64, 64, 19, 28), (5, 64, 80, 41, 56), (16, 96, 96, 30, 30), (17, 128, 128, 16, 16), (5, 128, 192, 28, 28),
    (3, 64, 96, 64, 64), (200, 64, 64, 5, 4), (30, 128, 64, 13, 22), (2, 64, 112, 90, 81), (150, 96, 160, 8, 9)])
def test_shapes_above_run_by_pairs(shape):
    cout = shape[2]
    # the data gradient reads blocks of 32 output channels, up to 128 of them
    assert _pairs(*shape) == (True, cout % 32 == 0 and cout <= 128)


def test_whole_rows_of_28_pixels():
    test_forward_and_data_gradient(40, 64, 64, 19, 28)


# input channels that are no blocks of 32: the filter's boxes reach into the next tap and past the last one
@pytest.mark.parametrize("n,cin,cout,h,w", [(20, 80, 64, 32, 32), (12, 112, 128, 28, 28), (30, 80, 96, 13, 22), (9, 208, 64, 40, 41)])
def test_data_gradient_of_odd_blocks(n, cin, cout, h, w):
    import gpu_util as g

    assert _pairs(n, cin, cout, h, w)[1]
    rng = np.random.default_rng(n + cin)
    f32 = lambda *s: rng.standard_normal(s).astype(np.float32)
    x, wt, dy = f32(n, cin, h, w), f32(cout, cin, 3, 3), f32(n, cout, h, w)
    dx = g.host(g.op("conv2d_backward")(g.dev(dy), g.dev(x, True), g.dev(wt), None, (1, 1), (1, 1))[0])
    rdy, turned = O.round_tf32(dy).astype(np.float64), O.round_tf32(wt).astype(np.float64)[:, :, ::-1, ::-1].transpose(1, 0, 2, 3)
    assert (np.abs(dx - _product(rdy, turned)) <= (9 * cout + 3) * 2.0 ** -23 * _product(abs(rdy), abs(turned))).all()
