"""Convolutions over few input channels (packed into blocks of 32), and 1x1 data gradients that add a tensor in their epilogue.

TF32 products of K terms against FP32 ones: 5e-3 of the largest result, the bound of every TF32 convolution here."""
import numpy as np
import pytest

from conftest import rel_err
from oracle import ops as O

pytestmark = pytest.mark.gpu
TF32_TOL = 5e-3


@pytest.mark.parametrize("n,cin,cout,h,w,kh,kw,stride,pad", [
    (3, 3, 64, 33, 31, 3, 3, (1, 1), (1, 1)), (2, 3, 36, 65, 63, 7, 7, (2, 2), (3, 3)), (4, 2, 32, 40, 37, 4, 4, (3, 2), (0, 2)),
    (2, 4, 64, 32, 48, 2, 4, (1, 1), (0, 0)), (2, 8, 32, 31, 33, 5, 4, (1, 2), (2, 0)), (2, 20, 32, 33, 30, 3, 3, (2, 1), (1, 1)),
    (9, 3, 64, 32, 32, 1, 1, (1, 1), (0, 0)), (3, 3, 30, 32, 32, 3, 3, (1, 1), (1, 1))])
def test_few_input_channels(n, cin, cout, h, w, kh, kw, stride, pad):
    import gpu_util as g

    rng = np.random.default_rng(cin * 31 + kh)
    x, wt = rng.standard_normal((n, cin, h, w)).astype(np.float32), rng.standard_normal((cout, cin, kh, kw)).astype(np.float32)
    b = rng.standard_normal(cout).astype(np.float32)
    want = O.conv2d_forward(x, wt, b, stride, pad)
    dy = rng.standard_normal(want.shape).astype(np.float32)
    xt, wtt, bt = g.dev(x, True), g.dev(wt, True), g.dev(b, True)
    y = g.op("conv2d")(xt, wtt, bt, stride, pad)
    assert rel_err(g.host(y), want) < TF32_TOL
    rdx, rdw, rdb = O.conv2d_backward(dy, x, wt, True, stride, pad)
    for _ in range(2):  # every call packs the input it is given
        dx, dw, db = g.op("conv2d_backward")(g.dev(dy), xt, wtt, bt, stride, pad)
        assert rel_err(g.host(dx), rdx) < TF32_TOL and rel_err(g.host(dw), rdw) < TF32_TOL
        assert rel_err(g.host(db), rdb) < 1e-5  # 32-bit sums of at most 9216 terms
    x2 = rng.standard_normal(x.shape).astype(np.float32)  # a refilled input is packed again
    xt.copy_(g.dev(x2))
    assert rel_err(g.host(g.op("conv2d")(xt, wtt, bt, stride, pad)), O.conv2d_forward(x2, wt, b, stride, pad)) < TF32_TOL


@pytest.mark.parametrize("n,h,w", [(1, 5, 9), (2, 33, 40), (7, 224, 224)])  # a pixel a thread, and several
def test_packed_filter_rows(n, h, w):
    import gpu_util as g
    from mytorch_b200.backends.cuda.env import CudaEnv, CudaMemory

    env = CudaEnv.instance()
    x = np.random.default_rng(w).standard_normal((n, 3, h, w)).astype(np.float32)
    ow = (w + 6 - 7) // 2 + 1
    out = CudaMemory(0, n * h * ow * 32 * 4)
    env.lib.pack_patches_f32(n, 3, h, w, 1, 7, 1, 2, 0, 3, g.dev(x), out.ptr, env.stream())
    padded = np.pad(x.transpose(0, 2, 3, 1), ((0, 0), (0, 0), (3, 3), (0, 0)))
    want = np.zeros((n, h, ow, 32), np.float32)
    for dw in range(7):
        want[..., 3 * dw:3 * dw + 3] = padded[:, :, dw:dw + 2 * ow - 1:2]
    assert np.array_equal(out.read(want.shape, np.float32), want)


@pytest.mark.parametrize("n,cin,cout,hw", [(3, 256, 64, 28), (2, 64, 32, 33), (5, 68, 64, 17), (2, 132, 96, 29)])
def test_pointwise_data_gradient_adds_in_its_epilogue(n, cin, cout, hw):
    import gpu_util as g

    rng = np.random.default_rng(cin)
    x, wt = rng.standard_normal((n, cin, hw, hw)).astype(np.float32), rng.standard_normal((cout, cin, 1, 1)).astype(np.float32)
    dy, add = rng.standard_normal((n, cout, hw, hw)).astype(np.float32), rng.standard_normal(x.shape).astype(np.float32)
    xt, addt = g.dev(x, True), g.dev(add)
    dx, _, _ = g.op("conv2d_backward")(g.dev(dy), xt, g.dev(wt, True), None, (1, 1), (0, 0), accumulate_dx=addt)
    want = O.conv2d_backward(dy, x, wt, False, (1, 1), (0, 0))[0] + add
    assert rel_err(g.host(dx), want) < TF32_TOL
    assert np.array_equal(g.host(addt), add)
