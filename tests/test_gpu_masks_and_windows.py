"""The ReLU mask that BatchNorm + addition + ReLU hands to its backward, the vectorised pooling windows and the packed stems, at
ragged sizes: bits equal to the forms they replace (masks, windows), exact copies (packing)."""
import numpy as np
import pytest

from oracle import ops as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,c,h,w", [(1, 4, 1, 1), (3, 36, 5, 7), (2, 64, 16, 16), (5, 260, 9, 3), (1, 2048, 7, 7), (2, 6, 5, 5)])
def test_backward_from_the_mask_equals_backward_from_the_added_tensor(n, c, h, w):
    import gpu_util as g
    import mytorch_b200 as mt

    rng = np.random.default_rng(c)
    arr = lambda *s: g.dev(rng.standard_normal(s).astype(np.float32), True)
    x, res, dy, gamma, beta = arr(n, c, h, w), arr(n, c, h, w), arr(n, c, h, w), arr(c), arr(c)
    with_mask = g.op("batch_norm2d_add_relu")(x, res, gamma, beta, 1e-5, True, 0.1, None, None)
    with mt.no_grad():
        without = g.op("batch_norm2d_add_relu")(x, res, gamma, beta, 1e-5, True, 0.1, None, None)
    assert hasattr(with_mask[1], "_relu_mask") == (c % 4 == 0) and not hasattr(without[1], "_relu_mask")
    for a, b in zip(with_mask, without):
        assert np.array_equal(g.host(a), g.host(b))
    got = g.op("batch_norm2d_add_relu_backward")(dy, with_mask[1], with_mask[2], x, res, gamma, beta, 1e-5)
    want = g.op("batch_norm2d_add_relu_backward")(dy, without[1], without[2], x, res, gamma, beta, 1e-5)
    for a, b in zip(got, want):
        assert np.array_equal(g.host(a), g.host(b))


@pytest.mark.parametrize("k,s,p", [(3, 2, 1), (3, 2, 0), (3, 1, 1), (3, 1, 0), (2, 2, 0), (2, 2, 1)])
@pytest.mark.parametrize("n,c,h,w", [(2, 4, 3, 3), (3, 12, 7, 10), (1, 64, 23, 17), (2, 8, 4, 31)])
def test_pooling_windows(n, c, h, w, k, s, p):
    import gpu_util as g
    from mytorch_b200.backends.cuda.ops import max_pool2d_argmax

    rng = np.random.default_rng(h * w)
    x = rng.integers(-2, 3, (n, c, h, w)).astype(np.float32)  # many ties
    xt = g.dev(x, True)
    y = g.op("max_pool2d")(xt, (k, k), (s, s), (p, p))
    want = O.max_pool2d_forward(x, k, s, p)
    assert np.array_equal(g.host(y), want)
    assert np.array_equal(max_pool2d_argmax(y), O.max_pool2d_argmax(x, k, s, p).astype(np.uint8))
    dy = rng.integers(-4, 5, want.shape).astype(np.float32)  # small whole numbers: sums are exact
    (dx,) = g.op("max_pool2d_backward")(g.dev(dy), y, xt, (k, k), (s, s), (p, p))
    assert np.array_equal(g.host(dx), O.max_pool2d_backward(dy, want, x, k, s, p))


@pytest.mark.parametrize("n,c,h,w,kh,kw,sh,sw,ph,pw", [(2, 3, 9, 7, 3, 3, 1, 1, 1, 1), (1, 3, 20, 13, 1, 7, 1, 2, 0, 3), (3, 32, 4, 5, 1, 1, 2, 1, 0, 0),
                                                       (2, 5, 6, 6, 2, 3, 2, 3, 1, 2)])
def test_packed_patches(n, c, h, w, kh, kw, sh, sw, ph, pw):
    import gpu_util as g
    from mytorch_b200.backends.cuda.env import CudaEnv, CudaMemory

    env = CudaEnv.instance()
    x = np.random.default_rng(c).standard_normal((n, c, h, w)).astype(np.float32)
    oh, ow = (h + 2 * ph - kh) // sh + 1, (w + 2 * pw - kw) // sw + 1
    xt, out = g.dev(x), CudaMemory(0, n * oh * ow * 128)
    env.lib.pack_patches_f32(n, c, h, w, kh, kw, sh, sw, ph, pw, xt._native_array, out, env.stream())
    padded = np.pad(x, ((0, 0), (0, 0), (ph, ph), (pw, pw)))
    want = np.zeros((n, oh, ow, 32), np.float32)
    for a in range(kh):
        for b in range(kw):
            at = (a * kw + b) * c
            want[..., at:at + c] = padded[:, :, a:a + sh * oh:sh, b:b + sw * ow:sw][:, :, :oh, :ow].transpose(0, 2, 3, 1)
    assert np.array_equal(out.read((n, oh, ow, 32), np.float32), want)
