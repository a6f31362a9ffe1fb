"""The backward pass of 3x3 / stride 2 max-pooling that takes four inputs a thread, and the broadcast of an average's gradient."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,c,h,w,pad", [(2, 4, 3, 3, 0), (1, 8, 4, 7, 1), (3, 4, 5, 5, 1), (2, 12, 9, 8, 0), (1, 4, 1, 6, 1), (2, 64, 12, 17, 1), (1, 4, 2, 2, 1)])
def test_max_pool_3x3_stride_2(n, c, h, w, pad):
    import gpu_util as g

    rng = np.random.default_rng(h * w)
    x = rng.integers(-3, 4, (n, c, h, w)).astype(np.float32)  # ties
    args = ((3, 3), (2, 2), (pad, pad))
    xt = g.dev(x)
    y = g.op("max_pool2d")(xt, *args)
    dy = rng.standard_normal(y.shape).astype(np.float32)
    dx, = g.op("max_pool2d_backward")(g.dev(dy), y, xt, *args)
    yh, want = g.host(y), np.zeros((n, c, h + 2 * pad, w + 2 * pad), np.float32)
    xp = np.pad(x, ((0, 0), (0, 0), (pad, pad), (pad, pad)))
    for i in range(y.shape[2]):
        for j in range(y.shape[3]):
            window = np.s_[:, :, 2 * i:2 * i + 3, 2 * j:2 * j + 3]
            assert np.array_equal(yh[:, :, i, j], xp[window].max((2, 3)))
            want[window] += np.where(xp[window] == yh[:, :, i:i + 1, j:j + 1], dy[:, :, i:i + 1, j:j + 1], 0)
    assert np.array_equal(g.host(dx), want[:, :, pad:pad + h, pad:pad + w])  # at most four terms, added in the order of the windows


@pytest.mark.parametrize("n,c,hw,offset", [(1, 1, 1, 0), (3, 5, 7, 0), (2, 8, 49, 0), (128, 512, 16, 0), (5, 260, 1000, 0), (2, 8, 49, 1), (300, 4, 3, 0),
                                           (2, 3, 1000, 0), (1, 4, 5000, 0), (3, 63, 17, 0), (2, 8, 2049, 1), (2, 1, 200000, 0)])
def test_spatial_broadcast(n, c, hw, offset):
    import gpu_util as g
    from mytorch_b200.backends.cuda.env import CudaEnv, CudaMemory

    env = CudaEnv.instance()
    dy = np.random.default_rng(c).standard_normal((n, c)).astype(np.float32)
    src, dst = g.dev(np.concatenate([np.zeros(offset, np.float32), dy.reshape(-1)])), CudaMemory(0, 4 * (n * c * hw + offset))
    env.lib.nhwc_spatial_bcast_f32(src._native_array.ptr + 4 * offset, dst.ptr + 4 * offset, n, c, hw, 1 / hw, env.stream())
    got = dst.read((n * c * hw + offset,), np.float32)[offset:].reshape(n, hw, c)
    assert np.array_equal(got, np.broadcast_to((dy * np.float32(1 / hw))[:, None], (n, hw, c)))
