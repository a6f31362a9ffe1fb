"""BatchNorm2d + ReLU + max-pool of stride 2 (2x2, or 3x3 with padding 1) as one operator: the very bits of the three, forward (with the tie mask) and backward; odd extents, whose last line
and column no window holds, ties, one to many column blocks, running statistics, gradients off 16 bytes, and the layers of a Sequential."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,c,h,w,training", [(64, 32, 28, 28, True), (5, 128, 7, 7, True), (3, 4, 2, 3, True), (2, 1028, 5, 4, True), (7, 36, 9, 2, False), (1, 64, 33, 31, True)])
@pytest.mark.parametrize("window", [2, 3])
def test_same_bits_as_the_three_operators(n, c, h, w, training, window):
    import gpu_util as g
    from mytorch_b200.backends.cuda.env import CudaMemory, CudaMemoryView

    rng = np.random.default_rng(n + c + h)
    x = np.round(rng.standard_normal((n, c, h, w)) * 4).astype(np.float32) / 4  # ties
    vec = lambda lo, hi: rng.uniform(lo, hi, c).astype(np.float32)
    gamma, beta, rm, rv = vec(0.5, 1.5), vec(-0.5, 0.5), vec(-1, 1), vec(0.5, 2)
    dy = rng.standard_normal((n, c, h // 2, w // 2) if window == 2 else (n, c, (h + 1) // 2, (w + 1) // 2)).astype(np.float32)
    pool = ((window, window), (2, 2), (window - 2, window - 2))

    def stats():
        return g.dev(rm), g.dev(rv)

    xt, gt, bt, dyt = g.dev(x, True), g.dev(gamma, True), g.dev(beta, True), g.dev(dy)
    running = stats()
    y, mean, var = g.op("batch_norm2d_relu_halved")(xt, gt, bt, 1e-5, training, 0.1, *running, window)
    dx, dg, db = g.op("batch_norm2d_relu_halved_backward")(dyt, mean, var, xt, gt, bt, 1e-5, window)
    separate = stats()
    a, mean0, var0 = g.op("batch_norm2d_relu")(xt, gt, bt, 1e-5, training, 0.1, *separate)
    y0 = g.op("max_pool2d")(a, *pool)
    da, = g.op("max_pool2d_backward")(dyt, y0, a, *pool)
    dx0, dg0, db0 = g.op("batch_norm2d_relu_backward")(da, mean0, var0, xt, gt, bt, 1e-5)
    for u, v in zip((y, mean, var, dx, dg, db, *running), (y0, mean0, var0, dx0, dg0, db0, *separate)):
        assert np.array_equal(g.host(u), g.host(v))
    count = y._native_array.nbytes // 4
    assert np.array_equal(y._pool_tiemask.read((count,), np.uint16), y0._pool_tiemask.read((count,), np.uint16))
    block = CudaMemory(0, dyt._native_array.nbytes + 16)
    off = CudaMemoryView(block, 4, dyt._native_array.nbytes, 0)
    off.copy_from(dyt._native_array, off.nbytes)
    dyt._native_array = off
    assert np.array_equal(g.host(g.op("batch_norm2d_relu_halved_backward")(dyt, mean, var, xt, gt, bt, 1e-5, window)[0]), g.host(dx0))


def test_shapes_that_keep_three_operators():
    import gpu_util as g

    for shape in ((2, 6, 8, 8), (2, 8, 1, 8), (2, 8, 8, 1)):
        assert g.op("batch_norm2d_relu_halved")(g.dev(np.ones(shape, np.float32)), None, None, 1e-5, True, 0.1, None, None) is None


def test_layers_of_a_sequential():
    import gpu_util as g
    import mytorch_b200 as mt
    import mytorch_b200.nn as nn

    rng = np.random.default_rng(1)
    xa, target = rng.standard_normal((6, 3, 21, 18)).astype(np.float32), g.dev(rng.integers(0, 4, 6).astype(np.int64))

    class Apart(nn.ReLU):  # not the class's own: every operator by itself
        pass

    results = []
    for relu in (nn.ReLU, Apart):
        mt.manual_seed(2)
        net = nn.Sequential(nn.Conv2d(3, 8, 3, padding=1), nn.BatchNorm2d(8), relu(), nn.MaxPool2d(2, 2), nn.Conv2d(8, 12, 3), nn.BatchNorm2d(12), relu(), nn.MaxPool2d(2, 2))
        head = nn.Linear(12 * 4 * 3, 4)
        net.to(g.DEV), head.to(g.DEV)
        x = g.dev(xa, True)
        loss = nn.functional.cross_entropy(head(net(x).reshape((6, 12 * 4 * 3))), target)
        loss.backward()
        results.append([g.host(loss), g.host(x.grad)] + [g.host(p.grad) for p in (*net.parameters(), *head.parameters())] + [g.host(b) for _, b in net.named_buffers()])
    assert all(np.array_equal(u, v) for u, v in zip(*results))
