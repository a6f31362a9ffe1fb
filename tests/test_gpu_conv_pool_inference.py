"""Convolution + BatchNorm with running statistics + ReLU + 2x2 max-pool in one launch: the very bits, and the tie masks, of the separate
operators; odd extents (a last line and column that no window holds), rows and columns that end inside a tile, split reductions, single
floats and vectors, and the shapes that keep their own pooling pass."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,cin,cout,h,w,k,stride,pad,takes", [
    (1, 1, 32, 28, 28, 3, 1, 1, True), (1, 32, 128, 14, 14, 3, 1, 1, True), (1, 128, 32, 7, 7, 3, 1, 1, True), (3, 5, 6, 9, 7, 3, 1, 1, True),
    (2, 64, 33, 5, 11, 3, 1, 0, True), (1, 6, 70, 2, 3, 1, 1, 0, True), (4, 3, 17, 21, 20, 5, 2, 2, True), (1, 256, 64, 4, 4, 3, 1, 1, True),
    (64, 32, 128, 14, 14, 3, 1, 1, False), (2, 8, 8, 1, 9, 1, 1, 0, False), (2, 1, 32, 40, 40, 3, 1, 1, False)])
def test_same_bits_as_separate_operators(n, cin, cout, h, w, k, stride, pad, takes):
    import gpu_util as g

    rng = np.random.default_rng(cin + cout + h)
    s, p = (stride, stride), (pad, pad)
    x, wt = g.dev(rng.standard_normal((n, cin, h, w)).astype(np.float32)), g.dev(rng.standard_normal((cout, cin, k, k)).astype(np.float32))
    vec = lambda lo, hi: g.dev(rng.uniform(lo, hi, cout).astype(np.float32))
    bias, gamma, beta, mean, var = vec(-1, 1), vec(0.5, 1.5), vec(-1, 1), vec(-1, 1), vec(0.5, 2)
    fused = g.op("conv2d_batch_norm")
    for b, gm, bt in ((None, gamma, beta), (bias, gamma, beta), (bias, None, None)):
        y = fused(x, wt, b, s, p, gm, bt, mean, var, 1e-5, True, None, True)
        assert (y is not None) == takes
        if not takes:
            return
        want = g.op("max_pool2d")(fused(x, wt, b, s, p, gm, bt, mean, var, 1e-5, True), (2, 2), (2, 2), (0, 0))
        assert np.array_equal(g.host(y), g.host(want))
        masks = [t._pool_tiemask.read((t._native_array.nbytes // 4,), np.uint16) for t in (y, want)]
        assert np.array_equal(*masks)


def test_sequential_takes_it_only_for_the_class_s_own_layers():
    import gpu_util as g
    import mytorch_b200 as mt
    import mytorch_b200.nn as nn

    mt.manual_seed(4)
    x = g.dev(np.random.default_rng(0).standard_normal((2, 3, 9, 9)).astype(np.float32))
    for pool in (nn.MaxPool2d(2, 2), nn.MaxPool2d(2), nn.MaxPool2d(2, 2, 1), nn.MaxPool2d(3, 2)):
        net = nn.Sequential(nn.Conv2d(3, 8, 3, padding=1), nn.BatchNorm2d(8), nn.ReLU(), pool, nn.Conv2d(8, 4, 3, padding=1), nn.BatchNormReLU2d(4), nn.MaxPool2d(2, 2))
        net.to(g.DEV)
        net.eval()
        want = g.host(net(x).detach())  # gradients wanted: layer by layer
        with mt.no_grad():
            assert np.array_equal(g.host(net(x)), want)


# odd extents, where the pixels in windows alone would be priced for another split of the reduction than all pixels
@pytest.mark.parametrize("n,cin,cout,h,w", [(1, 32, 128, 25, 25), (1, 32, 128, 21, 29), (1, 32, 96, 25, 31)])
def test_split_of_the_reduction_follows_from_all_pixels(n, cin, cout, h, w):
    test_same_bits_as_separate_operators(n, cin, cout, h, w, 3, 1, 1, True)


@pytest.mark.parametrize("batch", [1, 2, 16])
def test_one_operator_call_per_convolution(batch, monkeypatch):
    """Whether a convolution's pool goes along is the operator's own decision: no second attempt, with its checks, behind a refused one."""
    import gpu_util as g
    import mytorch_b200 as mt
    import mytorch_b200.nn.batch_norm as B
    from mytorch_b200.examples.mnist import CNN

    mt.manual_seed(7)
    net = CNN()
    net.to(g.DEV)
    net.eval()
    x = g.dev(np.random.default_rng(batch).standard_normal((batch, 1, 28, 28)).astype(np.float32))
    want = g.host(net(x).detach())  # gradients wanted: layer by layer
    calls, dispatch = [], B.dispatch
    monkeypatch.setattr(B, "dispatch", lambda device, name: calls.append(name) or dispatch(device, name))
    with mt.no_grad():
        assert np.array_equal(g.host(net(x)), want)
    assert len(calls) == 3
