"""Convolution + BatchNorm with running statistics (+ addition) (+ ReLU) in one launch: the very bits of the separate operators.

The shapes reach every kernel that carries it: row-staged with resident and streamed filters, one and two tiles per
stage, im2col with whole and ragged column tiles, split reductions, CUDA-core tiles, packed stems."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,cin,cout,h,w,k,stride,pad", [
    (70, 64, 64, 32, 32, 3, 1, 1), (40, 128, 128, 16, 16, 3, 1, 1), (100, 64, 128, 32, 32, 3, 1, 1), (3, 64, 256, 40, 40, 1, 1, 0),
    (9, 64, 72, 17, 19, 3, 2, 1), (20, 256, 100, 8, 8, 3, 1, 1), (16, 512, 512, 4, 4, 3, 1, 1), (4, 32, 36, 33, 31, 5, 1, 2), (2, 3, 64, 64, 64, 7, 2, 3),
    (1, 1, 32, 28, 28, 3, 1, 1), (1, 32, 128, 14, 14, 3, 1, 1), (3, 5, 6, 9, 7, 3, 1, 1), (40, 20, 130, 30, 30, 3, 1, 1)])
def test_same_bits_as_separate_operators(n, cin, cout, h, w, k, stride, pad):
    import gpu_util as g

    rng = np.random.default_rng(cin + cout)
    x, wt = g.dev(rng.standard_normal((n, cin, h, w)).astype(np.float32)), g.dev(rng.standard_normal((cout, cin, k, k)).astype(np.float32))
    vec = lambda lo, hi: g.dev(rng.uniform(lo, hi, cout).astype(np.float32))
    bias, gamma, beta, mean, var = vec(-1, 1), vec(0.5, 1.5), vec(-1, 1), vec(-1, 1), vec(0.5, 2)
    conv = lambda b: g.op("conv2d")(x, wt, b, (stride, stride), (pad, pad))
    fused = lambda b, gm, bt, relu, res=None: g.op("conv2d_batch_norm")(x, wt, b, (stride, stride), (pad, pad), gm, bt, mean, var, 1e-5, relu, res)
    res = g.dev(rng.standard_normal(conv(None).shape).astype(np.float32))
    for b, gm, bt in ((None, gamma, beta), (bias, gamma, beta), (None, None, None)):
        y = conv(b)
        plain = g.op("batch_norm2d")(y, gm, bt, 1e-5, False, 0.1, mean, var)[0]
        assert np.array_equal(g.host(fused(b, gm, bt, False)), g.host(plain))
        assert np.array_equal(g.host(fused(b, gm, bt, True)), g.host(g.op("relu")(plain)))
        assert np.array_equal(g.host(fused(b, gm, bt, True, res)), g.host(g.op("add_relu")(plain, res)))


def test_models_evaluate_to_the_bits_of_their_layers():
    import gpu_util as g
    import mytorch_b200 as mt
    from mytorch_b200.examples.mnist import CNN
    from mytorch_b200.examples.models import ResNet18Cifar

    rng = np.random.default_rng(3)
    for make, shape in ((CNN, (5, 1, 28, 28)), (lambda: ResNet18Cifar((32, 32, 64, 64)), (6, 3, 32, 32))):
        mt.manual_seed(5)
        net = make()
        net.to(g.DEV)
        x = g.dev(rng.standard_normal(shape).astype(np.float32))
        net(x)  # training mode: the running statistics move
        net.eval()
        want = g.host(net(x).detach())  # gradients wanted: layer by layer
        with mt.no_grad():
            assert np.array_equal(g.host(net(x)), want)
