"""Convolution + BatchNorm in evaluation mode run as one operator only where nothing is differentiated: every operand
that can carry a gradient counts, the biases as much as the weights."""
import numpy as np
import pytest

import mytorch_b200 as mt
import mytorch_b200.nn as nn
from mytorch_b200.nn.batch_norm import inference_conv_norm

NAMES = ("conv.weight", "conv.bias", "norm.weight", "norm.bias")


def _layers(trainable):
    mt.manual_seed(4)
    conv, norm = nn.Conv2d(8, 8, 3, padding=1), nn.BatchNorm2d(8)
    norm.eval()
    params = dict(zip(NAMES, (conv.weight, conv.bias, norm.weight, norm.bias)))
    for name, p in params.items():
        p.requires_grad = name in trainable
    return conv, norm, params


@pytest.mark.parametrize("trainable", [(), *((name,) for name in NAMES)])
def test_one_operator_only_without_gradients(trainable, monkeypatch):
    from mytorch_b200.backends.backend_dispatcher import BackendDispatcher
    from mytorch_b200.tensor import Device, Tensor

    fused = []
    monkeypatch.setitem(BackendDispatcher.instance()._impls["cuda"], "conv2d_batch_norm", lambda *a: fused.append(a) or a[0])
    device = Device("cuda:0")
    conv, norm, params = _layers(trainable)
    for t in (*params.values(), norm.running_mean, norm.running_var):
        t.device = device
    x = Tensor._on_device((2, 8, 4, 4), mt.float32, device, None)
    assert (inference_conv_norm(conv, norm, x) is None) == bool(trainable) and len(fused) == (not trainable)
    with mt.no_grad():
        assert inference_conv_norm(conv, norm, x) is not None
    x.requires_grad = True
    assert inference_conv_norm(conv, norm, x) is None


@pytest.mark.gpu
@pytest.mark.parametrize("trainable", [("conv.bias",), ("norm.bias",), ("conv.bias", "norm.bias")])
def test_biases_train_behind_frozen_weights(trainable):
    import gpu_util as g

    rng = np.random.default_rng(6)
    x = rng.standard_normal((4, 8, 6, 6)).astype(np.float32)
    conv, norm, _ = _layers(trainable)
    net = nn.Sequential(conv, norm, nn.ReLU())
    net.to(g.DEV)
    conv, norm = net._modules["0"], net._modules["1"]
    params = dict(zip(NAMES, (conv.weight, conv.bias, norm.weight, norm.bias)))
    for name, p in params.items():
        p.requires_grad = name in trainable
    net.eval()
    y = net(g.dev(x))
    y.sum().backward()
    # BatchNorm's backward is that of batch statistics in either mode, as in the reference; fresh statistics, gamma = 1, beta = 0
    scale = 1 / np.sqrt(1 + 1e-5)
    with mt.no_grad():
        normal = g.host(conv(g.dev(x))).astype(np.float64) * scale
    passed = (normal >= 0).astype(np.float64)
    axes = (0, 2, 3)
    mean = lambda a: a.mean(axes, keepdims=True)
    want = {"conv.bias": ((passed - mean(passed) - normal * mean(passed * normal)) * scale).sum(axes), "norm.bias": passed.sum(axes)}
    for name, p in params.items():
        assert (p.grad is None) == (name not in trainable)
        if name in trainable:
            np.testing.assert_allclose(g.host(p.grad), want[name], rtol=1e-5, atol=1e-4)  # sums of 144 terms of about 1, 32-bit
