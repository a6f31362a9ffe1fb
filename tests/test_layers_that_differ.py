"""Layers are replaced by one operator only where they are what they look like: a subclass with a forward of its own, or a
forward put on an instance, is called."""
import pytest

import mytorch_b200 as mt
import mytorch_b200.nn as nn
from mytorch_b200.examples.models import _conv_norm


class Renamed(nn.BatchNorm2d):
    """A BatchNorm layer (without a ReLU) under another name."""


class LoudConv(nn.Conv2d):
    calls = 0

    def forward(self, x):
        LoudConv.calls += 1
        return super().forward(x)


@pytest.fixture
def operators(monkeypatch):
    """The names of the operators that are called, in order; their result is their first argument."""
    from mytorch_b200.backends.backend_dispatcher import BackendDispatcher

    called = []

    def stand_in(name):
        def run(x, *args, **kwargs):
            called.append((name, *[a for a in args if isinstance(a, bool)]))
            return (x, None, None) if name.startswith("batch") else x
        return run

    table = BackendDispatcher.instance()._impls["cuda"]
    for name in ("conv2d", "conv2d_batch_norm", "batch_norm2d", "batch_norm2d_relu", "batch_norm2d_add_relu", "relu"):
        monkeypatch.setitem(table, name, stand_in(name))
    return called


def _on_device(*layers):
    from mytorch_b200.tensor import Device, Tensor

    device = Device("cuda:0")
    for layer in layers:
        layer.eval()
        for t in (*layer._parameters.values(), *layer._buffers.values()):
            t.device = device
    return Tensor._on_device((2, 4, 5, 5), mt.float32, device, None)


@pytest.mark.parametrize("make,want", [
    (lambda: (nn.Conv2d(4, 4, 1), nn.BatchNorm2d(4)), [("conv2d_batch_norm", False)]),
    (lambda: (nn.Conv2d(4, 4, 1), nn.BatchNormReLU2d(4)), [("conv2d_batch_norm", True)]),
    (lambda: (nn.Conv2d(4, 4, 1), Renamed(4)), [("conv2d",), ("batch_norm2d", False)]),
    (lambda: (LoudConv(4, 4, 1), nn.BatchNorm2d(4)), [("conv2d",), ("batch_norm2d", False)])])
def test_models_and_sequential(operators, make, want):
    conv, norm = make()
    x = _on_device(conv, norm)
    with mt.no_grad():
        _conv_norm(conv, norm, x)
        assert operators == want
        nn.Sequential(conv, norm)(x)
    assert operators == 2 * want


def test_forward_on_an_instance_is_called(operators):
    seen = []
    for wrapped in range(3):
        layers = nn.Conv2d(4, 4, 1), nn.BatchNorm2d(4), nn.ReLU()
        x = _on_device(*layers)
        plain = layers[wrapped].forward
        layers[wrapped].forward = lambda t, plain=plain: seen.append(plain.__self__) or plain(t)
        with mt.no_grad():
            nn.Sequential(*layers)(x)
            if wrapped < 2:
                _conv_norm(*layers[:2], x)
        assert seen == [layers[wrapped]] * (2 if wrapped < 2 else 1)
        seen.clear()


@pytest.mark.parametrize("name", ["weight", "bias", "running_mean", "running_var"])
def test_vectors_of_another_length_go_to_the_layer_that_checks_them(operators, name):
    conv, norm = nn.Conv2d(4, 4, 1), nn.BatchNorm2d(4)
    other = nn.BatchNorm2d(3)
    x = _on_device(conv, norm, other)
    setattr(norm, name, getattr(other, name))
    with mt.no_grad():
        if name in ("weight", "bias"):
            with pytest.raises(RuntimeError, match="shape"):
                _conv_norm(conv, norm, x)
        else:
            _conv_norm(conv, norm, x)
    assert "conv2d_batch_norm" not in [o[0] for o in operators]


def test_residual_goes_to_the_layer_that_adds_it(operators):
    conv, norm = nn.Conv2d(4, 4, 1), nn.BatchNormAddReLU2d(4)
    x = _on_device(conv, norm)
    with mt.no_grad():
        _conv_norm(conv, norm, x, x)
        assert operators == [("conv2d_batch_norm", True)]
        with pytest.raises(TypeError):
            _conv_norm(conv, norm, x)
