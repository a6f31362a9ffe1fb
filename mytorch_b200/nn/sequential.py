from mytorch_b200.nn.batch_norm import BatchNorm2d, BatchNormReLU2d, inference_conv_norm
from mytorch_b200.nn.conv import Conv2d
from mytorch_b200.nn.functional.batch_norm import _batch_norm2d_relu, _batch_norm2d_relu_halved
from mytorch_b200.nn.functional.linear import _linear_relu
from mytorch_b200.nn.linear import Linear
from mytorch_b200.nn.max_pool import MaxPool2d
from mytorch_b200.nn.module import Module
from mytorch_b200.nn.relu import ReLU

_NORMS = (BatchNorm2d, BatchNormReLU2d)


def _halves(layer):
    """A 2x2 max-pool of stride 2 that runs the class's own forward."""
    return type(layer) is MaxPool2d and layer.kernel_size == layer.stride == (2, 2) and layer.padding == (0, 0) and not layer._forward_replaced


class Sequential(Module):
    """Layers one after the other.  Neighbours that exist as one operator with the same bits run as one on CUDA: BatchNorm2d +
    ReLU (+ MaxPool2d(2, 2)), Linear + ReLU, and, where nothing is differentiated, Conv2d + BatchNorm2d (+ ReLU (+ MaxPool2d(2, 2)))
    with running statistics.  A step of the MNIST example is 300 library calls of a few microseconds each, so every operator left
    out shows."""

    def __init__(self, *args):
        super().__init__()
        for i, module in enumerate(args):
            self.register_module(str(i), module)

    def forward(self, input):
        layers = list(self._modules.values()) + [None, None, None]
        i = 0
        while layers[i] is not None:
            layer, after = layers[i], layers[i + 1]
            kind, kind_after = type(layer), type(after)
            if kind is Conv2d and kind_after in _NORMS and not (after.training or layer._forward_replaced or after._forward_replaced):
                behind = layers[i + 2]
                relu = kind_after is BatchNorm2d and type(behind) is ReLU and not behind._forward_replaced
                step = 3 if relu else 2
                relu = relu or kind_after is BatchNormReLU2d
                pooled = relu and _halves(layers[i + step])
                y = inference_conv_norm(layer, after, input, relu, None, pooled)
                if y is not None:
                    if pooled:
                        y, pooled = y
                    input = y
                    i += step + pooled
                    continue
            if kind is BatchNorm2d and kind_after is ReLU and input.device.type == "cuda" and not (layer._forward_replaced or after._forward_replaced):
                if _halves(layers[i + 2]):
                    y = _batch_norm2d_relu_halved(input, layer.weight, layer.bias, layer.eps, layer.training, layer.momentum, layer.running_mean,
                                                  layer.running_var)
                    if y is not None:
                        input = y
                        i += 3
                        continue
                input = _batch_norm2d_relu(input, layer.weight, layer.bias, layer.eps, layer.training, layer.momentum, layer.running_mean,
                                           layer.running_var)
                i += 2
                continue
            if (kind is Linear and kind_after is ReLU and input.device.type == "cuda" and len(input.shape) == 2
                    and not (layer._forward_replaced or after._forward_replaced)):
                input = _linear_relu(input, layer.weight, layer.bias)
                i += 2
                continue
            input = layer(input)
            i += 1
        return input
