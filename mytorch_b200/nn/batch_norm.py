"""BatchNorm2d (``mytorch/nn/batch_norm.py:7-135``): affine weight=1 / bias=0, running mean 0 /
running var 1; training mode normalises with batch statistics and blends the *biased* batch
variance into ``running_var``."""
from mytorch_b200.dtype import float32
from mytorch_b200.nn.functional.batch_norm import _batch_norm2d, _batch_norm2d_add_relu, _batch_norm2d_relu
from mytorch_b200.nn.module import Module
from mytorch_b200.nn.parameter import Parameter
from mytorch_b200.ops._common import dispatch, grad_enabled
from mytorch_b200.tensor import Tensor


class BatchNorm2d(Module):
    def __init__(self, num_features, eps=1e-5, momentum=0.1, affine=True, track_running_stats=True, device="cpu", dtype=float32):
        super().__init__()
        self.num_features, self.eps, self.momentum = num_features, eps, momentum
        self.affine, self.track_running_stats = affine, track_running_stats
        if affine:
            self.weight = Parameter(Tensor(shape=(num_features,), dtype=dtype, device=device))
            self.bias = Parameter(Tensor(shape=(num_features,), dtype=dtype, device=device))
        else:
            self.register_parameter("weight", None)
            self.register_parameter("bias", None)
        if track_running_stats:
            self.running_mean = Tensor(shape=(num_features,), dtype=dtype, device=device)
            self.running_var = Tensor(shape=(num_features,), dtype=dtype, device=device)
        else:
            self.register_buffer("running_mean", None)
            self.register_buffer("running_var", None)
        self.reset_parameters()

    def reset_parameters(self):
        if self.track_running_stats:
            self.running_mean.fill_(0)
            self.running_var.fill_(1)
        if self.affine:
            self.weight.fill_(1)
            self.bias.fill_(0)

    def forward(self, x):
        return _batch_norm2d(x, self.weight, self.bias, self.eps, self.training, self.momentum, self.running_mean, self.running_var)


class BatchNormReLU2d(BatchNorm2d):
    """``BatchNorm2d`` immediately followed by ``ReLU`` as one fused operator.  Same parameters,
    buffers and state-dict keys as ``BatchNorm2d``; results equal ``ReLU()(BatchNorm2d(...)(x))``."""

    def forward(self, x):
        return _batch_norm2d_relu(x, self.weight, self.bias, self.eps, self.training, self.momentum, self.running_mean, self.running_var)


class BatchNormAddReLU2d(BatchNorm2d):
    """The tail of a residual block as one fused operator: ``forward(x, residual)`` returns
    ``ReLU()(BatchNorm2d(...)(x) + residual)``.  Same parameters, buffers and state-dict keys as ``BatchNorm2d``."""

    def forward(self, x, residual):
        return _batch_norm2d_add_relu(x, residual, self.weight, self.bias, self.eps, self.training, self.momentum, self.running_mean,
                                      self.running_var)


class BatchNorm1d(BatchNorm2d):
    """BatchNorm over [N, C] or [N, C, L] inputs (``mytorch/nn/batch_norm.py:92-106``): the same per-channel
    statistics over every non-channel dimension, computed by the BatchNorm2d kernels on the input viewed
    as [N, C, L, 1]."""

    def forward(self, x):
        if len(x.shape) not in (2, 3):
            raise RuntimeError(f"BatchNorm1d expects a 2-D or 3-D input, got shape {x.shape}")
        n, c = x.shape[0], x.shape[1]
        length = x.shape[2] if len(x.shape) == 3 else 1
        y = _batch_norm2d(x.reshape((n, c, length, 1)), self.weight, self.bias, self.eps, self.training, self.momentum, self.running_mean,
                          self.running_var)
        return y.reshape(x.shape)


def runs_as_written(layer, *kinds):
    """Whether a layer is one of these classes itself and runs its class's forward: what may be replaced by an operator that does
    the same.  A subclass, or a forward put on the instance (to wrap or trace it), is called."""
    return type(layer) in kinds and "forward" not in layer.__dict__


def inference_conv_norm(conv, norm, x, relu=False, residual=None):
    """``norm(conv(x))``, then optionally ``+ residual``, then optionally ReLU, as one operator where that is possible: a
    convolution and a BatchNorm layer that normalises with its running statistics, on CUDA, with no gradient to record.
    None elsewhere.  Same bits as the separate layers."""
    if norm.training or norm.running_mean is None or x.device.type != "cuda":
        return None
    if grad_enabled(x, conv.weight, conv.bias, norm.weight, norm.bias, residual):
        return None
    weight, device, dtype = conv.weight, x.device, x.dtype
    ok = weight.shape[0] == norm.num_features
    for t in (norm.weight, norm.bias, norm.running_mean, norm.running_var):  # layers' tensors may have been replaced
        ok = ok and (t is None or t.shape == weight.shape[:1])
    for t in (weight, norm.running_mean, norm.running_var, conv.bias, norm.weight, norm.bias, residual):
        ok = ok and (t is None or (t.device is device and t.dtype is dtype))
    if not ok:
        return None  # the separate operators say what is wrong
    affine = norm.weight is not None and norm.bias is not None
    return dispatch(x.device, "conv2d_batch_norm")(x, conv.weight, conv.bias, conv.stride, conv.padding, norm.weight if affine else None,
                                                   norm.bias if affine else None, norm.running_mean, norm.running_var, norm.eps, relu, residual)
