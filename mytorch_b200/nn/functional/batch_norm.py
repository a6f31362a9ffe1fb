"""Fused BatchNorm2d front-end (``mytorch/nn/functional/batch_norm.py:8-51``)."""
from mytorch_b200.ops._common import dispatch, record, tracker
from mytorch_b200.tensor import Tensor


def _batch_norm2d(input: Tensor, weight, bias, eps, training, momentum, running_mean, running_var):
    requires_grad = input.requires_grad
    channels = input.shape[1]
    if weight is not None and bias is not None:
        ok = (input.dtype == weight.dtype == bias.dtype and input.device == weight.device == bias.device
              and weight.shape == (channels,) and bias.shape == (channels,))
        if not ok:
            raise RuntimeError("batch_norm2d shape, dtype or device mismatch")
        requires_grad = requires_grad or weight.requires_grad or bias.requires_grad
    out, mean, var = dispatch(input.device, "batch_norm2d")(input, weight, bias, eps, training, momentum, running_mean, running_var)
    out.requires_grad = requires_grad and not tracker.no_grad
    return record("batch_norm2d", [input, weight, bias, eps], out, [mean, var])


@tracker.register_backward_function("batch_norm2d")
def _batch_norm2d_backward(output_grad, mean, var, input, weight, bias, eps):
    return dispatch(input.device, "batch_norm2d_backward")(output_grad, mean, var, input, weight, bias, eps)


def _batch_norm2d_relu(input: Tensor, weight, bias, eps, training, momentum, running_mean, running_var):
    """relu(batch_norm2d(x)) as one operator: the normalise pass applies max(0, .) before it stores,
    and backward re-derives the ReLU mask from x, so the intermediate is never written or read.
    Same arithmetic as ``BatchNorm2d`` followed by ``ReLU`` (``mytorch/nn/batch_norm.py:123-135``,
    ``mytorch/nn/relu.py:5-10``); the reference runs them as two operators."""
    requires_grad = input.requires_grad
    channels = input.shape[1]
    if weight is not None and bias is not None:
        ok = (input.dtype == weight.dtype == bias.dtype and input.device == weight.device == bias.device
              and weight.shape == (channels,) and bias.shape == (channels,))
        if not ok:
            raise RuntimeError("batch_norm2d shape, dtype or device mismatch")
        requires_grad = requires_grad or weight.requires_grad or bias.requires_grad
    out, mean, var = dispatch(input.device, "batch_norm2d_relu")(input, weight, bias, eps, training, momentum, running_mean, running_var)
    out.requires_grad = requires_grad and not tracker.no_grad
    return record("batch_norm2d_relu", [input, weight, bias, eps], out, [mean, var])


@tracker.register_backward_function("batch_norm2d_relu")
def _batch_norm2d_relu_backward(output_grad, mean, var, input, weight, bias, eps):
    return dispatch(input.device, "batch_norm2d_relu_backward")(output_grad, mean, var, input, weight, bias, eps)


def _batch_norm2d_relu_halved(input: Tensor, weight, bias, eps, training, momentum, running_mean, running_var, window=2):
    """max_pool2d(relu(batch_norm2d(x)), 2, 2) (``window`` 3: max_pool2d(.., 3, 2, 1)) as one operator on CUDA, None where it does not exist.  The reference runs three
    (``mytorch/nn/batch_norm.py:123-135``, ``mytorch/nn/relu.py:5-10``, ``mytorch/nn/max_pool.py:5-21``); here neither the normalised
    tensor nor its gradient is stored."""
    requires_grad = input.requires_grad
    channels = input.shape[1]
    if channels % 4:
        return None
    if weight is not None and bias is not None:
        ok = (input.dtype == weight.dtype == bias.dtype and input.device == weight.device == bias.device
              and weight.shape == (channels,) and bias.shape == (channels,))
        if not ok:
            return None  # the separate operators say what is wrong
        requires_grad = requires_grad or weight.requires_grad or bias.requires_grad
    made = dispatch(input.device, "batch_norm2d_relu_halved")(input, weight, bias, eps, training, momentum, running_mean, running_var, window)
    if made is None:
        return None
    out, mean, var = made
    out.requires_grad = requires_grad and not tracker.no_grad
    return record("batch_norm2d_relu_halved", [input, weight, bias, eps, window], out, [mean, var])


@tracker.register_backward_function("batch_norm2d_relu_halved")
def _batch_norm2d_relu_halved_backward(output_grad, mean, var, input, weight, bias, eps, window):
    return dispatch(input.device, "batch_norm2d_relu_halved_backward")(output_grad, mean, var, input, weight, bias, eps, window)


def _batch_norm2d_add_relu(input: Tensor, residual: Tensor, weight, bias, eps, training, momentum, running_mean, running_var):
    """relu(batch_norm2d(x) + residual) as one operator: the tail of a residual block.  The reference runs
    three operators (``mytorch/nn/batch_norm.py:123-135``, ``mytorch/tensor.py:292-300``,
    ``mytorch/nn/relu.py:5-10``); here the BatchNorm output and the sum are never stored, and backward
    re-derives the ReLU mask from x, the statistics and the residual."""
    channels = input.shape[1]
    requires_grad = input.requires_grad or residual.requires_grad
    if input.shape != residual.shape or input.device != residual.device or input.dtype != residual.dtype:
        raise RuntimeError("batch_norm2d_add_relu: x and the tensor to add must agree in shape, dtype and device")
    if weight is not None and bias is not None:
        ok = (input.dtype == weight.dtype == bias.dtype and input.device == weight.device == bias.device
              and weight.shape == (channels,) and bias.shape == (channels,))
        if not ok:
            raise RuntimeError("batch_norm2d shape, dtype or device mismatch")
        requires_grad = requires_grad or weight.requires_grad or bias.requires_grad
    out, mean, var = dispatch(input.device, "batch_norm2d_add_relu")(input, residual, weight, bias, eps, training, momentum, running_mean, running_var)
    out.requires_grad = requires_grad and not tracker.no_grad
    return record("batch_norm2d_add_relu", [input, residual, weight, bias, eps], out, [mean, var])


@tracker.register_backward_function("batch_norm2d_add_relu")
def _batch_norm2d_add_relu_backward(output_grad, mean, var, input, residual, weight, bias, eps):
    return dispatch(input.device, "batch_norm2d_add_relu_backward")(output_grad, mean, var, input, residual, weight, bias, eps)
