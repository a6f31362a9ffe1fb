"""conv2d front-end (``mytorch/nn/functional/conv.py:10-49``)."""
from mytorch_b200.ops._common import dispatch, grad_enabled, record, tracker
from mytorch_b200.tensor import MismatchDataTypesError, MismatchDevicesError, Tensor


def conv2d(input: Tensor, weight: Tensor, bias=None, stride=1, padding=0, bn_stats=False) -> Tensor:
    """``bn_stats`` (no counterpart in the reference): the result goes straight into a BatchNorm layer
    in training mode; the CUDA backend then lets the convolution reduce the batch statistics of its
    own output, which BatchNorm picks up instead of re-reading the tensor.  Results are unchanged."""
    if weight.device is not input.device or (bias is not None and bias.device is not input.device):
        raise MismatchDevicesError([t.device for t in (input, weight, bias) if t is not None])
    if weight.dtype is not input.dtype or (bias is not None and bias.dtype is not input.dtype):
        raise MismatchDataTypesError([t.dtype for t in (input, weight, bias) if t is not None])
    stride = (stride, stride) if isinstance(stride, int) else tuple(stride)
    padding = (padding, padding) if isinstance(padding, int) else tuple(padding)
    packed = [] if weight.requires_grad and not tracker.no_grad else None
    if input.device.type == "cuda" and (bn_stats or packed is not None):
        out = dispatch(input.device, "conv2d")(input, weight, bias, stride, padding, bn_stats, packed)
    else:
        out = dispatch(input.device, "conv2d")(input, weight, bias, stride, padding)
    out.requires_grad = grad_enabled(input, weight, bias)
    record("conv2d", [input, weight, bias, stride, padding], out)
    if packed:  # kept by this node alone: it lives as long as the graph and belongs to the values forward saw
        out._grad_node.keywords = {"packed_input": packed[0]}
    return out


@tracker.register_backward_function("conv2d")
def conv2d_backward(output_grad, input, weight, bias, stride, padding, accumulate_dx=None, accumulate_shared=False, defer_weight_gradient=False,
                    packed_input=None):
    """``accumulate_dx`` is the gradient ``input`` already holds (the tape passes it for operators
    listed in ``DAGTracker.fused_accumulate``): the returned dx then includes it.  ``accumulate_shared``: others may
    hold that tensor too (``DAGTracker.accumulates_in_place``), so it is only read.
    ``defer_weight_gradient`` (passed by the tape for operators in ``DAGTracker.deferrable``): the backend
    may compute dw beside the rest of the pass; it is complete after the tape's next ``join_hook()``.
    ``packed_input``: the input as forward had it packed for its kernel."""
    backend = dispatch(input.device, "conv2d_backward")
    extra = {}
    if accumulate_dx is not None:
        extra["accumulate_dx"] = accumulate_dx
        if accumulate_shared:
            extra["accumulate_shared"] = True
    if packed_input is not None:
        extra["packed_input"] = packed_input
    if defer_weight_gradient and input.device.type == "cuda":
        extra["defer_weight_gradient"] = True
    dx, dw, db = backend(output_grad, input, weight, bias, stride, padding, **extra)
    return [dx, dw, db]


tracker.fused_accumulate["conv2d"] = 0  # input 0's accumulated gradient can be folded into the backward
tracker.accumulates_in_place.add("conv2d")
tracker.deferrable.add("conv2d")        # the weight gradient may run beside the rest of backward
