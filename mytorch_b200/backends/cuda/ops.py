"""CUDA operator wrappers: allocate outputs, marshal shapes and scalars, call the kernel library.

One function per registry name, with the positional signatures and return containers of the
reference's ``mytorch/backends/cuda/ops/*.py`` (e.g. ``conv2d`` / ``conv2d_backward``
``conv.py:9-90``, ``batch_norm2d`` ``batch_norm.py:10-105``, ``max_pool2d`` ``pool_ops.py:95-104``,
``sgd`` ``sgd.py:8-35``).  No wrapper synchronises, copies metadata to the device or touches the
host copy of a tensor, so a whole training step can be captured in a CUDA graph.

4-D float32 tensors are channels-last in device memory (see ``tensor.py``); helpers below give
the logical-dimension strides of either layout to the generic strided kernels.
"""
from __future__ import annotations

import ctypes

import numpy as np

from mytorch_b200.autograd import DAGTracker
from mytorch_b200.backends.backend_dispatcher import BackendDispatcher
from mytorch_b200.backends.cuda.env import CudaEnv, CudaMemory, _binding
from mytorch_b200.backends.utils import calculate_broadcast_shape, calculate_reduce_shape, calculate_reshaped_shape
from mytorch_b200.dtype import float32, int32, int64
from mytorch_b200.tensor import InvalidDataTypeError, MismatchShapesError, Tensor

_tracker = DAGTracker.instance()
_reg = BackendDispatcher.instance().register_backend_function
_on_device = Tensor._on_device


# Native (csrc/binding.cpp): _env(tensor) makes the tensor's device current and returns the CUDA state; _new(shape, like,
# dtype=None) is an uninitialised result tensor.  Tensors and blocks are pointer arguments as they are, tuples and lists of
# ints are shapes and strides.
_env = getattr(_binding, "enter", None)
_new = getattr(_binding, "new_like", None)


def _numel(shape):
    n = 1
    for s in shape:
        n *= s
    return n


def _grad_buffer(param):
    """Output tensor for a parameter's gradient.  Under the data-parallel wrapper every parameter
    owns a window of the flat all-reduce buffer (``param._grad_slot``) and its first gradient of a
    backward pass is written straight into it; otherwise (no wrapper, or a second contribution that
    the tape will add to the first) a fresh tensor."""
    slot = getattr(param, "_grad_slot", None)
    if slot is None or param.grad is not None:
        return _new(param.shape, param)
    return _on_device(param.shape, param.dtype, param.device, slot)


def _f32(*tensors):
    for t in tensors:
        if t is not None and t.dtype is not float32:
            raise InvalidDataTypeError(t.dtype)


def _nontrivial_nhwc(t):
    return t._nhwc and t.shape[1] > 1 and t.shape[2] * t.shape[3] > 1


def _strides(t):
    """Element strides of the logical dimensions in device memory."""
    shape = t.shape
    if t._nhwc:
        n, c, h, w = shape
        return [h * w * c, 1, w * c, c]
    out, acc = [0] * len(shape), 1
    for i in range(len(shape) - 1, -1, -1):
        out[i] = acc
        acc *= shape[i]
    return out


def _aligned(*tensors):
    """All on 16-byte boundaries: windows of larger blocks may start at any float."""
    for t in tensors:
        if t._native_array.ptr % 16:
            return False
    return True


# ---------------------------------------------------------------------------- host <-> device

@_reg("cuda", "upload")
def cuda_upload(t, array):
    """Host ndarray (logical layout) -> device storage of ``t`` (channels-last when 4-D float32)."""
    env = _env(t)
    array = np.ascontiguousarray(array, dtype=t.dtype.np_dtype)
    if _nontrivial_nhwc(t):
        stage = CudaMemory(t.device.index, array.nbytes)
        stage.write(array)
        n, c, h, w = t.shape
        env.lib.nchw_to_nhwc_f32(stage.ptr, t, n, c, h, w, env.stream())
    else:
        t._native_array.write(array)


def upload_into(t, host):
    """Asynchronously refill an existing device tensor from host memory holding the logical (NCHW)
    layout: a NumPy array (page-locked, e.g. ``env.PinnedBuffer(...).array``, for a truly asynchronous
    copy) or an object with ``data_ptr()`` such as a pinned PyTorch CPU tensor.  The memory must stay
    valid until the copy has run.  The staging buffer of a channels-last tensor is allocated once and reused."""
    env = _env(t)
    src = host if hasattr(host, "data_ptr") else np.ascontiguousarray(host)
    if _nontrivial_nhwc(t):
        stage = getattr(t, "_stage", None)
        if stage is None:
            stage = t._stage = CudaMemory(t.device.index, t._native_array.nbytes)
        stage.write_from(src)
        n, c, h, w = t.shape
        env.lib.nchw_to_nhwc_f32(stage.ptr, t, n, c, h, w, env.stream())
    else:
        t._native_array.write_from(src)
        if not hasattr(host, "data_ptr") and src is not host:
            env.lib.stream_synchronize(env.stream())  # `src` is a temporary: let the copy finish before it goes away


@_reg("cuda", "download")
def cuda_download(t):
    env = _env(t)
    if _nontrivial_nhwc(t):
        tmp = CudaMemory(t.device.index, t._native_array.nbytes)
        n, c, h, w = t.shape
        env.lib.nhwc_to_nchw_f32(t, tmp.ptr, n, c, h, w, env.stream())
        return tmp.read(t.shape, t.dtype.np_dtype)
    return t._native_array.read(t.shape, t.dtype.np_dtype)


# ---------------------------------------------------------------------------- convolution

def _conv_args(x, w, stride, padding):
    """(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout)"""
    n, cin, h, wd = x.shape
    cout, cin2, kh, kw = w.shape
    if cin != cin2:
        raise MismatchShapesError([x.shape, w.shape])
    return (n, cin, h, wd, kh, kw, stride[0], stride[1], padding[0], padding[1], cout)


_TC_CHANNELS = 32  # the tensor-core convolution reads activations in blocks of 32 channels


def _stem_form(x_shape, w_shape, stride, padding):
    """How a convolution over fewer than 32 channels (an image stem) reaches the tensor-core kernels, or None when it
    does not (too small for them, or an output width they do not take).

    ``(pack, args)``: ``mtb_pack_patches_f32`` with the window ``pack`` = (kh, kw, sh, sw, ph, pw) turns the input into
    blocks of 32 channels, on which the convolution has the arguments ``args``.  Where the whole filter fits 32 entries (3x3
    over 3 channels) the window disappears and each output reads one block; where one filter row does (7x7 over 3
    channels: 21) a window of a single column stays, 7 blocks instead of the 49 of zero-padded channels.
    ``pack`` is None where not even a row fits: the channels are padded with zeros to one block."""
    n, c, h, w = x_shape
    cout, _, kh, kw = w_shape
    (sh, sw), (ph, pw) = stride, padding
    if c >= _TC_CHANNELS or cout % 4 or n * h * w * _TC_CHANNELS * 4 < (1 << 17):
        return None
    oh, ow = (h + 2 * ph - kh) // sh + 1, (w + 2 * pw - kw) // sw + 1
    if c == 1:  # measured on 28x28 digits only, where a step is all launches and fewer blocks gain nothing; larger images were not
        return None, (n, _TC_CHANNELS, h, w, kh, kw, sh, sw, ph, pw, cout)
    if kh * kw * c <= _TC_CHANNELS:
        return (kh, kw, sh, sw, ph, pw), (n, _TC_CHANNELS, oh, ow, 1, 1, 1, 1, 0, 0, cout)
    if kw * c <= _TC_CHANNELS:
        return (1, kw, 1, sw, 0, pw), (n, _TC_CHANNELS, h, ow, kh, 1, sh, 1, ph, 0, cout)
    return None, (n, _TC_CHANNELS, h, w, kh, kw, sh, sw, ph, pw, cout)


def _stem_input(env, x, form):
    """The input in the form the convolution reads."""
    pack, args = form
    if pack is None:
        return _pad_channels(env, x, _TC_CHANNELS)
    n, c, h, w = x.shape
    out = _new((n, _TC_CHANNELS, args[2], args[3]), x)
    env.lib.pack_patches_f32(n, c, h, w, *pack, x, out, env.stream())
    return out


def _stem_filter_rows(w_shape, form):
    """(rows, entries per row) of the filter as that form reads it: a row is widened to one block of 32."""
    cout, c, kh, kw = w_shape
    if form[0] is None:
        return cout * kh * kw, c
    return cout * form[1][4], form[0][0] * kw * c


def _pad_channels(env, t, channels):
    """A channels-last tensor copied into one with `channels` channels (dim 1), the new ones zero."""
    n, c, h, w = t.shape
    out = _new((n, channels, h, w), t)
    env.lib.resize_channels_f32(t, out, n * h * w, c, channels, env.stream())
    return out


def _take_channels(env, t, channels, like, out=None):
    """First `channels` channels (dim 1) of a channels-last tensor, as a new tensor (or into `out`)."""
    n, c, h, w = t.shape
    out = _new((n, channels, h, w), like) if out is None else out
    env.lib.resize_channels_f32(t, out, n * h * w, c, channels, env.stream())
    return out


_BIAS_BESIDE_BYTES = 16 << 20


def _conv_operands(env, input, weight, stride, padding, packed=None):
    """(arguments, input, filter, output tensor) of a forward convolution, the operands in the form its kernel reads.
    ``packed``: a list that takes the input as it was packed, if it was."""
    return _operands_of(env, input, weight, *_conv_form(input, weight, stride, padding), packed)


def _conv_form(input, weight, stride, padding):
    """(arguments, how the input is packed or None) of a forward convolution."""
    a = _conv_args(input, weight, stride, padding)
    return a, _stem_form(input.shape, weight.shape, stride, padding) if a[1] < _TC_CHANNELS else None


def _operands_of(env, input, weight, a, form, packed=None):
    x, wt = input, weight
    n, cin, h, w, kh, kw, sh, sw, ph, pw, cout = a
    oh, ow = (h + 2 * ph - kh) // sh + 1, (w + 2 * pw - kw) // sw + 1
    if form is not None:
        a = form[1]
        x = _stem_input(env, input, form)
        if packed is not None:
            packed.append(x)
        rows, entries = _stem_filter_rows(weight.shape, form)
        block = CudaMemory(weight.device.index, rows * _TC_CHANNELS * 4)
        env.lib.resize_channels_f32(weight, block, rows, entries, _TC_CHANNELS, env.stream())
        wt = _on_device((rows, _TC_CHANNELS), float32, weight.device, block)
    return a, x, wt, _new((n, cout, oh, ow), input)


@_reg("cuda", "conv2d_batch_norm")
def cuda_conv2d_batch_norm(input, weight, bias, stride, padding, gamma, beta, running_mean, running_var, eps, relu, residual=None, pool=False):
    """Inference: relu?(batch_norm2d(conv2d(input)) + residual) with running statistics, in the convolution's launch.
    ``pool``: with a ReLU and a 2x2 max-pool of stride 2 behind it; None where that takes more than one launch."""
    _f32(input, weight, bias, gamma, beta, running_mean, running_var, residual)
    env = _env(input)
    if pool:
        a, form = _conv_form(input, weight, stride, padding)
        if form is not None or not env.lib.conv2d_bn_pool_takes(*a):
            return None
        return _conv_bn_pooled(env, a, input, weight, bias, gamma, beta, running_mean, running_var, eps)
    a, x, wt, out = _conv_operands(env, input, weight, stride, padding)
    if residual is not None and residual.shape != out.shape:
        raise MismatchShapesError([out.shape, residual.shape])
    ws, ws_bytes = env.workspace(env.lib.conv2d_workspace_bytes(*a))
    env.lib.conv2d_bn_forward_f32(*a, x, wt, bias, gamma, beta, running_mean, running_var, float(eps),
                                  residual, int(bool(relu)), out, ws, ws_bytes, env.stream())
    return out


@_reg("cuda", "conv2d_batch_norm_halved")
def cuda_conv2d_batch_norm_halved(input, weight, bias, stride, padding, gamma, beta, running_mean, running_var, eps):
    """Inference: relu(batch_norm2d(conv2d(input))) with running statistics in the convolution's launch, and a 2x2 max-pool of stride 2 in the same
    launch where that exists: (result, whether the pool is in it)."""
    _f32(input, weight, bias, gamma, beta, running_mean, running_var)
    env = _env(input)
    a, form = _conv_form(input, weight, stride, padding)
    scratch = 0  # an image stem that is packed for the tensor cores is not a small convolution, and takes none
    if form is None:
        scratch = env.lib.conv2d_bn_pool_scratch_bytes(*a)
        if scratch < 0:
            return _conv_bn_pooled(env, a, input, weight, bias, gamma, beta, running_mean, running_var, eps), True
    a, x, wt, out = _operands_of(env, input, weight, a, form)
    ws, ws_bytes = env.workspace(scratch) if scratch else (None, 0)
    env.lib.conv2d_bn_forward_f32(*a, x, wt, bias, gamma, beta, running_mean, running_var, float(eps), None, 1, out, ws, ws_bytes, env.stream())
    return out, False


def _conv_bn_pooled(env, a, input, weight, bias, gamma, beta, running_mean, running_var, eps):
    n, _, h, w, kh, kw, sh, sw, ph, pw, cout = a
    out = _new((n, cout, ((h + 2 * ph - kh) // sh + 1) // 2, ((w + 2 * pw - kw) // sw + 1) // 2), input)
    out._pool_tiemask = mask = CudaMemory(input.device.index, out._native_array.nbytes // 2)
    env.lib.conv2d_bn_pool_forward_f32(*a, input, weight, bias, gamma, beta, running_mean, running_var, float(eps), out, mask, env.stream())
    return out


@_reg("cuda", "conv2d")
def cuda_conv2d(input, weight, bias, stride, padding, bn_stats=False, packed=None):
    """``bn_stats``: the output feeds a BatchNorm layer in training mode; where the kernel allows, the
    convolution's epilogue also reduces the per-channel batch statistics of the output and leaves them
    on the result (``_bn_partials``) for ``batch_norm2d``, which then skips its own pass over the tensor.
    ``packed`` (a list): takes the input in the form the kernel read, where few channels had to be packed; the weight
    gradient of the same values can read it again (``packed_input`` of the backward)."""
    _f32(input, weight, bias)
    env = _env(input)
    a, x, wt, out = _conv_operands(env, input, weight, stride, padding, packed)
    ws, ws_bytes = env.workspace(env.lib.conv2d_workspace_bytes(*a))
    if bn_stats:
        partials = CudaMemory(input.device.index, env.lib.conv2d_stats_max_rows() * 3 * a[-1] * 4)
        rows = (ctypes.c_int * 1)()
        env.lib.conv2d_forward_stats_f32(*a, x, wt, bias, out, 0, partials.ptr, rows, ws, ws_bytes,
                                         env.stream())
        if rows[0] > 0:
            out._bn_partials = (partials, rows[0])
        return out
    env.lib.conv2d_forward_f32(*a, x, wt, bias, out, 0, ws, ws_bytes, env.stream())
    return out


@_reg("cuda", "conv2d_backward")
def cuda_conv2d_backward(output_grad, input, weight, bias, stride, padding, accumulate_dx=None, defer_weight_gradient=False,
                         accumulate_shared=False, packed_input=None):
    """``accumulate_dx``: a gradient the input has already received from another consumer; when given,
    the returned dx is the data gradient PLUS that tensor (added in the convolution's epilogue where
    the kernel allows), and the caller stores it instead of adding the two itself.  The returned tensor may be that
    tensor, changed in place, unless ``accumulate_shared`` says that others hold it too.
    ``defer_weight_gradient``: the caller (the tape) does not need dw until it calls ``CudaEnv.join_side``;
    the weight gradient then runs on the device's side stream, beside whatever the caller enqueues next."""
    _f32(output_grad, input, weight)
    env = _env(input)
    want_dx, want_dw, cin = input.requires_grad, weight.requires_grad, input.shape[1]
    form = _stem_form(input.shape, weight.shape, stride, padding) if cin < _TC_CHANNELS else None
    x, wt = input, weight
    a = _conv_args(x, weight, stride, padding)
    # a data gradient of 1 or 3 channels fits no tensor-core tile: 32 are computed (the filter padded with zeros) and the first taken
    padded = want_dx and form is not None and cin % 4 != 0 and a[-1] % 32 == 0
    if padded:
        wt = _pad_channels(env, weight, _TC_CHANNELS)
        a = (a[0], _TC_CHANNELS) + a[2:]
    st = env.stream()
    need = env.lib.conv2d_workspace_bytes(*a)
    dx = dw = db = None
    # The bias gradient reads all of dY and needs little else of an SM, so it goes beside the tensor-core kernels of this call on
    # the side stream, if dY is large enough for the two events to pay (64 channels, 128 images of 56x56, forward and
    # backward, cold L2: 287 -> 266 us; 48 -> 82 channels, 32 images of 37x37, under the limit: 442 us with and without; no
    # sizes in between were measured).  For direct calls of the operator: the tape defers weight gradients, and a deferred one
    # has the side stream already, and the longer of the two queues.
    want_db = bias is not None and bias.requires_grad
    beside = (want_db and want_dx and not defer_weight_gradient and env.overlap_weight_gradients
              and output_grad._native_array.nbytes >= _BIAS_BESIDE_BYTES)
    if beside:
        # Memory before the fork: a block that is free now was last used by work the side stream waits for, one that the calls
        # below give back is still used by theirs.
        db, scratch = _grad_buffer(bias), env.side_workspace(env.lib.colsum_workspace_bytes(a[-1]))
        side = env.fork_side((output_grad, db))
    if want_dx:
        ws, ws_bytes = env.workspace(need)
        if accumulate_dx is not None and not padded and not accumulate_shared and env.lib.conv2d_dgrad_accumulates_in_place(
                *a, output_grad, wt, accumulate_dx):
            # a filter smaller than its stride (the 1x1 / stride-2 shortcut) reaches only some pixels: it adds
            # to those in the gradient the input already holds, which is then the returned tensor
            dx = accumulate_dx
            env.lib.conv2d_dgrad_add_f32(*a, output_grad, wt, dx, dx, ws, ws_bytes, st)
        elif accumulate_dx is not None and not padded:
            dx = _new(x.shape, x)
            env.lib.conv2d_dgrad_add_f32(*a, output_grad, wt, accumulate_dx, dx, ws, ws_bytes, st)
        else:
            dx = _new((a[0], a[1], a[2], a[3]), x)
            env.lib.conv2d_dgrad_f32(*a, output_grad, wt, dx, ws, ws_bytes, st)
            if padded:
                dx = _take_channels(env, dx, cin, dx)
            if accumulate_dx is not None:
                dx = BackendDispatcher.instance().dispatch("cuda", "add")(dx, accumulate_dx, 1)
    if beside:
        _bias_gradient(env, output_grad, a[-1], db, scratch, side)
    if want_dw:
        # Nothing in the rest of backward reads this layer's weight gradient, so it runs on the side
        # stream, beside the data-gradient / BatchNorm chain that the next layer waits for, and is
        # joined when backward ends (or before anything touches the gradient: see DAGTracker.backward).
        # A weight that already holds a gradient (shared weights) accumulates on the compute stream.
        wa = a
        if form is not None:
            x = _stem_input(env, input, form) if packed_input is None else packed_input
            wa = form[1]
            need = env.lib.conv2d_workspace_bytes(*wa)
        wst = st
        if defer_weight_gradient and env.overlap_weight_gradients and weight.grad is None:
            wst = env.fork_side((x, output_grad))
            wws, wws_bytes = env.side_workspace(need)
        else:
            wws, wws_bytes = env.workspace(need)
        if form is not None:
            rows, entries = _stem_filter_rows(weight.shape, form)
            wide = CudaMemory(weight.device.index, rows * _TC_CHANNELS * 4)
            env.lib.conv2d_wgrad_f32(*wa, x, output_grad, wide, wws, wws_bytes, wst)
            dw = _grad_buffer(weight)
            env.lib.resize_channels_f32(wide, dw, rows, _TC_CHANNELS, entries, wst)
            if wst is not st:
                env._side_keepalive.append(wide)
        else:
            dw = _grad_buffer(weight)
            env.lib.conv2d_wgrad_f32(*a, x, output_grad, dw, wws, wws_bytes, wst)
    if beside:
        env.join_side()
    elif want_db:
        db = _grad_buffer(bias)
        _bias_gradient(env, output_grad, a[-1], db, env.workspace(env.lib.colsum_workspace_bytes(a[-1])), st)
    return [dx, dw, db]


def _bias_gradient(env, output_grad, channels, out, scratch, stream):
    env.lib.colsum_f32(output_grad, _numel(output_grad.shape) // channels, channels, 1.0, out, *scratch, stream)


def _colsum(env, mat, rows, cols, like, scale=1.0, out=None):
    out = _new((cols,), like) if out is None else out
    ws, ws_bytes = env.workspace(env.lib.colsum_workspace_bytes(cols))
    env.lib.colsum_f32(mat, rows, cols, scale, out, ws, ws_bytes, env.stream())
    return out


# ---------------------------------------------------------------------------- linear / mm

def _gemm(env, m, n, k, a, ta, b, tb, bias, relu, c):
    env.lib.gemm_f32(m, n, k, a, ta, b, tb, bias, relu, c, env.stream())


@_reg("cuda", "linear")
def cuda_linear(x, weight, bias):
    _f32(x, weight, bias)
    env = _env(x)
    b, fin = x.shape
    fout = weight.shape[0]
    if weight.shape[1] != fin:
        raise MismatchShapesError([x.shape, weight.shape])
    y = _new((b, fout), x)
    _gemm(env, b, fout, fin, x, 0, weight, 1, bias, 0, y)
    return y


@_reg("cuda", "linear_relu")
def cuda_linear_relu(x, weight, bias, keep):
    """(relu(x Wᵀ + b), x Wᵀ + b or None): a Linear layer and the ReLU behind it in one launch.  ``keep``: a backward pass will
    ask for the second, whose sign masks the gradient."""
    _f32(x, weight, bias)
    env = _env(x)
    b, fin = x.shape
    fout = weight.shape[0]
    if weight.shape[1] != fin:
        raise MismatchShapesError([x.shape, weight.shape])
    y, pre = _new((b, fout), x), _new((b, fout), x) if keep else None
    env.lib.linear_relu_f32(b, fout, fin, x, weight, bias, pre, y, env.stream())
    return y, pre


@_reg("cuda", "linear_relu_backward")
def cuda_linear_relu_backward(output_grad, pre, x, weight, bias):
    env = _env(x)
    masked = _new(pre.shape, pre)
    env.lib.relu_backward_f32(output_grad, pre, masked, _numel(pre.shape), env.stream())
    return cuda_linear_backward(masked, x, weight, bias)


@_reg("cuda", "linear_backward")
def cuda_linear_backward(output_grad, x, weight, bias):
    env = _env(x)
    b, fin = x.shape
    fout = weight.shape[0]
    dx = dw = db = None
    if x.requires_grad:
        dx = _new(x.shape, x)
        _gemm(env, b, fin, fout, output_grad, 0, weight, 0, None, 0, dx)
    if weight.requires_grad:
        dw = _grad_buffer(weight)
        _gemm(env, fout, fin, b, output_grad, 1, x, 0, None, 0, dw)
    if bias is not None and bias.requires_grad:
        db = _colsum(env, output_grad, b, fout, bias, out=_grad_buffer(bias))
    return [dx, dw, db]


@_reg("cuda", "mm")
def cuda_mm(x, y):
    _f32(x, y)
    env = _env(x)
    (m, k), (k2, n) = x.shape, y.shape
    if k != k2:
        raise MismatchShapesError([x.shape, y.shape])
    z = _new((m, n), x)
    _gemm(env, m, n, k, x, 0, y, 0, None, 0, z)
    return z


@_reg("cuda", "mm_backward")
def cuda_mm_backward(output_grad, x, y):
    env = _env(x)
    (m, k), n = x.shape, y.shape[1]
    dx, dy = _new(x.shape, x), _new(y.shape, y)
    _gemm(env, m, k, n, output_grad, 0, y, 1, None, 0, dx)
    _gemm(env, k, n, m, x, 1, output_grad, 0, None, 0, dy)
    return dx, dy


# ---------------------------------------------------------------------------- batch norm

@_reg("cuda", "batch_norm2d")
def cuda_batch_norm2d(x, weight, bias, eps, training, momentum, running_mean, running_var, relu=False):
    _f32(x, weight, bias, running_mean, running_var)
    env = _env(x)
    n, c, h, w = x.shape
    y, mean, var = _new(x.shape, x), _new((c,), x), _new((c,), x)
    ws, ws_bytes = env.workspace(env.lib.batch_norm2d_workspace_bytes(n, c, h, w))
    # without running statistics the reference normalises with batch statistics in eval mode too
    # (``mytorch/backends/cpu/ops/batch_norm.py:40-46``)
    use_batch_stats = bool(training) or running_mean is None or running_var is None
    pre = getattr(x, "_bn_partials", None)
    if use_batch_stats and pre is not None:  # the convolution that produced x already reduced its statistics
        env.lib.batch_norm2d_forward_prestats_f32(n, c, h, w, x, weight, bias, float(eps), float(momentum), running_mean,
                                                  running_var, y, mean, var, int(bool(relu)), pre[0].ptr, pre[1], ws, ws_bytes,
                                                  env.stream())
        return y, mean, var
    env.lib.batch_norm2d_forward_f32(n, c, h, w, x, weight, bias, float(eps), int(use_batch_stats), float(momentum),
                                     running_mean, running_var, y, mean, var, int(bool(relu)), ws, ws_bytes, env.stream())
    return y, mean, var


@_reg("cuda", "batch_norm2d_add_relu")
def cuda_batch_norm2d_add_relu(x, residual, weight, bias, eps, training, momentum, running_mean, running_var):
    """max(0, batch_norm2d(x) + residual) in one normalise pass; returns (y, mean, var)."""
    _f32(x, residual, weight, bias, running_mean, running_var)
    if x.shape != residual.shape:
        raise MismatchShapesError([x.shape, residual.shape])
    env = _env(x)
    n, c, h, w = x.shape
    y, mean, var = _new(x.shape, x), _new((c,), x), _new((c,), x)
    ws, ws_bytes = env.workspace(env.lib.batch_norm2d_workspace_bytes(n, c, h, w))
    use_batch_stats = bool(training) or running_mean is None or running_var is None
    pre = getattr(x, "_bn_partials", None) if use_batch_stats else None
    head = (n, c, h, w, x, residual, weight, bias, float(eps), int(use_batch_stats), float(momentum), running_mean,
            running_var, y, mean, var)
    tail = (pre[0] if pre else None, pre[1] if pre else 0, ws, ws_bytes, env.stream())
    if c % 4 == 0 and not _tracker.no_grad and _aligned(x, residual):  # the ReLU's mask goes to backward with the statistics
        mean._relu_mask = CudaMemory(x.device.index, n * c * h * w // 4)
        env.lib.batch_norm2d_add_relu_forward_masked_f32(*head, mean._relu_mask, *tail)
    else:
        env.lib.batch_norm2d_add_relu_forward_f32(*head, *tail)
    return y, mean, var


@_reg("cuda", "batch_norm2d_add_relu_backward")
def cuda_batch_norm2d_add_relu_backward(output_grad, mean, var, x, residual, weight, bias, eps):
    """[dx, dresidual, dgamma, dbeta]"""
    env = _env(x)
    n, c, h, w = x.shape
    dx, dres = _new(x.shape, x), _new(x.shape, x)
    affine = weight is not None and bias is not None
    dg = _grad_buffer(weight) if affine else None
    db = _grad_buffer(bias) if affine else None
    ws, ws_bytes = env.workspace(env.lib.batch_norm2d_workspace_bytes(n, c, h, w))
    tail = (weight, bias, float(eps), dx, dres, dg, db, ws, ws_bytes, env.stream())
    mask = getattr(mean, "_relu_mask", None)
    if mask is not None and _aligned(x, output_grad):
        env.lib.batch_norm2d_add_relu_backward_masked_f32(n, c, h, w, output_grad, mean, var, x, mask, *tail)
    else:
        env.lib.batch_norm2d_add_relu_backward_f32(n, c, h, w, output_grad, mean, var, x, residual, *tail)
    return [dx, dres, dg, db]


@_reg("cuda", "batch_norm2d_relu")
def cuda_batch_norm2d_relu(x, weight, bias, eps, training, momentum, running_mean, running_var):
    """BatchNorm2d followed by ReLU in one normalise pass (the ReLU input is never stored)."""
    return cuda_batch_norm2d(x, weight, bias, eps, training, momentum, running_mean, running_var, relu=True)


@_reg("cuda", "batch_norm2d_relu_backward")
def cuda_batch_norm2d_relu_backward(output_grad, mean, var, x, weight, bias, eps):
    return cuda_batch_norm2d_backward(output_grad, mean, var, x, weight, bias, eps, relu=True)


@_reg("cuda", "batch_norm2d_relu_halved")
def cuda_batch_norm2d_relu_halved(x, weight, bias, eps, training, momentum, running_mean, running_var, window=2):
    """BatchNorm2d, ReLU and a max-pool of stride 2 (2x2, or 3x3 with padding 1: ``window``): (y, mean, var), or None where the
    channels are no fours, no window fits or a tensor starts off 16 bytes.  Same bits as the three operators."""
    _f32(x, weight, bias, running_mean, running_var)
    n, c, h, w = x.shape
    if c % 4 or h < 2 or w < 2 or n * c * h * w >= 1 << 29 or not _aligned(x) or bias is not None and not _aligned(bias):
        return None
    env = _env(x)
    y, mean, var = _new((n, c, h // 2, w // 2) if window == 2 else (n, c, (h + 1) // 2, (w + 1) // 2), x), _new((c,), x), _new((c,), x)
    ws, ws_bytes = env.workspace(env.lib.batch_norm2d_workspace_bytes(n, c, h, w))
    use_batch_stats = bool(training) or running_mean is None or running_var is None
    pre = getattr(x, "_bn_partials", None) if use_batch_stats else None
    y._pool_tiemask = mean._pool_tiemask = mask = CudaMemory(x.device.index, y._native_array.nbytes // 2)
    env.lib.batch_norm2d_relu_pool_forward_f32(n, c, h, w, window, x, weight, bias, float(eps), int(use_batch_stats), float(momentum), running_mean, running_var,
                                               y, mean, var, mask, pre[0] if pre else None, pre[1] if pre else 0, ws, ws_bytes, env.stream())
    return y, mean, var


@_reg("cuda", "batch_norm2d_relu_halved_backward")
def cuda_batch_norm2d_relu_halved_backward(output_grad, mean, var, x, weight, bias, eps, window=2):
    env = _env(x)
    n, c, h, w = x.shape
    if window == 3:
        behind = _new(x.shape, x)
        env.lib.max_pool2d_backward_f32(n, c, h, w, 3, 3, 2, 2, 1, 1, output_grad, mean._pool_tiemask, None, None, behind, env.stream())
        return cuda_batch_norm2d_backward(behind, mean, var, x, weight, bias, eps, relu=True)
    dy, dx = output_grad, _new(x.shape, x)
    if not _aligned(dy):
        dy = _new(output_grad.shape, output_grad)
        env.lib.copy_f32(dy, output_grad, _numel(dy.shape), env.stream())
    affine = weight is not None and bias is not None
    dg = _grad_buffer(weight) if affine else None
    db = _grad_buffer(bias) if affine else None
    ws, ws_bytes = env.workspace(env.lib.batch_norm2d_workspace_bytes(n, c, h, w))
    env.lib.batch_norm2d_relu_pool_backward_f32(n, c, h, w, dy, mean, var, x, mean._pool_tiemask, weight, bias, float(eps), dx, dg, db, ws, ws_bytes, env.stream())
    return [dx, dg, db]


@_reg("cuda", "batch_norm2d_backward")
def cuda_batch_norm2d_backward(output_grad, mean, var, x, weight, bias, eps, relu=False):
    env = _env(x)
    n, c, h, w = x.shape
    dx = _new(x.shape, x)
    affine = weight is not None and bias is not None
    dg = _grad_buffer(weight) if affine else None
    db = _grad_buffer(bias) if affine else None
    ws, ws_bytes = env.workspace(env.lib.batch_norm2d_workspace_bytes(n, c, h, w))
    env.lib.batch_norm2d_backward_f32(n, c, h, w, output_grad, mean, var, x, weight, bias, float(eps),
                                      int(bool(relu)), dx, dg, db, ws, ws_bytes, env.stream())
    return [dx, dg, db]


# ---------------------------------------------------------------------------- pooling

def _pool_args(x, kernel_size, stride, padding):
    if stride is None:
        stride = kernel_size
    kh, kw = (kernel_size, kernel_size) if isinstance(kernel_size, int) else kernel_size
    sh, sw = (stride, stride) if isinstance(stride, int) else stride
    ph, pw = (padding, padding) if isinstance(padding, int) else padding
    return (*x.shape, kh, kw, sh, sw, ph, pw)


@_reg("cuda", "max_pool2d")
def cuda_max_pool2d(x, kernel_size, stride, padding):
    _f32(x)
    env = _env(x)
    a = _pool_args(x, kernel_size, stride, padding)
    n, c, h, w, kh, kw, sh, sw, ph, pw = a
    oh, ow = (2 * ph + h - kh) // sh + 1, (2 * pw + w - kw) // sw + 1
    y = _new((n, c, oh, ow), x)
    mask = CudaMemory(x.device.index, 2 * n * c * oh * ow) if kh * kw <= 16 else None
    env.lib.max_pool2d_forward_f32(*a, x, y, mask, env.stream())
    y._pool_tiemask = mask  # uint16 per output element, channels-last like y
    return y


@_reg("cuda", "max_pool2d_backward")
def cuda_max_pool2d_backward(output_grad, output, x, kernel_size, stride, padding):
    env = _env(x)
    a = _pool_args(x, kernel_size, stride, padding)
    dx = _new(x.shape, x)
    mask = getattr(output, "_pool_tiemask", None)
    env.lib.max_pool2d_backward_f32(*a, output_grad, mask, output, x, dx, env.stream())
    return [dx]


def max_pool2d_argmax(output):
    """Window-local index (kh*KW + kw) of the first maximum for every output element, as a host
    uint8 array in logical [N,C,OH,OW] order.  Derived from the tie mask written by forward."""
    env = _env(output)
    mask = getattr(output, "_pool_tiemask", None)
    if mask is None:
        raise RuntimeError("this tensor was not produced by max_pool2d with a window of at most 16 elements")
    n, c, oh, ow = output.shape
    total = n * c * oh * ow
    arg = CudaMemory(output.device.index, total)
    env.lib.max_pool2d_argmax_u8(mask.ptr, arg.ptr, total, env.stream())
    return arg.read((n, oh, ow, c), np.uint8).transpose(0, 3, 1, 2).copy()


# ---------------------------------------------------------------------------- elementwise

@_reg("cuda", "relu")
def cuda_relu(x):
    _f32(x)
    env = _env(x)
    y = _new(x.shape, x)
    env.lib.relu_forward_f32(x, y, _numel(x.shape), env.stream())
    return y


@_reg("cuda", "relu_backward")
def cuda_relu_backward(output_grad, x):
    env = _env(x)
    dx = _new(x.shape, x)
    env.lib.relu_backward_f32(output_grad, x, dx, _numel(x.shape), env.stream())
    return [dx]


@_reg("cuda", "add_relu")
def cuda_add_relu(x, y):
    """max(0, x + y) for same-shape operands (residual connection followed by ReLU)."""
    _f32(x, y)
    if x.shape != y.shape:
        raise MismatchShapesError([x.shape, y.shape])
    env = _env(x)
    z = _new(x.shape, x)
    env.lib.add_relu_f32(x, y, z, _numel(x.shape), env.stream())
    return z


@_reg("cuda", "add_relu_backward")
def cuda_add_relu_backward(output_grad, x, y):
    env = _env(x)
    g = _new(x.shape, x)
    env.lib.add_relu_backward_f32(output_grad, x, y, g, _numel(x.shape), env.stream())
    return g, g  # one tensor serves both operands: gradients are never modified in place


@_reg("cuda", "fill")
def cuda_fill(x, value):
    env = _env(x)
    if x.dtype is float32:
        env.lib.fill_f32(x, _numel(x.shape), float(value), env.stream())
    else:
        x._native_array.write(np.full(x.shape, value, dtype=x.dtype.np_dtype))


def _host_random(x, array):
    cuda_upload(x, array.astype(x.dtype.np_dtype))


@_reg("cuda", "uniform")
def cuda_uniform(x, seed, a, b):
    # Initialisation only: drawn on the host with the reference CPU recipe, then uploaded, so a
    # model initialised on the GPU has the same weights as one initialised on the CPU.
    np.random.seed(seed)
    _host_random(x, np.random.uniform(low=a, high=b, size=x.shape))


@_reg("cuda", "normal")
def cuda_normal(x, seed, mean, stddev):
    np.random.seed(seed)
    _host_random(x, np.random.normal(mean, stddev, x.shape))


@_reg("cuda", "copy")
def cuda_copy(dst, src):
    env = _env(dst)
    if dst.shape != src.shape:
        raise MismatchShapesError([dst.shape, src.shape])
    if dst.dtype is float32:
        env.lib.copy_f32(dst, src, _numel(dst.shape), env.stream())
    else:
        dst._native_array.copy_from(src._native_array, dst._native_array.nbytes)


@_reg("cuda", "cast")
def cuda_cast(x, dtype):
    env = _env(x)
    from mytorch_b200.dtype import int8

    kinds = {(int32, int64): 0, (int64, float32): 1, (float32, int64): 2, (int8, float32): 3}
    kind = kinds.get((x.dtype, dtype))
    if kind is None:
        raise RuntimeError(f"cast from {x.dtype} to {dtype} is not available on the cuda backend")
    if x._nhwc or (len(x.shape) == 4 and dtype is float32):
        raise RuntimeError("cast of 4-D tensors between float32 and integer types is not available on the cuda backend")
    out = _new(x.shape, x, dtype)
    env.lib.cast(kind, x, out, _numel(x.shape), env.stream())
    return out


# ---------------------------------------------------------------------------- broadcast binary ops

_OPS = {"add": 0, "sub": 1, "mul": 2, "div": 3, "pow": 4, "pow_dx": 6, "pow_dy": 7}


def _bstrides(t, out_shape):
    """Strides of ``t`` along the dimensions of ``out_shape`` (0 where ``t`` broadcasts)."""
    pad = len(out_shape) - len(t.shape)
    st = _strides(t)
    return [0] * pad + [0 if t.shape[i] == 1 and out_shape[pad + i] != 1 else st[i] for i in range(len(t.shape))]


def _binary(name, x, y, alpha=1.0):
    _f32(x, y)
    env = _env(x)
    shape = x.shape if x.shape == y.shape else calculate_broadcast_shape(x.shape, y.shape)
    z = _new(shape, x)
    if x.shape == y.shape and name in ("add", "sub", "mul"):
        if name == "mul":
            env.lib.mul_f32(x, y, z, _numel(shape), env.stream())
        else:
            env.lib.add_f32(x, y, z, _numel(shape), float(alpha) if name == "add" else -float(alpha), env.stream())
        return z
    if name == "add" and len(x.shape) == 2 and y.shape == (x.shape[1],):
        env.lib.add_bias_rows_f32(x, y, z, x.shape[0], x.shape[1], float(alpha), env.stream())
        return z
    env.lib.binary_strided_f32(_OPS[name], len(shape), shape, _bstrides(x, shape), _bstrides(y, shape),
                               _strides(z), x, y, z, float(alpha), env.stream())
    return z


def _scaled(t, scale):
    if scale == 1:
        return t
    env = _env(t)
    out = _new(t.shape, t)
    env.lib.scale_f32(out, t, _numel(t.shape), float(scale), env.stream())
    return out


def _reduce_to(g, shape, like):
    """Sum ``g`` over the dimensions along which a tensor of ``shape`` was broadcast."""
    if tuple(g.shape) == tuple(shape):
        return g
    pad = len(g.shape) - len(shape)
    dims = tuple(i for i in range(len(g.shape)) if i < pad or (shape[i - pad] == 1 and g.shape[i] != 1))
    out = cuda_sum_scale(g, dims, True, 1)
    return cuda_reshape(out, shape)


@_reg("cuda", "add")
def cuda_add(x, y, alpha):
    return _binary("add", x, y, alpha)


@_reg("cuda", "sub")
def cuda_sub(x, y, alpha):
    return _binary("sub", x, y, alpha)


@_reg("cuda", "mul")
def cuda_mul(x, y):
    return _binary("mul", x, y)


@_reg("cuda", "div")
def cuda_div(x, y):
    return _binary("div", x, y)


@_reg("cuda", "pow")
def cuda_pow(x, y):
    return _binary("pow", x, y)


# ``needed``: which of the two gradients the caller will use (the tape has no use for one towards a constant, such as the
# exponent of ``x ** 2``); the other is then None instead of being computed.  The front-end hands it to functions that are
# marked for it (``skips_gradients``).
_BOTH = (True, True)


@_reg("cuda", "add_backward")
def cuda_add_backward(output_grad, x, y, alpha, needed=_BOTH):
    # Same-shape operands receive the upstream gradient itself (no copy): the tape lets no operator change a
    # gradient in place that is not its tensor's alone.
    return (_reduce_to(output_grad, x.shape, x) if needed[0] else None,
            _reduce_to(_scaled(output_grad, alpha), y.shape, y) if needed[1] else None)


@_reg("cuda", "sub_backward")
def cuda_sub_backward(output_grad, x, y, alpha, needed=_BOTH):
    return cuda_add_backward(output_grad, x, y, -alpha, needed)


@_reg("cuda", "mul_backward")
def cuda_mul_backward(output_grad, x, y, needed=_BOTH):
    return (_reduce_to(_binary("mul", output_grad, y), x.shape, x) if needed[0] else None,
            _reduce_to(_binary("mul", output_grad, x), y.shape, y) if needed[1] else None)


@_reg("cuda", "div_backward")
def cuda_div_backward(output_grad, x, y, needed=_BOTH):
    """dx = dy / y, dy_ = -x / y^2 * dy (``mytorch/backends/cpu/ops/broadcast_binary_ops.py:108-115``)."""
    gx = gy = None
    if needed[0]:
        gx = _reduce_to(_binary("div", output_grad, y), x.shape, x)
    if needed[1]:
        gy = _reduce_to(_scaled(_binary("div", _binary("mul", output_grad, x), _binary("mul", y, y)), -1.0), y.shape, y)
    return gx, gy


@_reg("cuda", "pow_backward")
def cuda_pow_backward(output_grad, x, y, needed=_BOTH):
    """dx = y x^(y-1) dy, dy_ = x^y ln(x) dy (``mytorch/backends/cpu/ops/broadcast_binary_ops.py:130-137``)."""
    return (_reduce_to(_binary("mul", _binary("pow_dx", x, y), output_grad), x.shape, x) if needed[0] else None,
            _reduce_to(_binary("mul", _binary("pow_dy", x, y), output_grad), y.shape, y) if needed[1] else None)


for _f in (cuda_add_backward, cuda_sub_backward, cuda_mul_backward, cuda_div_backward, cuda_pow_backward):
    _f.skips_gradients = True


# ---------------------------------------------------------------------------- max / eq / bmm

@_reg("cuda", "max")
def cuda_max(tensor, dim, keepdim):
    """(values, int64 indices) of the maximum along ``dim`` (``None``: over everything, index into the
    flattened logical tensor); ties go to the first element (``mytorch/backends/cuda/ops/max.py:10-75``)."""
    _f32(tensor)
    if dim is not None and not isinstance(dim, int):
        raise RuntimeError(f"max dimension must be a integer or None: {dim}")
    env = _env(tensor)
    nd = len(tensor.shape)
    src = tensor
    if dim is None:
        if _nontrivial_nhwc(tensor):  # flat indices refer to the logical order
            src = cuda_reshape(tensor, (_numel(tensor.shape),))
        kept_shape, kept_strides, red_len, red_stride = [], [], _numel(tensor.shape), 1
        out_shape = calculate_reduce_shape(tensor.shape, tuple(range(nd)), keepdim)
    else:
        dim = dim + nd if dim < 0 else dim
        st = _strides(tensor)
        kept = [i for i in range(nd) if i != dim]
        kept_shape, kept_strides = [tensor.shape[i] for i in kept], [st[i] for i in kept]
        red_len, red_stride = tensor.shape[dim], st[dim]
        out_shape = calculate_reduce_shape(tensor.shape, (dim,), keepdim)
    n_out = _numel(out_shape)
    values = Tensor(shape=(n_out,), dtype=tensor.dtype, device=tensor.device)
    indices = Tensor(shape=tuple(out_shape), dtype=int64, device=tensor.device)
    env.lib.max_strided_f32(src, values, indices, len(kept_shape), kept_shape, kept_strides, red_len, red_stride,
                            env.stream())
    return cuda_reshape(values, tuple(out_shape)), indices


@_reg("cuda", "max_backward")
def cuda_max_backward(output_grad, indices_tensor, tensor, dim, keepdim):
    env = _env(tensor)
    nd = len(tensor.shape)
    dx = _new(tensor.shape, tensor)
    g = output_grad
    if _nontrivial_nhwc(g):  # the kernel reads dy in logical (dense) order, like the indices
        g = cuda_reshape(g, (_numel(g.shape),))
    if dim is None:
        flat = Tensor(shape=(_numel(tensor.shape),), dtype=tensor.dtype, device=tensor.device)
        env.lib.max_backward_f32(g, indices_tensor, flat, _numel(tensor.shape), 0, [], [], 1, env.stream())
        return [cuda_reshape(flat, tensor.shape)]
    dim = dim + nd if dim < 0 else dim
    st = _strides(dx)
    kept = [i for i in range(nd) if i != dim]
    env.lib.max_backward_f32(g, indices_tensor, dx, _numel(tensor.shape), len(kept), [tensor.shape[i] for i in kept],
                             [st[i] for i in kept], st[dim], env.stream())
    return [dx]


@_reg("cuda", "eq")
def cuda_eq(x, y):
    """int8 tensor of element-wise equality (``mytorch/backends/cuda/ops/eq.py:9``)."""
    from mytorch_b200.dtype import int8
    if x.shape != y.shape:
        raise MismatchShapesError([x.shape, y.shape])
    kinds = {float32: 0, int64: 1}
    if x.dtype not in kinds or y.dtype is not x.dtype:
        raise InvalidDataTypeError(x.dtype)
    env = _env(x)
    out = Tensor(shape=x.shape, dtype=int8, device=x.device)
    env.lib.eq_strided(kinds[x.dtype], len(x.shape), x.shape, _strides(x), _strides(y), x, y, out, env.stream())
    return out


def _bmm_into(env, batch, m, n, k, a, ta, b, tb, c):
    """c[i] = op(a[i]) op(b[i]) for i < batch; dense 3-D operands, one GEMM per batch entry."""
    sa, sb, sc = 4 * (a.shape[1] * a.shape[2]), 4 * (b.shape[1] * b.shape[2]), 4 * m * n
    pa, pb, pc = a._native_array.ptr, b._native_array.ptr, c._native_array.ptr
    for i in range(batch):
        env.lib.gemm_f32(m, n, k, pa + i * sa, ta, pb + i * sb, tb, None, 0, pc + i * sc, env.stream())


@_reg("cuda", "bmm")
def cuda_bmm(x, y):
    """[B,M,K] x [B,K,N] -> [B,M,N] (``mytorch/backends/cuda/ops/mm.py:131-138``)."""
    _f32(x, y)
    if len(x.shape) != 3 or len(y.shape) != 3 or x.shape[0] != y.shape[0] or x.shape[2] != y.shape[1]:
        raise MismatchShapesError([x.shape, y.shape])
    env = _env(x)
    bsz, m, k = x.shape
    n = y.shape[2]
    z = _new((bsz, m, n), x)
    _bmm_into(env, bsz, m, n, k, x, 0, y, 0, z)
    return z


@_reg("cuda", "bmm_backward")
def cuda_bmm_backward(output_grad, x, y):
    env = _env(x)
    bsz, m, k = x.shape
    n = y.shape[2]
    dx, dy = _new(x.shape, x), _new(y.shape, y)
    _bmm_into(env, bsz, m, k, n, output_grad, 0, y, 1, dx)   # dx[i] = dz[i] y[i]^T
    _bmm_into(env, bsz, k, n, m, x, 1, output_grad, 0, dy)   # dy[i] = x[i]^T dz[i]
    return dx, dy


# ---------------------------------------------------------------------------- reductions

@_reg("cuda", "sum_scale")
def cuda_sum_scale(x, dim, keepdim, scale):
    _f32(x)
    env = _env(x)
    dim = tuple(dim)
    out_shape = calculate_reduce_shape(x.shape, dim, keepdim)
    out = _new(out_shape, x)
    st = env.stream()
    if x._nhwc and dim == (2, 3):
        n, c, h, w = x.shape
        env.lib.nhwc_spatial_sum_f32(x, out, n, c, h * w, float(scale), st)
        return out
    if x._nhwc and dim == (0, 2, 3):
        n, c, h, w = x.shape
        ws, ws_bytes = env.workspace(env.lib.colsum_workspace_bytes(c))
        env.lib.colsum_f32(x, n * h * w, c, float(scale), out, ws, ws_bytes, st)
        return out
    xs = _strides(x)
    kept = [i for i in range(len(x.shape)) if i not in dim]
    red = list(dim)
    dense = out if not _nontrivial_nhwc(out) else Tensor(shape=(_numel(out_shape),), dtype=x.dtype, device=x.device)
    env.lib.sum_strided_f32(x, dense, len(kept), [x.shape[i] for i in kept], [xs[i] for i in kept],
                            len(red), [x.shape[i] for i in red], [xs[i] for i in red], float(scale), st)
    if dense is not out:
        n, c, h, w = out_shape
        env.lib.nchw_to_nhwc_f32(dense, out, n, c, h, w, st)
    return out


@_reg("cuda", "sum_scale_backward")
def cuda_sum_scale_backward(output_grad, x, dim, keepdim, scale):
    env = _env(x)
    dim = tuple(dim)
    dx = _new(x.shape, x)
    st = env.stream()
    if x._nhwc and dim == (2, 3):
        n, c, h, w = x.shape
        env.lib.nhwc_spatial_bcast_f32(output_grad, dx, n, c, h * w, float(scale), st)
        return [dx]
    gs = _strides(output_grad)
    if keepdim:
        src = [0 if i in dim else gs[i] for i in range(len(x.shape))]
    else:
        it = iter(gs)
        src = [0 if i in dim else next(it) for i in range(len(x.shape))]
    env.lib.binary_strided_f32(5, len(x.shape), x.shape, src, src, _strides(dx), output_grad, None,
                               dx, float(scale), st)
    return [dx]


# ---------------------------------------------------------------------------- shape ops

def _dense_copy(env, t):
    """Logical row-major copy of a channels-last tensor."""
    n, c, h, w = t.shape
    out = CudaMemory(t.device.index, t._native_array.nbytes)
    env.lib.nhwc_to_nchw_f32(t, out, n, c, h, w, env.stream())
    return out


@_reg("cuda", "reshape")
def cuda_reshape(x, shape):
    env = _env(x)
    new_shape = calculate_reshaped_shape(x.shape, shape)
    new_shape = tuple(new_shape)
    mem = x._native_array
    if _nontrivial_nhwc(x):
        mem = _dense_copy(env, x)
    out = _on_device(new_shape, x.dtype, x.device, mem)
    if _nontrivial_nhwc(out):
        n, c, h, w = new_shape
        dst = CudaMemory(x.device.index, mem.nbytes)
        env.lib.nchw_to_nhwc_f32(mem, dst, n, c, h, w, env.stream())
        out._native_array = dst
    return out


@_reg("cuda", "permute")
def cuda_permute(x, dims):
    _f32(x)
    env = _env(x)
    out = _new(tuple(x.shape[d] for d in dims), x)
    xs = _strides(x)
    src = [xs[d] for d in dims]
    env.lib.binary_strided_f32(5, len(dims), out.shape, src, src, _strides(out), x, None, out, 1.0,
                               env.stream())
    return out


@_reg("cuda", "permute_backward")
def cuda_permute_backward(output_grad, x, dims):
    inverse = [0] * len(dims)
    for i, d in enumerate(dims):
        inverse[d] = i
    return [cuda_permute(output_grad, tuple(inverse))]


# ---------------------------------------------------------------------------- loss

@_reg("cuda", "cross_entropy")
def cuda_cross_entropy(input, target):
    if target.dtype is not int64:
        raise InvalidDataTypeError(target.dtype)
    _f32(input)
    env = _env(input)
    b, c = input.shape
    loss = _new((1,), input)
    ws, ws_bytes = env.workspace(env.lib.cross_entropy_workspace_bytes(b))
    env.lib.cross_entropy_forward_f32(b, c, input, target, loss, ws, ws_bytes, env.stream())
    return loss


@_reg("cuda", "cross_entropy_backward")
def cuda_cross_entropy_backward(output_grad, input, target):
    env = _env(input)
    b, c = input.shape
    dx = _new(input.shape, input)
    env.lib.cross_entropy_backward_f32(b, c, input, target, output_grad, dx, env.stream())
    return [dx]


# ---------------------------------------------------------------------------- optimiser

def _refuse_first_step_in_capture(env, is_first_time):
    """A captured first step would bake "momentum buffer = gradient" into the graph and every replay
    would reset the momentum; the momentum buffers must exist (one eager step) before capture."""
    if is_first_time and env.capturing():
        raise RuntimeError("optimizer state does not exist yet: run one eager optimizer step before capturing the step in a CUDA graph")


@_reg("cuda", "sgd")
def cuda_sgd(param, momentum_buffer, is_first_time, lr, weight_decay, momentum, dampening, nesterov, maximize):
    env = _env(param)
    _refuse_first_step_in_capture(env, is_first_time)
    env.lib.sgd_f32(param, param.grad, momentum_buffer, _numel(param.shape), int(bool(is_first_time)), float(lr),
                    float(weight_decay), float(momentum), float(dampening), int(bool(nesterov)), int(bool(maximize)), 1.0, env.stream())


@_reg("cuda", "sgd_multi")
def cuda_sgd_multi(entries, lr, weight_decay, momentum, dampening, nesterov, maximize, grad_scale=1.0):
    """entries: [(param, momentum_buffer, is_first_time)]; one launch per 96 tensors."""
    if not entries:
        return
    env = _env(entries[0][0])
    _refuse_first_step_in_capture(env, any([f for _, _, f in entries]))
    _binding.sgd_step(list(entries), lr, weight_decay, momentum, dampening, bool(nesterov), bool(maximize), grad_scale, env.stream())
