"""CUDA runtime glue: the kernel library (a CPython binding of its C ABI), device memory, streams, events.

Plays the role of the reference's ``mytorch/backends/cuda/env.py`` (library loader
``:341-393``, ``CudaMemory`` ``:524-561``, ``allocate_memory`` / ``transfer_memory``
``:564-580``) and ``memory_allocator.py:16-51``.  Everything comes from ``libmytorch_b200.so``:
the arithmetic kernels and the runtime around them (a size-keyed device memory pool whose blocks
keep their addresses from step to step, asynchronous copies, one compute stream per device,
events, whole-step graph capture).  This module imports neither PyTorch nor any other CUDA
binding; ``mytorch_b200.parallel`` alone uses ``torch.distributed`` for the NCCL all-reduce.

There is no fallback: if the library is missing or the device is not sm_100, the first CUDA
operation raises.
"""
from __future__ import annotations

import ctypes
import importlib.machinery
import importlib.util
import os

import numpy as np

from mytorch_b200.backends.backend_dispatcher import BackendDispatcher

LIBRARY_PATH = os.environ.get(
    "MYTORCH_B200_LIB",
    os.path.join(os.path.dirname(os.path.dirname(os.path.dirname(os.path.abspath(__file__)))), "lib", "libmytorch_b200.so"),
)
BINDING_PATH = os.path.join(os.path.dirname(os.path.dirname(os.path.dirname(os.path.abspath(__file__)))), "lib", "_mtb_binding.so")


class NativeError(RuntimeError):
    pass


def _load_binding():
    """The CPython binding of the C ABI (``csrc/binding.cpp``), or None when it has not been built."""
    if not os.path.exists(BINDING_PATH):
        return None
    loader = importlib.machinery.ExtensionFileLoader("_mtb_binding", BINDING_PATH)
    module = importlib.util.module_from_spec(importlib.util.spec_from_loader("_mtb_binding", loader))
    loader.exec_module(module)
    return module


_binding = _load_binding()
# every entry point the Python layer binds (argument types come from the public header, compiled into the binding)
_SIGNATURES = _binding.entry_points if _binding is not None else ()


class NativeLibrary:
    """The entry points of ``libmytorch_b200.so`` as attributes, without their ``mtb_`` prefix; a call raises on a
    non-zero status (or a NULL pointer from the entry points that return one).  Pointer arguments are None,
    addresses, ``CudaMemory`` blocks or tensors; those that the header calls HOST are None, addresses or ctypes storage
    (arrays, ``byref``), shapes and strides also tuples or lists."""

    def __init__(self, path=LIBRARY_PATH):
        if not os.path.exists(path) or _binding is None:
            missing = path if not os.path.exists(path) else BINDING_PATH
            raise NativeError(
                f"kernel library not found at {missing}; build it with `python -m mytorch_b200.build` "
                "(there is no fallback implementation)")
        _binding.load(path, NativeError)
        for name in _SIGNATURES:
            setattr(self, name[4:], getattr(_binding, name[4:]))

    @property
    def launches(self):
        """Calls so far of entry points that enqueue kernels."""
        return _binding.launches()

    def exported(self, name):
        return name in _SIGNATURES


class Event:
    """A CUDA event (``timing=True`` to measure elapsed time between two of them)."""

    def __init__(self, timing=False):
        self._lib = CudaEnv.instance().lib
        self.handle = self._lib.event_create(int(bool(timing)))

    def record(self, stream=None):
        self._lib.event_record(self.handle, CudaEnv.instance().stream() if stream is None else stream)

    def synchronize(self):
        self._lib.event_synchronize(self.handle)

    def elapsed_ms(self, later):
        ms = ctypes.c_float(0)
        self._lib.event_elapsed_ms(self.handle, later.handle, ctypes.byref(ms))
        return ms.value

    def __del__(self):
        try:
            self._lib.event_destroy(self.handle)
        except Exception:
            pass


class PinnedBuffer:
    """Page-locked host memory, viewed as a NumPy array: copies from it to the device are asynchronous."""

    def __init__(self, shape, np_dtype):
        self._lib = CudaEnv.instance().lib
        self.nbytes = int(np.prod(shape, dtype=np.int64)) * np.dtype(np_dtype).itemsize
        self.ptr = self._lib.host_alloc_pinned(self.nbytes)
        raw = (ctypes.c_ubyte * max(self.nbytes, 1)).from_address(self.ptr)
        self.array = np.frombuffer(raw, dtype=np_dtype, count=int(np.prod(shape, dtype=np.int64))).reshape(shape)

    def __del__(self):
        try:
            self.array = None
            self._lib.host_free_pinned(self.ptr)
        except Exception:
            pass


class CudaEnv:
    """Per-process CUDA state: the library, one compute stream and one grow-only scratch buffer per device."""

    _instance = None

    @classmethod
    def instance(cls):
        if cls._instance is None:
            cls._instance = cls()
        return cls._instance

    def __init__(self):
        self.lib = NativeLibrary()
        count = ctypes.c_int(0)
        try:
            self.lib.device_count(ctypes.byref(count))
        except NativeError as e:
            raise NativeError(f"no CUDA device is available; the cuda backend has no CPU fallback ({e})") from None
        if count.value == 0:
            raise NativeError("no CUDA device is available; the cuda backend has no CPU fallback")
        self.lib.device_check()
        self._scratch = ({}, {})  # per device: of the compute stream, of the side stream
        self._retired_scratch = []
        self._capturing = False
        # weight gradients run beside the rest of backward on a second stream (see fork_side / join_side)
        self._side_streams = {}
        self._side_keepalive = []
        self._side_busy = set()
        self._fork_events, self._join_events = {}, {}
        self.overlap_weight_gradients = not os.environ.get("MTB_SERIAL_WGRAD")
        from mytorch_b200.autograd import DAGTracker
        from mytorch_b200.dtype import float32
        from mytorch_b200.tensor import Tensor

        # Every operator asks for these, so they are native (csrc/binding.cpp):
        self.stream = _binding.stream  # () -> the compute stream of the current device: every operator enqueues its work there
        # (nbytes) -> (address, bytes) of scratch for kernels that need it (split-K partials, per-CTA reduction partials): one
        # buffer per device, shared by all operators, which run in order on one stream; the side stream has its own
        self.workspace, self.side_workspace = _binding.workspace, _binding.side_workspace
        _binding.set_state(Tensor, float32, CudaMemory, self, self.lib.stream_create, self._grow_scratch)
        DAGTracker.instance().join_hook = self.join_side

    # ---- devices, streams
    def current_device(self):
        return _binding.current_device()

    def set_device(self, index):
        if index is not None and index != _binding.current_device():
            self.lib.set_device(int(index))

    def new_stream(self):
        return self.lib.stream_create()

    def synchronize(self):
        self.lib.device_synchronize()

    def capturing(self):
        return self._capturing

    def mem_get_info(self):
        free, total = ctypes.c_longlong(0), ctypes.c_longlong(0)
        self.lib.mem_get_info(ctypes.byref(free), ctypes.byref(total))
        return free.value, total.value

    def tensor_core_status(self):
        """Synchronises and returns the status word of the tensor-core kernels (0 = fine; non-zero
        = a bounded wait inside a kernel ran out and the kernel gave up).  Reading clears it."""
        out = ctypes.c_int(0)
        self.lib.tc_status(ctypes.byref(out))
        return out.value

    # ---- a second stream for work nothing on the compute stream waits for until backward ends
    def fork_side(self, keepalive=()):
        """The side stream of the current device, ordered after everything enqueued on the compute
        stream so far.  ``keepalive``: objects whose device memory the side-stream work reads or writes;
        they are held until ``join_side`` so that the pool cannot hand their blocks to compute-stream
        work while the side stream still uses them."""
        dev = self.current_device()
        side = self._side_streams.get(dev)
        if side is None:
            side = self._side_streams[dev] = self.lib.stream_create()
        # one event per device is enough: a wait refers to the record that precedes it, later records do not move it
        ev = self._fork_events.get(dev)
        if ev is None:
            ev = self._fork_events[dev] = Event()
        self.lib.event_record(ev.handle, self.stream())
        self.lib.stream_wait_event(side, ev.handle)
        self._side_keepalive.extend(keepalive)
        self._side_busy.add(dev)
        return side

    def side_event(self):
        """An event after everything enqueued so far on the current device's side stream (None if idle):
        a third stream that consumes side-stream results (the gradient all-reduce) waits on it directly,
        without making the compute stream wait."""
        dev = self.current_device()
        if dev not in self._side_busy:
            return None
        ev = Event()
        ev.record(self._side_streams[dev])
        return ev

    def join_side(self):
        """Make the compute stream of every device wait for its side stream; release the kept objects."""
        if not self._side_busy:
            return
        current = self.current_device()
        for dev in list(self._side_busy):
            self.set_device(dev)
            ev = self._join_events.get(dev)
            if ev is None:
                ev = self._join_events[dev] = Event()
            self.lib.event_record(ev.handle, self._side_streams[dev])
            self.lib.stream_wait_event(self.stream(), ev.handle)
        self.set_device(current)
        self._side_busy.clear()
        self._side_keepalive.clear()

    # ---- memory
    def _grow_scratch(self, which, nbytes):
        table, dev = self._scratch[which], self.current_device()
        buf = table.get(dev)
        if buf is None or buf.nbytes < nbytes:
            if buf is not None:
                # a captured graph may hold this block's address: it is kept for the life of the
                # process so that the pool can never hand it to a tensor a replay would overwrite
                self._retired_scratch.append(buf)
            buf = CudaMemory(dev, max(int(nbytes), 1 << 20))
            table[dev] = buf
        return buf.ptr, buf.nbytes


if _binding is not None:
    _binding.on_first_use(CudaEnv.instance)


class CudaMemory(_binding.Block if _binding is not None else object):
    """A device allocation from the library's pool (``CudaMemory(device_index, nbytes)``; allocation, ``destroy`` and
    the release when the object goes away are native, see ``csrc/binding.cpp``). ``ptr`` is the raw device address,
    ``nbytes`` and ``device_index`` say how much and where; ``read`` / ``write`` move bytes between it and NumPy
    arrays without interpreting any layout."""

    __slots__ = ()

    def read(self, shape, np_dtype):
        env = CudaEnv.instance()
        env.join_side()  # a host read must see what the side stream has produced, too
        env.set_device(self.device_index)
        out = np.empty(shape, dtype=np_dtype)
        env.lib.memcpy_d2h_async(out.ctypes.data, self.ptr, out.nbytes, env.stream())
        env.lib.stream_synchronize(env.stream())
        return out

    def write(self, array):
        """Copy a NumPy array in (pageable memory: the call returns once the bytes are staged)."""
        env = CudaEnv.instance()
        env.set_device(self.device_index)
        a = np.ascontiguousarray(array)
        env.lib.memcpy_h2d_async(self.ptr, a.ctypes.data, a.nbytes, env.stream())
        env.lib.stream_synchronize(env.stream())

    def write_from(self, host, stream=None):
        """Asynchronous copy from host memory that stays valid until the copy has run: a NumPy array
        (page-locked, e.g. ``PinnedBuffer.array``, for a truly asynchronous copy) or any object with
        ``data_ptr()`` / ``numel()`` / ``element_size()`` (a pinned PyTorch CPU tensor)."""
        env = CudaEnv.instance()
        env.set_device(self.device_index)
        src, nbytes = host_pointer(host)
        env.lib.memcpy_h2d_async(self.ptr, src, min(nbytes, self.nbytes), env.stream() if stream is None else stream)

    def copy_from(self, other, nbytes=None):
        env = CudaEnv.instance()
        env.set_device(self.device_index)
        env.lib.memcpy_d2d_async(self.ptr, other.ptr, self.nbytes if nbytes is None else nbytes, env.stream())


def host_pointer(host):
    """(address, bytes) of a contiguous host buffer: NumPy array or an object with ``data_ptr()``."""
    if hasattr(host, "data_ptr"):
        return host.data_ptr(), host.numel() * host.element_size()
    if not host.flags["C_CONTIGUOUS"]:
        raise ValueError("host buffer must be contiguous")
    return host.ctypes.data, host.nbytes


@BackendDispatcher.instance().register_backend_function("cuda", "allocate_memory")
def cuda_allocate_memory(device_index, nbytes):
    return CudaMemory(device_index, nbytes)


@BackendDispatcher.instance().register_backend_function("cuda", "transfer_memory")
def cuda_transfer_memory(dst, src):
    dst.copy_from(src, src.nbytes)


class CudaMemoryView(CudaMemory):
    """A window into another allocation (used for gradient tensors that live inside one flat
    all-reduce buffer). Keeps the parent alive; frees nothing."""

    __slots__ = ("_parent",)

    def __init__(self, parent, offset_bytes, nbytes, device_index):
        self.device_index = parent.device_index if device_index is None else device_index
        self.nbytes = int(nbytes)
        self._parent = parent
        self.ptr = parent.ptr + int(offset_bytes)
