"""What the binding takes where an entry point wants device memory, and where it wants host memory.  Calls over no
elements: they return before they would need a GPU."""
import ctypes

import numpy as np
import pytest

from mytorch_b200.backends.cuda.env import LIBRARY_PATH, NativeError, _binding

ADDRESS = 1 << 20  # never dereferenced


@pytest.fixture(scope="module")
def lib():
    _binding.load(LIBRARY_PATH, NativeError)
    return _binding


@pytest.mark.parametrize("address", [None, 0, ADDRESS, ctypes.c_void_p(ADDRESS), ctypes.cast(ADDRESS, ctypes.POINTER(ctypes.c_float))])
def test_addresses_are_device_memory(lib, address):
    assert lib.fill_f32(address, 0, 1.0, None) == 0 and lib.copy_f32(address, address, 0, address) == 0


@pytest.mark.parametrize("storage", [np.zeros(4, np.float32), np.int64(ADDRESS), np.zeros((), np.int64), (ctypes.c_float * 4)(),
                                     ctypes.byref(ctypes.c_float()), ctypes.c_longlong(ADDRESS), b"bytes", bytearray(8), memoryview(bytes(8)),
                                     (1, 2), [1, 2], 1.0, "text", object()], ids=lambda s: type(s).__name__)
def test_host_storage_is_no_device_memory(lib, storage):
    for call in (lambda: lib.fill_f32(storage, 0, 1.0, None), lambda: lib.fill_f32(None, 0, 1.0, storage),
                 lambda: lib.cross_entropy_forward_f32(4, 10, ADDRESS, storage, ADDRESS, ADDRESS, 1 << 20, None)):
        with pytest.raises(TypeError):
            call()


def test_host_arguments(lib):
    shape = (ctypes.c_longlong * 2)(0, 3)
    for dims in ((0, 3), [0, 3], shape, ctypes.byref(shape), ctypes.addressof(shape), ctypes.cast(shape, ctypes.POINTER(ctypes.c_longlong))):
        assert lib.eq_strided(0, 2, dims, dims, dims, ADDRESS, ADDRESS, ADDRESS, None) == 0
    for wrong in (np.zeros(2, np.int64), np.int64(ADDRESS), 1.0, object()):
        with pytest.raises((TypeError, ctypes.ArgumentError)):
            lib.eq_strided(0, 2, wrong, (0, 3), (0, 3), ADDRESS, ADDRESS, ADDRESS, None)
    plan = (ctypes.c_int * 27)()  # one past the end on either side stays untouched
    plan[0] = plan[26] = -7
    lib.conv2d_plan_f32(64, 64, 32, 32, 3, 3, 1, 1, 1, 1, 64, ctypes.byref(plan, 4))
    assert plan[0] == plan[26] == -7 and any(plan[1:26])


def test_header_and_binding_agree_on_host_arguments(lib):
    """The binding's list against the public header: parameters of HOST kind are the ones the header's comments name."""
    import os
    import re

    from conftest import ROOT

    names = {"shape", "x_strides", "y_strides", "z_strides", "kept_shape", "kept_strides", "red_shape", "red_strides", "params", "grads",
             "momentum_buffers", "sizes", "is_first", "srcs", "offsets", "stats_rows", "status_out", "device", "count", "free_bytes",
             "total_bytes", "src_host", "dst_host", "ms", "graph_exec_out"}
    text = re.sub(r"/\*.*?\*/", " ", open(os.path.join(ROOT, "include", "mytorch_b200.h")).read(), flags=re.S)
    source = open(os.path.join(ROOT, "mytorch_b200", "csrc", "binding.cpp")).read()
    entries = dict(re.findall(r"X\((\w+), [A-Z]+, (0|HOST\([^)]*\))\)", source))
    checked = 0
    for name, params in re.findall(r"\bmtb_(\w+)\(([^()]*)\);", text):
        if name not in entries:
            continue
        host = [i for i, p in enumerate(params.split(",")) if "*" in p and
                (p.split()[-1].lstrip("*") in names or (name, p.split()[-1].lstrip("*")) in {("conv2d_plan_f32", "out"), ("host_free_pinned", "ptr")})]
        assert host == ([] if entries[name] == "0" else [int(v) for v in re.findall(r"\d+", entries[name])]), name
        checked += 1
    assert checked == len(entries) == len(_binding.entry_points)
