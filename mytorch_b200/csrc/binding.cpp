// CPython binding of the C ABI: one vectorcall function per entry point, and the device-memory object.
//
// What bounds it: a training step issued operator by operator makes about 300 library calls, and a step of a
// small network is over in a fraction of a millisecond on the GPU, so the host's cost per call IS the step time.
// Through ctypes one call of the convolution entry points (18 arguments) took 3-4 us, an allocation plus its
// release 3.5 us.  Here the argument conversion is compiled per signature (taken from the public header, so the
// two cannot drift apart), and a device block is a C object whose constructor and destructor call the pool
// directly.  Host time to enqueue a step, before and after: the MNIST example at 64 images 1100 -> 616 us, ResNet-18
// training 3230 -> 1530 us, ResNet-18 inference 1070 -> 408 us (with leaner tensor construction and tape loops).
//
// Nothing here touches CUDA: the kernel library is opened at run time (load()), so importing this module needs
// neither a GPU nor the driver.
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <dlfcn.h>
#include <structmember.h>

#include <string>
#include <cstring>
#include <tuple>
#include <type_traits>
#include <utility>
#include <vector>

#include "../../include/mytorch_b200.h"

namespace {

PyObject* g_error = nullptr;  // NativeError, handed over by load()
PyObject* g_first_use = nullptr;  // called when memory is asked for before load(): sets the CUDA state up or raises
const char* (*g_last_error)() = nullptr;

// Handed over by the Python layer when its CUDA state exists (set_state).
PyTypeObject *g_tensor_type = nullptr, *g_memory_type = nullptr;
PyObject *g_float32 = nullptr, *g_env = nullptr, *g_make_stream = nullptr, *g_grow_scratch = nullptr;
#define MTB_NAMES(X) X(shape) X(dtype) X(device) X(index) X(_nhwc) X(_native_array) X(_itemsize) X(grad)
#define X(n) PyObject* N_##n = nullptr;
MTB_NAMES(X)
#undef X
long long g_launches = 0;

// ------------------------------------------------------------------ device memory

struct Block {
  PyObject_HEAD
  unsigned long long ptr;
  long long nbytes;
  int device_index;
  char owned;  // a view of another block owns nothing
};
PyTypeObject BlockType = {PyVarObject_HEAD_INIT(nullptr, 0)};

// ------------------------------------------------------------------ argument conversion

inline bool from_py(PyObject* o, int& v) {
  const long x = PyLong_AsLong(o);
  if (x == -1 && PyErr_Occurred()) return false;
  if (x != (int)x) { PyErr_SetString(PyExc_OverflowError, "argument does not fit a C int"); return false; }
  v = (int)x;
  return true;
}
inline bool from_py(PyObject* o, long long& v) {
  v = PyLong_AsLongLong(o);
  return !(v == -1 && PyErr_Occurred());
}
inline bool from_py(PyObject* o, double& v) {
  v = PyFloat_AsDouble(o);
  return !(v == -1.0 && PyErr_Occurred());
}
inline bool from_py(PyObject* o, float& v) {
  double d;
  if (!from_py(o, d)) return false;
  v = (float)d;
  return true;
}

// ctypes, for the objects that hold or describe an address (imported on the first of them).
struct CTypes {
  PyObject *cast, *c_void_p, *pointer, *array;
};
const CTypes* ctypes() {
  static CTypes c{};
  if (!c.array) {
    PyObject* m = PyImport_ImportModule("ctypes");
    if (!m) return nullptr;
    c.cast = PyObject_GetAttrString(m, "cast");
    c.c_void_p = PyObject_GetAttrString(m, "c_void_p");
    c.pointer = PyObject_GetAttrString(m, "_Pointer");
    c.array = PyObject_GetAttrString(m, "Array");
    Py_DECREF(m);
    if (!c.cast || !c.c_void_p || !c.pointer || !c.array) { c.array = nullptr; return nullptr; }
  }
  return &c;
}
bool ctypes_address(const CTypes& c, PyObject* o, void*& v) {  // refuses what a c_void_p argument refuses
  PyObject* p = PyObject_CallFunctionObjArgs(c.cast, o, c.c_void_p, nullptr);
  PyObject* value = p ? PyObject_GetAttrString(p, "value") : nullptr;
  Py_XDECREF(p);
  if (!value) return false;
  v = value == Py_None ? nullptr : PyLong_AsVoidPtr(value);
  Py_DECREF(value);
  return !PyErr_Occurred();
}

// Where the header says HOST: None, an integer, or ctypes storage (an array, byref(x), a pointer); for shapes and strides
// also a tuple or list.
bool host_address(PyObject* o, void*& v) {
  const CTypes* c = ctypes();
  if (!c) return false;
  const int array = PyObject_IsInstance(o, c->array);
  if (array <= 0) return array == 0 && ctypes_address(*c, o, v);
  Py_buffer view;
  if (PyObject_GetBuffer(o, &view, PyBUF_SIMPLE)) return false;
  v = view.buf;
  PyBuffer_Release(&view);  // the caller's argument keeps the storage alive during the call
  return true;
}
// Everywhere else (device memory, streams, events, graphs): None, an integer, a block, a tensor, or a ctypes pointer's value.
// Anything that merely has storage is host memory, which a kernel must not be given.
bool device_address(PyObject* o, void*& v) {
  if (PyObject_TypeCheck(o, &BlockType)) { v = (void*)((Block*)o)->ptr; return true; }
  if (g_tensor_type && PyObject_TypeCheck(o, g_tensor_type)) {
    PyObject* memory = PyObject_GetAttr(o, N__native_array);
    if (!memory) return false;
    const bool block = PyObject_TypeCheck(memory, &BlockType);
    v = block ? (void*)((Block*)memory)->ptr : nullptr;
    Py_DECREF(memory);  // the tensor holds it
    // not NULL: an optional operand (a bias, running statistics) would be taken as absent
    if (!block) PyErr_SetString(PyExc_TypeError, "a tensor without device memory");
    return block;
  }
  const CTypes* c = ctypes();
  if (!c) return false;
  int value = PyObject_IsInstance(o, c->c_void_p);
  if (!value) value = PyObject_IsInstance(o, c->pointer);
  if (value > 0) return ctypes_address(*c, o, v);
  if (value == 0) PyErr_Format(PyExc_TypeError, "device memory, a tensor, an address or None expected, not %.80s", Py_TYPE(o)->tp_name);
  return false;
}

template <bool HOST, class T>
inline bool pointer(PyObject* o, T*& v) {
  if (o == Py_None) { v = nullptr; return true; }
  if (PyLong_Check(o)) {
    v = (T*)PyLong_AsVoidPtr(o);
    return !(v == nullptr && PyErr_Occurred());
  }
  if constexpr (HOST && std::is_same_v<T, const long long>) {
    if (PyTuple_CheckExact(o) || PyList_CheckExact(o)) {
      // shapes and strides: read by the entry point before it returns, so a few slots per thread taken in turn are enough
      constexpr int kSlots = 16, kLength = 64;
      thread_local long long values[kSlots][kLength];
      thread_local int next = 0;
      const Py_ssize_t n = PySequence_Fast_GET_SIZE(o);
      if (n > kLength) { PyErr_SetString(PyExc_ValueError, "too many dimensions"); return false; }
      long long* slot = values[next++ % kSlots];
      for (Py_ssize_t i = 0; i < n; ++i)
        if (!from_py(PySequence_Fast_GET_ITEM(o, i), slot[i])) return false;
      v = slot;
      return true;
    }
  }
  void* p = nullptr;
  if (!(HOST ? host_address(o, p) : device_address(o, p))) return false;
  v = (T*)p;
  return true;
}
// One argument of an entry point; HOST: it is a pointer to host memory.
template <bool HOST, class T>
inline bool argument(PyObject* o, T& v) {
  if constexpr (std::is_pointer_v<T>) return pointer<HOST>(o, v);
  else return from_py(o, v);
}

inline PyObject* to_py(int v) { return PyLong_FromLong(v); }
inline PyObject* to_py(long long v) { return PyLong_FromLongLong(v); }
inline PyObject* to_py(void* v) { return PyLong_FromVoidPtr(v); }

// ------------------------------------------------------------------ one function per entry point

enum Kind {
  LAUNCH,   // status; counted as work enqueued on the GPU
  STATUS,   // status; bookkeeping
  POINTER,  // NULL means failure
  VALUE,    // host arithmetic: the result itself
};

PyObject* raise_native(const char* name, int rc) {
  if (rc) PyErr_Format(g_error, "%s failed (%d): %s", name, rc, g_last_error());
  else PyErr_Format(g_error, "%s failed: %s", name, g_last_error());
  return nullptr;
}

template <int ID, Kind K, unsigned HOST, class Sig>
struct Entry;
template <int ID, Kind K, unsigned HOST, class R, class... A>
struct Entry<ID, K, HOST, R(A...)> {
  static inline R (*fn)(A...) = nullptr;
  static inline const char* name = nullptr;

  template <size_t... I>
  static PyObject* invoke(PyObject* const* args, std::index_sequence<I...>) {
    std::tuple<A...> a;
    if (!(argument<(HOST >> I & 1u) != 0>(args[I], std::get<I>(a)) && ... && true)) return nullptr;
    if constexpr (K == VALUE) {
      return to_py(fn(std::get<I>(a)...));
    } else {
      // released: a launch waits when the stream's queue is full, and other Python threads feed it meanwhile
      R r;
      Py_BEGIN_ALLOW_THREADS
      r = fn(std::get<I>(a)...);
      Py_END_ALLOW_THREADS
      if constexpr (K == POINTER) {
        if (!r) return raise_native(name, 0);
      } else {
        if (r) return raise_native(name, r);
        if (K == LAUNCH) ++g_launches;
      }
      return to_py(r);
    }
  }
  static PyObject* call(PyObject*, PyObject* const* args, Py_ssize_t n) {
    if (!fn) { PyErr_SetString(PyExc_RuntimeError, "the kernel library is not loaded"); return nullptr; }
    if (n != (Py_ssize_t)sizeof...(A)) {
      PyErr_Format(PyExc_TypeError, "%s takes %zu arguments (%zd given)", name, sizeof...(A), n);
      return nullptr;
    }
    return invoke(args, std::index_sequence_for<A...>{});
  }
};

// name, kind, and which arguments (counted from 0) the public header calls HOST memory
template <class... I>
constexpr unsigned HOST(I... i) { return (0u | ... | (1u << i)); }
#define MTB_ENTRIES(X) \
  X(version, VALUE, 0) X(device_check, STATUS, 0) X(fill_f32, LAUNCH, 0) X(copy_f32, LAUNCH, 0) X(scale_f32, LAUNCH, 0) \
  X(relu_forward_f32, LAUNCH, 0) X(relu_backward_f32, LAUNCH, 0) X(add_f32, LAUNCH, 0) X(mul_f32, LAUNCH, 0) \
  X(add_bias_rows_f32, LAUNCH, 0) X(binary_strided_f32, LAUNCH, HOST(2, 3, 4, 5)) X(resize_channels_f32, LAUNCH, 0) \
  X(pack_patches_f32, LAUNCH, 0) X(nchw_to_nhwc_f32, LAUNCH, 0) X(nhwc_to_nchw_f32, LAUNCH, 0) X(cast, LAUNCH, 0) \
  X(batch_norm2d_workspace_bytes, VALUE, 0) X(batch_norm2d_forward_f32, LAUNCH, 0) X(batch_norm2d_backward_f32, LAUNCH, 0) \
  X(batch_norm2d_relu_pool_forward_f32, LAUNCH, 0) X(batch_norm2d_relu_pool_backward_f32, LAUNCH, 0) X(batch_norm2d_add_relu_forward_f32, LAUNCH, 0) X(batch_norm2d_add_relu_forward_masked_f32, LAUNCH, 0) \
  X(batch_norm2d_add_relu_backward_masked_f32, LAUNCH, 0) X(batch_norm2d_add_relu_backward_f32, LAUNCH, 0) X(add_relu_f32, LAUNCH, 0) \
  X(add_relu_backward_f32, LAUNCH, 0) X(colsum_workspace_bytes, VALUE, 0) X(colsum_f32, LAUNCH, 0) X(colsum_noalloc_f32, LAUNCH, 0) \
  X(nhwc_spatial_sum_f32, LAUNCH, 0) X(nhwc_spatial_bcast_f32, LAUNCH, 0) X(sum_strided_f32, LAUNCH, HOST(3, 4, 6, 7)) \
  X(max_strided_f32, LAUNCH, HOST(4, 5)) X(max_backward_f32, LAUNCH, HOST(5, 6)) X(eq_strided, LAUNCH, HOST(2, 3, 4)) \
  X(max_pool2d_forward_f32, LAUNCH, 0) X(max_pool2d_backward_f32, LAUNCH, 0) X(max_pool2d_argmax_u8, LAUNCH, 0) \
  X(cross_entropy_workspace_bytes, VALUE, 0) X(cross_entropy_forward_f32, LAUNCH, 0) X(cross_entropy_backward_f32, LAUNCH, 0) \
  X(sgd_f32, LAUNCH, 0) X(sgd_multi_f32, LAUNCH, HOST(1, 2, 3, 4, 5)) X(pack_scale_f32, LAUNCH, HOST(1, 2, 3)) \
  X(conv2d_workspace_bytes, VALUE, 0) X(conv2d_plan_f32, STATUS, HOST(11)) X(conv2d_pair_plan_f32, STATUS, HOST(11)) X(conv2d_pair_choice_f32, STATUS, HOST(11)) X(conv2d_pair_smem_bytes, VALUE, 0) X(conv2d_forward_f32, LAUNCH, 0) \
  X(conv2d_stats_max_rows, VALUE, 0) X(conv2d_forward_stats_f32, LAUNCH, HOST(17)) X(conv2d_bn_forward_f32, LAUNCH, 0) X(conv2d_bn_pool_takes, VALUE, 0) X(conv2d_bn_pool_scratch_bytes, VALUE, 0) X(conv2d_bn_pool_forward_f32, LAUNCH, 0) \
  X(batch_norm2d_forward_prestats_f32, LAUNCH, 0) X(conv2d_dgrad_f32, LAUNCH, 0) X(conv2d_dgrad_add_f32, LAUNCH, 0) \
  X(conv2d_dgrad_accumulates_in_place, VALUE, 0) X(conv2d_wgrad_f32, LAUNCH, 0) X(gemm_f32, LAUNCH, 0) X(linear_relu_f32, LAUNCH, 0) X(tc_status, STATUS, HOST(0)) \
  X(tc_wait_selftest, LAUNCH, 0) X(malloc, POINTER, 0) X(free, STATUS, 0) X(malloc_if_ready, VALUE, 0) \
  X(free_if_ready, VALUE, 0) X(pool_reserved_bytes, VALUE, 0) X(pool_in_use_bytes, VALUE, 0) \
  X(pool_trim, STATUS, 0) X(set_device, STATUS, 0) X(get_device, STATUS, HOST(0)) X(device_count, STATUS, HOST(0)) \
  X(device_synchronize, STATUS, 0) X(mem_get_info, STATUS, HOST(0, 1)) X(memcpy_h2d_async, STATUS, HOST(1)) \
  X(memcpy_d2h_async, STATUS, HOST(0)) X(memcpy_d2d_async, STATUS, 0) X(memset_async, STATUS, 0) X(host_alloc_pinned, POINTER, 0) \
  X(host_free_pinned, STATUS, HOST(0)) X(stream_create, POINTER, 0) X(stream_destroy, STATUS, 0) X(stream_synchronize, STATUS, 0) \
  X(stream_wait_event, STATUS, 0) X(event_create, POINTER, 0) X(event_destroy, STATUS, 0) X(event_record, STATUS, 0) \
  X(event_synchronize, STATUS, 0) X(event_elapsed_ms, STATUS, HOST(2)) X(graph_begin_capture, STATUS, 0) \
  X(graph_end_capture, STATUS, HOST(1)) X(graph_launch, STATUS, 0) X(graph_destroy, STATUS, 0)

#define X(n, k, h) ID_##n,
enum EntryId { MTB_ENTRIES(X) kEntries };
#undef X
#define X(n, k, h) using E_##n = Entry<ID_##n, k, h, std::remove_pointer_t<decltype(&mtb_##n)>>;
MTB_ENTRIES(X)
#undef X

// ------------------------------------------------------------------ Block

// The Python layer's CUDA state exists (created on the first use), or an exception is set.
bool ready() {
  if (g_env) return true;
  PyObject* r = g_first_use ? PyObject_CallNoArgs(g_first_use) : nullptr;
  if (!r) {
    if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, "the kernel library is not loaded");
    return false;
  }
  Py_DECREF(r);
  if (!g_env) { PyErr_SetString(PyExc_RuntimeError, "the kernel library is not loaded"); return false; }
  return true;
}
// Make `device` (an index, or None: the current one) the current device.
bool enter_device(PyObject* device, int& want) {
  int current = 0;
  if (int rc = E_get_device::fn(&current)) { raise_native("mtb_get_device", rc); return false; }
  want = current;
  if (device != Py_None && !from_py(device, want)) return false;
  if (want != current)
    if (int rc = E_set_device::fn(want)) { raise_native("mtb_set_device", rc); return false; }
  return true;
}
// The interpreter is let go of where the pool would wait or grow (milliseconds in the driver): other threads, a data
// loader's, run meanwhile.  Letting go on every call: a step of the MNIST example 366 us instead of 362.
void give_back(unsigned long long ptr) {
  if (E_free_if_ready::fn((void*)ptr)) return;
  Py_BEGIN_ALLOW_THREADS
  E_free::fn((void*)ptr);
  Py_END_ALLOW_THREADS
}
bool block_allocate(Block* b, PyObject* device, long long nbytes) {
  int want = 0;
  if (!ready() || !enter_device(device, want)) return false;
  void* p = E_malloc_if_ready::fn(nbytes > 0 ? nbytes : 1);
  if (!p) {
    Py_BEGIN_ALLOW_THREADS
    p = E_malloc::fn(nbytes > 0 ? nbytes : 1);
    Py_END_ALLOW_THREADS
  }
  if (!p) { raise_native("mtb_malloc", 0); return false; }
  if (b->owned && b->ptr) give_back(b->ptr);
  b->ptr = (unsigned long long)p;
  b->nbytes = nbytes;
  b->device_index = want;
  b->owned = 1;
  return true;
}
int block_init(PyObject* self, PyObject* args, PyObject* kwargs) {
  static const char* names[] = {"device_index", "nbytes", nullptr};
  PyObject* device = nullptr;
  long long nbytes = 0;
  if (!PyArg_ParseTupleAndKeywords(args, kwargs, "OL", (char**)names, &device, &nbytes)) return -1;
  return block_allocate((Block*)self, device, nbytes) ? 0 : -1;
}
void block_release(Block* b) {
  const unsigned long long ptr = b->owned && E_free::fn ? b->ptr : 0;
  b->ptr = 0;  // first: another thread may see the block while the pool is asked
  b->owned = 0;
  if (ptr) give_back(ptr);
}
void block_dealloc(PyObject* self) {
  block_release((Block*)self);
  Py_TYPE(self)->tp_free(self);
}
PyObject* block_destroy(PyObject* self, PyObject*) {
  block_release((Block*)self);
  Py_RETURN_NONE;
}
PyMemberDef block_members[] = {
    {"ptr", T_ULONGLONG, offsetof(Block, ptr), 0, "device address"},
    {"nbytes", T_LONGLONG, offsetof(Block, nbytes), 0, "size in bytes"},
    {"device_index", T_INT, offsetof(Block, device_index), 0, "device the block lives on"},
    {nullptr, 0, 0, 0, nullptr}};
PyMethodDef block_methods[] = {{"destroy", block_destroy, METH_NOARGS, "Give the block back to the pool now."}, {nullptr, nullptr, 0, nullptr}};

// ------------------------------------------------------------------ what every operator wrapper does
//
// A training step makes about 50 result tensors and as many stream and scratch look-ups; in Python these were a quarter of
// the host time of a small step (0.9 us for a result with its block, 0.4 us for a stream).  With them, the optimiser's
// tables and the shape tuples converted here, and no gradients towards constants: the MNIST example's step at 64 images
// 393 -> 336 us, a three-layer perceptron's at 1000 rows 270 -> 172 us, inference of one MNIST image 90 -> 80 us.

struct Ref {  // an owned reference
  PyObject* p;
  explicit Ref(PyObject* q) : p(q) {}
  Ref(const Ref&) = delete;
  ~Ref() { Py_XDECREF(p); }
  operator PyObject*() const { return p; }
};

// new_like(shape, like, dtype=None): an uninitialised tensor on the device of `like` (its dtype unless one is given).
PyObject* new_like(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n < 2 || n > 3 || !PyTuple_Check(args[0])) { PyErr_SetString(PyExc_TypeError, "new_like(shape, like, dtype=None)"); return nullptr; }
  if (!ready()) return nullptr;
  PyObject* shape = args[0];
  Ref device(PyObject_GetAttr(args[1], N_device));
  if (!device) return nullptr;
  Ref dtype(n == 3 && args[2] != Py_None ? (Py_INCREF(args[2]), args[2]) : PyObject_GetAttr(args[1], N_dtype));
  if (!dtype) return nullptr;
  long long bytes = 4;
  if (dtype.p != g_float32) {
    Ref size(PyObject_GetAttr(dtype, N__itemsize));
    if (!size || !from_py(size, bytes)) return nullptr;
  }
  const Py_ssize_t dims = PyTuple_GET_SIZE(shape);
  for (Py_ssize_t i = 0; i < dims; ++i) {
    long long extent;
    if (!from_py(PyTuple_GET_ITEM(shape, i), extent)) return nullptr;
    bytes *= extent;
  }
  Ref index(PyObject_GetAttr(device, N_index));
  if (!index) return nullptr;
  Ref memory(g_memory_type->tp_alloc(g_memory_type, 0));
  if (!memory || !block_allocate((Block*)memory.p, index, bytes)) return nullptr;
  PyObject* t = g_tensor_type->tp_alloc(g_tensor_type, 0);
  if (!t) return nullptr;
  PyObject* nhwc = dtype.p == g_float32 && dims == 4 ? Py_True : Py_False;
  if (PyObject_SetAttr(t, N_shape, shape) < 0 || PyObject_SetAttr(t, N_dtype, dtype) < 0 || PyObject_SetAttr(t, N_device, device) < 0 ||
      PyObject_SetAttr(t, N__nhwc, nhwc) < 0 || PyObject_SetAttr(t, N__native_array, memory) < 0) {
    Py_DECREF(t);
    return nullptr;
  }
  return t;
}

// enter(tensor): make the tensor's device current; returns the CUDA state.
PyObject* enter(PyObject*, PyObject* t) {
  if (!ready()) return nullptr;
  Ref device(PyObject_GetAttr(t, N_device));
  if (!device) return nullptr;
  Ref index(PyObject_GetAttr(device, N_index));
  int current;
  if (!index || !enter_device(index, current)) return nullptr;
  Py_INCREF(g_env);
  return g_env;
}

// Per device: the compute stream, and what the scratch buffers (0: compute stream, 1: side stream) are at the moment.
constexpr int kDevices = 64;
struct DeviceState {
  PyObject* stream = nullptr;
  struct { PyObject* pair = nullptr; long long nbytes = -1; } scratch[2];
} g_devices[kDevices];

DeviceState* device_state() {
  int device = 0;
  if (!ready()) return nullptr;
  if (int rc = E_get_device::fn(&device)) { raise_native("mtb_get_device", rc); return nullptr; }
  if (device < 0 || device >= kDevices) { PyErr_SetString(PyExc_RuntimeError, "device index out of range"); return nullptr; }
  return &g_devices[device];
}

// stream(): the compute stream of the current device, made on the first use.
PyObject* stream(PyObject*, PyObject*) {
  DeviceState* d = device_state();
  if (!d) return nullptr;
  if (!d->stream && !(d->stream = PyObject_CallNoArgs(g_make_stream))) return nullptr;
  Py_INCREF(d->stream);
  return d->stream;
}

// workspace(nbytes): (address, bytes) of at least that much scratch on the current device.
template <int SLOT>
PyObject* workspace(PyObject*, PyObject* nbytes) {
  long long want;
  DeviceState* d = device_state();
  if (!d || !from_py(nbytes, want)) return nullptr;
  auto& s = d->scratch[SLOT];
  if (want > s.nbytes || !s.pair) {
    PyObject* pair = PyObject_CallFunction(g_grow_scratch, "iL", SLOT, want);
    if (!pair) return nullptr;
    if (!PyTuple_Check(pair) || PyTuple_GET_SIZE(pair) != 2 || !from_py(PyTuple_GET_ITEM(pair, 1), s.nbytes)) {
      Py_DECREF(pair);
      if (!PyErr_Occurred()) PyErr_SetString(PyExc_TypeError, "scratch: (address, bytes) expected");
      return nullptr;
    }
    Py_XSETREF(s.pair, pair);
  }
  Py_INCREF(s.pair);
  return s.pair;
}

// sgd_step(entries, lr, weight_decay, momentum, dampening, nesterov, maximize, grad_scale, stream): one update of every
// (parameter, momentum buffer, first time) of the list; the tables that the entry point reads are gathered here.
PyObject* sgd_step(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 9 || !PyList_CheckExact(args[0])) { PyErr_SetString(PyExc_TypeError, "sgd_step takes a list and 8 values"); return nullptr; }
  if (!ready()) return nullptr;
  const Py_ssize_t count = PyList_GET_SIZE(args[0]);
  std::vector<float*> params(count), bufs(count);
  std::vector<const float*> grads(count);
  std::vector<long long> sizes(count);
  std::vector<int> first(count);
  double h[4], scale;
  int nesterov, maximize;
  void* st;
  for (int i = 0; i < 4; ++i)
    if (!from_py(args[1 + i], h[i])) return nullptr;
  if (!from_py(args[5], nesterov) || !from_py(args[6], maximize) || !from_py(args[7], scale) || !pointer<false>(args[8], st)) return nullptr;
  for (Py_ssize_t i = 0; i < count; ++i) {
    PyObject* e = PyList_GET_ITEM(args[0], i);
    if (!PyTuple_CheckExact(e) || PyTuple_GET_SIZE(e) != 3) { PyErr_SetString(PyExc_TypeError, "(parameter, buffer, first) expected"); return nullptr; }
    PyObject* param = PyTuple_GET_ITEM(e, 0);
    Ref grad(PyObject_GetAttr(param, N_grad)), shape(PyObject_GetAttr(param, N_shape));
    if (!grad || !shape || !pointer<false>(param, params[i]) || !pointer<false>((PyObject*)grad, grads[i]) ||
        !pointer<false>(PyTuple_GET_ITEM(e, 1), bufs[i]))
      return nullptr;
    const int is_first = PyObject_IsTrue(PyTuple_GET_ITEM(e, 2));
    if (is_first < 0 || !params[i] || !grads[i] || !bufs[i] || !PyTuple_Check(shape)) { if (!PyErr_Occurred()) PyErr_SetString(PyExc_TypeError, "sgd_step: a parameter without device memory, gradient or buffer"); return nullptr; }
    first[i] = is_first;
    sizes[i] = 1;
    for (Py_ssize_t k = 0; k < PyTuple_GET_SIZE(shape.p); ++k) {
      long long extent;
      if (!from_py(PyTuple_GET_ITEM(shape.p, k), extent)) return nullptr;
      sizes[i] *= extent;
    }
  }
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = E_sgd_multi_f32::fn((int)count, params.data(), grads.data(), bufs.data(), sizes.data(), first.data(), h[0], h[1], h[2], h[3], nesterov, maximize,
                           scale, st);
  Py_END_ALLOW_THREADS
  if (rc) return raise_native("mtb_sgd_multi_f32", rc);
  ++g_launches;
  Py_RETURN_NONE;
}

// set_state(Tensor, float32, CudaMemory, env, make_stream, grow_scratch)
PyObject* set_state(PyObject*, PyObject* args) {
  PyObject *tensor, *f32, *memory, *env, *make, *grow;
  if (!PyArg_ParseTuple(args, "O!OO!OOO", &PyType_Type, &tensor, &f32, &PyType_Type, &memory, &env, &make, &grow)) return nullptr;
  if (!PyType_IsSubtype((PyTypeObject*)memory, &BlockType)) { PyErr_SetString(PyExc_TypeError, "a Block type expected"); return nullptr; }
#define MTB_KEEP(slot, type, value) { Py_INCREF(value); type old = slot; slot = (type)value; Py_XDECREF((PyObject*)old); }
  MTB_KEEP(g_tensor_type, PyTypeObject*, tensor)
  MTB_KEEP(g_memory_type, PyTypeObject*, memory)
  MTB_KEEP(g_float32, PyObject*, f32)
  MTB_KEEP(g_make_stream, PyObject*, make)
  MTB_KEEP(g_grow_scratch, PyObject*, grow)
  MTB_KEEP(g_env, PyObject*, env)
#undef MTB_KEEP
  Py_RETURN_NONE;
}

// ------------------------------------------------------------------ module

// load(path, error_class): open the kernel library and resolve every entry point.
PyObject* load(PyObject*, PyObject* args) {
  const char* path;
  PyObject* error;
  if (!PyArg_ParseTuple(args, "sO", &path, &error)) return nullptr;
  void* dll = dlopen(path, RTLD_NOW | RTLD_LOCAL);
  if (!dll) { PyErr_Format(error, "cannot open %s: %s", path, dlerror()); return nullptr; }
  Py_INCREF(error);
  Py_XSETREF(g_error, error);
  auto find = [&](const char* name) {
    void* p = dlsym(dll, name);
    if (!p) PyErr_Format(error, "%s does not export %s", path, name);
    return p;
  };
  if (!(g_last_error = (decltype(g_last_error))find("mtb_last_error"))) return nullptr;
#define X(n, k, h) \
  E_##n::name = "mtb_" #n; \
  if (!(E_##n::fn = (decltype(E_##n::fn))find("mtb_" #n))) return nullptr;
  MTB_ENTRIES(X)
#undef X
  Py_RETURN_NONE;
}

PyObject* on_first_use(PyObject*, PyObject* f) {
  Py_INCREF(f);
  Py_XSETREF(g_first_use, f);
  Py_RETURN_NONE;
}

// Entry-point calls so far that enqueue kernels.
PyObject* launches(PyObject*, PyObject*) { return PyLong_FromLongLong(g_launches); }

PyObject* current_device(PyObject*, PyObject*) {
  int device = 0;
  if (!E_get_device::fn) { PyErr_SetString(PyExc_RuntimeError, "the kernel library is not loaded"); return nullptr; }
  if (int rc = E_get_device::fn(&device)) return raise_native("mtb_get_device", rc);
  return PyLong_FromLong(device);
}

PyMethodDef methods[] = {
    {"load", load, METH_VARARGS, nullptr},
    {"on_first_use", on_first_use, METH_O, nullptr},
    {"launches", launches, METH_NOARGS, nullptr},
    {"current_device", current_device, METH_NOARGS, nullptr},
    {"set_state", set_state, METH_VARARGS, nullptr},
    {"new_like", (PyCFunction)(void (*)())new_like, METH_FASTCALL, "An uninitialised tensor: (shape, like, dtype=None)."},
    {"enter", enter, METH_O, "Make the tensor's device current; the CUDA state."},
    {"stream", stream, METH_NOARGS, "The compute stream of the current device."},
    {"sgd_step", (PyCFunction)(void (*)())sgd_step, METH_FASTCALL, "One SGD update of a list of (parameter, buffer, first)."},
    {"workspace", workspace<0>, METH_O, "(address, bytes) of scratch for compute-stream kernels."},
    {"side_workspace", workspace<1>, METH_O, "(address, bytes) of scratch for side-stream kernels."},
#define X(n, k, h) {#n, (PyCFunction)(void (*)())E_##n::call, METH_FASTCALL, nullptr},
    MTB_ENTRIES(X)
#undef X
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_mtb_binding", "C ABI of libmytorch_b200.so", -1, methods};

}  // namespace

PyMODINIT_FUNC PyInit__mtb_binding() {
  BlockType.tp_name = "mytorch_b200.Block";
  BlockType.tp_basicsize = sizeof(Block);
  BlockType.tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_BASETYPE;
  BlockType.tp_doc = "A device allocation from the library's pool.";
  BlockType.tp_new = PyType_GenericNew;
  BlockType.tp_init = block_init;
  BlockType.tp_dealloc = block_dealloc;
  BlockType.tp_members = block_members;
  BlockType.tp_methods = block_methods;
  if (PyType_Ready(&BlockType) < 0) return nullptr;
  PyObject* m = PyModule_Create(&module);
  if (!m) return nullptr;
#define X(n) if (!(N_##n = PyUnicode_InternFromString(#n))) return nullptr;
  MTB_NAMES(X)
#undef X
  PyObject* names = PyTuple_New(kEntries);
#define X(n, k, h) PyTuple_SET_ITEM(names, ID_##n, PyUnicode_FromString("mtb_" #n));
  MTB_ENTRIES(X)
#undef X
  Py_INCREF(&BlockType);
  if (PyModule_AddObject(m, "entry_points", names) < 0 || PyModule_AddObject(m, "Block", (PyObject*)&BlockType) < 0) return nullptr;
  return m;
}
