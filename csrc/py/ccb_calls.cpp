// The package's frequent calls from Python to libccb.so in one step each: tensors to pointers, checks, results
// allocated, the call. As Python and ctypes a small all-reduce of eight ranks took 8 us for that, longer than its
// launch and kernel.
//
// Every function takes what the Python function around it takes and answers None where anything is out of the
// ordinary (an argument of another type, a tensor elsewhere, strided, wrapped or of a subclass, a mode that watches
// torch's functions): the Python function then goes its general way, which raises what there is to raise.
// Otherwise it answers with the library's return code, or with the result and the code's place taken by it.
// The interpreter's lock is released around the library's call, as ctypes does: a launch may wait.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/ops/empty.h>
#include <ATen/ops/empty_like.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <cuda_runtime_api.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include "ccb/ccb.h"
#include "ccb/ccb_lossless.h"
#include "ccb/ccb_moe.h"
#include "ccb/ccb_sz.h"

namespace {

#define CCB_CALLS(X)                                                                                                          \
  X(ccb_all_reduce) X(ccb_reduce_scatter) X(ccb_all_gather) X(ccb_moe_dispatch) X(ccb_moe_combine) X(ccb_wire_bytes)           \
  X(ccb_encode) X(ccb_decode) X(ccb_reduce_recode) X(ccb_lossless_max_bytes) X(ccb_lossless_encode) X(ccb_lossless_decode)     \
  X(ccb_sz_capacity) X(ccb_sz_compress) X(ccb_sz_decompress) X(ccb_sz_container_sums) X(ccb_sz_container_open)                 \
  X(ccb_sz_container_pack) X(ccb_sz_container_unpack)
struct Library {
#define CCB_FIELD(f) decltype(&::f) f;
  CCB_CALLS(CCB_FIELD)
#undef CCB_FIELD
} lib;
PyObject *kOps, *kCodecs, *kAlgos, *kParameter;   // name -> number; torch.nn.Parameter

constexpr int kMost = CCB_MAX_RANKS;
typedef PyObject* const* Args;

// A tensor of plain torch type whose memory is what it says.
const at::Tensor* plain(PyObject* o) {
  if (!THPVariable_CheckExact(o) && (PyObject*)Py_TYPE(o) != kParameter) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(o);
  if (!t.defined() || !t.is_cuda() || t.layout() != at::kStrided || !t.has_storage() || !t.is_contiguous()) return nullptr;
  using K = c10::DispatchKey;
  static const c10::DispatchKeySet wrapped({K::Python, K::Functionalize, K::FuncTorchBatched, K::BatchedNestedTensor, K::FuncTorchGradWrapper, K::Batched});
  if (t.key_set().has_any(wrapped) || t.get_device() != c10::cuda::current_device()) return nullptr;
  return &t;
}
bool watched() { return at::impl::torch_function_mode_enabled() || c10::impl::TorchDispatchModeTLS::any_modes_set(); }

int dtype_of(at::ScalarType t) { return t == at::kFloat ? CCB_F32 : t == at::kBFloat16 ? CCB_BF16 : t == at::kHalf ? CCB_F16 : -1; }

struct Tensors {
  void* ptr[kMost];
  const at::Tensor* first = nullptr;
  int n = 0;
  bool take(PyObject* o) {
    const at::Tensor* t = n < kMost ? plain(o) : nullptr;
    if (!t) return false;
    if (!n) first = t;
    ptr[n++] = t->data_ptr();
    return true;
  }
  // one tensor, or a list or tuple of them: `want` of them
  bool read(PyObject* o, int want) {
    if (PyList_CheckExact(o) || PyTuple_CheckExact(o)) {
      const Py_ssize_t k = PySequence_Fast_GET_SIZE(o);
      if (k != want) return false;
      for (Py_ssize_t i = 0; i < k; ++i)
        if (!take(PySequence_Fast_GET_ITEM(o, i))) return false;
      return n > 0;
    }
    return want == 1 && take(o);
  }
  // an attribute of one object, or of each of a list
  bool read_of(PyObject* o, const char* name, int want) {
    const bool many = PyList_CheckExact(o);
    if (many ? PyList_GET_SIZE(o) != want : want != 1) return false;
    for (int i = 0; i < want; ++i) {
      PyObject* a = PyObject_GetAttrString(many ? PyList_GET_ITEM(o, i) : o, name);
      const bool ok = a && take(a);   // the object keeps its attribute
      Py_XDECREF(a);
      if (!ok) {
        PyErr_Clear();
        return false;
      }
    }
    return true;
  }
};

bool number(PyObject* o, uint64_t& v) {
  if (!PyLong_CheckExact(o)) return false;
  v = PyLong_AsUnsignedLongLong(o);
  if (PyErr_Occurred()) {
    PyErr_Clear();
    return false;
  }
  return true;
}
bool code(PyObject* o, PyObject* table, int& v) {
  PyObject* hit = PyUnicode_CheckExact(o) ? PyDict_GetItemWithError(table, o) : nullptr;
  if (!hit || !PyLong_Check(hit)) {
    PyErr_Clear();
    return false;
  }
  v = (int)PyLong_AsLong(hit);
  return true;
}
bool real(PyObject* o, float& v) {
  if (!PyFloat_CheckExact(o)) return false;
  v = (float)PyFloat_AS_DOUBLE(o);
  return true;
}
bool extents(PyObject* o, int (&e)[3]) {
  if (!PyTuple_Check(o) || PyTuple_GET_SIZE(o) != 3) return false;
  for (int i = 0; i < 3; ++i) {
    uint64_t v;
    if (!number(PyTuple_GET_ITEM(o, i), v) || v < 1 || v > 0x7fffffff) return false;
    e[i] = (int)v;
  }
  return true;
}
ccb_comm* comm_of(PyObject* o) { return static_cast<ccb_comm*>(PyLong_AsVoidPtr(o)); }
cudaStream_t stream() { return c10::cuda::getCurrentCUDAStream().stream(); }
at::Tensor made(at::IntArrayRef size, at::ScalarType t, const at::Tensor& like) { return at::empty(size, at::TensorOptions().dtype(t).device(like.device())); }

#define NOT_TAKEN Py_RETURN_NONE
#define FUNCTION(name, count)                                          \
  PyObject* name(PyObject*, Args a, Py_ssize_t given) {                \
    HANDLE_TH_ERRORS                                                   \
    if (given != count || watched()) NOT_TAKEN;
#define END     \
  END_HANDLE_TH_ERRORS \
  }
struct Unlocked {
  PyThreadState* state = PyEval_SaveThread();
  ~Unlocked() { PyEval_RestoreThread(state); }
};
template <class F>
int unlocked(F f) {
  const Unlocked now;
  return f();
}
// the result, or the code where the call failed
PyObject* result(int rc, const at::Tensor& t) { return rc ? PyLong_FromLong(rc) : THPVariable_Wrap(t); }

// (handle, ranks here, send, recv, error feedback, op, codec, algo)
FUNCTION(all_reduce, 8)
  const int n = (int)PyLong_AsLong(a[1]);
  Tensors s, r, e;
  int op, codec, algo;
  if (!s.read(a[2], n) || !r.read(a[3], n) || !code(a[5], kOps, op) || !code(a[6], kCodecs, codec) || !code(a[7], kAlgos, algo)) NOT_TAKEN;
  const int dt = dtype_of(s.first->scalar_type());
  if (dt < 0) NOT_TAKEN;
  const uint64_t count = (uint64_t)s.first->numel();
  if (a[4] != Py_None) {
    if (!e.read(a[4], n)) NOT_TAKEN;
    for (int i = 0; i < n; ++i) {
      const at::Tensor& t = THPVariable_Unpack(PyList_CheckExact(a[4]) || PyTuple_CheckExact(a[4]) ? PySequence_Fast_GET_ITEM(a[4], i) : a[4]);
      if (t.scalar_type() != at::kFloat || (uint64_t)t.numel() != count) NOT_TAKEN;
    }
  }
  ccb_comm* c = comm_of(a[0]);
  const cudaStream_t st = stream();
  float* const* ef = a[4] == Py_None ? nullptr : reinterpret_cast<float* const*>(e.ptr);
  return PyLong_FromLong(unlocked([&] { return lib.ccb_all_reduce(c, s.ptr, r.ptr, count, dt, op, codec, algo, ef, st); }));
END

// (handle, ranks here, ranks, send, recv, op, codec)
FUNCTION(reduce_scatter, 7)
  const int n = (int)PyLong_AsLong(a[1]);
  Tensors s, r;
  int op, codec;
  if (!s.read(a[3], n) || !r.read(a[4], n) || !code(a[5], kOps, op) || !code(a[6], kCodecs, codec)) NOT_TAKEN;
  const int dt = dtype_of(s.first->scalar_type());
  if (dt < 0 || s.first->numel() != r.first->numel() * PyLong_AsLong(a[2])) NOT_TAKEN;
  const uint64_t count = (uint64_t)r.first->numel();
  ccb_comm* c = comm_of(a[0]);
  const cudaStream_t st = stream();
  return PyLong_FromLong(unlocked([&] { return lib.ccb_reduce_scatter(c, s.ptr, r.ptr, count, dt, op, codec, nullptr, st); }));
END

// (handle, ranks here, ranks, send, recv, codec)
FUNCTION(all_gather, 6)
  const int n = (int)PyLong_AsLong(a[1]);
  Tensors s, r;
  int codec;
  if (!s.read(a[3], n) || !r.read(a[4], n) || !code(a[5], kCodecs, codec)) NOT_TAKEN;
  const int dt = dtype_of(s.first->scalar_type());
  if (dt < 0 || r.first->numel() != s.first->numel() * PyLong_AsLong(a[2])) NOT_TAKEN;
  const uint64_t count = (uint64_t)s.first->numel();
  ccb_comm* c = comm_of(a[0]);
  const cudaStream_t st = stream();
  return PyLong_FromLong(unlocked([&] { return lib.ccb_all_gather(c, s.ptr, r.ptr, count, dt, codec, st); }));
END

bool matrix(PyObject* o, int n, uint64_t (&m)[kMost * kMost]) {
  if (n > kMost || !PyList_CheckExact(o) || PyList_GET_SIZE(o) != n) return false;
  for (int i = 0; i < n; ++i) {
    PyObject* row = PyList_GET_ITEM(o, i);
    if (!PyList_CheckExact(row) || PyList_GET_SIZE(row) != n) return false;
    for (int k = 0; k < n; ++k)
      if (!number(PyList_GET_ITEM(row, k), m[i * n + k])) return false;
  }
  return true;
}

// (handle, ranks here, ranks, x, recv, routes, counts, codec)
FUNCTION(moe_dispatch, 8)
  const int n = (int)PyLong_AsLong(a[1]);
  Tensors x, r, perm;
  uint64_t counts[kMost * kMost];
  int codec;
  if (!x.read(a[3], n) || !r.read(a[4], n) || !perm.read_of(a[5], "perm", n) || !matrix(a[6], (int)PyLong_AsLong(a[2]), counts) || !code(a[7], kCodecs, codec)) NOT_TAKEN;
  const int dt = dtype_of(x.first->scalar_type());
  if (dt < 0 || x.first->dim() < 1) NOT_TAKEN;
  const uint64_t hidden = (uint64_t)x.first->size(-1);
  ccb_comm* c = comm_of(a[0]);
  const cudaStream_t st = stream();
  return PyLong_FromLong(unlocked([&] { return lib.ccb_moe_dispatch(c, x.ptr, r.ptr, reinterpret_cast<const int32_t* const*>(perm.ptr), counts, hidden, dt, codec, st); }));
END

// (handle, ranks here, ranks, y, out, routes, counts, codec)
FUNCTION(moe_combine, 8)
  const int n = (int)PyLong_AsLong(a[1]);
  Tensors y, o, dest, pos, gate;
  uint64_t counts[kMost * kMost], topk;
  int codec;
  if (!y.read(a[3], n) || !o.read(a[4], n) || !dest.read_of(a[5], "dest_rank", n) || !pos.read_of(a[5], "pos", n) || !gate.read_of(a[5], "gate", n) ||
      !matrix(a[6], (int)PyLong_AsLong(a[2]), counts) || !code(a[7], kCodecs, codec)) NOT_TAKEN;
  PyObject* k = PyObject_GetAttrString(PyList_CheckExact(a[5]) ? PyList_GET_ITEM(a[5], 0) : a[5], "topk");
  const bool ok = k && number(k, topk) && topk <= 0x7fffffff;
  Py_XDECREF(k);
  if (!ok) {
    PyErr_Clear();
    NOT_TAKEN;
  }
  const int dt = dtype_of(o.first->scalar_type());
  if (dt < 0 || o.first->dim() < 1) NOT_TAKEN;
  const uint64_t tokens = (uint64_t)o.first->size(0), hidden = (uint64_t)o.first->size(-1);
  ccb_comm* c = comm_of(a[0]);
  const cudaStream_t st = stream();
  return PyLong_FromLong(unlocked([&] {
    return lib.ccb_moe_combine(c, y.ptr, o.ptr, reinterpret_cast<const int32_t* const*>(dest.ptr), reinterpret_cast<const int32_t* const*>(pos.ptr),
                               reinterpret_cast<const float* const*>(gate.ptr), counts, tokens, (int)topk, hidden, dt, codec, st);
  }));
END

// (x, codec) -> wire
FUNCTION(encode, 2)
  const at::Tensor* x = plain(a[0]);
  int codec;
  if (!x || !code(a[1], kCodecs, codec)) NOT_TAKEN;
  const int dt = dtype_of(x->scalar_type());
  if (dt < 0) NOT_TAKEN;
  const uint64_t count = (uint64_t)x->numel();
  const at::Tensor wire = made({(int64_t)lib.ccb_wire_bytes(codec, dt, count)}, at::kByte, *x);
  const void *in = x->data_ptr();
  void* out = wire.data_ptr();
  const cudaStream_t st = stream();
  return result(unlocked([&] { return lib.ccb_encode(codec, dt, in, count, out, st); }), wire);
END

// (wire, codec, count, dtype) -> values
FUNCTION(decode, 4)
  const at::Tensor* wire = plain(a[0]);
  int codec;
  uint64_t count;
  if (!wire || !code(a[1], kCodecs, codec) || !number(a[2], count) || !THPDtype_Check(a[3])) NOT_TAKEN;
  const at::ScalarType type = reinterpret_cast<THPDtype*>(a[3])->scalar_type;
  const int dt = dtype_of(type);
  if (dt < 0 || count >> 62) NOT_TAKEN;
  const at::Tensor out = made({(int64_t)count}, type, *wire);
  const void* in = wire->data_ptr();
  void* to = out.data_ptr();
  const cudaStream_t st = stream();
  return result(unlocked([&] { return lib.ccb_decode(codec, dt, in, count, to, st); }), out);
END

// (wires, codec, count) -> wire
FUNCTION(reduce_recode, 3)
  int codec;
  uint64_t count;
  if (!PyList_CheckExact(a[0]) || !code(a[1], kCodecs, codec) || !number(a[2], count)) NOT_TAKEN;
  const Py_ssize_t n = PyList_GET_SIZE(a[0]);
  const void* in[16];
  if (n < 1 || n > 16) NOT_TAKEN;
  const at::Tensor* first = nullptr;
  for (Py_ssize_t i = 0; i < n; ++i) {
    const at::Tensor* t = plain(PyList_GET_ITEM(a[0], i));
    if (!t) NOT_TAKEN;
    if (!i) first = t;
    in[i] = t->data_ptr();
  }
  const at::Tensor out = at::empty_like(*first);
  void* to = out.data_ptr();
  const cudaStream_t st = stream();
  return result(unlocked([&] { return lib.ccb_reduce_recode(codec, in, (int)n, count, to, st); }), out);
END

// (x) -> container
FUNCTION(lossless_encode, 1)
  const at::Tensor* x = plain(a[0]);
  if (!x) NOT_TAKEN;
  const int dt = dtype_of(x->scalar_type());
  if (dt < 0) NOT_TAKEN;
  const uint64_t count = (uint64_t)x->numel();
  const at::Tensor out = made({(int64_t)lib.ccb_lossless_max_bytes(dt, count)}, at::kByte, *x);
  const void* in = x->data_ptr();
  void* to = out.data_ptr();
  const cudaStream_t st = stream();
  return result(unlocked([&] { return lib.ccb_lossless_encode(dt, in, count, to, st); }), out);
END

// (container, count, dtype) -> values
FUNCTION(lossless_decode, 3)
  const at::Tensor* comp = plain(a[0]);
  uint64_t count;
  if (!comp || !number(a[1], count) || count >> 62 || !THPDtype_Check(a[2])) NOT_TAKEN;
  const at::ScalarType type = reinterpret_cast<THPDtype*>(a[2])->scalar_type;
  const int dt = dtype_of(type);
  if (dt < 0) NOT_TAKEN;
  const at::Tensor out = made({(int64_t)count}, type, *comp);
  const void* in = comp->data_ptr();
  void* to = out.data_ptr();
  const cudaStream_t st = stream();
  return result(unlocked([&] { return lib.ccb_lossless_decode(dt, in, count, to, 0, st); }), out);
END

// (field, bound) -> (slots, used bytes)
FUNCTION(sz_compress, 2)
  const at::Tensor* f = plain(a[0]);
  float eb;
  if (!f || f->scalar_type() != at::kFloat || f->dim() != 3 || f->numel() < 1 || f->numel() >> 31 || !real(a[1], eb)) NOT_TAKEN;
  const int nz = (int)f->size(0), ny = (int)f->size(1), nx = (int)f->size(2);
  const at::Tensor buf = made({(int64_t)lib.ccb_sz_capacity(nx, ny, nz)}, at::kByte, *f), used = made({1}, at::kLong, *f);
  const float* in = static_cast<const float*>(f->data_ptr());
  void* to = buf.data_ptr();
  unsigned long long* sum = static_cast<unsigned long long*>(used.data_ptr());
  const cudaStream_t st = stream();
  const int rc = unlocked([&] { return lib.ccb_sz_compress(in, nx, ny, nz, eb, to, sum, st); });
  if (rc) return PyLong_FromLong(rc);
  return Py_BuildValue("NN", THPVariable_Wrap(buf), THPVariable_Wrap(used));
END

// (slots, shape, bound) -> field
FUNCTION(sz_decompress, 3)
  const at::Tensor* buf = plain(a[0]);
  int e[3];
  float eb;
  if (!buf || !extents(a[1], e) || !real(a[2], eb)) NOT_TAKEN;
  const at::Tensor out = made({e[0], e[1], e[2]}, at::kFloat, *buf);
  const void* in = buf->data_ptr();
  float* to = static_cast<float*>(out.data_ptr());
  const cudaStream_t st = stream();
  return result(unlocked([&] { return lib.ccb_sz_decompress(in, e[2], e[1], e[0], eb, to, st); }), out);
END

// A capture cannot be read back from: the general way says so.
bool capturing(cudaStream_t st) {
  cudaStreamCaptureStatus now;
  return cudaStreamIsCapturing(st, &now) != cudaSuccess || now != cudaStreamCaptureStatusNone;
}
int ended(cudaStream_t st) { return cudaStreamSynchronize(st) == cudaSuccess ? 0 : CCB_ERR_CUDA; }
at::Tensor pinned(int64_t words) { return at::empty({words}, at::TensorOptions().dtype(at::kLong).pinned_memory(true)); }

// (slots, stride of a group) -> (offsets, total, largest): the scan of a buffer's groups
FUNCTION(sz_scan, 2)
  const at::Tensor* buf = plain(a[0]);
  uint64_t stride;
  if (!buf || buf->scalar_type() != at::kByte || !number(a[1], stride)) NOT_TAKEN;
  const uint64_t groups = (uint64_t)buf->numel() / stride;
  if (!groups || groups * stride != (uint64_t)buf->numel() || (reinterpret_cast<uintptr_t>(buf->data_ptr()) & 15)) NOT_TAKEN;
  const cudaStream_t st = stream();
  if (capturing(st)) NOT_TAKEN;
  const at::Tensor offsets = made({(int64_t)groups + 2}, at::kLong, *buf), host = pinned(2);
  const void* slots = buf->data_ptr();
  unsigned long long* at = static_cast<unsigned long long*>(offsets.data_ptr());
  unsigned long long* sums = static_cast<unsigned long long*>(host.data_ptr());   // see sz_open
  const int rc = unlocked([&] {
    const int code = lib.ccb_sz_container_sums(slots, groups, at, sums, st);
    return code ? code : ended(st);
  });
  if (rc) return PyLong_FromLong(rc);
  const int64_t* v = static_cast<const int64_t*>(host.data_ptr());
  return Py_BuildValue("NLL", THPVariable_Wrap(offsets), (long long)v[0], (long long)v[1]);
END

// (container, room) -> (offsets, header and the two sums as 56 bytes): see ccb_sz_container_open
FUNCTION(sz_open, 2)
  const at::Tensor* blob = plain(a[0]);
  uint64_t room;
  if (!blob || blob->scalar_type() != at::kByte || !number(a[1], room) || !room || room >> 31) NOT_TAKEN;
  const cudaStream_t st = stream();
  if (capturing(st)) NOT_TAKEN;
  const at::Tensor offsets = made({(int64_t)room + 2}, at::kLong, *blob), host = pinned(7);
  const void* in = blob->data_ptr();
  const uint64_t bytes = (uint64_t)blob->numel();
  unsigned long long* at = static_cast<unsigned long long*>(offsets.data_ptr());
  void* found = host.data_ptr();   // pinned memory is the device's as well: the kernel's last words, without a copy
  const int rc = unlocked([&] {
    const int code = lib.ccb_sz_container_open(in, bytes, room, at, found, st);
    return code ? code : ended(st);
  });
  if (rc) return PyLong_FromLong(rc);
  return Py_BuildValue("Ny#", THPVariable_Wrap(offsets), static_cast<const char*>(host.data_ptr()), (Py_ssize_t)56);
END

// (slots, offsets, shape, bound, groups, bytes) -> container
FUNCTION(sz_pack, 6)
  const at::Tensor *buf = plain(a[0]), *offsets = plain(a[1]);
  int e[3];
  float eb;
  uint64_t groups, bytes;
  if (!buf || !offsets || !extents(a[2], e) || !real(a[3], eb) || !number(a[4], groups) || !number(a[5], bytes) || bytes >> 62) NOT_TAKEN;
  const at::Tensor out = made({(int64_t)bytes}, at::kByte, *buf);
  const void* slots = buf->data_ptr();
  const unsigned long long* at = static_cast<const unsigned long long*>(offsets->data_ptr());
  void* to = out.data_ptr();
  const cudaStream_t st = stream();
  return result(unlocked([&] { return lib.ccb_sz_container_pack(slots, at, e[2], e[1], e[0], eb, groups, to, st); }), out);
END

// (container, bytes before the payload, offsets, groups, stride of a group) -> slots
FUNCTION(sz_unpack, 5)
  const at::Tensor *blob = plain(a[0]), *offsets = plain(a[2]);
  uint64_t head, groups, stride;
  if (!blob || !offsets || !number(a[1], head) || !number(a[3], groups) || !number(a[4], stride)) NOT_TAKEN;
  const at::Tensor out = made({(int64_t)(groups * stride)}, at::kByte, *blob);
  const char* payload = static_cast<const char*>(blob->data_ptr()) + head;
  const unsigned long long* at = static_cast<const unsigned long long*>(offsets->data_ptr());
  void* to = out.data_ptr();
  const cudaStream_t st = stream();
  return result(unlocked([&] { return lib.ccb_sz_container_unpack(payload, at, groups, to, st); }), out);
END

// (name -> address of the library's function, ops, codecs, algos, torch.nn.Parameter): once, before any call
PyObject* setup(PyObject*, PyObject* args) {
  PyObject* where;
  if (!PyArg_ParseTuple(args, "O!O!O!O!O", &PyDict_Type, &where, &PyDict_Type, &kOps, &PyDict_Type, &kCodecs, &PyDict_Type, &kAlgos, &kParameter)) return nullptr;
  for (PyObject* o : {kOps, kCodecs, kAlgos, kParameter}) Py_INCREF(o);
#define CCB_FIND(f)                                                              \
  {                                                                              \
    PyObject* v = PyDict_GetItemString(where, #f);                               \
    if (!v) return PyErr_Format(PyExc_KeyError, "no address of %s", #f);         \
    lib.f = reinterpret_cast<decltype(lib.f)>(PyLong_AsVoidPtr(v));              \
  }
  CCB_CALLS(CCB_FIND)
#undef CCB_FIND
  if (PyErr_Occurred()) return nullptr;
  Py_RETURN_NONE;
}
// What this file was compiled for, looked for in the built file before it is loaded: the objects above are read by
// the layout that the headers of one torch give them.
PyObject* built_for(PyObject*, PyObject*) { return PyUnicode_FromString(CCB_BUILT_FOR); }
PyObject* names(PyObject*, PyObject*) {
#define CCB_NAME(f) #f " "
  return PyUnicode_FromString(CCB_CALLS(CCB_NAME));
#undef CCB_NAME
}

#define METHOD(f) {#f, (PyCFunction)(void (*)(void))f, METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    {"setup", setup, METH_VARARGS, nullptr}, {"names", names, METH_NOARGS, nullptr}, {"built_for", built_for, METH_NOARGS, nullptr},
    METHOD(all_reduce), METHOD(reduce_scatter), METHOD(all_gather), METHOD(moe_dispatch), METHOD(moe_combine), METHOD(encode), METHOD(decode),
    METHOD(reduce_recode), METHOD(lossless_encode), METHOD(lossless_decode), METHOD(sz_compress), METHOD(sz_decompress), METHOD(sz_scan), METHOD(sz_open),
    METHOD(sz_pack), METHOD(sz_unpack), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "ccb_calls", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_ccb_calls(void) { return PyModule_Create(&module); }
