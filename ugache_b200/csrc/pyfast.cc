// The per-step calls of the Python face in native code: argument checks, output tensors from
// torch's caching allocator, the current stream, the library call.  A lookup of a few hundred keys
// takes less time on the GPU than the same steps took in Python and ctypes (11 us per call, of
// which the library's own part is 3).  Row movement stays in libugache_b200.so; its entry points
// arrive as addresses, so this module links against torch alone.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/ugache_b200.h"

namespace {

struct Entry {
  decltype(&ugc_lookup_i64) lookup_i64;
  decltype(&ugc_lookup_u32) lookup_u32;
  decltype(&ugc_lookup_unique) lookup_unique;
  decltype(&ugc_lookup_pool) lookup_pool;
  decltype(&ugc_record) record;
};
Entry g_ugc = {};
PyObject* g_check = nullptr;  // raises for a status other than UGC_OK

PyObject* raise_status(int status) {
  PyObject* r = PyObject_CallFunction(g_check, "i", status);
  if (r) {  // cannot be: a failing status raises
    Py_DECREF(r);
    PyErr_SetString(PyExc_RuntimeError, "ugache_b200: failed");
  }
  return nullptr;
}

// Key tensor of the call and its bytes per key; `on_gpu`: its device decides the stream or where the
// outputs go (else pinned host keys will do).  False with a Python error set.
bool key_tensor(PyObject* o, const at::Tensor** keys, int* key_bytes, bool reject_other, bool on_gpu) {
  if (!THPVariable_Check(o)) {
    PyErr_SetString(PyExc_TypeError, "keys must be a torch tensor");
    return false;
  }
  const at::Tensor& t = THPVariable_Unpack(o);
  const at::ScalarType ty = t.scalar_type();
  if (reject_other && ty != at::kLong && ty != at::kInt && ty != at::kUInt32) {
    PyErr_SetString(PyExc_TypeError, "keys must be int64, int32 or uint32");
    return false;
  }
  if (on_gpu && !t.is_cuda()) {
    PyErr_SetString(PyExc_ValueError, "keys must be a CUDA tensor");
    return false;
  }
  *keys = &t;
  *key_bytes = ty == at::kLong ? 8 : 4;
  return true;
}

// The stream argument: an integer, or None for the device's current stream.
bool stream_arg(PyObject* o, at::DeviceIndex dev, void** stream) {
  if (o == Py_None) {
    *stream = c10::cuda::getCurrentCUDAStream(dev).stream();
    return true;
  }
  *stream = PyLong_AsVoidPtr(o);
  return !PyErr_Occurred();
}

bool tensor_or_none(PyObject* o, const char* what, const at::Tensor** t) {
  *t = nullptr;
  if (o == Py_None) return true;
  if (!THPVariable_Check(o)) {
    PyErr_Format(PyExc_TypeError, "%s must be a torch tensor", what);
    return false;
  }
  *t = &THPVariable_Unpack(o);
  return true;
}

at::Tensor device_empty(at::IntArrayRef sizes, at::ScalarType ty, at::Device dev) {
  return at::Tensor(at::detail::empty_cuda(sizes, ty, dev, std::nullopt));
}

bool arg_count(Py_ssize_t n, Py_ssize_t want) {
  if (n == want) return true;
  PyErr_Format(PyExc_TypeError, "%zd arguments expected, got %zd", want, n);
  return false;
}

// C++ exceptions become the Python ones torch raises for them (by its translation alone: the buffer for
// warnings that torch's own macros set up besides would be made on every call)
#define UGC_PY_TRY try {
#define UGC_PY_END                                                  \
  }                                                                 \
  catch (...) {                                                     \
    torch::translate_exception_to_python(std::current_exception()); \
    return nullptr;                                                 \
  }

// lookup(ctx, replica, row_bytes, keys, out | None, stream | None) -> out
PyObject* fast_lookup(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
  if (!arg_count(n_args, 6)) return nullptr;
  UGC_PY_TRY
  ugc_ctx* ctx = static_cast<ugc_ctx*>(PyLong_AsVoidPtr(a[0]));
  const int replica = (int)PyLong_AsLong(a[1]);
  const int64_t row_bytes = PyLong_AsLongLong(a[2]);
  if (PyErr_Occurred()) return nullptr;
  const at::Tensor *keys, *out;
  int kb;
  void* stream;
  if (!key_tensor(a[3], &keys, &kb, true, a[4] == Py_None || a[5] == Py_None) || !tensor_or_none(a[4], "out", &out) ||
      !stream_arg(a[5], keys->device().index(), &stream))
    return nullptr;
  const int64_t n = keys->numel();
  at::Tensor made;
  if (!out) {
    made = device_empty({n, row_bytes}, at::kByte, keys->device());
    out = &made;
  }
  const void* kp = keys->data_ptr();
  void* op = out->data_ptr();
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = kb == 8 ? g_ugc.lookup_i64(ctx, replica, static_cast<const int64_t*>(kp), (size_t)n, op, stream)
               : g_ugc.lookup_u32(ctx, replica, static_cast<const uint32_t*>(kp), (size_t)n, op, stream);
  Py_END_ALLOW_THREADS
  if (rc != UGC_OK) return raise_status(rc);
  if (!made.defined()) return Py_NewRef(a[4]);
  return THPVariable_Wrap(std::move(made));
  UGC_PY_END
}

// lookup_unique(ctx, replica, row_bytes, keys, stream | None) -> (rows, unique_keys, inverse, n_unique)
PyObject* fast_lookup_unique(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
  if (!arg_count(n_args, 5)) return nullptr;
  UGC_PY_TRY
  ugc_ctx* ctx = static_cast<ugc_ctx*>(PyLong_AsVoidPtr(a[0]));
  const int replica = (int)PyLong_AsLong(a[1]);
  const int64_t row_bytes = PyLong_AsLongLong(a[2]);
  if (PyErr_Occurred()) return nullptr;
  const at::Tensor* keys;
  int kb;
  void* stream;
  if (!key_tensor(a[3], &keys, &kb, false, true) || !stream_arg(a[4], keys->device().index(), &stream)) return nullptr;
  const int64_t n = keys->numel();
  const at::Device dev = keys->device();
  at::Tensor rows = device_empty({n, row_bytes}, at::kByte, dev);
  at::Tensor uniq = device_empty({n}, keys->scalar_type(), dev);
  at::Tensor inverse = device_empty({n}, at::kInt, dev);
  at::Tensor n_unique = device_empty({1}, at::kInt, dev);  // the call writes it, whatever n
  void *rp = rows.data_ptr(), *up = uniq.data_ptr();
  int32_t* ip = inverse.data_ptr<int32_t>();
  uint32_t* np = reinterpret_cast<uint32_t*>(n_unique.data_ptr<int32_t>());
  const void* kp = keys->data_ptr();
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = g_ugc.lookup_unique(ctx, replica, kp, kb, (size_t)n, rp, up, ip, np, stream);
  Py_END_ALLOW_THREADS
  if (rc != UGC_OK) return raise_status(rc);
  PyObject* t = PyTuple_New(4);
  if (!t) return nullptr;
  PyTuple_SET_ITEM(t, 0, THPVariable_Wrap(std::move(rows)));
  PyTuple_SET_ITEM(t, 1, THPVariable_Wrap(std::move(uniq)));
  PyTuple_SET_ITEM(t, 2, THPVariable_Wrap(std::move(inverse)));
  PyTuple_SET_ITEM(t, 3, THPVariable_Wrap(std::move(n_unique)));
  return t;
  UGC_PY_END
}

// lookup_pool(ctx, replica, keys, offsets | None, n_bags, bag_size, elem_type, mode, dim, out | None,
//             stream | None) -> out
PyObject* fast_lookup_pool(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
  if (!arg_count(n_args, 11)) return nullptr;
  UGC_PY_TRY
  ugc_ctx* ctx = static_cast<ugc_ctx*>(PyLong_AsVoidPtr(a[0]));
  const int replica = (int)PyLong_AsLong(a[1]);
  const int64_t n_bags = PyLong_AsLongLong(a[4]), bag_size = PyLong_AsLongLong(a[5]);
  const int elem = (int)PyLong_AsLong(a[6]), mode = (int)PyLong_AsLong(a[7]);
  const int64_t dim = PyLong_AsLongLong(a[8]);
  if (PyErr_Occurred()) return nullptr;
  const at::Tensor *keys, *offsets, *out;
  int kb;
  void* stream;
  if (!key_tensor(a[2], &keys, &kb, false, a[9] == Py_None || a[10] == Py_None) || !tensor_or_none(a[3], "offsets", &offsets) ||
      !tensor_or_none(a[9], "out", &out) || !stream_arg(a[10], keys->device().index(), &stream))
    return nullptr;
  at::Tensor made;
  if (!out) {
    made = device_empty({n_bags, dim}, at::kFloat, keys->device());
    out = &made;
  }
  const void* kp = keys->data_ptr();
  const int64_t* fp = offsets ? offsets->data_ptr<int64_t>() : nullptr;
  float* op = static_cast<float*>(out->data_ptr());
  const size_t n = (size_t)keys->numel();
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = g_ugc.lookup_pool(ctx, replica, kp, kb, n, fp, (size_t)n_bags, (size_t)bag_size, elem, mode, op, stream);
  Py_END_ALLOW_THREADS
  if (rc != UGC_OK) return raise_status(rc);
  if (!made.defined()) return Py_NewRef(a[9]);
  return THPVariable_Wrap(std::move(made));
  UGC_PY_END
}

// record(ctx, replica, keys, stream | None)
PyObject* fast_record(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
  if (!arg_count(n_args, 4)) return nullptr;
  UGC_PY_TRY
  ugc_ctx* ctx = static_cast<ugc_ctx*>(PyLong_AsVoidPtr(a[0]));
  const int replica = (int)PyLong_AsLong(a[1]);
  if (PyErr_Occurred()) return nullptr;
  const at::Tensor* keys;
  int kb;
  void* stream;
  if (!key_tensor(a[2], &keys, &kb, false, a[3] == Py_None) || !stream_arg(a[3], keys->device().index(), &stream)) return nullptr;
  const void* kp = keys->data_ptr();
  const size_t n = (size_t)keys->numel();
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = g_ugc.record(ctx, replica, kp, kb, n, stream);
  Py_END_ALLOW_THREADS
  if (rc != UGC_OK) return raise_status(rc);
  Py_RETURN_NONE;
  UGC_PY_END
}

// bind(check, {entry point name: address})
PyObject* fast_bind(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
  if (!arg_count(n_args, 2)) return nullptr;
  auto address = [&](const char* name, auto* slot) {
    PyObject* v = PyDict_GetItemString(a[1], name);
    void* p = v ? PyLong_AsVoidPtr(v) : nullptr;
    if (!p && !PyErr_Occurred()) PyErr_Format(PyExc_KeyError, "%s", name);
    *slot = reinterpret_cast<std::remove_pointer_t<decltype(slot)>>(p);
    return p != nullptr;
  };
  if (!address("ugc_lookup_i64", &g_ugc.lookup_i64) || !address("ugc_lookup_u32", &g_ugc.lookup_u32) ||
      !address("ugc_lookup_unique", &g_ugc.lookup_unique) || !address("ugc_lookup_pool", &g_ugc.lookup_pool) ||
      !address("ugc_record", &g_ugc.record))
    return nullptr;
  Py_XDECREF(g_check);
  g_check = Py_NewRef(a[0]);
  Py_RETURN_NONE;
}

PyMethodDef kMethods[] = {
    {"bind", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(fast_bind)), METH_FASTCALL, nullptr},
    {"lookup", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(fast_lookup)), METH_FASTCALL, nullptr},
    {"lookup_unique", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(fast_lookup_unique)), METH_FASTCALL, nullptr},
    {"lookup_pool", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(fast_lookup_pool)), METH_FASTCALL, nullptr},
    {"record", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(fast_record)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_fast", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__fast() {
  PyObject* m = PyModule_Create(&kModule);
  if (m && PyModule_AddStringConstant(m, "built_for", UGC_BUILT_FOR) < 0) {
    Py_DECREF(m);
    return nullptr;
  }
  return m;
}
