// CPython module _gcb200_host: the call path of the small, repeated calls (one matmul, one attention, one execute of a
// partition) from Python objects to the C ABI of libGcDnnlApi.so.
//
// Through ctypes a call spends 8 us (matmul, four tensors) to 50 us (execute, a dozen tensors) on attribute look-ups,
// argument conversion and structure building in the interpreter - more than the kernels of a small problem.  Here the
// tensors' addresses and shapes go straight into C structures.  Only the C API of Python is used: no torch headers, no
// ABI beyond the methods data_ptr / shape / is_cuda / dtype / is_contiguous of the tensors.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <cstddef>
#include <cstdint>

#include "../../include/dnnl_graph_compiler.h"
#include "../../include/gc_b200.h"

namespace {

// interned names and cached objects of the torch module (set by setup())
PyObject *s_data_ptr, *s_shape, *s_is_cuda, *s_dtype, *s_is_contiguous;
PyObject *t_tensor, *t_bf16, *f_get_device, *f_raw_stream, *t_ndarray;

struct Ref {   // owned reference
  PyObject *p;
  explicit Ref(PyObject *o) : p(o) {}
  ~Ref() { Py_XDECREF(p); }
  Ref(const Ref &) = delete;
  operator PyObject *() const { return p; }
};

bool address(PyObject *t, void **out) {
  Ref r(PyObject_CallMethodNoArgs(t, s_data_ptr));
  if (!r.p) return false;
  *out = PyLong_AsVoidPtr(r);
  return !PyErr_Occurred();
}
// Shape of a tensor; -1 on error, -2 when it has more than `cap` dimensions.
int shape(PyObject *t, int64_t *dims, int cap) {
  Ref r(PyObject_GetAttr(t, s_shape));
  if (!r.p) return -1;
  if (!PyTuple_Check(r.p)) {
    PyErr_SetString(PyExc_TypeError, "shape is not a tuple");
    return -1;
  }
  const Py_ssize_t n = PyTuple_GET_SIZE(r.p);
  if (n > cap) return -2;
  for (Py_ssize_t i = 0; i < n; ++i) {
    dims[i] = PyLong_AsLongLong(PyTuple_GET_ITEM(r.p, i));
    if (dims[i] == -1 && PyErr_Occurred()) return -1;
  }
  return int(n);
}
bool is_true(PyObject *t, PyObject *attr, bool call, bool *out) {
  Ref r(call ? PyObject_CallMethodNoArgs(t, attr) : PyObject_GetAttr(t, attr));
  if (!r.p) return false;
  *out = r.p == Py_True;
  return true;
}
bool require(bool ok, const char *what) {
  if (!ok) PyErr_SetString(PyExc_AssertionError, what);
  return ok;
}
// A bf16 CUDA tensor (contiguous): its address and two-dimensional or larger shape.
bool operand(PyObject *t, bool check_type, void **ptr, int64_t *dims, int *nd) {
  bool v = false;
  if (check_type) {
    if (!is_true(t, s_is_cuda, false, &v) || !require(v, "the operands must be CUDA tensors")) return false;
    Ref dt(PyObject_GetAttr(t, s_dtype));
    if (!dt.p || !require(dt.p == t_bf16, "the operands must be bfloat16")) return false;
  }
  if (!is_true(t, s_is_contiguous, true, &v) || !require(v, "the operands must be contiguous")) return false;
  *nd = shape(t, dims, DNNL_MAX_NDIMS);
  if (*nd == -2) PyErr_SetString(PyExc_ValueError, "too many dimensions");
  return *nd >= 0 && address(t, ptr);
}
bool current_stream(void **out) {
  Ref dev(PyObject_CallNoArgs(f_get_device));
  if (!dev.p) return false;
  Ref st(PyObject_CallOneArg(f_raw_stream, dev));
  if (!st.p) return false;
  *out = PyLong_AsVoidPtr(st);
  return !PyErr_Occurred();
}

// matmul_bf16(A, B, bias | None, relu, transpose_a, transpose_b, out) -> status
PyObject *matmul_bf16(PyObject *, PyObject *const *a, Py_ssize_t n) {
  if (n != 7) return PyErr_Format(PyExc_TypeError, "matmul_bf16 takes 7 arguments"), nullptr;
  void *pa, *pb, *pbias = nullptr, *po, *stream;
  int64_t da[DNNL_MAX_NDIMS], db[DNNL_MAX_NDIMS];
  int na, nb;
  const int relu = PyObject_IsTrue(a[3]), ta = PyObject_IsTrue(a[4]), tb = PyObject_IsTrue(a[5]);
  if (relu < 0 || ta < 0 || tb < 0) return nullptr;
  if (!operand(a[0], true, &pa, da, &na) || !operand(a[1], false, &pb, db, &nb)) return nullptr;
  if (!require(na == 2 && nb == 2, "the operands must be matrices")) return nullptr;
  const int64_t M = ta ? da[1] : da[0], K = ta ? da[0] : da[1], N = tb ? db[0] : db[1];
  if (!require((tb ? db[1] : db[0]) == K, "inner dimensions differ")) return nullptr;
  if (a[2] != Py_None && !address(a[2], &pbias)) return nullptr;
  if (!address(a[6], &po) || !current_stream(&stream)) return nullptr;
  int st;
  Py_BEGIN_ALLOW_THREADS
  st = gcb200_matmul_bf16(pa, pb, pbias, po, M, N, K, ta, tb, relu, stream);
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(st);
}

// attention_bf16(Q, K, V, scale, causal, out) -> status
PyObject *attention_bf16(PyObject *, PyObject *const *a, Py_ssize_t n) {
  if (n != 6) return PyErr_Format(PyExc_TypeError, "attention_bf16 takes 6 arguments"), nullptr;
  void *q, *k, *v, *o, *stream;
  int64_t d[DNNL_MAX_NDIMS];
  int nd;
  if (!operand(a[1], false, &k, d, &nd) || !operand(a[2], false, &v, d, &nd) || !operand(a[0], true, &q, d, &nd)) return nullptr;
  if (!require(nd >= 2, "Q must have at least two dimensions")) return nullptr;
  const double scale = PyFloat_AsDouble(a[3]);
  const int causal = PyObject_IsTrue(a[4]);
  if (PyErr_Occurred() || causal < 0 || !address(a[5], &o) || !current_stream(&stream)) return nullptr;
  int64_t bh = 1;
  for (int i = 0; i + 2 < nd; ++i) bh *= d[i];
  int st;
  Py_BEGIN_ALLOW_THREADS
  st = gcb200_attention_bf16(q, k, v, o, bh, d[nd - 2], d[nd - 1], float(scale), causal, stream);
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(st);
}

constexpr int kMaxTensors = 64;
struct Pack {
  dnnl_graph_compiler_tensor t[kMaxTensors + 1];
  int64_t dims[kMaxTensors][DNNL_MAX_NDIMS];
  Py_buffer views[kMaxTensors];
  PyObject *held[kMaxTensors];   // the call runs without the interpreter's lock: another thread may change the dictionary
  int n = 0, n_views = 0, n_held = 0;
  ~Pack() {
    for (int i = 0; i < n_views; ++i) PyBuffer_Release(&views[i]);
    for (int i = 0; i < n_held; ++i) Py_DECREF(held[i]);
  }
  // 1: packed, 0: something this path does not take (the caller packs it in Python), -1: error.  Only tensors and numpy
  // arrays are taken: other objects with a buffer (bytes, memoryview) are no arguments of a partition, and an output among
  // them could be memory that must not change.
  int add(PyObject *key, PyObject *val) {
    if (n == kMaxTensors) return 0;
    const bool tensor = PyObject_TypeCheck(val, reinterpret_cast<PyTypeObject *>(t_tensor));
    if (!tensor && !(t_ndarray && PyObject_TypeCheck(val, reinterpret_cast<PyTypeObject *>(t_ndarray)))) return 0;
    const size_t id = PyLong_AsSize_t(key);
    if (id == size_t(-1) && PyErr_Occurred()) {
      PyErr_Clear();
      return 0;
    }
    Py_INCREF(val);
    held[n_held++] = val;
    int64_t *d = dims[n];
    void *p;
    int nd;
    if (tensor) {
      nd = shape(val, d, DNNL_MAX_NDIMS);
      if (nd == -2) return 0;
      if (nd < 0 || !address(val, &p)) return -1;
    } else {
      Py_buffer *b = &views[n_views];
      if (PyObject_GetBuffer(val, b, PyBUF_STRIDED_RO) != 0) {
        PyErr_Clear();
        return 0;
      }
      ++n_views;
      nd = b->ndim;
      if (nd > DNNL_MAX_NDIMS) return 0;
      for (int i = 0; i < nd; ++i) d[i] = b->shape[i];
      p = b->buf;
    }
    t[n].id = id;
    t[n].ndims = uint8_t(nd);
    t[n].dims = d;
    t[n].data = p;
    ++n;
    return 1;
  }
  int add_all(PyObject *dict) {
    PyObject *k, *v;
    Py_ssize_t pos = 0;
    while (PyDict_Next(dict, &pos, &k, &v)) {
      const int r = add(k, v);
      if (r != 1) return r;
    }
    for (int i = n; i <= kMaxTensors; ++i) t[i].id = ~size_t(0);   // a call with too few tensors finds none of these
    return 1;
  }
};

// execute(handle, inputs, outputs, stream): stream None = the synchronous call, True = the current stream, else a raw
// handle.  Returns the status, or None when an argument is nothing this path takes.
PyObject *execute(PyObject *, PyObject *const *a, Py_ssize_t n) {
  if (n != 4) return PyErr_Format(PyExc_TypeError, "execute takes 4 arguments"), nullptr;
  if (!PyDict_CheckExact(a[1]) || !PyDict_CheckExact(a[2])) Py_RETURN_NONE;
  auto *exe = static_cast<const dnnl_graph_compiler_executable *>(PyLong_AsVoidPtr(a[0]));
  if (PyErr_Occurred()) return nullptr;
  Pack in, out;
  for (int i = 0; i < 2; ++i) {
    const int r = i == 0 ? in.add_all(a[1]) : out.add_all(a[2]);
    if (r < 0) return nullptr;
    if (r == 0) Py_RETURN_NONE;
  }
  void *stream = nullptr;
  if (a[3] == Py_True) {
    if (!current_stream(&stream)) return nullptr;
  } else if (a[3] != Py_None) {
    stream = PyLong_AsVoidPtr(a[3]);
    if (PyErr_Occurred()) return nullptr;
  }
  int st;
  Py_BEGIN_ALLOW_THREADS
  st = a[3] == Py_None ? int(dnnl_graph_compiler_execute(exe, in.t, out.t)) : gcb200_execute_on_stream(exe, in.t, out.t, stream);
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(st);
}

// setup(torch.Tensor, torch.bfloat16, get_device, get_raw_stream, numpy.ndarray)
PyObject *setup(PyObject *, PyObject *const *a, Py_ssize_t n) {
  if (n != 5) return PyErr_Format(PyExc_TypeError, "setup takes 5 arguments"), nullptr;
  PyObject **slots[5] = {&t_tensor, &t_bf16, &f_get_device, &f_raw_stream, &t_ndarray};
  for (int i = 0; i < 5; ++i) {
    Py_INCREF(a[i]);
    Py_XSETREF(*slots[i], a[i]);
  }
  Py_RETURN_NONE;
}

PyMethodDef methods[] = {
    {"setup", reinterpret_cast<PyCFunction>(reinterpret_cast<void *>(setup)), METH_FASTCALL, nullptr},
    {"matmul_bf16", reinterpret_cast<PyCFunction>(reinterpret_cast<void *>(matmul_bf16)), METH_FASTCALL, nullptr},
    {"attention_bf16", reinterpret_cast<PyCFunction>(reinterpret_cast<void *>(attention_bf16)), METH_FASTCALL, nullptr},
    {"execute", reinterpret_cast<PyCFunction>(reinterpret_cast<void *>(execute)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_gcb200_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

} // namespace

PyMODINIT_FUNC PyInit__gcb200_host() {
  s_data_ptr = PyUnicode_InternFromString("data_ptr");
  s_shape = PyUnicode_InternFromString("shape");
  s_is_cuda = PyUnicode_InternFromString("is_cuda");
  s_dtype = PyUnicode_InternFromString("dtype");
  s_is_contiguous = PyUnicode_InternFromString("is_contiguous");
  return PyModule_Create(&module);
}
