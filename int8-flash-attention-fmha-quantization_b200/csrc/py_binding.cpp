// Native Python binding of the C ABI (include/fmha_i8_c.h): reads the descriptor objects, tensor addresses and the
// stream straight from the Python arguments and calls the library with the GIL released.
//
// Why it exists: a forward call on a short sequence keeps the GPU busy for 5-7 us, and building the same call from
// ctypes arrays and torch.cuda.current_stream() costs about 8 us of Python per call (measured on the B200 host: two
// descriptor arrays 1.1 us, five addresses 1.3 us, the stream object 3.6 us, the foreign call 1.5 us), so the host was
// what bounded it.
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <cstdint>

#include "../../include/fmha_i8_c.h"

namespace {

PyObject *s_q_amax, *s_k_amax, *s_v_amax, *s_o_amax, *s_s_max;
PyObject *s_batch_num, *s_seq_len, *s_seq_len_q, *s_seq_len_k, *s_head_num, *s_head_dim;
PyObject *s_data_ptr, *s_ctypes, *s_data, *s_cuda_stream;

// torch's raw-stream getters (device index -> stream handle, and the current device index), once torch's CUDA state is
// initialised; until then the Python-level slow path, which initialises it.
PyObject *g_raw_stream, *g_get_device, *g_slow_stream;

bool get_float(PyObject* obj, PyObject* name, float* out) {
  PyObject* v = PyObject_GetAttr(obj, name);
  if (!v) return false;
  const double d = PyFloat_AsDouble(v);
  Py_DECREF(v);
  if (d == -1.0 && PyErr_Occurred()) return false;
  *out = static_cast<float>(d);
  return true;
}
bool get_int(PyObject* obj, PyObject* name, int* out) {
  PyObject* v = PyObject_GetAttr(obj, name);
  if (!v) return false;
  PyObject* i = PyNumber_Index(v);
  Py_DECREF(v);
  if (!i) return false;
  *out = static_cast<int>(PyLong_AsUnsignedLongLongMask(i));
  Py_DECREF(i);
  return true;
}
// Whatever int() takes.
bool as_int(PyObject* v, int* out) {
  PyObject* i = PyNumber_Long(v);
  if (!i) return false;
  *out = static_cast<int>(PyLong_AsUnsignedLongLongMask(i));
  Py_DECREF(i);
  return true;
}
bool as_address(PyObject* v, void** out) {
  const unsigned long long a = PyLong_AsUnsignedLongLongMask(v);
  if (a == static_cast<unsigned long long>(-1) && PyErr_Occurred()) return false;
  *out = reinterpret_cast<void*>(static_cast<uintptr_t>(a));
  return true;
}

// Device or host address of None, an int, a torch tensor or a numpy array.
bool get_ptr(PyObject* x, void** out) {
  if (x == Py_None) { *out = nullptr; return true; }
  if (PyLong_Check(x)) return as_address(x, out);
  PyObject* r = PyObject_CallMethodNoArgs(x, s_data_ptr);
  if (!r && PyErr_ExceptionMatches(PyExc_AttributeError)) {
    PyErr_Clear();
    PyObject* c = PyObject_GetAttr(x, s_ctypes);
    if (c) {
      r = PyObject_GetAttr(c, s_data);
      Py_DECREF(c);
    } else {
      PyErr_Clear();
      PyErr_Format(PyExc_TypeError, "cannot take the address of %R", reinterpret_cast<PyObject*>(Py_TYPE(x)));
    }
  }
  if (!r) return false;
  const bool ok = as_address(r, out);
  Py_DECREF(r);
  return ok;
}

bool get_stream(PyObject* s, void** out) {
  PyObject* r;
  if (s == Py_None) {
    if (g_raw_stream) {
      PyObject* dev = PyObject_CallNoArgs(g_get_device);
      if (!dev) return false;
      r = PyObject_CallOneArg(g_raw_stream, dev);
      Py_DECREF(dev);
    } else {
      r = PyObject_CallNoArgs(g_slow_stream);
    }
  } else if (PyLong_Check(s)) {
    return as_address(s, out);
  } else {
    r = PyObject_GetAttr(s, s_cuda_stream);
  }
  if (!r) return false;
  const bool ok = as_address(r, out);
  Py_DECREF(r);
  return ok;
}

bool get_param(PyObject* p, float (&a)[5]) {
  return get_float(p, s_q_amax, &a[0]) && get_float(p, s_k_amax, &a[1]) && get_float(p, s_v_amax, &a[2]) && get_float(p, s_o_amax, &a[3]) &&
         get_float(p, s_s_max, &a[4]);
}
bool get_desc4(PyObject* d, int (&a)[4]) {
  return get_int(d, s_batch_num, &a[0]) && get_int(d, s_seq_len, &a[1]) && get_int(d, s_head_num, &a[2]) && get_int(d, s_head_dim, &a[3]);
}
bool get_desc5(PyObject* d, int (&a)[5]) {
  return get_int(d, s_batch_num, &a[0]) && get_int(d, s_seq_len_q, &a[1]) && get_int(d, s_seq_len_k, &a[2]) && get_int(d, s_head_num, &a[3]) &&
         get_int(d, s_head_dim, &a[4]);
}
bool want(Py_ssize_t got, Py_ssize_t n) {
  if (got == n) return true;
  PyErr_Format(PyExc_TypeError, "expected %zd arguments, got %zd", n, got);
  return false;
}

// infer(stream, param, desc, q, k, v, mask, o, flags) -> status
PyObject* py_infer(PyObject*, PyObject* const* a, Py_ssize_t n) {
  void *stream, *t[5];
  float amax[5];
  int desc[4], flags, st;
  if (!want(n, 9) || !get_stream(a[0], &stream) || !get_param(a[1], amax) || !get_desc4(a[2], desc) || !as_int(a[8], &flags)) return nullptr;
  for (int i = 0; i < 5; ++i)
    if (!get_ptr(a[3 + i], &t[i])) return nullptr;
  Py_BEGIN_ALLOW_THREADS
  st = fmha_i8_sm100_infer(stream, amax, desc, t[0], t[1], t[2], t[3], t[4], static_cast<unsigned>(flags));
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(st);
}

// infer_slice(stream, param, desc, q, k, v, mask, o, bh_begin, bh_count, flags) -> status
PyObject* py_infer_slice(PyObject*, PyObject* const* a, Py_ssize_t n) {
  void *stream, *t[5];
  float amax[5];
  int desc[4], begin, count, flags, st;
  if (!want(n, 11) || !get_stream(a[0], &stream) || !get_param(a[1], amax) || !get_desc4(a[2], desc) || !as_int(a[8], &begin) ||
      !as_int(a[9], &count) || !as_int(a[10], &flags))
    return nullptr;
  for (int i = 0; i < 5; ++i)
    if (!get_ptr(a[3 + i], &t[i])) return nullptr;
  Py_BEGIN_ALLOW_THREADS
  st = fmha_i8_sm100_infer_slice(stream, amax, desc, t[0], t[1], t[2], t[3], t[4], begin, count, static_cast<unsigned>(flags));
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(st);
}

// bh_count == None: all heads from bh_begin on
bool get_slice(PyObject* begin, PyObject* count, const int (&desc)[5], int* b, int* c) {
  if (!as_int(begin, b)) return false;
  if (count == Py_None) {
    *c = static_cast<int>(static_cast<long long>(desc[0]) * desc[3] - *b);
    return true;
  }
  return as_int(count, c);
}

// infer_cross(stream, param, desc_x, q, k, v, mask, o, bh_begin, bh_count, flags) -> status
PyObject* py_infer_cross(PyObject*, PyObject* const* a, Py_ssize_t n) {
  void *stream, *t[5];
  float amax[5];
  int desc[5], begin, count, flags, st;
  if (!want(n, 11) || !get_stream(a[0], &stream) || !get_param(a[1], amax) || !get_desc5(a[2], desc) || !get_slice(a[8], a[9], desc, &begin, &count) ||
      !as_int(a[10], &flags))
    return nullptr;
  for (int i = 0; i < 5; ++i)
    if (!get_ptr(a[3 + i], &t[i])) return nullptr;
  Py_BEGIN_ALLOW_THREADS
  st = fmha_i8_sm100_infer_cross(stream, amax, desc, t[0], t[1], t[2], t[3], t[4], begin, count, static_cast<unsigned>(flags));
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(st);
}

// infer_policy(stream, param, desc_x, q, k, v, mask, o, bh_begin, bh_count, flags, policy, row_scratch) -> status
PyObject* py_infer_policy(PyObject*, PyObject* const* a, Py_ssize_t n) {
  void *stream, *t[5], *scratch;
  float amax[5];
  int desc[5], begin, count, flags, policy, st;
  if (!want(n, 13) || !get_stream(a[0], &stream) || !get_param(a[1], amax) || !get_desc5(a[2], desc) || !get_slice(a[8], a[9], desc, &begin, &count) ||
      !as_int(a[10], &flags) || !as_int(a[11], &policy) || !get_ptr(a[12], &scratch))
    return nullptr;
  for (int i = 0; i < 5; ++i)
    if (!get_ptr(a[3 + i], &t[i])) return nullptr;
  Py_BEGIN_ALLOW_THREADS
  st = fmha_i8_sm100_infer_policy(stream, amax, desc, t[0], t[1], t[2], t[3], t[4], begin, count, static_cast<unsigned>(flags), policy,
                                  static_cast<float*>(scratch));
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(st);
}

// infer_host(param, desc, q, k, v, mask, o, bh_begin, bh_count, flags) -> status; bh_begin None: the whole problem
PyObject* py_infer_host(PyObject*, PyObject* const* a, Py_ssize_t n) {
  void* t[5];
  float amax[5];
  int desc[4], begin = 0, count = 0, flags, st;
  if (!want(n, 10) || !get_param(a[0], amax) || !get_desc4(a[1], desc) || !as_int(a[9], &flags)) return nullptr;
  const bool whole = a[7] == Py_None;
  if (!whole && (!as_int(a[7], &begin) || !as_int(a[8], &count))) return nullptr;
  for (int i = 0; i < 5; ++i)
    if (!get_ptr(a[2 + i], &t[i])) return nullptr;
  Py_BEGIN_ALLOW_THREADS
  st = whole ? fmha_i8_sm100_infer_host(amax, desc, t[0], t[1], t[2], t[3], t[4], static_cast<unsigned>(flags))
             : fmha_i8_sm100_infer_host_slice(amax, desc, t[0], t[1], t[2], t[3], t[4], begin, count, static_cast<unsigned>(flags));
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(st);
}

// quantize(stream, x, n, out, amax_out, no_alloc) -> status
PyObject* py_quantize(PyObject*, PyObject* const* a, Py_ssize_t n) {
  void *stream, *x, *out, *amax;
  int st;
  if (!want(n, 6) || !get_stream(a[0], &stream) || !get_ptr(a[1], &x) || !get_ptr(a[3], &out) || !get_ptr(a[4], &amax)) return nullptr;
  const long long count = PyLong_AsLongLong(a[2]);
  if (count == -1 && PyErr_Occurred()) return nullptr;
  const int no_alloc = PyObject_IsTrue(a[5]);
  if (no_alloc < 0) return nullptr;
  Py_BEGIN_ALLOW_THREADS
  st = (no_alloc ? fmha_i8_sm100_quantize_f32_noalloc : fmha_i8_sm100_quantize_f32)(stream, static_cast<const float*>(x), count,
                                                                                    static_cast<int8_t*>(out), static_cast<float*>(amax));
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(st);
}

// set_stream_source(slow) before first use; set_raw_stream(raw_stream, get_device) once torch's CUDA state exists
PyObject* py_set_stream_source(PyObject*, PyObject* slow) {
  Py_INCREF(slow);
  Py_XSETREF(g_slow_stream, slow);
  Py_RETURN_NONE;
}
PyObject* py_set_raw_stream(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (!want(n, 2)) return nullptr;
  Py_INCREF(a[1]);
  Py_XSETREF(g_get_device, a[1]);
  Py_INCREF(a[0]);
  Py_XSETREF(g_raw_stream, a[0]);
  Py_RETURN_NONE;
}

#define FAST(name) reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(name)), METH_FASTCALL, nullptr
PyMethodDef g_methods[] = {
    {"infer", FAST(py_infer)},
    {"infer_slice", FAST(py_infer_slice)},
    {"infer_cross", FAST(py_infer_cross)},
    {"infer_policy", FAST(py_infer_policy)},
    {"infer_host", FAST(py_infer_host)},
    {"quantize", FAST(py_quantize)},
    {"set_stream_source", py_set_stream_source, METH_O, nullptr},
    {"set_raw_stream", FAST(py_set_raw_stream)},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_fmha_i8_py", nullptr, -1, g_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__fmha_i8_py(void) {
  struct { PyObject** slot; const char* text; } names[] = {
      {&s_q_amax, "q_amax"}, {&s_k_amax, "k_amax"}, {&s_v_amax, "v_amax"}, {&s_o_amax, "o_amax"}, {&s_s_max, "s_max"},
      {&s_batch_num, "batch_num"}, {&s_seq_len, "seq_len"}, {&s_seq_len_q, "seq_len_q"}, {&s_seq_len_k, "seq_len_k"},
      {&s_head_num, "head_num"}, {&s_head_dim, "head_dim"}, {&s_data_ptr, "data_ptr"}, {&s_ctypes, "ctypes"}, {&s_data, "data"},
      {&s_cuda_stream, "cuda_stream"}};
  for (auto& x : names)
    if (!(*x.slot = PyUnicode_InternFromString(x.text))) return nullptr;
  return PyModule_Create(&g_module);
}
