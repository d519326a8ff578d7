// The operators a program calls once per layer, as functions of a CPython extension module: tensors are taken as they are and
// the call goes straight to the C ABI. Through ctypes a call spent 1.7 of its 4 to 5.5 us of host time on converting its
// arguments (the launch itself is most of the rest); here 0.5. Anything else goes through ctypes (_lib.py).
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include "../include/et_cuda.h"

namespace {

PyObject *g_data_ptr, *g_ctypes, *g_data;

// The address a tensor, array, integer or None stands for (as _ptr in __init__.py).
bool address(PyObject* o, void** out) {
  *out = nullptr;
  if (o == Py_None) return true;
  PyObject* number = nullptr;
  if (PyLong_Check(o)) {
    number = Py_NewRef(o);
  } else {
    number = PyObject_CallMethodNoArgs(o, g_data_ptr);
    if (!number && PyErr_ExceptionMatches(PyExc_AttributeError)) {  // a numpy array
      PyErr_Clear();
      PyObject* view = PyObject_GetAttr(o, g_ctypes);
      if (!view) return false;
      number = PyObject_GetAttr(view, g_data);
      Py_DECREF(view);
    }
  }
  if (!number) return false;
  *out = reinterpret_cast<void*>(PyLong_AsUnsignedLongLongMask(number));
  Py_DECREF(number);
  return !(PyErr_Occurred());
}

// Arguments one after the other; the first that cannot be converted leaves the Python error and ok == false.
struct Arguments {
  PyObject* const* args;
  Py_ssize_t left;
  bool ok;
  Arguments(PyObject* const* a, Py_ssize_t n, Py_ssize_t expected) : args(a), left(n), ok(n == expected) {
    if (!ok) PyErr_Format(PyExc_TypeError, "expected %zd arguments, got %zd", expected, n);
  }
  PyObject* next() { return ok && left-- > 0 ? *args++ : nullptr; }
  template <typename T = void>
  T* pointer() {
    void* p = nullptr;
    if (PyObject* o = next()) ok = address(o, &p);
    return reinterpret_cast<T*>(p);
  }
  unsigned long long bits() {  // as ctypes: whole numbers of any sign, cut to the parameter's width
    PyObject* o = next();
    if (!o) return 0;
    if (!PyIndex_Check(o)) {
      PyErr_Format(PyExc_TypeError, "expected a whole number, got %.100s", Py_TYPE(o)->tp_name);
      ok = false;
      return 0;
    }
    const unsigned long long v = PyLong_AsUnsignedLongLongMask(o);
    if (v == (unsigned long long)-1 && PyErr_Occurred()) ok = false;
    return v;
  }
  int64_t wide() { return (int64_t)bits(); }
  int narrow() { return (int)bits(); }
  double real() {
    PyObject* o = next();
    if (!o) return 0.0;
    const double v = PyFloat_AsDouble(o);
    if (v == -1.0 && PyErr_Occurred()) ok = false;
    return v;
  }
};

// Calls into the library without the interpreter's lock; the status, which the caller turns into its exception.
template <typename F>
PyObject* finish(const Arguments& a, F&& call) {
  if (!a.ok) return nullptr;
  int status;
  Py_BEGIN_ALLOW_THREADS
  status = (int)call();
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(status);
}

PyObject* dequantize_into(PyObject*, PyObject* const* args, Py_ssize_t n) {
  Arguments a(args, n, 6);
  auto* rt = a.pointer<etc_runtime>();
  const auto codec = (etc_codec)a.narrow();
  const void* packed = a.pointer();
  const int64_t rows = a.wide(), columns = a.wide();
  float* out = a.pointer<float>();
  return finish(a, [&] { return etc_dequantize_into(rt, codec, packed, rows, columns, out); });
}

PyObject* quantize_into(PyObject*, PyObject* const* args, Py_ssize_t n) {
  Arguments a(args, n, 6);
  auto* rt = a.pointer<etc_runtime>();
  const auto codec = (etc_codec)a.narrow();
  const float* x = a.pointer<float>();
  const int64_t rows = a.wide(), columns = a.wide();
  void* packed = a.pointer();
  return finish(a, [&] { return etc_quantize_into(rt, codec, x, rows, columns, packed); });
}

PyObject* qlinear_into(PyObject*, PyObject* const* args, Py_ssize_t n) {
  Arguments a(args, n, 9);
  auto* rt = a.pointer<etc_runtime>();
  const auto codec = (etc_codec)a.narrow();
  const float* x = a.pointer<float>();
  const int64_t vectors = a.wide(), columns = a.wide();
  const void* weight = a.pointer();
  const int64_t rows = a.wide();
  const float* bias = a.pointer<float>();
  float* out = a.pointer<float>();
  return finish(a, [&] { return etc_qlinear_into(rt, codec, x, vectors, columns, weight, rows, bias, out, nullptr); });
}

PyObject* qlinear_tiled_into(PyObject*, PyObject* const* args, Py_ssize_t n) {
  Arguments a(args, n, 10);
  auto* rt = a.pointer<etc_runtime>();
  const auto* w = a.pointer<etc_qweight>();
  const float* x = a.pointer<float>();
  const int64_t vectors = a.wide();
  const float *bias = a.pointer<float>(), *residual = a.pointer<float>();
  const auto epilogue = (etc_epilogue)a.narrow();
  float* out = a.pointer<float>();
  void* scratch = a.pointer();
  const size_t scratch_bytes = (size_t)a.bits();
  return finish(a, [&] { return etc_qlinear_tiled_into(rt, w, x, vectors, bias, residual, epilogue, out, scratch, scratch_bytes); });
}

PyObject* sample_rows_into(PyObject*, PyObject* const* args, Py_ssize_t n) {
  Arguments a(args, n, 12);
  auto* rt = a.pointer<etc_runtime>();
  const float* logits = a.pointer<float>();
  const int64_t rows = a.wide(), vocab = a.wide();
  const double temperature = a.real();
  const int64_t top_k = a.wide();
  const double top_p = a.real();
  const uint64_t seed = a.bits(), counter = a.bits();
  const uint64_t *seeds = a.pointer<uint64_t>(), *counters = a.pointer<uint64_t>();
  uint32_t* tokens = a.pointer<uint32_t>();
  return finish(a, [&] { return etc_sample_rows_into(rt, logits, rows, vocab, temperature, top_k, top_p, seed, counter, seeds, counters, tokens); });
}

PyObject* paged_attention_into(PyObject*, PyObject* const* args, Py_ssize_t n) {
  Arguments a(args, n, 14);
  auto* rt = a.pointer<etc_runtime>();
  auto* pool = a.pointer<etc_pool>();
  const int layer = a.narrow();
  const auto* lanes = a.pointer<etc_lane>();
  const int* tables = a.pointer<int>();
  const int batch = a.narrow(), max_pages = a.narrow();
  const float* q = a.pointer<float>();
  const int q_heads = a.narrow();
  const double scale = a.real();
  const int64_t window = a.wide();
  float* out = a.pointer<float>();
  void* scratch = a.pointer();
  const size_t scratch_bytes = (size_t)a.bits();
  return finish(a, [&] { return etc_paged_attention_into(rt, pool, layer, lanes, tables, batch, max_pages, q, q_heads, scale, window, out, scratch, scratch_bytes); });
}

#define CALL(name) {#name, (PyCFunction)(void (*)(void))name, METH_FASTCALL, nullptr}
PyMethodDef g_methods[] = {CALL(dequantize_into), CALL(quantize_into),    CALL(qlinear_into), CALL(qlinear_tiled_into),
                           CALL(sample_rows_into), CALL(paged_attention_into), {nullptr, nullptr, 0, nullptr}};
#undef CALL
PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_calls", "Operators of the C ABI without ctypes.", -1, g_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__calls() {
  g_data_ptr = PyUnicode_InternFromString("data_ptr");
  g_ctypes = PyUnicode_InternFromString("ctypes");
  g_data = PyUnicode_InternFromString("data");
  if (!g_data_ptr || !g_ctypes || !g_data) return nullptr;
  return PyModule_Create(&g_module);
}
