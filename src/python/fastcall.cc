// Calls of the native library with lists of tensors, for the Python front end.
//
// A small collective is bound by the way to its launch.  Through ctypes a call of eight ranks spent more than a third of its 7.2 us on packing addresses and converting a
// dozen arguments; here the addresses go from the tensors straight into the tables that the library takes.  (us per call of a small collective, ctypes and this: two ranks 5.7 / 3.9, four 6.4 / 4.3, eight 7.3 / 4.9.)
// The library's functions come as addresses, so that nothing here is linked against it.  The interpreter's lock is released around them, as ctypes does.
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <cstring>

namespace {

constexpr Py_ssize_t kMost = 64;
PyObject* g_data_ptr = nullptr;      // "data_ptr"

// Addresses of the tensors of a list or tuple; None where it is allowed: 0.
bool addresses(PyObject* seq, Py_ssize_t n, bool none, void** out) {
  PyObject* const fast = PySequence_Fast(seq, "a sequence of tensors is wanted");
  if (!fast) return false;
  bool ok = PySequence_Fast_GET_SIZE(fast) == n;
  if (!ok) PyErr_Format(PyExc_ValueError, "%zd tensors are wanted, one per rank, got %zd", n, PySequence_Fast_GET_SIZE(fast));
  for (Py_ssize_t i = 0; ok && i < n; i++) {
    PyObject* const t = PySequence_Fast_GET_ITEM(fast, i);
    if (none && t == Py_None) { out[i] = nullptr; continue; }
    PyObject* const p = PyObject_CallMethodNoArgs(t, g_data_ptr);
    if (!p) { ok = false; break; }
    out[i] = PyLong_AsVoidPtr(p);
    Py_DECREF(p);
    ok = !PyErr_Occurred();
  }
  Py_DECREF(fast);
  return ok;
}
bool comms(PyObject* bytes, Py_ssize_t n, void** out) {
  char* b; Py_ssize_t len;
  if (PyBytes_AsStringAndSize(bytes, &b, &len)) return false;
  if (n < 1 || n > kMost || len != n * (Py_ssize_t)sizeof(void*)) { PyErr_SetString(PyExc_ValueError, "a table of communicators is wanted"); return false; }
  memcpy(out, b, (size_t)len);
  return true;
}
bool ints(PyObject* const* args, int n, int* out) {
  for (int i = 0; i < n; i++) {
    const long v = PyLong_AsLong(args[i]);
    if (v == -1 && PyErr_Occurred()) return false;
    out[i] = (int)v;
  }
  return true;
}

// collective(function, communicators, nranks, send, recv, count, coll, dtype, op, root, algo, k, stream) -> code
PyObject* collective(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  typedef int (*Fn)(void**, int, int, const void* const*, void* const*, size_t, int, int, int, int, int, void*);
  if (nargs != 13) { PyErr_SetString(PyExc_TypeError, "13 arguments are wanted"); return nullptr; }
  const Fn fn = reinterpret_cast<Fn>(PyLong_AsVoidPtr(args[0]));
  const Py_ssize_t n = PyLong_AsSsize_t(args[2]);
  void *c[kMost], *send[kMost], *recv[kMost];
  int v[6];
  if (PyErr_Occurred() || !comms(args[1], n, c) || !addresses(args[3], n, false, send) || !addresses(args[4], n, true, recv)) return nullptr;
  const size_t count = PyLong_AsSize_t(args[5]);
  if (PyErr_Occurred() || !ints(args + 6, 6, v)) return nullptr;
  void* const stream = PyLong_AsVoidPtr(args[12]);
  if (PyErr_Occurred()) return nullptr;
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = fn(c, (int)n, v[0], send, recv, count, v[1], v[2], v[3], v[4], v[5], stream);
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(rc);
}
// product(function, communicators, nranks, A, B, out, M, N, K, stream) -> code
PyObject* product(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  typedef int (*Fn)(void**, int, const void* const*, const void* const*, void* const*, int, int, int, void*);
  if (nargs != 10) { PyErr_SetString(PyExc_TypeError, "10 arguments are wanted"); return nullptr; }
  const Fn fn = reinterpret_cast<Fn>(PyLong_AsVoidPtr(args[0]));
  const Py_ssize_t n = PyLong_AsSsize_t(args[2]);
  void *c[kMost], *a[kMost], *b[kMost], *out[kMost];
  int v[3];
  if (PyErr_Occurred() || !comms(args[1], n, c) || !addresses(args[3], n, false, a) || !addresses(args[4], n, false, b) || !addresses(args[5], n, false, out) || !ints(args + 6, 3, v)) return nullptr;
  void* const stream = PyLong_AsVoidPtr(args[9]);
  if (PyErr_Occurred()) return nullptr;
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = fn(c, (int)n, a, b, out, v[0], v[1], v[2], stream);
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(rc);
}

PyMethodDef g_methods[] = {{"collective", (PyCFunction)(void (*)(void))collective, METH_FASTCALL, nullptr}, {"product", (PyCFunction)(void (*)(void))product, METH_FASTCALL, nullptr}, {nullptr, nullptr, 0, nullptr}};
PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_fastcall", nullptr, -1, g_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__fastcall(void) {
  g_data_ptr = PyUnicode_InternFromString("data_ptr");
  return g_data_ptr ? PyModule_Create(&g_module) : nullptr;
}
