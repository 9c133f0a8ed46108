// Calls from Python into libscirust_b200_cuda.so without ctypes: one typed function per entry point of the C ABI. A launch
// of the decode path has about 20 arguments, which ctypes turns into as many objects (4.8 us); a conversion here is one
// test and one read (0.5 us). Arguments are ints, None (a null pointer), arrays of ctypes (their address) and floats; anything
// else raises TypeError, and the caller (ops/_lib.py) makes that call through ctypes. Built by _build.py;
// py_calls.inc lists the entry points.
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <dlfcn.h>
#include <tuple>
#include <type_traits>
#include <utility>
#include "api.h"

namespace {

bool bad_arg(const char* want, PyObject* got) {
  PyErr_Format(PyExc_TypeError, "expected %s, got %s", want, Py_TYPE(got)->tp_name);
  return false;
}

PyTypeObject* ctypes_array = nullptr;            // _ctypes.Array

bool is_array(PyObject* o) { return PyType_IsSubtype(Py_TYPE(o), ctypes_array); }

// The address of a ctypes array; it stays where it is while the caller holds the array.
void* array_address(PyObject* o) {
  Py_buffer view;
  if (PyObject_GetBuffer(o, &view, PyBUF_SIMPLE)) return nullptr;
  void* at = view.buf;
  PyBuffer_Release(&view);
  return at;
}

template <class T>
bool read_arg(PyObject* o, T& out) {
  if constexpr (std::is_floating_point_v<T>) {
    if (PyFloat_Check(o)) out = static_cast<T>(PyFloat_AS_DOUBLE(o));
    else if (PyLong_Check(o)) out = static_cast<T>(PyLong_AsDouble(o));
    else return bad_arg("a number", o);
  } else {
    if constexpr (std::is_pointer_v<T>) {
      if (o == Py_None) { out = T{}; return true; }
      if (!PyLong_Check(o) && is_array(o)) { out = reinterpret_cast<T>(array_address(o)); return !PyErr_Occurred(); }
    }
    if (!PyLong_Check(o)) return bad_arg(std::is_pointer_v<T> ? "an address or None" : "an integer", o);
    const unsigned long long v = PyLong_AsUnsignedLongLongMask(o);       // out of range: the low bits, as ctypes does
    if constexpr (std::is_pointer_v<T>) out = reinterpret_cast<T>(static_cast<uintptr_t>(v));
    else out = static_cast<T>(v);
  }
  return !PyErr_Occurred();
}

template <class R, class... A, size_t... I>
PyObject* invoke(R (*fn)(A...), PyObject* const* args, Py_ssize_t n, std::index_sequence<I...>) {
  if (n != static_cast<Py_ssize_t>(sizeof...(A))) {
    PyErr_Format(PyExc_TypeError, "expected %zu arguments, got %zd", sizeof...(A), n);
    return nullptr;
  }
  std::tuple<std::remove_cv_t<A>...> v;
  if (!(read_arg(args[I], std::get<I>(v)) && ...)) return nullptr;
  R rc;
  Py_BEGIN_ALLOW_THREADS                       // a launch may wait for room in the queue
  rc = fn(std::get<I>(v)...);
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(static_cast<long>(rc));
}

template <class R, class... A>
PyObject* invoke(R (*fn)(A...), PyObject* const* args, Py_ssize_t n) {
  return invoke(fn, args, n, std::index_sequence_for<A...>{});
}

// One function per entry point; `at` is filled in by bind().
#define SB_ENTRY(name)                                                                     \
  void* at_##name = nullptr;                                                               \
  PyObject* call_##name(PyObject*, PyObject* const* args, Py_ssize_t n) {                  \
    return invoke(reinterpret_cast<decltype(&name)>(at_##name), args, n);                  \
  }                                                                                        \
  PyMethodDef def_##name = {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(call_##name)), METH_FASTCALL, nullptr};
#include "py_calls.inc"
#undef SB_ENTRY

// bind(path) -> {entry point: function} of the library at `path`, which the process has loaded already.
PyObject* bind(PyObject*, PyObject* arg) {
  const char* path = PyUnicode_AsUTF8(arg);
  if (!path) return nullptr;
  if (!ctypes_array) {
    PyObject* ctypes = PyImport_ImportModule("_ctypes");
    PyObject* array = ctypes ? PyObject_GetAttrString(ctypes, "Array") : nullptr;
    Py_XDECREF(ctypes);
    if (!array) return nullptr;
    if (!PyType_Check(array)) { Py_DECREF(array); return PyErr_Format(PyExc_TypeError, "_ctypes.Array is not a type"); }
    ctypes_array = reinterpret_cast<PyTypeObject*>(array);   // kept for the life of the process
  }
  void* lib = dlopen(path, RTLD_NOW | RTLD_NOLOAD);
  if (!lib) return PyErr_Format(PyExc_OSError, "%s is not loaded", path);
  PyObject* out = PyDict_New();
  if (!out) return nullptr;
#define SB_ENTRY(name)                                                                     \
  if ((at_##name = dlsym(lib, #name)) != nullptr) {                                        \
    PyObject* f = PyCFunction_New(&def_##name, nullptr);                                   \
    if (!f || PyDict_SetItemString(out, #name, f) < 0) { Py_XDECREF(f); Py_DECREF(out); return nullptr; } \
    Py_DECREF(f);                                                                          \
  }
#include "py_calls.inc"
#undef SB_ENTRY
  return out;
}

PyMethodDef methods[] = {{"bind", bind, METH_O, nullptr}, {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "sb_py_calls", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_sb_py_calls() {
  PyObject* m = PyModule_Create(&module);
  if (m && PyModule_AddStringConstant(m, "api_digest", SB_API_DIGEST) < 0) Py_CLEAR(m);   // of the api.h compiled in
  return m;
}
