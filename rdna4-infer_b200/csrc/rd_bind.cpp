// Python callables for the entry points of a layer loop, without ctypes.
//
// ctypes converts the 17 arguments of a decode call in 4.3 us -- more than the call itself, and with
// the pre-attention call twice per layer more than the GPU needs for a short context. Here every
// argument is converted by the type that include/rd_attn.h declares for it: about 0.3 us. Anything but
// plain numbers and None (a ctypes byref, an array, a wrong type) goes to the ctypes function.
//
// The module does not link the library: install(name, address, fallback) binds one entry point.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <cstring>
#include <tuple>
#include <type_traits>
#include <utility>

#include "rd_attn.h"

namespace {

template <class T>
bool convert(PyObject *o, T &out) {
  if constexpr (std::is_pointer_v<T>) {
    if (o == Py_None) {
      out = nullptr;
      return true;
    }
    if (!PyLong_Check(o)) return false;
    out = reinterpret_cast<T>(PyLong_AsUnsignedLongLongMask(o));
    return true;
  } else if constexpr (std::is_floating_point_v<T>) {
    if (PyFloat_CheckExact(o)) {
      out = (T)PyFloat_AS_DOUBLE(o);
      return true;
    }
    if (!PyLong_CheckExact(o)) return false;
    const double d = PyLong_AsDouble(o);
    if (d == -1.0 && PyErr_Occurred()) {
      PyErr_Clear();
      return false;
    }
    out = (T)d;
    return true;
  } else {
    if (!PyLong_Check(o)) return false;
    out = (T)PyLong_AsUnsignedLongLongMask(o);   // out of range: wraps, as ctypes does
    return true;
  }
}

// One entry point (told apart by N): its address, and the ctypes function for what this one does not take.
template <int N, class F>
struct Entry;
template <int N, class R, class... A>
struct Entry<N, R (*)(A...)> {
  static inline R (*fn)(A...) = nullptr;
  static inline PyObject *fallback = nullptr;

  template <size_t... I>
  static bool take(PyObject *const *args, std::tuple<A...> &a, std::index_sequence<I...>) {
    return (convert(args[I], std::get<I>(a)) && ...);
  }
  static PyObject *py(PyObject *, PyObject *const *args, Py_ssize_t n) {
    std::tuple<A...> a;
    if (n != (Py_ssize_t)sizeof...(A) || !take(args, a, std::index_sequence_for<A...>()))
      return PyObject_Vectorcall(fallback, args, (size_t)n, nullptr);
    R r;
    Py_BEGIN_ALLOW_THREADS
    r = std::apply(fn, a);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong((long)r);
  }
  static void set(void *address, PyObject *ctypes_function) {
    fn = reinterpret_cast<R (*)(A...)>(address);
    Py_INCREF(ctypes_function);
    Py_XSETREF(fallback, ctypes_function);
  }
};

struct Bound {
  void (*set)(void *, PyObject *);
  PyMethodDef def;
};
#define RD_ENTRY(name)                                                                                  \
  {&Entry<__LINE__, decltype(&::name)>::set,                                                            \
   {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(                                  \
               &Entry<__LINE__, decltype(&::name)>::py)),                                               \
    METH_FASTCALL, "see include/rd_attn.h"}},

Bound g_entries[] = {
    RD_ENTRY(rd_kv_store_rows)
    RD_ENTRY(rd_kv_append)
    RD_ENTRY(rd_rope)
    RD_ENTRY(rd_deinterleave_q_gate)
    RD_ENTRY(rd_sigmoid_gate)
    RD_ENTRY(rd_rms_norm)
    RD_ENTRY(rd_pre_attn_fused)
    RD_ENTRY(rd_attn_decode)
    RD_ENTRY(rd_attn_decode_split)
    RD_ENTRY(rd_attn_decode_ws)
    RD_ENTRY(rd_attn_decode_append_ws)
    RD_ENTRY(rd_attn_decode_multi)
    RD_ENTRY(rd_attn_multi_plan)
    RD_ENTRY(rd_attn_multi_launch)
    RD_ENTRY(rd_attn_decode_sharded)
    RD_ENTRY(rd_attn_decode_sharded_append)
    RD_ENTRY(rd_attn_shard_push)
    RD_ENTRY(rd_attn_shard_merge)
    RD_ENTRY(rd_attn_decode_noalloc)
    RD_ENTRY(rd_attn_merge)
    RD_ENTRY(rd_attn_batch)
    RD_ENTRY(rd_attn_split_batch)
    RD_ENTRY(rd_fa2_prefill)
    RD_ENTRY(rd_attn_prefill_fused)
    RD_ENTRY(rd_attn_prefill_append_fused)
    RD_ENTRY(rd_attn_prefill_typed)
};

// install(name, address, ctypes function) -> callable, or None for an entry that is not bound here
PyObject *install(PyObject *, PyObject *args) {
  const char *name;
  unsigned long long address;
  PyObject *ctypes_function;
  if (!PyArg_ParseTuple(args, "sKO", &name, &address, &ctypes_function)) return nullptr;
  for (Bound &b : g_entries)
    if (std::strcmp(b.def.ml_name, name) == 0) {
      b.set(reinterpret_cast<void *>(address), ctypes_function);
      return PyCFunction_New(&b.def, nullptr);
    }
  Py_RETURN_NONE;
}

PyMethodDef g_methods[] = {{"install", install, METH_VARARGS, nullptr}, {nullptr, nullptr, 0, nullptr}};
PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_rd_bind", nullptr, -1, g_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__rd_bind(void) { return PyModule_Create(&g_module); }
