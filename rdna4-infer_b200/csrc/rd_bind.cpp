// Python callables for the entry points of a layer loop, without ctypes.
//
// ctypes converts the 17 arguments of a decode call in 4.3 us -- more than the call itself, and with
// the pre-attention call twice per layer more than the GPU needs for a short context. Here every
// argument is converted by the type that include/rd_attn.h declares for it: about 0.3 us. Anything but
// plain numbers and None (a ctypes byref, an array, a wrong type) goes to the ctypes function.
//
// The module does not link the library: install(name, address, fallback) gives a callable for one entry point of
// one library. What it is bound to belongs to the callable, so libraries loaded side by side keep their own.
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

// What a callable is bound to: the entry point, and the ctypes function for what convert does not take.
struct Binding {
  void *address;
  PyObject *fallback;
};
constexpr const char *kBinding = "rd_bind.binding";
void release(PyObject *self) {
  Binding *b = static_cast<Binding *>(PyCapsule_GetPointer(self, kBinding));
  Py_XDECREF(b->fallback);
  delete b;
}

template <class F>
struct Entry;
template <class R, class... A>
struct Entry<R (*)(A...)> {
  template <size_t... I>
  static bool take(PyObject *const *args, std::tuple<A...> &a, std::index_sequence<I...>) {
    return (convert(args[I], std::get<I>(a)) && ...);
  }
  static PyObject *py(PyObject *self, PyObject *const *args, Py_ssize_t n) {
    const Binding *b = static_cast<const Binding *>(PyCapsule_GetPointer(self, kBinding));
    if (b == nullptr) return nullptr;
    std::tuple<A...> a;
    if (n != (Py_ssize_t)sizeof...(A) || !take(args, a, std::index_sequence_for<A...>()))
      return PyObject_Vectorcall(b->fallback, args, (size_t)n, nullptr);
    R r;
    Py_BEGIN_ALLOW_THREADS
    r = std::apply(reinterpret_cast<R (*)(A...)>(b->address), a);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong((long)r);
  }
};

#define RD_ENTRY(name)                                                                                             \
  {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(Entry<decltype(&::name)>::py)), METH_FASTCALL, \
   "see include/rd_attn.h"},

PyMethodDef g_entries[] = {
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
  for (PyMethodDef &def : g_entries)
    if (std::strcmp(def.ml_name, name) == 0) {
      Binding *b = new Binding{reinterpret_cast<void *>(address), Py_NewRef(ctypes_function)};
      PyObject *self = PyCapsule_New(b, kBinding, release);
      if (self == nullptr) {
        Py_DECREF(b->fallback);
        delete b;
        return nullptr;
      }
      PyObject *callable = PyCFunction_New(&def, self);
      Py_DECREF(self);
      return callable;
    }
  Py_RETURN_NONE;
}

PyMethodDef g_methods[] = {{"install", install, METH_VARARGS, nullptr}, {nullptr, nullptr, 0, nullptr}};
PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_rd_bind", nullptr, -1, g_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__rd_bind(void) { return PyModule_Create(&g_module); }
