// CPython binding of the C ABI for calls that are made thousands of times per training step.
//
// What bounds such a program is the host: the driver's launch call takes 2.3 us and a call through
// ctypes with a dozen arguments another 2 to 3 us on top (argument objects, type checks, a Python
// frame for the return code).  Here every entry point gets a wrapper generated from its own
// declaration: each argument goes from the interpreter's object to a register, the library is called
// with the GIL released (as ctypes does), and only a failure returns to Python code.  Measured on an
// elementwise operation of 64 elements, back to back: 5.3 us per call through ctypes, 2.7 us here.
//
// An argument that is neither a number nor None (a ctypes array or reference) is left to the ctypes
// path: the wrappers report it and the call goes to the fallback it was created with.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <cstdint>
#include <cstddef>
#include <tuple>
#include <type_traits>
#include <utility>

#include "../../include/primitiv_b200_ops.h"

namespace {

// One argument.  False: not a plain value, or (with the error indicator set) a failed conversion.
template <typename T>
inline bool convert(PyObject *o, T *out) {
  if constexpr (std::is_floating_point<T>::value) {
    if (PyFloat_CheckExact(o)) {
      *out = static_cast<T>(PyFloat_AS_DOUBLE(o));
      return true;
    }
    if (!PyLong_Check(o)) return false;
    const double v = PyLong_AsDouble(o);
    if (v == -1.0 && PyErr_Occurred()) return false;
    *out = static_cast<T>(v);
    return true;
  } else {
    if (PyLong_Check(o)) {
      // as ctypes does, integers are taken modulo the parameter's width
      const unsigned long long v = PyLong_AsUnsignedLongLongMask(o);
      if (v == static_cast<unsigned long long>(-1) && PyErr_Occurred()) return false;
      if constexpr (std::is_pointer<T>::value) *out = reinterpret_cast<T>(static_cast<std::uintptr_t>(v));
      else *out = static_cast<T>(v);
      return true;
    }
    if constexpr (std::is_pointer<T>::value) {
      if (o == Py_None) {
        *out = nullptr;
        return true;
      }
    }
    return false;
  }
}

enum { kNotPlain = -1 };   // no code of the library is negative

// Calls Fn(ctx, args...) and returns its code, or kNotPlain without calling it.
typedef long (*Wrapper)(b200_ctx *, PyObject *const *, Py_ssize_t);

template <auto Fn>
struct Wrap;
template <typename... A, int (*Fn)(b200_ctx *, A...)>
struct Wrap<Fn> {
  template <std::size_t... I>
  static long run(b200_ctx *ctx, PyObject *const *args, std::index_sequence<I...>) {
    std::tuple<A...> v;
    if (!(convert(args[I], &std::get<I>(v)) && ...)) return kNotPlain;
    long code;
    Py_BEGIN_ALLOW_THREADS
    code = Fn(ctx, std::get<I>(v)...);
    Py_END_ALLOW_THREADS
    return code;
  }
  static long call(b200_ctx *ctx, PyObject *const *args, Py_ssize_t n) {
    if (n != static_cast<Py_ssize_t>(sizeof...(A))) return kNotPlain;   // ctypes words the error
    return run(ctx, args, std::index_sequence_for<A...>{});
  }
};

struct Named {
  const char *name;
  Wrapper fn;
};
#define B200_ENTRY(name) {#name, &Wrap<&name>::call}
const Named kEntries[] = {
    B200_ENTRY(b200_matmul_fw), B200_ENTRY(b200_matmul_bw), B200_ENTRY(b200_matmul_bw_ex),
    B200_ENTRY(b200_matmul_fw_bw_host), B200_ENTRY(b200_gemm), B200_ENTRY(b200_operand_cache_invalidate),
    B200_ENTRY(b200_unary_fw), B200_ENTRY(b200_unary_bw), B200_ENTRY(b200_scalar_fw), B200_ENTRY(b200_binary_fw),
    B200_ENTRY(b200_binary_bw), B200_ENTRY(b200_inplace_add), B200_ENTRY(b200_inplace_add_ex),
    B200_ENTRY(b200_inplace_multiply_const), B200_ENTRY(b200_fill), B200_ENTRY(b200_identity),
    B200_ENTRY(b200_im2col), B200_ENTRY(b200_col2im), B200_ENTRY(b200_max_pool2d_fw), B200_ENTRY(b200_max_pool2d_bw),
    B200_ENTRY(b200_upload), B200_ENTRY(b200_download), B200_ENTRY(b200_copy), B200_ENTRY(b200_slice_fw),
    B200_ENTRY(b200_slice_bw), B200_ENTRY(b200_slice_bw_ex), B200_ENTRY(b200_concat_part), B200_ENTRY(b200_pick_fw),
    B200_ENTRY(b200_pick_bw), B200_ENTRY(b200_broadcast_fw), B200_ENTRY(b200_batch_pick_fw),
    B200_ENTRY(b200_batch_pick_bw), B200_ENTRY(b200_transpose), B200_ENTRY(b200_permute_dims), B200_ENTRY(b200_flip),
    B200_ENTRY(b200_reduce_fw), B200_ENTRY(b200_minmax_bw), B200_ENTRY(b200_argminmax), B200_ENTRY(b200_batch_sum_fw),
    B200_ENTRY(b200_random),
};
#undef B200_ENTRY

PyObject *g_by_name = nullptr;    // name -> capsule-free integer: index into kEntries

// ---- Caller: op(name, *args) ----
//
// It comes in two forms.  Over a fixed address it is a function of one context, whose owner outlives it.  Without one it is a
// method, to be an attribute of a class: it is called with the object first and takes the context's address from
// that object's `_address`, an integer, at each call.  The object is then kept alive by whoever holds the bound
// method, a closed one has a 0 there, and a subclass can put its own method in place, as with a function
// written in Python.

struct Caller {
  PyObject_HEAD
  vectorcallfunc vectorcall;
  bool method;
  b200_ctx *ctx;        // unless it is a method
  PyObject *fallback;   // called with the same arguments for what the wrappers do not take
  PyObject *fail;       // called with (code, name); raises
};

PyObject *g_address = nullptr;   // "_address"

// The context of the object that a method is called on.  False, with no error set: it has no such integer.
bool context_of(PyObject *object, b200_ctx **ctx) {
  PyObject *address = PyObject_GetAttr(object, g_address);
  const bool ok = address && PyLong_Check(address);
  if (ok) *ctx = static_cast<b200_ctx *>(PyLong_AsVoidPtr(address));
  Py_XDECREF(address);
  if (!PyErr_Occurred()) return ok;
  PyErr_Clear();
  return false;
}

PyObject *caller_call(PyObject *self, PyObject *const *args, size_t nargsf, PyObject *kwnames) {
  Caller *c = reinterpret_cast<Caller *>(self);
  const Py_ssize_t n = PyVectorcall_NARGS(nargsf), skip = c->method ? 1 : 0;
  if (n > skip && !kwnames && PyUnicode_CheckExact(args[skip])) {
    PyObject *at = PyDict_GetItemWithError(g_by_name, args[skip]);   // borrowed
    if (!at && PyErr_Occurred()) return nullptr;
    b200_ctx *ctx = c->ctx;
    if (at && (!c->method || context_of(args[0], &ctx))) {
      const long code = kEntries[PyLong_AsLong(at)].fn(ctx, args + skip + 1, n - skip - 1);
      if (code == 0) Py_RETURN_NONE;
      if (code > 0) return PyObject_CallFunction(c->fail, "lO", code, args[skip]);
      if (PyErr_Occurred()) return nullptr;
    }
  }
  return PyObject_Vectorcall(c->fallback, args, nargsf, kwnames);
}

PyObject *caller_get(PyObject *self, PyObject *object, PyObject *) {
  return object ? PyMethod_New(self, object) : Py_NewRef(self);
}

int caller_traverse(PyObject *self, visitproc visit, void *arg) {
  Py_VISIT(reinterpret_cast<Caller *>(self)->fallback);
  Py_VISIT(reinterpret_cast<Caller *>(self)->fail);
  return 0;
}

int caller_clear(PyObject *self) {
  Py_CLEAR(reinterpret_cast<Caller *>(self)->fallback);
  Py_CLEAR(reinterpret_cast<Caller *>(self)->fail);
  return 0;
}

void caller_dealloc(PyObject *self) {
  PyObject_GC_UnTrack(self);
  caller_clear(self);
  PyObject_GC_Del(self);
}

PyTypeObject caller_type = {PyVarObject_HEAD_INIT(nullptr, 0)};

PyObject *make_caller(PyObject *, PyObject *args) {
  PyObject *address, *fallback, *fail;
  if (!PyArg_ParseTuple(args, "OOO", &address, &fallback, &fail)) return nullptr;
  std::uintptr_t ctx = 0;
  if (address != Py_None) {
    ctx = reinterpret_cast<std::uintptr_t>(PyLong_AsVoidPtr(address));
    if (!ctx && PyErr_Occurred()) return nullptr;
  }
  Caller *c = PyObject_GC_New(Caller, &caller_type);
  if (!c) return nullptr;
  c->vectorcall = caller_call;
  c->method = address == Py_None;
  c->ctx = reinterpret_cast<b200_ctx *>(ctx);
  c->fallback = Py_NewRef(fallback);
  c->fail = Py_NewRef(fail);
  PyObject_GC_Track(reinterpret_cast<PyObject *>(c));
  return reinterpret_cast<PyObject *>(c);
}

PyMethodDef methods[] = {
    {"caller", make_caller, METH_VARARGS,
     "caller(context, fallback, fail): op(name, *args) of the context at that address, or with None a method of objects with an `_address`"},
    {nullptr, nullptr, 0, nullptr},
};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_native", "Fast calls into libprimitiv_b200.so", -1, methods,
                      nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native() {
  caller_type.tp_name = "primitiv_b200._native.Caller";
  caller_type.tp_basicsize = sizeof(Caller);
  caller_type.tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_GC | Py_TPFLAGS_HAVE_VECTORCALL | Py_TPFLAGS_METHOD_DESCRIPTOR;
  caller_type.tp_vectorcall_offset = offsetof(Caller, vectorcall);
  caller_type.tp_call = PyVectorcall_Call;
  caller_type.tp_descr_get = caller_get;
  caller_type.tp_traverse = caller_traverse;
  caller_type.tp_clear = caller_clear;
  caller_type.tp_dealloc = caller_dealloc;
  if (PyType_Ready(&caller_type) < 0) return nullptr;
  g_by_name = PyDict_New();
  g_address = PyUnicode_InternFromString("_address");
  if (!g_by_name || !g_address) return nullptr;
  for (long i = 0; i < static_cast<long>(sizeof(kEntries) / sizeof(kEntries[0])); ++i) {
    PyObject *at = PyLong_FromLong(i);
    if (!at || PyDict_SetItemString(g_by_name, kEntries[i].name, at) < 0) return nullptr;
    Py_DECREF(at);
  }
  return PyModule_Create(&module);
}
