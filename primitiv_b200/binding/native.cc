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
// path: the wrappers report it and `op` hands the call to the fallback it was created with.
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

// ---- Caller: op(name, *args) of one context ---------------------------------------------------

struct Caller {
  PyObject_HEAD
  vectorcallfunc vectorcall;
  b200_ctx *ctx;
  PyObject *fallback;   // called with (name, *args) for what the wrappers do not take
  PyObject *fail;       // called with (code, name); raises
};

PyObject *caller_call(PyObject *self, PyObject *const *args, size_t nargsf, PyObject *kwnames) {
  Caller *c = reinterpret_cast<Caller *>(self);
  const Py_ssize_t n = PyVectorcall_NARGS(nargsf);
  if (n >= 1 && !kwnames && PyUnicode_CheckExact(args[0])) {
    PyObject *at = PyDict_GetItemWithError(g_by_name, args[0]);   // borrowed
    if (!at && PyErr_Occurred()) return nullptr;
    if (at) {
      const long code = kEntries[PyLong_AsLong(at)].fn(c->ctx, args + 1, n - 1);
      if (code == 0) Py_RETURN_NONE;
      if (code > 0) return PyObject_CallFunction(c->fail, "lO", code, args[0]);
      if (PyErr_Occurred()) return nullptr;
    }
  }
  return PyObject_Vectorcall(c->fallback, args, nargsf, kwnames);
}

int caller_traverse(PyObject *self, visitproc visit, void *arg) {
  Py_VISIT(reinterpret_cast<Caller *>(self)->fallback);
  Py_VISIT(reinterpret_cast<Caller *>(self)->fail);
  return 0;
}

void caller_dealloc(PyObject *self) {
  PyObject_GC_UnTrack(self);
  Py_CLEAR(reinterpret_cast<Caller *>(self)->fallback);
  Py_CLEAR(reinterpret_cast<Caller *>(self)->fail);
  PyObject_GC_Del(self);
}

PyTypeObject caller_type = {PyVarObject_HEAD_INIT(nullptr, 0)};

PyObject *make_caller(PyObject *, PyObject *args) {
  unsigned long long ctx = 0;
  PyObject *fallback, *fail;
  if (!PyArg_ParseTuple(args, "KOO", &ctx, &fallback, &fail)) return nullptr;
  Caller *c = PyObject_GC_New(Caller, &caller_type);
  if (!c) return nullptr;
  c->vectorcall = caller_call;
  c->ctx = reinterpret_cast<b200_ctx *>(static_cast<std::uintptr_t>(ctx));
  c->fallback = Py_NewRef(fallback);
  c->fail = Py_NewRef(fail);
  PyObject_GC_Track(reinterpret_cast<PyObject *>(c));
  return reinterpret_cast<PyObject *>(c);
}

PyMethodDef methods[] = {
    {"caller", make_caller, METH_VARARGS, "caller(context, fallback, fail): op(name, *args) of one context"},
    {nullptr, nullptr, 0, nullptr},
};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_native", "Fast calls into libprimitiv_b200.so", -1, methods,
                      nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native() {
  caller_type.tp_name = "primitiv_b200._native.Caller";
  caller_type.tp_basicsize = sizeof(Caller);
  caller_type.tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_GC | Py_TPFLAGS_HAVE_VECTORCALL;
  caller_type.tp_vectorcall_offset = offsetof(Caller, vectorcall);
  caller_type.tp_call = PyVectorcall_Call;
  caller_type.tp_traverse = caller_traverse;
  caller_type.tp_dealloc = caller_dealloc;
  if (PyType_Ready(&caller_type) < 0) return nullptr;
  g_by_name = PyDict_New();
  if (!g_by_name) return nullptr;
  for (long i = 0; i < static_cast<long>(sizeof(kEntries) / sizeof(kEntries[0])); ++i) {
    PyObject *at = PyLong_FromLong(i);
    if (!at || PyDict_SetItemString(g_by_name, kEntries[i].name, at) < 0) return nullptr;
    Py_DECREF(at);
  }
  return PyModule_Create(&module);
}
