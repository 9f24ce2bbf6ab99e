// CPython calls of the C ABI: the calls that a decode step makes op by op, without ctypes' conversion of up to nineteen
// arguments (two to four microseconds a call, as long as the kernels of a small layer run).
//
// bind(name, address, slow, on_error) gives a callable for the library's function `name` at `address`.  The argument types come
// from include/tlcuda.h.  Integers, floats, pointers given as int or None and descriptors as bytes of their size are converted here, as
// ctypes does; a call with anything else (a ctypes pointer, an array, another kind of integer, too few arguments) goes to `slow`, the
// same call through ctypes, whose rules then hold.  A status other than TL_OK is handed to on_error(context, status), which raises.  The
// GIL is released around the call.  For tl_alloc the call is (context, bytes) and its result, as that of `slow`, the block's address.
// quant(scheme, group size, scales dtype, convention) and epilogue(ops, inputs) give the bytes of the descriptors.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <cstdint>
#include <cstring>
#include <iterator>
#include <tuple>
#include <type_traits>
#include <utility>

#include "../../include/tlcuda.h"

namespace {

template <typename T> bool convert(PyObject* o, T* out) {
  if constexpr (std::is_pointer_v<T>) {
    if (o == Py_None) { *out = nullptr; return true; }
    if (PyLong_Check(o)) { *out = reinterpret_cast<T>(static_cast<uintptr_t>(PyLong_AsUnsignedLongLongMask(o))); return true; }
    using Pointee = std::remove_const_t<std::remove_pointer_t<T>>;
    if constexpr (std::is_same_v<Pointee, tl_quant_desc> || std::is_same_v<Pointee, tl_epilogue>) {
      if (PyBytes_CheckExact(o) && PyBytes_GET_SIZE(o) == Py_ssize_t(sizeof(Pointee))) { *out = reinterpret_cast<T>(PyBytes_AS_STRING(o)); return true; }
    }
    return false;
  } else if constexpr (std::is_floating_point_v<T>) {
    if (!PyFloat_Check(o)) return false;
    *out = static_cast<T>(PyFloat_AS_DOUBLE(o));
    return true;
  } else {
    if (!PyLong_Check(o)) return false;
    *out = static_cast<T>(PyLong_AsUnsignedLongLongMask(o));
    return true;
  }
}

// The same for what has no slow path: any object that is an integer by __index__.
template <typename T> bool convert_index(PyObject* o, T* out) {
  if (convert(o, out)) return true;
  PyObject* i = PyNumber_Index(o);
  if (!i) { PyErr_Clear(); return false; }
  const bool ok = convert(i, out);
  Py_DECREF(i);
  return ok;
}

using Thunk = bool (*)(void* fn, PyObject* const* args, int32_t* status);  // false: an argument is not for here

template <typename F> struct Call;
template <typename... A> struct Call<int32_t(A...)> {
  static constexpr Py_ssize_t kArgs = sizeof...(A);
  template <size_t... I> static bool go(void* fn, PyObject* const* args, int32_t* status, std::index_sequence<I...>) {
    std::tuple<std::decay_t<A>...> v;
    if (!(convert(args[I], &std::get<I>(v)) && ...)) return false;
    Py_BEGIN_ALLOW_THREADS
    *status = reinterpret_cast<int32_t (*)(A...)>(fn)(std::get<I>(v)...);
    Py_END_ALLOW_THREADS
    return true;
  }
  static bool thunk(void* fn, PyObject* const* args, int32_t* status) { return go(fn, args, status, std::index_sequence_for<A...>{}); }
};

struct Entry { const char* name; Thunk thunk; Py_ssize_t args; };
#define TL_ENTRY(F) {#F, Call<decltype(F)>::thunk, Call<decltype(F)>::kArgs}
const Entry kEntries[] = {TL_ENTRY(tl_free),     TL_ENTRY(tl_copy2d),    TL_ENTRY(tl_quantize_linear_weight_device),
                          TL_ENTRY(tl_qmatmul_nt), TL_ENTRY(tl_matmul),  TL_ENTRY(tl_unary_op),
                          TL_ENTRY(tl_binary_op), TL_ENTRY(tl_rmsnorm),  TL_ENTRY(tl_rope),
                          TL_ENTRY(tl_attention), TL_ENTRY(tl_decode_attention)};

struct Bound {
  PyObject_HEAD
  vectorcallfunc vectorcall;
  Thunk thunk;  // null: tl_alloc
  Py_ssize_t args;
  void* fn;
  PyObject *slow, *on_error;
};

PyObject* fail(Bound* self, PyObject* ctx, int32_t status) {
  PyObject* r = PyObject_CallFunction(self->on_error, "Oi", ctx, int(status));
  if (!r) return nullptr;
  Py_DECREF(r);
  PyErr_Format(PyExc_RuntimeError, "tl status %d", int(status));
  return nullptr;
}
PyObject* bound_call(PyObject* callable, PyObject* const* args, size_t nargsf, PyObject* kwnames) {
  Bound* self = reinterpret_cast<Bound*>(callable);
  int32_t status = TL_OK;
  if (!kwnames && PyVectorcall_NARGS(nargsf) == self->args && self->thunk(self->fn, args, &status)) {
    if (status == TL_OK) Py_RETURN_NONE;
    return fail(self, args[0], status);
  }
  PyObject* r = PyObject_Vectorcall(self->slow, args, nargsf, kwnames);
  if (!r) return nullptr;
  const long slow_status = PyLong_AsLong(r);
  Py_DECREF(r);
  if (slow_status == -1 && PyErr_Occurred()) return nullptr;
  if (slow_status == TL_OK) Py_RETURN_NONE;
  return fail(self, args[0], int32_t(slow_status));
}
PyObject* alloc_call(PyObject* callable, PyObject* const* args, size_t nargsf, PyObject* kwnames) {
  Bound* self = reinterpret_cast<Bound*>(callable);
  tl_ctx* ctx;
  size_t bytes;
  if (kwnames || PyVectorcall_NARGS(nargsf) != 2 || !convert(args[0], &ctx) || !convert(args[1], &bytes))
    return PyObject_Vectorcall(self->slow, args, nargsf, kwnames);
  void* p = nullptr;
  int32_t status;
  Py_BEGIN_ALLOW_THREADS
  status = reinterpret_cast<decltype(&tl_alloc)>(self->fn)(ctx, bytes, &p);
  Py_END_ALLOW_THREADS
  if (status != TL_OK) return fail(self, args[0], status);
  if (!p) Py_RETURN_NONE;
  return PyLong_FromVoidPtr(p);
}
void bound_dealloc(PyObject* o) {
  Bound* self = reinterpret_cast<Bound*>(o);
  Py_XDECREF(self->slow);
  Py_XDECREF(self->on_error);
  Py_TYPE(o)->tp_free(o);
}
PyTypeObject BoundType = [] {
  PyTypeObject t = {PyVarObject_HEAD_INIT(nullptr, 0)};
  t.tp_name = "_tlcall.Bound";
  t.tp_basicsize = sizeof(Bound);
  t.tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_VECTORCALL;
  t.tp_vectorcall_offset = offsetof(Bound, vectorcall);
  t.tp_call = PyVectorcall_Call;
  t.tp_dealloc = bound_dealloc;
  return t;
}();

PyObject* make(vectorcallfunc call, Thunk thunk, Py_ssize_t args, unsigned long long address, PyObject* slow, PyObject* on_error) {
  Bound* b = PyObject_New(Bound, &BoundType);
  if (!b) return nullptr;
  b->vectorcall = call;
  b->thunk = thunk;
  b->args = args;
  b->fn = reinterpret_cast<void*>(static_cast<uintptr_t>(address));
  b->slow = Py_NewRef(slow);
  b->on_error = Py_NewRef(on_error);
  return reinterpret_cast<PyObject*>(b);
}
PyObject* py_bind(PyObject*, PyObject* args) {
  const char* name;
  unsigned long long address;
  PyObject *slow, *on_error;
  if (!PyArg_ParseTuple(args, "sKOO", &name, &address, &slow, &on_error)) return nullptr;
  if (!std::strcmp(name, "tl_alloc")) return make(alloc_call, nullptr, 2, address, slow, on_error);
  for (const Entry& e : kEntries)
    if (!std::strcmp(name, e.name)) return make(bound_call, e.thunk, e.args, address, slow, on_error);
  PyErr_Format(PyExc_KeyError, "%s", name);
  return nullptr;
}

// quant(scheme, group size, scales dtype, convention): a tl_quant_desc
PyObject* py_quant(PyObject*, PyObject* const* args, Py_ssize_t n) {
  tl_quant_desc q{};
  if (n != 4 || !convert_index(args[0], &q.scheme) || !convert_index(args[1], &q.group_size) || !convert_index(args[2], &q.scales_dtype) ||
      !convert_index(args[3], &q.scale_convention)) {
    PyErr_SetString(PyExc_TypeError, "quant: four integers");
    return nullptr;
  }
  return PyBytes_FromStringAndSize(reinterpret_cast<const char*>(&q), sizeof(q));
}
// epilogue(((kind, op, input index, to dtype), ...), (address, ...)): a tl_epilogue; the caller has checked the counts
PyObject* py_epilogue(PyObject*, PyObject* const* args, Py_ssize_t n) {
  tl_epilogue e{};
  bool ok = n == 2 && PyTuple_Check(args[0]) && PyTuple_Check(args[1]) && PyTuple_GET_SIZE(args[0]) <= TL_EPI_MAX_OPS &&
            PyTuple_GET_SIZE(args[1]) <= TL_EPI_MAX_INPUTS;
  if (ok) {
    e.n_ops = int32_t(PyTuple_GET_SIZE(args[0]));
    e.n_inputs = int32_t(PyTuple_GET_SIZE(args[1]));
    for (int i = 0; ok && i < e.n_ops; ++i) {
      PyObject* t = PyTuple_GET_ITEM(args[0], i);
      ok = PyTuple_Check(t) && PyTuple_GET_SIZE(t) == 4 && convert_index(PyTuple_GET_ITEM(t, 0), &e.ops[i].kind) &&
           convert_index(PyTuple_GET_ITEM(t, 1), &e.ops[i].op) && convert_index(PyTuple_GET_ITEM(t, 2), &e.ops[i].input_index) &&
           convert_index(PyTuple_GET_ITEM(t, 3), &e.ops[i].to_dtype);
    }
    for (int i = 0; ok && i < e.n_inputs; ++i) ok = convert_index(PyTuple_GET_ITEM(args[1], i), &e.inputs[i]);
  }
  if (!ok) {
    PyErr_SetString(PyExc_TypeError, "epilogue: tuples of integers");
    return nullptr;
  }
  return PyBytes_FromStringAndSize(reinterpret_cast<const char*>(&e), sizeof(e));
}

PyMethodDef kMethods[] = {{"bind", py_bind, METH_VARARGS, nullptr},
                          {"quant", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(py_quant)), METH_FASTCALL, nullptr},
                          {"epilogue", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(py_epilogue)), METH_FASTCALL, nullptr},
                          {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_tlcall", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__tlcall(void) {
  if (PyType_Ready(&BoundType) < 0) return nullptr;
  PyObject* m = PyModule_Create(&kModule);
  if (m) {
    PyObject* names = PyTuple_New(Py_ssize_t(std::size(kEntries)) + 1);
    if (!names) return nullptr;
    PyTuple_SET_ITEM(names, 0, PyUnicode_FromString("tl_alloc"));
    for (size_t i = 0; i < std::size(kEntries); ++i) PyTuple_SET_ITEM(names, Py_ssize_t(i) + 1, PyUnicode_FromString(kEntries[i].name));
    PyModule_AddObject(m, "names", names);
  }
  return m;
}
