// The per-layer entry points of libjllama_b200.so as built-in Python functions.
//
// A step of a small layer is a handful of launches of a few microseconds, and the host issues them: through ctypes a call of 18 arguments costs 1.7 us before the
// library's first instruction, through these wrappers a fraction of that.  A wrapper is generated from the entry point's own declaration: it converts whole
// numbers, floats and None as the declared types say, lets other Python threads run during the call, and hands anything else it is given (ctypes arrays,
// numbers out of range, a wrong count) to the ctypes function it stands for, which then answers as always.
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <dlfcn.h>
#include <limits.h>

#include <string>
#include <tuple>
#include <type_traits>
#include <utility>

#include "jllama_b200.h"

namespace {

template <typename T>
bool convert(PyObject* o, T* out) {
  if constexpr (std::is_pointer_v<T>) {
    if (o == Py_None) { *out = nullptr; return true; }
    if (!PyLong_Check(o)) return false;
    void* p = PyLong_AsVoidPtr(o);
    if (p == nullptr && PyErr_Occurred()) return false;
    *out = (T)p;
    return true;
  } else if constexpr (std::is_floating_point_v<T>) {
    if (PyFloat_Check(o)) { *out = (T)PyFloat_AS_DOUBLE(o); return true; }
    if (!PyLong_Check(o)) return false;
    const double v = PyLong_AsDouble(o);
    if (v == -1.0 && PyErr_Occurred()) return false;
    *out = (T)v;
    return true;
  } else if constexpr (std::is_signed_v<T>) {
    if (!PyLong_Check(o)) return false;
    int over = 0;
    const long long v = PyLong_AsLongLongAndOverflow(o, &over);
    if (over != 0 || (v == -1 && PyErr_Occurred()) || v != (long long)(T)v) return false;
    *out = (T)v;
    return true;
  } else {
    if (!PyLong_Check(o)) return false;
    const unsigned long long v = PyLong_AsUnsignedLongLong(o);
    if ((v == (unsigned long long)-1 && PyErr_Occurred()) || v != (unsigned long long)(T)v) return false;
    *out = (T)v;
    return true;
  }
}

template <typename R>
PyObject* to_python(R r) {
  if constexpr (std::is_signed_v<R>) return PyLong_FromLongLong(r);
  else return PyLong_FromUnsignedLongLong(r);
}

template <typename F>
struct Entry;
template <typename R, typename... A>
struct Entry<R (*)(A...)> {
  template <std::size_t... I>
  static bool all(PyObject* const* a, std::tuple<A...>& v, std::index_sequence<I...>) { return (convert(a[I], &std::get<I>(v)) && ...); }

  // self: the ctypes function of the same name
  template <R (**fn)(A...)>
  static PyObject* call(PyObject* self, PyObject* const* a, Py_ssize_t n) {
    std::tuple<A...> v{};
    if (n != (Py_ssize_t)sizeof...(A) || !all(a, v, std::index_sequence_for<A...>())) {
      PyErr_Clear();
      return PyObject_Vectorcall(self, a, (size_t)n, nullptr);
    }
    R r;
    Py_BEGIN_ALLOW_THREADS
    r = std::apply(*fn, v);
    Py_END_ALLOW_THREADS
    return to_python(r);
  }
};

#define JL_ENTRIES(X)                                                                                                                    \
  X(jl_rmsnorm) X(jl_rope_kv_write) X(jl_gemv) X(jl_gemm) X(jl_gemm_2cta) X(jl_decode_attn) X(jl_decode_attn_fused) X(jl_flash_prefill)  \
  X(jl_prefill_attn_mma) X(jl_sample_full) X(jl_swiglu) X(jl_argmax)                                                                     \
  X(jl_embed_f32) X(jl_norm_f32) X(jl_postnorm_add) X(jl_headnorm_gate) X(jl_act_cast) X(jl_act_inplace) X(jl_linear_any)                \
  X(jl_linear_resident) X(jl_linear_exact) X(jl_linear_f32_pair_ws) X(jl_linear_f32_pair) X(jl_attn_prep) X(jl_attn_prep_ex)             \
  X(jl_attn_step) X(jl_attn_generic) X(jl_attn_generic_splits) X(jl_head_gate) X(jl_gla_scan) X(jl_gla_scan_exact) X(jl_gla_step)           \
  X(jl_gla_scan_ws_floats) X(jl_retention_scan) X(jl_branch_add_norm) X(jl_moe_route) X(jl_moe_route_ex) X(jl_moe_sort)                      \
  X(jl_moe_sorted_rows) X(jl_moe_gather) X(jl_moe_combine) X(jl_moe_combine_ex) X(jl_gemm_grouped) X(jl_gemm_grouped_act) X(jl_gemm_glu) \
  X(jl_glu_act) X(jl_linear_grouped) X(jl_latent_prep) X(jl_latent_heads) X(jl_rotary_slice) X(jl_attn_masked) X(jl_attn_windowed)       \
  X(jl_flash_prefill_masked) X(jl_causal_conv) X(jl_ssd_gates) X(jl_ssd_scan) X(jl_gated_groupnorm) X(jl_delta_scan)                     \
  X(jl_delta_scan_ws_floats) X(jl_delta_head_scan) X(jl_delta_head_scan_ws_floats) X(jl_weighted_sum2) X(jl_rownorm_gate)                \
  X(jl_postnorm_cast) X(jl_branch_add_cast) X(jl_attn_prep_all) X(jl_activated_scan) X(jl_mlstm_gates) X(jl_mlstm_scan)                  \
  X(jl_mlstm_finish)

#define JL_SLOT(name) decltype(&name) slot_##name = nullptr;
JL_ENTRIES(JL_SLOT)

struct Row {
  const char* name;
  void** slot;
  PyMethodDef def;
};
#define JL_ROW(name)                 \
  Row{#name, (void**)&slot_##name,   \
      {#name, (PyCFunction)(void (*)(void)) & Entry<decltype(&name)>::template call<&slot_##name>, METH_FASTCALL, nullptr}},
Row rows[] = {JL_ENTRIES(JL_ROW)};

// bind(handle of the library as dlopen gave it, {name: ctypes function}) -> {name: built-in function} for the entry points that both know
PyObject* bind(PyObject*, PyObject* args) {
  unsigned long long handle = 0;
  PyObject* fallback = nullptr;
  if (!PyArg_ParseTuple(args, "KO!", &handle, &PyDict_Type, &fallback)) return nullptr;
  PyObject* out = PyDict_New();
  if (out == nullptr) return nullptr;
  for (Row& r : rows) {
    PyObject* slow = PyDict_GetItemString(fallback, r.name);               // borrowed
    void* fn = slow != nullptr ? dlsym((void*)handle, r.name) : nullptr;
    if (fn == nullptr) continue;
    *r.slot = fn;
    PyObject* f = PyCFunction_New(&r.def, slow);
    if (f == nullptr || PyDict_SetItemString(out, r.name, f) != 0) {
      Py_XDECREF(f);
      Py_DECREF(out);
      return nullptr;
    }
    Py_DECREF(f);
  }
  return out;
}

PyMethodDef methods[] = {{"bind", bind, METH_VARARGS, "bind(handle, {name: ctypes function}) -> {name: built-in function}"}, {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_jl_binding", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__jl_binding(void) { return PyModule_Create(&module); }
