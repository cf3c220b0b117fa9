// The calls of libspd.so as Python functions without ctypes.  A call of 16 arguments costs ctypes 2.2 us and these 0.2,
// and where few tokens make every kernel short, a step's time is its host time: an expert layer of 2 tokens 98.6 -> 88.3 us,
// the extend of 10 tokens through two Llama layers 328 -> 293, decode attention for 4 requests of 100 keys 16.5 -> 14.2.
// What goes in is what the header declares, as plain ints (addresses: ints or None) and floats; anything else that
// ctypes would take (byref, arrays, numpy's integers) or refuse goes to the ctypes function of the same name, so that
// what is taken and what is refused stays as it was.  The C function runs without the interpreter's lock, as there.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <type_traits>

#include "../../include/spd.h"

namespace {

// the value of one argument; false: not a plain one, or out of range (a Python error may be set)
template <typename T>
bool take(PyObject* o, T* out) {
  if constexpr (std::is_pointer_v<T>) {
    if (o == Py_None) {
      *out = nullptr;
      return true;
    }
    if (!PyLong_CheckExact(o)) return false;
    *out = static_cast<T>(PyLong_AsVoidPtr(o));
    return *out || !PyErr_Occurred();
  } else if constexpr (std::is_same_v<T, float>) {
    if (!PyFloat_CheckExact(o)) return false;
    *out = static_cast<float>(PyFloat_AS_DOUBLE(o));
    return true;
  } else {
    if (!PyLong_Check(o)) return false;  // a bool too
    *out = static_cast<T>(PyLong_AsUnsignedLongLongMask(o));  // cut to the parameter's width, as ctypes does
    return true;
  }
}

template <typename... A>
struct Args;
template <>
struct Args<> {
  bool load(PyObject* const*) { return true; }
  template <typename F, typename... V>
  int call(F f, V... v) { return f(v...); }
};
template <typename T, typename... A>
struct Args<T, A...> {
  T value;
  Args<A...> rest;
  bool load(PyObject* const* o) { return take(*o, &value) && rest.load(o + 1); }
  template <typename F, typename... V>
  int call(F f, V... v) { return rest.call(f, v..., value); }
};

template <typename F>
struct Call;
template <typename... A>
struct Call<int(A...)> {
  // self: (capsule of the C function, the ctypes function)
  static PyObject* run(PyObject* self, PyObject* const* args, Py_ssize_t n) {
    Args<A...> a;
    if (n != static_cast<Py_ssize_t>(sizeof...(A)) || !a.load(args)) {
      PyErr_Clear();
      return PyObject_Vectorcall(PyTuple_GET_ITEM(self, 1), args, n, nullptr);
    }
    auto f = reinterpret_cast<int (*)(A...)>(PyCapsule_GetPointer(PyTuple_GET_ITEM(self, 0), nullptr));
    int rc;
    Py_BEGIN_ALLOW_THREADS rc = a.call(f);
    Py_END_ALLOW_THREADS return PyLong_FromLong(rc);
  }
};

#define SPD_CALLS \
  X(spd_wait_selftest) X(spd_rmsnorm) X(spd_fused_add_rmsnorm) X(spd_silu_and_mul) X(spd_rope_inplace) X(spd_rope_kvwrite) \
  X(spd_rope_inplace_sms) X(spd_rope_kvwrite_sms) \
  X(spd_kv_write) X(spd_gather_rows) X(spd_argmax_f32) X(spd_argmax_partial_f32) X(spd_argmax_merge) \
  X(spd_compute_positions) X(spd_decode_positions) X(spd_build_kv_indices) X(spd_write_req_to_token) X(spd_layernorm) \
  X(spd_bias_act_residual) X(spd_gemm) X(spd_attn_prefill_ragged) X(spd_attn_decode_paged) X(spd_attn_decode_paged_own) \
  X(spd_attn_prefill_simt) X(spd_attn_decode_simt) X(spd_gemm_grouped) X(spd_gemm_grouped_rows) X(spd_moe_route) \
  X(spd_moe_align) X(spd_moe_align_groups) X(spd_moe_gather) X(spd_moe_combine) X(spd_moe_dense_act) \
  X(spd_mla_rotary_store) X(spd_mla_rotary_store_inplace) X(spd_mla_gather) X(spd_attn_mla_prefill) X(spd_attn_mla) \
  X(spd_attn_mla_own) X(spd_residual_rmsnorm) X(spd_embed_f32) X(spd_act_and_mul) X(spd_headnorm_gate) X(spd_linear_simt) \
  X(spd_moe_route_scores) X(spd_moe_gather_scaled) X(spd_moe_combine_gated) X(spd_kv_store) X(spd_attn_general) \
  X(spd_retention) X(spd_retention_extend) X(spd_retention_extend_ws) X(spd_retention_extend_tiles) \
  X(spd_residual_rmsnorm2) X(spd_linear_simt_block_diag) X(spd_gated_recurrence) X(spd_token_shift_mix) X(spd_embed_sincos) \
  X(spd_cast_concat) X(spd_activation) X(spd_rmsnorm_store) X(spd_head_gate_sigmoid) X(spd_scale_f32) \
  X(spd_embed_norm_streams) X(spd_streams_mix_norm) X(spd_rotary_bias_store) X(spd_matrix_memory) X(spd_attn_general_ex) \
  X(spd_embed_pair) X(spd_residual_tanh_norm) X(spd_heads_gate) X(spd_residual_postnorm) X(spd_softcap_f32) \
  X(spd_attn_general_blocks) X(spd_attn_general_keys) X(spd_attn_general_sms) X(spd_pool_key_blocks) X(spd_head_decay) \
  X(spd_short_conv) X(spd_gated_group_norm)

PyMethodDef calls[] = {
#define X(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(&Call<decltype(name)>::run)), METH_FASTCALL, nullptr},
    SPD_CALLS
#undef X
    {nullptr, nullptr, 0, nullptr}};

// bind({name: (address, ctypes function)}) -> {name: function} for the names that are here
PyObject* bind(PyObject*, PyObject* functions) {
  if (!PyDict_Check(functions)) return PyErr_Format(PyExc_TypeError, "bind takes a dict");
  PyObject* out = PyDict_New();
  for (PyMethodDef* m = calls; out && m->ml_name; ++m) {
    PyObject* pair = PyDict_GetItemString(functions, m->ml_name);  // borrowed
    if (!pair) continue;
    PyObject *address, *slow;
    PyObject *capsule = nullptr, *self = nullptr, *f = nullptr;
    if (PyArg_ParseTuple(pair, "OO", &address, &slow)) {
      void* p = PyLong_AsVoidPtr(address);
      if (!PyErr_Occurred()) capsule = PyCapsule_New(p, nullptr, nullptr);  // an error for a null address
    }
    if (capsule) self = PyTuple_Pack(2, capsule, slow);
    if (self) f = PyCFunction_New(m, self);
    if (!f || PyDict_SetItemString(out, m->ml_name, f) < 0) Py_CLEAR(out);
    Py_XDECREF(f);
    Py_XDECREF(self);
    Py_XDECREF(capsule);
  }
  return out;
}

PyMethodDef methods[] = {{"bind", bind, METH_O, nullptr}, {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_calls", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__calls() { return PyModule_Create(&module); }
