// The kernel library's entry points as a Python module (`pfeife_b200_calls`).
//
// A launch costs the host some 4 us; going through ctypes added 4 to 6 for the objects that carry 20
// to 30 arguments and their conversion.  Here the signatures of api.h become argument parsers at
// compile time: integers and floats as they are, pointers as None, an address or a tensor (whose
// data_ptr() is asked for), and `const long long*` also as a tuple of up to eight integers.  The
// interpreter lock is released around the call, which may wait for room in the launch queue.
// Host time of a GEMM with a bias, its output's allocation included: 13.2 us through ctypes, 9.5 so;
// attention on a fused projection 28.8 and 23.5; ViT-Tiny logits of 4 images 3.02 and 2.49 ms.
//
// The library itself is loaded by the caller beforehand with its symbols global.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <type_traits>
#include <tuple>
#include <utility>

#include "api.h"

namespace {

constexpr int MAX_TUPLE = 8;
PyObject* s_data_ptr = nullptr;

// One converted argument; tuples live here until the call has returned.
template <typename T>
struct Arg {
  T value{};
  long long items[std::is_same_v<T, const long long*> ? MAX_TUPLE : 1];

  bool from(PyObject* o) {
    if constexpr (std::is_floating_point_v<T>) {
      value = static_cast<T>(PyFloat_AsDouble(o));
      return !PyErr_Occurred();
    } else if constexpr (std::is_integral_v<T>) {
      const long long v = PyLong_AsLongLong(o);
      if (v == -1 && PyErr_Occurred()) return false;
      if (static_cast<long long>(static_cast<T>(v)) != v) {
        PyErr_SetString(PyExc_OverflowError, "argument does not fit its C type");
        return false;
      }
      value = static_cast<T>(v);
      return true;
    } else {
      if (o == Py_None) return true;
      if (PyLong_Check(o)) {
        value = reinterpret_cast<T>(PyLong_AsUnsignedLongLong(o));
        return !PyErr_Occurred();
      }
      if constexpr (std::is_same_v<T, const long long*>) {
        if (PyTuple_Check(o)) {
          const Py_ssize_t n = PyTuple_GET_SIZE(o);
          if (n > MAX_TUPLE) {
            PyErr_SetString(PyExc_ValueError, "tuple argument too long");
            return false;
          }
          for (Py_ssize_t i = 0; i < n; ++i) {
            items[i] = PyLong_AsLongLong(PyTuple_GET_ITEM(o, i));
            if (items[i] == -1 && PyErr_Occurred()) return false;
          }
          value = items;
          return true;
        }
      }
      PyObject* p = PyObject_CallMethodNoArgs(o, s_data_ptr);
      if (!p) return false;
      value = reinterpret_cast<T>(PyLong_AsUnsignedLongLong(p));
      Py_DECREF(p);
      return !PyErr_Occurred();
    }
  }
};

template <auto F> struct Call;
template <typename... A, int (*F)(A...)>
struct Call<F> {
  template <size_t... I>
  static PyObject* run(PyObject* const* args, std::index_sequence<I...>) {
    std::tuple<Arg<A>...> a;
    if (!(std::get<I>(a).from(args[I]) && ...)) return nullptr;
    int r;
    Py_BEGIN_ALLOW_THREADS
    r = F(std::get<I>(a).value...);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(r);
  }
  static PyObject* fast(PyObject*, PyObject* const* args, Py_ssize_t n) {
    if (n != static_cast<Py_ssize_t>(sizeof...(A)))
      return PyErr_Format(PyExc_TypeError, "expected %zu arguments, got %zd", sizeof...(A), n);
    return run(args, std::index_sequence_for<A...>());
  }
};

#define PF_CALL(name) \
  {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&Call<&name>::fast)), \
   METH_FASTCALL, nullptr}

PyMethodDef methods[] = {
    PF_CALL(pf_bind_device), PF_CALL(pf_gemm), PF_CALL(pf_gemm_workspace), PF_CALL(pf_elementwise), PF_CALL(pf_glu_fwd),
    PF_CALL(pf_glu_bwd),
    PF_CALL(pf_axpy_f32), PF_CALL(pf_cast), PF_CALL(pf_colsum), PF_CALL(pf_transpose16),
    PF_CALL(pf_norm_fwd), PF_CALL(pf_norm_bwd_ctas), PF_CALL(pf_norm_bwd), PF_CALL(pf_nonfinite),
    PF_CALL(pf_adamw), PF_CALL(pf_step_advance), PF_CALL(pf_sgd), PF_CALL(pf_loss_scale_update),
    PF_CALL(pf_ce_fwd), PF_CALL(pf_ce_mean_parts), PF_CALL(pf_ce_mean), PF_CALL(pf_ce_bwd),
    PF_CALL(pf_mse_fwd), PF_CALL(pf_mse_bwd), PF_CALL(pf_embed_fwd), PF_CALL(pf_embed_bwd),
    PF_CALL(pf_rope), PF_CALL(pf_rope_qkv), PF_CALL(pf_attn_fwd),
    PF_CALL(pf_attn_bwd_scratch), PF_CALL(pf_attn_bwd), PF_CALL(pf_im2col), PF_CALL(pf_col2im), PF_CALL(pf_groupnorm_slabs),
    PF_CALL(pf_groupnorm_fwd), PF_CALL(pf_groupnorm_bwd), PF_CALL(pf_upsample2x),
    PF_CALL(pf_conv_gemm), PF_CALL(pf_conv_wgrad), PF_CALL(pf_conv_pack), PF_CALL(pf_conv_unpack),
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "pfeife_b200_calls",
                      "entry points of the kernel library", -1, methods,
                      nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_pfeife_b200_calls() {
  if (!s_data_ptr && !(s_data_ptr = PyUnicode_InternFromString("data_ptr"))) return nullptr;
  return PyModule_Create(&module);
}
