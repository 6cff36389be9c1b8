// CPython entry points for the single-GPU kernels (nkb_api.h): the same functions that
// _lib.py reaches through ctypes, as positional C calls.
//
// Small models are bound by the host: through ctypes a GEMM call with its 28 arguments is
// converted argument by argument by generic code (6.7 us with the launch).  Here the conversions are
// compiled from the C signature (4.4 us).  None is a null pointer, a pointer is an integer.  The interpreter lock is
// released around the call as ctypes does (a launch waits while the device's queue is full).
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <tuple>
#include <utility>

#include "nkb_api.h"

namespace {

template <typename T>
struct Arg;
template <typename T>
struct Arg<T*> {
  static bool get(PyObject* o, T*& v) {
    if (o == Py_None) {
      v = nullptr;
      return true;
    }
    void* p = PyLong_AsVoidPtr(o);
    if (!p && PyErr_Occurred()) return false;
    v = static_cast<T*>(p);
    return true;
  }
};
template <>
struct Arg<long long> {
  static bool get(PyObject* o, long long& v) {
    v = PyLong_AsLongLong(o);
    return v != -1 || !PyErr_Occurred();
  }
};
template <>
struct Arg<int> {
  static bool get(PyObject* o, int& v) {
    const long long x = PyLong_AsLongLong(o);
    if (x == -1 && PyErr_Occurred()) return false;
    v = static_cast<int>(x);
    if (v != x) {
      PyErr_SetString(PyExc_OverflowError, "argument does not fit a C int");
      return false;
    }
    return true;
  }
};
template <>
struct Arg<float> {
  static bool get(PyObject* o, float& v) {
    const double x = PyFloat_AsDouble(o);
    if (x == -1.0 && PyErr_Occurred()) return false;
    v = static_cast<float>(x);
    return true;
  }
};

template <auto F>
struct Call;
template <typename... A, int (*F)(A...)>
struct Call<F> {
  template <size_t... I>
  static PyObject* run(PyObject* const* args, std::index_sequence<I...>) {
    std::tuple<A...> v;
    if (!(Arg<A>::get(args[I], std::get<I>(v)) && ...)) return nullptr;
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = F(std::get<I>(v)...);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(rc);
  }
  static PyObject* py(PyObject*, PyObject* const* args, Py_ssize_t n) {
    if (n != (Py_ssize_t)sizeof...(A))
      return PyErr_Format(PyExc_TypeError, "%zd arguments, %zd wanted", n,
                          (Py_ssize_t)sizeof...(A));
    return run(args, std::index_sequence_for<A...>{});
  }
};

#define ENTRY(name)                                                                         \
  {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&Call<&name>::py)), \
   METH_FASTCALL, nullptr}

PyMethodDef methods[] = {
    ENTRY(nkb_gemm_bf16),        ENTRY(nkb_norm_fwd),         ENTRY(nkb_norm_bwd_all),
    ENTRY(nkb_norm_bwd_dx),      ENTRY(nkb_norm_bwd_dx_res),  ENTRY(nkb_colsum),
    ENTRY(nkb_colsum_fused),     ENTRY(nkb_f32_to_bf16),      ENTRY(nkb_ce_fwd_bwd),
    ENTRY(nkb_ce_stats),         ENTRY(nkb_ce_grad),          ENTRY(nkb_loss_mean),
    ENTRY(nkb_loss_corr),        ENTRY(nkb_embed_fwd),        ENTRY(nkb_embed_bwd),
    ENTRY(nkb_adam_flat),        ENTRY(nkb_hyper_advance),    ENTRY(nkb_sgd_flat),
    ENTRY(nkb_clip_coef),        ENTRY(nkb_quant2_flat),      ENTRY(nkb_dequant2_flat),
    ENTRY(nkb_quant2_matrix),    ENTRY(nkb_dequant2_matrix),  ENTRY(nkb_scale_cast),
    ENTRY(nkb_sumsq),            ENTRY(nkb_attn_fwd),         ENTRY(nkb_attn_bwd),
    ENTRY(nkb_rope),             ENTRY(nkb_swiglu_fwd),       ENTRY(nkb_swiglu_bwd),
    ENTRY(nkb_im2col_nhwc),      ENTRY(nkb_col2im_nhwc),      ENTRY(nkb_conv_fwd),
    ENTRY(nkb_conv_dgrad),       ENTRY(nkb_conv_wgrad_split), ENTRY(nkb_conv_wgrad),
    ENTRY(nkb_bn_fwd),           ENTRY(nkb_bn_apply),         ENTRY(nkb_bn_bwd),
    ENTRY(nkb_bn_eval),          ENTRY(nkb_maxpool3x3s2_fwd), ENTRY(nkb_maxpool3x3s2_bwd),
    ENTRY(nkb_avgpool_fwd),      ENTRY(nkb_avgpool_bwd),      ENTRY(nkb_gemm_slices),
    ENTRY(nkb_gemm_bf16_ws),     ENTRY(nkb_capture_id),       ENTRY(nkb_conv_route),
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_nkpy", nullptr, -1, methods,
                      nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__nkpy() { return PyModule_Create(&module); }
