// Operators on tensors: what ops/*.py does around a kernel call, compiled.
//
// A forward or backward operator of a small model costs the host more than the device: reading
// shapes, strides and addresses of its tensors one attribute at a time, a handful of checks, views to
// two dimensions and back, an allocation per output and a call with up to 30 arguments are 8 to 15 us
// of Python for a kernel of 5 us.  Each function here does that for the form that models use (bf16,
// contiguous, 16-byte aligned) and gives None for any other, which the caller then takes the general
// way; it holds no state.  A native error code comes back as an int.
//
// Optional like _nkpy (pycall.cpp): without it every operator takes the general way.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/version.h>

#include <climits>
#include <cmath>

#include "nkb_api.h"

namespace {

using at::Tensor;

struct Args {
  PyObject* const* v;
  const Tensor* tensor(int i) const {  // null for None
    return v[i] == Py_None ? nullptr : &THPVariable_Unpack(v[i]);
  }
  bool tensors(std::initializer_list<int> at) const {  // these arguments are tensors or None
    for (int i : at)
      if (v[i] != Py_None && !THPVariable_Check(v[i])) return false;
    return true;
  }
  long long num(int i) const { return PyLong_AsLongLong(v[i]); }
  double real(int i) const { return PyFloat_AsDouble(v[i]); }
  bool flag(int i) const { return PyObject_IsTrue(v[i]) == 1; }
  int* status(int i) const { return static_cast<int*>(PyLong_AsVoidPtr(v[i])); }
};

inline uintptr_t address(const Tensor& t) { return reinterpret_cast<uintptr_t>(t.data_ptr()); }
inline void* ptr(const Tensor* t) { return t ? t->data_ptr() : nullptr; }
// what the functions take: values of 16 bits in rows without gaps
inline bool plain(const Tensor& t) {
  return t.is_cuda() && t.scalar_type() == at::kBFloat16 && t.is_contiguous() && t.dim() > 0 &&
         t.numel() > 0 && !(address(t) & 15);
}
inline bool plain_or_none(const Tensor* t) { return !t || plain(*t); }
inline bool vec_or_none(const Tensor* t, long long n) {  // a bias: any alignment
  return !t || (t->is_cuda() && t->scalar_type() == at::kBFloat16 && t->is_contiguous() &&
                t->numel() == n);
}
inline long long rows_of(const Tensor& t) { return t.numel() / t.size(-1); }
inline bool fits(long long a) { return a > 0 && a <= INT_MAX; }
inline void* stream() { return c10::cuda::getCurrentCUDAStream().stream(); }
inline at::TensorOptions of(const Tensor& like, at::ScalarType type) {
  return at::TensorOptions().dtype(type).device(like.device());
}
inline Tensor empty_with_cols(const Tensor& x, long long cols) {
  auto s = x.sizes().vec();
  s.back() = cols;
  return at::empty(s, of(x, at::kBFloat16));
}

PyObject* none() {
  PyErr_Clear();  // an argument of another kind
  Py_RETURN_NONE;
}
PyObject* code(int rc) { return PyLong_FromLong(rc); }
PyObject* wrap(Tensor t) { return THPVariable_Wrap(std::move(t)); }
template <typename... T>
PyObject* tuple(T... t) {
  PyObject* r = PyTuple_New(sizeof...(T));
  if (!r) return nullptr;
  int i = 0;
  bool ok = true;
  auto put = [&](Tensor x) {
    PyObject* o = ok ? wrap(std::move(x)) : nullptr;
    ok = ok && o;
    if (o) PyTuple_SET_ITEM(r, i++, o);
  };
  (put(std::move(t)), ...);
  if (!ok) {
    Py_DECREF(r);
    return nullptr;
  }
  return r;
}

// A launch waits while the device's queue is full: other threads may run meanwhile.
template <typename F>
int launch(F f) {
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = f();
  Py_END_ALLOW_THREADS
  return rc;
}

// One GEMM; K is split like in ops/gemm.py.
struct Gemm {
  const void *a = nullptr, *b = nullptr;
  long long lda = 0, ldb = 0;
  int a_mn = 0, b_mn = 0;
  void* c = nullptr;
  long long ldc = 0;
  int fp32 = 0, accumulate = 0;
  long long M = 0, N = 0, K = 0;
  float alpha = 1.f;
  const void *bias = nullptr, *res = nullptr;
  long long ldres = 0;
  int epi = NKB_EPI_NONE;
  void* aux = nullptr;
  long long ldaux = 0;
  int bn = 0;
  const float* alpha_dev = nullptr;

  bool ok() const {
    return fits(M) && fits(N) && fits(K) && !(lda & 7) && !(ldb & 7) &&
           !((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b)) & 15);
  }
  int run(const Tensor& like, int* status) const {
    int slices = 1;
    Tensor ws;  // the call's own: the allocator orders its reuse on the stream
    auto at = [](const void* p) { return reinterpret_cast<uintptr_t>(p); };
    if (K >= 2048 && epi == NKB_EPI_NONE && !(at(c) & (fp32 ? 15 : 7)) &&
        !((at(bias) | at(res)) & 7) && !(ldres & 3)) {
      slices = nkb_gemm_slices((int)M, (int)N, (int)K, ldc, bn);
      if (slices > 1) ws = at::empty({slices * M * N}, of(like, at::kFloat));
    }
    void* s = stream();
    float* w = slices > 1 ? ws.data_ptr<float>() : nullptr;
    return launch([&] {
      return nkb_gemm_bf16_ws(a, lda, a_mn, b, ldb, b_mn, c, ldc, fp32, accumulate, (int)M, (int)N,
                              (int)K, alpha, bias, res, ldres, epi, aux, ldaux, status, nullptr, 0,
                              0, 0, bn, alpha_dev, w, slices, s);
    });
  }
};

// y [M, N] = x [M, K] w [N, K]^T
Gemm fwd(const Tensor& x, const Tensor& w, const Tensor& y) {
  Gemm g;
  g.K = x.size(-1); g.M = rows_of(x); g.N = w.size(0);
  g.a = x.data_ptr(); g.lda = g.K; g.b = w.data_ptr(); g.ldb = g.K;
  g.c = y.data_ptr(); g.ldc = g.N;
  return g;
}
// dx [M, K] = dy [M, N] w [N, K]
Gemm dgrad(const Tensor& dy, const Tensor& w, const Tensor& dx) {
  Gemm g;
  g.M = rows_of(dy); g.K = w.size(0); g.N = w.size(1);
  g.a = dy.data_ptr(); g.lda = g.K; g.b = w.data_ptr(); g.ldb = g.N; g.b_mn = 1;
  g.c = dx.data_ptr(); g.ldc = g.N;
  return g;
}
// dw [N, K] (+)= dy [M, N]^T x [M, K]
Gemm wgrad(const Tensor& dy, const Tensor& x, const Tensor& dw, bool accumulate) {
  Gemm g;
  g.M = dy.size(-1); g.N = x.size(-1); g.K = rows_of(dy);
  g.a = dy.data_ptr(); g.lda = g.M; g.a_mn = 1; g.b = x.data_ptr(); g.ldb = g.N; g.b_mn = 1;
  g.c = dw.data_ptr(); g.ldc = g.N; g.accumulate = accumulate;
  return g;
}
// where a gradient goes: bf16, the weight's shape
bool target(const Tensor* t, const Tensor& like) {
  return !t || (t->is_cuda() && t->scalar_type() == at::kBFloat16 && t->is_contiguous() &&
                t->sizes() == like.sizes());
}
bool bias_target(const Tensor* t, long long n) { return vec_or_none(t, n) && !(n & 1); }

// The columns' fp32 accumulator and ticket counters (ops.gemm.colsum_scratch), arguments i and i + 1
struct Scratch {
  float* acc = nullptr;
  int* tickets = nullptr;
  Scratch(const Args& a, int i) {
    if (const Tensor* t = a.tensor(i)) {
      acc = t->data_ptr<float>();
      tickets = a.tensor(i + 1)->data_ptr<int>();
    }
  }
};

int colsum(const Tensor& dy, const Tensor& out, bool accumulate, const Scratch& sc) {
  const int rows = (int)rows_of(dy), C = (int)dy.size(-1);
  void* s = stream();
  return launch([&] {
    return nkb_colsum_fused(dy.data_ptr(), sc.acc, sc.tickets, out.data_ptr(), accumulate, rows, C,
                            C, s);
  });
}

#define NK_FUNCTION(name, count)                                                          \
  PyObject* name(const Args& a);                                                          \
  PyObject* name##_py(PyObject*, PyObject* const* v, Py_ssize_t n) {                      \
    HANDLE_TH_ERRORS                                                                      \
    if (n != count)                                                                       \
      return PyErr_Format(PyExc_TypeError, #name ": %zd arguments, %d wanted", n, count); \
    return name(Args{v});                                                                 \
    END_HANDLE_TH_ERRORS                                                                  \
  }                                                                                       \
  PyObject* name(const Args& a)

// gemm(a, b, a_mn, b_mn, out, fp32, accumulate, alpha, bias, res, epi, aux, bn, alpha_dev, status)
// -> out.  Operands may have rows apart; see ops.gemm.gemm.
NK_FUNCTION(gemm, 15) {
  if (!a.tensors({0, 1, 4, 8, 9, 11, 13})) return none();
  const Tensor *A = a.tensor(0), *B = a.tensor(1), *out = a.tensor(4), *bias = a.tensor(8),
               *res = a.tensor(9), *aux = a.tensor(11), *alpha_dev = a.tensor(13);
  auto matrix = [](const Tensor& t) {
    return t.is_cuda() && t.scalar_type() == at::kBFloat16 && t.dim() == 2 && t.stride(1) == 1;
  };
  if (!A || !B || !matrix(*A) || !matrix(*B)) return none();
  Gemm g;
  g.a_mn = a.flag(2); g.b_mn = a.flag(3);
  g.M = A->size(g.a_mn ? 1 : 0); g.K = A->size(g.a_mn ? 0 : 1); g.N = B->size(g.b_mn ? 1 : 0);
  if (B->size(g.b_mn ? 0 : 1) != g.K) return none();
  g.fp32 = a.flag(5); g.accumulate = a.flag(6); g.alpha = (float)a.real(7);
  g.epi = (int)a.num(10); g.bn = (int)a.num(12);
  if (PyErr_Occurred()) return none();
  g.a = A->data_ptr(); g.lda = A->stride(0); g.b = B->data_ptr(); g.ldb = B->stride(0);
  if (!g.ok() || !vec_or_none(bias, g.N)) return none();
  auto like_out = [&](const Tensor* t) {
    return !t || (matrix(*t) && t->size(0) == g.M && t->size(1) == g.N);
  };
  const bool gelu = g.epi == NKB_EPI_GELU_FWD || g.epi == NKB_EPI_GELU_BWD;
  if (!like_out(res) || (gelu ? !aux || !like_out(aux) : aux != nullptr)) return none();
  if (alpha_dev && (!alpha_dev->is_cuda() || alpha_dev->scalar_type() != at::kFloat)) return none();
  Tensor y;
  if (out) {
    g.fp32 = out->scalar_type() == at::kFloat;
    if (!out->is_cuda() || (!g.fp32 && out->scalar_type() != at::kBFloat16) || out->dim() != 2 ||
        out->size(0) != g.M || out->size(1) != g.N || out->stride(1) != 1)
      return none();
  } else {
    if (g.accumulate) return none();
    y = at::empty({g.M, g.N}, of(*A, g.fp32 ? at::kFloat : at::kBFloat16));
  }
  const Tensor& c = out ? *out : y;
  g.c = c.data_ptr(); g.ldc = c.stride(0);
  g.bias = ptr(bias);
  if (res) { g.res = res->data_ptr(); g.ldres = res->stride(0); }
  if (aux) { g.aux = aux->data_ptr(); g.ldaux = aux->stride(0); }
  if (alpha_dev) g.alpha_dev = alpha_dev->data_ptr<float>();
  if (int rc = g.run(*A, a.status(14))) return code(rc);
  if (out) {
    Py_INCREF(a.v[4]);
    return a.v[4];
  }
  return wrap(std::move(y));
}

// linear(x, w, b, residual, status) -> x w^T (+ b) (+ residual), in x's leading dimensions
NK_FUNCTION(linear, 5) {
  if (!a.tensors({0, 1, 2, 3})) return none();
  const Tensor *x = a.tensor(0), *w = a.tensor(1), *b = a.tensor(2), *r = a.tensor(3);
  if (!x || !w || !plain(*x) || !plain(*w) || w->dim() != 2 || x->size(-1) != w->size(1) ||
      !vec_or_none(b, w->size(0)) || !plain_or_none(r))
    return none();
  const long long N = w->size(0);
  if (r && (r->numel() != rows_of(*x) * N || r->size(-1) != N)) return none();
  Tensor y = empty_with_cols(*x, N);
  Gemm g = fwd(*x, *w, y);
  g.bias = ptr(b); g.res = ptr(r); g.ldres = r ? N : 0;
  if (!g.ok()) return none();
  if (int rc = g.run(*x, a.status(4))) return code(rc);
  return wrap(std::move(y));
}

// linear_bwd(dy, x, w, need_dx, dw, acc_w, db, acc_b, acc, tickets, status) -> (dx,) or ()
NK_FUNCTION(linear_bwd, 11) {
  if (!a.tensors({0, 1, 2, 4, 6, 8, 9})) return none();
  const Tensor *dy = a.tensor(0), *x = a.tensor(1), *w = a.tensor(2), *dw = a.tensor(4),
               *db = a.tensor(6);
  if (!dy || !x || !w || !plain(*dy) || !plain(*x) || !plain(*w) || w->dim() != 2) return none();
  const long long N = w->size(0), K = w->size(1), M = rows_of(*dy);
  if (dy->size(-1) != N || x->size(-1) != K || rows_of(*x) != M || ((N | K) & 7) || !fits(M) ||
      !fits(N) || !fits(K) || !target(dw, *w) || !bias_target(db, N))
    return none();
  const Scratch s(a, 8);
  if (db && !s.acc) return none();
  int* status = a.status(10);
  Tensor dx;
  if (a.flag(3)) {
    dx = empty_with_cols(*dy, K);
    if (int rc = dgrad(*dy, *w, dx).run(*dy, status)) return code(rc);
  }
  if (dw)
    if (int rc = wgrad(*dy, *x, *dw, a.flag(5)).run(*dy, status)) return code(rc);
  if (db)
    if (int rc = colsum(*dy, *db, a.flag(7), s)) return code(rc);
  return dx.defined() ? tuple(std::move(dx)) : tuple();
}

// mlp(x, w1, b1, w2, b2, residual, status) -> (y, h, z): z = x w1^T + b1, h = gelu(z),
// y = h w2^T + b2 (+ residual)
NK_FUNCTION(mlp, 7) {
  if (!a.tensors({0, 1, 2, 3, 4, 5})) return none();
  const Tensor *x = a.tensor(0), *w1 = a.tensor(1), *b1 = a.tensor(2), *w2 = a.tensor(3),
               *b2 = a.tensor(4), *r = a.tensor(5);
  if (!x || !w1 || !w2 || !plain(*x) || !plain(*w1) || !plain(*w2) || w1->dim() != 2 ||
      w2->dim() != 2)
    return none();
  const long long F = w1->size(0), N = w2->size(0), M = rows_of(*x);
  if (x->size(-1) != w1->size(1) || w2->size(1) != F || !vec_or_none(b1, F) ||
      !vec_or_none(b2, N) || !plain_or_none(r) ||
      (r && (r->numel() != M * N || r->size(-1) != N)))
    return none();
  Tensor z = at::empty({M, F}, of(*x, at::kBFloat16)), h = at::empty({M, F}, of(*x, at::kBFloat16));
  Tensor y = empty_with_cols(*x, N);
  Gemm g1 = fwd(*x, *w1, h), g2 = fwd(h, *w2, y);
  g1.bias = ptr(b1); g1.epi = NKB_EPI_GELU_FWD; g1.aux = z.data_ptr(); g1.ldaux = F;
  g2.bias = ptr(b2); g2.res = ptr(r); g2.ldres = r ? N : 0;
  if (!g1.ok() || !g2.ok()) return none();
  if (int rc = g1.run(*x, a.status(6))) return code(rc);
  if (int rc = g2.run(*x, a.status(6))) return code(rc);
  return tuple(std::move(y), std::move(h), std::move(z));
}

// mlp_bwd(dy, x, w1, w2, h, z, need_dx, dw1, acc, db1, acc, dw2, acc, db2, acc, acc, tickets, status)
// -> (dx,) or ()
NK_FUNCTION(mlp_bwd, 18) {
  if (!a.tensors({0, 1, 2, 3, 4, 5, 7, 9, 11, 13, 15, 16})) return none();
  const Tensor *dy = a.tensor(0), *x = a.tensor(1), *w1 = a.tensor(2), *w2 = a.tensor(3),
               *h = a.tensor(4), *z = a.tensor(5), *dw1 = a.tensor(7), *db1 = a.tensor(9),
               *dw2 = a.tensor(11), *db2 = a.tensor(13);
  for (const Tensor* t : {dy, x, w1, w2, h, z})
    if (!t || !plain(*t)) return none();
  if (w1->dim() != 2 || w2->dim() != 2) return none();
  const long long F = w1->size(0), K = w1->size(1), N = w2->size(0), M = rows_of(*dy);
  if (dy->size(-1) != N || w2->size(1) != F || x->size(-1) != K || rows_of(*x) != M ||
      h->numel() != M * F || h->size(-1) != F || z->numel() != M * F || z->size(-1) != F ||
      ((N | F | K) & 7) || !fits(M) || !fits(N) || !fits(F) || !fits(K) || !target(dw1, *w1) ||
      !target(dw2, *w2) || !bias_target(db1, F) || !bias_target(db2, N))
    return none();
  const Scratch s(a, 15);
  if ((db1 || db2) && !s.acc) return none();
  int* status = a.status(17);
  Tensor dz = at::empty({M, F}, of(*dy, at::kBFloat16));
  Gemm g = dgrad(*dy, *w2, dz);
  g.epi = NKB_EPI_GELU_BWD; g.aux = z->data_ptr(); g.ldaux = F;
  if (int rc = g.run(*dy, status)) return code(rc);
  if (dw2)
    if (int rc = wgrad(*dy, *h, *dw2, a.flag(12)).run(*dy, status)) return code(rc);
  if (db2)
    if (int rc = colsum(*dy, *db2, a.flag(14), s)) return code(rc);
  Tensor dx;
  if (a.flag(6)) {
    dx = empty_with_cols(*dy, K);
    if (int rc = dgrad(dz, *w1, dx).run(*dy, status)) return code(rc);
  }
  if (dw1)
    if (int rc = wgrad(dz, *x, *dw1, a.flag(8)).run(*dy, status)) return code(rc);
  if (db1)
    if (int rc = colsum(dz, *db1, a.flag(10), s)) return code(rc);
  return dx.defined() ? tuple(std::move(dx)) : tuple();
}

// norm(x, w, b, eps, rms) -> (y, stats [rows, 2])
NK_FUNCTION(norm, 5) {
  if (!a.tensors({0, 1, 2})) return none();
  const Tensor *x = a.tensor(0), *w = a.tensor(1), *b = a.tensor(2);
  if (!x || !w || !plain(*x) || !plain(*w) || !plain_or_none(b)) return none();
  const long long C = x->size(-1), rows = rows_of(*x);
  if (w->numel() != C || (b && b->numel() != C) || (C & 7) || !fits(rows) || !fits(C)) return none();
  const float eps = (float)a.real(3);
  const int rms = a.flag(4);
  if (PyErr_Occurred()) return none();
  Tensor y = at::empty(x->sizes(), of(*x, at::kBFloat16));
  Tensor stats = at::empty({rows, 2}, of(*x, at::kFloat));
  void* s = stream();
  if (int rc = launch([&] {
        return nkb_norm_fwd(x->data_ptr(), w->data_ptr(), ptr(b), y.data_ptr(),
                            stats.data_ptr<float>(), (int)rows, (int)C, eps, rms, s);
      }))
    return code(rc);
  return tuple(std::move(y), std::move(stats));
}

// norm_bwd(dy, x, w, stats, dres, rms, dw, acc_w, db, acc_b, acc, tickets) -> dx
NK_FUNCTION(norm_bwd, 12) {
  if (!a.tensors({0, 1, 2, 3, 4, 6, 8, 10, 11})) return none();
  const Tensor *dy = a.tensor(0), *x = a.tensor(1), *w = a.tensor(2), *stats = a.tensor(3),
               *dres = a.tensor(4), *dw = a.tensor(6), *db = a.tensor(8);
  if (!dy || !x || !w || !stats || !dw || !plain(*dy) || !plain(*x) || !plain(*w) ||
      !plain_or_none(dres) || dy->numel() != x->numel() || dy->size(-1) != x->size(-1) ||
      (dres && (dres->numel() != x->numel() || dres->size(-1) != x->size(-1))))
    return none();
  const long long C = x->size(-1), rows = rows_of(*x);
  if (w->numel() != C || (C & 7) || !fits(rows) || !fits(C) || !target(dw, *w) ||
      !vec_or_none(db, C) || !stats->is_cuda() || stats->scalar_type() != at::kFloat ||
      !stats->is_contiguous() || stats->numel() != 2 * rows)
    return none();
  const Scratch s(a, 10);
  if (!s.acc) return none();
  Tensor dx = at::empty(dy->sizes(), of(*x, at::kBFloat16));
  const int rms = a.flag(5), aw = a.flag(7), ab = a.flag(9);
  void* st = stream();
  if (int rc = launch([&] {
        return nkb_norm_bwd_all(dy->data_ptr(), x->data_ptr(), w->data_ptr(),
                                stats->data_ptr<float>(), dx.data_ptr(), ptr(dres), (int)rows,
                                (int)C, rms, s.acc, s.tickets, dw->data_ptr(), ptr(db), aw, ab, st);
      }))
    return code(rc);
  return wrap(std::move(dx));
}

struct Heads {  // of a packed [B, S, 3 H D]
  long long B, S, C, D;
  int H;
  float scale;
  bool of(const Tensor& qkv, long long n_head) {
    if (!plain(qkv) || qkv.dim() != 3 || n_head <= 0 || qkv.size(2) % (3 * n_head)) return false;
    B = qkv.size(0); S = qkv.size(1); C = qkv.size(2) / 3; H = (int)n_head; D = C / n_head;
    scale = (float)(1.0 / std::sqrt((double)D));
    return (D == 64 || D == 128) && fits(B * H) && fits(S);
  }
};

// attn(qkv, H, causal, status) -> (out [B, S, C], lse [B, H, S])
NK_FUNCTION(attn, 4) {
  if (!a.tensors({0}) || a.v[0] == Py_None) return none();
  const Tensor& qkv = *a.tensor(0);
  Heads n;
  if (!n.of(qkv, a.num(1))) return none();
  const int causal = a.flag(2);
  Tensor out = at::empty({n.B, n.S, n.C}, of(qkv, at::kBFloat16));
  Tensor lse = at::empty({n.B, n.H, n.S}, of(qkv, at::kFloat));
  const char* q = static_cast<const char*>(qkv.data_ptr());
  int* status = a.status(3);
  void* s = stream();
  if (int rc = launch([&] {
        return nkb_attn_fwd(q, q + 2 * n.C, q + 4 * n.C, out.data_ptr(), lse.data_ptr<float>(),
                            (int)n.B, n.H, (int)n.S, (int)n.D, n.S * 3 * n.C, n.D, 3 * n.C,
                            n.S * n.C, n.D, n.C, n.scale, causal, status, s);
      }))
    return code(rc);
  return tuple(std::move(out), std::move(lse));
}

// attn_bwd(qkv, out, lse, dout, H, causal, status) -> dqkv
NK_FUNCTION(attn_bwd, 7) {
  if (!a.tensors({0, 1, 2, 3})) return none();
  const Tensor *qkv = a.tensor(0), *out = a.tensor(1), *lse = a.tensor(2), *dout = a.tensor(3);
  Heads n;
  if (!qkv || !out || !lse || !dout || !n.of(*qkv, a.num(4)) || !plain(*out) || !plain(*dout) ||
      out->numel() != n.B * n.S * n.C || dout->numel() != n.B * n.S * n.C || !lse->is_cuda() ||
      !lse->is_contiguous() || lse->scalar_type() != at::kFloat ||
      lse->numel() != n.B * n.H * n.S)
    return none();
  const int causal = a.flag(5);
  Tensor dqkv = at::empty(qkv->sizes(), of(*qkv, at::kBFloat16));
  Tensor delta = at::empty({n.B, n.H, n.S}, of(*qkv, at::kFloat));
  Tensor dq_acc = at::empty({n.B, n.H, n.S, n.D}, of(*qkv, at::kFloat));  // cleared by the call
  const char* q = static_cast<const char*>(qkv->data_ptr());
  char* dq = static_cast<char*>(dqkv.data_ptr());
  int* status = a.status(6);
  void* s = stream();
  if (int rc = launch([&] {
        return nkb_attn_bwd(q, q + 2 * n.C, q + 4 * n.C, out->data_ptr(), dout->data_ptr(),
                            lse->data_ptr<float>(), dq, dq + 2 * n.C, dq + 4 * n.C,
                            delta.data_ptr<float>(), dq_acc.data_ptr<float>(), (int)n.B, n.H,
                            (int)n.S, (int)n.D, n.S * 3 * n.C, n.D, 3 * n.C, n.S * n.C, n.D, n.C,
                            n.scale, causal, status, s);
      }))
    return code(rc);
  return wrap(std::move(dqkv));
}

// conv(x [N,H,W,C], w, KH, KW, stride, pad, status) -> y on the image itself
NK_FUNCTION(conv, 7) {
  if (!a.tensors({0, 1}) || a.v[0] == Py_None || a.v[1] == Py_None) return none();
  const Tensor &x = *a.tensor(0), &w = *a.tensor(1);
  const long long KH = a.num(2), KW = a.num(3), st = a.num(4), pad = a.num(5);
  if (PyErr_Occurred() || !plain(x) || !plain(w) || x.dim() != 4 || w.dim() != 2 || st < 1)
    return none();
  const long long N = x.size(0), H = x.size(1), W = x.size(2), C = x.size(3);
  if (w.size(1) != KH * KW * C || H + 2 * pad < KH || W + 2 * pad < KW || !fits(N) || !fits(H) ||
      !fits(W) || !fits(C) || !fits(w.size(0)))
    return none();
  Tensor y = at::empty({N, (H + 2 * pad - KH) / st + 1, (W + 2 * pad - KW) / st + 1, w.size(0)},
                       of(x, at::kBFloat16));
  int* status = a.status(6);
  void* s = stream();
  if (int rc = launch([&] {
        return nkb_conv_fwd(x.data_ptr(), w.data_ptr(), y.data_ptr(), (int)N, (int)H, (int)W, (int)C,
                            (int)w.size(0), (int)KH, (int)KW, (int)st, (int)pad, status, s);
      }))
    return code(rc);
  return wrap(std::move(y));
}

// bn_eval(x, mean, var, eps, w, b, residual, relu) -> y
NK_FUNCTION(bn_eval, 8) {
  if (!a.tensors({0, 1, 2, 4, 5, 6})) return none();
  const Tensor *x = a.tensor(0), *mean = a.tensor(1), *var = a.tensor(2), *w = a.tensor(4),
               *b = a.tensor(5), *r = a.tensor(6);
  if (!x || !mean || !var || !w || !b || !plain(*x) || !plain(*w) || !plain(*b) || !plain_or_none(r))
    return none();
  const long long C = x->size(-1);
  const double eps = a.real(3);
  if (PyErr_Occurred()) return none();
  for (const Tensor* t : {mean, var})
    if (!t->is_cuda() || t->scalar_type() != at::kFloat || !t->is_contiguous() || t->numel() != C)
      return none();
  if (w->numel() != C || b->numel() != C || (C & 7) || !fits(C) || !(eps >= 0) ||
      (r && (r->numel() != x->numel() || r->size(-1) != C)))
    return none();
  Tensor y = at::empty(x->sizes(), of(*x, at::kBFloat16));
  const int relu = a.flag(7);
  void* s = stream();
  if (int rc = launch([&] {
        return nkb_bn_eval(x->data_ptr(), mean->data_ptr<float>(), var->data_ptr<float>(), (float)eps,
                           w->data_ptr(), b->data_ptr(), ptr(r), y.data_ptr(), rows_of(*x), (int)C,
                           relu, s);
      }))
    return code(rc);
  return wrap(std::move(y));
}

#define ENTRY(name)                                                                \
  {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&name##_py)), \
   METH_FASTCALL, nullptr}

PyMethodDef methods[] = {ENTRY(gemm),     ENTRY(linear),  ENTRY(linear_bwd), ENTRY(mlp),
                         ENTRY(mlp_bwd),  ENTRY(norm),    ENTRY(norm_bwd),   ENTRY(attn),
                         ENTRY(attn_bwd), ENTRY(conv),    ENTRY(bn_eval),
                         {nullptr, nullptr, 0, nullptr}};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_nkops", nullptr, -1, methods,
                      nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__nkops() {
  PyObject* m = PyModule_Create(&module);
  // the tensors' layout is that of the torch it was built with
  if (m && PyModule_AddStringConstant(m, "torch_version", TORCH_VERSION) < 0) Py_CLEAR(m);
  return m;
}
