// Launch sequences of whole decoder sub-layers: what runs between two library attention calls, forward or backward, as ONE call from
// Python.  Written in Python, a launch of these sequences costs 15 to 25 us of host time (allocation, strides, addresses, plan, call),
// more than most kernels of a short batch run; here 3 to 4.
//
// The functions allocate their results and launch the library's kernels (bound by address, see api.h) on the current stream; they
// keep nothing.  The callers (models/gpt2.py, models/llama.py) have checked types, layouts and alignment, fit() checks here that the
// operands belong together.  A launch that fails raises through the
// Python check that the other entry points use; no C++ exception leaves a function.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <algorithm>
#include <array>
#include <initializer_list>
#include <map>
#include <vector>

#include "api.h"

#ifdef OB_DIGEST
__attribute__((used)) static const char digest[] = OB_DIGEST;      // of this file, api.h and torch's version (utils/build.py)
#endif

namespace {

using at::Tensor;

#define OB_ENTRIES(X)                                                                                                          \
  X(ob_gemm_tn) X(ob_gemm_tn_act) X(ob_gemm_pair) X(ob_gemm_pair_glu_bwd) X(ob_glu_bwd) X(ob_rmsnorm_fwd) X(ob_rmsnorm_bwd) X(ob_layernorm_fwd)  \
  X(ob_layernorm_bwd_dx) X(ob_layernorm_bwd_sums) X(ob_add_layernorm_fwd) X(ob_add_layernorm_bwd_dx) X(ob_activation) X(ob_merge_heads3) X(ob_lora_pack) \
  X(ob_rope_qk_oop) X(ob_rope_qkv_gather) X(ob_wgrad_clip_batch) X(ob_wgrad_clip_pe_batch) \
  X(ob_ghost_norm_batch) X(ob_rows_sum_batch)
#define X(name) decltype(&name) p_##name = nullptr;
OB_ENTRIES(X)
#undef X

// lib.check(rc, what); (M, N, K, K2, mode) -> 0 pair, 64 or 256: tile width; (tiles, rows, most, peer) -> splits of a weight gradient
PyObject *g_check = nullptr, *g_plan = nullptr, *g_splits = nullptr;
int g_sms = 0;
double g_budget = 0.0;

struct PythonError {};                               // a Python exception is set

void done(int rc, const char* what) {
  PyObject* r = PyObject_CallFunction(g_check, "is", rc, what);
  if (r == nullptr) throw PythonError();
  Py_DECREF(r);
}
void* stream() { return c10::cuda::getCurrentCUDAStream().stream(); }
// Launches without the interpreter lock (a full launch queue blocks); the arguments are evaluated before it is given up.
template <class F, class... A>
void launch(const char* what, F entry, A... args) {
  void* const st = stream();
  PyThreadState* const thread = PyEval_SaveThread();
  const int rc = entry(args..., st);
  PyEval_RestoreThread(thread);
  done(rc, what);
}
#define LAUNCH(name, ...) launch(#name, p_##name, __VA_ARGS__)

// The shape checks of the Python entry points: a ValueError before a kernel is given a size that an operand does not have.
void fit(bool ok, const char* what) {
  if (ok) return;
  PyErr_SetString(PyExc_ValueError, what);
  throw PythonError();
}

void* ptr(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }
const float* f32(const Tensor& t) { return static_cast<const float*>(ptr(t)); }
Tensor empty(std::initializer_list<int64_t> shape, const Tensor& like) { return at::empty(shape, like.options()); }
Tensor empty_f32(std::initializer_list<int64_t> shape, const Tensor& like) { return at::empty(shape, like.options().dtype(at::kFloat)); }
// contiguous and on a 16-byte boundary
Tensor vec16(const Tensor& t) {
  if (!t.is_contiguous()) return t.contiguous();
  return (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15) == 0 ? t : t.clone(at::MemoryFormat::Contiguous);
}
Tensor rows(const Tensor& t) { return t.defined() ? vec16(t.reshape({-1, t.size(-1)})) : t; }

// ------------------------------------------------------------------------------------------------------- single launches

// The choice of kernel and tile is the Python rule's; it is asked once per shape.
enum : int { ANY = 0, SINGLE = 1, ACTIVATION = 2 };
int plan(int64_t M, int64_t N, int64_t K, int64_t K2, int mode) {
  static std::map<std::array<int64_t, 5>, int> known;
  const std::array<int64_t, 5> key{M, N, K, K2, mode};
  const auto at = known.find(key);
  if (at != known.end()) return at->second;
  PyObject* r = PyObject_CallFunction(g_plan, "LLLLi", (long long)M, (long long)N, (long long)K, (long long)K2, mode);
  if (r == nullptr) throw PythonError();
  const int width = static_cast<int>(PyLong_AsLong(r));
  Py_DECREF(r);
  if (PyErr_Occurred()) throw PythonError();
  if (known.size() >= 4096) known.clear();
  return known[key] = width;
}

struct Opt {                                         // the optional parts of a product
  Tensor bias, a2, b2;
  bool kn2 = false, single = false;
  float alpha = 1.f;
};
// a [M, K] times b ([N, K], or [K, N] with kn), as ops.gemm
Tensor product(const Tensor& a, const Tensor& b, int64_t N, bool kn, const Opt& o = {}) {
  const int64_t M = a.size(0), K = a.size(1), K2 = o.a2.defined() ? o.a2.size(1) : 0;
  fit(b.dim() == 2 && b.size(kn ? 0 : 1) == K && b.size(kn ? 1 : 0) == N, "inner dimensions differ");
  fit(K2 == 0 || (o.a2.size(0) == M && o.b2.size(o.kn2 ? 0 : 1) == K2 && o.b2.size(o.kn2 ? 1 : 0) == N), "low-rank segment: a2 [M, r], b2 [N, r] (or [r, N])");
  fit(!o.bias.defined() || o.bias.numel() == N, "bias must hold N contiguous values");
  Tensor out = empty({M, N}, a);
  const int width = plan(M, N, K, K2, o.single ? SINGLE : ANY);
  const int64_t lda2 = K2 ? o.a2.stride(0) : 0, ldb2 = K2 ? o.b2.stride(0) : 0;
  if (width == 0)
    LAUNCH(ob_gemm_pair, ptr(a), ptr(b), nullptr, ptr(o.a2), ptr(o.b2), nullptr, ptr(o.bias), ptr(out), nullptr, nullptr, M, (int)N, (int)K, (int)K2,
           a.stride(0), b.stride(0), lda2, ldb2, N, kn, o.kn2, 0, 0, -1, nullptr, g_budget, g_sms);
  else
    LAUNCH(ob_gemm_tn, ptr(a), ptr(b), ptr(o.a2), ptr(o.b2), ptr(o.bias), ptr(out), M, (int)N, (int)K, (int)K2, a.stride(0), b.stride(0), lda2, ldb2,
           N, kn, o.kn2, o.alpha, nullptr, 0, width, nullptr, g_budget, g_sms);
  return out;
}
Opt with_bias(const Tensor& bias) { Opt o; o.bias = bias; return o; }
Opt scaled(double alpha) { Opt o; o.alpha = static_cast<float>(alpha); o.single = true; return o; }
Opt segment(const Tensor& a2, const Tensor& b2, bool kn2) { Opt o; o.a2 = a2; o.b2 = b2; o.kn2 = kn2; return o; }

void fit_norm(const Tensor& x, const Tensor& r, const Tensor& w) {
  fit(w.numel() == x.size(1), "a norm's weight and bias hold one value per column");
  fit(!r.defined() || r.sizes() == x.sizes(), "the two parts of the stream have one shape");
}
// s = x + r (s = x without r) and its norm; stats: mean and rstd [2, rows]
struct Normed {
  Tensor y, s, stats;
};
Normed layer_norm(const Tensor& x, const Tensor& r, const Tensor& w, const Tensor& b, double eps) {
  const int64_t R = x.size(0);
  fit_norm(x, r, w);
  fit_norm(x, r, b);
  Normed n{empty({R, x.size(1)}, x), x, empty_f32({2, R}, x)};
  float* mean = n.stats.data_ptr<float>();
  if (!r.defined()) {
    LAUNCH(ob_layernorm_fwd, ptr(x), ptr(w), ptr(b), ptr(n.y), mean, mean + R, R, (int)x.size(1), (float)eps);
  } else {
    n.s = empty({R, x.size(1)}, x);
    LAUNCH(ob_add_layernorm_fwd, ptr(x), ptr(r), ptr(w), ptr(b), ptr(n.y), ptr(n.s), mean, mean + R, R, (int)x.size(1), (float)eps);
  }
  return n;
}
// sums_w, sums_b [examples, H] (windows of the per-example buffer): the weight's and bias's gradients of every example are added there
struct Sums {
  Tensor w, b;
};
Tensor layer_norm_bwd(const Tensor& dy, const Tensor& s, const Tensor& w, const Tensor& stats, const Tensor& ds, const Sums& sums) {
  const int64_t R = s.size(0);
  Tensor dx = empty({R, s.size(1)}, s);
  const float* mean = f32(stats);
  if (sums.w.defined()) {
    const int64_t E = sums.w.size(0);
    if (R % E != 0 || sums.w.scalar_type() != at::kFloat || sums.b.scalar_type() != at::kFloat || sums.w.size(1) != s.size(1) ||
        sums.b.sizes() != sums.w.sizes() || sums.b.stride(0) != sums.w.stride(0) || sums.w.stride(1) != 1 || sums.b.stride(1) != 1) {
      PyErr_SetString(PyExc_ValueError, "layer_norm_bwd: the sums are fp32 [examples, H] windows of one buffer, rows a multiple of examples");
      throw PythonError();
    }
    LAUNCH(ob_layernorm_bwd_sums, ptr(dy), ptr(s), ptr(w), mean, mean + R, ptr(ds), ptr(dx), (int)E, (int)(R / E), (int)s.size(1),
           sums.w.data_ptr<float>(), sums.b.data_ptr<float>(), sums.w.stride(0));
  } else if (!ds.defined())
    LAUNCH(ob_layernorm_bwd_dx, ptr(dy), ptr(s), ptr(w), mean, mean + R, ptr(dx), R, (int)s.size(1));
  else
    LAUNCH(ob_add_layernorm_bwd_dx, ptr(dy), ptr(s), ptr(w), mean, mean + R, ptr(ds), ptr(dx), R, (int)s.size(1));
  return dx;
}
Normed rms_norm(const Tensor& x, const Tensor& r, const Tensor& w, double eps, double offset, int mode) {
  const int64_t R = x.size(0);
  fit_norm(x, r, w);
  Normed n{empty({R, x.size(1)}, x), r.defined() ? empty({R, x.size(1)}, x) : x, empty_f32({R}, x)};
  LAUNCH(ob_rmsnorm_fwd, ptr(x), ptr(r), ptr(w), ptr(n.y), r.defined() ? ptr(n.s) : nullptr, n.stats.data_ptr<float>(), R, (int)x.size(1),
         (float)eps, (float)offset, mode);
  return n;
}
Tensor rms_norm_bwd(const Tensor& dy, const Tensor& s, const Tensor& w, const Tensor& rstd, const Tensor& ds, double offset) {
  Tensor dx = empty({s.size(0), s.size(1)}, s);
  LAUNCH(ob_rmsnorm_bwd, ptr(dy), ptr(s), ptr(w), f32(rstd), ptr(ds), ptr(dx), nullptr, nullptr, 0, 0, s.size(0), (int)s.size(1), (float)offset);
  return dx;
}
constexpr int GELU_TANH = 2;
Tensor gelu(const Tensor& x, const Tensor& dy) {
  Tensor out = empty({x.size(0), x.size(1)}, x);
  LAUNCH(ob_activation, ptr(x), ptr(dy), ptr(out), x.numel(), GELU_TANH, g_sms);
  return out;
}
// GPT-2's GELU in the epilogue of the product around it: the pair kernel's or, with 64-column tiles, the single-CTA kernel's.
// -> gelu(x b^T + bias) and, with `pre`, its argument there (allocated)
Tensor product_gelu(const Tensor& x, const Tensor& b, const Tensor& bias, Tensor* pre) {
  const int64_t M = x.size(0), N = b.size(0), K = x.size(1);
  if (N % 64 != 0) {
    const Tensor f = product(x, b, N, false, with_bias(bias));
    if (pre != nullptr) *pre = f;
    return gelu(f, Tensor());
  }
  fit(b.size(1) == K, "inner dimensions differ");
  fit(bias.numel() == N, "bias must hold N contiguous values");
  Tensor h = empty({M, N}, x);
  if (pre != nullptr) *pre = empty({M, N}, x);
  void* const f = pre != nullptr ? ptr(*pre) : nullptr;
  if (plan(M, N, K, 0, ACTIVATION) == 0)
    LAUNCH(ob_gemm_pair, ptr(x), ptr(b), nullptr, nullptr, nullptr, nullptr, ptr(bias), ptr(h), f, nullptr, M, (int)N, (int)K, 0, x.stride(0),
           b.stride(0), 0, 0, N, 0, 0, 2, GELU_TANH, -1, nullptr, g_budget, g_sms);
  else
    LAUNCH(ob_gemm_tn_act, ptr(x), ptr(b), ptr(bias), ptr(h), f, M, (int)N, (int)K, x.stride(0), b.stride(0), 0, GELU_TANH, 0, nullptr, g_budget, g_sms);
  return h;
}
// -> (g w) * gelu'(f)
Tensor product_gelu_bwd(const Tensor& g, const Tensor& w, const Tensor& f) {
  const int64_t M = g.size(0), N = w.size(1), K = g.size(1);
  if (N % 64 != 0) return gelu(f, product(g, w, N, true));
  fit(w.size(0) == K && f.size(0) == M && f.size(1) == N, "inner dimensions differ");
  Tensor df = empty({M, N}, g);
  if (plan(M, N, K, 0, ACTIVATION) == 0)
    LAUNCH(ob_gemm_pair_glu_bwd, ptr(g), ptr(w), ptr(f), nullptr, ptr(df), nullptr, M, (int)N, (int)K, g.stride(0), w.stride(0), N, N, 1, GELU_TANH,
           nullptr, g_budget, g_sms);
  else
    LAUNCH(ob_gemm_tn_act, ptr(g), ptr(w), nullptr, ptr(df), ptr(f), M, (int)N, (int)K, g.stride(0), w.stride(0), 1, GELU_TANH, 1, nullptr, g_budget,
           g_sms);
  return df;
}
// q, k [B, T, heads, hd] through their strides -> rotated, contiguous
bool rope_reads(const Tensor& t) {
  return t.stride(3) == 1 && (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15) == 0 && ((t.stride(0) | t.stride(1) | t.stride(2)) & 7) == 0;
}
std::pair<Tensor, Tensor> rope(const Tensor& q, const Tensor& k, const Tensor& cs, const Tensor& sn) {
  const int64_t B = q.size(0), T = q.size(1), hd = q.size(3);
  for (const Tensor* t : {&cs, &sn}) fit(t->dim() == 2 && t->size(0) >= T && t->size(1) == hd / 2, "rotary tables [positions, head size / 2] of too few positions");
  Tensor qo = empty({B, T, q.size(2), hd}, q), ko = empty({B, T, k.size(2), hd}, k);
  LAUNCH(ob_rope_qk_oop, ptr(q), ptr(k), ptr(qo), ptr(ko), f32(cs), f32(sn), nullptr, B * T, (int)T, (int)q.size(2), (int)k.size(2), (int)hd, q.stride(0),
         q.stride(1), q.stride(2), k.stride(0), k.stride(1), k.stride(2), 0, g_sms);
  return {qo, ko};
}
// gradients [B, heads, T, hd] -> [B * T, (heads + 2 kv heads) * hd], query and key rotated back
Tensor rope_backward(Tensor q, Tensor k, Tensor v, const Tensor& cs, const Tensor& sn) {
  long long strides[9];
  int i = 0;
  for (Tensor* t : {&q, &k, &v}) {
    if (!rope_reads(*t)) *t = t->clone(at::MemoryFormat::Contiguous);
    for (int d : {0, 2, 1}) strides[i++] = t->stride(d);
  }
  const int64_t B = q.size(0), Hq = q.size(1), T = q.size(2), hd = q.size(3), Hk = k.size(1);
  Tensor out = empty({B * T, (Hq + 2 * Hk) * hd}, q);
  LAUNCH(ob_rope_qkv_gather, ptr(q), ptr(k), ptr(v), ptr(out), f32(cs), f32(sn), strides, B * T, (int)T, (int)Hq, (int)Hk, (int)hd, 1, g_sms);
  return out;
}
// three gradients [B, heads, T, hd] -> [B * T, 3 * heads * hd]
Tensor merge_heads(const Tensor& q, const Tensor& k, const Tensor& v) {
  const int64_t B = q.size(0), H = q.size(1), T = q.size(2), hd = q.size(3);
  Tensor out = empty({B * T, 3 * H * hd}, q);
  const Tensor* parts[3] = {&q, &k, &v};
  long long strides[9];
  bool ok = hd % 8 == 0;
  for (int i = 0; i < 3; ++i) {
    ok = ok && parts[i]->scalar_type() == at::kBFloat16 && rope_reads(*parts[i]);
    for (int j = 0; j < 3; ++j) strides[3 * i + j] = parts[i]->stride(j);
  }
  if (ok) {
    LAUNCH(ob_merge_heads3, ptr(q), ptr(k), ptr(v), strides, ptr(out), B, (int)T, (int)H, (int)hd, g_sms);
  } else {
    Tensor v5 = out.view({B, T, 3, H, hd});
    for (int i = 0; i < 3; ++i) v5.select(2, i).copy_(parts[i]->transpose(1, 2));
  }
  return out;
}

// ------------------------------------------------------------------------------------------------------- Python arguments

struct Args {
  PyObject* const* a;
  Py_ssize_t n, i = 0;
  PyObject* next() {
    if (i >= n) {
      PyErr_SetString(PyExc_TypeError, "too few arguments");
      throw PythonError();
    }
    return a[i++];
  }
  Tensor tensor() {
    PyObject* o = next();
    if (!THPVariable_Check(o)) {
      PyErr_Format(PyExc_TypeError, "expected a tensor, got %.80s", Py_TYPE(o)->tp_name);
      throw PythonError();
    }
    return THPVariable_Unpack(o);
  }
  Tensor optional() {
    if (i < n && a[i] == Py_None) {
      ++i;
      return Tensor();
    }
    return tensor();
  }
  double number() {
    const double v = PyFloat_AsDouble(next());
    if (v == -1.0 && PyErr_Occurred()) throw PythonError();
    return v;
  }
  long long integer() {
    const long long v = PyLong_AsLongLong(next());
    if (v == -1 && PyErr_Occurred()) throw PythonError();
    return v;
  }
};
PyObject* pack(std::initializer_list<Tensor> ts) {
  PyObject* out = PyTuple_New(static_cast<Py_ssize_t>(ts.size()));
  if (out == nullptr) throw PythonError();
  Py_ssize_t i = 0;
  for (const Tensor& t : ts) {
    PyObject* o = t.defined() ? THPVariable_Wrap(t) : Py_NewRef(Py_None);
    if (o == nullptr) {
      Py_DECREF(out);
      throw PythonError();
    }
    PyTuple_SET_ITEM(out, i++, o);
  }
  return out;
}
template <PyObject* (*F)(Args&)>
PyObject* call(PyObject*, PyObject* const* a, Py_ssize_t n) {
  Args args{a, n};
  try {
    return F(args);
  } catch (const PythonError&) {
  } catch (const std::exception&) {                 // of the type that torch's own calls raise: torch.OutOfMemoryError, IndexError, ...
    torch::translate_exception_to_python(std::current_exception());
  } catch (...) {
    PyErr_SetString(PyExc_RuntimeError, "unknown C++ exception");
  }
  return nullptr;
}

// ------------------------------------------------------------------------------------------------------- GPT-2

// (x, residual | None, ln_w, ln_b, w, b, eps) -> y, s, stats, qkv
PyObject* gpt2_in(Args& a) {
  const Tensor x = rows(a.tensor()), r = rows(a.optional()), lw = a.tensor(), lb = a.tensor(), w = a.tensor(), b = a.tensor();
  const Normed n = layer_norm(x, r, lw, lb, a.number());
  return pack({n.y, n.s, n.stats, product(n.y, w, w.size(0), false, with_bias(b))});
}
// (dq, dk, dv, w, s, ln_w, stats, ds | None, need_dx, sums_w | None, sums_b | None) -> g, dy, dx
PyObject* gpt2_in_bwd(Args& a) {
  const Tensor dq = a.tensor(), dk = a.tensor(), dv = a.tensor(), w = a.tensor(), s = a.tensor(), lw = a.tensor(), stats = a.tensor(),
               ds = rows(a.optional()), g = merge_heads(dq, dk, dv);
  Tensor dy, dx;
  if (a.integer()) {
    const Tensor sums_w = a.optional(), sums_b = a.optional();
    dy = product(g, w, s.size(1), true);
    dx = layer_norm_bwd(dy, s, lw, stats, ds, {sums_w, sums_b});
  }
  return pack({g, dy, dx});
}
// (o [B, heads, T, hd], residual, wo, bo, ln_w, ln_b, w1, b1, w2, b2, eps, keep) -> o2, y, s, stats, f | None, h, m
PyObject* gpt2_out(Args& a) {
  const Tensor o = a.tensor(), r = rows(a.tensor()), wo = a.tensor(), bo = a.tensor(), lw = a.tensor(), lb = a.tensor(), w1 = a.tensor(),
               b1 = a.tensor(), w2 = a.tensor(), b2 = a.tensor();
  const Tensor o2 = vec16(o.transpose(1, 2).reshape({o.size(0) * o.size(2), o.size(1) * o.size(3)}));
  const Normed n = layer_norm(product(o2, wo, wo.size(0), false, with_bias(bo)), r, lw, lb, a.number());
  Tensor f;
  const Tensor h = product_gelu(n.y, w1, b1, a.integer() ? &f : nullptr);
  return pack({o2, n.y, n.s, n.stats, f, h, product(h, w2, w2.size(0), false, with_bias(b2))});
}
// (dm, f, w2, w1, s, ln_w, stats, ds, wo, sums_w | None, sums_b | None) -> g2, g1, dy, dx, do [rows, heads * hd]
PyObject* gpt2_out_bwd(Args& a) {
  const Tensor g2 = rows(a.tensor()), f = a.tensor(), w2 = a.tensor(), w1 = a.tensor(), s = a.tensor(), lw = a.tensor(), stats = a.tensor(),
               ds = rows(a.tensor()), wo = a.tensor(), sums_w = a.optional(), sums_b = a.optional();
  const Tensor g1 = product_gelu_bwd(g2, w2, f), dy = product(g1, w1, w1.size(1), true);
  const Tensor dx = layer_norm_bwd(dy, s, lw, stats, ds, {sums_w, sums_b});
  return pack({g2, g1, dy, dx, product(dx, wo, wo.size(1), true)});
}

// ------------------------------------------------------------------------------------------------------- Llama with LoRA

// (x [B, T, d], residual | None, norm_w, eps, offset, mode, aq, bq, ak, bk, av, bv, scaling, w_all, cos, sin, heads, kv heads, hd)
//   -> y, s, rstd, a_cat, b_block, xa, q, k [B, T, heads, hd] rotated, qkv
PyObject* lora_in(Args& a) {
  const Tensor x3 = a.tensor(), x = rows(x3), r = rows(a.optional()), nw = a.tensor();
  const double eps = a.number(), offset = a.number();
  const int mode = static_cast<int>(a.integer());
  const Tensor aq = a.tensor(), bq = a.tensor(), ak = a.tensor(), bk = a.tensor(), av = a.tensor(), bv = a.tensor();
  const double scaling = a.number();
  const Tensor w_all = a.tensor(), cs = a.tensor(), sn = a.tensor();
  const int64_t nh = a.integer(), nkv = a.integer(), hd = a.integer(), rank = aq.size(0);
  for (const Tensor* f : {&aq, &ak, &av}) fit(f->sizes() == aq.sizes() && f->size(1) == x.size(1), "LoRA factors A [r, in] of one rank");
  for (const Tensor* f : {&bq, &bk, &bv}) fit(f->size(1) == rank, "LoRA factors B [out, r] of one rank");
  const Normed n = rms_norm(x, r, nw, eps, offset, mode);
  const Tensor a_cat = empty({3 * rank, aq.size(1)}, aq), b_block = empty({bq.size(0) + bk.size(0) + bv.size(0), 3 * rank}, aq);
  LAUNCH(ob_lora_pack, ptr(aq), ptr(ak), ptr(av), ptr(bq), ptr(bk), ptr(bv), ptr(a_cat), ptr(b_block), (int)rank, (int)aq.size(1), (int)bq.size(0),
         (int)bk.size(0), (int)bv.size(0), g_sms);
  const Tensor xa = product(n.y, a_cat, 3 * rank, false, scaled(scaling)), qkv = product(n.y, w_all, w_all.size(0), false, segment(xa, b_block, false));
  const Tensor heads = qkv.view({x3.size(0), x3.size(1), nh + 2 * nkv, hd});
  const auto [q, k] = rope(heads.narrow(2, 0, nh), heads.narrow(2, nh, nkv), cs, sn);
  return pack({n.y, n.s, n.stats, a_cat, b_block, xa, q, k, qkv});
}
// (dq, dk, dv [B, heads, T, hd], cos, sin, b_block, scaling, w_all, a_cat, s, norm_w, rstd, ds | None, offset, need_dx) -> g, q_all, dx
PyObject* lora_in_bwd(Args& a) {
  const Tensor dq = a.tensor(), dk = a.tensor(), dv = a.tensor(), cs = a.tensor(), sn = a.tensor(), b_block = a.tensor();
  const double scaling = a.number();
  const Tensor w_all = a.tensor(), a_cat = a.tensor(), s = a.tensor(), nw = a.tensor(), rstd = a.tensor(), ds = rows(a.optional());
  const double offset = a.number();
  const Tensor g = rope_backward(dq, dk, dv, cs, sn), q_all = product(g, b_block, b_block.size(1), true, scaled(scaling));
  Tensor dx;
  if (a.integer()) dx = rms_norm_bwd(product(g, w_all, w_all.size(1), true, segment(q_all, a_cat, true)), s, nw, rstd, ds, offset);
  return pack({g, q_all, dx});
}
// (o [B, heads, T, hd], a, scaling, wo, b, residual, norm_w, eps, offset, mode, w_gate, w_up, act, w_down, keep)
//   -> o2, xa, s, rstd, g | None, u | None, m
PyObject* lora_out(Args& a) {
  const Tensor o = a.tensor(), la = a.tensor();
  const double scaling = a.number();
  const Tensor wo = a.tensor(), lb = a.tensor(), r = rows(a.tensor()), nw = a.tensor();
  const double eps = a.number(), offset = a.number();
  const int mode = static_cast<int>(a.integer());
  const Tensor wg = a.tensor(), wu = a.tensor();
  const int act = static_cast<int>(a.integer());
  const Tensor wd = a.tensor();
  const bool keep = a.integer() != 0;
  const Tensor o2 = vec16(o.transpose(1, 2).reshape({o.size(0) * o.size(2), o.size(1) * o.size(3)})), xa = product(o2, la, la.size(0), false, scaled(scaling));
  const Normed n = rms_norm(product(o2, wo, wo.size(0), false, segment(xa, lb, false)), r, nw, eps, offset, mode);
  const int64_t M = o2.size(0), I = wg.size(0), K = wg.size(1);
  fit(K == n.y.size(1) && wu.sizes() == wg.sizes(), "gate and up projections [I, K]");
  const Tensor h = empty({M, I}, o2), g = keep ? empty({M, I}, o2) : Tensor(), u = keep ? empty({M, I}, o2) : Tensor();
  LAUNCH(ob_gemm_pair, ptr(n.y), ptr(wg), ptr(wu), nullptr, nullptr, nullptr, nullptr, ptr(h), ptr(g), ptr(u), M, (int)(2 * I), (int)K, 0, K,
         wg.stride(0), 0, 0, I, 0, 0, 1, act, -1, nullptr, g_budget, g_sms);
  return pack({o2, xa, n.s, n.stats, g, u, product(h, wd, wd.size(0), false)});
}
// (dm, w_down, g, u, act, fused, w_gate, w_up, s, norm_w, rstd, ds, offset, b, scaling, wo, a) -> dx, q, do [rows, heads * hd]
PyObject* lora_out_bwd(Args& a) {
  const Tensor d2 = rows(a.tensor()), wd = a.tensor(), g = a.tensor(), u = a.tensor();
  const int act = static_cast<int>(a.integer());
  const bool one_launch = a.integer() != 0;
  const Tensor wg = a.tensor(), wu = a.tensor(), s = a.tensor(), nw = a.tensor(), rstd = a.tensor(), ds = rows(a.tensor());
  const double offset = a.number();
  const Tensor lb = a.tensor();
  const double scaling = a.number();
  const Tensor wo = a.tensor(), la = a.tensor();
  const int64_t M = g.size(0), I = g.size(1);
  fit(d2.size(0) == M && wd.size(0) == d2.size(1) && wd.size(1) == I, "inner dimensions differ");
  Tensor dg = empty({M, I}, g), du = empty({M, I}, g);
  if (one_launch) {
    LAUNCH(ob_gemm_pair_glu_bwd, ptr(d2), ptr(wd), ptr(g), ptr(u), ptr(dg), ptr(du), M, (int)I, (int)d2.size(1), d2.stride(0), wd.stride(0), I, I, 1,
           act, nullptr, g_budget, g_sms);
  } else {
    const Tensor dh = product(d2, wd, I, true);
    LAUNCH(ob_glu_bwd, ptr(dh), ptr(g), ptr(u), ptr(dg), ptr(du), M, (int)I, I, I, act, g_sms);
  }
  const Tensor dy = product(dg, wg, wg.size(1), true, segment(du, wu, true));
  dg.reset();
  du.reset();
  const Tensor dx = rms_norm_bwd(dy, s, nw, rstd, ds, offset), q = product(dx, lb, lb.size(1), true, scaled(scaling));
  return pack({dx, q, product(dx, wo, wo.size(1), true, segment(q, la, true))});
}

// Stored (not accumulated) weight gradients of every example, one launch:
// (jobs, out, seg_offsets, groups, group_stride, status address), jobs: (a, b, out_offset, ldm, ldn, n_valid), tiles of 64 columns.
PyObject* store_wgrads(Args& args) {
  PyObject* jobs = args.next();
  const Tensor out = args.tensor(), seg = args.tensor();
  const long long groups = args.integer(), group_stride = args.integer(), status = args.integer();
  if (!PyTuple_Check(jobs) || PyTuple_GET_SIZE(jobs) > 8 || out.scalar_type() != at::kFloat) {
    PyErr_SetString(PyExc_TypeError, "store_wgrads: at most eight jobs and an fp32 destination");
    throw PythonError();
  }
  const int count = static_cast<int>(PyTuple_GET_SIZE(jobs));
  const long long room = static_cast<long long>(out.storage().nbytes() / 4) - out.storage_offset();
  ob_wgrad_desc d[8] = {};
  for (int i = 0; i < count; ++i) {
    PyObject* t = PyTuple_GET_ITEM(jobs, i);
    if (!PyTuple_Check(t) || PyTuple_GET_SIZE(t) != 6) {
      PyErr_SetString(PyExc_TypeError, "store_wgrads: a job is (a, b, out_offset, ldm, ldn, n_valid)");
      throw PythonError();
    }
    Args j{&PyTuple_GET_ITEM(t, 0), 6};
    const Tensor a = j.tensor(), b = j.tensor();
    ob_wgrad_desc& p = d[i];
    p.out_offset = j.integer();
    p.ldm = j.integer();
    p.ldn = j.integer();
    p.n_valid = static_cast<int>(j.integer());
    p.a = ptr(a);
    p.b = ptr(b);
    p.seg_offsets = static_cast<const int*>(ptr(seg));
    p.lda = a.stride(0);
    p.ldb = b.stride(0);
    p.group_stride = group_stride;
    p.T = static_cast<int>(a.size(0));
    p.M = static_cast<int>(a.size(1));
    p.N = static_cast<int>(b.size(1));
    p.num_groups = static_cast<int>(groups);
    p.splits = 1;
    const long long n_lim = p.n_valid && p.n_valid < p.N ? p.n_valid : p.N;
    const long long hi = p.out_offset + (groups - 1) * group_stride + (p.M - 1) * p.ldm + (n_lim - 1) * p.ldn;
    if (a.scalar_type() != at::kBFloat16 || b.scalar_type() != at::kBFloat16 || b.size(0) != p.T || a.stride(1) != 1 || b.stride(1) != 1 ||
        p.out_offset < 0 || p.ldm < 0 || p.ldn < 0 || hi >= room) {
      PyErr_Format(PyExc_ValueError, "store_wgrads: job %d is not a pair of row-major bf16 matrices or would write element %lld of %lld", i, hi, room);
      throw PythonError();
    }
  }
  LAUNCH(ob_wgrad_clip_batch, d, count, out.data_ptr<float>(), nullptr, 0, 64, reinterpret_cast<int*>(status), g_budget, g_sms);
  Py_RETURN_NONE;
}

// ------------------------------------------------------------------------------------------------------- batches of problems
//
// The descriptions of ops.ghost_norm_batch, wgrad_clip_batch, wgrad_clip_per_example_batch and functional.rows_sum_batch_, packed here: 4 us a
// problem in Python.  Each takes the same list of problems and returns True, or False, having launched nothing, where an argument is
// not of the plain form: the Python function then says what is wrong with it, or packs it itself.

bool bf16_rows(const Tensor& t) { return t.defined() && t.scalar_type() == at::kBFloat16 && t.dim() == 2 && t.is_cuda(); }
struct Declined {};
void need(bool ok) {
  if (!ok) throw Declined();
}
Tensor tensor_or_none(PyObject* o) {
  need(o != nullptr);
  if (o == Py_None) return Tensor();
  need(THPVariable_Check(o));
  return THPVariable_Unpack(o);
}
long long whole(PyObject* o) {
  need(o != nullptr && PyLong_Check(o));
  const long long v = PyLong_AsLongLong(o);
  if (v == -1 && PyErr_Occurred()) throw PythonError();
  return v;
}
long long splits(long long tiles, long long rows, long long most, bool peer) {
  PyObject* r = PyObject_CallFunction(g_splits, "LLLi", tiles, rows, most, (int)peer);
  if (r == nullptr) throw PythonError();
  const long long v = PyLong_AsLongLong(r);
  Py_DECREF(r);
  return v;
}
struct Problems {
  PyObject* seq;
  explicit Problems(PyObject* o) : seq(o) { need(PyList_Check(o) || PyTuple_Check(o)); }
  Py_ssize_t size() const { return PySequence_Fast_GET_SIZE(seq); }
  PyObject* at(Py_ssize_t i) const { return PySequence_Fast_GET_ITEM(seq, i); }
  // item i, a tuple of `n` values
  PyObject* tuple(Py_ssize_t i, Py_ssize_t n) const {
    PyObject* t = at(i);
    need(PyTuple_Check(t) && PyTuple_GET_SIZE(t) == n);
    return t;
  }
};
Tensor field(PyObject* tuple, Py_ssize_t i) { return tensor_or_none(PyTuple_GET_ITEM(tuple, i)); }
long long room(const Tensor& out) { return static_cast<long long>(out.storage().nbytes() / 4) - out.storage_offset(); }
template <PyObject* (*F)(Args&)>
PyObject* or_false(Args& a) {
  try {
    return F(a);
  } catch (const Declined&) {
    Py_RETURN_FALSE;
  }
}

// (problems (a | None, g, norm2, tokens, ids | None, seg | None, seg_out | None), status)
PyObject* ghost_batch(Args& args) {
  const Problems ps(args.next());
  const long long status = args.integer();
  std::vector<ob_ghost_desc> d;
  for (Py_ssize_t i = 0; i < ps.size(); ++i) {
    PyObject* t = ps.tuple(i, 7);
    const Tensor a = field(t, 0), g = field(t, 1), norm2 = field(t, 2), ids = field(t, 4), seg = field(t, 5), seg_out = field(t, 6);
    const long long tokens = whole(PyTuple_GET_ITEM(t, 3));
    need(bf16_rows(g) && norm2.defined() && tokens > 0);
    ob_ghost_desc p = {};
    p.total_rows = g.size(0);
    if (seg.defined()) {
      need(seg.scalar_type() == at::kInt && (!seg_out.defined() || (seg_out.scalar_type() == at::kInt && seg_out.numel() == seg.numel() - 1)));
      p.B = static_cast<int>(seg.numel() - 1);
    } else {
      p.B = static_cast<int>(p.total_rows / tokens);
      need(p.B * tokens == p.total_rows && norm2.numel() >= p.B);
    }
    if (ids.defined()) {
      need(ids.scalar_type() == at::kInt && ids.numel() == p.total_rows);
    } else {
      need(bf16_rows(a) && a.size(0) == p.total_rows);
      p.a = ptr(a);
      p.lda = a.stride(0);
      p.Da = static_cast<int>(a.size(1));
    }
    p.g = ptr(g);
    p.ids = static_cast<const int*>(ptr(ids));
    p.norm2 = static_cast<float*>(ptr(norm2));
    p.seg = static_cast<const int*>(ptr(seg));
    p.seg_out = static_cast<const int*>(ptr(seg_out));
    p.ldg = g.stride(0);
    p.T = static_cast<int>(tokens);
    p.Dg = static_cast<int>(g.size(1));
    d.push_back(p);
  }
  std::stable_sort(d.begin(), d.end(), [](const ob_ghost_desc& x, const ob_ghost_desc& y) { return x.Da + x.Dg > y.Da + y.Dg; });
  LAUNCH(ob_ghost_norm_batch, d.data(), (int)d.size(), reinterpret_cast<int*>(status), g_budget, g_sms);
  Py_RETURN_TRUE;
}

// (problems {a, b, row_scale, seg_offsets, num_groups, out_offset, ldm, group_stride}, out | None, peer_table | None, shard_elems, status):
// accumulating, tiles of 256 columns
PyObject* wgrad_batch(Args& args) {
  const Problems ps(args.next());
  const Tensor out = args.optional(), peers = args.optional();
  const long long shard = args.integer(), status = args.integer();
  need(out.defined() ? out.scalar_type() == at::kFloat : peers.defined() && shard > 0);
  struct Job {
    double key;
    ob_wgrad_desc d;
  };
  std::vector<Job> jobs;
  long long tiles = 0;
  for (Py_ssize_t i = 0; i < ps.size(); ++i) {
    PyObject* o = ps.at(i);
    need(PyDict_Check(o));
    Tensor a, b, scale, seg;
    ob_wgrad_desc p = {};
    p.num_groups = 1;
    p.ldn = 1;
    p.accumulate = 1;
    bool pitch = false;                              // given by the caller
    PyObject *k, *v;
    Py_ssize_t pos = 0;
    while (PyDict_Next(o, &pos, &k, &v)) {
      const char* name = PyUnicode_Check(k) ? PyUnicode_AsUTF8(k) : nullptr;
      need(name != nullptr);
      if (!strcmp(name, "a")) a = tensor_or_none(v);
      else if (!strcmp(name, "b")) b = tensor_or_none(v);
      else if (!strcmp(name, "row_scale")) scale = tensor_or_none(v);
      else if (!strcmp(name, "seg_offsets")) seg = tensor_or_none(v);
      else if (!strcmp(name, "num_groups")) p.num_groups = static_cast<int>(whole(v));
      else if (!strcmp(name, "out_offset")) p.out_offset = whole(v);
      else if (!strcmp(name, "ldm")) p.ldm = whole(v), pitch = true;
      else if (!strcmp(name, "group_stride")) p.group_stride = whole(v);
      else throw Declined();
    }
    need(bf16_rows(a) && bf16_rows(b) && a.size(0) == b.size(0) && a.stride(1) == 1 && b.stride(1) == 1);
    p.a = ptr(a);
    p.b = ptr(b);
    p.row_scale = f32(scale);
    p.seg_offsets = static_cast<const int*>(ptr(seg));
    p.lda = a.stride(0);
    p.ldb = b.stride(0);
    p.T = static_cast<int>(a.size(0));
    p.M = static_cast<int>(a.size(1));
    p.N = static_cast<int>(b.size(1));
    if (!pitch) p.ldm = p.N;
    need(p.num_groups >= 1);
    if (out.defined())
      need(p.out_offset >= 0 && p.ldm >= 0 &&
           p.out_offset + (p.num_groups - 1) * p.group_stride + (p.M - 1) * p.ldm + p.N - 1 < room(out));
    tiles += static_cast<long long>(p.num_groups) * ((p.M + 127) / 128) * ((p.N + 255) / 256);
    jobs.push_back({0.0, p});
  }
  for (Job& j : jobs) {
    j.d.splits = j.d.num_groups == 1 ? static_cast<int>(splits(tiles, j.d.T, -1, peers.defined())) : 1;
    j.key = static_cast<double>(j.d.T) / (static_cast<double>(j.d.num_groups) * j.d.splits);
  }
  std::stable_sort(jobs.begin(), jobs.end(), [](const Job& x, const Job& y) { return x.key > y.key; });
  std::vector<ob_wgrad_desc> d;
  for (const Job& j : jobs) d.push_back(j.d);
  LAUNCH(ob_wgrad_clip_batch, d.data(), (int)d.size(), static_cast<float*>(ptr(out)), static_cast<float* const*>(ptr(peers)), shard, 256,
         reinterpret_cast<int*>(status), g_budget, g_sms);
  Py_RETURN_TRUE;
}

// (problems (a, b, ex_scale | None, out_offset, ldm), out | None, rows_per_example, peer_table | None, shard_elems, status)
PyObject* wgrad_pe_batch(Args& args) {
  const Problems ps(args.next());
  const Tensor out = args.optional();
  const long long rows = args.integer();
  const Tensor peers = args.optional();
  const long long shard = args.integer(), status = args.integer();
  need(rows > 0 && (out.defined() ? out.scalar_type() == at::kFloat : peers.defined() && shard > 0));
  std::vector<ob_wgrad_pe_desc> d;
  long long tiles = 0;
  for (Py_ssize_t i = 0; i < ps.size(); ++i) {
    PyObject* t = ps.tuple(i, 5);
    const Tensor a = field(t, 0), b = field(t, 1), scale = field(t, 2);
    need(bf16_rows(a) && bf16_rows(b) && a.size(0) == b.size(0) && a.stride(1) == 1 && b.stride(1) == 1 && a.size(0) % rows == 0);
    ob_wgrad_pe_desc p = {};
    p.a = ptr(a);
    p.b = ptr(b);
    p.ex_scale = f32(scale);
    p.lda = a.stride(0);
    p.ldb = b.stride(0);
    p.out_offset = whole(PyTuple_GET_ITEM(t, 3));
    p.ldm = whole(PyTuple_GET_ITEM(t, 4));
    p.num_examples = static_cast<int>(a.size(0) / rows);
    p.ex_rows = static_cast<int>(rows);
    p.M = static_cast<int>(a.size(1));
    p.N = static_cast<int>(b.size(1));
    p.accumulate = 1;
    need(!scale.defined() || (scale.scalar_type() == at::kFloat && scale.numel() >= p.num_examples && scale.is_contiguous()));
    if (out.defined()) need(p.out_offset >= 0 && p.ldm >= 0 && p.out_offset + (p.M - 1) * p.ldm + p.N - 1 < room(out));
    tiles += static_cast<long long>((p.M + 127) / 128) * ((p.N + 255) / 256);
    d.push_back(p);
  }
  for (ob_wgrad_pe_desc& p : d)
    p.splits = static_cast<int>(splits(tiles, static_cast<long long>(p.num_examples) * rows, p.num_examples, peers.defined()));
  LAUNCH(ob_wgrad_clip_pe_batch, d.data(), (int)d.size(), static_cast<float*>(ptr(out)), static_cast<float* const*>(ptr(peers)), shard,
         reinterpret_cast<int*>(status), g_budget, g_sms);
  Py_RETURN_TRUE;
}

// (jobs (out, g) or (out, g, x, mean | None, rstd, out_plain | None), examples), all of the same rows
PyObject* sums_batch(Args& args) {
  const Problems ps(args.next());
  const long long examples = args.integer();
  std::vector<ob_rowsum_desc> d;
  long long rows = -1;
  for (Py_ssize_t i = 0; i < ps.size(); ++i) {
    PyObject* t = ps.at(i);
    need(PyTuple_Check(t) && (PyTuple_GET_SIZE(t) == 2 || PyTuple_GET_SIZE(t) == 6));
    const bool norm = PyTuple_GET_SIZE(t) == 6;
    const Tensor out = field(t, 0), g = field(t, 1), x = norm ? field(t, 2) : Tensor(), mean = norm ? field(t, 3) : Tensor(),
                 rstd = norm ? field(t, 4) : Tensor(), plain = norm ? field(t, 5) : Tensor();
    need(bf16_rows(g) && (rows < 0 || g.size(0) == rows) && g.stride(1) == 1 && examples > 0 && g.size(0) % examples == 0);
    rows = g.size(0);
    for (const Tensor* o : {&out, &plain})
      need((!o->defined() && o == &plain) || (o->defined() && o->scalar_type() == at::kFloat && o->dim() == 2 && o->size(0) == examples &&
                                              o->size(1) == g.size(1) && o->stride(1) == 1));
    need(!x.defined() || (bf16_rows(x) && x.sizes() == g.sizes() && x.stride(1) == 1 && x.stride(0) == g.stride(0)));
    ob_rowsum_desc p = {};
    p.g = ptr(g);
    p.x = ptr(x);
    p.mean = f32(mean);
    p.rstd = f32(rstd);
    p.out = static_cast<float*>(ptr(out));
    p.out2 = static_cast<float*>(ptr(plain));
    p.ldg = g.stride(0);
    p.ld_out = out.stride(0);
    p.ld_out2 = plain.defined() ? plain.stride(0) : 0;
    p.N = static_cast<int>(g.size(1));
    p.mode = !x.defined() ? 0 : (mean.defined() ? 1 : 2);
    d.push_back(p);
  }
  need(!d.empty());
  LAUNCH(ob_rows_sum_batch, d.data(), (int)d.size(), (int)examples, (int)(rows / examples));
  Py_RETURN_TRUE;
}

// bind(name, address); setup(check, plan, splits, sms, budget)
PyObject* bind(Args& a) {
  const char* name = PyUnicode_AsUTF8(a.next());
  if (name == nullptr) throw PythonError();
  void* p = PyLong_AsVoidPtr(a.next());
  if (p == nullptr) throw PythonError();
#define X(entry) \
  if (!strcmp(name, #entry)) { p_##entry = reinterpret_cast<decltype(&entry)>(p); Py_RETURN_NONE; }
  OB_ENTRIES(X)
#undef X
  PyErr_Format(PyExc_KeyError, "%s", name);
  throw PythonError();
}
PyObject* setup(Args& a) {
  PyObject *check = a.next(), *plan_fn = a.next(), *splits_fn = a.next();
  const long long sms = a.integer();
  g_budget = a.number();
  g_sms = static_cast<int>(sms);
  Py_XDECREF(g_check);
  Py_XDECREF(g_plan);
  Py_XDECREF(g_splits);
  g_splits = Py_NewRef(splits_fn);
  g_check = Py_NewRef(check);
  g_plan = Py_NewRef(plan_fn);
  const char* missing = nullptr;
#define X(entry) \
  if (p_##entry == nullptr) missing = #entry;
  OB_ENTRIES(X)
#undef X
  if (missing != nullptr) {
    PyErr_Format(PyExc_RuntimeError, "%s is not bound", missing);
    throw PythonError();
  }
  Py_RETURN_NONE;
}
PyObject* entries(Args&) {
#define X(entry) #entry " "
  return PyUnicode_FromString(OB_ENTRIES(X));
#undef X
}

#define METHOD(f) {#f, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(&call<f>)), METH_FASTCALL, nullptr}
#define BATCH(f) {#f, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(&call<or_false<f>>)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {METHOD(gpt2_in), METHOD(gpt2_in_bwd), METHOD(gpt2_out), METHOD(gpt2_out_bwd), METHOD(lora_in), METHOD(lora_in_bwd),
                         METHOD(lora_out), METHOD(lora_out_bwd), METHOD(store_wgrads), BATCH(ghost_batch), BATCH(wgrad_batch),
                         BATCH(wgrad_pe_batch), BATCH(sums_batch), METHOD(bind), METHOD(setup), METHOD(entries),
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_blocks", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__blocks(void) { return PyModule_Create(&module); }
