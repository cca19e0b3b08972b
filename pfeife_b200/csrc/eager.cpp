// Eager calls of the differentiable ops, from Python's arguments to the launches and the autograd node,
// as a Python module (`pfeife_b200_eager`).
//
// What bounds a small call is the host: through Python an op took the caller 20 to 30 us forward and as
// much again backward, where autograd's thread also has to wait for the interpreter lock.  Here it takes
// a few: linear 6.1 us, MLP 9.8, LayerNorm with residual 6.1, attention 5.4.  (As a caller sees them, forward
// and backward of a LayerNorm with residual 160 -> 81 us, what is left being autograd's hop to its thread
// and back; logits of 4 images by ViT-Tiny 2540 -> 753 us.)
//
// Only the usual call is taken: plain CUDA tensors of one device and one 16-bit type, no autocast, nothing
// that observes ops (dispatch or function modes, transforms, traces, forward-mode gradients).  For every
// other call the functions return None, and the caller goes on in Python (ops/functional.py), which
// defines what each op means.  A backward whose tensors are not plain any more, or that is itself
// recorded, calls the registered backward op through the dispatcher, as the Python formulas do.  So does
// one that unpacks something in another order or type than the forward saved: hooks on saved tensors may
// return any tensor, and what the kernels assume of their operands is tested again in each backward.
//
// The kernel library is loaded by the caller beforehand with its symbols global.
#include <ATen/autocast_mode.h>
#include <ATen/core/PythonFallbackKernel.h>
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/EmptyTensor.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/autograd/variable.h>
#include <torch/csrc/jit/frontend/tracer.h>

#include <atomic>

#include "api.h"

namespace pfeife {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

// ------------------------------------------------------------------------------ launching
struct Failed { int code; const char* what; };      // an entry point refused the call
std::atomic<long long> g_launches{0};
PyObject* g_status_word = nullptr;                  // kernels.status_word
PyObject* g_check = nullptr;                        // _lib.check: raises for a code
constexpr int MAX_DEVICES = 64;
Tensor g_status[MAX_DEVICES];                       // kept: the buffer lives as long as the process

void ok(int code, const char* what) {
  if (code) throw Failed{code, what};
  g_launches.fetch_add(1, std::memory_order_relaxed);
}

// Called with the interpreter lock in forwards, which come before any backward on a device.
bool learn_status(int dev) {
  if (g_status[dev].defined()) return true;
  PyObject* d = THPDevice_New(at::Device(at::kCUDA, dev));
  PyObject* t = d ? PyObject_CallOneArg(g_status_word, d) : nullptr;
  Py_XDECREF(d);
  if (!t) return false;
  g_status[dev] = THPVariable_Unpack(t);
  Py_DECREF(t);
  return true;
}

struct Env {
  int dev, sms;
  int* status;
  void* stream;
  explicit Env(const Tensor& t) : dev(t.get_device()) {
    if (const int code = pf_bind_device(dev)) throw Failed{code, "pf_bind_device"};
    sms = at::cuda::getDeviceProperties(dev)->multiProcessorCount;
    status = static_cast<int*>(g_status[dev].data_ptr());
    stream = at::cuda::getCurrentCUDAStream(dev).stream();
  }
};

int code_of(at::ScalarType t) { return t == at::kFloat ? 0 : t == at::kHalf ? 1 : 2; }
int code_of(const Tensor& t) { return code_of(t.scalar_type()); }
const void* at_or_null(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }
bool aligned(const Tensor& t) { return (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15) == 0; }
// packed values are read 16 bytes at a time; others are packed into memory of their own first
template <typename... T>
bool on_vectors(const T&... t) {
  return ((!t.defined() || !t.is_contiguous() || aligned(t)) && ...);
}
bool half(const Tensor& t) { return t.scalar_type() == at::kHalf || t.scalar_type() == at::kBFloat16; }

Tensor empty(at::IntArrayRef sizes, at::ScalarType type, const Tensor& like) {
  return Tensor(at::detail::empty_cuda(sizes, type, like.device(), std::nullopt));
}
Tensor empty(at::IntArrayRef sizes, const Tensor& like) { return empty(sizes, like.scalar_type(), like); }
Tensor floats(long long n, const Tensor& like) { return empty({n}, at::kFloat, like); }

// ------------------------------------------------------------------------------ which calls are taken
bool unobserved() {
  return !c10::impl::TorchDispatchModeTLS::any_modes_set() && !at::impl::torch_function_mode_enabled() &&
         !c10::impl::tls_is_dispatch_key_included(at::DispatchKey::FuncTorchDynamicLayerFrontMode) &&
         !torch::jit::tracer::isTracing();
}

// A tensor whose memory holds its values: no wrapper, negative view or the like (each is a dispatch key),
// no forward-mode gradient, and not empty.  The usual keys are those of a tensor made outside inference mode,
// in which tensors lack some of them, whatever the mode of the first call.
bool plain(const Tensor& t, int dev) {
  static const uint64_t usual = [] {
    const c10::InferenceMode off(false);
    return at::empty({0}, at::device(at::kCUDA).dtype(at::kHalf)).key_set().raw_repr();
  }();
  return (t.key_set().raw_repr() & ~usual) == 0 && t.get_device() == dev && t.data_ptr() != nullptr &&
         !t._fw_grad(0).defined();
}
template <typename... T>
bool all_plain(const Tensor& first, const T&... more) {
  const int dev = first.get_device();
  return plain(first, dev) && ((!more.defined() || plain(more, dev)) && ...);
}

template <typename... T>
bool recorded(const T&... t) {
  return at::GradMode::is_enabled() && ((t.defined() && t.requires_grad()) || ...) &&
         !c10::impl::tls_is_dispatch_key_excluded(at::DispatchKey::AutogradOther);
}

// Whether a backward may launch kernels itself.
template <typename... T>
bool direct(const Tensor& first, const T&... more) {
  return !at::GradMode::is_enabled() && unobserved() && all_plain(first, more...);
}

// fp32 values one after the other, as a forward kernel wrote them or as a caller's parameters are taken
bool packed_floats(const Tensor& t, int64_t n) {
  return t.scalar_type() == at::kFloat && t.numel() == n && t.is_contiguous();
}
// values of the type and sizes of `like`
bool matches(const Tensor& t, const Tensor& like) {
  return t.scalar_type() == like.scalar_type() && t.sizes() == like.sizes();
}

c10::IValue opt(const Tensor& t) { return t.defined() ? c10::IValue(t) : c10::IValue(); }

// A registered op through the dispatcher.
torch::jit::Stack dispatched(const char* name, torch::jit::Stack stack) {
  c10::Dispatcher::singleton().findSchemaOrThrow(name, "").callBoxed(stack);
  return stack;
}
Tensor given(const c10::IValue& v) {                // an empty tensor stands for "not needed"
  const Tensor& t = v.toTensor();
  return t.numel() ? t : Tensor();
}
Tensor as(const Tensor& t, const c10::IValue& saved) {       // in the type that a forward took down
  const auto type = static_cast<at::ScalarType>(saved.toInt());
  return !t.defined() || t.scalar_type() == type ? t : t.to(type);
}

// Tensors that a call may leave out reach a node as optionals, which count as inputs only when given.
using Maybe = std::optional<Tensor>;
Maybe maybe(const Tensor& t) { return t.defined() ? Maybe(t) : std::nullopt; }
Tensor value(const Maybe& t) { return t ? *t : Tensor(); }

// Runs the launches of a backward below autograd; a refused call raises what it raises in Python.
template <typename F>
auto below(F&& f) {
  try {
    at::AutoDispatchBelowADInplaceOrView guard;
    return f();
  } catch (const Failed& e) {
    pybind11::gil_scoped_acquire lock;
    PyObject* r = PyObject_CallFunction(g_check, "is", e.code, e.what);
    Py_XDECREF(r);
    python_error raised;
    raised.persist();
    throw raised;
  }
}

// ------------------------------------------------------------------------------ GEMM
enum Epi { NONE, GELU, DGELU, GELU_TANH, DGELU_TANH, SILU };          // gemm_sm100.cu
constexpr int EPI_OF_ACT[4] = {NONE, GELU, GELU_TANH, SILU};

// x as rows the TMA can read
Tensor rows(const Tensor& x) {
  Tensor r = x.dim() == 2 ? x : x.reshape({-1, x.size(-1)});
  if (r.stride(1) != 1 || r.stride(0) % 8 || !aligned(r)) r = r.contiguous();
  return r;
}
bool readable(const Tensor& m) {
  return m.dim() == 2 && m.stride(1) == 1 && m.stride(0) % 8 == 0 && aligned(m);
}
// all operands of 16 bits, as is the result
Tensor gemm(const Env& e, const Tensor& a, const Tensor& b, bool a_mn, bool b_mn, const Tensor& bias = {},
            const Tensor& residual = {}, const Tensor& aux = {}, int epi = NONE) {
  const long long M = a.size(a_mn), K = a.size(!a_mn), N = b.size(b_mn);
  Tensor out = empty({M, N}, a);
  ok(pf_gemm(a.data_ptr(), b.data_ptr(), out.data_ptr(), (int)M, (int)N, (int)K, a.stride(0), b.stride(0), N,
             a_mn, b_mn, code_of(a), code_of(a), at_or_null(bias), bias.defined() ? code_of(bias) : 0,
             at_or_null(residual), residual.defined() ? residual.stride(0) : 0,
             const_cast<void*>(at_or_null(aux)), aux.defined() ? aux.stride(0) : 0, epi, 0, 1.0f, e.status,
             e.sms, 0, nullptr, 0, e.stream),
     "pf_gemm");
  return out;
}
Tensor colsum(const Env& e, const Tensor& x) {
  Tensor out = at::zeros({x.size(1)}, x.options().dtype(at::kFloat));
  ok(pf_colsum(x.data_ptr(), out.data_ptr(), x.size(0), (int)x.size(1), x.stride(0), code_of(x), e.sms,
               e.stream),
     "pf_colsum");
  return out;
}

std::vector<int64_t> with_last(const Tensor& x, int64_t n) {
  auto s = x.sizes().vec();
  s.back() = n;
  return s;
}

// ------------------------------------------------------------------------------ linear
bool bias_fits(const Tensor& b, int64_t n) { return !b.defined() || (b.dim() == 1 && b.size(0) == n && b.is_contiguous() && (half(b) || b.scalar_type() == at::kFloat)); }
bool layer_fits(const Tensor& x, const Tensor& w, const Tensor& b) {
  return x.dim() >= 2 && half(x) && w.scalar_type() == x.scalar_type() && readable(w) &&
         w.size(1) == x.size(-1) && w.size(1) % 8 == 0 && bias_fits(b, w.size(0)) &&
         x.numel() / x.size(-1) < (1ll << 31) && w.size(0) < (1ll << 31);
}
bool residual_fits(const Tensor& r, const Tensor& x, int64_t n) {
  return !r.defined() || (r.scalar_type() == x.scalar_type() && r.dim() == x.dim() && r.size(-1) == n &&
                          r.numel() / n == x.numel() / x.size(-1));
}

std::pair<Tensor, Tensor> linear_forward(const Tensor& x, const Tensor& w, const Tensor& b, const Tensor& res,
                                         int act) {
  const Env e(x);
  const Tensor x2 = rows(x), r2 = res.defined() ? rows(res) : Tensor();
  const Tensor aux = act ? empty({x2.size(0), w.size(0)}, x) : Tensor();
  const Tensor y = gemm(e, x2, w, false, false, b, r2, aux, EPI_OF_ACT[act]);
  const auto shape = with_last(x, w.size(0));
  return {y.view(shape), act ? aux.view(shape) : aux};
}
// whether linear_gradients can read what a backward unpacked, beside a gradient of the output
bool gradients_fit(const Tensor& dz, const Tensor& x, const Tensor& w) {
  return layer_fits(x, w, {}) && x.scalar_type() == dz.scalar_type() && dz.size(-1) == w.size(0) &&
         x.numel() / x.size(-1) == dz.numel() / dz.size(-1);
}
// gradients of x, w, b from that of the pre-activation
void linear_gradients(const Env& e, const Tensor& dz2, const Tensor& x, const Tensor& w, bool need_dx,
                      bool need_dw, bool need_db, Tensor& dx, Tensor& dw, Tensor& db) {
  if (need_dx) dx = gemm(e, dz2, w, false, true).view(x.sizes());
  if (need_dw) dw = gemm(e, dz2, rows(x), true, true);
  if (need_db) db = colsum(e, dz2);
}

struct DirectLinear : torch::autograd::Function<DirectLinear> {
  static Tensor forward(AutogradContext* ctx, Tensor x, Tensor w, Maybe bias, Maybe residual, int64_t act) {
    at::AutoDispatchBelowADInplaceOrView guard;
    const Tensor b = value(bias), res = value(residual);
    auto [y, aux] = linear_forward(x, w, b, res, (int)act);
    ctx->set_materialize_grads(false);
    ctx->save_for_backward({x, w, b, aux});
    ctx->saved_data["act"] = act;
    if (bias) ctx->saved_data["type"] = (int64_t)b.scalar_type();
    ctx->saved_data["res"] = res.defined();
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto s = ctx->get_saved_variables();
    const Tensor &x = s[0], &w = s[1], &b = s[2], &aux = s[3];
    if (!grads[0].defined()) return variable_list(5);
    const Tensor dy = grads[0].contiguous();
    const int act = (int)ctx->saved_data["act"].toInt();
    const bool nx = ctx->needs_input_grad(0), nw = ctx->needs_input_grad(1),
               nb = b.defined() && ctx->needs_input_grad(2),
               nr = ctx->saved_data["res"].toBool() && ctx->needs_input_grad(2 + b.defined());
    Tensor dx, dw, db;
    if (direct(dy, x, w, b, aux) && gradients_fit(dy, x, w) && (!act || matches(aux, dy))) {
      below([&] {
        const Env e(dy);
        Tensor dz = rows(dy);
        if (act) {
          constexpr int DACT[4] = {0, 10, 11, 12};                    // elementwise.cu
          const Tensor z = rows(aux).contiguous();
          Tensor out = empty(dz.sizes(), dz);
          dz = dz.contiguous();
          ok(pf_elementwise(dz.data_ptr(), z.data_ptr(), out.data_ptr(), dz.numel(), DACT[act], code_of(dz),
                            e.sms, e.stream),
             "pf_elementwise");
          dz = out;
        }
        linear_gradients(e, dz, x, w, nx, nw, nb, dx, dw, db);
        return 0;
      });
    } else {
      auto out = dispatched("pfeife::linear_bwd", {dy, x, w, aux.defined() ? aux : dy.new_empty({0}),
                                                   (int64_t)act, nx, nw, nb, opt(b)});
      dx = given(out[0]); dw = given(out[1]); db = given(out[2]);
    }
    return {nx ? dx : Tensor(), nw ? dw : Tensor(), nb ? as(db, ctx->saved_data["type"]) : Tensor(),
            nr ? dy : Tensor(), Tensor()};
  }
};

// ------------------------------------------------------------------------------ feed-forward block
struct DirectMlp : torch::autograd::Function<DirectMlp> {
  static Tensor forward(AutogradContext* ctx, Tensor x, Tensor w1, Maybe bias1, Tensor w2, Maybe bias2,
                        Maybe residual, int64_t act) {
    at::AutoDispatchBelowADInplaceOrView guard;
    const Tensor b1 = value(bias1), b2 = value(bias2), res = value(residual);
    auto [a1, z1] = linear_forward(x, w1, b1, {}, (int)act);
    const Tensor y = linear_forward(a1, w2, b2, res, 0).first;
    ctx->set_materialize_grads(false);
    ctx->save_for_backward({x, w1, w2, z1, a1, b1, b2});
    ctx->saved_data["act"] = act;
    if (bias1) ctx->saved_data["type1"] = (int64_t)b1.scalar_type();
    if (bias2) ctx->saved_data["type2"] = (int64_t)b2.scalar_type();
    ctx->saved_data["res"] = res.defined();
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto s = ctx->get_saved_variables();
    const Tensor &x = s[0], &w1 = s[1], &w2 = s[2], &z1 = s[3], &a1 = s[4], &b1 = s[5], &b2 = s[6];
    if (!grads[0].defined()) return variable_list(7);
    const Tensor dy = grads[0].contiguous();
    const int act = (int)ctx->saved_data["act"].toInt();
    const bool nx = ctx->needs_input_grad(0),
               nr = ctx->saved_data["res"].toBool() &&
                    ctx->needs_input_grad(3 + b1.defined() + b2.defined());
    Tensor dx, dw1, db1, dw2, db2, none;
    if (direct(dy, x, w1, w2, z1, a1, b1, b2) && gradients_fit(dy, a1, w2) && gradients_fit(a1, x, w1) &&
        matches(z1, a1)) {
      below([&] {
        const Env e(dy);
        const Tensor dy2 = rows(dy);
        const Tensor dz1 = gemm(e, dy2, w2, false, true, {}, {}, rows(z1), act == 1 ? DGELU : DGELU_TANH);
        linear_gradients(e, dy2, a1, w2, false, true, b2.defined(), none, dw2, db2);
        linear_gradients(e, dz1, x, w1, nx, true, b1.defined(), dx, dw1, db1);
        return 0;
      });
    } else {
      auto out = dispatched("pfeife::mlp_bwd", {dy, x, w1, w2, z1, a1, (int64_t)act, nx, b1.defined(),
                                                b2.defined(), opt(b1), opt(b2)});
      dx = given(out[0]); dw1 = given(out[1]); db1 = given(out[2]); dw2 = given(out[3]); db2 = given(out[4]);
    }
    return {nx ? dx : Tensor(), dw1, b1.defined() ? as(db1, ctx->saved_data["type1"]) : Tensor(), dw2,
            b2.defined() ? as(db2, ctx->saved_data["type2"]) : Tensor(), nr ? dy : Tensor(), Tensor()};
  }
};

// ------------------------------------------------------------------------------ norms
struct NormOut { Tensor y, h, mean, rstd; };
NormOut norm_forward(const Tensor& x, const Tensor& gamma, const Tensor& beta, const Tensor& res, double eps,
                     bool rms) {
  const Env e(x);
  const Tensor xc = x.contiguous(), rc = res.defined() ? res.contiguous() : res;
  const int64_t N = x.size(-1), n = x.numel() / N;
  NormOut o;
  o.y = empty(x.sizes(), x);
  if (res.defined()) o.h = empty(x.sizes(), x);
  o.mean = floats(n, x);
  o.rstd = floats(n, x);
  ok(pf_norm_fwd(xc.data_ptr(), at_or_null(rc), gamma.data_ptr(), at_or_null(beta), o.y.data_ptr(),
                 const_cast<void*>(at_or_null(o.h)), o.mean.data_ptr(), o.rstd.data_ptr(), n, (int)N, (float)eps,
                 rms, code_of(x), e.stream),
     "pf_norm_fwd");
  return o;
}

struct DirectNorm : torch::autograd::Function<DirectNorm> {
  static variable_list forward(AutogradContext* ctx, Tensor x, Tensor gamma, Maybe bias, Maybe residual,
                               double eps, bool rms) {
    at::AutoDispatchBelowADInplaceOrView guard;
    const Tensor beta = value(bias), res = value(residual);
    const NormOut o = norm_forward(x, gamma, beta, res, eps, rms);
    ctx->set_materialize_grads(false);
    ctx->save_for_backward({res.defined() ? o.h : x, gamma, beta, o.mean, o.rstd});
    ctx->saved_data["rms"] = rms;
    ctx->saved_data["res"] = res.defined();
    if (res.defined()) return {o.y, o.h};
    return {o.y};
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto s = ctx->get_saved_variables();
    const Tensor &h = s[0], &gamma = s[1], &beta = s[2], &mean = s[3], &rstd = s[4];
    const bool rms = ctx->saved_data["rms"].toBool(), has_res = ctx->saved_data["res"].toBool();
    Tensor dh, dy = grads[0];
    if (has_res && grads[1].defined()) dh = grads[1].contiguous();
    if (!dy.defined()) {
      if (!dh.defined()) return variable_list(6);
      dy = at::zeros_like(h);
    }
    dy = dy.contiguous();
    const int64_t n = h.numel() / h.size(-1);
    Tensor dx, dg, db;
    if (direct(dy, dh, h, gamma, beta, mean, rstd) && half(h) && matches(h, dy) &&
        (!dh.defined() || matches(dh, dy)) && on_vectors(dy, dh, h, gamma) && packed_floats(gamma, h.size(-1)) && packed_floats(mean, n) &&
        packed_floats(rstd, n)) {
      below([&] {
        const Env e(dy);
        const Tensor hc = h.contiguous();
        const int64_t N = h.size(-1);
        dx = empty(h.sizes(), h);
        dg = floats(N, h);
        if (beta.defined() && !rms) db = floats(N, h);
        const Tensor scratch = floats((int64_t)pf_norm_bwd_ctas(n, e.sms) * 2 * N, h);
        ok(pf_norm_bwd(dy.data_ptr(), hc.data_ptr(), gamma.data_ptr(), mean.data_ptr(), rstd.data_ptr(),
                       at_or_null(dh), dx.data_ptr(), dg.data_ptr(), const_cast<void*>(at_or_null(db)),
                       scratch.data_ptr(), n, (int)N, rms, 0, code_of(h), e.sms, e.stream),
           "pf_norm_bwd");
        return 0;
      });
    } else {
      auto out = dispatched("pfeife::norm_bwd",
                            {dy, opt(dh), h, gamma, mean, rstd, rms, beta.defined(), opt(beta)});
      dx = out[0].toTensor(); dg = given(out[1]); db = given(out[2]);
    }
    return {dx, dg, beta.defined() ? db : Tensor(), has_res ? dx : Tensor(), Tensor(), Tensor()};
  }
};

// ------------------------------------------------------------------------------ attention
struct View { const char* at; long long strides[3]; };                // of q, k or v: batch, seq, head
View view_of(const Tensor& t) {
  return {static_cast<const char*>(t.data_ptr()), {t.stride(0), t.stride(1), t.stride(2)}};
}
View slice_of(const Tensor& qkv, int i) {
  return {static_cast<const char*>(qkv.data_ptr()) + i * qkv.stride(2) * 2,
          {qkv.stride(0), qkv.stride(1), qkv.stride(3)}};
}
Tensor readable_heads(const Tensor& t) {
  const bool fits = t.stride(3) == 1 && aligned(t) && t.stride(0) % 8 == 0 && t.stride(1) % 8 == 0 &&
                    t.stride(2) % 8 == 0;
  return fits ? t : t.contiguous();
}

std::pair<Tensor, Tensor> attention_forward(const Tensor& like, const View& q, const View& k, const View& v,
                                            int64_t B, int64_t Sq, int64_t Sk, int64_t H, int64_t D,
                                            bool causal, double scale) {
  const Env e(like);
  const Tensor o = empty({B, Sq, H, D}, like), lse = empty({B, H, Sq}, at::kFloat, like);
  ok(pf_attn_fwd(q.at, k.at, v.at, o.data_ptr(), lse.data_ptr(), (int)B, (int)H, (int)Sq, (int)Sk, (int)D,
                 q.strides, k.strides, v.strides, causal, (float)scale, code_of(like), e.status, e.stream),
     "pf_attn_fwd");
  return {o, lse};
}
// gradients to views of equal strides for k and v
void attention_backward(const Tensor& dout, const View& q, const View& k, const View& v, const Tensor& o,
                        const Tensor& lse, const View& dq, const View& dk, const View& dv, int64_t Sk,
                        bool causal, double scale) {
  const Env e(dout);
  const int B = (int)o.size(0), Sq = (int)o.size(1), H = (int)o.size(2), D = (int)o.size(3);
  const Tensor stats = floats((int64_t)B * H * ((Sq + 127) / 128) * 256, dout);
  const int kib = pf_attn_bwd_scratch(B, H, Sq, (int)Sk, D, causal);
  const Tensor scratch = kib ? floats(kib * 256ll, dout) : Tensor();
  ok(pf_attn_bwd(dout.data_ptr(), q.at, k.at, v.at, o.data_ptr(), lse.data_ptr(), stats.data_ptr(),
                 const_cast<void*>(at_or_null(scratch)), const_cast<char*>(dq.at), const_cast<char*>(dk.at),
                 const_cast<char*>(dv.at), B, H, Sq, (int)Sk, D, q.strides, k.strides, v.strides, dq.strides,
                 dk.strides, causal, (float)scale, code_of(dout), e.status, e.sms, e.stream),
     "pf_attn_bwd");
}

std::pair<Tensor, Tensor> heads_forward(const Tensor& q, const Tensor& k, const Tensor& v, bool causal,
                                        double scale) {
  const Tensor qr = readable_heads(q), kr = readable_heads(k), vr = readable_heads(v);
  return attention_forward(q, view_of(qr), view_of(kr), view_of(vr), q.size(0), q.size(1), k.size(1),
                           q.size(2), q.size(3), causal, scale);
}

// whether a backward can read what it unpacked, beside a gradient of the output
bool heads_fit(const Tensor& dout, const Tensor& o, const Tensor& lse) {
  return half(dout) && matches(o, dout) && on_vectors(o) &&
         packed_floats(lse, dout.size(0) * dout.size(1) * dout.size(2));
}

struct DirectAttention : torch::autograd::Function<DirectAttention> {
  static Tensor forward(AutogradContext* ctx, Tensor q, Tensor k, Tensor v, bool causal, double scale) {
    at::AutoDispatchBelowADInplaceOrView guard;
    auto [o, lse] = heads_forward(q, k, v, causal, scale);
    ctx->set_materialize_grads(false);
    ctx->save_for_backward({q, k, v, o, lse});
    ctx->saved_data["causal"] = causal;
    ctx->saved_data["scale"] = scale;
    return o;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto s = ctx->get_saved_variables();
    const Tensor &q = s[0], &k = s[1], &v = s[2], &o = s[3], &lse = s[4];
    if (!grads[0].defined()) return variable_list(5);
    const Tensor dout = grads[0].contiguous();
    const bool causal = ctx->saved_data["causal"].toBool();
    const double scale = ctx->saved_data["scale"].toDouble();
    Tensor dq, dk, dv;
    if (direct(dout, q, k, v, o, lse) && heads_fit(dout, o, lse) && matches(q, dout) &&
        matches(k, v) && k.scalar_type() == q.scalar_type()) {
      below([&] {
        const Tensor qr = readable_heads(q), kr = readable_heads(k), vr = readable_heads(v);
        dq = empty(q.sizes(), q);
        dk = empty(k.sizes(), k);
        dv = empty(v.sizes(), v);
        attention_backward(aligned(dout) ? dout : dout.clone(), view_of(qr), view_of(kr), view_of(vr),
                           o.contiguous(), lse, view_of(dq), view_of(dk), view_of(dv), k.size(1), causal,
                           scale);
        return 0;
      });
    } else {
      auto out = dispatched("pfeife::attn_bwd", {dout, q, k, v, o, lse, causal, scale});
      dq = out[0].toTensor(); dk = out[1].toTensor(); dv = out[2].toTensor();
    }
    return {dq, dk, dv, Tensor(), Tensor()};
  }
};

bool packed_fits(const Tensor& t) {                  // [B, S, 3, H, D], read in place
  return t.stride(4) == 1 && aligned(t) && t.stride(0) % 8 == 0 && t.stride(1) % 8 == 0 &&
         t.stride(2) % 8 == 0 && t.stride(3) % 8 == 0;
}
std::pair<Tensor, Tensor> packed_forward(const Tensor& t, bool causal, double scale) {
  return attention_forward(t, slice_of(t, 0), slice_of(t, 1), slice_of(t, 2), t.size(0), t.size(1), t.size(1),
                           t.size(3), t.size(4), causal, scale);
}

struct DirectAttentionQkv : torch::autograd::Function<DirectAttentionQkv> {
  static Tensor forward(AutogradContext* ctx, Tensor qkv, bool causal, double scale) {
    at::AutoDispatchBelowADInplaceOrView guard;
    auto [o, lse] = packed_forward(qkv, causal, scale);
    ctx->set_materialize_grads(false);
    ctx->save_for_backward({qkv, o, lse});
    ctx->saved_data["causal"] = causal;
    ctx->saved_data["scale"] = scale;
    return o;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto s = ctx->get_saved_variables();
    const Tensor &qkv = s[0], &o = s[1], &lse = s[2];
    if (!grads[0].defined()) return variable_list(3);
    const Tensor dout = grads[0].contiguous();
    const bool causal = ctx->saved_data["causal"].toBool();
    const double scale = ctx->saved_data["scale"].toDouble();
    Tensor d;
    if (direct(dout, qkv, o, lse) && heads_fit(dout, o, lse) && qkv.scalar_type() == dout.scalar_type() &&
        qkv.dim() == 5 && qkv.numel() == 3 * dout.numel() && packed_fits(qkv)) {
      below([&] {
        d = empty(qkv.sizes(), qkv);
        attention_backward(aligned(dout) ? dout : dout.clone(), slice_of(qkv, 0), slice_of(qkv, 1),
                           slice_of(qkv, 2), o.contiguous(), lse, slice_of(d, 0), slice_of(d, 1),
                           slice_of(d, 2), qkv.size(1), causal, scale);
        return 0;
      });
    } else {
      d = dispatched("pfeife::attn_qkv_bwd", {dout, qkv, o, lse, causal, scale})[0].toTensor();
    }
    return {d, Tensor(), Tensor()};
  }
};

// ------------------------------------------------------------------------------ rotary embedding, GLU
Tensor rope_forward(const Tensor& x, const Tensor& cos, const Tensor& sin, bool inverse) {
  const Env e(x);
  const Tensor out = empty(x.sizes(), x);
  ok(pf_rope_qkv(x.data_ptr(), out.data_ptr(), cos.data_ptr(), sin.data_ptr(), x.size(0) * x.size(1),
                 (int)x.size(1), (int)x.size(3), (int)x.size(4), inverse, code_of(x), e.stream),
     "pf_rope_qkv");
  return out;
}
bool table_fits(const Tensor& t, const Tensor& x) {  // of cosines or sines, for x [B, S, 3, H, D]
  return t.scalar_type() == at::kFloat && t.dim() == 2 && t.is_contiguous() && aligned(t) &&
         t.size(0) >= x.size(1) && t.size(1) == x.size(4) / 2;
}
struct DirectRopeQkv : torch::autograd::Function<DirectRopeQkv> {
  static Tensor forward(AutogradContext* ctx, Tensor x, Tensor cos, Tensor sin) {
    at::AutoDispatchBelowADInplaceOrView guard;
    ctx->save_for_backward({cos, sin});
    return rope_forward(x, cos, sin, false);
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto s = ctx->get_saved_variables();
    const Tensor &cos = s[0], &sin = s[1];
    const Tensor dy = grads[0].contiguous();
    Tensor dx;
    if (direct(dy, cos, sin) && half(dy) && aligned(dy) && table_fits(cos, dy) && table_fits(sin, dy))
      below([&] { dx = rope_forward(dy, cos, sin, true); return 0; });
    else dx = dispatched("pfeife::rope_qkv_apply", {dy, cos, sin, true})[0].toTensor();
    return {dx, Tensor(), Tensor()};
  }
};

Tensor glu_forward(const Tensor& gu, bool gelu) {
  const Env e(gu);
  const int64_t H = gu.size(-1) / 2;
  const Tensor out = empty(with_last(gu, H), gu);
  ok(pf_glu_fwd(gu.data_ptr(), out.data_ptr(), gu.numel() / (2 * H), (int)H, gelu, code_of(gu), e.sms,
                e.stream),
     "pf_glu_fwd");
  return out;
}
struct DirectGlu : torch::autograd::Function<DirectGlu> {
  static Tensor forward(AutogradContext* ctx, Tensor gu, bool gelu) {
    at::AutoDispatchBelowADInplaceOrView guard;
    ctx->save_for_backward({gu});
    ctx->saved_data["gelu"] = gelu;
    return glu_forward(gu, gelu);
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const Tensor gu = ctx->get_saved_variables()[0];
    const Tensor dy = grads[0].contiguous();
    const bool gelu = ctx->saved_data["gelu"].toBool();
    Tensor d;
    if (direct(dy, gu) && gu.is_contiguous() && half(gu) && gu.scalar_type() == dy.scalar_type() &&
        gu.numel() == 2 * dy.numel() && on_vectors(gu, dy)) {
      below([&] {
        const Env e(dy);
        const int64_t H = gu.size(-1) / 2;
        d = empty(gu.sizes(), gu);
        ok(pf_glu_bwd(gu.data_ptr(), dy.data_ptr(), d.data_ptr(), gu.numel() / (2 * H), (int)H, gelu,
                      code_of(gu), e.sms, e.stream),
           "pf_glu_bwd");
        return 0;
      });
    } else {
      d = dispatched("pfeife::glu_bwd", {dy, gu, gelu})[0].toTensor();
    }
    return {d, Tensor()};
  }
};

// ------------------------------------------------------------------------------ mean cross entropy
struct LossOut { Tensor mean, lse, inv; };
LossOut loss_forward(const Tensor& logits, const Tensor& target, int64_t ignore) {
  const Env e(logits);
  const Tensor lc = logits.contiguous(), tc = target.contiguous();
  const int64_t n = lc.size(0), V = lc.size(1);
  const Tensor loss = floats(n, lc);
  LossOut o{empty({}, at::kFloat, lc), floats(n, lc), empty({}, at::kFloat, lc)};
  ok(pf_ce_fwd(lc.data_ptr(), tc.data_ptr(), loss.data_ptr(), o.lse.data_ptr(), n, (int)V, V, ignore,
               code_of(lc), e.sms, e.stream),
     "pf_ce_fwd");
  const int parts = pf_ce_mean_parts(n, e.sms);
  const Tensor scratch = parts > 1 ? floats(2 * parts, lc) : Tensor();
  ok(pf_ce_mean(loss.data_ptr(), tc.data_ptr(), const_cast<void*>(at_or_null(scratch)), o.mean.data_ptr(),
                o.inv.data_ptr(), n, ignore, e.sms, e.stream),
     "pf_ce_mean");
  return o;
}
struct DirectCrossEntropy : torch::autograd::Function<DirectCrossEntropy> {
  static Tensor forward(AutogradContext* ctx, Tensor logits, Tensor target, int64_t ignore) {
    at::AutoDispatchBelowADInplaceOrView guard;
    const LossOut o = loss_forward(logits, target, ignore);
    ctx->set_materialize_grads(false);
    ctx->save_for_backward({logits, target, o.lse, o.inv});
    ctx->saved_data["ignore"] = ignore;
    return o.mean;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto s = ctx->get_saved_variables();
    const Tensor &logits = s[0], &target = s[1], &lse = s[2], &inv = s[3];
    const Tensor& g = grads[0];
    if (!g.defined()) return variable_list(3);
    const int64_t ignore = ctx->saved_data["ignore"].toInt();
    const Tensor scale = g * inv;
    Tensor d;
    if (direct(scale, logits, target, lse) && logits.dim() == 2 &&
        (half(logits) || logits.scalar_type() == at::kFloat) && target.scalar_type() == at::kLong &&
        target.numel() == logits.size(0) && packed_floats(lse, logits.size(0)) && packed_floats(scale, 1)) {
      below([&] {
        const Env e(scale);
        const Tensor lc = logits.contiguous(), tc = target.contiguous();
        d = empty(lc.sizes(), lc);
        ok(pf_ce_bwd(lc.data_ptr(), tc.data_ptr(), lse.data_ptr(), scale.data_ptr(), d.data_ptr(), lc.size(0),
                     (int)lc.size(1), lc.size(1), ignore, 0, code_of(lc), e.sms, e.stream),
           "pf_ce_bwd");
        return 0;
      });
    } else {
      d = dispatched("pfeife::ce_bwd", {scale.expand({logits.size(0)}), logits, target, lse, ignore})[0]
              .toTensor();
    }
    return {d, Tensor(), Tensor()};
  }
};

// ------------------------------------------------------------------------------ GroupNorm
Tensor group_scratch(const Env& e, const Tensor& x, int64_t width) {
  const int64_t B = x.size(0), C = x.size(3), HW = x.size(1) * x.size(2);
  return floats(B * pf_groupnorm_slabs((int)B, (int)HW, (int)C, e.sms) * 2 * width, x);
}
NormOut group_norm_forward(const Tensor& x, const Tensor& gamma, const Tensor& beta, int64_t groups, double eps,
                           bool silu) {
  const Env e(x);
  const Tensor xc = x.contiguous();
  const int64_t B = x.size(0), C = x.size(3), HW = x.size(1) * x.size(2);
  NormOut o{empty(x.sizes(), x), {}, floats(B * groups, x), floats(B * groups, x)};
  const Tensor scratch = group_scratch(e, x, groups);
  ok(pf_groupnorm_fwd(xc.data_ptr(), gamma.data_ptr(), beta.data_ptr(), o.y.data_ptr(), o.mean.data_ptr(),
                      o.rstd.data_ptr(), scratch.data_ptr(), (int)B, (int)HW, (int)C, (int)groups, (float)eps,
                      silu, code_of(x), e.sms, e.stream),
     "pf_groupnorm_fwd");
  return o;
}
struct DirectGroupNorm : torch::autograd::Function<DirectGroupNorm> {
  static Tensor forward(AutogradContext* ctx, Tensor x, Tensor gamma, Tensor beta, int64_t groups, double eps,
                        bool silu) {
    at::AutoDispatchBelowADInplaceOrView guard;
    const NormOut o = group_norm_forward(x, gamma, beta, groups, eps, silu);
    ctx->set_materialize_grads(false);
    ctx->save_for_backward({x, o.mean, o.rstd, gamma, beta});
    ctx->saved_data["groups"] = groups;
    ctx->saved_data["silu"] = silu;
    return o.y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto s = ctx->get_saved_variables();
    const Tensor &x = s[0], &mean = s[1], &rstd = s[2], &gamma = s[3], &beta = s[4];
    if (!grads[0].defined()) return variable_list(6);
    const Tensor dy = grads[0].contiguous();
    const int64_t groups = ctx->saved_data["groups"].toInt();
    const bool silu = ctx->saved_data["silu"].toBool();
    const int64_t stats = dy.size(0) * groups, C = dy.size(3);
    Tensor dx, dg, db;
    if (direct(dy, x, mean, rstd, gamma, beta) && half(x) && matches(x, dy) && packed_floats(mean, stats) &&
        packed_floats(rstd, stats) && packed_floats(gamma, C) && packed_floats(beta, C) && on_vectors(dy, x)) {
      below([&] {
        const Env e(dy);
        const Tensor xc = x.contiguous();
        const int64_t B = x.size(0), HW = x.size(1) * x.size(2);
        dx = empty(x.sizes(), x);
        dg = floats(C, x);
        db = floats(C, x);
        const Tensor sums = floats(2 * B * groups, x), scratch = group_scratch(e, x, C + groups);
        ok(pf_groupnorm_bwd(dy.data_ptr(), xc.data_ptr(), mean.data_ptr(), rstd.data_ptr(), gamma.data_ptr(),
                            beta.data_ptr(), dx.data_ptr(), dg.data_ptr(), db.data_ptr(), sums.data_ptr(),
                            scratch.data_ptr(), (int)B, (int)HW, (int)C, (int)groups, silu, code_of(x), e.sms,
                            e.stream),
           "pf_groupnorm_bwd");
        return 0;
      });
    } else {
      auto out = dispatched("pfeife::group_norm_bwd", {dy, x, mean, rstd, gamma, beta, groups, silu});
      dx = out[0].toTensor(); dg = out[1].toTensor(); db = out[2].toTensor();
    }
    return {dx, dg, db, Tensor(), Tensor(), Tensor()};
  }
};

// ------------------------------------------------------------------------------ convolution
// The implicit-GEMM route (kernels.conv_gemm_supported, kernels.conv_wgrad_supported).
struct ConvShape {
  int64_t B, H, W, C, N, KH, KW, stride, pad, Ho, Wo;
  ConvShape(const Tensor& x, const Tensor& w, int64_t s, int64_t p)
      : B(x.size(0)), H(x.size(1)), W(x.size(2)), C(x.size(3)), N(w.size(0)), KH(w.size(2)), KW(w.size(3)),
        stride(s), pad(p), Ho((H + 2 * p - KH) / s + 1), Wo((W + 2 * p - KW) / s + 1) {}
  bool output_fits(const Tensor& y) const {
    return y.dim() == 4 && y.size(0) == B && y.size(1) == Ho && y.size(2) == Wo && y.size(3) == N;
  }
  bool one() const { return KH == 1 && KW == 1 && stride == 1 && pad == 0; }
  bool forward_fits() const {
    return !one() && C % 64 == 0 && N % 8 == 0 && KH * KW <= 64 && Wo > 0 && Ho > 0 && Wo <= 128 &&
           128 % Wo == 0 && Ho * Wo % 128 == 0 && (stride == 1 || stride == 2);
  }
  // Tiles of the input gradient are whole rows of the input.  Python keeps the gradients that take several
  // routes: strides, kernels that are not square, and up to 64 filters, which it pads.
  bool backward_fits() const {
    return stride == 1 && KH == KW && pad < KH && N % 64 == 0 && N > 64 && (64 % Wo == 0 || Wo % 64 == 0) && W <= 128 &&
           128 % W == 0 && H * W % 128 == 0;
  }
};
Tensor conv_pack(const Env& e, const Tensor& w, const ConvShape& s, bool flip) {
  const int64_t taps = s.KH * s.KW;
  const Tensor wc = w.contiguous();
  const Tensor out = flip ? empty({s.C, taps * s.N}, w) : empty({s.N, taps * s.C}, w);
  ok(pf_conv_pack(wc.data_ptr(), out.data_ptr(), (int)s.N, (int)s.C, (int)taps, (int)s.N, (int)s.C, flip,
                  e.stream),
     "pf_conv_pack");
  return out;
}
// images that the implicit GEMM reads in place
bool operands_fit(const Tensor& x, const Tensor& w) {
  return x.dim() == 4 && w.dim() == 4 && half(x) && w.scalar_type() == x.scalar_type() &&
         w.size(1) == x.size(3) && x.is_contiguous() && aligned(x);
}
Tensor conv_forward(const Tensor& x, const Tensor& w, const Tensor& b, int64_t stride, int64_t pad) {
  const Env e(x);
  const ConvShape s(x, w, stride, pad);
  const Tensor w2 = conv_pack(e, w, s, false), y = empty({s.B, s.Ho, s.Wo, s.N}, x);
  ok(pf_conv_gemm(x.data_ptr(), w2.data_ptr(), y.data_ptr(), (int)s.B, (int)s.H, (int)s.W, (int)s.C, (int)s.N,
                  (int)s.KH, (int)s.KW, (int)stride, (int)pad, w2.size(1), s.N, code_of(x), code_of(x),
                  at_or_null(b), 0, nullptr, 0, NONE, e.status, e.sms, e.stream),
     "pf_conv_gemm");
  return y;
}
struct DirectConv2d : torch::autograd::Function<DirectConv2d> {
  static Tensor forward(AutogradContext* ctx, Tensor x, Tensor w, Maybe bias, int64_t stride, int64_t pad) {
    at::AutoDispatchBelowADInplaceOrView guard;
    const Tensor b = value(bias);
    ctx->save_for_backward({x, w});
    ctx->saved_data["pad"] = pad;
    ctx->saved_data["bias"] = b.defined();
    return conv_forward(x, w, b, stride, pad);
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto v = ctx->get_saved_variables();
    const Tensor &x = v[0], &w = v[1];
    const Tensor dy = grads[0].contiguous();
    const int64_t pad = ctx->saved_data["pad"].toInt();
    const bool bias = ctx->saved_data["bias"].toBool();
    const bool nx = ctx->needs_input_grad(0), nw = ctx->needs_input_grad(1);
    Tensor dx, dw, db;
    if (direct(dy, x, w) && operands_fit(x, w) && x.scalar_type() == dy.scalar_type() &&
        ConvShape(x, w, 1, pad).output_fits(dy)) {
      below([&] {
        const Env e(dy);
        const ConvShape s(x, w, 1, pad);
        const Tensor dyc = aligned(dy) ? dy : dy.clone();
        const int64_t K = s.KH * s.KW * s.C, pixels = s.B * s.Ho * s.Wo;
        const Tensor dw2 = empty({s.N, K}, at::kFloat, x);
        const int kib = pf_gemm_workspace((int)s.N, (int)K, (int)pixels, 0, 2, e.sms, 0);
        const Tensor ws = kib ? floats(kib * 256ll, x) : Tensor();
        ok(pf_conv_wgrad(dyc.data_ptr(), x.data_ptr(), dw2.data_ptr(), (int)s.B, (int)s.H, (int)s.W, (int)s.C,
                         (int)s.N, (int)s.KH, (int)s.KW, 1, (int)pad, code_of(x), 0, e.status, e.sms,
                         const_cast<void*>(at_or_null(ws)), kib, e.stream),
           "pf_conv_wgrad");
        dw = empty(w.sizes(), w);
        ok(pf_conv_unpack(dw2.data_ptr(), dw.data_ptr(), (int)s.N, (int)s.C, (int)(s.KH * s.KW), (int)s.C,
                          code_of(w), e.stream),
           "pf_conv_unpack");
        if (nx) {
          const Tensor wt = conv_pack(e, w, s, true);
          dx = empty(x.sizes(), x);
          ok(pf_conv_gemm(dyc.data_ptr(), wt.data_ptr(), dx.data_ptr(), (int)s.B, (int)s.Ho, (int)s.Wo,
                          (int)s.N, (int)s.C, (int)s.KH, (int)s.KW, 1, (int)(s.KH - 1 - pad), wt.size(1), s.C,
                          code_of(x), code_of(x), nullptr, 0, nullptr, 0, NONE, e.status, e.sms, e.stream),
             "pf_conv_gemm");
        }
        if (bias) db = colsum(e, dyc.view({pixels, s.N}));
        return 0;
      });
    } else {
      auto out = dispatched("pfeife::conv2d_bwd", {dy, x, w, (int64_t)1, pad, nx, bias});
      dx = given(out[0]); dw = out[1].toTensor(); db = given(out[2]);
    }
    return {nx ? dx : Tensor(), nw ? dw : Tensor(), bias ? db : Tensor(), Tensor(), Tensor()};
  }
};

// ------------------------------------------------------------------------------ Python
// Arguments of one call.  `fits` turns false at the first that is not what the usual call has.
struct Args {
  PyObject* const* a;
  bool fits;
  Args(PyObject* const* args, Py_ssize_t n, Py_ssize_t expected) : a(args), fits(n == expected) {
    if (!fits) PyErr_Format(PyExc_TypeError, "expected %zd arguments, got %zd", expected, n);
    else fits = unobserved() && !at::autocast::is_autocast_enabled(at::kCUDA);
  }
  Tensor tensor(int i, bool optional = false) {
    if (!fits) return {};
    if (optional && a[i] == Py_None) return {};
    if (!THPVariable_CheckTypeExact(Py_TYPE(a[i]))) { fits = false; return {}; }
    const Tensor& t = THPVariable_Unpack(a[i]);
    if (!t.is_cuda()) fits = false;
    return t;
  }
  int64_t integer(int i) {
    if (!fits) return 0;
    if (!PyLong_CheckExact(a[i])) { fits = false; return 0; }
    const long long v = PyLong_AsLongLong(a[i]);
    if (v == -1 && PyErr_Occurred()) { PyErr_Clear(); fits = false; }
    return v;
  }
  bool boolean(int i) {
    if (a[i] != Py_True && a[i] != Py_False) fits = false;
    return a[i] == Py_True;
  }
  double real(int i) {
    if (!fits) return 0;
    if (!PyFloat_CheckExact(a[i])) { fits = false; return 0; }
    return PyFloat_AS_DOUBLE(a[i]);
  }
};

// Runs `f`, which returns the outputs, without the interpreter lock; None where the kernels refuse the
// call (Python repeats it and reports why).
template <typename F>
PyObject* run(const Tensor& first, F&& f) {
  if (first.get_device() >= MAX_DEVICES) Py_RETURN_NONE;
  if (!learn_status(first.get_device())) return nullptr;
  try {
    decltype(f()) out;
    {
      pybind11::gil_scoped_release free;
      out = f();
    }
    if constexpr (std::is_same_v<decltype(out), Tensor>) {
      return THPVariable_Wrap(std::move(out));
    } else {
      if (out.size() == 1) return THPVariable_Wrap(std::move(out[0]));
      PyObject* t = PyTuple_New((Py_ssize_t)out.size());
      for (size_t i = 0; t && i < out.size(); ++i) PyTuple_SET_ITEM(t, (Py_ssize_t)i, THPVariable_Wrap(out[i]));
      return t;
    }
  } catch (const Failed&) {
    Py_RETURN_NONE;
  }
}
// HANDLE_TH_ERRORS turns C++ exceptions into Python's.
#define PF_OP(name) PyObject* name(PyObject*, PyObject* const* args, Py_ssize_t n)
template <typename F>
Tensor unrecorded(F&& f) {
  at::AutoDispatchBelowADInplaceOrView guard;
  return f();
}

PF_OP(linear) {
  HANDLE_TH_ERRORS
  Args a(args, n, 5);
  if (PyErr_Occurred()) return nullptr;
  const Tensor x = a.tensor(0), w = a.tensor(1), b = a.tensor(2, true), r = a.tensor(3, true);
  const int64_t act = a.integer(4);
  if (!a.fits || act < 0 || act > 3 || !all_plain(x, w, b, r) || !layer_fits(x, w, b) ||
      !residual_fits(r, x, w.size(0)))
    Py_RETURN_NONE;
  if (!recorded(x, w, b, r))
    return run(x, [&] { return unrecorded([&] { return linear_forward(x, w, b, r, (int)act).first; }); });
  if (w.size(0) % 8) Py_RETURN_NONE;                  // the backward's products need whole vectors
  return run(x, [&] { return DirectLinear::apply(x, w, maybe(b), maybe(r), act); });
  END_HANDLE_TH_ERRORS
}

PF_OP(mlp) {
  HANDLE_TH_ERRORS
  Args a(args, n, 7);
  if (PyErr_Occurred()) return nullptr;
  const Tensor x = a.tensor(0), w1 = a.tensor(1), b1 = a.tensor(2, true), w2 = a.tensor(3),
               b2 = a.tensor(4, true), r = a.tensor(5, true);
  const int64_t act = a.integer(6);
  if (!a.fits || act < 1 || act > 2 || !all_plain(x, w1, b1, w2, b2, r) || !layer_fits(x, w1, b1) ||
      w2.scalar_type() != x.scalar_type() || !readable(w2) || w2.size(1) != w1.size(0) || w2.size(1) % 8 ||
      !bias_fits(b2, w2.size(0)) || !residual_fits(r, x, w2.size(0)))
    Py_RETURN_NONE;
  if (!recorded(x, w1, b1, w2, b2, r))
    return run(x, [&] {
      return unrecorded([&] {
        const Tensor a1 = linear_forward(x, w1, b1, {}, (int)act).first;
        return linear_forward(a1, w2, b2, r, 0).first;
      });
    });
  if (w2.size(0) % 8) Py_RETURN_NONE;
  return run(x, [&] { return DirectMlp::apply(x, w1, maybe(b1), w2, maybe(b2), maybe(r), act); });
  END_HANDLE_TH_ERRORS
}

PF_OP(norm) {
  HANDLE_TH_ERRORS
  Args a(args, n, 6);
  if (PyErr_Occurred()) return nullptr;
  const Tensor x = a.tensor(0), g = a.tensor(1), b = a.tensor(2, true), r = a.tensor(3, true);
  const double eps = a.real(4);
  const bool rms = a.boolean(5);
  auto vector = [&](const Tensor& t) {
    return !t.defined() || (t.scalar_type() == at::kFloat && t.dim() == 1 && t.size(0) == x.size(-1) &&
                            t.is_contiguous());
  };
  if (!a.fits || !all_plain(x, g, b, r) || x.dim() < 1 || !half(x) || !vector(g) || !vector(b) ||
      !on_vectors(x, g, b, r) || (r.defined() && (r.scalar_type() != x.scalar_type() || r.sizes() != x.sizes())))
    Py_RETURN_NONE;
  if (!recorded(x, g, b, r))
    return run(x, [&]() -> variable_list {
      at::AutoDispatchBelowADInplaceOrView guard;
      const NormOut o = norm_forward(x, g, b, r, eps, rms);
      if (r.defined()) return {o.y, o.h};
      return {o.y};
    });
  return run(x, [&] { return DirectNorm::apply(x, g, maybe(b), maybe(r), eps, rms); });
  END_HANDLE_TH_ERRORS
}

PF_OP(attention) {
  HANDLE_TH_ERRORS
  Args a(args, n, 5);
  if (PyErr_Occurred()) return nullptr;
  const Tensor q = a.tensor(0), k = a.tensor(1), v = a.tensor(2);
  const bool causal = a.boolean(3);
  const double scale = a.real(4);
  if (!a.fits || !all_plain(q, k, v) || q.dim() != 4 || k.dim() != 4 || !half(q) ||
      k.scalar_type() != q.scalar_type() || v.scalar_type() != q.scalar_type() || k.sizes() != v.sizes() ||
      k.size(0) != q.size(0) || k.size(2) != q.size(2) || k.size(3) != q.size(3) || q.size(3) % 8 ||
      q.size(3) > 128 || q.stride(3) != 1 || k.stride(3) != 1 || v.stride(3) != 1)
    Py_RETURN_NONE;
  if (!recorded(q, k, v))
    return run(q, [&] { return unrecorded([&] { return heads_forward(q, k, v, causal, scale).first; }); });
  return run(q, [&] { return DirectAttention::apply(q, k, v, causal, scale); });
  END_HANDLE_TH_ERRORS
}

PF_OP(attention_qkv) {
  HANDLE_TH_ERRORS
  Args a(args, n, 3);
  if (PyErr_Occurred()) return nullptr;
  const Tensor t = a.tensor(0);
  const bool causal = a.boolean(1);
  const double scale = a.real(2);
  if (!a.fits || !all_plain(t) || t.dim() != 5 || !half(t) || t.size(2) != 3 || t.size(4) % 8 ||
      t.size(4) > 128 || !packed_fits(t))
    Py_RETURN_NONE;
  if (!recorded(t))
    return run(t, [&] { return unrecorded([&] { return packed_forward(t, causal, scale).first; }); });
  return run(t, [&] { return DirectAttentionQkv::apply(t, causal, scale); });
  END_HANDLE_TH_ERRORS
}

PF_OP(rope_qkv) {
  HANDLE_TH_ERRORS
  Args a(args, n, 3);
  if (PyErr_Occurred()) return nullptr;
  const Tensor x = a.tensor(0), cos = a.tensor(1), sin = a.tensor(2);
  if (!a.fits || !all_plain(x, cos, sin) || x.dim() != 5 || !half(x) || x.size(2) != 3 || x.size(4) % 16 ||
      !x.is_contiguous() || !aligned(x) || !table_fits(cos, x) || !table_fits(sin, x))
    Py_RETURN_NONE;
  if (!recorded(x, cos, sin))
    return run(x, [&] { return unrecorded([&] { return rope_forward(x, cos, sin, false); }); });
  return run(x, [&] { return DirectRopeQkv::apply(x, cos, sin); });
  END_HANDLE_TH_ERRORS
}

PF_OP(glu) {
  HANDLE_TH_ERRORS
  Args a(args, n, 2);
  if (PyErr_Occurred()) return nullptr;
  const Tensor gu = a.tensor(0);
  const bool gelu = a.boolean(1);
  if (!a.fits || !all_plain(gu) || gu.dim() < 1 || !half(gu) || gu.size(-1) % 16 || !gu.is_contiguous() ||
      !on_vectors(gu))
    Py_RETURN_NONE;
  if (!recorded(gu)) return run(gu, [&] { return unrecorded([&] { return glu_forward(gu, gelu); }); });
  return run(gu, [&] { return DirectGlu::apply(gu, gelu); });
  END_HANDLE_TH_ERRORS
}

PF_OP(cross_entropy) {
  HANDLE_TH_ERRORS
  Args a(args, n, 3);
  if (PyErr_Occurred()) return nullptr;
  const Tensor x = a.tensor(0), t = a.tensor(1);
  const int64_t ignore = a.integer(2);
  if (!a.fits || !all_plain(x, t) || x.dim() != 2 || !(half(x) || x.scalar_type() == at::kFloat) ||
      t.scalar_type() != at::kLong || t.dim() != 1 || t.size(0) != x.size(0))
    Py_RETURN_NONE;
  if (!recorded(x))
    return run(x, [&] { return unrecorded([&] { return loss_forward(x, t, ignore).mean; }); });
  return run(x, [&] { return DirectCrossEntropy::apply(x, t, ignore); });
  END_HANDLE_TH_ERRORS
}

PF_OP(group_norm) {
  HANDLE_TH_ERRORS
  Args a(args, n, 6);
  if (PyErr_Occurred()) return nullptr;
  const Tensor x = a.tensor(0), g = a.tensor(1), b = a.tensor(2);
  const int64_t groups = a.integer(3);
  const double eps = a.real(4);
  const bool silu = a.boolean(5);
  auto vector = [&](const Tensor& t) {
    return t.scalar_type() == at::kFloat && t.dim() == 1 && t.size(0) == x.size(3) && t.is_contiguous();
  };
  if (!a.fits || !all_plain(x, g, b) || x.dim() != 4 || !half(x) || x.size(3) % 8 || x.size(3) > 8192 ||
      groups <= 0 || x.size(3) % groups || !vector(g) || !vector(b) || !on_vectors(x))
    Py_RETURN_NONE;
  if (!recorded(x, g, b))
    return run(x, [&] { return unrecorded([&] { return group_norm_forward(x, g, b, groups, eps, silu).y; }); });
  return run(x, [&] { return DirectGroupNorm::apply(x, g, b, groups, eps, silu); });
  END_HANDLE_TH_ERRORS
}

PF_OP(conv2d) {
  HANDLE_TH_ERRORS
  Args a(args, n, 5);
  if (PyErr_Occurred()) return nullptr;
  const Tensor x = a.tensor(0), w = a.tensor(1), b = a.tensor(2, true);
  const int64_t stride = a.integer(3), pad = a.integer(4);
  if (!a.fits || !all_plain(x, w, b) || !operands_fit(x, w) || stride < 1 || pad < 0 ||
      !ConvShape(x, w, stride, pad).forward_fits() ||
      (b.defined() && (b.scalar_type() != at::kFloat || !bias_fits(b, w.size(0)))))
    Py_RETURN_NONE;
  if (!recorded(x, w, b))
    return run(x, [&] { return unrecorded([&] { return conv_forward(x, w, b, stride, pad); }); });
  if (!ConvShape(x, w, stride, pad).backward_fits()) Py_RETURN_NONE;
  return run(x, [&] { return DirectConv2d::apply(x, w, maybe(b), stride, pad); });
  END_HANDLE_TH_ERRORS
}

PyObject* setup(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 2) return PyErr_Format(PyExc_TypeError, "setup(status_word, check)");
  Py_INCREF(args[0]);
  Py_INCREF(args[1]);
  g_status_word = args[0];
  g_check = args[1];
  Py_RETURN_NONE;
}
PyObject* launches(PyObject*, PyObject*) { return PyLong_FromLongLong(g_launches.load()); }

#define PF_ENTRY(name) \
  {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&name)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    PF_ENTRY(linear), PF_ENTRY(mlp), PF_ENTRY(norm), PF_ENTRY(attention), PF_ENTRY(attention_qkv),
    PF_ENTRY(rope_qkv), PF_ENTRY(glu), PF_ENTRY(cross_entropy), PF_ENTRY(group_norm), PF_ENTRY(conv2d),
    PF_ENTRY(setup), {"launches", launches, METH_NOARGS, nullptr}, {nullptr, nullptr, 0, nullptr}};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "pfeife_b200_eager", "eager calls of the ops", -1, methods,
                          nullptr, nullptr, nullptr, nullptr};

}  // namespace pfeife

PyMODINIT_FUNC PyInit_pfeife_b200_eager() {
  PyObject* m = PyModule_Create(&pfeife::module_def);
  // the sources it was built from: the loader takes no module of others
  if (m && PyModule_AddStringConstant(m, "SOURCES", PF_SOURCES) < 0) Py_CLEAR(m);
  return m;
}
