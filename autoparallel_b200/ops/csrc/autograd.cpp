// Native autograd of the apb200 operators for CUDA tensors.
//
// The formulas are those that ops/library.py and ops/moe_ops.py register for every device; here they are registered
// again, for the AutogradCUDA key only, so that a call on CUDA tensors passes through no Python on its way to the CUDA
// kernel's entry and its gradient node is a C++ one.  What that costs on the host per call (forward alone / forward that
// records a gradient): 18 -> 8 us / 38 -> 10 us, the CUDA entry apart.
// CPU, meta and fake CPU tensors (planning) keep the Python registration.  Everything below autograd - dispatch modes, fake
// tensors, functionalisation, the CUDA entries at the end of binding.cpp - is reached as before, by redispatch; functorch
// transforms and forward-mode differentiation of a recorded call are refused by the C++ function itself as they are by the Python
// one; a dual tensor in a call that records nothing loses its tangent, as it does there.
#include <ATen/core/dispatch/Dispatcher.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/library.h>

#include <tuple>

namespace {

using at::ScalarType;
using at::Tensor;
using c10::DispatchKeySet;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

// A typed operator of this namespace, looked up once.  ``below`` runs what is under the autograd layer.
template <typename Sig>
struct Op;
template <typename R, typename... Args>
struct Op<R(Args...)> {
  c10::TypedOperatorHandle<R(Args...)> h;
  explicit Op(const char* name) : h(c10::Dispatcher::singleton().findSchemaOrThrow(name, "").typed<R(Args...)>()) {}
  R operator()(Args... args) const { return h.call(args...); }
  R below(DispatchKeySet ks, Args... args) const {
    at::AutoDispatchBelowAutograd guard;
    return h.redispatch(ks & c10::after_autograd_keyset, args...);
  }
};

template <typename... Ts>
bool records(const Ts&... ts) {
  return at::GradMode::is_enabled() && (ts.requires_grad() || ...);
}

#define APB_OP(var, name, ...) static const Op<__VA_ARGS__> var("apb200::" name)
using Pair = std::tuple<Tensor, Tensor>;
using Triple = std::tuple<Tensor, Tensor, Tensor>;

using CastSig = Tensor(const Tensor&, ScalarType);
using MmNdSig = Tensor(const Tensor&, const Tensor&, bool, ScalarType);
using WgradSig = Tensor(const Tensor&, const Tensor&, ScalarType);
using GemmSig = Tensor(const Tensor&, const Tensor&, bool, bool, ScalarType);
using RmsSig = Pair(const Tensor&, const Tensor&, double);
using RmsBwdSig = Pair(const Tensor&, const Tensor&, const Tensor&, const Tensor&);
using RopeSig = Tensor(const Tensor&, const Tensor&, const Tensor&, bool);
using SwigluSig = Tensor(const Tensor&, const Tensor&);
using SwigluBwdSig = Pair(const Tensor&, const Tensor&, const Tensor&);
using AttnSig = Pair(const Tensor&, const Tensor&, const Tensor&, bool, double);
using AttnBwdSig = Triple(const Tensor&, const Tensor&, const Tensor&, const Tensor&, const Tensor&, const Tensor&, bool, double);
using XentSig = Pair(const Tensor&, const Tensor&);
using XentBwdSig = Tensor(const Tensor&, const Tensor&, const Tensor&, const Tensor&);
using EmbSig = Tensor(const Tensor&, const Tensor&);
using EmbBwdSig = Tensor(const Tensor&, const Tensor&, int64_t);
using ScatterSig = Tensor(const Tensor&, const Tensor&, const Tensor&, int64_t, int64_t, int64_t);
using GatherSig = Tensor(const Tensor&, const Tensor&, const Tensor&);

// Gradient of the first output of an operator whose second one (1 / rms, log-sum-exp) is seldom used.  The engine would fill a tensor of zeros for
// the second one's gradient, which no formula reads: a launch, an allocation and 8 us of host time per call (RMSNorm of 2047 x 2048 fp32, forward
// and backward, 81 -> 73 us).  So these operators take gradients as they come; where only the second output was used, the first one's is zeros.
Tensor first_grad(const variable_list& g, const Tensor& like) { return g[0].defined() ? g[0] : at::zeros_like(like); }

// The dispatch keys of the call travel to ``forward`` in a wrapper, so that they are not taken for an input.
struct Keys {
  DispatchKeySet ks;
};

// ---------------------------------------------------------------------------------------------- dtype_cast
const Op<CastSig>& op_cast() { APB_OP(o, "dtype_cast", CastSig); return o; }
struct Cast : torch::autograd::Function<Cast> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, ScalarType dtype, Keys k) {
    ctx->saved_data["dtype"] = x.scalar_type();
    return op_cast().below(k.ks, x, dtype);
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& g) {
    return {op_cast()(g[0], ctx->saved_data["dtype"].toScalarType()), Tensor(), Tensor()};
  }
};
Tensor cast(DispatchKeySet ks, const Tensor& x, ScalarType dtype) {
  return records(x) ? Cast::apply(x, dtype, Keys{ks}) : op_cast().below(ks, x, dtype);
}

// ---------------------------------------------------------------------------------------------- projections
const Op<MmNdSig>& op_mm_nd() { APB_OP(o, "mm_nd", MmNdSig); return o; }
const Op<WgradSig>& op_mm_wgrad() { APB_OP(o, "mm_wgrad", WgradSig); return o; }
struct MmNd : torch::autograd::Function<MmNd> {
  static Tensor forward(AutogradContext* ctx, const Tensor& a, const Tensor& b, bool tb, ScalarType dtype, Keys k) {
    ctx->save_for_backward({a, b});
    ctx->saved_data["tb"] = tb;
    return op_mm_nd().below(k.ks, a, b, tb, dtype);
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& g) {
    const auto s = ctx->get_saved_variables();
    const Tensor &a = s[0], &b = s[1], &dc = g[0];
    const bool tb = ctx->saved_data["tb"].toBool();
    Tensor da, db;
    if (ctx->needs_input_grad(0)) da = op_mm_nd()(dc, b, !tb, a.scalar_type());
    if (ctx->needs_input_grad(1)) db = tb ? op_mm_wgrad()(dc, a, b.scalar_type()) : op_mm_wgrad()(a, dc, b.scalar_type());
    return {da, db, Tensor(), Tensor(), Tensor()};
  }
};
Tensor mm_nd(DispatchKeySet ks, const Tensor& a, const Tensor& b, bool tb, ScalarType dtype) {
  return records(a, b) ? MmNd::apply(a, b, tb, dtype, Keys{ks}) : op_mm_nd().below(ks, a, b, tb, dtype);
}

const Op<GemmSig>& op_gemm() { APB_OP(o, "gemm", GemmSig); return o; }
struct Gemm : torch::autograd::Function<Gemm> {
  static Tensor forward(AutogradContext* ctx, const Tensor& a, const Tensor& b, bool ta, bool tb, ScalarType dtype, Keys k) {
    ctx->save_for_backward({a, b});
    ctx->saved_data["ta"] = ta;
    ctx->saved_data["tb"] = tb;
    return op_gemm().below(k.ks, a, b, ta, tb, dtype);
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& g) {
    const auto s = ctx->get_saved_variables();
    const Tensor &a = s[0], &b = s[1], &dc = g[0];
    const bool ta = ctx->saved_data["ta"].toBool(), tb = ctx->saved_data["tb"].toBool();
    // C = op(A) op(B): dA_op = dC op(B)^T, dB_op = op(A)^T dC, then the storage transpose is undone
    Tensor da, db;
    if (ctx->needs_input_grad(0)) da = ta ? op_gemm()(b, dc, tb, true, a.scalar_type()) : op_gemm()(dc, b, false, !tb, a.scalar_type());
    if (ctx->needs_input_grad(1)) db = tb ? op_gemm()(dc, a, true, ta, b.scalar_type()) : op_gemm()(a, dc, !ta, false, b.scalar_type());
    return {da, db, Tensor(), Tensor(), Tensor(), Tensor()};
  }
};
Tensor gemm(DispatchKeySet ks, const Tensor& a, const Tensor& b, bool ta, bool tb, ScalarType dtype) {
  return records(a, b) ? Gemm::apply(a, b, ta, tb, dtype, Keys{ks}) : op_gemm().below(ks, a, b, ta, tb, dtype);
}

const Op<MmNdSig>& op_grouped_mm() { APB_OP(o, "grouped_mm", MmNdSig); return o; }
const Op<WgradSig>& op_grouped_wgrad() { APB_OP(o, "grouped_mm_wgrad", WgradSig); return o; }
struct GroupedMm : torch::autograd::Function<GroupedMm> {
  static Tensor forward(AutogradContext* ctx, const Tensor& a, const Tensor& b, bool tb, ScalarType dtype, Keys k) {
    ctx->save_for_backward({a, b});
    ctx->saved_data["tb"] = tb;
    return op_grouped_mm().below(k.ks, a, b, tb, dtype);
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& g) {
    const auto s = ctx->get_saved_variables();
    const Tensor &a = s[0], &b = s[1], &dc = g[0];
    const bool tb = ctx->saved_data["tb"].toBool();
    Tensor da, db;
    if (ctx->needs_input_grad(0)) da = op_grouped_mm()(dc, b, !tb, a.scalar_type());
    if (ctx->needs_input_grad(1)) db = tb ? op_grouped_wgrad()(dc, a, b.scalar_type()) : op_grouped_wgrad()(a, dc, b.scalar_type());
    return {da, db, Tensor(), Tensor(), Tensor()};
  }
};
Tensor grouped_mm(DispatchKeySet ks, const Tensor& a, const Tensor& b, bool tb, ScalarType dtype) {
  return records(a, b) ? GroupedMm::apply(a, b, tb, dtype, Keys{ks}) : op_grouped_mm().below(ks, a, b, tb, dtype);
}

// ---------------------------------------------------------------------------------------------- norm, rotary, SwiGLU
const Op<RmsSig>& op_rms() { APB_OP(o, "rms_norm", RmsSig); return o; }
const Op<RmsBwdSig>& op_rms_bwd() { APB_OP(o, "rms_norm_bwd", RmsBwdSig); return o; }
struct Rms : torch::autograd::Function<Rms> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& w, double eps, Keys k) {
    auto [y, rstd] = op_rms().below(k.ks, x, w, eps);
    ctx->save_for_backward({x, w, rstd});
    ctx->set_materialize_grads(false);
    return {y, rstd};
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& g) {
    const auto s = ctx->get_saved_variables();
    auto [dx, dw] = op_rms_bwd()(first_grad(g, s[0]), s[0], s[1], s[2]);
    return {dx, dw, Tensor(), Tensor()};
  }
};
Pair rms_norm(DispatchKeySet ks, const Tensor& x, const Tensor& w, double eps) {
  if (!records(x, w)) return op_rms().below(ks, x, w, eps);
  auto o = Rms::apply(x, w, eps, Keys{ks});
  return {o[0], o[1]};
}

const Op<RopeSig>& op_rope() { APB_OP(o, "rope", RopeSig); return o; }
struct Rope : torch::autograd::Function<Rope> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& cos, const Tensor& sin, bool conj, Keys k) {
    ctx->save_for_backward({cos, sin});
    ctx->saved_data["conj"] = conj;
    return op_rope().below(k.ks, x, cos, sin, conj);
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& g) {
    const auto s = ctx->get_saved_variables();
    return {op_rope()(g[0], s[0], s[1], !ctx->saved_data["conj"].toBool()), Tensor(), Tensor(), Tensor(), Tensor()};
  }
};
Tensor rope(DispatchKeySet ks, const Tensor& x, const Tensor& cos, const Tensor& sin, bool conj) {
  return records(x, cos, sin) ? Rope::apply(x, cos, sin, conj, Keys{ks}) : op_rope().below(ks, x, cos, sin, conj);
}

const Op<SwigluSig>& op_swiglu() { APB_OP(o, "swiglu", SwigluSig); return o; }
const Op<SwigluBwdSig>& op_swiglu_bwd() { APB_OP(o, "swiglu_bwd", SwigluBwdSig); return o; }
struct Swiglu : torch::autograd::Function<Swiglu> {
  static Tensor forward(AutogradContext* ctx, const Tensor& a, const Tensor& b, Keys k) {
    ctx->save_for_backward({a, b});
    return op_swiglu().below(k.ks, a, b);
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& g) {
    const auto s = ctx->get_saved_variables();
    auto [da, db] = op_swiglu_bwd()(g[0], s[0], s[1]);
    return {da, db, Tensor()};
  }
};
Tensor swiglu(DispatchKeySet ks, const Tensor& a, const Tensor& b) {
  return records(a, b) ? Swiglu::apply(a, b, Keys{ks}) : op_swiglu().below(ks, a, b);
}

// ---------------------------------------------------------------------------------------------- attention, loss, embedding
const Op<AttnSig>& op_attn() { APB_OP(o, "attention", AttnSig); return o; }
const Op<AttnBwdSig>& op_attn_bwd() { APB_OP(o, "attention_bwd", AttnBwdSig); return o; }
struct Attn : torch::autograd::Function<Attn> {
  static variable_list forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v, bool causal, double scale, Keys key) {
    auto [out, lse] = op_attn().below(key.ks, q, k, v, causal, scale);
    ctx->save_for_backward({q, k, v, out, lse});
    ctx->set_materialize_grads(false);
    ctx->saved_data["causal"] = causal;
    ctx->saved_data["scale"] = scale;
    return {out, lse};
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& g) {
    const auto s = ctx->get_saved_variables();
    auto [dq, dk, dv] =
        op_attn_bwd()(first_grad(g, s[3]), s[0], s[1], s[2], s[3], s[4], ctx->saved_data["causal"].toBool(), ctx->saved_data["scale"].toDouble());
    return {dq, dk, dv, Tensor(), Tensor(), Tensor()};
  }
};
Pair attention(DispatchKeySet ks, const Tensor& q, const Tensor& k, const Tensor& v, bool causal, double scale) {
  if (!records(q, k, v)) return op_attn().below(ks, q, k, v, causal, scale);
  auto o = Attn::apply(q, k, v, causal, scale, Keys{ks});
  return {o[0], o[1]};
}

const Op<XentSig>& op_xent() { APB_OP(o, "cross_entropy", XentSig); return o; }
const Op<XentBwdSig>& op_xent_bwd() { APB_OP(o, "cross_entropy_bwd", XentBwdSig); return o; }
struct Xent : torch::autograd::Function<Xent> {
  static variable_list forward(AutogradContext* ctx, const Tensor& logits, const Tensor& labels, Keys k) {
    auto [loss, lse] = op_xent().below(k.ks, logits, labels);
    ctx->save_for_backward({logits, labels, lse});
    ctx->set_materialize_grads(false);
    return {loss, lse};
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& g) {
    const auto s = ctx->get_saved_variables();
    return {op_xent_bwd()(first_grad(g, s[2]), s[0], s[1], s[2]), Tensor(), Tensor()};
  }
};
Pair cross_entropy(DispatchKeySet ks, const Tensor& logits, const Tensor& labels) {
  if (!records(logits)) return op_xent().below(ks, logits, labels);
  auto o = Xent::apply(logits, labels, Keys{ks});
  return {o[0], o[1]};
}

const Op<EmbSig>& op_emb() { APB_OP(o, "embedding", EmbSig); return o; }
const Op<EmbBwdSig>& op_emb_bwd() { APB_OP(o, "embedding_bwd", EmbBwdSig); return o; }
struct Emb : torch::autograd::Function<Emb> {
  static Tensor forward(AutogradContext* ctx, const Tensor& weight, const Tensor& ids, Keys k) {
    ctx->save_for_backward({ids});
    ctx->saved_data["rows"] = weight.sym_size(0).guard_int(__FILE__, __LINE__);
    return op_emb().below(k.ks, weight, ids);
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& g) {
    const auto s = ctx->get_saved_variables();
    return {op_emb_bwd()(g[0], s[0], ctx->saved_data["rows"].toInt()), Tensor(), Tensor()};
  }
};
Tensor embedding(DispatchKeySet ks, const Tensor& weight, const Tensor& ids) {
  return records(weight) ? Emb::apply(weight, ids, Keys{ks}) : op_emb().below(ks, weight, ids);
}

// ---------------------------------------------------------------------------------------------- mixture-of-experts dispatch
const Op<ScatterSig>& op_scatter() { APB_OP(o, "moe_scatter", ScatterSig); return o; }
const Op<GatherSig>& op_gather() { APB_OP(o, "moe_gather", GatherSig); return o; }
const Op<GatherSig>& op_gate_grad() { APB_OP(o, "moe_gate_grad", GatherSig); return o; }
struct Scatter : torch::autograd::Function<Scatter> {
  static Tensor forward(AutogradContext* ctx, const Tensor& src, const Tensor& slot, const Tensor& w, int64_t E, int64_t C, int64_t nb, Keys k) {
    ctx->save_for_backward({src, slot, w});
    return op_scatter().below(k.ks, src, slot, w, E, C, nb);
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& g) {
    const auto s = ctx->get_saved_variables();
    Tensor dsrc, dw;
    if (ctx->needs_input_grad(0)) dsrc = op_gather()(g[0], s[1], s[2]);
    if (ctx->needs_input_grad(2)) dw = op_gate_grad()(g[0], s[1], s[0]).to(s[2].scalar_type());
    return {dsrc, Tensor(), dw, Tensor(), Tensor(), Tensor(), Tensor()};
  }
};
Tensor moe_scatter(DispatchKeySet ks, const Tensor& src, const Tensor& slot, const Tensor& w, int64_t E, int64_t C, int64_t nb) {
  return records(src, w) ? Scatter::apply(src, slot, w, E, C, nb, Keys{ks}) : op_scatter().below(ks, src, slot, w, E, C, nb);
}
struct Gather : torch::autograd::Function<Gather> {
  static Tensor forward(AutogradContext* ctx, const Tensor& buf, const Tensor& slot, const Tensor& w, Keys k) {
    ctx->save_for_backward({buf, slot, w});
    return op_gather().below(k.ks, buf, slot, w);
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& g) {
    const auto s = ctx->get_saved_variables();
    const Tensor &buf = s[0], &slot = s[1], &w = s[2];
    Tensor dbuf, dw;
    if (ctx->needs_input_grad(0))
      dbuf = op_scatter()(g[0], slot, w, buf.sym_size(0).guard_int(__FILE__, __LINE__), buf.sym_size(2).guard_int(__FILE__, __LINE__),
                          buf.sym_size(1).guard_int(__FILE__, __LINE__));
    if (ctx->needs_input_grad(2)) dw = op_gate_grad()(buf, slot, g[0]).to(w.scalar_type());
    return {dbuf, Tensor(), dw, Tensor()};
  }
};
Tensor moe_gather(DispatchKeySet ks, const Tensor& buf, const Tensor& slot, const Tensor& w) {
  return records(buf, w) ? Gather::apply(buf, slot, w, Keys{ks}) : op_gather().below(ks, buf, slot, w);
}

}  // namespace

TORCH_LIBRARY_IMPL(apb200, AutogradCUDA, m) {
  m.impl("dtype_cast", cast);
  m.impl("mm_nd", mm_nd);
  m.impl("gemm", gemm);
  m.impl("grouped_mm", grouped_mm);
  m.impl("rms_norm", rms_norm);
  m.impl("rope", rope);
  m.impl("swiglu", swiglu);
  m.impl("attention", attention);
  m.impl("cross_entropy", cross_entropy);
  m.impl("embedding", embedding);
  m.impl("moe_scatter", moe_scatter);
  m.impl("moe_gather", moe_gather);
}
