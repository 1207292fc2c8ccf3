// Differentiable front ends of the kernels: the autograd nodes of linear, bias + activation,
// bias + dropout + residual, the normalisations, flash attention and T5's relative bias, as C++
// functions.
//
// A layer of a small model is a few kernels of some microseconds each; a Python autograd function
// costs about 30 us per direction on the host (argument packing, the interpreter, one operator
// call per kernel), which is what such a layer then takes.  Here the host work of a direction is
// one operator call from Python and the launches.
//
// The kernels are reached through their registered operators, so that each keeps its checks.
#include <ATen/ATen.h>
#include <ATen/core/dispatch/Dispatcher.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/library.h>

namespace {

using at::Tensor;
using c10::optional;
using torch::autograd::AutogradContext;
using torch::autograd::Function;
using torch::autograd::tensor_list;
using torch::autograd::variable_list;

template <typename Sig>
auto op(const char* name) {
  return c10::Dispatcher::singleton().findSchemaOrThrow(name, "").typed<Sig>();
}

// Tensors that may be missing are optional arguments of the nodes below (an undefined tensor is
// not a valid input of a node) and undefined among the saved ones.
optional<Tensor> opt(const Tensor& t) { return t.defined() ? optional<Tensor>(t) : optional<Tensor>(); }
Tensor or_undefined(const optional<Tensor>& t) { return t.has_value() ? *t : Tensor(); }

Tensor philox_reserve(int64_t n) {
  static auto f = op<Tensor(int64_t)>("slapo_b200::philox_reserve");
  return f.call(n);
}
Tensor gemm(const Tensor& a, const Tensor& b, const optional<Tensor>& bias, int64_t act, bool a_mn, bool b_mn,
            bool split_k) {
  static auto f = op<Tensor(const Tensor&, const Tensor&, const optional<Tensor>&, int64_t, bool, bool,
                            const optional<Tensor>&, const optional<Tensor>&, int64_t, bool)>(
      "slapo_b200::gemm_out");
  return f.call(a, b, bias, act, a_mn, b_mn, c10::nullopt, c10::nullopt, 0, split_k);
}
Tensor colsum(const Tensor& x) {
  static auto f = op<Tensor(const Tensor&)>("slapo_b200::colsum");
  return f.call(x);
}

std::tuple<Tensor, Tensor> gemm_act_fwd(const Tensor& a, const Tensor& w, const optional<Tensor>& bias,
                                        int64_t act, bool keep, bool sum) {
  static auto f = op<std::tuple<Tensor, Tensor>(const Tensor&, const Tensor&, const optional<Tensor>&, int64_t, bool,
                                                bool)>("slapo_b200::gemm_act_fwd");
  return f.call(a, w, bias, act, keep, sum);
}
constexpr int64_t kRelu = 2;
Tensor bias_act_fwd(const Tensor& x, const optional<Tensor>& bias, int64_t act) {
  static auto f = op<Tensor(const Tensor&, const optional<Tensor>&, int64_t)>("slapo_b200::bias_act_fwd");
  return f.call(x, bias, act);
}
std::tuple<Tensor, Tensor> bias_act_bwd(const Tensor& dy, const Tensor& x, const optional<Tensor>& bias,
                                        int64_t act) {
  static auto f = op<std::tuple<Tensor, Tensor>(const Tensor&, const Tensor&, const optional<Tensor>&,
                                                int64_t)>("slapo_b200::bias_act_bwd");
  return f.call(dy, x, bias, act);
}

// `t` as a 2-D matrix with contiguous rows whose stride TMA accepts
Tensor rows_of(const Tensor& t) {
  Tensor t2 = t.reshape({-1, t.size(-1)});
  if (t2.stride(1) != 1 || t2.stride(0) % 8 != 0 ||
      reinterpret_cast<uintptr_t>(t2.data_ptr()) % 16 != 0)
    t2 = t2.contiguous();
  return t2;
}
std::vector<int64_t> with_last(at::IntArrayRef shape, int64_t last) {
  std::vector<int64_t> s = shape.vec();
  s.back() = last;
  return s;
}

// ------------------------------------------------------------------------ //
// y = act(x W^T + b) (act < 0: no activation): three GEMMs, none of them transposing an operand in
// memory.  Bias and activation ride in the forward GEMM's epilogue; the backward reads ReLU's derivative
// off the output (y > 0) and GeLU's off the product, which the same epilogue leaves where a backward
// will follow (`keep`).  GeLU's values and gradients are to the bit those of the plain layer followed
// by BiasActFn.  `transposed`: W is stored [in, out] (x W + b).
struct LinearFn : public Function<LinearFn> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& weight,
                        const optional<Tensor>& bias, int64_t act, bool transposed, bool keep) {
    Tensor x2 = rows_of(x);
    Tensor y, at;         // at: where the activation's derivative is read off
    const bool gelu = act >= 0 && act != kRelu;
    if (gelu && transposed) {       // (the epilogue forms take W as [out, in])
      at = gemm(x2, weight, c10::nullopt, -1, false, true, false);
      y = bias_act_fwd(at, bias, act);
    } else if (gelu) {
      std::tie(y, at) = gemm_act_fwd(x2, weight, bias, act, keep, false);
    } else {
      y = gemm(x2, weight, bias, act, false, transposed, false);
      if (act >= 0) at = y;
    }
    ctx->saved_data["act"] = act;
    ctx->saved_data["transposed"] = transposed;
    ctx->saved_data["bias"] = bias.has_value();
    ctx->saved_data["shape"] = x.sizes().vec();
    ctx->save_for_backward({x2, weight, at, gelu ? or_undefined(bias) : Tensor()});
    return y.view(with_last(x.sizes(), weight.size(transposed ? 1 : 0)));
  }
  static tensor_list backward(AutogradContext* ctx, tensor_list grads) {
    const variable_list saved = ctx->get_saved_variables();
    const Tensor &x2 = saved[0], &weight = saved[1], &at = saved[2];
    const int64_t act = ctx->saved_data["act"].toInt();
    const bool transposed = ctx->saved_data["transposed"].toBool();
    const bool has_bias = ctx->saved_data["bias"].toBool();
    Tensor dy = rows_of(grads[0]);
    Tensor dx, dw, db;
    if (act == kRelu) {
      static auto f = op<std::tuple<Tensor, Tensor>(const Tensor&, const Tensor&, int64_t)>(
          "slapo_b200::act_bwd_colsum");
      std::tie(dy, db) = f.call(dy.contiguous(), at, act);
    } else if (act >= 0) {
      std::tie(dy, db) = bias_act_bwd(dy.contiguous(), at, opt(saved[3]), act);
    } else if (has_bias && ctx->needs_input_grad(2)) {
      db = colsum(dy);
    }
    if (ctx->needs_input_grad(0))
      dx = gemm(dy, weight, c10::nullopt, -1, false, !transposed, false)
               .view(ctx->saved_data["shape"].toIntVector());
    if (ctx->needs_input_grad(1))
      // few tiles and a long contraction, hence split-K
      dw = transposed ? gemm(x2, dy, c10::nullopt, -1, true, true, true)
                      : gemm(dy, x2, c10::nullopt, -1, true, true, true);
    return {dx, dw, has_bias ? db : Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

// y = dropout(act(x W1^T + b1) W2^T + b2): a feed-forward block as one node.  The input gradient of the
// second layer goes through the activation's derivative and its column sums in that product's epilogue,
// which as separate nodes is a pass of its own over the inner width (16384 x 4096 bf16: 94 + 72 -> 137 us), and
// the host enters autograd once per direction instead of three or four times.
struct MlpFn : public Function<MlpFn> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w1, const Tensor& b1,
                        const Tensor& w2, const Tensor& b2, int64_t act, double p, bool keep) {
    Tensor x2 = rows_of(x);
    Tensor h, at, y;
    if (act != kRelu) {
      std::tie(h, at) = gemm_act_fwd(x2, w1, b1, act, keep, true);
    } else {
      h = gemm(x2, w1, b1, act, false, false, false);
      at = h;
    }
    if (p > 0.0) {
      Tensor rng = philox_reserve(h.size(0) * w2.size(0));
      if (h.size(0) > 16 && w2.size(0) % 16 == 0) {      // dropout in the product's epilogue
        static auto f = op<Tensor(const Tensor&, const Tensor&, const optional<Tensor>&, double, const Tensor&)>(
            "slapo_b200::gemm_dropout_fwd");
        y = f.call(h, w2, b2, p, rng);
      } else {
        static auto f = op<Tensor(const Tensor&, const optional<Tensor>&, const optional<Tensor>&, double,
                                  const Tensor&)>("slapo_b200::bias_dropout_add_fwd");
        y = f.call(gemm(h, w2, c10::nullopt, -1, false, false, false), b2, c10::nullopt, p, rng);
      }
      ctx->saved_data["rng"] = rng;
    } else {
      y = gemm(h, w2, b2, -1, false, false, false);
    }
    ctx->saved_data["act"] = act;
    ctx->saved_data["p"] = p;
    ctx->saved_data["shape"] = x.sizes().vec();
    ctx->save_for_backward({x2, w1, w2, h, at});
    return y.view(with_last(x.sizes(), w2.size(0)));
  }
  static tensor_list backward(AutogradContext* ctx, tensor_list grads) {
    const variable_list s = ctx->get_saved_variables();
    const Tensor &x2 = s[0], &w1 = s[1], &w2 = s[2], &h = s[3], &at = s[4];
    const double p = ctx->saved_data["p"].toDouble();
    tensor_list out(8);
    Tensor dy;
    if (p > 0.0) {
      static auto f = op<std::tuple<Tensor, Tensor>(const Tensor&, double, const Tensor&, bool)>(
          "slapo_b200::bias_dropout_add_bwd");
      Tensor g = grads[0].contiguous();
      std::tie(dy, out[4]) = f.call(g.view({-1, g.size(-1)}), p, ctx->saved_data["rng"].toTensor(),
                                    ctx->needs_input_grad(4));
      if (!ctx->needs_input_grad(4)) out[4] = Tensor();
    } else {
      dy = rows_of(grads[0]);
      if (ctx->needs_input_grad(4)) out[4] = colsum(dy);
    }
    if (ctx->needs_input_grad(3)) out[3] = gemm(dy, h, c10::nullopt, -1, true, true, true);
    if (ctx->needs_input_grad(0) || ctx->needs_input_grad(1) || ctx->needs_input_grad(2)) {
      static auto f = op<std::tuple<Tensor, Tensor>(const Tensor&, const Tensor&, const Tensor&, int64_t)>(
          "slapo_b200::gemm_act_bwd");
      auto [dz, db1] = f.call(dy, w2, at, ctx->saved_data["act"].toInt());
      out[2] = db1;
      if (ctx->needs_input_grad(0))
        out[0] = gemm(dz, w1, c10::nullopt, -1, false, true, false).view(ctx->saved_data["shape"].toIntVector());
      if (ctx->needs_input_grad(1)) out[1] = gemm(dz, x2, c10::nullopt, -1, true, true, true);
    }
    return out;
  }
};

struct BiasActFn : public Function<BiasActFn> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const optional<Tensor>& bias,
                        int64_t act) {
    ctx->saved_data["act"] = act;
    ctx->save_for_backward({x, or_undefined(bias)});
    return bias_act_fwd(x.contiguous(), bias, act);
  }
  static tensor_list backward(AutogradContext* ctx, tensor_list grads) {
    const variable_list saved = ctx->get_saved_variables();
    auto [dx, db] = bias_act_bwd(grads[0].contiguous(), saved[0].contiguous(), opt(saved[1]),
                                 ctx->saved_data["act"].toInt());
    return {dx, saved[1].defined() ? db : Tensor(), Tensor()};
  }
};

struct BiasDropoutAddFn : public Function<BiasDropoutAddFn> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const optional<Tensor>& bias,
                        const optional<Tensor>& residual, double p) {
    Tensor rng = philox_reserve(x.numel());
    ctx->saved_data["p"] = p;
    ctx->saved_data["rng"] = rng;
    ctx->saved_data["bias"] = bias.has_value();
    ctx->saved_data["residual"] = residual.has_value();
    static auto f = op<Tensor(const Tensor&, const optional<Tensor>&, const optional<Tensor>&, double,
                              const Tensor&)>("slapo_b200::bias_dropout_add_fwd");
    return f.call(x.contiguous(), bias,
                  residual.has_value() ? optional<Tensor>(residual->contiguous()) : c10::nullopt, p, rng);
  }
  static tensor_list backward(AutogradContext* ctx, tensor_list grads) {
    const bool has_bias = ctx->saved_data["bias"].toBool();
    Tensor g = grads[0].contiguous();
    static auto f = op<std::tuple<Tensor, Tensor>(const Tensor&, double, const Tensor&, bool)>(
        "slapo_b200::bias_dropout_add_bwd");
    auto [dx, db] = f.call(g, ctx->saved_data["p"].toDouble(), ctx->saved_data["rng"].toTensor(), has_bias);
    return {dx, has_bias ? db : Tensor(), ctx->saved_data["residual"].toBool() ? g : Tensor(), Tensor()};
  }
};

struct LayerNormFn : public Function<LayerNormFn> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& weight,
                        const optional<Tensor>& bias, double eps, bool rms) {
    Tensor x2 = x.contiguous().view({-1, x.size(-1)});
    static auto f = op<std::tuple<Tensor, Tensor, Tensor>(const Tensor&, const Tensor&,
                                                          const optional<Tensor>&, double, bool)>(
        "slapo_b200::layer_norm_fwd");
    auto [y, mean, rstd] = f.call(x2, weight, bias, eps, rms);
    ctx->saved_data["rms"] = rms;
    ctx->saved_data["bias"] = bias.has_value();
    ctx->save_for_backward({x2, weight, mean, rstd});
    return y.view(x.sizes());
  }
  static tensor_list backward(AutogradContext* ctx, tensor_list grads) {
    const variable_list s = ctx->get_saved_variables();
    Tensor g = grads[0].contiguous();
    static auto f = op<std::tuple<Tensor, Tensor, Tensor>(const Tensor&, const Tensor&, const Tensor&,
                                                          const Tensor&, const Tensor&, bool)>(
        "slapo_b200::layer_norm_bwd");
    auto [dx, dw, db] = f.call(g.view({-1, g.size(-1)}), s[0], s[1], s[2], s[3],
                               ctx->saved_data["rms"].toBool());
    return {dx.view(g.sizes()), dw, ctx->saved_data["bias"].toBool() ? db : Tensor(), Tensor(), Tensor()};
  }
};

// z = dropout(x + bias) + residual ; y = LayerNorm(z) ; returns (y, z).  An output without a
// consumer has no gradient: nothing is filled with zeros or read for it.
struct DropoutAddNormFn : public Function<DropoutAddNormFn> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const optional<Tensor>& bias,
                               const Tensor& residual, const Tensor& weight,
                               const optional<Tensor>& ln_bias, double p, double eps) {
    ctx->set_materialize_grads(false);
    const int64_t cols = x.size(-1);
    optional<Tensor> rng;
    Tensor x2 = x.contiguous().view({-1, cols}), r2 = residual.contiguous().view({-1, cols});
    if (p > 0.0) rng = philox_reserve(x.numel());
    static auto f = op<std::tuple<Tensor, Tensor, Tensor, Tensor>(
        const Tensor&, const optional<Tensor>&, const Tensor&, const Tensor&, const optional<Tensor>&,
        double, double, const optional<Tensor>&)>("slapo_b200::dropout_add_ln_fwd");
    auto [y, z, mean, rstd] = f.call(x2, bias, r2, weight, ln_bias, p, eps, rng);
    ctx->saved_data["p"] = p;
    if (rng.has_value()) ctx->saved_data["rng"] = *rng;
    ctx->saved_data["bias"] = bias.has_value();
    ctx->saved_data["ln_bias"] = ln_bias.has_value();
    ctx->saved_data["shape"] = x.sizes().vec();
    ctx->save_for_backward({z, weight, mean, rstd});
    return {y.view(x.sizes()), z.view(x.sizes())};
  }
  static tensor_list backward(AutogradContext* ctx, tensor_list grads) {
    tensor_list out(7);
    if (!grads[0].defined() && !grads[1].defined()) return out;
    const variable_list s = ctx->get_saved_variables();
    const std::vector<int64_t> shape = ctx->saved_data["shape"].toIntVector();
    const int64_t cols = shape.back();
    Tensor gy = grads[0].defined() ? grads[0].contiguous().view({-1, cols}) : at::zeros_like(s[0]);
    optional<Tensor> gz, rng;
    if (grads[1].defined()) gz = grads[1].contiguous().view({-1, cols});
    const double p = ctx->saved_data["p"].toDouble();
    if (p > 0.0) rng = ctx->saved_data["rng"].toTensor();
    const bool has_bias = ctx->saved_data["bias"].toBool();
    static auto f = op<std::tuple<Tensor, Tensor, Tensor, Tensor, Tensor>(
        const Tensor&, const optional<Tensor>&, const Tensor&, const Tensor&, const Tensor&,
        const Tensor&, double, const optional<Tensor>&, bool)>("slapo_b200::dropout_add_ln_bwd");
    auto [dx, dres, dw, db, dbias] = f.call(gy, gz, s[0], s[1], s[2], s[3], p, rng, has_bias);
    out[0] = dx.view(shape);
    if (has_bias) out[1] = dbias;
    out[2] = dres.view(shape);
    out[3] = dw;
    if (ctx->saved_data["ln_bias"].toBool()) out[4] = db;
    return out;
  }
};

// ------------------------------------------------------------------------ //
using FlashFwd = std::tuple<Tensor, Tensor>(const Tensor&, const Tensor&, const Tensor&,
                                            const optional<Tensor>&, const optional<Tensor>&, bool,
                                            double, double, const optional<Tensor>&);
using FlashBwd = std::tuple<Tensor, Tensor, Tensor, Tensor>(
    const Tensor&, const Tensor&, const Tensor&, const Tensor&, const Tensor&, const Tensor&,
    const optional<Tensor>&, const optional<Tensor>&, bool, double, double, const optional<Tensor>&,
    bool, int64_t);

// Attention on separate q, k, v [B, S, H, D] (q only given: the packed [B, S, H, 3, D], read in
// place through strided views and its gradient written into one tensor of that layout).
struct FlashFn : public Function<FlashFn> {
  static Tensor forward(AutogradContext* ctx, const Tensor& q_or_qkv, const optional<Tensor>& k,
                        const optional<Tensor>& v, const optional<Tensor>& key_bias,
                        const optional<Tensor>& rel, bool causal, double scale, double p) {
    const bool packed = !k.has_value();
    const Tensor q = packed ? q_or_qkv.select(3, 0) : q_or_qkv;
    const Tensor kk = packed ? q_or_qkv.select(3, 1) : *k, vv = packed ? q_or_qkv.select(3, 2) : *v;
    optional<Tensor> rng;
    if (p > 0.0) rng = philox_reserve(q.size(0) * q.size(2) * q.size(1) * kk.size(1));
    static auto f = op<FlashFwd>("slapo_b200::flash_attn_fwd");
    auto [out, lse] = f.call(q, kk, vv, key_bias, rel, causal, scale, p, rng);
    ctx->save_for_backward({q_or_qkv, or_undefined(k), or_undefined(v), out, lse,
                            or_undefined(key_bias), or_undefined(rel)});
    ctx->saved_data["causal"] = causal;
    ctx->saved_data["scale"] = scale;
    ctx->saved_data["p"] = p;
    if (rng.has_value()) ctx->saved_data["rng"] = *rng;
    return out;
  }
  static tensor_list backward(AutogradContext* ctx, tensor_list grads) {
    const variable_list s = ctx->get_saved_variables();
    const bool packed = !s[1].defined();
    const Tensor q = packed ? s[0].select(3, 0) : s[0];
    const Tensor k = packed ? s[0].select(3, 1) : s[1], v = packed ? s[0].select(3, 2) : s[2];
    optional<Tensor> rng;
    const double p = ctx->saved_data["p"].toDouble();
    if (p > 0.0) rng = ctx->saved_data["rng"].toTensor();
    static auto f = op<FlashBwd>("slapo_b200::flash_attn_bwd");
    auto [dq, dk, dv, drel] =
        f.call(grads[0].contiguous(), q, k, v, s[3], s[4], opt(s[5]), opt(s[6]),
               ctx->saved_data["causal"].toBool(), ctx->saved_data["scale"].toDouble(), p, rng, packed, /*keep_words=*/0);
    tensor_list out(8);
    out[0] = dq;
    if (!packed) {
      out[1] = dk;
      out[2] = dv;
    }
    if (s[6].defined()) out[4] = drel;
    return out;
  }
};

// T5's relative-position table by distance, [buckets, H] -> [H, n] fp32, and the sum over the
// distances of each bucket: linear maps, each the other's derivative (of any order).
struct RelBiasFn : public Function<RelBiasFn> {
  static Tensor forward(AutogradContext* ctx, const Tensor& table, const Tensor& buckets);
  static tensor_list backward(AutogradContext* ctx, tensor_list grads);
};
struct RelBiasSumFn : public Function<RelBiasSumFn> {
  static Tensor forward(AutogradContext* ctx, const Tensor& grad, const Tensor& buckets,
                        const Tensor& table) {
    ctx->save_for_backward({buckets});
    static auto f = op<Tensor(const Tensor&, const Tensor&, const Tensor&)>("slapo_b200::rel_bias_bwd");
    return f.call(grad.contiguous(), buckets, table);
  }
  static tensor_list backward(AutogradContext* ctx, tensor_list grads) {
    return {RelBiasFn::apply(grads[0], ctx->get_saved_variables()[0]), Tensor(), Tensor()};
  }
};
Tensor RelBiasFn::forward(AutogradContext* ctx, const Tensor& table, const Tensor& buckets) {
  ctx->save_for_backward({table, buckets});
  static auto f = op<Tensor(const Tensor&, const Tensor&)>("slapo_b200::rel_bias_fwd");
  return f.call(table.contiguous(), buckets);
}
tensor_list RelBiasFn::backward(AutogradContext* ctx, tensor_list grads) {
  const variable_list s = ctx->get_saved_variables();
  return {RelBiasSumFn::apply(grads[0], s[1], s[0].detach()), Tensor()};
}

// ------------------------------------------------------------------------ //
// A bias that starts anywhere, as the kernels read it: 16 bytes at a time.  (A copy that is differentiated.)
Tensor aligned(const Tensor& bias) {
  return bias.is_cuda() && reinterpret_cast<uintptr_t>(bias.data_ptr()) % 16 != 0 ? bias.clone() : bias;
}
optional<Tensor> aligned(const optional<Tensor>& bias) {
  return bias.has_value() && bias->defined() ? optional<Tensor>(aligned(*bias)) : c10::nullopt;
}

Tensor linear(const Tensor& x, const Tensor& weight, const optional<Tensor>& bias_in, int64_t act,
              bool transposed) {
  const optional<Tensor> bias = aligned(bias_in);
  const bool keep = at::GradMode::is_enabled() &&
                    (x.requires_grad() || weight.requires_grad() || (bias.has_value() && bias->requires_grad()));
  return LinearFn::apply(x, weight, bias, act, transposed, keep);
}
Tensor mlp(const Tensor& x, const Tensor& w1, const Tensor& b1, const Tensor& w2, const Tensor& b2,
           int64_t act, double p) {
  TORCH_CHECK(w1.dim() == 2 && w2.dim() == 2 && x.dim() >= 1 && x.size(-1) == w1.size(1) &&
                  w2.size(1) == w1.size(0) && b1.numel() == w1.size(0) && b2.numel() == w2.size(0),
              "mlp: x [.., in], w1 [inner, in], b1 [inner], w2 [out, inner] and b2 [out] required");
  for (const Tensor* t : {&w1, &b1, &w2, &b2})
    TORCH_CHECK(t->device() == x.device() && t->scalar_type() == x.scalar_type() && t->stride(-1) == 1,
                "mlp: contiguous parameters of x's type and device required");
  const bool keep = at::GradMode::is_enabled() && (x.requires_grad() || w1.requires_grad() || b1.requires_grad() ||
                                                   w2.requires_grad() || b2.requires_grad());
  return MlpFn::apply(x, w1, aligned(b1), w2, aligned(b2), act, p, keep);
}
Tensor bias_act(const Tensor& x, const optional<Tensor>& bias, int64_t act) {
  return BiasActFn::apply(x, aligned(bias), act);
}
Tensor bias_dropout_add(const Tensor& x, const optional<Tensor>& bias, const optional<Tensor>& residual,
                        double p) {
  return BiasDropoutAddFn::apply(x, aligned(bias), residual, p);
}
Tensor norm(const Tensor& x, const Tensor& weight, const optional<Tensor>& bias, double eps, bool rms) {
  return LayerNormFn::apply(x, weight, bias, eps, rms);
}
std::tuple<Tensor, Tensor> dropout_add_norm(const Tensor& x, const optional<Tensor>& bias,
                                            const Tensor& residual, const Tensor& weight,
                                            const optional<Tensor>& ln_bias, double p, double eps) {
  variable_list r = DropoutAddNormFn::apply(x, aligned(bias), residual, weight, ln_bias, p, eps);
  return {r[0], r[1]};
}
Tensor flash(const Tensor& q, const optional<Tensor>& k, const optional<Tensor>& v,
             const optional<Tensor>& key_bias, const optional<Tensor>& rel, bool causal, double scale,
             double p) {
  return FlashFn::apply(q, k, v, key_bias, rel, causal, scale, p);
}

Tensor rel_bias(const Tensor& table, const Tensor& buckets) { return RelBiasFn::apply(table, buckets); }

}  // namespace

void register_autograd_ops(torch::Library& m) {
  m.def("linear(Tensor x, Tensor weight, Tensor? bias, int act, bool transposed) -> Tensor", &linear);
  m.def("mlp(Tensor x, Tensor w1, Tensor b1, Tensor w2, Tensor b2, int act, float p) -> Tensor", &mlp);
  m.def("bias_act(Tensor x, Tensor? bias, int act) -> Tensor", &bias_act);
  m.def("bias_dropout_add(Tensor x, Tensor? bias, Tensor? residual, float p) -> Tensor",
        &bias_dropout_add);
  m.def("norm(Tensor x, Tensor weight, Tensor? bias, float eps, bool rms) -> Tensor", &norm);
  m.def("dropout_add_norm(Tensor x, Tensor? bias, Tensor residual, Tensor weight, Tensor? ln_bias, float p, float eps) -> (Tensor, Tensor)",
        &dropout_add_norm);
  m.def("rel_bias(Tensor table, Tensor buckets) -> Tensor", &rel_bias);
  m.def("flash(Tensor q, Tensor? k, Tensor? v, Tensor? key_bias, Tensor? rel, bool causal, float scale, float p) -> Tensor",
        &flash);
}
