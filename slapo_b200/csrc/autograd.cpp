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
// y = x W^T + b (act < 0) or its ReLU: three GEMMs, none of them transposing an operand in
// memory.  The bias rides in the forward GEMM's epilogue and so does ReLU, whose derivative the
// backward reads off the output (y > 0).  `transposed`: W is stored [in, out] (x W + b).
struct LinearFn : public Function<LinearFn> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& weight,
                        const optional<Tensor>& bias, int64_t act, bool transposed) {
    Tensor x2 = rows_of(x);
    Tensor y = gemm(x2, weight, bias, act, false, transposed, false);
    ctx->saved_data["act"] = act;
    ctx->saved_data["transposed"] = transposed;
    ctx->saved_data["bias"] = bias.has_value();
    ctx->saved_data["shape"] = x.sizes().vec();
    ctx->save_for_backward({x2, weight, act >= 0 ? y : Tensor()});
    return y.view(with_last(x.sizes(), weight.size(transposed ? 1 : 0)));
  }
  static tensor_list backward(AutogradContext* ctx, tensor_list grads) {
    const variable_list saved = ctx->get_saved_variables();
    const Tensor &x2 = saved[0], &weight = saved[1], &y = saved[2];
    const int64_t act = ctx->saved_data["act"].toInt();
    const bool transposed = ctx->saved_data["transposed"].toBool();
    const bool has_bias = ctx->saved_data["bias"].toBool();
    Tensor dy = rows_of(grads[0]);
    Tensor dx, dw, db;
    if (act >= 0) {
      // relu'(z) = (y > 0): the saved output stands in for the pre-activation
      static auto f = op<std::tuple<Tensor, Tensor>(const Tensor&, const Tensor&, int64_t)>(
          "slapo_b200::act_bwd_colsum");
      std::tie(dy, db) = f.call(dy.contiguous(), y, act);
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
    return {dx, dw, has_bias ? db : Tensor(), Tensor(), Tensor()};
  }
};

struct BiasActFn : public Function<BiasActFn> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const optional<Tensor>& bias,
                        int64_t act) {
    ctx->saved_data["act"] = act;
    ctx->save_for_backward({x, or_undefined(bias)});
    static auto f = op<Tensor(const Tensor&, const optional<Tensor>&, int64_t)>("slapo_b200::bias_act_fwd");
    return f.call(x.contiguous(), bias, act);
  }
  static tensor_list backward(AutogradContext* ctx, tensor_list grads) {
    const variable_list saved = ctx->get_saved_variables();
    static auto f = op<std::tuple<Tensor, Tensor>(const Tensor&, const Tensor&, const optional<Tensor>&,
                                                  int64_t)>("slapo_b200::bias_act_bwd");
    auto [dx, db] = f.call(grads[0].contiguous(), saved[0].contiguous(), opt(saved[1]),
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
Tensor linear(const Tensor& x, const Tensor& weight, const optional<Tensor>& bias, int64_t act,
              bool transposed) {
  return LinearFn::apply(x, weight, bias, act, transposed);
}
Tensor bias_act(const Tensor& x, const optional<Tensor>& bias, int64_t act) {
  return BiasActFn::apply(x, bias, act);
}
Tensor bias_dropout_add(const Tensor& x, const optional<Tensor>& bias, const optional<Tensor>& residual,
                        double p) {
  return BiasDropoutAddFn::apply(x, bias, residual, p);
}
Tensor norm(const Tensor& x, const Tensor& weight, const optional<Tensor>& bias, double eps, bool rms) {
  return LayerNormFn::apply(x, weight, bias, eps, rms);
}
std::tuple<Tensor, Tensor> dropout_add_norm(const Tensor& x, const optional<Tensor>& bias,
                                            const Tensor& residual, const Tensor& weight,
                                            const optional<Tensor>& ln_bias, double p, double eps) {
  variable_list r = DropoutAddNormFn::apply(x, bias, residual, weight, ln_bias, p, eps);
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
