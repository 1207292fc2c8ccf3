// torch bindings of the tcgen05 flash-attention kernels.
#include <ATen/ATen.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/library.h>

#include "kernels.h"

int* slapo_status_ptr(int device);
slapo::PhiloxArgs unpack_rng(const c10::optional<at::Tensor>& rng);      // bindings.cpp

namespace {

using at::Tensor;
using c10::optional;

void check_bshd(const Tensor& t, const char* name) {
  TORCH_CHECK(t.is_cuda() && t.dim() == 4, name, " must be a CUDA tensor [B, S, H, D]");
  TORCH_CHECK(t.stride(3) == 1, name, ": D must be contiguous");
  TORCH_CHECK(t.stride(0) % 8 == 0 && t.stride(1) % 8 == 0 && t.stride(2) % 8 == 0,
              name, ": strides must be multiples of 8 elements");
  TORCH_CHECK(reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0, name, " must be 16-byte aligned");
}

const float* opt_f32(const optional<Tensor>& t, const char* name) {
  if (!t.has_value() || !t->defined()) return nullptr;
  TORCH_CHECK(t->is_cuda() && t->scalar_type() == at::kFloat && t->is_contiguous(), name,
              " must be a contiguous fp32 CUDA tensor");
  return t->data_ptr<float>();
}

std::tuple<Tensor, Tensor> flash_attn_fwd(const Tensor& q, const Tensor& k, const Tensor& v,
                                          const optional<Tensor>& kbias,
                                          const optional<Tensor>& rel, bool causal, double scale,
                                          double p_drop, const optional<Tensor>& rng) {
  check_bshd(q, "q"); check_bshd(k, "k"); check_bshd(v, "v");
  TORCH_CHECK(q.scalar_type() == at::kBFloat16 || q.scalar_type() == at::kHalf, "bf16/fp16 only");
  TORCH_CHECK(k.scalar_type() == q.scalar_type() && v.scalar_type() == q.scalar_type());
  c10::cuda::CUDAGuard guard(q.device());
  const int B = q.size(0), Sq = q.size(1), H = q.size(2), D = q.size(3), Sk = k.size(1);
  TORCH_CHECK(k.size(0) == B && k.size(2) == H && k.size(3) == D && v.sizes() == k.sizes());
  if (kbias.has_value() && kbias->defined()) TORCH_CHECK(kbias->numel() == (int64_t)B * Sk);
  if (rel.has_value() && rel->defined()) TORCH_CHECK(rel->numel() == (int64_t)H * (Sq + Sk - 1));
  Tensor o = at::empty({B, Sq, H, D}, q.options());
  Tensor lse = at::empty({B, H, Sq}, q.options().dtype(at::kFloat));
  const int64_t qs[3] = {q.stride(0), q.stride(1), q.stride(2)};
  const int64_t ks[3] = {k.stride(0), k.stride(1), k.stride(2)};
  const int64_t vs[3] = {v.stride(0), v.stride(1), v.stride(2)};
  // few row tiles: the keys are split over work items, whose shares a second kernel combines
  const int64_t splits = slapo::flash_fwd_splits(B, H, Sq, Sk, D);
  Tensor scratch;
  if (splits > 1)
    scratch = at::empty({splits * B * H * Sq * (D + 2)}, q.options().dtype(at::kFloat));
  int rc = slapo::launch_flash_fwd(
      q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), lse.data_ptr<float>(),
      splits > 1 ? scratch.data_ptr<float>() : nullptr,
      opt_f32(kbias, "key bias"), opt_f32(rel, "relative bias"), B, H, Sq, Sk, D, qs, ks, vs,
      static_cast<float>(scale), causal ? 1 : 0, static_cast<float>(p_drop), unpack_rng(rng),
      q.scalar_type() == at::kBFloat16, slapo_status_ptr(q.get_device()),
      at::cuda::getCurrentCUDAStream().stream());
  TORCH_CHECK(rc == 0, "flash_attn_fwd: launch refused (code ", rc, ")");
  return {o, lse};
}

// keep_words: see flash_bwd_plan (0: its default)
std::tuple<Tensor, Tensor, Tensor, Tensor> flash_attn_bwd(
    const Tensor& dout, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& o,
    const Tensor& lse, const optional<Tensor>& kbias, const optional<Tensor>& rel, bool causal,
    double scale, double p_drop, const optional<Tensor>& rng, bool packed_qkv, int64_t keep_words) {
  check_bshd(q, "q"); check_bshd(k, "k"); check_bshd(v, "v");
  TORCH_CHECK(dout.is_contiguous() && o.is_contiguous(), "dout and out must be contiguous");
  c10::cuda::CUDAGuard guard(q.device());
  const int B = q.size(0), Sq = q.size(1), H = q.size(2), D = q.size(3), Sk = k.size(1);
  // packed_qkv: q, k, v are the slices [..., 0/1/2, :] of one [B, S, H, 3, D]
  // projection output; the gradients are written into one tensor of that
  // layout so that autograd needs no concatenation
  Tensor dq, dk, dv, dqkv;
  int64_t row_stride = D;
  if (packed_qkv) {
    TORCH_CHECK(Sq == Sk, "packed QKV needs equal query and key lengths");
    dqkv = at::empty({B, Sq, H, 3, D}, q.options());
    dq = dqkv.select(3, 0);
    dk = dqkv.select(3, 1);
    dv = dqkv.select(3, 2);
    row_stride = 3 * D;
  } else {
    dq = at::empty({B, Sq, H, D}, q.options());
    dk = at::empty({B, Sk, H, D}, q.options());
    dv = at::empty({B, Sk, H, D}, q.options());
  }
  const bool has_bias = kbias.has_value() && kbias->defined();
  const bool has_rel = rel.has_value() && rel->defined();
  const slapo::FlashBwdPlan plan = slapo::flash_bwd_plan(
      B, H, Sq, Sk, D, packed_qkv, causal, has_bias, has_rel, static_cast<float>(p_drop), keep_words);
  Tensor scratch = at::empty({plan.total()}, q.options().dtype(at::kFloat));
  Tensor drel;
  if (has_rel) drel = at::zeros_like(*rel);
  else drel = at::empty({0}, q.options().dtype(at::kFloat));
  const int64_t qs[3] = {q.stride(0), q.stride(1), q.stride(2)};
  const int64_t ks[3] = {k.stride(0), k.stride(1), k.stride(2)};
  const int64_t vs[3] = {v.stride(0), v.stride(1), v.stride(2)};
  int rc = slapo::launch_flash_bwd(
      q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), dout.data_ptr(),
      lse.data_ptr<float>(), plan, scratch.data_ptr<float>(), dq.data_ptr(), dk.data_ptr(),
      dv.data_ptr(), row_stride, row_stride, opt_f32(kbias, "key bias"),
      opt_f32(rel, "relative bias"),
      has_rel ? drel.data_ptr<float>() : nullptr, B, H, Sq, Sk, D, qs, ks, vs,
      static_cast<float>(scale), causal ? 1 : 0, static_cast<float>(p_drop), unpack_rng(rng),
      q.scalar_type() == at::kBFloat16, slapo_status_ptr(q.get_device()),
      at::cuda::getCurrentCUDAStream().stream());
  TORCH_CHECK(rc == 0, "flash_attn_bwd: launch refused (code ", rc, ")");
  if (packed_qkv) return {dqkv, dk, dv, drel};
  return {dq, dk, dv, drel};
}

Tensor flash_attn_dropout_mask(int64_t B, int64_t H, int64_t Sq, int64_t Sk, double p_drop,
                               const Tensor& rng) {
  Tensor mask = at::empty({B, H, Sq, Sk}, at::TensorOptions().dtype(at::kByte).device(at::kCUDA));
  slapo::launch_flash_dropout_mask(mask.data_ptr<uint8_t>(), B, H, Sq, Sk,
                                   static_cast<float>(p_drop), unpack_rng(rng),
                                   at::cuda::getCurrentCUDAStream().stream());
  return mask;
}

// Whether one launch takes the four tensors: plain CUDA tensors outside of autograd and of functorch
// / forward-mode transforms, one type and device, contiguous caches, 16-byte aligned heads.
bool kv_append_takes(const Tensor* const (&past)[2], const Tensor* const (&fresh)[2]) {
  static constexpr c10::DispatchKeySet kWrapped({c10::DispatchKey::FuncTorchBatched,
                                                 c10::DispatchKey::FuncTorchGradWrapper,
                                                 c10::DispatchKey::Functionalize, c10::DispatchKey::Python,
                                                 c10::DispatchKey::ZeroTensor, c10::DispatchKey::Negative});
  const Tensor& k = *fresh[0];
  const auto dtype = k.scalar_type();
  if (dtype != at::kBFloat16 && dtype != at::kHalf && dtype != at::kFloat) return false;
  const bool grad = at::GradMode::is_enabled();
  for (const Tensor* t : {past[0], past[1], fresh[0], fresh[1]}) {
    if (t->key_set().has_any(kWrapped) || t->layout() != at::kStrided || !t->is_cuda() || t->dim() != 4 ||
        t->scalar_type() != dtype || t->get_device() != k.get_device() || (grad && t->requires_grad()) ||
        t->_fw_grad(/*level=*/0).defined() || reinterpret_cast<uintptr_t>(t->data_ptr()) % 16 != 0)
      return false;
  }
  const int64_t e = k.element_size();
  for (int i = 0; i < 2; ++i) {
    const Tensor &p = *past[i], &f = *fresh[i];
    if (f.sizes() != k.sizes() || p.sizes() != past[0]->sizes() || !p.is_contiguous() || f.stride(3) != 1)
      return false;
    for (int d = 0; d < 3; ++d)
      if (f.stride(d) * e % 16 != 0) return false;
  }
  const Tensor& p = *past[0];
  return k.numel() > 0 && p.size(0) == k.size(0) && p.size(2) == k.size(2) && p.size(3) == k.size(3) &&
         k.size(3) * e % 16 == 0 && k.size(0) <= 65535;
}

// Key / value caches [B, S, H, D] followed by the new tokens [B, n, H, D] (slices of a packed
// projection are read in place): two new tensors, by one launch where kv_append_takes says so.  The
// checks live here because they cost a Python caller more than the launch (15 us against 9 for both).
std::tuple<Tensor, Tensor> append_kv(const Tensor& past_k, const Tensor& past_v, const Tensor& k,
                                     const Tensor& v) {
  const Tensor* const past[2] = {&past_k, &past_v};
  const Tensor* const fresh[2] = {&k, &v};
  if (!kv_append_takes(past, fresh)) return {at::cat({past_k, k}, 1), at::cat({past_v, v}, 1)};
  c10::cuda::CUDAGuard guard(k.device());
  const int64_t B = k.size(0), n = k.size(1), H = k.size(2), D = k.size(3), len = past_k.size(1);
  const int64_t e = k.element_size();
  Tensor out[2];
  const void* past_ptr[2];
  const void* fresh_ptr[2];
  void* out_ptr[2];
  int64_t strides[2][3];
  for (int i = 0; i < 2; ++i) {
    for (int d = 0; d < 3; ++d) strides[i][d] = fresh[i]->stride(d) * e;
    out[i] = at::empty({B, len + n, H, D}, k.options());
    past_ptr[i] = past[i]->data_ptr();
    fresh_ptr[i] = fresh[i]->data_ptr();
    out_ptr[i] = out[i].data_ptr();
  }
  slapo::launch_kv_append(past_ptr, fresh_ptr, out_ptr, B, len, n, H, D * e, strides,
                          at::cuda::getCurrentCUDAStream().stream());
  return {out[0], out[1]};
}

// T5's table [buckets, H] by distance, and its gradient (see rel_bias.cu)
int rel_dtype(const Tensor& t) {
  return t.scalar_type() == at::kBFloat16 ? 0 : (t.scalar_type() == at::kHalf ? 1 : 2);
}

// (indexes outside of the table are the kernels' to check)
void check_rel(const Tensor& table, const Tensor& buckets) {
  TORCH_CHECK(table.is_cuda() && table.dim() == 2 && table.is_contiguous() &&
                  (rel_dtype(table) < 2 || table.scalar_type() == at::kFloat),
              "rel_bias: a contiguous [buckets, H] CUDA table of fp32, bf16 or fp16 required");
  TORCH_CHECK(buckets.is_cuda() && buckets.dim() == 1 && buckets.is_contiguous() &&
                  buckets.scalar_type() == at::kLong && buckets.get_device() == table.get_device(),
              "rel_bias: contiguous int64 buckets on the table's device required");
  TORCH_CHECK(table.size(0) <= INT_MAX && table.size(1) <= 65535 && buckets.numel() <= INT_MAX - 256,
              "rel_bias: table or distances too large");
}

// int64 [sq + sk - 1]: the buckets of the distances -(sk - 1) .. sq - 1, on the device of `table`
Tensor rel_buckets(const Tensor& table, int64_t sq, int64_t sk, bool bidirectional, double inv_exact,
                   double inv_log) {
  TORCH_CHECK(table.is_cuda() && table.dim() == 2 && sq > 0 && sk > 0 && sq + sk <= INT_MAX - 256 &&
                  table.size(0) >= (bidirectional ? 4 : 2) && table.size(0) <= INT_MAX,
              "rel_buckets: a [buckets, H] CUDA table and positive lengths required");
  c10::cuda::CUDAGuard guard(table.device());
  const int n = static_cast<int>(sq + sk - 1);
  Tensor out = at::empty({n}, table.options().dtype(at::kLong));
  slapo::launch_rel_buckets(out.data_ptr<int64_t>(), n, static_cast<int>(sk - 1), static_cast<int>(table.size(0)),
                            bidirectional ? 1 : 0, static_cast<float>(inv_exact), static_cast<float>(inv_log),
                            at::cuda::getCurrentCUDAStream().stream());
  return out;
}

Tensor rel_bias_fwd(const Tensor& table, const Tensor& buckets) {
  check_rel(table, buckets);
  c10::cuda::CUDAGuard guard(table.device());
  const int n = static_cast<int>(buckets.numel()), H = static_cast<int>(table.size(1));
  Tensor out = at::empty({H, n}, table.options().dtype(at::kFloat));
  slapo::launch_rel_bias_fwd(table.data_ptr(), buckets.data_ptr<int64_t>(), out.data_ptr<float>(), n, H,
                             static_cast<int>(table.size(0)), rel_dtype(table),
                             at::cuda::getCurrentCUDAStream().stream());
  return out;
}

// `table`: only its sizes and type
Tensor rel_bias_bwd(const Tensor& grad, const Tensor& buckets, const Tensor& table) {
  Tensor dtable = at::empty(table.sizes(), table.options(), at::MemoryFormat::Contiguous);
  check_rel(dtable, buckets);
  TORCH_CHECK(grad.is_cuda() && grad.is_contiguous() && grad.scalar_type() == at::kFloat &&
                  grad.get_device() == table.get_device() && grad.dim() == 2 &&
                  grad.size(0) == table.size(1) && grad.size(1) == buckets.numel(),
              "rel_bias: a contiguous fp32 [H, distances] gradient on the table's device required");
  c10::cuda::CUDAGuard guard(table.device());
  slapo::launch_rel_bias_bwd(grad.data_ptr<float>(), buckets.data_ptr<int64_t>(), dtable.data_ptr(),
                             static_cast<int>(buckets.numel()), static_cast<int>(table.size(1)),
                             static_cast<int>(table.size(0)), rel_dtype(table),
                             at::cuda::getCurrentCUDAStream().stream());
  return dtable;
}

}  // namespace

void register_attn_ops(torch::Library& m) {
  m.def("flash_attn_fwd(Tensor q, Tensor k, Tensor v, Tensor? kbias, Tensor? rel, bool causal, float scale, float p_drop, Tensor? rng) -> (Tensor, Tensor)",
        &flash_attn_fwd);
  m.def("flash_attn_bwd(Tensor dout, Tensor q, Tensor k, Tensor v, Tensor o, Tensor lse, Tensor? kbias, Tensor? rel, bool causal, float scale, float p_drop, Tensor? rng, bool packed_qkv, int keep_words=0) -> (Tensor, Tensor, Tensor, Tensor)",
        &flash_attn_bwd);
  m.def("append_kv(Tensor past_k, Tensor past_v, Tensor k, Tensor v) -> (Tensor, Tensor)", &append_kv);
  m.def("rel_buckets(Tensor table, int sq, int sk, bool bidirectional, float inv_exact, float inv_log) -> Tensor",
        &rel_buckets);
  m.def("rel_bias_fwd(Tensor table, Tensor buckets) -> Tensor", &rel_bias_fwd);
  m.def("rel_bias_bwd(Tensor grad, Tensor buckets, Tensor table) -> Tensor", &rel_bias_bwd);
  m.def("flash_attn_dropout_mask(int B, int H, int Sq, int Sk, float p_drop, Tensor rng) -> Tensor",
        &flash_attn_dropout_mask);
}
