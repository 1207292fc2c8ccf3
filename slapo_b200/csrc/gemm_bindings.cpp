// torch bindings of the tcgen05 GEMM family.
#include <ATen/ATen.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/library.h>

#include "kernels.h"

slapo::PhiloxArgs unpack_rng(const c10::optional<at::Tensor>& rng);      // bindings.cpp

namespace {

using at::Tensor;

// One int32 error word per device, written by kernels whose bounded waits ran
// out.  Read (with a device sync) through device_status().
Tensor& status_word(int device) {
  static std::vector<Tensor> words(64);
  if (!words[device].defined()) {
    words[device] = at::zeros({4}, at::TensorOptions().dtype(at::kInt).device(at::kCUDA, device));
  }
  return words[device];
}

int64_t device_status() {
  int dev = at::cuda::current_device();
  Tensor& w = status_word(dev);
  int64_t v = w.cpu().data_ptr<int>()[0];
  if (v != 0) w.zero_();
  return v;
}

// fp32 scratch of the split-K pair GEMM (one slice per split; contents do not matter), one per
// device, grown on demand.  All GEMMs of a device run on one stream at a time.
Tensor& split_scratch(int device, int64_t floats) {
  static std::vector<Tensor> s(64);
  if (!s[device].defined() || s[device].numel() < floats)
    s[device] = at::empty({floats}, at::TensorOptions().dtype(at::kFloat).device(at::kCUDA, device));
  return s[device];
}

// impl: 0 = pick (CTA-pair kernel when the problem has at least one pair tile, else the
// single-CTA kernel), 1 = single-CTA kernel, 2 = CTA-pair kernel or fail.
// split_k: allow several CTA pairs per output tile (weight gradients).
// the word itself (device tensor), for callers that copy it out asynchronously
Tensor device_status_tensor() { return status_word(at::cuda::current_device()); }

// A bias [N] as the kernels read it, 16 bytes at a time, or null
const void* bias_words(const c10::optional<Tensor>& bias, const Tensor& a, int N) {
  if (!bias.has_value() || !bias->defined()) return nullptr;
  TORCH_CHECK(bias->device() == a.device() && bias->scalar_type() == a.scalar_type() && bias->numel() == N &&
                  bias->is_contiguous(),
              "gemm: bias must be a contiguous [N] tensor of the operands' type and device");
  return bias->data_ptr();
}

Tensor gemm_out(const Tensor& a, const Tensor& b, const c10::optional<Tensor>& bias, int64_t act,
                bool a_mn, bool b_mn, const c10::optional<Tensor>& out,
                const c10::optional<Tensor>& pre_act, int64_t impl, bool split_k) {
  TORCH_CHECK(a.is_cuda() && b.device() == a.device(), "gemm: tensors on one CUDA device required");
  TORCH_CHECK(a.dim() == 2 && b.dim() == 2, "gemm: 2-D operands required");
  TORCH_CHECK(a.scalar_type() == b.scalar_type() &&
                  (a.scalar_type() == at::kBFloat16 || a.scalar_type() == at::kHalf),
              "gemm: bf16 or fp16 operands of the same type required");
  TORCH_CHECK(a.stride(1) == 1 && b.stride(1) == 1, "gemm: innermost dimension must be contiguous");
  c10::cuda::CUDAGuard guard(a.device());
  const int M = static_cast<int>(a_mn ? a.size(1) : a.size(0));
  const int K = static_cast<int>(a_mn ? a.size(0) : a.size(1));
  const int N = static_cast<int>(b_mn ? b.size(1) : b.size(0));
  const int Kb = static_cast<int>(b_mn ? b.size(0) : b.size(1));
  TORCH_CHECK(K == Kb, "gemm: contraction sizes differ: ", K, " vs ", Kb);
  Tensor c;
  if (out.has_value() && out->defined()) {
    c = *out;
    TORCH_CHECK(c.dim() == 2 && c.size(0) == M && c.size(1) == N && c.stride(1) == 1 &&
                    c.scalar_type() == a.scalar_type() && c.device() == a.device(),
                "gemm: `out` must be an [M, N] tensor of the operand dtype with contiguous rows");
  } else {
    c = at::empty({M, N}, a.options());
  }
  void* c2 = nullptr;
  if (pre_act.has_value() && pre_act->defined()) {
    TORCH_CHECK(pre_act->sizes() == c.sizes() && pre_act->strides() == c.strides() &&
                    pre_act->scalar_type() == c.scalar_type() && pre_act->device() == c.device(),
                "gemm: `pre_act` must match the output's shape, strides and dtype");
    c2 = pre_act->data_ptr();
  }
  const void* bias_ptr = bias_words(bias, a, N);
  const int dev = a.get_device();
  const bool bf16 = a.scalar_type() == at::kBFloat16;
  auto stream = at::cuda::getCurrentCUDAStream().stream();
  int rc = 5;
  const int splits = split_k && impl != 1 ? slapo::gemm2_splits(M, N, K, N > 128 ? 256 : 128) : 1;
  // a second output and several pairs per tile exist on the pair kernel's default tile only
  slapo::GemmTile tile{impl != 1, 0};
  if (impl == 0 && splits == 1 && c2 == nullptr) {
    if (!a_mn && !b_mn && slapo::gemm_rows_takes(M, N, K)) {
      rc = slapo::launch_gemm_rows(a.data_ptr(), b.data_ptr(), c.data_ptr(), bias_ptr, M, N, K,
                                   static_cast<int>(a.stride(0)), static_cast<int>(b.stride(0)),
                                   static_cast<int>(c.stride(0)), bf16, static_cast<int>(act), stream);
      TORCH_CHECK(rc == 0, "gemm: launch refused (code ", rc,
                  "): sizes must be multiples of 8 and pointers 16-byte aligned");
      return c;
    }
    tile = slapo::gemm_tile(M, N);
  }
  if (tile.pair) {
    float* ws = nullptr;
    if (splits > 1) ws = split_scratch(dev, static_cast<int64_t>(splits) * M * N).data_ptr<float>();
    rc = slapo::launch_gemm2(a.data_ptr(), b.data_ptr(), c.data_ptr(), c2, bias_ptr, M, N, K,
                             static_cast<int>(a.stride(0)), static_cast<int>(b.stride(0)),
                             static_cast<int>(c.stride(0)), a_mn, b_mn, bf16,
                             static_cast<int>(act), tile.bn, ws,
                             status_word(dev).data_ptr<int>(), stream);
    TORCH_CHECK(impl != 2 || rc == 0, "gemm: the CTA-pair kernel refused the launch (code ", rc, ")");
  }
  if (rc == 5) {
    TORCH_CHECK(c2 == nullptr, "gemm: `pre_act` needs a problem of at least one 256 x 128 tile");
    rc = slapo::launch_gemm(a.data_ptr(), b.data_ptr(), c.data_ptr(), bias_ptr, M, N, K,
                            static_cast<int>(a.stride(0)), static_cast<int>(b.stride(0)),
                            static_cast<int>(c.stride(0)), a_mn, b_mn, bf16, static_cast<int>(act),
                            tile.pair ? 0 : tile.bn, status_word(dev).data_ptr<int>(), stream);
  }
  TORCH_CHECK(rc == 0, "gemm: launch refused (code ", rc,
              "): sizes must be multiples of 8 and pointers 16-byte aligned");
  return c;
}

// Operands of a product with an activation in its epilogue, a [M, K] K-major
struct GemmCall {
  const Tensor &a, &w;
  bool b_mn, bf16;
  int M, N, K;
  GemmCall(const Tensor& a_, const Tensor& w_, bool b_mn_) : a(a_), w(w_), b_mn(b_mn_) {
    TORCH_CHECK(a.is_cuda() && w.device() == a.device() && a.dim() == 2 && w.dim() == 2,
                "gemm: 2-D operands on one CUDA device required");
    TORCH_CHECK(a.scalar_type() == w.scalar_type() &&
                    (a.scalar_type() == at::kBFloat16 || a.scalar_type() == at::kHalf),
                "gemm: bf16 or fp16 operands of the same type required");
    TORCH_CHECK(a.stride(1) == 1 && w.stride(1) == 1, "gemm: innermost dimension must be contiguous");
    bf16 = a.scalar_type() == at::kBFloat16;
    M = static_cast<int>(a.size(0));
    K = static_cast<int>(a.size(1));
    N = static_cast<int>(b_mn ? w.size(1) : w.size(0));
    TORCH_CHECK(K == (b_mn ? w.size(0) : w.size(1)), "gemm: contraction sizes differ");
  }
  void run(const Tensor& c, const void* bias, const slapo::GemmEpi& epi) const {
    const int dev = a.get_device();
    auto stream = at::cuda::getCurrentCUDAStream().stream();
    int* status = status_word(dev).data_ptr<int>();
    const int lda = static_cast<int>(a.stride(0)), ldb = static_cast<int>(w.stride(0));
    const slapo::GemmTile tile = slapo::gemm_tile(M, N);
    int rc = 5;
    if (epi.z == nullptr && !b_mn && slapo::gemm_rows_takes(M, N, K))
      rc = slapo::launch_gemm_rows(a.data_ptr(), w.data_ptr(), c.data_ptr(), bias, M, N, K, lda, ldb, N, bf16, -1,
                                   stream, &epi);
    else if (tile.pair)
      rc = slapo::launch_gemm2(a.data_ptr(), w.data_ptr(), c.data_ptr(), epi.c2, bias, M, N, K, lda, ldb, N,
                               false, b_mn, bf16, -1, tile.bn, nullptr, status, stream, &epi);
    if (rc == 5)
      rc = slapo::launch_gemm(a.data_ptr(), w.data_ptr(), c.data_ptr(), bias, M, N, K, lda, ldb, N, false, b_mn,
                              bf16, -1, tile.pair ? 0 : tile.bn, status, stream, &epi);
    TORCH_CHECK(rc == 0, "gemm: launch refused (code ", rc,
                "): sizes must be multiples of 8 and pointers 16-byte aligned");
  }
};

Tensor gemm(const Tensor& a, const Tensor& b, const c10::optional<Tensor>& bias, int64_t act,
            bool a_mn, bool b_mn) {
  return gemm_out(a, b, bias, act, a_mn, b_mn, c10::nullopt, c10::nullopt, 0, false);
}

// act(a w^T + bias) with the activation (0 GeLU, 1 GeLU tanh) in the epilogue, and the value before it
// (empty unless `keep`): the product, or with `sum` product + bias.
std::tuple<Tensor, Tensor> gemm_act_fwd(const Tensor& a, const Tensor& w, const c10::optional<Tensor>& bias,
                                        int64_t act, bool keep, bool sum) {
  TORCH_CHECK(act == 0 || act == 1, "gemm_act_fwd: GeLU only");
  GemmCall g(a, w, false);
  const void* bias_ptr = bias_words(bias, a, g.N);
  c10::cuda::CUDAGuard guard(a.device());
  Tensor y = at::empty({g.M, g.N}, a.options());
  Tensor z = keep ? at::empty({g.M, g.N}, a.options()) : at::empty({0}, a.options());
  slapo::GemmEpi epi{act == 0 ? 1 : 2, sum, keep ? z.data_ptr() : nullptr, nullptr, nullptr};
  g.run(y, bias_ptr, epi);
  return {y, z};
}

// dropout(a w^T + bias) with the decisions of bias_dropout_add_fwd, more than 16 rows and N % 16 == 0
Tensor gemm_dropout_fwd(const Tensor& a, const Tensor& w, const c10::optional<Tensor>& bias, double p,
                        const Tensor& rng) {
  GemmCall g(a, w, false);
  TORCH_CHECK(g.N % 16 == 0 && !slapo::gemm_rows_takes(g.M, g.N, g.K), "gemm_dropout_fwd: N % 16 == 0 and more rows");
  const void* bias_ptr = bias_words(bias, a, g.N);
  c10::cuda::CUDAGuard guard(a.device());
  const slapo::PhiloxArgs state = unpack_rng(rng);
  Tensor y = at::empty({g.M, g.N}, a.options());
  slapo::GemmEpi epi{6, false, nullptr, nullptr, nullptr, &state, static_cast<float>(p)};
  g.run(y, bias_ptr, epi);
  return y;
}

// dz = (dy w) * act'(z) and its column sums: the input gradient of the layer that follows an
// activation, on to that activation's input.  z: for ReLU (act 2) the activation's output.  w is the
// following layer's weight [K, N].
std::tuple<Tensor, Tensor> gemm_act_bwd(const Tensor& dy, const Tensor& w, const Tensor& z, int64_t act) {
  TORCH_CHECK(act >= 0 && act <= 2, "gemm_act_bwd: unknown activation");
  GemmCall g(dy, w, true);
  TORCH_CHECK(z.device() == dy.device() && z.is_contiguous() && z.scalar_type() == dy.scalar_type() && z.dim() == 2 &&
                  z.size(0) == g.M && z.size(1) == g.N,
              "gemm_act_bwd: z must be a contiguous [M, N] tensor of the operand dtype");
  c10::cuda::CUDAGuard guard(dy.device());
  Tensor dz = at::empty({g.M, g.N}, dy.options()), db = at::empty({g.N}, dy.options());
  const int parts = (g.M + 31) / 32;
  Tensor part = at::empty({parts, g.N}, dy.options().dtype(at::kFloat));
  slapo::GemmEpi epi{3 + static_cast<int>(act), false, nullptr, z.data_ptr(), part.data_ptr<float>()};
  g.run(dz, nullptr, epi);
  slapo::launch_colsum_finalize(part.data_ptr<float>(), db.data_ptr(), parts, g.N, g.bf16 ? 0 : 1,
                                at::cuda::getCurrentCUDAStream().stream());
  return {dz, db};
}

}  // namespace

int* slapo_status_ptr(int device) { return status_word(device).data_ptr<int>(); }

void register_gemm_ops(torch::Library& m) {
  m.def("gemm(Tensor a, Tensor b, Tensor? bias, int act, bool a_mn, bool b_mn) -> Tensor", &gemm);
  m.def("gemm_out(Tensor a, Tensor b, Tensor? bias, int act, bool a_mn, bool b_mn, Tensor? out, "
        "Tensor? pre_act, int impl, bool split_k) -> Tensor", &gemm_out);
  m.def("gemm_act_fwd(Tensor a, Tensor w, Tensor? bias, int act, bool keep, bool sum=True) -> (Tensor, Tensor)",
        &gemm_act_fwd);
  m.def("gemm_dropout_fwd(Tensor a, Tensor w, Tensor? bias, float p, Tensor rng) -> Tensor", &gemm_dropout_fwd);
  m.def("gemm_act_bwd(Tensor dy, Tensor w, Tensor z, int act) -> (Tensor, Tensor)",
        &gemm_act_bwd);
  // which tile a product without split K gets: a CTA pair's or one CTA's, and its columns (0: the widest)
  m.def("gemm_tile(int M, int N) -> (bool, int)", [](int64_t M, int64_t N) -> std::tuple<bool, int64_t> {
    const slapo::GemmTile t = slapo::gemm_tile(static_cast<int>(M), static_cast<int>(N));
    return {t.pair, t.bn};
  });
  m.def("gemm2_splits(int M, int N, int K) -> int", [](int64_t M, int64_t N, int64_t K) -> int64_t {
    return slapo::gemm2_splits(static_cast<int>(M), static_cast<int>(N), static_cast<int>(K),
                               N > 128 ? 256 : 128);
  });
  m.def("device_status() -> int", &device_status);
  m.def("device_status_tensor() -> Tensor", &device_status_tensor);
}
