// Launchers that take a PhiloxArgs by value need its full definition; it is
// kept free of device-only constructs so that host compilers can include it.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#ifndef __CUDACC__
namespace slapo {
struct PhiloxArgs {
  uint64_t seed;
  uint64_t offset;
  const int64_t* seed_ptr;
  const int64_t* offset_ptr;
  uint32_t offset_intragraph;
  int captured;
};
}  // namespace slapo
#endif

namespace slapo {
void launch_bias_dropout_add_fwd(const void* x, const void* bias, const void* residual, void* y,
                                 int64_t rows, int cols, float p, PhiloxArgs rng, int dtype,
                                 cudaStream_t stream);
void launch_bias_dropout_add_bwd(const void* dy, void* dx, void* dbias, float* partial, int rows,
                                 int cols, float p, PhiloxArgs rng, int dtype,
                                 cudaStream_t stream);
void launch_ln_fwd(const void* x, const void* bias, const void* residual, const void* gamma,
                   const void* beta, void* y, void* z, float* mean, float* rstd, int rows,
                   int cols, float eps, float p, PhiloxArgs rng, int rms, int dtype,
                   cudaStream_t stream);
void launch_ln_bwd(const void* gy, const void* gz, const void* zin, const void* gamma,
                   const float* mean, const float* rstd, void* dx, void* dres, void* dgamma,
                   void* dbeta, void* dbias, float* partial, int rows, int cols, float p,
                   PhiloxArgs rng, int rms, int dtype, cudaStream_t stream);
}  // namespace slapo

namespace slapo {
// Flash attention on [B, S, H, D] tensors (D contiguous, a multiple of 8 up to 128);
// *_strides = element strides of (B, S, H).  Return 0 on success.
int flash_fwd_splits(int B, int H, int Sq, int Sk, int D);
int launch_flash_fwd(const void* q, const void* k, const void* v, void* o, float* lse,
                     float* scratch,
                     const float* kbias, const float* rel, int B, int H, int Sq, int Sk, int D,
                     const int64_t* q_strides, const int64_t* k_strides, const int64_t* v_strides,
                     float scale, int causal, float p_drop, PhiloxArgs rng, bool bf16, int* status,
                     cudaStream_t stream);
// How the backward runs, and its scratch in floats: row statistics, padded key bias, keep bits
// (dropout in two launches) and shares of dQ (keys split over work items).
struct FlashBwdPlan {
  int pairs;         // (batch, head) pairs per launch: the keep bits of all would grow with B H Sq Sk
  int splits;        // work items per query tile in the dQ pass
  int q_ctas;        // both passes in one launch, this many CTAs for dQ; 0: one launch each
  int64_t stats, bias, keep, part;
  int64_t total() const { return stats + bias + keep + part; }
};
// keep_words: 32-bit words of keep bits at a time (one pair's at least); 0: 1 GB of them, and whether
// the passes run in one launch, without keep bits, is left to the plan.
FlashBwdPlan flash_bwd_plan(int B, int H, int Sq, int Sk, int D, bool packed, bool causal,
                            bool key_bias, bool rel, float p_drop, int64_t keep_words);
// dq_row_stride / dkv_row_stride: elements between consecutive (b, s, head) rows of the outputs
int launch_flash_bwd(const void* q, const void* k, const void* v, const void* o, const void* dout,
                     const float* lse, const FlashBwdPlan& plan, float* scratch, void* dq, void* dk,
                     void* dv, int64_t dq_row_stride, int64_t dkv_row_stride, const float* kbias,
                     const float* rel, float* drel, int B, int H, int Sq, int Sk, int D,
                     const int64_t* q_strides, const int64_t* k_strides, const int64_t* v_strides,
                     float scale, int causal, float p_drop, PhiloxArgs rng, bool bf16, int* status,
                     cudaStream_t stream);
void launch_flash_dropout_mask(uint8_t* mask, int B, int H, int Sq, int Sk, float p_drop,
                               PhiloxArgs rng, cudaStream_t stream);
}  // namespace slapo
