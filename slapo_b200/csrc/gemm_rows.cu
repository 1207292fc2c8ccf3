// C[M, N] = act(A[M, K] W[N, K]^T + bias) for at most 16 rows: a linear layer on the tokens of one step of
// generation, GeLU and what its backward wants included (gemm_epilogue.cuh).  bf16 / fp16, fp32 accumulation.
//
// Bound by reading W once.  A 128-row tcgen05 tile has few CTAs for it (2048 columns: 32) and each
// waits for its ring; here a CTA takes 8 columns and its eight warps a part of K each, lanes load W straight
// into the registers of mma.sync (m16n8k16) 16 bytes at a time, eight loads ahead, and the warps' sums meet in
// shared memory in a fixed order.  A contraction may be taken in any order of K, so a lane's 16 bytes (8
// values of k) are the operands of two products, with A's values picked alike.
// Measured, 64-column tcgen05 tiles -> this: 8 x 6144 x 2048 and 8 x 2048 x 2048 together 30.3 -> 19.0 us (weights not in L2).
#include "common.cuh"
#include "gemm_epilogue.cuh"
#include "kernels.h"

namespace slapo {

struct GemmRowsParams {
  const void *a, *w, *bias;
  void *c, *c2;         // c2: GeLU's (GemmEpi), or nullptr
  int M, N, K, lda, ldw, ldc, act;
  int gelu, c2_sum;     // kind of GemmEpi and what goes to c2; 0: bias and `act`
};

template <typename T>
__device__ __forceinline__ void mma_16x8x16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1);
template <>
__device__ __forceinline__ void mma_16x8x16<__nv_bfloat16>(float (&d)[4], const uint32_t (&a)[4], uint32_t b0,
                                                           uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
      "{%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
template <>
__device__ __forceinline__ void mma_16x8x16<__half>(float (&d)[4], const uint32_t (&a)[4], uint32_t b0,
                                                    uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
      "{%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

constexpr int kRowsWarps = 8, kRowsUnroll = 8;

// kRuns: a warp takes eight steps of K in a row (512 bytes of each row of W), otherwise every eighth one
template <typename T, bool kRuns>
__global__ void __launch_bounds__(32 * kRowsWarps) gemm_rows_kernel(const GemmRowsParams p) {
  __shared__ float s_sum[kRowsWarps][16][9];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n0 = blockIdx.x * 8;              // N % 8 == 0
  const int row = lane >> 2;                  // of A (and row + 8), and column of the tile
  const int k_lane = (lane & 3) * 8;          // a step is 32 values of k, a lane's eight of them here
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  const T* w = static_cast<const T*>(p.w) + static_cast<int64_t>(n0 + row) * p.ldw + k_lane;
  const T* a0 = static_cast<const T*>(p.a) + static_cast<int64_t>(min(row, p.M - 1)) * p.lda + k_lane;
  const T* a1 = static_cast<const T*>(p.a) + static_cast<int64_t>(min(row + 8, p.M - 1)) * p.lda + k_lane;
  const bool two = p.M > 8;
  float d[4] = {0.f, 0.f, 0.f, 0.f};
  const int steps = (p.K + 31) / 32;
  constexpr int kNext = kRuns ? 1 : kRowsWarps;
  for (int s0 = kRuns ? warp * kRowsUnroll : warp; s0 < steps; s0 += kRowsWarps * kRowsUnroll) {
    uint4 ww[kRowsUnroll], x[kRowsUnroll];
#pragma unroll
    for (int u = 0; u < kRowsUnroll; ++u) {
      const int k = (s0 + u * kNext) * 32;
      const bool ok = k + k_lane < p.K;       // K % 8 == 0: all eight or none
      ww[u] = ok ? __ldcs(reinterpret_cast<const uint4*>(w + k)) : zero;
      x[u] = ok ? __ldg(reinterpret_cast<const uint4*>(a0 + k)) : zero;
    }
#pragma unroll
    for (int u = 0; u < kRowsUnroll; ++u) {
      const int k = (s0 + u * kNext) * 32;
      uint4 y = zero;
      if (two && k + k_lane < p.K) y = __ldg(reinterpret_cast<const uint4*>(a1 + k));
      const uint32_t f0[4] = {x[u].x, y.x, x[u].y, y.y}, f1[4] = {x[u].z, y.z, x[u].w, y.w};
      mma_16x8x16<T>(d, f0, ww[u].x, ww[u].y);
      mma_16x8x16<T>(d, f1, ww[u].z, ww[u].w);
    }
  }
  // rows row and row + 8, columns 2 (lane % 4) and the next
  s_sum[warp][row][(lane & 3) * 2] = d[0];
  s_sum[warp][row][(lane & 3) * 2 + 1] = d[1];
  s_sum[warp][row + 8][(lane & 3) * 2] = d[2];
  s_sum[warp][row + 8][(lane & 3) * 2 + 1] = d[3];
  __syncthreads();
  if (threadIdx.x < 128) {
    const int r = threadIdx.x >> 3, c = threadIdx.x & 7;
    if (r < p.M) {
      float v = 0.f;
#pragma unroll
      for (int i = 0; i < kRowsWarps; ++i) v += s_sum[i][r][c];
      const float bias = p.bias != nullptr ? static_cast<float>(static_cast<const T*>(p.bias)[n0 + c]) : 0.f;
      const int64_t at = static_cast<int64_t>(r) * p.ldc + n0 + c;
      if (p.gelu != kEpiPlain) {        // as epi_finish has it
        const T product = static_cast<T>(v);
        v = static_cast<float>(product) + bias;
        if (p.c2 != nullptr) static_cast<T*>(p.c2)[at] = p.c2_sum ? static_cast<T>(v) : product;
        v = p.gelu == kEpiGelu ? epi_value<kEpiGelu>(v) : epi_value<kEpiGeluTanh>(v);
      } else {
        v += bias;
        if (p.act >= 0) v = act_fwd(v, p.act);
      }
      static_cast<T*>(p.c)[at] = static_cast<T>(v);
    }
  }
}

// All products on so few rows that fill a block of 64 columns and two steps of K: from 64 x 64 (5.2 -> 2.4 us
// with 8 rows) to a vocabulary's width (the table below).
bool gemm_rows_takes(int M, int N, int K) { return M <= 16 && K >= 64 && N >= 64; }

// Returns 0 on success; >0 = refused on the host, as launch_gemm does.
int launch_gemm_rows(const void* A, const void* W, void* C, const void* bias, int M, int N, int K, int lda,
                     int ldw, int ldc, bool bf16, int act, cudaStream_t stream, const GemmEpi* epi) {
  if (epi != nullptr && (epi_backward(epi->kind) || epi->kind == kEpiDropout)) return 1;
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if (M > 16 || N % 8 || K % 8 || lda % 8 || ldw % 8 || ldc % 8) return 1;
  if ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(W) | reinterpret_cast<uintptr_t>(C)) & 15)
    return 1;
  const GemmRowsParams p{A, W, bias, C, epi != nullptr ? epi->c2 : nullptr, M, N, K, lda, ldw, ldc, act,
                         epi != nullptr ? epi->kind : kEpiPlain, epi != nullptr && epi->c2_sum ? 1 : 0};
  // Runs where every warp has whole ones (K a multiple of 2048), otherwise steps one by one: at K = 768 runs
  // would be three of eight warps' work.  Measured (us, 8 rows; 64-column tcgen05 tiles / runs / one by one), W
  // not in L2: 2048 x 2048: 15.2 / 6.2 / 7.0; 2560 x 10240: 51.6 / 20.4 / 25.5; 2560 x 2560: 17.8 / 9.8 / 8.7; 3072 x
  // 768: 8.5 / 5.5 / 4.3; 30528 x 768: 21.9 / 24.7 / 20.5; 32000 x 512: 19.3 / 24.1 / 17.7; 50304 x 1024: 37.8 / 37.3 /
  // 35.8; 50304 x 2048: 54.0 / 44.5 / 52.4.
  const bool runs = K % (32 * kRowsWarps * kRowsUnroll) == 0;
  auto kernel = bf16 ? (runs ? gemm_rows_kernel<__nv_bfloat16, true> : gemm_rows_kernel<__nv_bfloat16, false>)
                     : (runs ? gemm_rows_kernel<__half, true> : gemm_rows_kernel<__half, false>);
  count_launch();
  kernel<<<N / 8, 32 * kRowsWarps, 0, stream>>>(p);
  return cudaGetLastError() == cudaSuccess ? 0 : 4;
}

}  // namespace slapo
