// T5's relative-position table [buckets, H] as a bias by distance [H, n], and its gradient.
//
// Both are latency-bound (n is a few thousand): one launch each, where indexing the table with
// torch operators took a cast, a gather and a transposing copy, and its gradient an index-add
// that serialises on the few rows of the table (85 us at 1023 distances x 16 heads).
#include "common.cuh"
#include "kernels.h"

namespace slapo {

// Row of the table that an index names: negative ones count from the end, as in torch; -1 for an
// index outside of the table, which reads nothing and gives NaN.
__device__ __forceinline__ int64_t rel_row_of(int64_t index, int n_buckets) {
  if (index < 0) index += n_buckets;
  return index >= 0 && index < n_buckets ? index : -1;
}

template <typename T>
__global__ void __launch_bounds__(256) rel_bias_fwd_kernel(const T* __restrict__ table,
                                                           const int64_t* __restrict__ buckets,
                                                           float* __restrict__ out, int n, int H,
                                                           int n_buckets) {
  const int d = blockIdx.x * 256 + threadIdx.x, h = blockIdx.y;
  if (d >= n) return;
  const int64_t row = rel_row_of(buckets[d], n_buckets);
  out[static_cast<int64_t>(h) * n + d] =
      row >= 0 ? static_cast<float>(table[row * H + h]) : __int_as_float(0x7fc00000);
}

// one block per head; each warp sums the distances of one bucket at a time (fp32, fixed order)
template <typename T>
__global__ void __launch_bounds__(256) rel_bias_bwd_kernel(const float* __restrict__ grad,
                                                           const int64_t* __restrict__ buckets,
                                                           T* __restrict__ dtable, int n, int H,
                                                           int n_buckets) {
  const int h = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const float* g = grad + static_cast<int64_t>(h) * n;
  for (int b = warp; b < n_buckets; b += 8) {
    float s = 0.f;
    for (int d = lane; d < n; d += 32)
      if (rel_row_of(buckets[d], n_buckets) == b) s += g[d];
    s = warp_sum(s);
    if (lane == 0) dtable[static_cast<int64_t>(b) * H + h] = static_cast<T>(s);
  }
}

// T5's bucket of every distance key - query, as the operators of t5_relative_position_bucket round it: fp32
// throughout, divisions by a number as products with its reciprocal, each rounded, and the logarithm that
// the operators call (this file is built without --use_fast_math).  Where a distance lies on a border between
// buckets the last bit of any of these decides.  One launch where those operators were fourteen (40 us of
// kernels and 150 us of the host's time at 1023 distances).
__global__ void __launch_bounds__(256) rel_buckets_kernel(int64_t* __restrict__ out, int n, int last_key,
                                                          int buckets, int bidirectional, float inv_exact,
                                                          float inv_log) {
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i >= n) return;
  const int dist = i - last_key;
  int base = 0, far = dist < 0 ? -dist : 0;
  if (bidirectional) {
    buckets /= 2;
    if (dist > 0) base = buckets;
    far = dist < 0 ? -dist : dist;
  }
  const int exact = buckets / 2;
  int b = far;
  if (far >= exact) {
    const float x = __fmul_rn(static_cast<float>(max(far, 1)), inv_exact);
    const float l = __fmul_rn(logf(x), inv_log);
    b = min(exact + static_cast<int>(__fmul_rn(l, static_cast<float>(buckets - exact))),
            buckets - 1);
  }
  out[i] = base + b;
}

#define DISPATCH_DTYPE(dtype, ...)                                   \
  switch (dtype) {                                                   \
    case 0: { using T = __nv_bfloat16; __VA_ARGS__; break; }         \
    case 1: { using T = __half; __VA_ARGS__; break; }                \
    default: { using T = float; __VA_ARGS__; break; }                \
  }

void launch_rel_buckets(int64_t* out, int n, int last_key, int buckets, int bidirectional, float inv_exact,
                        float inv_log, cudaStream_t stream) {
  if (n <= 0) return;
  count_launch();
  rel_buckets_kernel<<<(n + 255) / 256, 256, 0, stream>>>(out, n, last_key, buckets, bidirectional, inv_exact,
                                                          inv_log);
}

void launch_rel_bias_fwd(const void* table, const int64_t* buckets, float* out, int n, int H,
                         int n_buckets, int dtype, cudaStream_t stream) {
  if (n == 0 || H == 0) return;
  count_launch();
  DISPATCH_DTYPE(dtype, (rel_bias_fwd_kernel<T><<<dim3((n + 255) / 256, H), 256, 0, stream>>>(
      static_cast<const T*>(table), buckets, out, n, H, n_buckets)));
}

void launch_rel_bias_bwd(const float* grad, const int64_t* buckets, void* dtable, int n, int H,
                         int n_buckets, int dtype, cudaStream_t stream) {
  if (H == 0 || n_buckets == 0) return;
  count_launch();
  DISPATCH_DTYPE(dtype, (rel_bias_bwd_kernel<T><<<H, 256, 0, stream>>>(
      grad, buckets, static_cast<T*>(dtable), n, H, n_buckets)));
}

}  // namespace slapo
