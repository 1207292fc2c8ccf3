// Attention of one query per (batch, head) over all its keys: a token of generation.
//
// Bound by reading K and V (8 x 1500 keys x 16 heads of 128: 98 MB, 15 us from HBM, less where a cache
// grown just before is still in L2).  A 128-row tensor-core tile would be one row of work in 128, and
// its loads wait for its softmax; here every lane has 16 bytes of four rows of K and V on their way under
// the arithmetic of the four before.  L lanes share a key row, so that a warp's load is 32 / L whole rows;
// each such group of lanes keeps a running maximum, sum and output of its own, merged over the lanes and
// warps at the end.  Probabilities stay in fp32.
// A CTA of sixteen or four warps takes the keys of one work item: all of a head's, or a share of them that
// flash_combine_kernel adds up (the rule is flash_fwd_splits).
// Measured (us), tensor-core tiles -> this: 8 x 1500 keys x 16 heads of 128: 24.4 -> 19.5 after a cache was
// grown (32 -> 20 alone; without the rows fetched ahead 38); 16 x 2000 x 20 x 64: 90 -> 41; 1 x 300 x 12 x 64:
// 10.7 -> 4.6; 1 x 2000 x 16 x 128, keys split: 14.5 -> 9.4 with the combine kernel.
#include "flash_common.cuh"
#include "kernels.h"

namespace slapo {

struct FlashDecodeParams {
  const void *q, *k, *v;
  int64_t qb, qh, kb, ks, kh, vb, vs, vh;     // strides in elements
  int H, Sk, D, splits, keys_per_split;
  void* o;              // [B, 1, H, D]
  float* lse;           // [B, H, 1]
  float* part_o;        // splits > 1: [splits][B H][D] and (maximum, sum) [splits][B H]
  float2* part_ml;
  const float* kbias;   // [B, Sk] or nullptr
  float scale_log2;
  int rows;             // B H
};

constexpr int kDecodeUnroll = 4;

template <int L, int kWarps, typename T>
__global__ void __launch_bounds__(32 * kWarps, 16 / kWarps) flash_decode_kernel(const FlashDecodeParams p) {
  constexpr int kRows = 32 / L;                 // key rows of a warp's load
  __shared__ float s_o[kWarps][L * 8];
  __shared__ float2 s_ml[kWarps];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int bh = blockIdx.x / p.splits, split = blockIdx.x - bh * p.splits;
  const int b = bh / p.H, h = bh - b * p.H;
  const int d0 = (lane % L) * 8;
  const bool d_ok = d0 < p.D;
  const int first = split * p.keys_per_split, end = min(p.Sk, first + p.keys_per_split);
  const T* k = static_cast<const T*>(p.k) + b * p.kb + h * p.kh + d0;
  const T* v = static_cast<const T*>(p.v) + b * p.vb + h * p.vh + d0;
  float q[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (d_ok) Vec8<T>::load(static_cast<const T*>(p.q) + b * p.qb + h * p.qh + d0, q);
#pragma unroll
  for (int i = 0; i < 8; ++i) q[i] *= p.scale_log2;

  // a step's rows as they are in memory, the next step's on their way under this one's arithmetic
  struct Rows { uint4 k[kDecodeUnroll], v[kDecodeUnroll]; };
  constexpr int kStep = kWarps * kRows * kDecodeUnroll;
  auto load = [&](int at, Rows& r) {
#pragma unroll
    for (int u = 0; u < kDecodeUnroll; ++u) {
      const int key = at + u * kRows + lane / L;
      const bool ok = key < end && d_ok;
      const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
      r.k[u] = ok ? *reinterpret_cast<const uint4*>(k + key * p.ks) : zero;
      r.v[u] = ok ? *reinterpret_cast<const uint4*>(v + key * p.vs) : zero;
    }
  };
  float m = -INFINITY, l = 0.f, o[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  int at = first + warp * kRows * kDecodeUnroll;
  Rows rows, next;
  load(at, rows);
  for (; at < end; at += kStep) {
    load(at + kStep, next);
    float s[kDecodeUnroll], top = m;
#pragma unroll
    for (int u = 0; u < kDecodeUnroll; ++u) {
      const int key = at + u * kRows + lane / L;
      float x = 0.f, kk[8];
      Vec8<T>::load(reinterpret_cast<const T*>(&rows.k[u]), kk);
#pragma unroll
      for (int i = 0; i < 8; ++i) x = fmaf(kk[i], q[i], x);
#pragma unroll
      for (int w = L / 2; w > 0; w >>= 1) x += __shfl_xor_sync(0xffffffffu, x, w);
      if (p.kbias != nullptr && key < end) x = fmaf(p.kbias[static_cast<int64_t>(b) * p.Sk + key], kLog2e, x);
      s[u] = key < end ? x : -INFINITY;
      top = fmaxf(top, s[u]);
    }
    const float use = top == -INFINITY ? 0.f : top;
    const float shrink = exp2f(m - use);          // (0 at the first keys)
    l *= shrink;
#pragma unroll
    for (int i = 0; i < 8; ++i) o[i] *= shrink;
#pragma unroll
    for (int u = 0; u < kDecodeUnroll; ++u) {
      const float e = exp2f(s[u] - use);
      float vv[8];
      Vec8<T>::load(reinterpret_cast<const T*>(&rows.v[u]), vv);
      l += e;
#pragma unroll
      for (int i = 0; i < 8; ++i) o[i] = fmaf(e, vv[i], o[i]);
    }
    m = top;
    rows = next;
  }

  // the groups of the warp, then the warps
#pragma unroll
  for (int w = L; w < 32; w <<= 1) {
    const float om = __shfl_xor_sync(0xffffffffu, m, w), ol = __shfl_xor_sync(0xffffffffu, l, w);
    const float top = fmaxf(m, om), use = top == -INFINITY ? 0.f : top;
    const float a = exp2f(m - use), c = exp2f(om - use);
    l = l * a + ol * c;
#pragma unroll
    for (int i = 0; i < 8; ++i) o[i] = o[i] * a + __shfl_xor_sync(0xffffffffu, o[i], w) * c;
    m = top;
  }
  if (lane < L) Vec8<float>::store(&s_o[warp][d0], o);
  if (lane == 0) s_ml[warp] = make_float2(m, l);
  __syncthreads();
  float top = -INFINITY;
#pragma unroll
  for (int w = 0; w < kWarps; ++w) top = fmaxf(top, s_ml[w].x);
  const float use = top == -INFINITY ? 0.f : top;
  float sum = 0.f, x = 0.f;
  const int d = threadIdx.x;
#pragma unroll
  for (int w = 0; w < kWarps; ++w) {
    const float f = exp2f(s_ml[w].x - use);
    sum += s_ml[w].y * f;
    if (d < p.D) x += s_o[w][d] * f;
  }
  if (p.splits > 1) {
    const int64_t row = static_cast<int64_t>(split) * p.rows + bh;
    if (d < p.D) p.part_o[row * p.D + d] = x;
    if (d == 0) p.part_ml[row] = make_float2(top, sum);
    return;
  }
  // (no visible key: 0; a NaN among the scores or values stays one, as in the other kernels)
  if (d < p.D)
    static_cast<T*>(p.o)[static_cast<int64_t>(bh) * p.D + d] = static_cast<T>(x * (sum > 0.f ? 1.f / sum : 0.f));
  if (d == 0) p.lse[bh] = sum > 0.f ? use * 0.6931471805599453f + logf(sum) : -INFINITY;
}

// One query, no dropout and no relative bias (the caller has looked).  part_o, part_ml: with splits > 1.
int launch_flash_decode(const void* q, const void* k, const void* v, void* o, float* lse, float* part_o,
                        float2* part_ml, const float* kbias, int B, int H, int Sk, int D,
                        const int64_t* q_strides, const int64_t* k_strides, const int64_t* v_strides,
                        float scale, int splits, int keys_per_split, bool bf16, cudaStream_t stream) {
  if ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v)) & 15)
    return 1;
  for (int i = 0; i < 3; ++i)
    if ((i != 1 && q_strides[i] % 8) || k_strides[i] % 8 || v_strides[i] % 8) return 1;
  FlashDecodeParams p;
  p.q = q; p.k = k; p.v = v; p.o = o; p.lse = lse; p.part_o = part_o; p.part_ml = part_ml;
  p.qb = q_strides[0]; p.qh = q_strides[2];
  p.kb = k_strides[0]; p.ks = k_strides[1]; p.kh = k_strides[2];
  p.vb = v_strides[0]; p.vs = v_strides[1]; p.vh = v_strides[2];
  p.H = H; p.Sk = Sk; p.D = D; p.splits = splits; p.keys_per_split = keys_per_split;
  p.kbias = kbias; p.scale_log2 = scale * kLog2e; p.rows = B * H;
  const int64_t ctas = static_cast<int64_t>(p.rows) * splits;
  if (ctas > 0x7fffffff) return 1;
  const unsigned grid = static_cast<unsigned>(ctas);
  count_launch();
  // Sixteen warps where a work item has many keys and the items leave SMs idle, four (and four CTAs per SM)
  // where most of sixteen would have nothing to load or the items fill the SMs by themselves.  Measured (us;
  // 128-row tensor-core tiles / sixteen / four), bf16, items x keys x D: 96 x 16 x 64: 6.8 / 3.4 / 2.9; 96 x 256 x
  // 64: 8.0 / 4.2 / 4.6; 384 x 128 x 64: 10.5 / 8.8 / 4.6; 640 x 2000 x 64: 96 / 67 / 75; 2048 x 128 x 64: 28 / 48 /
  // 19; 4096 x 512 x 64: 147 / 144 / 93; 144 x 384 x 128: 11.8 / 8.1 / 13.1; 384 x 256 x 128: 19.8 / 17.5 / 12.9;
  // 2048 x 512 x 128: 110 / 111 / 89.
  const int step = D <= 64 ? 256 : 128;         // keys that sixteen warps take at a time
  const bool few = 2 * keys_per_split <= step || (2 * ctas >= 3 * sm_count() && keys_per_split <= 2 * step) ||
                   ctas >= 6 * sm_count();
#define FLASH_DECODE_CASE(L_, W_)                                                                     \
  if (bf16) flash_decode_kernel<L_, W_, __nv_bfloat16><<<grid, 32 * W_, 0, stream>>>(p);              \
  else flash_decode_kernel<L_, W_, __half><<<grid, 32 * W_, 0, stream>>>(p)
  if (D <= 64) {
    if (few) { FLASH_DECODE_CASE(8, 4); }
    else { FLASH_DECODE_CASE(8, 16); }
  } else {
    if (few) { FLASH_DECODE_CASE(16, 4); }
    else { FLASH_DECODE_CASE(16, 16); }
  }
#undef FLASH_DECODE_CASE
  return cudaGetLastError() == cudaSuccess ? 0 : 4;
}

}  // namespace slapo
