// Fused element-wise kernels (HBM-bound, one pass each):
//   bias_act          y = act(x + bias)                       fwd / bwd (+ reduced dbias)
//   bias_dropout_add  y = dropout(x + bias, p) + residual     fwd / bwd (+ reduced dbias)
//   fused_adamw       AdamW on flat fp32 master weights, writes the low-precision copy
// Dropout masks are regenerated from Philox (seed, offset, element index): no
// mask tensor exists.  Bias gradients are reduced in two stages through a
// small fp32 scratch buffer [row_chunks, cols] supplied by the caller.
#include "common.cuh"
#include "kernels.h"

#include <atomic>

namespace slapo {

static std::atomic<int64_t> g_launches{0};
void count_launch(int n) { g_launches.fetch_add(n, std::memory_order_relaxed); }
int64_t launch_count() { return g_launches.load(std::memory_order_relaxed); }

// ------------------------------------------------------------------------ //
// An activation and its derivative by the type of the data (common.cuh).
template <int kAct, typename T>
__device__ __forceinline__ float act_value(float x) {
  if constexpr (sizeof(T) == 2) return act_fwd16<kAct>(x);
  else return act_fwd(x, kAct);
}
template <int kAct, typename T>
__device__ __forceinline__ float act_slope(float x) {
  if constexpr (sizeof(T) == 2) return act_grad16<kAct>(x);
  else return act_grad(x, kAct);
}

// Four independent 16-byte loads per thread are issued before any of them is used: with
// 2048 resident threads per SM a single load each leaves too few bytes in flight to cover the
// HBM latency at full bandwidth.
template <int kAct, typename T>
__global__ void __launch_bounds__(256) bias_act_fwd_kernel(
    const T* __restrict__ x, const T* __restrict__ bias, T* __restrict__ y, int64_t n_vec,
    int cols) {
  constexpr int kUnroll = 4;
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  const int vpr = cols / kVec;  // vectors per row
  int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  // column (in vectors) of the first vector and its advance per step, kept in 32 bits
  int cv = static_cast<int>(i % vpr);
  const int step = static_cast<int>(stride % vpr);
  for (; i + (kUnroll - 1) * stride < n_vec; i += kUnroll * stride) {
    float v[kUnroll][8];
    int cvs[kUnroll];
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
      Vec8<T>::load(x + (i + u * stride) * kVec, v[u]);
      cvs[u] = cv;
      cv += step;
      if (cv >= vpr) cv -= vpr;
    }
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
      if (bias != nullptr) {
        float b[8];
        Vec8<T>::load(bias + cvs[u] * kVec, b);
#pragma unroll
        for (int k = 0; k < 8; ++k) v[u][k] += b[k];
      }
#pragma unroll
      for (int k = 0; k < 8; ++k) v[u][k] = act_value<kAct, T>(v[u][k]);
      Vec8<T>::store(y + (i + u * stride) * kVec, v[u]);
    }
  }
  for (; i < n_vec; i += stride) {
    float v[8];
    Vec8<T>::load(x + i * kVec, v);
    if (bias != nullptr) {
      float b[8];
      Vec8<T>::load(bias + cv * kVec, b);
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] += b[k];
    }
    cv += step;
    if (cv >= vpr) cv -= vpr;
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = act_value<kAct, T>(v[k]);
    Vec8<T>::store(y + i * kVec, v);
  }
}

// Column-slab layout shared by the backward kernels: a CTA of 8 warps covers
// 256 columns (lane -> 8 columns) and a chunk of rows (warp w takes rows
// w, w+8, ...), or, where rows of 16-bit values are whole groups of 16 on 32 bytes, a lane 16 columns and a warp two
// rows (2 w, 2 w + 1, and so on in steps of 16).  Per-thread partial column sums are combined across the 8
// warps in shared memory and written to partial[blockIdx.y][col].
__device__ __forceinline__ void slab_reduce_store(float acc[8], float* partial, int cols,
                                                  int col, bool col_ok) {
  __shared__ float red[8][256 + 8];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
  for (int k = 0; k < 8; ++k) red[warp][lane * 8 + k] = acc[k];
  __syncthreads();
  if (warp == 0 && col_ok) {
    float s[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      float t = 0.f;
#pragma unroll
      for (int w = 0; w < 8; ++w) t += red[w][lane * 8 + k];
      s[k] = t;
    }
    Vec8<float>::store(partial + static_cast<int64_t>(blockIdx.y) * cols + col, s);
  }
}

__device__ __forceinline__ void slab_reduce_store(const float (&acc16)[16], float* partial, int cols, int col0) {
  __shared__ float red16[8][16 * 17];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
  for (int k = 0; k < 16; ++k) {
    const float v = acc16[k] + __shfl_xor_sync(0xffffffffu, acc16[k], 16);
    if (lane < 16) red16[warp][k * 17 + lane] = v;
  }
  __syncthreads();
  const int c = threadIdx.x;
  float t = 0.f;
#pragma unroll
  for (int w = 0; w < 8; ++w) t += red16[w][(c & 15) * 17 + (c >> 4)];
  if (col0 + c < cols) partial[static_cast<int64_t>(blockIdx.y) * cols + col0 + c] = t;
}

// 32-byte accesses, and one Philox call per thread and row instead of one in each of two neighbours.  8 columns ->
// 16 columns per lane, L2 flushed (us):
//                       GeLU's backward      ReLU's             dropout's
//   16384 x  4096       96.2 -> 77.4         72.1 -> 66.2       64.9 -> 48.7
//    8192 x  4096       51.2 -> 42.9         40.0 -> 36.4       34.8 -> 26.2
//    4096 x 10240       77.3 -> 52.5         56.1 -> 44.1       42.3 -> 30.6
//    8192 x  1024       17.4 -> 13.5         13.8 -> 11.2       11.6 ->  8.4
//    4096 x  1024        9.2 -> 10.1          8.7 ->  8.2        7.5 ->  5.8
//     512 x  2048        4.3 ->  4.6          4.3 ->  4.2        3.6 ->  3.5
// (GeLU's at 16384 x 4096: 5.2 of 6.5 TB/s).
template <int kAct, typename T>
__global__ void __launch_bounds__(256) bias_act_bwd_wide_kernel(
    const T* __restrict__ dy, const T* __restrict__ x, const T* __restrict__ bias,
    T* __restrict__ dx, float* __restrict__ partial, int rows, int cols, int rows_per_chunk) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int col = blockIdx.x * 256 + (lane & 15) * 16;
  float acc[16];
#pragma unroll
  for (int k = 0; k < 16; ++k) acc[k] = 0.f;
  if (col < cols) {
    uint32_t bw[8] = {0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u};
    if (bias != nullptr) load16_raw(bias + col, bw);
    const int r0 = blockIdx.y * rows_per_chunk;
    const int r1 = min(rows, r0 + rows_per_chunk);
    constexpr int kRows = 2;  // whose loads are issued before any is used
    for (int r = r0 + warp * 2 + (lane >> 4); r < r1; r += 16 * kRows) {
      const int64_t e = static_cast<int64_t>(r) * cols + col;
      uint32_t gw[kRows][8], vw[kRows][8];
#pragma unroll
      for (int u = 0; u < kRows; ++u)
        if (r + 16 * u < r1) {
          load16_raw(dy + e + static_cast<int64_t>(16 * u) * cols, gw[u]);
          load16_raw(x + e + static_cast<int64_t>(16 * u) * cols, vw[u]);
        }
#pragma unroll
      for (int u = 0; u < kRows; ++u)
        if (r + 16 * u < r1) {
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            float2 g = pair_floats(gw[u][k], T());
            const float2 v = pair_floats(vw[u][k], T()), b = pair_floats(bw[k], T());
            g.x *= act_slope<kAct, T>(v.x + b.x);
            g.y *= act_slope<kAct, T>(v.y + b.y);
            acc[2 * k] += g.x;
            acc[2 * k + 1] += g.y;
            gw[u][k] = pair_word(g.x, g.y, T());
          }
          store16_raw(dx + e + static_cast<int64_t>(16 * u) * cols, gw[u]);
        }
    }
  }
  if (partial != nullptr) slab_reduce_store(acc, partial, cols, blockIdx.x * 256);
}

template <typename T>
__global__ void __launch_bounds__(256) bias_dropout_add_bwd_wide_kernel(
    const T* __restrict__ dy, T* __restrict__ dx, float* __restrict__ partial, int rows,
    int cols, int rows_per_chunk, float p, PhiloxArgs rng) {
  uint64_t seed, offset;
  philox_unpack(rng, seed, offset);
  const float scale = dropout_scale(p);
  const uint32_t add4 = (128u - dropout_thr7(p)) * 0x01010101u;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int col = blockIdx.x * 256 + (lane & 15) * 16;
  float acc[16];
#pragma unroll
  for (int k = 0; k < 16; ++k) acc[k] = 0.f;
  if (col < cols) {
    const int r0 = blockIdx.y * rows_per_chunk;
    const int r1 = min(rows, r0 + rows_per_chunk);
    constexpr int kRows = 2;
    for (int r = r0 + warp * 2 + (lane >> 4); r < r1; r += 16 * kRows) {
      const int64_t e0 = static_cast<int64_t>(r) * cols + col;
      uint32_t w[kRows][8];
#pragma unroll
      for (int u = 0; u < kRows; ++u)
        if (r + 16 * u < r1) load16_raw(dy + e0 + static_cast<int64_t>(16 * u) * cols, w[u]);
#pragma unroll
      for (int u = 0; u < kRows; ++u)
        if (r + 16 * u < r1) {
          const int64_t e = e0 + static_cast<int64_t>(16 * u) * cols;
          float g[16];
          unpack_values<T>(w[u], g);
          drop16(philox_keep16(seed, offset, static_cast<uint64_t>(e) >> 4, add4), scale, g);
#pragma unroll
          for (int k = 0; k < 16; ++k) acc[k] += g[k];
          pack_values<T>(g, w[u]);
          store16_raw(dx + e, w[u]);
        }
    }
  }
  if (partial != nullptr) slab_reduce_store(acc, partial, cols, blockIdx.x * 256);
}

template <int kAct, typename T>
__global__ void __launch_bounds__(256) bias_act_bwd_kernel(
    const T* __restrict__ dy, const T* __restrict__ x, const T* __restrict__ bias,
    T* __restrict__ dx, float* __restrict__ partial, int rows, int cols, int rows_per_chunk) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int col = blockIdx.x * 256 + lane * 8;
  const bool col_ok = col + 8 <= cols;
  float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  float b[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (col_ok) {
    if (bias != nullptr) Vec8<T>::load(bias + col, b);
    const int r0 = blockIdx.y * rows_per_chunk;
    const int r1 = min(rows, r0 + rows_per_chunk);
#pragma unroll 4
    for (int r = r0 + warp; r < r1; r += 8) {
      const int64_t e = static_cast<int64_t>(r) * cols + col;
      float g[8], v[8];
      Vec8<T>::load(dy + e, g);
      Vec8<T>::load(x + e, v);
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        g[k] *= act_slope<kAct, T>(v[k] + b[k]);
        acc[k] += g[k];
      }
      Vec8<T>::store(dx + e, g);
    }
  }
  if (partial != nullptr) slab_reduce_store(acc, partial, cols, col, col_ok);
}

// Column sums of a [rows, cols] matrix (the bias gradient of a plain linear layer): same slab
// decomposition as above, reading only.
template <typename T>
__global__ void __launch_bounds__(256) colsum_kernel(const T* __restrict__ x,
                                                     float* __restrict__ partial, int rows,
                                                     int cols, int64_t row_stride,
                                                     int rows_per_chunk) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int col = blockIdx.x * 256 + lane * 8;
  const bool col_ok = col + 8 <= cols;
  float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (col_ok) {
    const int r0 = blockIdx.y * rows_per_chunk;
    const int r1 = min(rows, r0 + rows_per_chunk);
#pragma unroll 4
    for (int r = r0 + warp; r < r1; r += 8) {
      float g[8];
      Vec8<T>::load(x + static_cast<int64_t>(r) * row_stride + col, g);
#pragma unroll
      for (int k = 0; k < 8; ++k) acc[k] += g[k];
    }
  }
  slab_reduce_store(acc, partial, cols, col, col_ok);
}

// 32 x 32 threads per 32 columns: threadIdx.y strides over the chunks (see ln_bwd_finalize).
template <typename T>
__global__ void __launch_bounds__(1024) colsum_finalize_kernel(
    const float* __restrict__ partial, T* __restrict__ out, int chunks, int cols) {
  __shared__ float red[32][33];
  const int c = blockIdx.x * 32 + threadIdx.x;
  float s = 0.f;
  if (c < cols) {
    for (int i = threadIdx.y; i < chunks; i += 32) s += partial[static_cast<int64_t>(i) * cols + c];
  }
  red[threadIdx.y][threadIdx.x] = s;
  __syncthreads();
  if (threadIdx.y == 0 && c < cols) {
    float t = 0.f;
#pragma unroll
    for (int y = 0; y < 32; ++y) t += red[y][threadIdx.x];
    if constexpr (sizeof(T) == 4) out[c] = t;
    else out[c] = static_cast<T>(t);
  }
}

// ------------------------------------------------------------------------ //
template <typename T>
__global__ void __launch_bounds__(256) bias_dropout_add_fwd_kernel(
    const T* __restrict__ x, const T* __restrict__ bias, const T* __restrict__ residual,
    T* __restrict__ y, int64_t n_vec, int cols, float p, PhiloxArgs rng) {
  uint64_t seed, offset;
  philox_unpack(rng, seed, offset);
  const float scale = dropout_scale(p);
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n_vec;
       i += stride) {
    const int64_t e = i * kVec;
    float v[8], t[8];
    bool keep[8];
    Vec8<T>::load(x + e, v);
    if (bias != nullptr) {
      Vec8<T>::load(bias + (e % cols), t);
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] += t[k];
    }
    dropout_keep8(seed, offset, static_cast<uint64_t>(e), p, keep);
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = keep[k] ? v[k] * scale : 0.f;
    if (residual != nullptr) {
      Vec8<T>::load(residual + e, t);
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] += t[k];
    }
    Vec8<T>::store(y + e, v);
  }
}

template <typename T>
__global__ void __launch_bounds__(256) bias_dropout_add_bwd_kernel(
    const T* __restrict__ dy, T* __restrict__ dx, float* __restrict__ partial, int rows,
    int cols, int rows_per_chunk, float p, PhiloxArgs rng) {
  uint64_t seed, offset;
  philox_unpack(rng, seed, offset);
  const float scale = dropout_scale(p);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int col = blockIdx.x * 256 + lane * 8;
  const bool col_ok = col + 8 <= cols;
  float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (col_ok) {
    const int r0 = blockIdx.y * rows_per_chunk;
    const int r1 = min(rows, r0 + rows_per_chunk);
    for (int r = r0 + warp; r < r1; r += 8) {
      const int64_t e = static_cast<int64_t>(r) * cols + col;
      float g[8];
      bool keep[8];
      Vec8<T>::load(dy + e, g);
      dropout_keep8(seed, offset, static_cast<uint64_t>(e), p, keep);
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        g[k] = keep[k] ? g[k] * scale : 0.f;
        acc[k] += g[k];
      }
      Vec8<T>::store(dx + e, g);
    }
  }
  if (partial != nullptr) slab_reduce_store(acc, partial, cols, col, col_ok);
}

// ------------------------------------------------------------------------ //
// Eight fp32 values that are read and written once per step: 32 bytes at a time where they start on them, past what
// the caches would keep.  Two requests of 16 bytes for each held AdamW at 84 % of the copy rate: 83.4 M
// parameters 437 -> 377 us (5.5 -> 6.4 TB/s).
template <bool kWide>
__device__ __forceinline__ void load8_once(const float* p, float (&v)[8]) {
  if constexpr (kWide)
    asm volatile("ld.global.cs.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
                 : "l"(p)
                 : "memory");
  else
    Vec8<float>::load(p, v);
}
template <bool kWide>
__device__ __forceinline__ void store8_once(float* p, const float (&v)[8]) {
  if constexpr (kWide)
    asm volatile("st.global.cs.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "f"(v[0]), "f"(v[1]),
                 "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7])
                 : "memory");
  else
    Vec8<float>::store(p, v);
}

template <bool kWide, typename T>
__global__ void __launch_bounds__(256) fused_adamw_kernel(
    T* __restrict__ param, const T* __restrict__ grad, float* __restrict__ master,
    float* __restrict__ exp_avg, float* __restrict__ exp_avg_sq,
    const uint8_t* __restrict__ decay_mask, const float* __restrict__ grad_scale, int64_t n_vec,
    float lr, float beta1, float beta2, float eps, float weight_decay, float bc1, float bc2,
    const float* __restrict__ hyper) {
  // hyper = {lr, bias correction 1, bias correction 2} in device memory: the values that change
  // from step to step, so that a captured CUDA graph of the step stays valid
  if (hyper != nullptr) { lr = hyper[0]; bc1 = hyper[1]; bc2 = hyper[2]; }
  const float gs = grad_scale != nullptr ? *grad_scale : 1.f;
  const float inv_bc1 = 1.f / bc1, inv_sqrt_bc2 = rsqrtf(bc2);
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n_vec;
       i += stride) {
    const int64_t e = i * kVec;
    float g[8], w[8], m[8], v[8];
    Vec8<T>::load(grad + e, g);
    load8_once<kWide>(master + e, w);
    load8_once<kWide>(exp_avg + e, m);
    load8_once<kWide>(exp_avg_sq + e, v);
    const uint2 dm = *reinterpret_cast<const uint2*>(decay_mask + e);
    const uint8_t* dmb = reinterpret_cast<const uint8_t*>(&dm);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const float gk = g[k] * gs;
      m[k] = beta1 * m[k] + (1.f - beta1) * gk;
      v[k] = beta2 * v[k] + (1.f - beta2) * gk * gk;
      const float denom = sqrtf(v[k]) * inv_sqrt_bc2 + eps;
      float upd = (m[k] * inv_bc1) / denom;
      if (dmb[k]) upd += weight_decay * w[k];
      w[k] -= lr * upd;
    }
    store8_once<kWide>(master + e, w);
    store8_once<kWide>(exp_avg + e, m);
    store8_once<kWide>(exp_avg_sq + e, v);
    Vec8<T>::store(param + e, w);
  }
}

// ------------------------------------------------------------------------ //
static inline int flat_grid(int64_t n_vec) {
  int64_t blocks = (n_vec + 255) / 256;
  int64_t cap = static_cast<int64_t>(sm_count()) * 16;
  return static_cast<int>(blocks < cap ? (blocks > 0 ? blocks : 1) : cap);
}

// most row chunks that any of the kernels below uses: what their scratch holds
int colsum_chunks(int rows, int cols) {
  const int slabs = (cols + 255) / 256;
  int chunks = (sm_count() * 8 + slabs - 1) / slabs;
  const int max_chunks = (rows + 7) / 8;
  if (chunks > max_chunks) chunks = max_chunks;
  if (chunks < 1) chunks = 1;
  return chunks;
}

// Row chunks of a launch: eight CTAs per SM at most, which is one wave of `colsum_kernel` and two of the others.  One
// CTA more waits for a wave of its own (8192 x 30528, sums alone: 1200 CTAs 109 us, 1080 CTAs 96; 8192 x 2560
// 12.4 -> 11.3).
static int wave_chunks(int rows, int cols) {
  const int most = colsum_chunks(rows, cols), fit = sm_count() * 8 / ((cols + 255) / 256);
  return fit < 1 ? 1 : (fit < most ? fit : most);
}

#define DISPATCH_DTYPE(dtype, ...)                                   \
  switch (dtype) {                                                   \
    case 0: { using T = __nv_bfloat16; __VA_ARGS__; break; }         \
    case 1: { using T = __half; __VA_ARGS__; break; }                \
    default: { using T = float; __VA_ARGS__; break; }                \
  }

#define DISPATCH_16BIT(dtype, ...)                                   \
  switch (dtype) {                                                   \
    case 0: { using T = __nv_bfloat16; __VA_ARGS__; break; }         \
    default: { using T = __half; __VA_ARGS__; break; }               \
  }
// The kernels with 16 columns per lane hold more registers and take longer over the sums at a CTA's end, so they run
// with fewer CTAs and from `least` values on.  (Summing alone, without a store, gained under 6 % and is not
// done that way.)
static bool slab_wide(int rows, int cols, int dtype, int64_t least) {
  return dtype < 2 && cols % 16 == 0 && static_cast<int64_t>(rows) * cols >= least;
}
// Row chunks of theirs: the most that fill one, two, three or four waves of `per_sm` CTAs, whichever takes least when a
// wave takes the rows of a CTA and some 16 rows' time for its sums.  That is one wave unless the slabs of 256 columns leave
// much of it empty (30528 columns, 120 slabs for 296 CTAs: two chunks up to some 500 rows, seven from there on).
// Operands in L2 / L2 flushed (us), general kernel, two waves, one wave:
//   GeLU's backward  8192 x 1024   13.0 / 17.1, 12.8 / 14.6, 11.9 / 13.5    1024 x 8192   12.7 / 17.1, 12.8 / 15.0, 11.9 / 14.1
//                   16384 x 4096   93.9 / 94.8, 76.5 / 77.5, 75.9 / 77.4    4096 x 10240     - / 77.3,    - / 62.1, 52.2 / 52.4
//                    8192 x 30528     -  /  - ,    -  / 329 , 277  / 275
//   ReLU's           8192 x 2048   19.3 / 22.0, 17.6 / 20.3, 14.3 / 19.8    819 x 10240    9.4 / 13.2, 9.0 / 11.8, 8.4 / 11.5
//   dropout's        1024 x 8192   11.1 / 11.5,  9.4 /  9.3,  8.4 /  8.3    68 x 30528     8.8 /  5.2, 8.8 /  5.7, 7.9 / 4.6
static int slab_chunks(int rows, int cols, int per_sm) {
  const int most = wave_chunks(rows, cols);
  const int64_t slabs = (cols + 255) / 256, resident = static_cast<int64_t>(sm_count()) * per_sm;
  int best = most;
  int64_t least = -1;
  for (int w = 1; w <= 4; ++w) {
    const int64_t fill = w * resident / slabs;
    const int c = fill < most ? static_cast<int>(fill) : most;
    if (c < 1) continue;
    const int64_t time = (c * slabs + resident - 1) / resident * ((rows + c - 1) / c + 16);
    if (least < 0 || time < least) { least = time; best = c; }
    if (c == most) break;
  }
  return best;
}

#define DISPATCH_ACT(act, ...)                                       \
  switch (act) {                                                     \
    case 0: { constexpr int kAct = 0; __VA_ARGS__; break; }          \
    case 1: { constexpr int kAct = 1; __VA_ARGS__; break; }          \
    default: { constexpr int kAct = 2; __VA_ARGS__; break; }         \
  }

void launch_bias_act_fwd(const void* x, const void* bias, void* y, int64_t rows, int cols,
                         int act, int dtype, cudaStream_t stream) {
  const int64_t n_vec = rows * cols / kVec;
  if (n_vec == 0) return;
  count_launch();
  DISPATCH_DTYPE(dtype, DISPATCH_ACT(act, (bias_act_fwd_kernel<kAct, T>
      <<<flat_grid(n_vec), 256, 0, stream>>>(
          static_cast<const T*>(x), static_cast<const T*>(bias), static_cast<T*>(y), n_vec, cols))));
}

void launch_colsum_finalize(const float* partial, void* out, int chunks, int cols, int dtype,
                            cudaStream_t stream) {
  count_launch();
  DISPATCH_DTYPE(dtype, (colsum_finalize_kernel<T><<<(cols + 31) / 32, dim3(32, 32), 0, stream>>>(
      partial, static_cast<T*>(out), chunks, cols)));
}

void launch_bias_act_bwd(const void* dy, const void* x, const void* bias, void* dx, void* dbias,
                         float* partial, int rows, int cols, int act, int dtype,
                         cudaStream_t stream) {
  if (rows == 0) return;
  const bool wide = slab_wide(rows, cols, dtype, 8 << 20) && on_32_bytes({dy, x, bias, dx});
  const int chunks = wide ? slab_chunks(rows, cols, 2) : wave_chunks(rows, cols);
  const int rows_per_chunk = (rows + chunks - 1) / chunks;
  dim3 grid((cols + 255) / 256, chunks);
  float* part = dbias != nullptr ? partial : nullptr;
  count_launch();
  if (wide) {
    DISPATCH_16BIT(dtype, DISPATCH_ACT(act, (bias_act_bwd_wide_kernel<kAct, T><<<grid, 256, 0, stream>>>(
        static_cast<const T*>(dy), static_cast<const T*>(x), static_cast<const T*>(bias),
        static_cast<T*>(dx), part, rows, cols, rows_per_chunk))));
  } else {
    DISPATCH_DTYPE(dtype, DISPATCH_ACT(act, (bias_act_bwd_kernel<kAct, T><<<grid, 256, 0, stream>>>(
        static_cast<const T*>(dy), static_cast<const T*>(x), static_cast<const T*>(bias),
        static_cast<T*>(dx), part, rows, cols, rows_per_chunk))));
  }
  if (dbias != nullptr) launch_colsum_finalize(partial, dbias, chunks, cols, dtype, stream);
}

void launch_colsum(const void* x, void* out, float* partial, int rows, int cols,
                   int64_t row_stride, int dtype, cudaStream_t stream) {
  if (rows == 0 || cols == 0) return;
  const int chunks = wave_chunks(rows, cols);
  const int rows_per_chunk = (rows + chunks - 1) / chunks;
  dim3 grid((cols + 255) / 256, chunks);
  count_launch();
  DISPATCH_DTYPE(dtype, (colsum_kernel<T><<<grid, 256, 0, stream>>>(
      static_cast<const T*>(x), partial, rows, cols, row_stride, rows_per_chunk)));
  launch_colsum_finalize(partial, out, chunks, cols, dtype, stream);
}

void launch_bias_dropout_add_fwd(const void* x, const void* bias, const void* residual, void* y,
                                 int64_t rows, int cols, float p, PhiloxArgs rng, int dtype,
                                 cudaStream_t stream) {
  const int64_t n_vec = rows * cols / kVec;
  if (n_vec == 0) return;
  count_launch();
  DISPATCH_DTYPE(dtype, (bias_dropout_add_fwd_kernel<T><<<flat_grid(n_vec), 256, 0, stream>>>(
      static_cast<const T*>(x), static_cast<const T*>(bias), static_cast<const T*>(residual),
      static_cast<T*>(y), n_vec, cols, p, rng)));
}

void launch_bias_dropout_add_bwd(const void* dy, void* dx, void* dbias, float* partial, int rows,
                                 int cols, float p, PhiloxArgs rng, int dtype,
                                 cudaStream_t stream) {
  if (rows == 0) return;
  const bool wide = slab_wide(rows, cols, dtype, 2 << 20) && on_32_bytes({dy, dx});
  const int chunks = wide ? slab_chunks(rows, cols, 4) : wave_chunks(rows, cols);
  const int rows_per_chunk = (rows + chunks - 1) / chunks;
  dim3 grid((cols + 255) / 256, chunks);
  float* part = dbias != nullptr ? partial : nullptr;
  count_launch();
  if (wide) {
    DISPATCH_16BIT(dtype, (bias_dropout_add_bwd_wide_kernel<T><<<grid, 256, 0, stream>>>(
        static_cast<const T*>(dy), static_cast<T*>(dx), part, rows, cols, rows_per_chunk, p, rng)));
  } else {
    DISPATCH_DTYPE(dtype, (bias_dropout_add_bwd_kernel<T><<<grid, 256, 0, stream>>>(
        static_cast<const T*>(dy), static_cast<T*>(dx), part, rows, cols, rows_per_chunk, p, rng)));
  }
  if (dbias != nullptr) launch_colsum_finalize(partial, dbias, chunks, cols, dtype, stream);
}

void launch_fused_adamw(void* param, const void* grad, float* master, float* exp_avg,
                        float* exp_avg_sq, const uint8_t* decay_mask, const float* grad_scale,
                        int64_t n, float lr, float beta1, float beta2, float eps,
                        float weight_decay, float bc1, float bc2, int dtype,
                        cudaStream_t stream, const float* hyper) {
  const int64_t n_vec = n / kVec;
  if (n_vec == 0) return;
  count_launch();
  const bool wide = ((reinterpret_cast<uintptr_t>(master) | reinterpret_cast<uintptr_t>(exp_avg) |
                      reinterpret_cast<uintptr_t>(exp_avg_sq)) & 31) == 0;
#define ADAMW_CASE(WIDE_)                                                                            \
  DISPATCH_DTYPE(dtype, (fused_adamw_kernel<WIDE_, T><<<flat_grid(n_vec), 256, 0, stream>>>(         \
      static_cast<T*>(param), static_cast<const T*>(grad), master, exp_avg, exp_avg_sq, decay_mask, \
      grad_scale, n_vec, lr, beta1, beta2, eps, weight_decay, bc1, bc2, hyper)))
  if (wide) {
    ADAMW_CASE(true)
  } else {
    ADAMW_CASE(false)
  }
#undef ADAMW_CASE
}

}  // namespace slapo
