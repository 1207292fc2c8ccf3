// LayerNorm / RMSNorm, optionally fused with "bias + dropout + residual add"
// in front:   z = dropout(x + bias, p) + residual ;  y = norm(z) * gamma + beta
//
// One pass over HBM per direction: a row lives in registers (VPL vectors of 8
// per thread, WPR warps per row; 16-bit rows of 257 to 4096 columns in whole groups of 16, as far as
// these start on 32 bytes: 16 values per thread, the `_rows` kernels), statistics are two-pass in fp32, the
// dropout mask is regenerated from Philox in the backward, and the gamma /
// beta / bias gradients are accumulated in registers over all rows a CTA
// visits, written once per CTA to an fp32 scratch [grid, 3, cols] and summed
// by a small second kernel.
#include "common.cuh"
#include "kernels.h"

namespace slapo {

// Threads of a CTA are organised as RG row groups of WPR warps; each group
// normalises one row per iteration (VPL vectors of 8 values per thread).
// Several rows in flight per CTA keep enough loads outstanding to cover the
// HBM latency; group-local reductions use named barriers.
template <int WPR>
__device__ __forceinline__ void group_sync(int group) {
  asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "r"(32 * WPR) : "memory");
}

template <int WPR>
__device__ __forceinline__ float row_sum(float v, float* red, int group, int wir) {
  v = warp_sum(v);
  if constexpr (WPR == 1) {
    return v;
  } else {
    const int lane = threadIdx.x & 31;
    if (lane == 0) red[group * WPR + wir] = v;
    group_sync<WPR>(group);
    float t = 0.f;
#pragma unroll
    for (int w = 0; w < WPR; ++w) t += red[group * WPR + w];
    group_sync<WPR>(group);
    return t;
  }
}

// Two sums at once for the backward.  `red`: [2][groups][WPR], used in turn, so that one barrier does: who
// writes a half again has passed the barrier that its last readers reached after reading it.  (In the
// forward the same was slower, 39.6 against 37.0 us at 16384 x 1024 with dropout.)
template <int WPR>
__device__ __forceinline__ float2 row_sums(float2 v, float2 (*red)[WPR], int groups, int group, int wir,
                                           int& turn) {
  v = make_float2(warp_sum(v.x), warp_sum(v.y));
  if constexpr (WPR == 1) {
    return v;
  } else {
    float2* mine = red[turn * groups + group];
    turn ^= 1;
    if ((threadIdx.x & 31) == 0) mine[wir] = v;
    group_sync<WPR>(group);
    float2 t = mine[0];
#pragma unroll
    for (int w = 1; w < WPR; ++w) t = make_float2(t.x + mine[w].x, t.y + mine[w].y);
    return t;
  }
}

template <typename T, int VPL, int WPR, int RG>
__global__ void __launch_bounds__(32 * WPR * RG, (VPL == 1 && WPR * RG == 16) ? 2 : 1) ln_fwd_kernel(
    const T* __restrict__ x, const T* __restrict__ bias, const T* __restrict__ residual,
    const T* __restrict__ gamma, const T* __restrict__ beta, T* __restrict__ y,
    T* __restrict__ z, float* __restrict__ mean_out, float* __restrict__ rstd_out, int rows,
    int cols, float eps, float p, PhiloxArgs rng, int rms) {
  __shared__ float red[WPR * RG];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int group = warp / WPR, wir = warp % WPR;
  uint64_t seed = 0, offset = 0;
  if (p > 0.f) philox_unpack(rng, seed, offset);
  const float scale = dropout_scale(p);
  const float inv_cols = 1.f / static_cast<float>(cols);

  float gw[VPL][8], gb[VPL][8];
#pragma unroll
  for (int i = 0; i < VPL; ++i) {
    const int col = (i * 32 * WPR + wir * 32 + lane) * 8;
    if (col < cols) {
      Vec8<T>::load(gamma + col, gw[i]);
      if (beta != nullptr) Vec8<T>::load(beta + col, gb[i]);
      else {
#pragma unroll
        for (int k = 0; k < 8; ++k) gb[i][k] = 0.f;
      }
    }
  }

  for (int row0 = blockIdx.x * RG; row0 < rows; row0 += gridDim.x * RG) {
    const int row = row0 + group;
    const bool row_ok = row < rows;
    float v[VPL][8];
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < VPL; ++i) {
      const int col = (i * 32 * WPR + wir * 32 + lane) * 8;
      if (row_ok && col < cols) {
        const int64_t e = static_cast<int64_t>(row) * cols + col;
        Vec8<T>::load(x + e, v[i]);
        if (bias != nullptr) {
          float t[8];
          Vec8<T>::load(bias + col, t);
#pragma unroll
          for (int k = 0; k < 8; ++k) v[i][k] += t[k];
        }
        if (p > 0.f) {
          bool keep[8];
          dropout_keep8(seed, offset, static_cast<uint64_t>(e), p, keep);
#pragma unroll
          for (int k = 0; k < 8; ++k) v[i][k] = keep[k] ? v[i][k] * scale : 0.f;
        }
        if (residual != nullptr) {
          float t[8];
          Vec8<T>::load(residual + e, t);
#pragma unroll
          for (int k = 0; k < 8; ++k) v[i][k] += t[k];
        }
        if (z != nullptr) {
          Vec8<T>::store(z + e, v[i]);
          // statistics must see exactly what the backward will re-read
          round_through<T>(v[i]);
        }
#pragma unroll
        for (int k = 0; k < 8; ++k) s += v[i][k];
      } else {
#pragma unroll
        for (int k = 0; k < 8; ++k) v[i][k] = 0.f;
      }
    }
    float mean = 0.f;
    if (!rms) mean = row_sum<WPR>(s, red, group, wir) * inv_cols;
    float sq = 0.f;
#pragma unroll
    for (int i = 0; i < VPL; ++i) {
      const int col = (i * 32 * WPR + wir * 32 + lane) * 8;
      if (col < cols) {
#pragma unroll
        for (int k = 0; k < 8; ++k) { const float d = v[i][k] - mean; sq += d * d; }
      }
    }
    const float rstd = rsqrtf(row_sum<WPR>(sq, red, group, wir) * inv_cols + eps);
    if (row_ok) {
#pragma unroll
      for (int i = 0; i < VPL; ++i) {
        const int col = (i * 32 * WPR + wir * 32 + lane) * 8;
        if (col < cols) {
          float o[8];
#pragma unroll
          for (int k = 0; k < 8; ++k) o[k] = (v[i][k] - mean) * rstd * gw[i][k] + gb[i][k];
          Vec8<T>::store(y + static_cast<int64_t>(row) * cols + col, o);
        }
      }
      if (lane == 0 && wir == 0) {
        mean_out[row] = mean;
        rstd_out[row] = rstd;
      }
    }
  }
}

// The forward for 16-bit rows of 16 values per thread: a 32-byte access and one Philox call for all of them (the
// kernel above draws each call twice, in neighbouring threads), WPR warps to a row, eight warps to a CTA, and the
// next row fetched before this one's sums.  A row's two sums are added up in another order, so that y differs from the
// kernel's above by single last places of 16 bits; z is the same to the bit.
// Both are bound by the instructions and reductions of a row more than by memory; two CTAs of 128 registers per SM
// hold 32 KB of loads in flight (16 without a residual).  Kernel above -> this one, L2 flushed, dropout + residual /
// LayerNorm alone (us):
//   64 x 1024    3.7 -> 3.7 /  3.3 ->  2.9       16384 x  512    32.8 -> 16.2 / 22.4 ->  9.6
//   2048 x 1024  7.6 -> 6.8 /  5.7 ->  4.5       16384 x 1536   100.6 -> 47.0 / 55.9 -> 29.3
//   16384 x 1024 36.4 -> 28.6 / 24.6 -> 16.9     8192 x 2560     63.2 -> 42.6 / 48.0 -> 28.1
//   8192 x 2048  55.6 -> 29.1 / 32.0 -> 17.6     8192 x 4096     74.9 -> 52.7 / 54.8 -> 32.8
// (4.7 TB/s of 6.5 at 16384 x 1024 x 4 passes).  Up to 256 columns half of the lanes and more would have no values:
// 16384 x 256 12.7 there, 13.1 here.
template <typename T, int WPR, bool kDrop>
__global__ void __launch_bounds__(256, 2) ln_fwd_rows_kernel(
    const T* __restrict__ x, const T* __restrict__ bias, const T* __restrict__ residual,
    const T* __restrict__ gamma, const T* __restrict__ beta, T* __restrict__ y,
    T* __restrict__ z, float* __restrict__ mean_out, float* __restrict__ rstd_out, int rows,
    int cols, float eps, float p, PhiloxArgs rng, int rms) {
  constexpr int RG = 8 / WPR;
  __shared__ float red[8];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int group = warp / WPR, wir = warp % WPR;
  uint64_t seed = 0, offset = 0;
  if constexpr (kDrop) philox_unpack(rng, seed, offset);
  const float scale = dropout_scale(p);
  const uint32_t add4 = (128u - dropout_thr7(p)) * 0x01010101u;
  const float inv_cols = 1.f / static_cast<float>(cols);
  const int stride = gridDim.x * RG, col = (wir * 32 + lane) * 16;
  const bool ok = col < cols;
  uint32_t xn[8], rn[8];
  auto fetch = [&](int row) {
    if (row < rows && ok) {
      const int64_t e = static_cast<int64_t>(row) * cols + col;
      load16_raw(x + e, xn);
      if (residual != nullptr) load16_raw(residual + e, rn);
    }
  };
  int row = blockIdx.x * RG + group;
  fetch(row);
  for (; row < rows; row += stride) {
    const int64_t e = static_cast<int64_t>(row) * cols + col;
    float v[16];
    float s = 0.f;
    if (ok) {
      unpack_values<T>(xn, v);
      if (bias != nullptr) {
        uint32_t w[8];
        float b[16];
        load16_raw(bias + col, w);
        unpack_values<T>(w, b);
#pragma unroll
        for (int k = 0; k < 16; ++k) v[k] += b[k];
      }
      if constexpr (kDrop) {
        const uint4 c = philox_keep16(seed, offset, static_cast<uint64_t>(e) >> 4, add4);
        drop16(c, scale, v);
      }
      if (residual != nullptr) {
        float r[16];
        unpack_values<T>(rn, r);
#pragma unroll
        for (int k = 0; k < 16; ++k) v[k] += r[k];
      }
      if (z != nullptr) {
        // statistics must see exactly what the backward will re-read
        uint32_t w[8];
        pack_values<T>(v, w);
        store16_raw(z + e, w);
        unpack_values<T>(w, v);
      }
#pragma unroll
      for (int k = 0; k < 16; ++k) s += v[k];
    }
    fetch(row + stride);
    const float mean = rms ? 0.f : row_sum<WPR>(s, red, group, wir) * inv_cols;
    float sq = 0.f;
    if (ok) {
#pragma unroll
      for (int k = 0; k < 16; ++k) { const float d = v[k] - mean; sq += d * d; }
    }
    const float rstd = rsqrtf(row_sum<WPR>(sq, red, group, wir) * inv_cols + eps);
    if (ok) {
      uint32_t w[8];
      float g[16], b[16];
      load16_raw(gamma + col, w);
      unpack_values<T>(w, g);
      if (beta != nullptr) {
        load16_raw(beta + col, w);
        unpack_values<T>(w, b);
      }
#pragma unroll
      for (int k = 0; k < 16; ++k) v[k] = (v[k] - mean) * rstd * g[k] + (beta != nullptr ? b[k] : 0.f);
      pack_values<T>(v, w);
      store16_raw(y + e, w);
    }
    if (lane == 0 && wir == 0) {
      mean_out[row] = mean;
      rstd_out[row] = rstd;
    }
  }
}

template <typename T, int VPL, int WPR, int RG>
__global__ void __launch_bounds__(32 * WPR * RG, (VPL == 1 && WPR * RG == 16) ? 2 : 1) ln_bwd_kernel(
    const T* __restrict__ gy, const T* __restrict__ gz, const T* __restrict__ zin,
    const T* __restrict__ gamma, const float* __restrict__ mean_in,
    const float* __restrict__ rstd_in, T* __restrict__ dx, T* __restrict__ dres,
    float* __restrict__ partial, int rows, int cols, float p, PhiloxArgs rng, int rms,
    int want_dbias) {
  __shared__ float2 red[2 * RG][WPR];
  int turn = 0;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int group = warp / WPR, wir = warp % WPR;
  uint64_t seed = 0, offset = 0;
  if (p > 0.f) philox_unpack(rng, seed, offset);
  const float scale = dropout_scale(p);
  const float inv_cols = 1.f / static_cast<float>(cols);

  float gw[VPL][8], dgam[VPL][8], dbet[VPL][8], dbia[VPL][8];
#pragma unroll
  for (int i = 0; i < VPL; ++i) {
    const int col = (i * 32 * WPR + wir * 32 + lane) * 8;
    if (col < cols) Vec8<T>::load(gamma + col, gw[i]);
#pragma unroll
    for (int k = 0; k < 8; ++k) { dgam[i][k] = 0.f; dbet[i][k] = 0.f; dbia[i][k] = 0.f; }
  }

  for (int row0 = blockIdx.x * RG; row0 < rows; row0 += gridDim.x * RG) {
    const int row = row0 + group;
    const bool row_ok = row < rows;
    const float mean = row_ok ? mean_in[row] : 0.f;
    const float rstd = row_ok ? rstd_in[row] : 0.f;
    float g[VPL][8], xh[VPL][8];
    uint4 gz_raw[VPL][sizeof(T) == 2 ? 1 : 2];  // fetched with the other operands, used after the reductions
    float s1 = 0.f, s2 = 0.f;
#pragma unroll
    for (int i = 0; i < VPL; ++i) {
      const int col = (i * 32 * WPR + wir * 32 + lane) * 8;
      if (row_ok && col < cols) {
        const int64_t e = static_cast<int64_t>(row) * cols + col;
        Vec8<T>::load(gy + e, g[i]);
        Vec8<T>::load(zin + e, xh[i]);
        if (gz != nullptr) {
#pragma unroll
          for (int q = 0; q < (sizeof(T) == 2 ? 1 : 2); ++q)
            gz_raw[i][q] = reinterpret_cast<const uint4*>(gz + e)[q];
        }
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          xh[i][k] = (xh[i][k] - mean) * rstd;
          dgam[i][k] += g[i][k] * xh[i][k];
          dbet[i][k] += g[i][k];
          g[i][k] *= gw[i][k];
          s1 += g[i][k];
          s2 += g[i][k] * xh[i][k];
        }
      } else {
#pragma unroll
        for (int k = 0; k < 8; ++k) { g[i][k] = 0.f; xh[i][k] = 0.f; }
      }
    }
    // (one exchange for both sums)
    const float2 sums = row_sums<WPR>(make_float2(s1, s2), red, RG, group, wir, turn);
    const float m1 = rms ? 0.f : sums.x * inv_cols, m2 = sums.y * inv_cols;
    if (row_ok) {
#pragma unroll
      for (int i = 0; i < VPL; ++i) {
        const int col = (i * 32 * WPR + wir * 32 + lane) * 8;
        if (col < cols) {
          const int64_t e = static_cast<int64_t>(row) * cols + col;
          float d[8];
#pragma unroll
          for (int k = 0; k < 8; ++k) d[k] = rstd * (g[i][k] - m1 - xh[i][k] * m2);
          if (gz != nullptr) {
            float t[8];
            Vec8<T>::load(reinterpret_cast<const T*>(gz_raw[i]), t);
#pragma unroll
            for (int k = 0; k < 8; ++k) d[k] += t[k];
          }
          if (dres != nullptr) Vec8<T>::store(dres + e, d);
          if (p > 0.f) {
            bool keep[8];
            dropout_keep8(seed, offset, static_cast<uint64_t>(e), p, keep);
#pragma unroll
            for (int k = 0; k < 8; ++k) d[k] = keep[k] ? d[k] * scale : 0.f;
          }
          if (want_dbias) {
#pragma unroll
            for (int k = 0; k < 8; ++k) dbia[i][k] += d[k];
          }
          Vec8<T>::store(dx + e, d);
        }
      }
    }
  }

  // one partial row per CTA: [grid][3][cols]; row groups are combined in
  // shared memory first
  float* out = partial + static_cast<int64_t>(blockIdx.x) * 3 * cols;
  if constexpr (RG > 1) {
    constexpr int kCap = 32 * WPR * VPL * 8;
    // the groups in turn, in vectors.  With atomics on single floats, and two barriers for each of a row's
    // sums, 16384 x 1024 with dropout took 47.7 us (now 41; floor 20) and 8192 x 1024 27 (23).
    __shared__ __align__(16) float acc[3][kCap];
    for (int r = 0; r < RG; ++r) {
      if (group == r) {
#pragma unroll
        for (int i = 0; i < VPL; ++i) {
          const int c = (i * 32 * WPR + wir * 32 + lane) * 8;
#pragma unroll
          for (int which = 0; which < 3; ++which) {
            const float* mine = which == 0 ? dgam[i] : which == 1 ? dbet[i] : dbia[i];
            float v[8];
            if (r > 0) Vec8<float>::load(&acc[which][c], v);
#pragma unroll
            for (int k = 0; k < 8; ++k) v[k] = r > 0 ? v[k] + mine[k] : mine[k];
            Vec8<float>::store(&acc[which][c], v);
          }
        }
      }
      __syncthreads();
    }
    for (int c = threadIdx.x; c < cols; c += blockDim.x) {
      out[c] = acc[0][c];
      out[cols + c] = acc[1][c];
      out[2 * cols + c] = acc[2][c];
    }
  } else {
#pragma unroll
    for (int i = 0; i < VPL; ++i) {
      const int col = (i * 32 * WPR + wir * 32 + lane) * 8;
      if (col < cols) {
        Vec8<float>::store(out + col, dgam[i]);
        Vec8<float>::store(out + cols + col, dbet[i]);
        Vec8<float>::store(out + 2 * cols + col, dbia[i]);
      }
    }
  }
}

// The backward in the same form.  The operands of a row stay as they came, half the registers of their values, because
// the sums for gamma, beta and the bias take 48 and the next row's operands 24 of the 128; without fetching ahead
// it is no faster than the kernel above (16384 x 1024: 40.3 us).  Kernel above -> this one, L2 flushed, with dropout,
// two gradients in and out / LayerNorm alone (us):
//   16384 x  512  37.2 -> 20.9 / 25.7 -> 17.2      16384 x 1024  41.1 -> 34.5 / 29.9 -> 27.1
//   16384 x 1536  92.9 -> 58.2 / 66.9 -> 46.0       8192 x 2048  54.3 -> 36.3 / 39.9 -> 28.1
//    8192 x 2560  66.4 -> 48.0 / 49.8 -> 39.5       8192 x 4096  85.5 -> 76.2 / 63.8 -> 61.2
// (which calls: rows_bwd_pays)
template <typename T, int WPR, bool kDrop>
__global__ void __launch_bounds__(256, 2) ln_bwd_rows_kernel(
    const T* __restrict__ gy, const T* __restrict__ gz, const T* __restrict__ zin,
    const T* __restrict__ gamma, const float* __restrict__ mean_in,
    const float* __restrict__ rstd_in, T* __restrict__ dx, T* __restrict__ dres,
    float* __restrict__ partial, int rows, int cols, float p, PhiloxArgs rng, int rms,
    int want_dbias) {
  constexpr int RG = 8 / WPR;
  __shared__ float2 red[2 * RG][WPR];
  int turn = 0;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int group = warp / WPR, wir = warp % WPR;
  uint64_t seed = 0, offset = 0;
  if constexpr (kDrop) philox_unpack(rng, seed, offset);
  const float scale = dropout_scale(p);
  const uint32_t add4 = (128u - dropout_thr7(p)) * 0x01010101u;
  const float inv_cols = 1.f / static_cast<float>(cols);
  const int stride = gridDim.x * RG, col = (wir * 32 + lane) * 16;
  const bool ok = col < cols;
  float dgam[16], dbet[16], dbia[16];
#pragma unroll
  for (int k = 0; k < 16; ++k) { dgam[k] = 0.f; dbet[k] = 0.f; dbia[k] = 0.f; }
  uint32_t gyn[8], zn[8], gzn[8];
  float mean_n = 0.f, rstd_n = 0.f;
  auto fetch = [&](int row) {
    if (row < rows) {
      if (ok) {
        const int64_t e = static_cast<int64_t>(row) * cols + col;
        load16_raw(gy + e, gyn);
        load16_raw(zin + e, zn);
        if (gz != nullptr) load16_raw(gz + e, gzn);
      }
      mean_n = mean_in[row];
      rstd_n = rstd_in[row];
    }
  };
  int row = blockIdx.x * RG + group;
  fetch(row);
  for (; row < rows; row += stride) {
    const int64_t e = static_cast<int64_t>(row) * cols + col;
    const float mean = mean_n, rstd = rstd_n;
    uint32_t gyw[8], zw[8], gzw[8], gamw[8];  // kept as they came: half the registers of their values
    float s1 = 0.f, s2 = 0.f;
    if (ok) {
      load16_raw(gamma + col, gamw);
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        gyw[k] = gyn[k];
        zw[k] = zn[k];
        gzw[k] = gzn[k];
        const float2 g = pair_floats(gyw[k], T()), zv = pair_floats(zw[k], T()), gw = pair_floats(gamw[k], T());
        const float xa = (zv.x - mean) * rstd, xb = (zv.y - mean) * rstd, ga = g.x * gw.x, gb = g.y * gw.y;
        dgam[2 * k] += g.x * xa;
        dgam[2 * k + 1] += g.y * xb;
        dbet[2 * k] += g.x;
        dbet[2 * k + 1] += g.y;
        s1 += ga;
        s2 += ga * xa;
        s1 += gb;
        s2 += gb * xb;
      }
    }
    fetch(row + stride);
    const float2 sums = row_sums<WPR>(make_float2(s1, s2), red, RG, group, wir, turn);
    const float m1 = rms ? 0.f : sums.x * inv_cols, m2 = sums.y * inv_cols;
    if (ok) {
      uint4 keep = make_uint4(0u, 0u, 0u, 0u);
      if constexpr (kDrop) {
        asm volatile("" : "+l"(seed));  // or the seven rounds' keys take a register each over the loop
        keep = philox_keep16(seed, offset, static_cast<uint64_t>(e) >> 4, add4);
      }
      const uint32_t kw[4] = {keep.x, keep.y, keep.z, keep.w};
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const float2 g = pair_floats(gyw[k], T()), zv = pair_floats(zw[k], T()), gw = pair_floats(gamw[k], T());
        float da = rstd * (g.x * gw.x - m1 - (zv.x - mean) * rstd * m2);
        float db = rstd * (g.y * gw.y - m1 - (zv.y - mean) * rstd * m2);
        if (gz != nullptr) {
          const float2 t = pair_floats(gzw[k], T());
          da += t.x;
          db += t.y;
        }
        if (dres != nullptr) gyw[k] = pair_word(da, db, T());
        if constexpr (kDrop) {
          da = (kw[k >> 1] & (0x80u << (16 * (k & 1)))) ? da * scale : 0.f;
          db = (kw[k >> 1] & (0x8000u << (16 * (k & 1)))) ? db * scale : 0.f;
        }
        if (want_dbias) {
          dbia[2 * k] += da;
          dbia[2 * k + 1] += db;
        }
        zw[k] = pair_word(da, db, T());
      }
      if (dres != nullptr) store16_raw(dres + e, gyw);
      store16_raw(dx + e, zw);
    }
  }

  // one partial row per CTA: [grid][3][cols]; its row groups add to one in shared memory in turn
  float* out = partial + static_cast<int64_t>(blockIdx.x) * 3 * cols;
  auto half = [](const float (&a)[16], int h, float (&v)[8]) {
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = h ? a[8 + k] : a[k];
  };
  if constexpr (RG > 1) {
    __shared__ __align__(16) float acc[3][32 * WPR * 16];
    for (int r = 0; r < RG; ++r) {
      if (group == r) {
#pragma unroll
        for (int which = 0; which < 3; ++which) {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            float v[8], m[8];
            half(which == 0 ? dgam : which == 1 ? dbet : dbia, h, m);
            float* dst = &acc[which][col + 8 * h];
            if (r > 0) Vec8<float>::load(dst, v);
#pragma unroll
            for (int k = 0; k < 8; ++k) v[k] = r > 0 ? v[k] + m[k] : m[k];
            Vec8<float>::store(dst, v);
          }
        }
      }
      __syncthreads();
    }
    for (int c = threadIdx.x; c < cols; c += blockDim.x) {
      out[c] = acc[0][c];
      out[cols + c] = acc[1][c];
      out[2 * cols + c] = acc[2][c];
    }
  } else if (ok) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      float m[8];
      half(dgam, h, m);
      Vec8<float>::store(out + col + 8 * h, m);
      half(dbet, h, m);
      Vec8<float>::store(out + cols + col + 8 * h, m);
      half(dbia, h, m);
      Vec8<float>::store(out + 2 * cols + col + 8 * h, m);
    }
  }
}

// Column sums of the per-CTA partials.  A 32 x 32 thread block owns 32 columns: threadIdx.y
// strides over the partial rows (coalesced 128-byte reads), shared memory combines the 32
// row groups - ~n_part / 32 dependent loads per thread instead of n_part.
template <typename T>
__global__ void __launch_bounds__(1024) ln_bwd_finalize_kernel(
    const float* __restrict__ partial, T* __restrict__ dgamma, T* __restrict__ dbeta,
    T* __restrict__ dbias, int n_part, int cols) {
  __shared__ float red[32][33];
  const int c = blockIdx.x * 32 + threadIdx.x;
  const int which = blockIdx.y;  // 0 gamma, 1 beta, 2 bias
  T* dst = which == 0 ? dgamma : (which == 1 ? dbeta : dbias);
  if (dst == nullptr) return;
  float s = 0.f;
  if (c < cols) {
    for (int i = threadIdx.y; i < n_part; i += 32)
      s += partial[(static_cast<int64_t>(i) * 3 + which) * cols + c];
  }
  red[threadIdx.y][threadIdx.x] = s;
  __syncthreads();
  if (threadIdx.y == 0 && c < cols) {
    float t = 0.f;
#pragma unroll
    for (int y = 0; y < 32; ++y) t += red[y][threadIdx.x];
    if constexpr (sizeof(T) == 4) dst[c] = t;
    else dst[c] = static_cast<T>(t);
  }
}

// ------------------------------------------------------------------------ //
struct LnShape { int vpl; int wpr; int rg; };

static LnShape pick_shape(int cols) {
  const int vecs = cols / 8;
  if (vecs <= 32) return {1, 1, 4};
  // for 1024 columns one warp per row (4 vectors per lane) and two warps per row were
  // measured slower (fwd 341 / 199 us, bwd 457 / 309 us on 65536 rows) than four warps per row
  // with four row groups per CTA (129 / 264 us): registers, which the `_rows` kernels save by
  // keeping operands in 16 bits
  if (vecs <= 128) return {1, 4, 4};
  if (vecs <= 256) return {2, 4, 4};
  if (vecs <= 512) return {1, 16, 1};
  if (vecs <= 1024) return {2, 16, 1};
  return {4, 16, 1};
}

static int ln_grid(int rows, int cols, int ctas_per_sm) {
  const LnShape s = pick_shape(cols);
  const int want = (rows + s.rg - 1) / s.rg;
  const int cap = sm_count() * ctas_per_sm;
  return want < cap ? (want > 0 ? want : 1) : cap;
}

// The kernels with 16 values per thread: which rows they take (16-bit, whole groups of 16 values on 32 bytes).
static bool rows_shape(int cols, int dtype) { return dtype < 2 && cols > 256 && cols <= 4096 && cols % 16 == 0; }
static int rows_wpr(int cols) { return cols <= 512 ? 1 : cols <= 1024 ? 2 : cols <= 2048 ? 4 : 8; }
// Which backward calls they take.  Times against the general kernel's, finalising kernel included, with the operands in
// L2 / the incoming gradients there and the rest not, as they are in a backward / L2 flushed:
//                   LayerNorm alone         with dropout                         LayerNorm alone         with dropout
//   512 x 3500      1.05 / 1.03 / 1.02      0.98 / 0.92 / 0.95       2048 x 296   0.94 /   -  /   -       0.91 /   -  /   -
//   512 x 4096      0.96 / 0.95 / 0.93      0.86 / 0.83 / 0.84       2048 x 304   1.18 / 1.09 /   -       1.14 / 1.10 /   -
//   768 x 4096      1.11 / 1.07 / 1.06      1.02 / 0.97 / 1.00       2048 x 592   1.19 / 1.10 /   -       1.14 / 1.09 /   -
//   768 x 6000      1.14 / 1.03 / 1.01      1.00 / 0.95 / 0.95       2048 x 700   0.86 / 0.79 /   -       0.81 / 0.77 /   -
//   768 x 8192      1.09 / 0.98 / 0.99      0.98 / 0.92 / 0.92       2048 x 4096  0.98 / 0.78 / 0.74      0.89 / 0.78 / 0.74
//  1024 x 8192      1.09 / 0.96 / 0.97      0.98 / 0.92 / 0.89       2064 x 296   1.05 /   -  /   -       1.07 /   -  /   -
//   768 x 16384     1.06 / 0.96 / 0.93      0.87 / 0.87 / 0.86       2064 x 1000  1.05 / 0.93 / 0.91      0.99 / 0.91 / 0.90
//  1536 x 64        0.89 /   -  /   -       0.85 /   -  /   -        4096 x 296   1.03 /   -  /   -       1.08 /   -  /   -
//  1536 x 2048      0.91 / 0.78 / 0.77      0.85 / 0.75 / 0.74       4096 x 1000  1.00 / 1.00 / 0.99      0.95 / 0.97 / 0.97
// Up to 1024 columns a CTA's four or eight groups add their column sums in turn at its end, which takes many rows to pay
// for.  Up to 2048 the general kernel has four rows to a CTA and this one two: between two and four rows an SM that one
// has a CTA for each SM, and here some SMs have two.
static bool rows_bwd_pays(int rows, int cols, bool drop) {
  if (cols <= 512) return rows >= 4096;
  if (cols <= 1024) return rows >= (drop ? 6000 : 8192);
  if (cols <= 2048) return rows <= 2 * sm_count() || rows > 4 * sm_count();
  return rows >= 1000;
}
static int rows_grid(int rows, int cols) {
  const int rg = 8 / rows_wpr(cols), want = (rows + rg - 1) / rg, cap = sm_count() * 2;
  return want < cap ? want : cap;
}

// partial rows that a backward may write, whichever kernel runs
int ln_bwd_grid(int rows, int cols) {
  const LnShape s = pick_shape(cols);
  const int grid = ln_grid(rows, cols, s.wpr * s.rg >= 16 ? 2 : 8);
  const int wide = rows_shape(cols, 0) ? rows_grid(rows, cols) : 0;
  return grid > wide ? grid : wide;
}

#define ROWS_WPR(W, dtype, p, ...)                                                  \
  {                                                                                 \
    constexpr int WPR = W;                                                          \
    if (dtype == 0) {                                                               \
      using T = __nv_bfloat16;                                                      \
      if (p > 0.f) { constexpr bool kDrop = true; __VA_ARGS__; }                    \
      else { constexpr bool kDrop = false; __VA_ARGS__; }                           \
    } else {                                                                        \
      using T = __half;                                                             \
      if (p > 0.f) { constexpr bool kDrop = true; __VA_ARGS__; }                    \
      else { constexpr bool kDrop = false; __VA_ARGS__; }                           \
    }                                                                               \
  }
#define ROWS_SWITCH(dtype, cols, p, ...)                                            \
  switch (rows_wpr(cols)) {                                                         \
    case 1: ROWS_WPR(1, dtype, p, __VA_ARGS__) break;                               \
    case 2: ROWS_WPR(2, dtype, p, __VA_ARGS__) break;                               \
    case 4: ROWS_WPR(4, dtype, p, __VA_ARGS__) break;                               \
    default: ROWS_WPR(8, dtype, p, __VA_ARGS__) break;                              \
  }

#define LN_SHAPE_SWITCH(s, ...)                                                     \
  if (s.wpr == 1) {                                                          \
    constexpr int WPR = 1, RG = 4, VPL = 1;                                         \
    __VA_ARGS__;                                                                    \
  } else if (s.wpr == 4) {                                                          \
    constexpr int WPR = 4, RG = 4;                                                  \
    if (s.vpl == 1) { constexpr int VPL = 1; __VA_ARGS__; }                         \
    else { constexpr int VPL = 2; __VA_ARGS__; }                                    \
  } else {                                                                          \
    constexpr int WPR = 16, RG = 1;                                                 \
    if (s.vpl == 1) { constexpr int VPL = 1; __VA_ARGS__; }                         \
    else if (s.vpl == 2) { constexpr int VPL = 2; __VA_ARGS__; }                    \
    else { constexpr int VPL = 4; __VA_ARGS__; }                                    \
  }

#define DISPATCH_DTYPE(dtype, ...)                                   \
  switch (dtype) {                                                   \
    case 0: { using T = __nv_bfloat16; __VA_ARGS__; break; }         \
    case 1: { using T = __half; __VA_ARGS__; break; }                \
    default: { using T = float; __VA_ARGS__; break; }                \
  }

void launch_ln_fwd(const void* x, const void* bias, const void* residual, const void* gamma,
                   const void* beta, void* y, void* z, float* mean, float* rstd, int rows,
                   int cols, float eps, float p, PhiloxArgs rng, int rms, int dtype,
                   cudaStream_t stream) {
  if (rows == 0) return;
  if (rows_shape(cols, dtype) && on_32_bytes({x, bias, residual, gamma, beta, y, z})) {
    const int grid = rows_grid(rows, cols);
    count_launch();
    ROWS_SWITCH(dtype, cols, p, (ln_fwd_rows_kernel<T, WPR, kDrop><<<grid, 256, 0, stream>>>(
        static_cast<const T*>(x), static_cast<const T*>(bias), static_cast<const T*>(residual),
        static_cast<const T*>(gamma), static_cast<const T*>(beta), static_cast<T*>(y),
        static_cast<T*>(z), mean, rstd, rows, cols, eps, p, rng, rms)));
    return;
  }
  const LnShape s = pick_shape(cols);
  const int grid = ln_grid(rows, cols, s.wpr * s.rg >= 16 ? 2 : 16);
  count_launch();
  DISPATCH_DTYPE(dtype, LN_SHAPE_SWITCH(s, (ln_fwd_kernel<T, VPL, WPR, RG>
      <<<grid, 32 * WPR * RG, 0, stream>>>(
          static_cast<const T*>(x), static_cast<const T*>(bias), static_cast<const T*>(residual),
          static_cast<const T*>(gamma), static_cast<const T*>(beta), static_cast<T*>(y),
          static_cast<T*>(z), mean, rstd, rows, cols, eps, p, rng, rms))));
}

void launch_ln_bwd(const void* gy, const void* gz, const void* zin, const void* gamma,
                   const float* mean, const float* rstd, void* dx, void* dres, void* dgamma,
                   void* dbeta, void* dbias, float* partial, int rows, int cols, float p,
                   PhiloxArgs rng, int rms, int dtype, cudaStream_t stream) {
  if (rows == 0) return;
  const int want_dbias = dbias != nullptr;
  int grid;
  count_launch(2);
  if (rows_shape(cols, dtype) && rows_bwd_pays(rows, cols, p > 0.f) &&
      on_32_bytes({gy, gz, zin, gamma, dx, dres})) {
    grid = rows_grid(rows, cols);
    ROWS_SWITCH(dtype, cols, p, (ln_bwd_rows_kernel<T, WPR, kDrop><<<grid, 256, 0, stream>>>(
        static_cast<const T*>(gy), static_cast<const T*>(gz), static_cast<const T*>(zin),
        static_cast<const T*>(gamma), mean, rstd, static_cast<T*>(dx), static_cast<T*>(dres),
        partial, rows, cols, p, rng, rms, want_dbias)));
  } else {
    const LnShape s = pick_shape(cols);
    grid = ln_grid(rows, cols, s.wpr * s.rg >= 16 ? 2 : 8);
    DISPATCH_DTYPE(dtype, LN_SHAPE_SWITCH(s, (ln_bwd_kernel<T, VPL, WPR, RG>
        <<<grid, 32 * WPR * RG, 0, stream>>>(
            static_cast<const T*>(gy), static_cast<const T*>(gz), static_cast<const T*>(zin),
            static_cast<const T*>(gamma), mean, rstd, static_cast<T*>(dx), static_cast<T*>(dres),
            partial, rows, cols, p, rng, rms, want_dbias))));
  }
  dim3 fgrid((cols + 31) / 32, 3);
  DISPATCH_DTYPE(dtype, (ln_bwd_finalize_kernel<T><<<fgrid, dim3(32, 32), 0, stream>>>(
      partial, static_cast<T*>(dgamma), static_cast<T*>(dbeta), static_cast<T*>(dbias), grid,
      cols)));
}

}  // namespace slapo
