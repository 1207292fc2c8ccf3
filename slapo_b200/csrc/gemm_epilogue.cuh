// What the GEMM kernels do with 32 columns of a row of the fp32 accumulator when an activation or its
// derivative rides in the epilogue (kEpi below); kind 0 is the kernels' own bias / ReLU path.
//
// GeLU's forward: the product is rounded to 16 bits, then C = act(product + bias): to the bit what a linear
// layer followed by a kernel for bias + activation gives.  (Adding the bias to the accumulator rounds once
// less and saves 5 of 122 us at 16384 x 4096, K = 1024, but moves every value that follows: after four BERT
// layers logits and gradients by 0.9 % of their norm.)  What the backward wants goes to C2: the product, or with
// `c2_sum` product + bias, rounded.  Backward: C = acc * act'(Z), with column sums of C (the bias gradient) over each 32 rows
// to `col_part` [ceil(M / 32)][N], which a second kernel adds up in a fixed order.
// An element is about 20 instructions and two of the special-function unit, which run under the next
// tile's products as far as those last.  Measured, L2 flushed, one machine (us; plain product / with the epilogue / the
// pass over memory that it replaces; eight or sixteen epilogue warps as in gemm2.cu at kManyEpiWarpsK):
//                                              16384 x 4096, K = 1024     4096 x 10240, K = 2560
//   GeLU                                               96 /  98 / 58             138 / 140 / 39
//   GeLU, the product kept                             96 / 111 / 58             138 / 146 / 39
//   tanh form                                          96 /  92 / 58             138 / 138 / 39
//   tanh form, the product kept                        96 / 109 / 58             138 / 145 / 39
//   GeLU's derivative and column sums                  94 / 137 / 72             138 / 156 / 50
//   tanh form's                                        94 / 143 / 73             138 / 156 / 49
//   ReLU's                                             94 / 126 / 54             138 / 153 / 36
// So the forward is all but hidden, while the derivative's epilogue is what bounds a product with K = 1024:
// of the pass of 72 us it saves 29, at K = 2560 32 of 50.
// Dropout (kEpiDropout): C = dropout(product + bias), again to the bit what a product and a kernel behind it give:
// the product is rounded first, and an element's decision is that of its index in C (16 to a Philox call, two calls
// for 32 columns; N % 16 == 0).  16384 x 1024, K = 4096: 98.8 -> 97.9 us, and a
// pass of 20 less; a whole feed-forward block of 8192 x 512 204 -> 187.
#pragma once
#include <type_traits>
#include "common.cuh"
#include "kernels.h"

namespace slapo {

enum GemmEpiKind {
  kEpiPlain = 0, kEpiGelu = 1, kEpiGeluTanh = 2, kEpiGeluBwd = 3, kEpiGeluTanhBwd = 4, kEpiReluBwd = 5, kEpiDropout = 6
};
constexpr bool epi_backward(int kind) { return kind >= kEpiGeluBwd && kind <= kEpiReluBwd; }

// Dropout's parameters, in that kernel's alone: with them among those of all, the plain kernel of gemm.cu was compiled
// to 64 registers instead of 80 and its tiles of 64 columns took 0.6 - 0.9 us longer (M x N x K, operands in L2:
// 200 x 2048 x 512 6.4 -> 7.3 us, 24 x 512 x 2048 4.6 -> 5.4).
template <typename P>
struct DropParams : P {
  PhiloxArgs rng;         // generator state
  uint32_t drop_add4;     // what a draw is compared by
  float drop_scale;       // factor of kept values
  void set(const GemmEpi& epi) {
    rng = *epi.rng;
    drop_add4 = (128u - dropout_thr7(epi.p)) * 0x01010101u;
    drop_scale = dropout_scale(epi.p);
  }
};
template <typename P, int kEpi>
using EpiParams = std::conditional_t<kEpi == kEpiDropout, DropParams<P>, P>;

template <int kEpi>
__device__ __forceinline__ float epi_value(float x) {
  return act_fwd16<kEpi == kEpiGelu ? 0 : 1>(x);
}
template <int kEpi>
__device__ __forceinline__ float epi_slope(float z) {
  return act_grad16<kEpi == kEpiGeluBwd ? 0 : (kEpi == kEpiGeluTanhBwd ? 1 : 2)>(z);
}

__device__ __forceinline__ float2 unpack_pair(uint32_t w, int bf16) {
  if (bf16) return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w));
  return __half22float2(*reinterpret_cast<const __half2*>(&w));
}
__device__ __forceinline__ uint32_t pack_pair(float a, float b, int bf16) {
  return bf16 ? pair_word(a, b, __nv_bfloat16()) : pair_word(a, b, __half());
}

// 32 columns of a row as 16 words, from and to 16-byte aligned memory (N % 8 == 0: whole groups of
// eight columns exist or do not)
__device__ __forceinline__ void load_row32(const void* base, int64_t off, int col0, int N, bool ok,
                                           uint32_t (&w)[16]) {
  const uint8_t* src = static_cast<const uint8_t*>(base) + off * 2;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    uint4 t = make_uint4(0u, 0u, 0u, 0u);
    if (ok && col0 + q * 8 < N) t = __ldcs(reinterpret_cast<const uint4*>(src + q * 16));
    w[4 * q] = t.x; w[4 * q + 1] = t.y; w[4 * q + 2] = t.z; w[4 * q + 3] = t.w;
  }
}
__device__ __forceinline__ void store_row32(void* base, int64_t off, int col0, int N, bool sectors,
                                            const uint32_t (&w)[16]) {
  uint8_t* dst = static_cast<uint8_t*>(base) + off * 2;
  if (sectors) {
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      if (col0 + q * 16 + 8 < N)
        asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(dst + q * 32),
                     "r"(w[8 * q]), "r"(w[8 * q + 1]), "r"(w[8 * q + 2]), "r"(w[8 * q + 3]),
                     "r"(w[8 * q + 4]), "r"(w[8 * q + 5]), "r"(w[8 * q + 6]), "r"(w[8 * q + 7])
                     : "memory");
      else if (col0 + q * 16 < N)
        *reinterpret_cast<uint4*>(dst + q * 32) = make_uint4(w[8 * q], w[8 * q + 1], w[8 * q + 2], w[8 * q + 3]);
    }
  } else {
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (col0 + q * 8 < N)
        *reinterpret_cast<uint4*>(dst + q * 16) = make_uint4(w[4 * q], w[4 * q + 1], w[4 * q + 2], w[4 * q + 3]);
  }
}

// Sums over the warp's 32 rows of 32 columns, column l in lane l: each step halves the columns that a
// lane holds and doubles the rows they are sums of.
__device__ __forceinline__ float column_sums32(float (&s)[32], int lane) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const bool upper = lane & o;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      if (i < o) {
        const float other = upper ? s[i] : s[i + o];
        const float mine = upper ? s[i + o] : s[i];
        s[i] = mine + __shfl_xor_sync(0xffffffffu, other, o);
      }
    }
  }
  return s[0];
}

// The whole warp calls it: lanes are 32 consecutive rows from row0 on, v the accumulator's columns
// [col0, col0 + 32) (col0 < N), aux the bias words (forward) or Z's (backward).
template <int kEpi, typename P>
__device__ __forceinline__ void epi_finish(const P& p, float (&v)[32], const uint32_t (&aux)[16], int row0,
                                           int lane, int col0, bool sectors) {
  const int row = row0 + lane;
  const int64_t off = static_cast<int64_t>(row) * p.ldc + col0;
  uint32_t w[16];
  if constexpr (epi_backward(kEpi)) {
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const float2 z = unpack_pair(aux[j], p.out_bf16);
      v[2 * j] *= epi_slope<kEpi>(z.x);
      v[2 * j + 1] *= epi_slope<kEpi>(z.y);
      w[j] = pack_pair(v[2 * j], v[2 * j + 1], p.out_bf16);
    }
    if (row < p.M) store_row32(p.C, off, col0, p.N, sectors, w);
    if (p.col_part != nullptr && row0 < p.M) {
      // (rows beyond M have a zero accumulator)
      const float s = column_sums32(v, lane);
      if (col0 + lane < p.N) p.col_part[static_cast<int64_t>(row0 >> 5) * p.N + col0 + lane] = s;
    }
  } else if constexpr (kEpi == kEpiDropout) {
    if (row >= p.M) return;
    uint64_t seed, offset;
    philox_unpack(p.rng, seed, offset);
    const uint64_t group = (static_cast<uint64_t>(row) * p.N + col0) >> 4;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const uint4 kw = philox_keep16(seed, offset, group + h, p.drop_add4);
      const uint32_t word[4] = {kw.x, kw.y, kw.z, kw.w};
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int j = h * 8 + i;
        const float2 a = unpack_pair(pack_pair(v[2 * j], v[2 * j + 1], p.out_bf16), p.out_bf16);
        const float2 b = unpack_pair(aux[j], p.out_bf16);
        w[j] = pack_pair((a.x + b.x) * p.drop_scale, (a.y + b.y) * p.drop_scale, p.out_bf16) &
               keep_mask_pair(word[i >> 1], i & 1);
      }
    }
    store_row32(p.C, off, col0, p.N, sectors, w);
  } else {
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      w[j] = pack_pair(v[2 * j], v[2 * j + 1], p.out_bf16);
      const float2 a = unpack_pair(w[j], p.out_bf16), b = unpack_pair(aux[j], p.out_bf16);
      v[2 * j] = a.x + b.x;
      v[2 * j + 1] = a.y + b.y;
    }
    if (row >= p.M) return;
    if (p.C2 != nullptr) {
      if (p.c2_sum) {
#pragma unroll
        for (int j = 0; j < 16; ++j) w[j] = pack_pair(v[2 * j], v[2 * j + 1], p.out_bf16);
      }
      store_row32(p.C2, off, col0, p.N, sectors, w);
    }
#pragma unroll
    for (int j = 0; j < 16; ++j)
      w[j] = pack_pair(epi_value<kEpi>(v[2 * j]), epi_value<kEpi>(v[2 * j + 1]), p.out_bf16);
    store_row32(p.C, off, col0, p.N, sectors, w);
  }
}

}  // namespace slapo
