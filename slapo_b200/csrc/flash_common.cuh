// Device helpers shared by the flash-attention forward and backward kernels: packed fp32
// arithmetic, 16-bit packing by type, exp2 on the special-function unit.
#pragma once
#include "common.cuh"
#include "tc05.cuh"

namespace slapo {

constexpr float kLog2e = 1.4426950408889634f;

// two fp32 values in one 64-bit register: sm_100 issues an FMA / add / multiply on both at once
__device__ __forceinline__ uint64_t f2_pack(float a, float b) {
  uint64_t d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(a), "f"(b));
  return d;
}
__device__ __forceinline__ void f2_unpack(uint64_t v, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ uint64_t f2_fma(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ uint64_t f2_add(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint64_t f2_mul(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

// 2^x on the special-function unit (what exp2f compiles to here), where it is written: not moved
// behind the waits that follow it
__device__ __forceinline__ float exp2_here(float x) {
  float r;
  asm volatile("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// two neighbouring words of a row of scores as one such pair
__device__ __forceinline__ uint64_t f2_load(const uint32_t* r) {
  return f2_pack(__uint_as_float(r[0]), __uint_as_float(r[1]));
}
__device__ __forceinline__ void f2_store(uint32_t* r, uint64_t v) {
  float a, b;
  f2_unpack(v, a, b);
  r[0] = __float_as_uint(a);
  r[1] = __float_as_uint(b);
}

// a 4-byte copy from global to shared memory that runs on its own, and the wait for all of a
// thread's copies
__device__ __forceinline__ void cp_async4(float* smem_dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(tc::smem_u32(smem_dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

template <typename T> __device__ __forceinline__ uint32_t pack16(float a, float b) { return pair_word(a, b, T()); }

// ... of values that count as 0 where they are negative
template <typename T> __device__ __forceinline__ uint32_t pack16_relu(float a, float b);
template <> __device__ __forceinline__ uint32_t pack16_relu<__nv_bfloat16>(float a, float b) {
  uint32_t d;
  asm("cvt.rn.relu.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(b), "f"(a));
  return d;
}
template <> __device__ __forceinline__ uint32_t pack16_relu<__half>(float a, float b) {
  uint32_t d;
  asm("cvt.rn.relu.f16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(b), "f"(a));
  return d;
}

// Columns col .. col + 15 of a row of `cols` 16-bit values (a multiple of 8; padded columns are not part of
// it).  Neighbouring rows lie whole lines apart, so that a store takes a cycle per row: one of 32 bytes
// where rows keep to 32 bytes.
__device__ __forceinline__ void store_cols16(void* row, int col, int cols, const uint32_t (&v)[8]) {
  uint8_t* dst = static_cast<uint8_t*>(row) + col * 2;
  if ((cols & 15) == 0) {
    if (col < cols)
      asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(dst), "r"(v[0]), "r"(v[1]),
                   "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
                   : "memory");
  } else {
    if (col < cols) *reinterpret_cast<uint4*>(dst) = make_uint4(v[0], v[1], v[2], v[3]);
    if (col + 8 < cols) *reinterpret_cast<uint4*>(dst + 16) = make_uint4(v[4], v[5], v[6], v[7]);
  }
}

// Overlap of a kernel's prologue with the kernel before it in the stream: a kernel that the next
// one may start under says so, and one that was launched that way waits until all work before it
// is complete and visible (at once, when it was launched the ordinary way).
__device__ __forceinline__ void pdl_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// the 16 decisions of one Philox call as bits
__device__ __forceinline__ uint32_t keep_bits16(const uint4& kw) {
  const uint32_t w[4] = {kw.x, kw.y, kw.z, kw.w};
  uint32_t m = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i)       // bit 7 of the four bytes, gathered by one multiply
    m |= ((((w[i] >> 7) & 0x01010101u) * 0x01020408u) >> 24) << (4 * i);
  return m;
}

// bits 0 .. n - 1 (none for n <= 0, all for n >= 32)
__device__ __forceinline__ uint32_t low_bits(int n) {
  return n >= 32 ? 0xffffffffu : (1u << max(n, 0)) - 1u;
}

// A generator's state in uniform registers: a reduction over the warp tells the compiler that all
// lanes have the same, and the round keys of a call then cost no per-lane instruction.
struct PhiloxUniform {
  uint32_t seed_lo, seed_hi, offset_lo, offset_hi;
};
__device__ __forceinline__ PhiloxUniform philox_uniform(const PhiloxArgs& a) {
  uint64_t seed, offset;
  philox_unpack(a, seed, offset);
  return {__reduce_or_sync(0xffffffffu, static_cast<uint32_t>(seed)),
          __reduce_or_sync(0xffffffffu, static_cast<uint32_t>(seed >> 32)),
          __reduce_or_sync(0xffffffffu, static_cast<uint32_t>(offset)),
          __reduce_or_sync(0xffffffffu, static_cast<uint32_t>(offset >> 32))};
}
// philox_keep16 (common.cuh) of such a state
__device__ __forceinline__ uint4 philox_keep16(const PhiloxUniform& s, uint64_t index, uint32_t add4) {
  uint4 c = make_uint4(s.offset_lo, s.offset_hi, static_cast<uint32_t>(index),
                       static_cast<uint32_t>(index >> 32));
  uint32_t kx = s.seed_lo, ky = s.seed_hi;
#pragma unroll
  for (int r = 0; r < 7; ++r) {
    const uint2 m0 = mulhilo32(0xD2511F53u, c.x);
    const uint2 m1 = mulhilo32(0xCD9E8D57u, c.z);
    c = make_uint4(m1.y ^ c.y ^ kx, m1.x, m0.y ^ c.w ^ ky, m0.x);
    kx += 0x9E3779B9u;
    ky += 0xBB67AE85u;
  }
  c.x = (c.x & 0x7f7f7f7fu) + add4;
  c.y = (c.y & 0x7f7f7f7fu) + add4;
  c.z = (c.z & 0x7f7f7f7fu) + add4;
  c.w = (c.w & 0x7f7f7f7fu) + add4;
  return c;
}

// Position in a ring of N slots
template <int N>
struct Ring {
  int slot = 0;
  uint32_t phase = 0;
  __device__ __forceinline__ void step() {
    if (++slot == N) { slot = 0; phase ^= 1; }
  }
};

// Division of 0 .. 2^31 - 1 by a number that is fixed for a launch: a product and a shift, for d <= 2^s with
// mul = ceil(2^(31 + s) / d) = (2^(31 + s) + e) / d, e < d: n mul / 2^(31 + s) exceeds n / d by n e / (d 2^(31 + s)) < 1 / d.
// (A division by a run-time number is some 40 dependent instructions.)
struct FastDiv {
  uint32_t mul = 0, shift = 0;
  __host__ void set(int d) {
    shift = 0;
    while ((1 << shift) < d && shift < 30) ++shift;
    if ((1 << shift) < d) ++shift;
    const uint64_t top = uint64_t(1) << (31 + shift);
    mul = static_cast<uint32_t>((top + d - 1) / d);
    shift += 31;
  }
  __device__ __forceinline__ int operator()(int n) const {
    return static_cast<int>((static_cast<uint64_t>(static_cast<uint32_t>(n)) * mul) >> shift);
  }
};

// Row tiles of 128 of all (batch, head) pairs, walked by a persistent grid.  Under a causal
// mask the tiles differ in cost: they are ordered by cost, heaviest first, over all heads.
// Otherwise the tiles of one head are neighbours, so that the tensors they share stay in L2.
struct TileWalk {
  int row_tiles;     // per (batch, head)
  int bh0, nbh;      // range of (batch, head) pairs of this launch
  int by_cost;       // 0 = head-major, 1 = first tile heaviest, 2 = last tile heaviest
  FastDiv div;       // by row_tiles, or by nbh when ordered by cost
  __host__ void set(int tiles, int first_bh, int bhs, int cost) {
    row_tiles = tiles;
    bh0 = first_bh;
    nbh = bhs;
    by_cost = cost;
    div.set(cost == 0 ? tiles : bhs);
  }
  __device__ __forceinline__ int items() const { return row_tiles * nbh; }
  __device__ __forceinline__ void at(int item, int& tile, int& bh_local) const {
    if (by_cost == 0) {
      bh_local = div(item);
      tile = item - bh_local * row_tiles;
    } else {
      tile = div(item);
      bh_local = item - tile * nbh;
      if (by_cost == 2) tile = row_tiles - 1 - tile;
    }
  }
};

}  // namespace slapo
