// Flash attention forward on tcgen05 / TMEM (sm_100a).
//
// Tensors are [B, S, H, D] with D contiguous and arbitrary strides on B, S, H
// (so q/k/v slices of a fused QKV projection are read in place through 4-D
// TMA maps - no .contiguous() copies).  D is 64 or 128.
//
// Two kernels.  flash_fwd_groups_kernel takes most calls with more than one tile of 128 query rows: persistent
// CTAs, one per SM, with two softmax groups that take the key tiles of a work item in turn.  Persistent CTAs of
// flash_fwd_kernel (D = 64: two per SM with 256 of the 512 TMEM columns each; D = 128: one) take those with a
// single row tile, where the keys may be split over work items, and short calls with few key tiles (fwd_in_groups).
// Both walk over work items of 128 query rows of one (batch, head), for each of which they stream the keys in tiles of 128:
//   a thread     TMA: Q, K ring, V ring (runs ahead over tiles and over work items)
//   a thread     tcgen05.mma:  S = Q K^T       (fp32, 128 TMEM columns)
//                              O += P V        (P read from TMEM, fp32 accumulator in TMEM)
//   four warps   one query row per thread: online softmax in the exp2 domain, P back to TMEM as bf16 / fp16
// P and O are scaled by the running row maximum: when that of any of a warp's rows has grown, the
// warp's O rows are scaled in TMEM.  (Raising it only after a growth of 2^8 saves 2 - 9 % of the
// forward, but then the probabilities that count lie anywhere in their binade instead of at or just below 1,
// and the result's rounding error grows by up to 5 %: 0.00230 against 0.00220 at 512 keys, bf16.)
// A single query goes to flash_decode.cu.
//
// What bounds it: the special-function unit (one exp2 per score, 1024 cycles per 128 x 128 tile and SM) next to
// the issue slots of the softmax warps, and what a tile's chain has between them: waits of 50 - 250 cycles, reads of
// tensor memory, issuing (40 cycles a product).  Dropout is a template parameter: skipped at run time its draws are
// branches over code that has to be fetched, and taken at run time they do not mix with the exponentials
// (us, run time -> template: 32 x 512 x 16 heads of 64, p 0.1: 105.5 -> 99.3, without 76.9 -> 75.3; 4 x 2048
// causal: 83.5 -> 77.5).
//
// Biases are added from shared memory, which asynchronous copies fill a tile ahead: a warp's 32
// queries see 159 distances in a tile of 128 keys, against 128 loads per query.  Fetched by each
// thread as it needed them they stood in the tile's chain: 73 -> 36 us with T5's bias, 65 -> 35 us
// with a key bias (8 x 512 x 16 x 64).
#include "flash_common.cuh"
#include "kernels.h"

#include <mutex>

namespace slapo {

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                  const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

void ensure_cuda_context();   // gemm.cu

bool make_tmap_bshd(CUtensorMap* out, const void* base, uint64_t B, uint64_t S, uint64_t H,
                    uint64_t D, uint64_t stride_b, uint64_t stride_s, uint64_t stride_h,
                    uint32_t box_s, bool is_bf16) {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, []() {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres) ==
            cudaSuccess && qres == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(ptr);
  });
  if (fn == nullptr) return false;
  ensure_cuda_context();
  cuuint64_t dims[4] = {D, H, S, B};
  cuuint64_t strides[3] = {stride_h * 2, stride_s * 2, stride_b * 2};
  cuuint32_t box[4] = {64, 1, box_s, 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  CUresult r = fn(out, is_bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16,
                  4, const_cast<void*>(base), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}

// ------------------------------------------------------------------------ //
constexpr int kBlockM = 128;   // query rows per work item
constexpr int kBlockN = 128;   // keys per tile

struct FlashFwdParams {
  int B, H, Sq, Sk;
  int Dr;              // the tensors' head dimension (<= the kernel's tile width D, % 8 == 0):
                       // TMA zero-fills columns Dr .. D - 1 of every Q / K / V tile
  int k_steps;         // ceil(Dr / 16): steps of the Q K^T contraction
  TileWalk walk;
  int splits;          // work items per row tile: each takes tiles_per_split of the key tiles
  int tiles_per_split;
  float* part_o;       // splits > 1: [splits][B H Sq][Dr] unnormalised outputs and
  float2* part_ml;     // [splits][B H Sq] (maximum in the log2 domain, sum), see combine kernel
  void* O;             // [B, Sq, H, Dr] contiguous
  float* lse;          // [B, H, Sq] natural-log sum-exp of the scaled scores
  const float* kbias;  // [B, Sk] additive key bias or nullptr
  const float* rel;    // [H, Sq + Sk - 1] additive bias by (key - query) + Sq - 1, or nullptr
  float scale_log2;    // softmax scale * log2(e)
  int causal;
  float p_drop;        // effective probability thr7 / 128
  uint32_t thr7;
  PhiloxArgs rng;
  uint32_t idesc_qk, idesc_pv;
  int* status;
};

// ---- what a softmax warp of either kernel does with the scores of its 32 query rows and 128 keys ----
// Biases in shared memory: the tile's 128 key biases, then the relative bias of the 32 + 128 - 1 distances
// between the warp's queries and the tile's keys.
constexpr int kBiasFloats = 128 + 160;

// Biases of key tile `jt` of a work item on their way to `dst`: copied a tile ahead, element by
// element (rows start anywhere).  What lies outside of the tensors is masked later.
__device__ __forceinline__ void fwd_fetch_bias(const FlashFwdParams& p, float* dst, int tile, int quarter, int lane,
                                               int bh, int jt) {
  const int batch = bh / p.H, head = bh - batch * p.H, k0 = jt * kBlockN;
  if (p.kbias != nullptr) {
    const float* src = p.kbias + static_cast<int64_t>(batch) * p.Sk;
#pragma unroll
    for (int i = lane; i < 128; i += 32) cp_async4(dst + i, src + min(k0 + i, p.Sk - 1));
  }
  if (p.rel != nullptr) {
    // key - query from that of the warp's last row and the first key on
    const float* src = p.rel + static_cast<int64_t>(head) * (p.Sq + p.Sk - 1) + p.Sq - 1;
    const int d0 = k0 - (tile * kBlockM + quarter * 32 + 31);
#pragma unroll
    for (int i = lane; i < 160; i += 32)
      cp_async4(dst + 128 + i, src + max(1 - p.Sq, min(d0 + i, p.Sk - 1)));
  }
}

// They have arrived, are visible to the warp, and the readers of its other buffer are done.
__device__ __forceinline__ void fwd_land_bias(const FlashFwdParams& p, float* bias, int lane) {
  cp_async_wait();
  if (p.kbias != nullptr) {
#pragma unroll
    for (int i = lane; i < 128; i += 32) bias[i] *= kLog2e;      // (the elements that this lane copied)
  }
  __syncwarp();
}

// A row's scores, scaled to the log2 domain, plus its biases
template <int kSets>
__device__ __forceinline__ void fwd_add_bias(const FlashFwdParams& p, uint32_t (&raw)[kSets][32], const float* bias,
                                             int lane) {
  const uint64_t scale2 = f2_pack(p.scale_log2, p.scale_log2);
  const uint64_t log2e2 = f2_pack(kLog2e, kLog2e);
  if (p.kbias != nullptr) {
#pragma unroll
    for (int c = 0; c < kSets; ++c)
#pragma unroll
      for (int i = 0; i < 32; i += 4) {
        const float4 b = *reinterpret_cast<const float4*>(bias + c * 32 + i);
        f2_store(raw[c] + i, f2_fma(f2_load(raw[c] + i), scale2, f2_pack(b.x, b.y)));
        f2_store(raw[c] + i + 2, f2_fma(f2_load(raw[c] + i + 2), scale2, f2_pack(b.z, b.w)));
      }
  } else {
#pragma unroll
    for (int c = 0; c < kSets; ++c)
#pragma unroll
      for (int i = 0; i < 32; i += 2) f2_store(raw[c] + i, f2_mul(f2_load(raw[c] + i), scale2));
  }
  if (p.rel != nullptr) {
    // neighbouring lanes (queries) read neighbouring words
    const float* rel = bias + 128 + 31 - lane;
#pragma unroll
    for (int c = 0; c < kSets; ++c)
#pragma unroll
      for (int i = 0; i < 32; i += 2)
        f2_store(raw[c] + i,
                 f2_fma(f2_pack(rel[c * 32 + i], rel[c * 32 + i + 1]), log2e2, f2_load(raw[c] + i)));
  }
}

// -inf for keys that a row does not see, of the tile from k0 on; row0: the warp's first row
template <int kSets>
__device__ __forceinline__ void fwd_mask(const FlashFwdParams& p, uint32_t (&raw)[kSets][32], int k0, int row0,
                                         int lane) {
  const int diag = p.Sk - p.Sq;         // key j visible to query i iff j <= i + diag (causal)
  const int first_limit = p.causal ? min(p.Sk, row0 + diag + 1) : p.Sk;
  if (k0 + kSets * 32 > first_limit) {     // some lane of the warp masks something
    const int limit = (p.causal ? min(p.Sk, row0 + lane + diag + 1) : p.Sk) - k0;
#pragma unroll
    for (int c = 0; c < kSets; ++c) {
      const uint32_t seen = low_bits(limit - c * 32);
#pragma unroll
      for (int i = 0; i < 32; ++i)
        if (!(seen & (1u << i))) raw[c][i] = 0xff800000u;   // -inf
    }
  }
}

template <int kSets>
__device__ __forceinline__ float fwd_max(const uint32_t (&raw)[kSets][32]) {
  float mm[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};  // 4 chains for ILP
#pragma unroll
  for (int c = 0; c < kSets; ++c)
#pragma unroll
    for (int i = 0; i < 32; i += 2) {
      float& m = mm[(i >> 1) & 3];
      m = fmaxf(m, fmaxf(__uint_as_float(raw[c][i]), __uint_as_float(raw[c][i + 1])));
    }
  return fmaxf(fmaxf(mm[0], mm[1]), fmaxf(mm[2], mm[3]));
}

template <int D>
struct FwdSmem {
  static constexpr int kTile = 128 * D * 2;          // one [128 x D] 16-bit tile
  static constexpr int kStages = 2;                  // K and V rings
  static constexpr int kCtas = D == 64 ? 2 : 1;      // per SM: shared memory and TMEM columns
  static constexpr int kK = kTile;
  static constexpr int kV = kK + kStages * kTile;
  // (per softmax warp, twice: this tile's biases and the next one's)
  static constexpr int kBias = kV + kStages * kTile;
  static constexpr int kBars = kBias + 4 * 2 * kBiasFloats * 4;
  static constexpr int kTotal = kBars + 20 * 8 + 1024;
};

// kGeneral: key bias, relative bias, causal mask, a ragged last key tile or a scale <= 0;
// without any of them the kernel takes row maxima on the raw scores and every probability is
// one fused multiply-add plus one exp2.
template <int D, bool kGeneral, bool kDrop, typename T>
__global__ void __launch_bounds__(192, D == 64 ? 2 : 1)
flash_fwd_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                 const __grid_constant__ CUtensorMap tm_v, const FlashFwdParams p) {
  using L = FwdSmem<D>;
  constexpr int kTileBytes = L::kTile;
  constexpr int kStages = L::kStages;
  constexpr int kBlkBytes = 128 * 128;      // one [128 rows x 64 cols] swizzled block
  constexpr int kDBlocks = D / 64;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint8_t* s_q = smem;
  uint8_t* s_k = smem + L::kK;
  uint8_t* s_v = smem + L::kV;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::kBars);
  uint64_t* q_full = bars;            // 1
  uint64_t* q_empty = bars + 1;       // 1
  uint64_t* k_full = bars + 2;        // 2
  uint64_t* k_empty = bars + 4;       // 2
  uint64_t* v_full = bars + 6;        // 2
  uint64_t* v_empty = bars + 8;       // 2
  uint64_t* s_full = bars + 10;       // S of a tile is in tensor memory
  uint64_t* s_free = bars + 11;       // ... and has been read out of it
  uint64_t* p_full = bars + 12;       // P of a tile is in tensor memory
  uint64_t* pv_done = bars + 13;      // O includes a tile
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 14);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int diag = p.Sk - p.Sq;  // key j visible to query i iff j <= i + diag (causal)
  constexpr uint32_t kTmemCols = D == 64 ? 256 : 512;
  constexpr uint32_t kColP = 128, kColO = 192;    // S: 0

  if (threadIdx.x == 0) {
    tc::mbar_init(q_full, 1);
    tc::mbar_init(q_empty, 1);
    for (int i = 0; i < 2; ++i) {
      tc::mbar_init(&k_full[i], 1);
      tc::mbar_init(&k_empty[i], 1);
      tc::mbar_init(&v_full[i], 1);
      tc::mbar_init(&v_empty[i], 1);
    }
    tc::mbar_init(s_full, 1);
    tc::mbar_init(s_free, 4);
    tc::mbar_init(p_full, 4);
    tc::mbar_init(pv_done, 1);
    *abort_flag = 0;
    tc::fence_barrier_init();
  }
  if (warp == 1) {
    tc::tmem_alloc(tmem_slot, kTmemCols);
    tc::tmem_relinquish();
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  const int items = p.walk.items() * p.splits;
  // row tile, (batch, head) and key tiles [j0, j0 + n) of a work item
  auto item_at = [&](int item, int& tile, int& bh, int& j0) {
    const int unit = p.splits == 1 ? item : item / p.splits;
    p.walk.at(unit, tile, bh);
    int n = (p.Sk + kBlockN - 1) / kBlockN;
    if (p.causal) {
      const int last_key = min(p.Sk, tile * kBlockM + kBlockM + diag);
      n = max(1, min(n, (last_key + kBlockN - 1) / kBlockN));
    }
    j0 = 0;
    if (p.splits > 1) {     // (one row tile per head: every split has at least one key tile)
      j0 = (item - unit * p.splits) * p.tiles_per_split;
      n = min(p.tiles_per_split, n - j0);
    }
    return n;
  };

  if (warp == 0) {
    if (tc::elect_one()) {
      tc::tma_prefetch_desc(&tm_q);
      tc::tma_prefetch_desc(&tm_k);
      tc::tma_prefetch_desc(&tm_v);
      bool ok = true;
      int t = 0, w = 0;
      for (int item = blockIdx.x; item < items && ok; item += gridDim.x, ++w) {
        int tile, bh, j0;
        const int n = item_at(item, tile, bh, j0);
        const int batch = bh / p.H, head = bh - batch * p.H;
        if (!tc::mbar_wait(q_empty, (w & 1) ^ 1, abort_flag)) { ok = false; break; }
        tc::mbar_arrive_expect_tx(q_full, kTileBytes);
#pragma unroll
        for (int d = 0; d < kDBlocks; ++d)
          tc::tma_load_4d(s_q + d * kBlkBytes, &tm_q, q_full, d * 64, head, tile * kBlockM, batch);
        for (int j = 0; j < n; ++j, ++t) {
          const int st = t % kStages;
          const uint32_t ph = (t / kStages) & 1;
          if (!tc::mbar_wait(&k_empty[st], ph ^ 1, abort_flag)) { ok = false; break; }
          tc::mbar_arrive_expect_tx(&k_full[st], kTileBytes);
#pragma unroll
          for (int d = 0; d < kDBlocks; ++d)
            tc::tma_load_4d(s_k + st * kTileBytes + d * kBlkBytes, &tm_k, &k_full[st], d * 64, head,
                            (j0 + j) * kBlockN, batch);
          if (!tc::mbar_wait(&v_empty[st], ph ^ 1, abort_flag)) { ok = false; break; }
          tc::mbar_arrive_expect_tx(&v_full[st], kTileBytes);
#pragma unroll
          for (int d = 0; d < kDBlocks; ++d)
            tc::tma_load_4d(s_v + st * kTileBytes + d * kBlkBytes, &tm_v, &v_full[st], d * 64, head,
                            (j0 + j) * kBlockN, batch);
        }
      }
    }
  } else if (warp == 1) {
    if (tc::elect_one()) {
      constexpr uint32_t kDescHi = tc::smem_desc_hi(1024);
      const uint32_t q_desc = tc::smem_desc_lo(tc::smem_u32(s_q), 16);
      const uint32_t k_desc = tc::smem_desc_lo(tc::smem_u32(s_k), 16);
      const uint32_t v_desc = tc::smem_desc_lo(tc::smem_u32(s_v), kBlkBytes);
      // S of tile t (the w-th item's; `last`: its last one)
      auto issue_qk = [&](int t, int w, bool first, bool last) -> bool {
        const int st = t % kStages;
        if (first && !tc::mbar_wait(q_full, w & 1, abort_flag)) return false;
        if (!tc::mbar_wait(&k_full[st], (t / kStages) & 1, abort_flag)) return false;
        tc::fence_after_sync();
        const uint32_t k_at = k_desc + st * (kTileBytes >> 4);
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
          if (kk < p.k_steps) {
            const uint32_t off = ((kk >> 2) * kBlkBytes + (kk & 3) * 32) >> 4;
            tc::umma_f16(tmem_base, tc::smem_desc_words(q_desc + off, kDescHi),
                         tc::smem_desc_words(k_at + off, kDescHi), p.idesc_qk, kk != 0 ? 1u : 0u);
          }
        }
        tc::umma_commit(s_full);
        tc::umma_commit(&k_empty[st]);
        if (last) tc::umma_commit(q_empty);
        return true;
      };
      bool ok = true;
      int t = 0, w = 0;
      int item = blockIdx.x;
      int n = 0;
      if (item < items) {
        int tile, bh, j0;
        n = item_at(item, tile, bh, j0);
        ok = issue_qk(0, 0, true, n == 1);
      }
      while (item < items && ok) {
        const int next_item = item + gridDim.x;
        int next_n = 0;
        if (next_item < items) {
          int tile, bh, j0;
          next_n = item_at(next_item, tile, bh, j0);
        }
        for (int j = 0; j < n; ++j, ++t) {
          auto issue_next = [&]() -> bool {
            if (j + 1 < n) return issue_qk(t + 1, w, false, j + 2 == n);
            if (next_n > 0) return issue_qk(t + 1, w + 1, true, next_n == 1);
            return true;
          };
          // S has been read out: the next tile's goes in its place under this one's softmax
          if (!tc::mbar_wait(s_free, t & 1, abort_flag) || !issue_next()) { ok = false; break; }
          const int st = t % kStages;
          if (!tc::mbar_wait(&v_full[st], (t / kStages) & 1, abort_flag) ||
              !tc::mbar_wait(p_full, t & 1, abort_flag)) { ok = false; break; }
          tc::fence_after_sync();
          const uint32_t v_at = v_desc + st * (kTileBytes >> 4);
#pragma unroll
          for (int kk = 0; kk < kBlockN / 16; ++kk)
            tc::umma_f16_ts(tmem_base + kColO, tmem_base + kColP + kk * 8,
                            tc::smem_desc_words(v_at + ((kk * 2048) >> 4), kDescHi), p.idesc_pv,
                            (j | kk) != 0 ? 1u : 0u);
          tc::umma_commit(pv_done);
          tc::umma_commit(&v_empty[st]);
        }
        item = next_item;
        n = next_n;
        ++w;
      }
    }
  } else {
    // ------------------------------ softmax warps ------------------------------
    const int quarter = warp & 3;
    const int row_in_tile = quarter * 32 + lane;
    const uint32_t tmem_row = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
    float* bias_buf = reinterpret_cast<float*>(smem + L::kBias) + (warp - 2) * 2 * kBiasFloats;
    PhiloxUniform rng{};
    if constexpr (kDrop) rng = philox_uniform(p.rng);
    const uint32_t add4 = (128u - p.thr7) * 0x01010101u;
    const int sk16 = (p.Sk + 15) >> 4;
    // scores are brought to the log2 domain before the maximum only where something is added
    // to them (or the scale would turn the maximum around)
    const bool biased = kGeneral && (p.kbias != nullptr || p.rel != nullptr || !(p.scale_log2 > 0.f));
    const float sc = biased ? 1.f : p.scale_log2;
    auto fetch_bias = [&](int tile, int bh, int jt, int buf) {
      fwd_fetch_bias(p, bias_buf + buf * kBiasFloats, tile, quarter, lane, bh, jt);
    };
    bool ok = true;
    int t = 0;
    if (biased && static_cast<int>(blockIdx.x) < items) {
      int tile, bh, j0;
      item_at(blockIdx.x, tile, bh, j0);
      fetch_bias(tile, bh, j0, 0);
    }
    for (int item = blockIdx.x; item < items && ok; item += gridDim.x) {
      int tile, bh, j0;
      const int n = item_at(item, tile, bh, j0);
      const int batch = bh / p.H, head = bh - batch * p.H;
      const int row = tile * kBlockM + row_in_tile;
      const uint64_t drop_row_base =
          (static_cast<uint64_t>(bh) * p.Sq + min(row, p.Sq - 1)) * sk16;
      float m_ref = -INFINITY;
      uint64_t l2 = 0;      // two fp32 partial row sums
      for (int j = 0; j < n; ++j, ++t) {
        const int k0 = (j0 + j) * kBlockN;
        const float* bias = bias_buf + (t & 1) * kBiasFloats;
        if (kGeneral && biased) {
          fwd_land_bias(p, bias_buf + (t & 1) * kBiasFloats, lane);
          if (j + 1 < n) {
            fetch_bias(tile, bh, j0 + j + 1, (t + 1) & 1);
          } else if (item + static_cast<int>(gridDim.x) < items) {
            int next_tile, next_bh, next_j0;
            item_at(item + gridDim.x, next_tile, next_bh, next_j0);
            fetch_bias(next_tile, next_bh, next_j0, (t + 1) & 1);
          }
        }
        if (!tc::mbar_wait_warp(s_full, t & 1, abort_flag)) { ok = false; break; }
        tc::fence_after_sync();
        uint32_t raw[4][32];
#pragma unroll
        for (int c = 0; c < 4; ++c) tc::tmem_ld_x32(tmem_row + c * 32, raw[c]);
        tc::tmem_ld_wait();
        tc::fence_before_sync();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(s_free);
        if constexpr (kGeneral) {
          if (biased) fwd_add_bias(p, raw, bias, lane);
          fwd_mask(p, raw, k0, tile * kBlockM + quarter * 32, lane);
        }
        const float m_tile = fwd_max(raw) * sc;
        // P of the tile before has been read (and O includes it)
        if (t > 0 && !tc::mbar_wait_warp(pv_done, (t - 1) & 1, abort_flag)) { ok = false; break; }
        tc::fence_after_sync();
        if (j == 0) {
          m_ref = m_tile;
        } else if (__any_sync(0xffffffffu, m_tile > m_ref)) {
          const float m_new = fmaxf(m_ref, m_tile);
          const float alpha = m_ref == -INFINITY ? 0.f : exp2f(m_ref - m_new);
          const uint64_t alpha2 = f2_pack(alpha, alpha);
#pragma unroll
          for (int c = 0; c < D / 16; ++c) {
            uint32_t o[16];
            tc::tmem_ld_x16(tmem_row + kColO + c * 16, o);
            tc::tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 16; ++i)
              o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
            tc::tmem_st_x16(tmem_row + kColO + c * 16, o);
          }
          l2 = f2_mul(l2, alpha2);
          m_ref = m_new;
        }
        const float m_use = m_ref == -INFINITY ? 0.f : m_ref;
        const uint64_t sc2 = f2_pack(sc, sc), nm2 = f2_pack(-m_use, -m_use);
        if (j == 0) l2 = 0;
        uint64_t la = l2, lb = 0;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint32_t pk[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const uint64_t x = f2_fma(
                f2_pack(__uint_as_float(raw[c][2 * i]), __uint_as_float(raw[c][2 * i + 1])), sc2, nm2);
            float a, b;
            f2_unpack(x, a, b);
            a = exp2f(a);
            b = exp2f(b);
            if (i & 1) lb = f2_add(lb, f2_pack(a, b));
            else la = f2_add(la, f2_pack(a, b));
            pk[i] = pack16<T>(a, b);
          }
          if constexpr (kDrop) {
            // dropped probabilities are cleared in the packed 16-bit pairs
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const uint4 kw = philox_keep16(rng, drop_row_base + ((k0 + c * 32 + h * 16) >> 4), add4);
              const uint32_t wd[4] = {kw.x, kw.y, kw.z, kw.w};
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                pk[h * 8 + i * 2 + 0] &= keep_mask_pair(wd[i], 0);
                pk[h * 8 + i * 2 + 1] &= keep_mask_pair(wd[i], 1);
              }
            }
          }
          tc::tmem_st_x16(tmem_row + kColP + c * 16, pk);
        }
        l2 = f2_add(la, lb);
        tc::tmem_st_wait();
        tc::fence_before_sync();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(p_full);
      }
      if (!ok) break;
      // O of this item (the next item's first P V product waits for this warp's next P)
      if (!tc::mbar_wait_warp(pv_done, (t - 1) & 1, abort_flag)) { ok = false; break; }
      tc::fence_after_sync();
      float l_run, l_hi;
      f2_unpack(l2, l_run, l_hi);
      l_run += l_hi;
      if (p.splits > 1) {
        // this split's share: unnormalised output, maximum and sum
        const int split = item - item / p.splits * p.splits;
        const int64_t at = (static_cast<int64_t>(split) * p.B * p.H + bh) * p.Sq + min(row, p.Sq - 1);
#pragma unroll
        for (int c = 0; c < D / 32; ++c) {
          uint32_t o[32];
          tc::tmem_ld_x32(tmem_row + kColO + c * 32, o);
          tc::tmem_ld_wait();
          if (row < p.Sq) {
#pragma unroll
            for (int g = 0; g < 8; ++g)
              if (c * 32 + g * 4 < p.Dr)
                *reinterpret_cast<uint4*>(p.part_o + at * p.Dr + c * 32 + g * 4) =
                    make_uint4(o[4 * g], o[4 * g + 1], o[4 * g + 2], o[4 * g + 3]);
          }
        }
        tc::fence_before_sync();
        if (row < p.Sq) p.part_ml[at] = make_float2(m_ref, l_run);
        continue;
      }
      const float inv = l_run > 0.f ? 1.f / (l_run * (1.f - p.p_drop)) : 0.f;
      uint8_t* dst = static_cast<uint8_t*>(p.O) +
                     ((static_cast<int64_t>(batch) * p.Sq + min(row, p.Sq - 1)) * p.H + head) * p.Dr * 2;
#pragma unroll
      for (int c = 0; c < D / 32; ++c) {
        uint32_t o[32];
        tc::tmem_ld_x32(tmem_row + kColO + c * 32, o);
        tc::tmem_ld_wait();
        if (row < p.Sq) {
#pragma unroll
          for (int g = 0; g < 4; ++g) {
            if (c * 32 + g * 8 < p.Dr) {     // padded columns are not part of the output
              uint32_t v[4];
#pragma unroll
              for (int i = 0; i < 4; ++i)
                v[i] = pack16<T>(__uint_as_float(o[g * 8 + 2 * i]) * inv,
                                 __uint_as_float(o[g * 8 + 2 * i + 1]) * inv);
              *reinterpret_cast<uint4*>(dst + (c * 32 + g * 8) * 2) = make_uint4(v[0], v[1], v[2], v[3]);
            }
          }
        }
      }
      tc::fence_before_sync();
      if (row < p.Sq) {
        const float m_nat = (m_ref == -INFINITY ? 0.f : m_ref) * 0.6931471805599453f;
        p.lse[static_cast<int64_t>(bh) * p.Sq + row] = l_run > 0.f ? m_nat + logf(l_run) : -INFINITY;
      }
    }
    if (kGeneral) cp_async_wait();      // (a give-up leaves copies under way)
  }

  tc::fence_before_sync();
  __syncthreads();
  if (threadIdx.x == 0 && *abort_flag != 0 && p.status != nullptr) atomicExch(p.status, 2);
  if (warp == 1) {
    tc::fence_after_sync();
    tc::tmem_dealloc(tmem_base, kTmemCols);
  }
}

// Registers per thread of the warpgroups: issuing, softmax (two), O; together the 128 per thread that
// 512 threads are launched with.
constexpr int kFwdRegsIssue = 72, kFwdRegsSoftmax = 176, kFwdRegsO = 88;
static_assert(kFwdRegsIssue + 2 * kFwdRegsSoftmax + kFwdRegsO <= 4 * 128, "more registers than the block has");

template <int D>
struct GroupsSmem {
  static constexpr int kTile = 128 * D * 2;          // one [128 x D] 16-bit tile
  static constexpr int kQ = 2;                       // Q tiles: this item's and the next one's
  static constexpr int kStages = D == 64 ? 4 : 2;    // K and V rings
  static constexpr int kK = kQ * kTile;
  static constexpr int kV = kK + kStages * kTile;
  // (per softmax warp, twice: this tile's biases and the next one's)
  static constexpr int kBias = kV + kStages * kTile;
  static constexpr int kAlpha = kBias + 8 * 2 * kBiasFloats * 4;     // [group][tile parity][128] floats
  static constexpr int kMl = kAlpha + 2 * 2 * 128 * 4;               // [group][item parity][128] float2
  static constexpr int kBars = kMl + 2 * 2 * 128 * 8;
  static constexpr int kTotal = kBars + 48 * 8 + 1024;
};

// The forward for more than one row tile: two softmax groups in one CTA that take the key tiles of a work
// item in turn, each with an online softmax and an accumulator of its own, which a third group of warps
// scales when maxima grow and merges at the end.
// One thread issues all products: two products' queue is served in the order it is filled in, so that
// a group's P V and next S do not wait behind each other's halves (a thread per group: 128 -> 153 us for 4 x 2048
// x 16 x 128).  Between two tiles of a group (some 4000 cycles) lie 2000 - 2500 of exponentials that the groups
// take together, the products and 300 - 500 each of reading S, its maximum, handing the factors for O over and
// waiting; D = 128 waits 1300 for P V and S, whose columns P lies in.  (The groups held apart, so that one has
// the special-function unit to itself: no difference.)
// The scores stay in tensor memory and come out of it twice, in pieces.  Held in registers from the maximum to
// the exponentials, 128 a row, they left too few for dropout's draws and biases, which spilled:
// 32 x 512 x 16 x 64, p 0.1: 87 -> 79 us; 4 x 1000 x 32 x 80 causal with key bias: 66 -> 60.
// Measured, all of that together (us; one softmax group in each of two CTAs per SM for D = 64, two issuing threads
// for D = 128 -> this): 32 x 512 x 16 x 64, p 0.1: 105.5 -> 78.7, without 76.9 -> 60.9; 4 x 2048 x 16 x 64 causal:
// 83.5 -> 74.9; 8 x 512 x 16 x 64 with T5's bias, key bias and p 0.1: 43.7 -> 41.2; 1 x 512 x 16 x 64, p 0.1: 12.9 ->
// 9.4; 4 x 2048 x 16 x 128 causal: 111 -> 91, all keys 154 -> 128; 4 x 1000 x 32 x 80 causal with key bias: 70 -> 60;
// 4 x 1024 x 16 x 128, p 0.1: 61 -> 49.  With a single row tile there are too few tiles to share out: 2 x 60 x 60 x
// 8 x 128: 6.5 -> 8.0 (which calls come here: fwd_in_groups).
template <int D, bool kGeneral, bool kDrop, typename T>
__global__ void __launch_bounds__(512, 1)
flash_fwd_groups_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                 const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ FlashFwdParams p) {
  using L = GroupsSmem<D>;
  constexpr int kTileBytes = L::kTile;
  constexpr int kStages = L::kStages, kQ = L::kQ;
  constexpr int kBlkBytes = 128 * 128;      // one [128 rows x 64 cols] swizzled block
  constexpr int kDBlocks = D / 64;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::kBars);
  uint64_t* q_full = bars;            // kQ (2)
  uint64_t* q_empty = bars + 2;
  uint64_t* k_full = bars + 4;        // kStages (<= 4)
  uint64_t* k_empty = bars + 8;
  uint64_t* v_full = bars + 12;
  uint64_t* v_empty = bars + 16;
  uint64_t* s_full = bars + 20;       // one per softmax group from here on: S of a tile is complete
  uint64_t* p_full = bars + 22;       // [group][half of the keys]: P is in tensor memory (4 warps)
  uint64_t* pv_done = bars + 26;      // O includes a tile
  uint64_t* o_ready = bars + 28;      // O is scaled (or free) for a tile (4 warps)
  uint64_t* alpha_ready = bars + 30;  // [group][tile parity]: a tile's factors (4 warps)
  uint64_t* ml_ready = bars + 34;     // [group][item parity]: an item's maxima and sums (4 warps)
  uint64_t* s_free = bars + 38;       // S of a tile has been read (4 warps; D = 64)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 40);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  float* s_alpha = reinterpret_cast<float*>(smem + L::kAlpha);
  float2* s_ml = reinterpret_cast<float2*>(smem + L::kMl);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int diag = p.Sk - p.Sq;  // key j visible to query i iff j <= i + diag (causal)
  constexpr uint32_t kTmemCols = 512;
  // S, O and P of the two groups.  For D = 128 P is written over S: the next S of a group goes into the
  // tensor core's queue behind the product that uses P up.  For D = 64 P has columns of its own and the next
  // S is formed as soon as this one has been read.
  // Relied on here: a later product of the same thread writes its result only after an earlier one has read its operands.
  // PTX promises two tcgen05.mma in their order of issue for the same accumulator and shape; these differ in both, and
  // a wait on pv_done, 400 - 650 cycles from commit to wait, would be what the documents ask for.  The order is
  // what the hardware shows: no difference in repeated and random calls, tests/test_flash_order_gpu.py.
  constexpr bool kOver = D == 128;
  constexpr uint32_t kColS = 0, kColO = 256, kColP = kOver ? kColS : 384, kPGroup = kOver ? 128 : 64;

  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) {
      tc::mbar_init(&q_full[i], 1);
      tc::mbar_init(&q_empty[i], 1);
      tc::mbar_init(&s_full[i], 1);
      tc::mbar_init(&pv_done[i], 1);
      tc::mbar_init(&o_ready[i], 4);
      tc::mbar_init(&s_free[i], 4);
    }
    for (int i = 0; i < kStages; ++i) {
      tc::mbar_init(&k_full[i], 1);
      tc::mbar_init(&k_empty[i], 1);
      tc::mbar_init(&v_full[i], 1);
      tc::mbar_init(&v_empty[i], 1);
    }
    for (int i = 0; i < 4; ++i) {
      tc::mbar_init(&p_full[i], 4);
      tc::mbar_init(&alpha_ready[i], 4);
      tc::mbar_init(&ml_ready[i], 4);
    }
    *abort_flag = 0;
    tc::fence_barrier_init();
  }
  if (warp == 1) {
    tc::tmem_alloc(tmem_slot, kTmemCols);
    tc::tmem_relinquish();
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  const int items = p.walk.items();       // (several row tiles: keys are not split)
  // row tile, (batch, head) and number of key tiles of a work item
  auto item_at = [&](int item, int& tile, int& bh) {
    p.walk.at(item, tile, bh);
    int n = (p.Sk + kBlockN - 1) / kBlockN;
    if (p.causal) {
      const int last_key = min(p.Sk, min(tile * kBlockM + kBlockM, p.Sq) + diag);
      n = max(1, min(n, (last_key + kBlockN - 1) / kBlockN));
    }
    return n;
  };

  if (warp < 4) {
    tc::regs_dec<kFwdRegsIssue>();
    if (tc::elect_one()) {
      constexpr uint32_t kDescHi = tc::smem_desc_hi(1024);
      constexpr uint32_t kStep = kTileBytes >> 4;
      bool ok = true;
      if (warp == 0) {
        // ------------------------------ loads ------------------------------
        tc::tma_prefetch_desc(&tm_q);
        tc::tma_prefetch_desc(&tm_k);
        tc::tma_prefetch_desc(&tm_v);
        Ring<kQ> q;
        Ring<kStages> r;
        for (int item = blockIdx.x; item < items && ok; item += gridDim.x, q.step()) {
          int tile, bh;
          const int n = item_at(item, tile, bh);
          const int batch = bh / p.H, head = bh - batch * p.H;
          ok = false;
          if (!tc::mbar_wait(&q_empty[q.slot], q.phase ^ 1, abort_flag)) break;
          tc::mbar_arrive_expect_tx(&q_full[q.slot], kTileBytes);
#pragma unroll
          for (int d = 0; d < kDBlocks; ++d)
            tc::tma_load_4d(smem + q.slot * kTileBytes + d * kBlkBytes, &tm_q, &q_full[q.slot], d * 64, head,
                            tile * kBlockM, batch);
          for (int j = 0; j < n; ++j, r.step()) {
            ok = false;
            const int k0 = j * kBlockN;
            if (!tc::mbar_wait(&k_empty[r.slot], r.phase ^ 1, abort_flag)) break;
            tc::mbar_arrive_expect_tx(&k_full[r.slot], kTileBytes);
#pragma unroll
            for (int d = 0; d < kDBlocks; ++d)
              tc::tma_load_4d(smem + L::kK + r.slot * kTileBytes + d * kBlkBytes, &tm_k, &k_full[r.slot], d * 64,
                              head, k0, batch);
            if (!tc::mbar_wait(&v_empty[r.slot], r.phase ^ 1, abort_flag)) break;
            tc::mbar_arrive_expect_tx(&v_full[r.slot], kTileBytes);
#pragma unroll
            for (int d = 0; d < kDBlocks; ++d)
              tc::tma_load_4d(smem + L::kV + r.slot * kTileBytes + d * kBlkBytes, &tm_v, &v_full[r.slot], d * 64,
                              head, k0, batch);
            ok = true;
          }
        }
      } else if (warp == 1) {
        // ------------------------------ products ------------------------------
        // In the order S(0), S(1), then for every tile u of the CTA's sequence P V(u) and S(u + 2), for D = 64
        // the other way round: S as soon as the one before it in its columns has been read.
        const uint32_t q_desc = tc::smem_desc_lo(tc::smem_u32(smem), 16);
        const uint32_t k_desc = tc::smem_desc_lo(tc::smem_u32(smem + L::kK), 16);
        const uint32_t v_desc = tc::smem_desc_lo(tc::smem_u32(smem + L::kV), kBlkBytes);
        Ring<kQ> q;
        Ring<kStages> rk, rv;
        int s_item = blockIdx.x, s_n = 0, s_j = 0;      // the next S
        int tile, bh;
        if (s_item < items) s_n = item_at(s_item, tile, bh);
        auto form_s = [&](int g) -> bool {
          if (s_item >= items) return true;
          if (s_j == 0 && !tc::mbar_wait(&q_full[q.slot], q.phase, abort_flag)) return false;
          if (!tc::mbar_wait(&k_full[rk.slot], rk.phase, abort_flag)) return false;
          tc::fence_after_sync();
#pragma unroll
          for (int kk = 0; kk < D / 16; ++kk) {
            if (kk < p.k_steps) {
              const uint32_t off = ((kk >> 2) * kBlkBytes + (kk & 3) * 32) >> 4;
              tc::umma_f16(tmem_base + kColS + g * 128, tc::smem_desc_words(q_desc + q.slot * kStep + off, kDescHi),
                           tc::smem_desc_words(k_desc + rk.slot * kStep + off, kDescHi), p.idesc_qk,
                           kk != 0 ? 1u : 0u);
            }
          }
          tc::umma_commit(&s_full[g]);
          tc::umma_commit(&k_empty[rk.slot]);
          rk.step();
          if (++s_j == s_n) {
            tc::umma_commit(&q_empty[q.slot]);
            q.step();
            s_j = 0;
            s_item += gridDim.x;
            if (s_item < items) s_n = item_at(s_item, tile, bh);
          }
          return true;
        };
        ok = form_s(0) && form_s(1);
        int u = 0;
        for (int item = blockIdx.x; item < items && ok; item += gridDim.x) {
          const int n = item_at(item, tile, bh);
          for (int j = 0; j < n; ++j, ++u, rv.step()) {
            const int g = u & 1;
            const uint32_t ph = (u >> 1) & 1;
            ok = false;
            if (!kOver && (!tc::mbar_wait(&s_free[g], ph, abort_flag) || !form_s(g))) break;
            if (!tc::mbar_wait(&v_full[rv.slot], rv.phase, abort_flag) ||
                !tc::mbar_wait(&o_ready[g], ph, abort_flag))
              break;
            // the first half of the keys' products run under the other half's softmax
#pragma unroll
            for (int half = 0; half < 2; ++half) {
              if (!tc::mbar_wait(&p_full[g * 2 + half], ph, abort_flag)) break;
              tc::fence_after_sync();
#pragma unroll
              for (int kk = half * 4; kk < half * 4 + 4; ++kk)
                tc::umma_f16_ts(tmem_base + kColO + g * D, tmem_base + kColP + g * kPGroup + kk * 8,
                                tc::smem_desc_words(v_desc + rv.slot * kStep + ((kk * 2048) >> 4), kDescHi),
                                p.idesc_pv, (j >= 2 || kk != 0) ? 1u : 0u);
            }
            if (*abort_flag != 0) break;
            tc::umma_commit(&pv_done[g]);
            tc::umma_commit(&v_empty[rv.slot]);
            // (no wait: S goes over a P that the products just issued still read; the order is explained at kOver)
            if (kOver && !form_s(g)) break;
            ok = true;
          }
        }
      }
    }
  } else if (warp >= 12) {
    tc::regs_dec<kFwdRegsO>();
    // ------------------------------ O: scaled when maxima grow, read out at the end ------------------
    const int quarter = warp & 3;
    const int row_in_tile = quarter * 32 + lane;
    const uint32_t tmem_row = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
    bool ok = true;
    int u = 0;
    int parts[2] = {0, 0};        // items that each group has had a part in
    // D = 64: the item before, its row of O packed, is stored once its columns have been given up
    constexpr bool kHold = D == 64;
    uint32_t done[kHold ? D / 16 : 1][8];
    T* done_at = nullptr;
    auto flush = [&]() {
      if (!kHold || done_at == nullptr) return;
#pragma unroll
      for (int c = 0; c < D / 16; ++c) store_cols16(done_at, c * 16, p.Dr, done[kHold ? c : 0]);
    };
    for (int item = blockIdx.x; item < items && ok; item += gridDim.x) {
      int tile, bh;
      const int n = item_at(item, tile, bh);
      const int first = u;
      // (O of the item before is in registers)
      __syncwarp();
      if (lane == 0) {
        tc::mbar_arrive(&o_ready[first & 1]);
        if (n > 1) tc::mbar_arrive(&o_ready[(first & 1) ^ 1]);
      }
      flush();
      u += n;
      for (int t = first + 2; t < u; ++t) {
        const int g = t & 1, k = t >> 1;
        if (!tc::mbar_wait_warp(&alpha_ready[g * 2 + (k & 1)], (k >> 1) & 1, abort_flag)) { ok = false; break; }
        const float alpha = s_alpha[(g * 2 + (k & 1)) * 128 + row_in_tile];
        // (also where nothing grows: a warp's arrivals for two tiles of a group must not meet in one phase)
        if (!tc::mbar_wait_warp(&pv_done[g], (k & 1) ^ 1, abort_flag)) { ok = false; break; }
        if (__any_sync(0xffffffffu, alpha != 1.f)) {
          tc::fence_after_sync();
          const uint64_t alpha2 = f2_pack(alpha, alpha);
#pragma unroll 1
          for (int c = 0; c < D; c += 32) {
            uint32_t o[32];
            tc::tmem_ld_x32(tmem_row + kColO + g * D + c, o);
            tc::tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; i += 2) f2_store(o + i, f2_mul(f2_load(o + i), alpha2));
            tc::tmem_st_x32(tmem_row + kColO + g * D + c, o);
          }
          tc::tmem_st_wait();
          tc::fence_before_sync();
        }
        __syncwarp();
        tc::mbar_arrive_if(&o_ready[g], lane == 0);
      }
      if (!ok) break;
      // both groups' maxima and sums, and their last products
      float m_g[2], l_g[2];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        m_g[i] = -INFINITY;
        l_g[i] = 0.f;
        const int last = u - 1 - ((u - 1 - i) & 1);      // the group's last tile so far
        if (last >= first) {
          const int c = parts[i]++;
          if (!tc::mbar_wait_warp(&ml_ready[i * 2 + (c & 1)], (c >> 1) & 1, abort_flag) ||
              !tc::mbar_wait_warp(&pv_done[i], (last >> 1) & 1, abort_flag)) { ok = false; break; }
          const float2 ml = s_ml[(i * 2 + (c & 1)) * 128 + row_in_tile];
          m_g[i] = ml.x;
          l_g[i] = ml.y;
        }
      }
      if (!ok) break;
      tc::fence_after_sync();
      const float m = fmaxf(m_g[0], m_g[1]);
      float f[2];
#pragma unroll
      for (int i = 0; i < 2; ++i) f[i] = m_g[i] == -INFINITY ? 0.f : exp2f(m_g[i] - m);
      const float l = f[0] * l_g[0] + f[1] * l_g[1];
      const bool two = n > 1;
      const int a = first & 1;                  // the group of the item's first tile
      float fa = f[a], fb = f[a ^ 1];
      const int row = tile * kBlockM + row_in_tile;
      const int batch = bh / p.H, head = bh - batch * p.H;
      const float inv = l > 0.f ? 1.f / (l * (1.f - p.p_drop)) : 0.f;
      fa *= inv;
      fb *= inv;
      done_at = nullptr;
      if (row < p.Sq) {
        done_at = static_cast<T*>(p.O) + ((static_cast<int64_t>(batch) * p.Sq + row) * p.H + head) * p.Dr;
        p.lse[static_cast<int64_t>(bh) * p.Sq + row] =
            l > 0.f ? (m == -INFINITY ? 0.f : m) * 0.6931471805599453f + logf(l) : -INFINITY;
      }
#pragma unroll
      for (int c = 0; c < D / 16; ++c) {
        uint32_t x[16], y[16];
        tc::tmem_ld_x16(tmem_row + kColO + a * D + c * 16, x);
        if (two) tc::tmem_ld_x16(tmem_row + kColO + (a ^ 1) * D + c * 16, y);
        tc::tmem_ld_wait();
        uint32_t(&w)[8] = done[kHold ? c : 0];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          float v[2];
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            v[e] = __uint_as_float(x[2 * i + e]) * fa;
            if (two) v[e] = fmaf(__uint_as_float(y[2 * i + e]), fb, v[e]);
          }
          w[i] = pack16<T>(v[0], v[1]);
        }
        if (!kHold && row < p.Sq) store_cols16(done_at, c * 16, p.Dr, w);
      }
      tc::fence_before_sync();
    }
    if (ok) flush();
  } else {
    tc::regs_inc<kFwdRegsSoftmax>();
    // ------------------------------ softmax groups ------------------------------
    const int quarter = warp & 3;
    const int g = (warp - 4) >> 2;        // takes tiles g, g + 2, ... of the CTA's sequence
    const int row_in_tile = quarter * 32 + lane;
    const uint32_t tmem_row = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
    float* bias_buf = reinterpret_cast<float*>(smem + L::kBias) + (warp - 4) * 2 * kBiasFloats;
    PhiloxUniform rng{};
    if constexpr (kDrop) rng = philox_uniform(p.rng);
    const uint32_t add4 = (128u - p.thr7) * 0x01010101u;
    const int sk16 = (p.Sk + 15) >> 4;
    // scores are brought to the log2 domain before the maximum only where something is added
    // to them (or the scale would turn the maximum around)
    const bool biased = kGeneral && (p.kbias != nullptr || p.rel != nullptr || !(p.scale_log2 > 0.f));
    const float sc = biased ? 1.f : p.scale_log2;
    const uint64_t sc2 = f2_pack(sc, sc);
    auto fetch_bias = [&](int tile, int bh, int jt, int buf) {
      fwd_fetch_bias(p, bias_buf + buf * kBiasFloats, tile, quarter, lane, bh, jt);
    };
    // a tile of the sequence: key tile j of a work item (j < n), u0 is the item's first
    struct Pos {
      int item, tile, bh, n, j, u0;
    };
    // the group's first one from sequence number pos.u0 and work item pos.item on
    auto enter = [&](Pos& pos) {
      while (pos.item < items) {
        pos.n = item_at(pos.item, pos.tile, pos.bh);
        pos.j = (pos.u0 & 1) ^ g;
        if (pos.j < pos.n) return;
        pos.u0 += pos.n;
        pos.item += gridDim.x;
      }
    };
    Pos pos{};
    pos.item = blockIdx.x;
    enter(pos);
    if (biased && pos.item < items) fetch_bias(pos.tile, pos.bh, pos.j, 0);
    bool ok = true;
    uint32_t k = 0, part = 0;       // tiles and items of the group so far
    while (pos.item < items && ok) {
      const int row = pos.tile * kBlockM + row_in_tile;
      const uint64_t drop_row = (static_cast<uint64_t>(pos.bh) * p.Sq + min(row, p.Sq - 1)) * sk16;
      float m_ref = -INFINITY;
      uint64_t l2 = 0;      // two fp32 partial row sums
      Pos next = pos;
      for (; pos.j < pos.n; pos.j += 2, ++k) {
        const uint32_t ph = k & 1;
        const int k0 = pos.j * kBlockN;
        const float* bias = bias_buf + ph * kBiasFloats;
        if (pos.j + 2 >= pos.n) {
          next.u0 += pos.n;
          next.item += gridDim.x;
          enter(next);
        } else {
          next.j = pos.j + 2;
        }
        if (kGeneral && biased) {
          fwd_land_bias(p, bias_buf + ph * kBiasFloats, lane);
          if (next.item < items) fetch_bias(next.tile, next.bh, next.j, ph ^ 1);
        }
        if (!tc::mbar_wait_warp(&s_full[g], ph, abort_flag)) { ok = false; break; }
        tc::fence_after_sync();
        // The tile's scores stay in tensor memory and come out of it twice, 64 for the maximum and 32 for the
        // exponentials at a time.
        const uint32_t tmem_s = tmem_row + kColS + g * 128;
        float m_tile = -INFINITY;
#pragma unroll
        for (int c = 0; c < 128; c += 64) {
          uint32_t raw[2][32];
#pragma unroll
          for (int b = 0; b < 2; ++b) tc::tmem_ld_x32(tmem_s + c + b * 32, raw[b]);
          tc::tmem_ld_wait();
          if constexpr (kGeneral) {
            if (biased) fwd_add_bias(p, raw, bias + c, lane);
            fwd_mask(p, raw, k0 + c, pos.tile * kBlockM + quarter * 32, lane);
#pragma unroll
            for (int b = 0; b < 2; ++b) tc::tmem_st_x32(tmem_s + c + b * 32, raw[b]);
          }
          m_tile = fmaxf(m_tile, fwd_max(raw));
        }
        uint32_t raw[2][32];
        if (kGeneral) tc::tmem_st_wait();
        tc::tmem_ld_x32(tmem_s, raw[0]);
        const float m_new = fmaxf(m_ref, m_tile * sc);
        const float m_use = m_new == -INFINITY ? 0.f : m_new;
        const uint64_t nm2 = f2_pack(-m_use, -m_use);
        const float alpha = m_new == m_ref ? 1.f : exp2f(m_ref - m_new);
        m_ref = m_new;
        s_alpha[(g * 2 + ph) * 128 + row_in_tile] = alpha;
        __syncwarp();
        tc::mbar_arrive_if(&alpha_ready[g * 2 + ph], lane == 0);
        uint64_t la = f2_mul(l2, f2_pack(alpha, alpha)), lb = 0;
        // P of the tile before has been used up
        if (!kOver && k > 0 && !tc::mbar_wait_warp(&pv_done[g], ph ^ 1, abort_flag)) { ok = false; break; }
        if (!kOver) tc::fence_after_sync();
        tc::tmem_ld_wait();
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint32_t(&r)[32] = raw[c & 1];
          if (c < 3) tc::tmem_ld_x32(tmem_s + (c + 1) * 32, raw[(c + 1) & 1]);
          uint32_t pk[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            float a, b;
            f2_unpack(f2_fma(f2_load(r + 2 * i), sc2, nm2), a, b);
            a = exp2f(a);
            b = exp2f(b);
            if (i & 1) lb = f2_add(lb, f2_pack(a, b));
            else la = f2_add(la, f2_pack(a, b));
            pk[i] = pack16<T>(a, b);
          }
          if constexpr (kDrop) {
            // dropped probabilities are cleared in the packed 16-bit pairs
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const uint4 kw = philox_keep16(rng, drop_row + ((k0 + c * 32 + h * 16) >> 4), add4);
              const uint32_t wd[4] = {kw.x, kw.y, kw.z, kw.w};
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                pk[h * 8 + i * 2 + 0] &= keep_mask_pair(wd[i], 0);
                pk[h * 8 + i * 2 + 1] &= keep_mask_pair(wd[i], 1);
              }
            }
          }
          if (c < 3) tc::tmem_ld_wait();
          tc::tmem_st_x16(tmem_row + kColP + g * kPGroup + c * 16, pk);
          if (!kOver && c == 2) {      // (the last scores are in registers)
            tc::fence_before_sync();
            __syncwarp();
            tc::mbar_arrive_if(&s_free[g], lane == 0);
          }
          if (c & 1) {
            tc::tmem_st_wait();
            tc::fence_before_sync();
            __syncwarp();
            tc::mbar_arrive_if(&p_full[g * 2 + (c >> 1)], lane == 0);
          }
        }
        l2 = f2_add(la, lb);
      }
      if (!ok) break;
      float l_run, l_hi;
      f2_unpack(l2, l_run, l_hi);
      s_ml[(g * 2 + (part & 1)) * 128 + row_in_tile] = make_float2(m_ref, l_run + l_hi);
      __syncwarp();
      tc::mbar_arrive_if(&ml_ready[g * 2 + (part & 1)], lane == 0);
      ++part;
      pos = next;
    }
    if (kGeneral) cp_async_wait();      // (a give-up leaves copies under way)
  }

  tc::fence_before_sync();
  __syncthreads();
  if (threadIdx.x == 0 && *abort_flag != 0 && p.status != nullptr) atomicExch(p.status, 2);
  if (warp == 1) {
    tc::fence_after_sync();
    tc::tmem_dealloc(tmem_base, kTmemCols);
  }
}

// Output and log-sum-exp of rows whose keys were split over work items: one warp per row, lanes
// along d (8 per thread for the 16 lanes that D = 128 needs, the other half idle).
template <typename T>
__global__ void __launch_bounds__(128) flash_combine_kernel(
    const float* __restrict__ part_o, const float2* __restrict__ part_ml, T* __restrict__ out,
    float* __restrict__ lse, int splits, int rows, int H, int Sq, int Dr, float keep_prob) {
  const int r = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (r >= rows) return;       // r = (b * H + h) * Sq + i
  float m = -INFINITY;
  for (int s = 0; s < splits; ++s) m = fmaxf(m, part_ml[static_cast<int64_t>(s) * rows + r].x);
  const float m_use = m == -INFINITY ? 0.f : m;
  float l = 0.f, v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  const int d = lane * 8;
  for (int s = 0; s < splits; ++s) {
    const int64_t at = static_cast<int64_t>(s) * rows + r;
    const float2 ml = part_ml[at];
    const float w = exp2f(ml.x - m_use);      // 0 for a split without a visible key
    l += w * ml.y;
    if (d < Dr) {
      float x[8];
      Vec8<float>::load(part_o + at * Dr + d, x);
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] += w * x[k];
    }
  }
  if (d < Dr) {
    const float inv = l > 0.f ? 1.f / (l * keep_prob) : 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] *= inv;
    const int i = r % Sq, bh = r / Sq;
    const int h = bh % H, b = bh / H;
    Vec8<T>::store(out + ((static_cast<int64_t>(b) * Sq + i) * H + h) * Dr + d, v);
  }
  if (lane == 0) lse[r] = l > 0.f ? m_use * 0.6931471805599453f + logf(l) : -INFINITY;
}

// Dropout keep-mask exactly as the attention kernels draw it (testing aid).
__global__ void flash_dropout_mask_kernel(uint8_t* mask, int B, int H, int Sq, int Sk, float p_drop,
                                          PhiloxArgs rng) {
  uint64_t seed, offset;
  philox_unpack(rng, seed, offset);
  const uint32_t add4 = (128u - dropout_thr7(p_drop)) * 0x01010101u;
  const int sk16 = (Sk + 15) >> 4;
  const int64_t total = static_cast<int64_t>(B) * H * Sq * sk16;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < total;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const uint4 kw = philox_keep16(seed, offset, static_cast<uint64_t>(i), add4);
    const uint32_t w[4] = {kw.x, kw.y, kw.z, kw.w};
    const int64_t rowi = i / sk16;
    const int k16 = static_cast<int>(i % sk16) * 16;
    for (int t = 0; t < 16; ++t)
      if (k16 + t < Sk) mask[rowi * Sk + k16 + t] = (w[t >> 2] >> (8 * (t & 3) + 7)) & 1u;
  }
}

void launch_flash_dropout_mask(uint8_t* mask, int B, int H, int Sq, int Sk, float p_drop,
                               PhiloxArgs rng, cudaStream_t stream) {
  count_launch();
  flash_dropout_mask_kernel<<<sm_count() * 4, 256, 0, stream>>>(mask, B, H, Sq, Sk, p_drop, rng);
}

template <int D, bool kGeneral, bool kDrop, typename T>
static int launch_fwd_groups(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv,
                             const FlashFwdParams& p, int64_t items, cudaStream_t stream) {
  constexpr int kSmem = GroupsSmem<D>::kTotal;
  static_assert(kSmem <= 227 * 1024, "flash forward: shared memory over the per-CTA limit");
  auto kernel = flash_fwd_groups_kernel<D, kGeneral, kDrop, T>;
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem) !=
        cudaSuccess)
      return 3;
    configured = true;
  }
  count_launch();
  kernel<<<static_cast<int>(items < sm_count() ? items : sm_count()), 512, kSmem, stream>>>(tq, tk, tv, p);
  return cudaGetLastError() == cudaSuccess ? 0 : 4;
}

// Whether a call without split keys goes to the two softmax groups.  At D = 64 they have one CTA per SM where the other
// kernel has two, so that calls which that one takes in a single wave, and whose few key tiles leave the groups little to
// share, stay with it.  Groups against the other kernel, times as long, by number of work items on 148 SMs
// (heads of 64 and 32, 129 - 2048 queries, all keys / with dropout / causal; 8 x 200 x 100 keys x 16 x 64: 9.9 against 8.5 us):
//   one key tile     up to 296: 0.98 - 1.17 / 0.95 - 1.11 / -    from 300 on: 0.79 - 1.01 / 0.79 - 0.98 / -
//   two              up to 148: 0.92 - 1.02 / 0.83 - 0.90 / 0.94 - 1.00    160 - 296: 0.97 - 1.11 / 0.94 - 1.04 / 1.14 - 1.18
//                    from 300 on: 0.86 - 1.00 / 0.83 - 1.02 / 0.90 - 1.05
//   three            up to 148: 0.94 - 1.04 / 0.83 - 0.91 / 0.95 - 1.02    150 - 296: 0.95 - 1.15 / 0.93 - 1.10 / 0.95 - 1.16
//                    from 300 on: 0.88 - 1.04 / 0.83 - 1.04 / 0.98 - 1.06
//   four and more    150 - 296: 0.90 - 1.14 / 0.84 - 1.06 / 0.80 - 1.04
// (dropout with nothing else, two or three key tiles, 150 - 296 items: 0.93 - 0.99)
template <int D, bool kGeneral, bool kDrop>
static bool fwd_in_groups(const FlashFwdParams& p, int64_t items) {
  if (p.walk.row_tiles == 1) return false;
  if (D != 64 || items > 2 * sm_count()) return true;
  const int key_tiles = (p.Sk + kBlockN - 1) / kBlockN;
  return key_tiles > 3 || (key_tiles > 1 && (items <= sm_count() || (kDrop && !kGeneral)));
}

template <int D, bool kGeneral, bool kDrop, typename T>
static int launch_fwd_d(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv,
                        const FlashFwdParams& p, cudaStream_t stream) {
  constexpr int kSmem = FwdSmem<D>::kTotal;
  static_assert(FwdSmem<D>::kCtas * (kSmem + 1024) <= 228 * 1024, "flash forward: shared memory");
  auto kernel = flash_fwd_kernel<D, kGeneral, kDrop, T>;
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem) !=
        cudaSuccess)
      return 3;
    configured = true;
  }
  const int64_t items = static_cast<int64_t>(p.walk.row_tiles) * p.walk.nbh * p.splits;
  if (fwd_in_groups<D, kGeneral, kDrop>(p, items))
    return launch_fwd_groups<D, kGeneral, kDrop, T>(tq, tk, tv, p, items, stream);
  const int64_t cap = FwdSmem<D>::kCtas * sm_count();
  count_launch();
  kernel<<<static_cast<int>(items < cap ? items : cap), 192, kSmem, stream>>>(tq, tk, tv, p);
  return cudaGetLastError() == cudaSuccess ? 0 : 4;
}

// Work items per row tile.  One row tile per (batch, head) - generation, short queries - and at
// most half as many of them as resident CTAs of flash_fwd_kernel (two per SM for D <= 64, one beyond): the
// keys are split as far as one wave of CTAs takes them.  The combine kernel, 3 us, has to be earned by a
// chain of four tiles less.  Several queries (1.4 - 1.7 us a tile), none -> split: 60 queries x 8 heads of 64: 600 keys 13.0 ->
// 10.3 us, 2000 keys 31 -> 14; 5 queries x 300 keys: 9.6 -> 9.9.  One query (flash_decode_kernel, 0.6 us for 128 keys
// with D <= 64 and 1.1 beyond), heads x keys x D: 12 x 2000 x 64: 13.0 -> 10.2, 12 x 8000 x 64: 40 -> 15, 12 x 1000 x 128:
// 12.7 -> 8.9, 48 x 2000 x 128: 21.9 -> 14.3, 74 x 4000 x 128: 42 -> 30, 48 x 450 x 128: 8.0 -> 8.3.  For one query with
// D <= 64 the line lies too low: seven tiles and one item per SM would be right (12 x 600 x 64: 6.5 -> 7.6, 48 x
// 1000 x 64: 8.5 -> 11.0, 96 x 2000 x 64: 13.0 -> 16.4).
int flash_fwd_splits(int B, int H, int Sq, int Sk, int D) {
  const int tiles = (Sk + kBlockN - 1) / kBlockN;
  const int64_t bh = static_cast<int64_t>(B) * H;
  const int64_t cap = (D <= 64 ? FwdSmem<64>::kCtas : FwdSmem<128>::kCtas) * sm_count();
  if (Sq > kBlockM || bh <= 0) return 1;
  int64_t s = cap / bh;
  if (s > tiles) s = tiles;
  if (s < 2) return 1;
  const int per = static_cast<int>((tiles + s - 1) / s);
  if (tiles - per < 4) return 1;
  return (tiles + per - 1) / per;     // no empty split
}

// `scratch`: flash_fwd_splits() * B * H * Sq * (D + 2) floats, or null with a single split
int launch_flash_fwd(const void* q, const void* k, const void* v, void* o, float* lse,
                     float* scratch,
                     const float* kbias, const float* rel, int B, int H, int Sq, int Sk, int D,
                     const int64_t* q_strides, const int64_t* k_strides, const int64_t* v_strides,
                     float scale, int causal, float p_drop, PhiloxArgs rng, bool bf16, int* status,
                     cudaStream_t stream) {
  // any head dimension up to 128 that is a multiple of 8 (16-byte rows for TMA): the kernels
  // work on 64- or 128-wide tiles whose columns beyond D are zero-filled by the tile loads
  if (D < 8 || D > 128 || D % 8 != 0) return 1;
  if (B <= 0 || H <= 0 || Sq <= 0 || Sk <= 0) return 1;     // (no tensor map without an address)
  FlashFwdParams p;
  p.B = B; p.H = H; p.Sq = Sq; p.Sk = Sk; p.Dr = D; p.O = o; p.lse = lse; p.kbias = kbias; p.rel = rel;
  p.k_steps = (D + 15) / 16;
  p.walk.set((Sq + kBlockM - 1) / kBlockM, 0, B * H, causal ? 2 : 0);
  p.splits = scratch != nullptr ? flash_fwd_splits(B, H, Sq, Sk, D) : 1;
  const int key_tiles = (Sk + kBlockN - 1) / kBlockN;
  p.tiles_per_split = (key_tiles + p.splits - 1) / p.splits;
  const int64_t rows = static_cast<int64_t>(B) * H * Sq;
  p.part_o = scratch;
  p.part_ml = reinterpret_cast<float2*>(scratch + (p.splits > 1 ? p.splits * rows * D : 0));
  p.scale_log2 = scale * kLog2e; p.causal = causal; p.rng = rng;
  // the dropout probability is quantised to a multiple of 1/128 (see philox_keep16)
  p.thr7 = dropout_thr7(p_drop);
  p.p_drop = p.thr7 / 128.f;
  p.status = status;
  p.idesc_qk = tc::instr_desc_f16(128, 128, bf16 ? 1 : 0, false, false);
  // only the columns that exist (a multiple of 16) take part in P V
  p.idesc_pv = tc::instr_desc_f16(128, p.k_steps * 16, bf16 ? 1 : 0, false, true);
  const bool general = kbias != nullptr || rel != nullptr || causal || Sk % kBlockN != 0 || !(scale > 0.f);
  int rc;
  if (Sq == 1 && p.thr7 == 0 && rel == nullptr) {
    // a single query sees all keys, causal or not; its kernel needs no tensor maps
    rc = launch_flash_decode(q, k, v, o, lse, p.part_o, p.part_ml, kbias, B, H, Sk, D, q_strides, k_strides,
                             v_strides, scale, p.splits, p.tiles_per_split * kBlockN, bf16, stream);
  } else {
    CUtensorMap tq, tk, tv;
    if (!make_tmap_bshd(&tq, q, B, Sq, H, D, q_strides[0], q_strides[1], q_strides[2], 128, bf16) ||
        !make_tmap_bshd(&tk, k, B, Sk, H, D, k_strides[0], k_strides[1], k_strides[2], 128, bf16) ||
        !make_tmap_bshd(&tv, v, B, Sk, H, D, v_strides[0], v_strides[1], v_strides[2], 128, bf16))
      return 2;
#define FLASH_FWD_CASE(D_, T_)                                            \
  rc = p.thr7 != 0 ? (general ? launch_fwd_d<D_, true, true, T_>(tq, tk, tv, p, stream)          \
                              : launch_fwd_d<D_, false, true, T_>(tq, tk, tv, p, stream))        \
                   : (general ? launch_fwd_d<D_, true, false, T_>(tq, tk, tv, p, stream)         \
                              : launch_fwd_d<D_, false, false, T_>(tq, tk, tv, p, stream))
    if (D <= 64) {
      if (bf16) FLASH_FWD_CASE(64, __nv_bfloat16);
      else FLASH_FWD_CASE(64, __half);
    } else {
      if (bf16) FLASH_FWD_CASE(128, __nv_bfloat16);
      else FLASH_FWD_CASE(128, __half);
    }
#undef FLASH_FWD_CASE
  }
  if (rc != 0 || p.splits == 1) return rc;
  count_launch();
  const unsigned blocks = static_cast<unsigned>((rows + 3) / 4);
  if (bf16)
    flash_combine_kernel<__nv_bfloat16><<<blocks, 128, 0, stream>>>(
        p.part_o, p.part_ml, static_cast<__nv_bfloat16*>(o), lse, p.splits, static_cast<int>(rows),
        H, Sq, D, 1.f - p.p_drop);
  else
    flash_combine_kernel<__half><<<blocks, 128, 0, stream>>>(
        p.part_o, p.part_ml, static_cast<__half*>(o), lse, p.splits, static_cast<int>(rows), H, Sq,
        D, 1.f - p.p_drop);
  return cudaGetLastError() == cudaSuccess ? 0 : 4;
}

}  // namespace slapo
