// Flash attention backward on tcgen05 / TMEM (sm_100a).
//
// Two passes of one kernel: a work item keeps a 128-row tile of two tensors (X1, X2) in shared
// memory, streams half tiles (64 rows) of two others (Y1, Y2) and accumulates in tensor memory -
// nothing is added up between work items.
//
//   pass      rows      X1  X2   streams   Y1  Y2     accumulators
//   dQ        queries   Q   dO   keys      K   V      dQ += dS K
//   dK / dV   keys      K   V    queries   Q   dO     dK += dS^T Q     dV += P^T dO
//
// Per half tile, with rows on the TMEM lanes:
//   tensor core   S = X1 Y1^T ,  dP = X2 Y2^T                       (fp32 in TMEM)
//   8 warps       p = exp2(s - lse) ;  ds = p * (dp - delta)        (half a row per thread; dropout
//                 replayed), P and dS written back to TMEM as 16 bit
//   tensor core   accumulators += dS Y1 , P Y2                      (A operand from TMEM)
// P and dS never pass through shared memory, and no transpose is needed: the two passes form
// S with its rows where they want them.
//
// Two groups of eight softmax warps take the half tiles in turn, each with its own barriers, so that one
// group's exponentials run under the other's waits, loads and conversions; two threads share a row, which
// needs no exchange here and halves what stands between two products.  Loads and products have threads of
// their own, which go through the sequence at their own pace, and four more warps read finished
// accumulators out under the next work item.  CTAs are persistent.  The
// passes run side by side in one launch where that fills the GPU better (both_q_ctas); the keys of few
// queries are split over work items.
//
// What that is for, measured by clocks in the kernel: one thread that issued all products under
// `lane == 0` took 400 - 700 cycles for the four to eight of each kind (under elect.sync half of
// that, their operands in uniform registers) and was what a tile of 128 waited for, with both halves
// of its columns in the same phase.  Bound now for D = 64: the chain of a half tile within its group, 2000 -
// 2700 cycles (waits, reads of tensor memory and hand-overs of 100 - 400 each next to 512 of exp2); for D = 128
// the products (48 - 64 cycles each, 20 or 24 to a half tile: the first operand's 4 KB from shared memory are as
// many for 64 columns as for 128).
// Measured (all kernels of the backward; whole tiles, one issuing thread -> half tiles, a thread for each kind of
// product): 32 x 512 x 16 heads of 64, p 0.1: 315 -> 262 us; 4 x 2048 x 16 x 128 causal: 400 -> 310; 4 x 1000 x 32 x 80
// causal with key bias: 227 -> 183; 8 x 512 x 16 x 64 with T5's bias, key bias and p 0.1: 155 -> 142; 4 x 2048 x 16 x 128:
// 553 -> 421.
//
// A single pass (5 products per tile instead of 7) has to add up dQ over the key tiles: one fp32
// partial of dQ per key tile written and read again was most of its time (BERT-large, 32 x 512
// tokens x 16 heads of 64: 268 MB each way).
//
// On top of that (us): dropout as a template parameter (its draws were branches over code that has to be
// fetched): dQ 117 -> 112, dK / dV 130 -> 123 for 32 x 512 x 16 x 64, p 0.1, dQ 82 -> 72 without; two sets of dK / dV
// accumulators at D = 64 and dV's read out a step before dK's, rows stored 32 bytes at a time (a store takes a
// cycle per row, and reads of shared memory queue behind it): dK / dV 123 -> 113 and, without dropout, 118 -> 101;
// 4 x 2048 x 16 x 128 causal 161 -> 140; 16 x 200 x 16 x 128, both passes: 85 -> 64.
//
// Two threads a row instead of one, and the next S / dP of the dK / dV pass queued by the thread that issues the
// product which uses up what stands in its place (us, dQ and dK / dV): 32 x 512 x 16 x 64, p 0.1: 110 -> 101 and 113 ->
// 106, without dropout 71 -> 63 and 101 -> 89; 8 x 512 x 16 x 64 with T5's bias and p 0.1: 52 -> 47 and 80 -> 65; 4 x 2048 x
// 16 x 64 causal: 98 -> 88 and 113 -> 110; 4 x 2048 x 16 x 128: 161 -> 156 and 230 -> 214.  (Two threads a row without the
// queue, causal: dK / dV 113 -> 117; the queue in the dQ pass too: dQ 63 -> 66; S and dP by one text with the operands in
// variables: dK / dV 89 -> 93.)
//
// With dropout the dQ pass draws the keep decisions (16 keys of a query row per Philox call, as
// in the forward) and leaves them as one bit each, [B H][key / 32][query] words, for the dK / dV
// pass, whose lanes are keys; side by side with the other, that pass draws them for itself.
#include "flash_common.cuh"
#include "kernels.h"

namespace slapo {

struct FlashBwdParams {
  int Sq, Sk, H;
  int Dr;                 // the tensors' head dimension (<= the tile width D, % 8 == 0)
  int k_steps;            // ceil(Dr / 16)
  int Rq, Rk;             // Sq and Sk rounded up to 128
  TileWalk walk;
  int splits;             // dQ pass: work items per row tile, each takes tiles_per_split key tiles
  int tiles_per_split;
  float* part;            // splits > 1: [splits][B Sq H][Dr] fp32 shares of dQ
  int64_t part_rows;      // B Sq H
  const float* nlse;      // [B H][Rq]  -log2(e) * lse ; -inf for rows without any key (and padding)
  const float* ndelta;    // [B H][Rq]  -rowsum(dO O) * keep probability ; 0 in the padding
  const float* kb2;       // [B][Rk] log2(e) * key bias, 0 in the padding, or nullptr
  uint32_t* keep;         // [B H of this launch][Rk / 32][Rq] keep bits (dropout in two launches)
  const float* rel;       // [H, Sq + Sk - 1] or nullptr
  float* drel;            // same shape fp32 accumulator or nullptr
  void* out1;             // dQ or dK: rows (b, s, head) spaced row_stride elements apart
  void* out2;             // dV
  int64_t row_stride1, row_stride2;
  float scale, scale_log2, inv_keep;
  int causal;
  uint32_t thr7;          // dropout: keep a draw >= thr7 of 128 ; 0 = no dropout
  PhiloxArgs rng;
  uint32_t idesc_s, idesc_acc;
  int* status;
};

// s + a.x b.x + a.y b.y of two 16-bit pairs
template <typename T> __device__ __forceinline__ float dot_pair(uint32_t a, uint32_t b, float s);
template <> __device__ __forceinline__ float dot_pair<__nv_bfloat16>(uint32_t a, uint32_t b, float s) {
  s = fmaf(__uint_as_float(a << 16), __uint_as_float(b << 16), s);
  return fmaf(__uint_as_float(a & 0xffff0000u), __uint_as_float(b & 0xffff0000u), s);
}
template <> __device__ __forceinline__ float dot_pair<__half>(uint32_t a, uint32_t b, float s) {
  const float2 x = __half22float2(*reinterpret_cast<const __half2*>(&a));
  const float2 y = __half22float2(*reinterpret_cast<const __half2*>(&b));
  return fmaf(x.y, y.y, fmaf(x.x, y.x, s));
}

// Row statistics in the layout the kernels read, one launch:
//   nlse   [B H][Rq]  -log2(e) * lse
//   ndelta [B H][Rq]  -keep_prob * sum_d dO[b, i, h, d] * O[b, i, h, d]
// dO and O are contiguous [B, Sq, H, Dr].  A block takes 32 query rows of one batch entry and
// 8 heads: lanes along d while reading (16-byte loads), then the sums pass through shared
// memory so that the stores run along the rows.  The blocks of the first heads also write
//   kb2    [B][Rk]    log2(e) * key bias, 0 in the padding
template <typename T>
__global__ void __launch_bounds__(256) flash_bwd_stats_kernel(
    const T* __restrict__ dout, const T* __restrict__ out, const float* __restrict__ lse,
    float* __restrict__ nlse, float* __restrict__ ndelta, const float* __restrict__ kbias,
    float* __restrict__ kb2, int H, int Sq, int Rq, int Sk, int Rk, int Dr, int lanes,
    float keep_prob) {
  __shared__ float sums[8][33];
  pdl_launch();
  const int i0 = blockIdx.x * 32, h0 = blockIdx.y * 8, b = blockIdx.z;
  if (kbias != nullptr && blockIdx.y == 0)
    for (int key = blockIdx.x * 256 + threadIdx.x; key < Rk; key += gridDim.x * 256)
      kb2[static_cast<int64_t>(b) * Rk + key] =
          key < Sk ? kbias[static_cast<int64_t>(b) * Sk + key] * kLog2e : 0.f;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // `lanes` (8 or 16) threads share a row of Dr; a warp's rows four at a time, all of their loads first (one at
  // a time the kernel ran at half of the memory's rate: 4 x 2048 x 16 x 128: 18.5 -> 13.3 us, 4 x 1000 x 32 x 80: 17 -> 12)
  const int rows_per_warp = 32 / lanes;
  const int d = (lane % lanes) * 8;
  constexpr int kAhead = 4;                    // (256 rows are 8 or 16 rounds)
  for (int r0 = warp * rows_per_warp + lane / lanes; r0 < 256; r0 += kAhead * 8 * rows_per_warp) {
    uint4 x[kAhead], y[kAhead];
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      const int r = r0 + u * 8 * rows_per_warp, i = i0 + (r >> 3), h = h0 + (r & 7);    // neighbouring heads are contiguous
      x[u] = y[u] = make_uint4(0u, 0u, 0u, 0u);
      if (i < Sq && h < H && d < Dr) {
        const int64_t at = ((static_cast<int64_t>(b) * Sq + i) * H + h) * Dr + d;
        x[u] = __ldg(reinterpret_cast<const uint4*>(dout + at));
        y[u] = __ldg(reinterpret_cast<const uint4*>(out + at));
      }
    }
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      float s = dot_pair<T>(x[u].x, y[u].x, 0.f);
      s = dot_pair<T>(x[u].y, y[u].y, s);
      s = dot_pair<T>(x[u].z, y[u].z, s);
      s = dot_pair<T>(x[u].w, y[u].w, s);
      for (int o = lanes >> 1; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      const int r = r0 + u * 8 * rows_per_warp;
      if (lane % lanes == 0) sums[r & 7][r >> 3] = s;
    }
  }
  __syncthreads();
  const int h = h0 + warp, i = i0 + lane;
  if (h < H && i < Rq) {
    const int64_t bh = static_cast<int64_t>(b) * H + h;
    float nl = -INFINITY;
    if (i < Sq) {
      const float l = lse[bh * Sq + i];
      nl = l == -INFINITY ? -INFINITY : -l * kLog2e;
    }
    nlse[bh * Rq + i] = nl;
    ndelta[bh * Rq + i] = i < Sq ? -sums[warp][lane] * keep_prob : 0.f;
  }
}

// Registers per thread of the warpgroups: issuing, softmax (four), reading out; together the 80 per thread
// that 768 threads are launched with.
constexpr int kBwdThreads = 768, kRegsLaunch = 80, kRegsSoftmax = 96;
template <bool kDrop>
struct BwdRegs {
  static constexpr int kIssue = kDrop ? 48 : 56, kOut = kDrop ? 48 : 40;
  static_assert(kIssue + 4 * kRegsSoftmax + kOut <= 6 * kRegsLaunch, "more registers than the block has");
};

template <int D, bool kKeys>
struct BwdSmem {
  static constexpr int kTile = 128 * D * 2;          // X1, X2
  static constexpr int kHalfTile = 64 * D * 2;       // Y1, Y2
  static constexpr int kX = D == 64 ? 2 : 1;         // X tiles: this item's (and the next one's)
  // Y1 is held from S to the accumulating product a step later, Y2 is not
  static constexpr int kY1 = D == 64 ? 6 : 5, kY2 = 4;
  // with each Y1 its column vectors: nlse, ndelta (256 B each) and four rows of keep bits (1 KB)
  // for the dK / dV pass, the key bias (256 B) for the dQ pass
  static constexpr int kVec = kKeys ? 512 + 1024 : 256;
  static constexpr int kX2 = kX * kTile;
  static constexpr int kY1At = 2 * kX * kTile;
  static constexpr int kY2At = kY1At + kY1 * kHalfTile;
  static constexpr int kVecs = kY2At + kY2 * kHalfTile;
  static constexpr int kDrel = kVecs + kY1 * kVec;           // [16 warps][32] floats
  // per softmax warp, twice: the relative bias of the 32 + 32 - 1 distances of its rows and columns
  static constexpr int kRelFloats = 64;
  static constexpr int kRel = kDrel + (kKeys ? 16 * 32 * 4 : 0);
  static constexpr int kBars = kRel + 16 * 2 * kRelFloats * 4;
  static constexpr int kTotal = kBars + 52 * 8 + 1024;
};

// 24 warps in six warpgroups: a thread each of warps 0 - 3 for the loads and the products; two softmax
// groups (warps 4 - 11 and 12 - 19), a row and half of a half tile's columns per thread, which take the half
// tiles in turn; and the warps that read the accumulators out (20 - 23).
// kKeys: the dK / dV pass.  kGeneral: key bias, relative bias, causal mask or ragged lengths.
// kDrop: with dropout.  kDraw: the dK / dV pass then draws the keep decisions itself, and the dQ pass leaves none.
// CTA `cta` of `ctas` that run the pass.
template <int D, bool kKeys, bool kGeneral, bool kDrop, bool kDraw, typename T>
__device__ __forceinline__ void bwd_pass(const CUtensorMap& tm_x1, const CUtensorMap& tm_x2,
                                         const CUtensorMap& tm_y1, const CUtensorMap& tm_y2,
                                         const FlashBwdParams& p, const int cta, const int ctas) {
  using L = BwdSmem<D, kKeys>;
  constexpr int kTileBytes = L::kTile, kHalfBytes = L::kHalfTile;
  constexpr int kBlkX = 128 * 128, kBlkY = 64 * 128;     // [rows x 64 columns], swizzled
  constexpr int kDBlocks = D / 64;
  constexpr int kX = L::kX, kY1 = L::kY1, kY2 = L::kY2;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint8_t* s_vec = smem + L::kVecs;       // [Y1 slot][kVec]
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::kBars);
  uint64_t* x1_full = bars;           // kX each (<= 2)
  uint64_t* x1_empty = bars + 2;
  uint64_t* x2_full = bars + 4;
  uint64_t* x2_empty = bars + 6;
  uint64_t* y1_full = bars + 8;       // kY1 (<= 6)
  uint64_t* y1_empty = bars + 14;
  uint64_t* y2_full = bars + 20;      // kY2 (4)
  uint64_t* y2_empty = bars + 24;
  uint64_t* s_full = bars + 28;       // one per softmax group from here on
  uint64_t* p_ready = bars + 30;      // 8 warps: S has been read (and P written)
  uint64_t* dp_full = bars + 32;
  uint64_t* a1_done = bars + 36;      // dQ pass: dS of a half tile has been used up
  uint64_t* ds_ready = bars + 34;     // 8 warps: dS written
  uint64_t* acc1_full = bars + 40;    // kAcc (<= 2) each
  uint64_t* acc1_free = bars + 42;    // 4 warps
  uint64_t* acc2_full = bars + 44;
  uint64_t* acc2_free = bars + 46;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 48);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int diag = p.Sk - p.Sq;
  constexpr uint32_t kTmemCols = 512;
  // S and dP of the two groups' half tiles, 64 columns each.  P is written over S, dS over dP, whose next
  // products wait for the ones that use them up.  Accumulators: two sets where they fit, so that an item's are
  // read out under the next one's products.  (dK / dV at D = 64 had one set and P in columns of its own, so that the next
  // S did not wait: a third of an item of eight half tiles went by between two items.)
  constexpr uint32_t kColS = 0, kColDP = 128, kColA1 = 256, kColA2 = 256 + D, kColP = kColS;
  constexpr uint32_t kAccCols = kKeys ? 2 * D : D;        // from one set to the next
  constexpr int kAcc = kKeys && D == 128 ? 1 : 2;
  const int items = p.walk.items() * (kKeys ? 1 : p.splits);
  constexpr bool drop = kDrop;

  // row tile and (batch, head) of a work item, its first streamed half tile and how many (at least
  // one: a row tile or a split that nothing reaches still has its zeros written)
  auto item_at = [&](int item, int& tile, int& bhl, int& first) {
    const int unit = kKeys || p.splits == 1 ? item : item / p.splits;
    p.walk.at(unit, tile, bhl);
    int n;
    first = 0;
    if constexpr (kKeys) {
      n = (p.Sq + 63) >> 6;
      if (p.causal) first = min(max(0, tile * 128 - diag) >> 6, n - 1);
      n -= first;
    } else {
      n = (p.Sk + 63) >> 6;
      if (p.causal) n = min(n, (min(tile * 128 + 128, p.Sq) + diag + 63) >> 6);
      if (p.splits > 1) {
        first = (item - unit * p.splits) * p.tiles_per_split * 2;
        n = min(p.tiles_per_split * 2, n - first);
      }
      n = max(1, n);
    }
    return n;
  };

  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) {
      tc::mbar_init(&x1_full[i], 1);
      tc::mbar_init(&x1_empty[i], 1);
      tc::mbar_init(&x2_full[i], 1);
      tc::mbar_init(&x2_empty[i], 1);
      tc::mbar_init(&s_full[i], 1);
      tc::mbar_init(&p_ready[i], 8);
      tc::mbar_init(&dp_full[i], 1);
      tc::mbar_init(&a1_done[i], 1);
      tc::mbar_init(&ds_ready[i], 8);
    }
    for (int i = 0; i < kY1; ++i) {
      tc::mbar_init(&y1_full[i], 1);
      tc::mbar_init(&y1_empty[i], 1);
    }
    for (int i = 0; i < kY2; ++i) {
      tc::mbar_init(&y2_full[i], 1);
      tc::mbar_init(&y2_empty[i], kKeys ? 2 : 1);      // dP and, of two threads, dV's product
    }
    for (int i = 0; i < kAcc; ++i) {
      tc::mbar_init(&acc1_full[i], 1);
      tc::mbar_init(&acc1_free[i], 4);
      tc::mbar_init(&acc2_full[i], 1);
      tc::mbar_init(&acc2_free[i], 4);
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
  // what the kernels before this one wrote is read from here on
  pdl_wait();
  pdl_launch();

  if (warp < 4) {
    tc::regs_dec<BwdRegs<kDrop>::kIssue>();
    if (tc::elect_one()) {
      // Threads that go through the half tiles at their own pace: loads, S, dP and the accumulating products.
      // One thread for all products was what a half tile waited for: issuing takes it 40 - 50 cycles a product or
      // commit and 80 a wait.
      constexpr uint32_t kDescHi = tc::smem_desc_hi(1024);
      constexpr uint32_t kXStep = kTileBytes >> 4, kYStep = kHalfBytes >> 4;
      // S / dP of a half tile (64 streamed rows); x, y: low descriptor words
      auto scores = [&](uint32_t col, uint32_t x, uint32_t y) {
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
          if (kk < p.k_steps)
            tc::umma_f16(tmem_base + col,
                         tc::smem_desc_words(x + (((kk >> 2) * kBlkX + (kk & 3) * 32) >> 4), kDescHi),
                         tc::smem_desc_words(y + (((kk >> 2) * kBlkY + (kk & 3) * 32) >> 4), kDescHi),
                         p.idesc_s, kk != 0 ? 1u : 0u);
        }
      };
      // accumulator += [128 rows x 64 streamed] 16-bit tile in TMEM times Y
      auto accumulate = [&](uint32_t col, uint32_t a_col, uint32_t y, bool fresh) {
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
          tc::umma_f16_ts(tmem_base + col, tmem_base + a_col + (kk >> 1) * 32 + (kk & 1) * 8,
                          tc::smem_desc_words(y + ((kk * 2048) >> 4), kDescHi), p.idesc_acc,
                          (fresh && kk == 0) ? 0u : 1u);
      };
      // where a thread of the dK / dV pass is with S / dP: half tile j of n of a work item
      struct Lead {
        int item, n, j;
      };
      auto lead_enter = [&](Lead& l) {
        int tile, bhl, first;
        l.j = 0;
        if (l.item < items) l.n = item_at(l.item, tile, bhl, first);
      };
      bool ok = true;
      if (warp == 0) {
        // ------------------------------ loads ------------------------------
        tc::tma_prefetch_desc(&tm_x1);
        tc::tma_prefetch_desc(&tm_x2);
        tc::tma_prefetch_desc(&tm_y1);
        tc::tma_prefetch_desc(&tm_y2);
        const bool load_keep = kKeys && !kDraw && drop;
        const uint32_t vec_bytes = kKeys ? 512u + (load_keep ? 1024u : 0u) : (p.kb2 != nullptr ? 256u : 0u);
        Ring<kX> x;
        Ring<kY1> r1;
        Ring<kY2> r2;
        for (int item = cta; item < items && ok; item += ctas, x.step()) {
          int tile, bhl, first;
          const int n = item_at(item, tile, bhl, first);
          const int bh = p.walk.bh0 + bhl;
          const int batch = bh / p.H, head = bh - batch * p.H;
          auto load_x = [&](const CUtensorMap* tm, uint64_t* full, uint64_t* empty, int at) -> bool {
            if (!tc::mbar_wait(&empty[x.slot], x.phase ^ 1, abort_flag)) return false;
            tc::mbar_arrive_expect_tx(&full[x.slot], kTileBytes);
#pragma unroll
            for (int d = 0; d < kDBlocks; ++d)
#pragma unroll
              for (int r = 0; r < 2; ++r)
                tc::tma_load_4d(smem + at + x.slot * kTileBytes + d * kBlkX + r * kBlkY, tm, &full[x.slot],
                                d * 64, head, tile * 128 + r * 64, batch);
            return true;
          };
          ok = false;
          if (!load_x(&tm_x1, x1_full, x1_empty, 0)) break;
          for (int j = 0; j < n; ++j, r1.step(), r2.step()) {
            ok = false;
            const int s0 = (first + j) * 64;
            // (the slot's column vectors were read before ds_ready, which y1_empty follows)
            if (!tc::mbar_wait(&y1_empty[r1.slot], r1.phase ^ 1, abort_flag)) break;
            uint64_t* full = &y1_full[r1.slot];
            tc::mbar_arrive_expect_tx(full, kHalfBytes + vec_bytes);
#pragma unroll
            for (int d = 0; d < kDBlocks; ++d)
              tc::tma_load_4d(smem + L::kY1At + r1.slot * kHalfBytes + d * kBlkY, &tm_y1, full, d * 64, head,
                              s0, batch);
            uint8_t* v = s_vec + r1.slot * L::kVec;
            if constexpr (kKeys) {
              tc::bulk_load(v, p.nlse + static_cast<int64_t>(bh) * p.Rq + s0, 256, full);
              tc::bulk_load(v + 256, p.ndelta + static_cast<int64_t>(bh) * p.Rq + s0, 256, full);
              if (load_keep)
#pragma unroll
                for (int r = 0; r < 4; ++r)
                  tc::bulk_load(v + 512 + r * 256,
                                p.keep + (static_cast<int64_t>(bhl) * (p.Rk >> 5) + tile * 4 + r) * p.Rq + s0,
                                256, full);
            } else {
              if (vec_bytes != 0)
                tc::bulk_load(v, p.kb2 + static_cast<int64_t>(batch) * p.Rk + s0, 256, full);
            }
            if (j == 0 && !load_x(&tm_x2, x2_full, x2_empty, L::kX2)) break;
            if (!tc::mbar_wait(&y2_empty[r2.slot], r2.phase ^ 1, abort_flag)) break;
            tc::mbar_arrive_expect_tx(&y2_full[r2.slot], kHalfBytes);
#pragma unroll
            for (int d = 0; d < kDBlocks; ++d)
              tc::tma_load_4d(smem + L::kY2At + r2.slot * kHalfBytes + d * kBlkY, &tm_y2, &y2_full[r2.slot],
                              d * 64, head, s0, batch);
            ok = true;
          }
        }
      } else if (!kKeys && warp < 3) {
        // ------------------------------ dQ pass: S (warp 1) and dP (warp 2) ------------------------------
        const bool is_s = warp == 1;
        const uint32_t x_desc = tc::smem_desc_lo(tc::smem_u32(smem + (is_s ? 0 : L::kX2)), 16);
        const uint32_t y_desc = tc::smem_desc_lo(tc::smem_u32(smem + (is_s ? L::kY1At : L::kY2At)), 16);
        const uint32_t col = is_s ? kColS : kColDP;
        uint64_t* x_full = is_s ? x1_full : x2_full;
        uint64_t* x_empty = is_s ? x1_empty : x2_empty;
        uint64_t* y_full = is_s ? y1_full : y2_full;
        uint64_t* out_full = is_s ? s_full : dp_full;
        uint64_t* out_free = is_s ? p_ready : a1_done;      // what stood there has been read (dS: used up)
        const int slots = is_s ? kY1 : kY2;
        Ring<kX> x;
        int slot = 0, h = 0;
        uint32_t phase = 0;
        for (int item = cta; item < items && ok; item += ctas, x.step()) {
          int tile, bhl, first;
          const int n = item_at(item, tile, bhl, first);
          if (!tc::mbar_wait(&x_full[x.slot], x.phase, abort_flag)) break;
          for (int j = 0; j < n; ++j, ++h) {
            const int g = h & 1;
            ok = false;
            if (!tc::mbar_wait(&y_full[slot], phase, abort_flag)) break;
            if (h >= 2 && !tc::mbar_wait(&out_free[g], ((h >> 1) & 1) ^ 1, abort_flag)) break;
            tc::fence_after_sync();
            scores(col + g * 64, x_desc + x.slot * kXStep, y_desc + slot * kYStep);
            tc::umma_commit(&out_full[g]);
            if (!is_s) tc::umma_commit(&y2_empty[slot]);
            if (j + 1 == n) tc::umma_commit(&x_empty[x.slot]);
            if (++slot == slots) { slot = 0; phase ^= 1; }
            ok = true;
          }
        }
      } else if (!kKeys) {
        // ------------------------------ accumulating products ------------------------------
        const uint32_t y1_desc = tc::smem_desc_lo(tc::smem_u32(smem + L::kY1At), kBlkY);
        Ring<kY1> r1;
        Ring<kAcc> acc;
        int h = 0;
        for (int item = cta; item < items && ok; item += ctas, acc.step()) {
          int tile, bhl, first;
          const int n = item_at(item, tile, bhl, first);
          // (what these accumulators held has been read out)
          ok = tc::mbar_wait(&acc1_free[acc.slot], acc.phase ^ 1, abort_flag);
          for (int j = 0; j < n && ok; ++j, ++h, r1.step()) {
            // (Y1 is there: S was formed from it before dS)
            ok = tc::mbar_wait(&ds_ready[h & 1], (h >> 1) & 1, abort_flag);
            if (!ok) break;
            tc::fence_after_sync();
            accumulate(kColA1 + acc.slot * kAccCols, kColDP + (h & 1) * 64, y1_desc + r1.slot * kYStep, j == 0);
            tc::umma_commit(&a1_done[h & 1]);
            tc::umma_commit(&y1_empty[r1.slot]);
          }
          if (ok) tc::umma_commit(&acc1_full[acc.slot]);
        }
      } else if (warp == 1) {
        // ------------------------------ dK / dV pass: S and dV ------------------------------
        // The next S of a group goes into the tensor core's queue behind the product that uses up the P in its
        // place, two half tiles ahead.  That S does not overtake that product's reads is the order in which the tensor core
        // takes one thread's products; PTX promises it for the same accumulator and shape only, and here both
        // differ (N = 64 for S, the head's columns for dV).  Same for dP over dS in the next warp.  Checked by
        // tests/test_flash_order_gpu.py; the dQ pass waits for the product (380 - 650 cycles from commit to wait).
        const uint32_t x_desc = tc::smem_desc_lo(tc::smem_u32(smem), 16);
        const uint32_t y_desc = tc::smem_desc_lo(tc::smem_u32(smem + L::kY1At), 16);
        const uint32_t y2_desc = tc::smem_desc_lo(tc::smem_u32(smem + L::kY2At), kBlkY);
        Ring<kX> x;
        Ring<kY1> r1;
        Ring<kY2> r2;
        Ring<kAcc> acc;
        Lead lead{cta, 0, 0};
        lead_enter(lead);
        auto next_s = [&](int g) -> bool {
          if (lead.item >= items) return true;
          if (lead.j == 0 && !tc::mbar_wait(&x1_full[x.slot], x.phase, abort_flag)) return false;
          if (!tc::mbar_wait(&y1_full[r1.slot], r1.phase, abort_flag)) return false;
          tc::fence_after_sync();
          scores(kColS + g * 64, x_desc + x.slot * kXStep, y_desc + r1.slot * kYStep);
          tc::umma_commit(&s_full[g]);
          r1.step();
          if (++lead.j == lead.n) {
            tc::umma_commit(&x1_empty[x.slot]);
            x.step();
            lead.item += ctas;
            lead_enter(lead);
          }
          return true;
        };
        ok = next_s(0) && next_s(1);
        int h = 0;
        for (int item = cta; item < items && ok; item += ctas, acc.step()) {
          int tile, bhl, first;
          const int n = item_at(item, tile, bhl, first);
          // (what these accumulators held has been read out)
          ok = tc::mbar_wait(&acc2_free[acc.slot], acc.phase ^ 1, abort_flag);
          for (int j = 0; j < n && ok; ++j, ++h) {
            ok = false;
            // (P comes of S and says nothing about Y2, which is loaded after Y1)
            if (!tc::mbar_wait(&y2_full[r2.slot], r2.phase, abort_flag) ||
                !tc::mbar_wait(&p_ready[h & 1], (h >> 1) & 1, abort_flag))
              break;
            tc::fence_after_sync();
            accumulate(kColA2 + acc.slot * kAccCols, kColP + (h & 1) * 64, y2_desc + r2.slot * kYStep, j == 0);
            tc::umma_commit(&y2_empty[r2.slot]);
            if (j + 1 == n) tc::umma_commit(&acc2_full[acc.slot]);
            r2.step();
            ok = next_s(h & 1);
          }
        }
      } else if (warp == 2) {
        // ------------------------------ accumulating products ------------------------------
        // (dK / dV pass: dP and dK, likewise)
        const uint32_t x_desc = tc::smem_desc_lo(tc::smem_u32(smem + L::kX2), 16);
        const uint32_t y_desc = tc::smem_desc_lo(tc::smem_u32(smem + L::kY2At), 16);
        const uint32_t y1_desc = tc::smem_desc_lo(tc::smem_u32(smem + L::kY1At), kBlkY);
        Ring<kX> x;
        Ring<kY1> r1;
        Ring<kY2> r2;
        Ring<kAcc> acc;
        Lead lead{cta, 0, 0};
        lead_enter(lead);
        auto next_dp = [&](int g) -> bool {
          if (lead.item >= items) return true;
          if (lead.j == 0 && !tc::mbar_wait(&x2_full[x.slot], x.phase, abort_flag)) return false;
          if (!tc::mbar_wait(&y2_full[r2.slot], r2.phase, abort_flag)) return false;
          tc::fence_after_sync();
          scores(kColDP + g * 64, x_desc + x.slot * kXStep, y_desc + r2.slot * kYStep);
          tc::umma_commit(&dp_full[g]);
          tc::umma_commit(&y2_empty[r2.slot]);
          r2.step();
          if (++lead.j == lead.n) {
            tc::umma_commit(&x2_empty[x.slot]);
            x.step();
            lead.item += ctas;
            lead_enter(lead);
          }
          return true;
        };
        ok = next_dp(0) && next_dp(1);
        int h = 0;
        for (int item = cta; item < items && ok; item += ctas, acc.step()) {
          int tile, bhl, first;
          const int n = item_at(item, tile, bhl, first);
          ok = tc::mbar_wait(&acc1_free[acc.slot], acc.phase ^ 1, abort_flag);
          for (int j = 0; j < n && ok; ++j, ++h) {
            // (Y1 is there: S was formed from it before dS)
            ok = tc::mbar_wait(&ds_ready[h & 1], (h >> 1) & 1, abort_flag);
            if (!ok) break;
            tc::fence_after_sync();
            accumulate(kColA1 + acc.slot * kAccCols, kColDP + (h & 1) * 64, y1_desc + r1.slot * kYStep, j == 0);
            tc::umma_commit(&y1_empty[r1.slot]);
            if (j + 1 == n) tc::umma_commit(&acc1_full[acc.slot]);
            r1.step();
            ok = next_dp(h & 1);
          }
        }
      }
    }
  } else if (warp >= 20) {
    tc::regs_dec<BwdRegs<kDrop>::kOut>();
    // ------------------------------ accumulators out of tensor memory ------------------------------
    // dS is formed without the factors scale and 1 / keep_prob; they are applied once to dQ and dK
    // (and 1 / keep_prob to dV) here
    const float out_scale = p.scale * p.inv_keep;
    const int r_in = (warp & 3) * 32 + lane;
    const uint32_t tmem_row = tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16);
    // D columns from `col` on, times f, to `dst` (or as they are to `share`)
    auto read_out = [&](uint32_t col, float f, T* dst, float* share, bool row_ok) {
#pragma unroll
      for (int c = 0; c < D; c += 16) {
        uint32_t r[16];
        tc::tmem_ld_x16(tmem_row + col + c, r);
        tc::tmem_ld_wait();
        if (!row_ok) continue;
        if (!kKeys && share != nullptr) {
#pragma unroll
          for (int g = 0; g < 16; g += 4)
            if (c + g < p.Dr)
              *reinterpret_cast<uint4*>(share + c + g) = make_uint4(r[g], r[g + 1], r[g + 2], r[g + 3]);
        } else {
          uint32_t v[8];
#pragma unroll
          for (int i = 0; i < 8; ++i)
            v[i] = pack16<T>(__uint_as_float(r[2 * i]) * f, __uint_as_float(r[2 * i + 1]) * f);
          store_cols16(dst, c, p.Dr, v);
        }
      }
    };
    Ring<kAcc> acc;
    for (int item = cta; item < items; item += ctas, acc.step()) {
      int tile, bhl, first;
      item_at(item, tile, bhl, first);
      const int bh = p.walk.bh0 + bhl;
      const int batch = bh / p.H, head = bh - batch * p.H;
      const int row = tile * 128 + r_in;
      const int rows = kKeys ? p.Sk : p.Sq;
      const int64_t at = (static_cast<int64_t>(batch) * rows + min(row, rows - 1)) * p.H + head;
      float* share = nullptr;
      if (!kKeys && p.splits > 1)
        share = p.part + (static_cast<int64_t>(item % p.splits) * p.part_rows + at) * p.Dr;
      if constexpr (kKeys) {      // (dV's last product is a step before dK's)
        if (!tc::mbar_wait_warp(&acc2_full[acc.slot], acc.phase, abort_flag)) break;
        tc::fence_after_sync();
        read_out(kColA2 + acc.slot * kAccCols, p.inv_keep, static_cast<T*>(p.out2) + at * p.row_stride2, nullptr,
                 row < rows);
        tc::fence_before_sync();
        __syncwarp();
        tc::mbar_arrive_if(&acc2_free[acc.slot], lane == 0);
      }
      if (!tc::mbar_wait_warp(&acc1_full[acc.slot], acc.phase, abort_flag)) break;
      tc::fence_after_sync();
      read_out(kColA1 + acc.slot * kAccCols, out_scale, static_cast<T*>(p.out1) + at * p.row_stride1, share,
               row < rows);
      tc::fence_before_sync();
      __syncwarp();
      tc::mbar_arrive_if(&acc1_free[acc.slot], lane == 0);
    }
  } else {
    tc::regs_inc<kRegsSoftmax>();
    // ------------------------------ softmax groups ------------------------------
    const int quarter = warp & 3;
    const int g = (warp - 4) >> 3;      // takes half tiles g, g + 2, ... of the CTA's sequence
    const int half = ((warp - 4) >> 2) & 1;      // ... and of each 32 columns
    const int r_in = quarter * 32 + lane;
    const uint32_t tmem_row = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + g * 64 + half * 32;
    PhiloxUniform rng{};
    if ((!kKeys || kDraw) && drop) rng = philox_uniform(p.rng);
    const uint32_t add4 = (128u - p.thr7) * 0x01010101u;
    const int sk16 = (p.Sk + 15) >> 4;
    const uint64_t sc2 = f2_pack(p.scale_log2, p.scale_log2);

    // a half tile of the sequence: half tile j of n of a work item, u0 is the item's first
    struct Pos {
      int item, tile, bhl, first, n, j, u0;
    };
    // the group's first one from sequence number pos.u0 and work item pos.item on
    auto enter = [&](Pos& pos) {
      while (pos.item < items) {
        pos.n = item_at(pos.item, pos.tile, pos.bhl, pos.first);
        pos.j = (pos.u0 & 1) ^ g;
        if (pos.j < pos.n) return;
        pos.u0 += pos.n;
        pos.item += ctas;
      }
    };
    // per-row scalars of a work item: the dQ pass's statistics, the dK / dV pass's key bias
    auto row_scalars = [&](const Pos& pos, float& a, float& b) {
      a = 0.f;
      b = 0.f;
      const int bh = p.walk.bh0 + pos.bhl;
      if constexpr (kKeys) {
        if (kGeneral && p.kb2 != nullptr)
          a = p.kb2[static_cast<int64_t>(bh / p.H) * p.Rk + pos.tile * 128 + r_in];
      } else {
        a = p.nlse[static_cast<int64_t>(bh) * p.Rq + pos.tile * 128 + r_in];
        b = p.ndelta[static_cast<int64_t>(bh) * p.Rq + pos.tile * 128 + r_in];
      }
    };

    // Relative bias of this warp's 32 rows and a half tile's 64 columns, on its way into buffer `buf`:
    // copied a half tile ahead, as in the forward.  A column further is a key further in the dQ
    // pass, a query further (a smaller distance) in the other.
    float* rel_buf = reinterpret_cast<float*>(smem + L::kRel) + (warp - 4) * 2 * L::kRelFloats;
    const bool has_rel = kGeneral && p.rel != nullptr;
    auto fetch_rel = [&](const Pos& pos, int buf) {
      const int head = (p.walk.bh0 + pos.bhl) % p.H;
      const float* src = p.rel + static_cast<int64_t>(head) * (p.Sq + p.Sk - 1) + p.Sq - 1;
      const int r0 = pos.tile * 128 + quarter * 32, c0 = (pos.first + pos.j) * 64 + half * 32;
      const int d0 = kKeys ? r0 - (c0 + 31) : c0 - (r0 + 31);
#pragma unroll
      for (int i = lane; i < L::kRelFloats; i += 32)
        cp_async4(rel_buf + buf * L::kRelFloats + i, src + max(1 - p.Sq, min(d0 + i, p.Sk - 1)));
    };

    Pos pos{};
    pos.item = cta;
    enter(pos);
    float row_a = 0.f, row_b = 0.f;
    if (pos.item < items) {
      row_scalars(pos, row_a, row_b);
      if (has_rel) fetch_rel(pos, 0);
    }
    bool ok = true;
    int slot = g;                         // of the Y1 ring
    uint32_t slot_phase = 0, ph = 0;      // ph: parity of the group's count of half tiles
    while (pos.item < items && ok) {
      const int bh = p.walk.bh0 + pos.bhl;
      const int row = pos.tile * 128 + r_in;
      const uint64_t ra2 = f2_pack(row_a, row_a), rb2 = f2_pack(row_b, row_b);
      const uint64_t drop_row = (static_cast<uint64_t>(bh) * p.Sq + min(row, p.Sq - 1)) * sk16;
      Pos next = pos;
      for (; pos.j < pos.n; pos.j += 2) {
        const int col0 = (pos.first + pos.j) * 64 + half * 32;       // this warp's first column
        const uint8_t* vec = s_vec + slot * L::kVec;
        if (pos.j + 2 >= pos.n) {       // the item's last: the next one's rows, under its work
          next.u0 += pos.n;
          next.item += ctas;
          enter(next);
          if (next.item < items) row_scalars(next, row_a, row_b);
        } else {
          next.j = pos.j + 2;
        }
        if (has_rel) {
          cp_async_wait();
          __syncwarp();     // (visible to the warp, and the other buffer's readers are done)
          if (next.item < items) fetch_rel(next, ph ^ 1);
        }
        // ---- dropout decisions of this row and the half tile's keys (dQ pass) ----
        uint32_t keep16[2][4];
        if (!kKeys && drop) {
          uint32_t bits = 0;
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            const uint4 kw = philox_keep16(rng, drop_row + (col0 >> 4) + q, add4);
            keep16[q][0] = kw.x; keep16[q][1] = kw.y; keep16[q][2] = kw.z; keep16[q][3] = kw.w;
            if constexpr (!kDraw) bits |= keep_bits16(kw) << (q * 16);
          }
          if constexpr (!kDraw)
            p.keep[(static_cast<int64_t>(pos.bhl) * (p.Rk >> 5) + (col0 >> 5)) * p.Rq + row] = bits;
        }
        // ---- ... of the warp's 32 keys and 32 queries (dK / dV pass), a query per lane, into the words that
        // the other form loads ----
        if constexpr (kKeys && kDraw) {
          if (drop) {
            uint32_t* words = reinterpret_cast<uint32_t*>(s_vec + slot * L::kVec + 512 + quarter * 256) + half * 32;
            const uint64_t at = (static_cast<uint64_t>(bh) * p.Sq + min(col0 + lane, p.Sq - 1)) * sk16 +
                                ((pos.tile * 128 + quarter * 32) >> 4);
            words[lane] = keep_bits16(philox_keep16(rng, at, add4)) |
                          keep_bits16(philox_keep16(rng, at + 1, add4)) << 16;
            __syncwarp();
          }
        }
        // ---- P ----
        if (!tc::mbar_wait_warp(&s_full[g], ph, abort_flag)) { ok = false; break; }
        // (complete since before s_full; waiting on it makes the column vectors visible)
        if (kKeys || (kGeneral && p.kb2 != nullptr)) {
          if (!tc::mbar_wait_warp(&y1_full[slot], slot_phase, abort_flag)) { ok = false; break; }
        }
        tc::fence_after_sync();
        float pr[32];
        {
          uint32_t s0[32];
          tc::tmem_ld_x32(tmem_row + kColS, s0);
          tc::tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 32; ++i) pr[i] = __uint_as_float(s0[i]);
        }
        if constexpr (!kKeys) {
          tc::fence_before_sync();
          __syncwarp();
          tc::mbar_arrive_if(&p_ready[g], lane == 0);
        }
        const float4* cv = reinterpret_cast<const float4*>(vec) + half * 8;
#pragma unroll
        for (int i = 0; i < 32; i += 4) {
          uint64_t x0 = f2_pack(pr[i], pr[i + 1]), x1 = f2_pack(pr[i + 2], pr[i + 3]);
          if constexpr (kKeys) {
            const float4 c = cv[i >> 2];
            x0 = f2_fma(x0, sc2, f2_pack(c.x, c.y));
            x1 = f2_fma(x1, sc2, f2_pack(c.z, c.w));
            if (kGeneral) {
              x0 = f2_add(x0, ra2);
              x1 = f2_add(x1, ra2);
            }
          } else {
            x0 = f2_fma(x0, sc2, ra2);
            x1 = f2_fma(x1, sc2, ra2);
          }
          f2_unpack(x0, pr[i], pr[i + 1]);
          f2_unpack(x1, pr[i + 2], pr[i + 3]);
        }
        if constexpr (kGeneral) {
          if (!kKeys && p.kb2 != nullptr) {
#pragma unroll
            for (int i = 0; i < 32; i += 4) {
              const float4 c = cv[i >> 2];
              f2_unpack(f2_add(f2_pack(pr[i], pr[i + 1]), f2_pack(c.x, c.y)), pr[i], pr[i + 1]);
              f2_unpack(f2_add(f2_pack(pr[i + 2], pr[i + 3]), f2_pack(c.z, c.w)), pr[i + 2], pr[i + 3]);
            }
          }
          if (has_rel) {
            const float* rel = rel_buf + ph * L::kRelFloats + (kKeys ? lane + 31 : 31 - lane);
            const uint64_t log2e2 = f2_pack(kLog2e, kLog2e);
#pragma unroll
            for (int i = 0; i < 32; i += 2) {
              const uint64_t x = f2_fma(kKeys ? f2_pack(rel[-i], rel[-i - 1]) : f2_pack(rel[i], rel[i + 1]),
                                        log2e2, f2_pack(pr[i], pr[i + 1]));
              f2_unpack(x, pr[i], pr[i + 1]);
            }
          }
          if constexpr (kKeys) {
            // key `row` is seen by queries >= row - diag (queries beyond Sq have nlse = -inf)
            if (p.causal && col0 + diag < pos.tile * 128 + quarter * 32 + 31) {
              const uint32_t hidden = low_bits(row - diag - col0);
#pragma unroll
              for (int i = 0; i < 32; ++i)
                if (hidden & (1u << i)) pr[i] = -INFINITY;
            }
          } else {
            const int first_limit = p.causal ? min(p.Sk, pos.tile * 128 + quarter * 32 + diag + 1) : p.Sk;
            if (col0 + 32 > first_limit) {
              const uint32_t seen = low_bits((p.causal ? min(p.Sk, row + diag + 1) : p.Sk) - col0);
#pragma unroll
              for (int i = 0; i < 32; ++i)
                if (!(seen & (1u << i))) pr[i] = -INFINITY;
            }
          }
        }
        // (kept before the waits that follow: the compiler would move it behind them)
#pragma unroll
        for (int i = 0; i < 32; ++i) pr[i] = exp2_here(pr[i]);
        if constexpr (kKeys) {
          if (drop) {
            // a dropped probability is kept as its negative: it still counts in dS's row term
            const uint4* kw4 = reinterpret_cast<const uint4*>(vec + 512 + quarter * 256) + half * 8;
            const uint32_t lane_bit = 1u << lane;
#pragma unroll
            for (int i = 0; i < 32; i += 4) {
              const uint4 kw = kw4[i >> 2];
              pr[i] = kw.x & lane_bit ? pr[i] : -pr[i];
              pr[i + 1] = kw.y & lane_bit ? pr[i + 1] : -pr[i + 1];
              pr[i + 2] = kw.z & lane_bit ? pr[i + 2] : -pr[i + 2];
              pr[i + 3] = kw.w & lane_bit ? pr[i + 3] : -pr[i + 3];
            }
          }
          uint32_t pk[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) pk[i] = pack16_relu<T>(pr[2 * i], pr[2 * i + 1]);
          tc::tmem_st_x16(tmem_row + kColP, pk);
          tc::tmem_st_wait();
          tc::fence_before_sync();
          __syncwarp();
          tc::mbar_arrive_if(&p_ready[g], lane == 0);
        }
        // ---- dS ----
        if (!tc::mbar_wait_warp(&dp_full[g], ph, abort_flag)) { ok = false; break; }
        tc::fence_after_sync();
        // Sums along the diagonals key - query = const, for the gradient of T5's table: the running sum moves
        // one lane up (next key) with every column (next query), so that it stays on its diagonal;
        // what leaves at lane 31 is collected and added to the result 32 at a time.
        float diagonal = 0.f;
        float* buf = reinterpret_cast<float*>(smem + L::kDrel) + (warp - 4) * 32;
#pragma unroll
        for (int c = 0; c < 32; c += 16) {
          uint32_t d[16];
          tc::tmem_ld_x16(tmem_row + kColDP + c, d);
          tc::tmem_ld_wait();
          if (!kKeys && drop) {
#pragma unroll
            for (int i = 0; i < 16; ++i) d[i] &= keep_mask_full(keep16[c >> 4][i >> 2], i & 3);
          }
          const float4* nd = reinterpret_cast<const float4*>(vec + 256) + half * 8 + (c >> 2);
          const float* v = pr + c;
          float ds[16];
          if (kKeys && drop) {
#pragma unroll
            for (int i = 0; i < 16; i += 4) {
              const float4 dl = nd[i >> 2];
              const float n4[4] = {dl.x, dl.y, dl.z, dl.w};
#pragma unroll
              for (int e = 0; e < 4; ++e)
                ds[i + e] = fmaf(fmaxf(v[i + e], 0.f), __uint_as_float(d[i + e]), fabsf(v[i + e]) * n4[e]);
            }
          } else {
#pragma unroll
            for (int i = 0; i < 16; i += 4) {
              uint64_t x0 = f2_load(d + i), x1 = f2_load(d + i + 2);
              if constexpr (kKeys) {
                const float4 dl = nd[i >> 2];
                x0 = f2_add(x0, f2_pack(dl.x, dl.y));
                x1 = f2_add(x1, f2_pack(dl.z, dl.w));
              } else {
                x0 = f2_add(x0, rb2);
                x1 = f2_add(x1, rb2);
              }
              x0 = f2_mul(x0, f2_pack(v[i], v[i + 1]));
              x1 = f2_mul(x1, f2_pack(v[i + 2], v[i + 3]));
              f2_unpack(x0, ds[i], ds[i + 1]);
              f2_unpack(x1, ds[i + 2], ds[i + 3]);
            }
          }
          if constexpr (kKeys && kGeneral) {
            if (p.drel != nullptr) {
#pragma unroll
              for (int i = 0; i < 16; ++i) {
                // padding: keys beyond Sk have a P (their rows go nowhere else), queries have none
                if (row < p.Sk) diagonal += ds[i];
                diagonal = __shfl_sync(0xffffffffu, diagonal, (lane + 31) & 31);
                if (lane == 0) {
                  buf[c + i] = diagonal;      // diagonal key0 + 31 - (col0 + c + i)
                  diagonal = 0.f;
                }
              }
            }
          }
          uint32_t pk[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) pk[i] = pack16<T>(ds[2 * i], ds[2 * i + 1]);
          tc::tmem_st_x8(tmem_row + kColDP + (c >> 1), pk);
        }
        if constexpr (kKeys && kGeneral) {
          if (p.drel != nullptr) {
            float* out = p.drel + static_cast<int64_t>(bh % p.H) * (p.Sq + p.Sk - 1);
            const int key0 = pos.tile * 128 + quarter * 32, last = p.Sq + p.Sk - 2;
            __syncwarp();
            const int at = key0 + 31 - (col0 + lane) + p.Sq - 1;
            if (at >= 0 && at <= last) atomicAdd(out + at, buf[lane] * p.inv_keep);
            const int rest = key0 + lane - (col0 + 32) + p.Sq - 1;     // still under way in the lanes
            if (lane > 0 && rest >= 0 && rest <= last) atomicAdd(out + rest, diagonal * p.inv_keep);
            __syncwarp();
          }
        }
        tc::tmem_st_wait();
        tc::fence_before_sync();
        __syncwarp();
        tc::mbar_arrive_if(&ds_ready[g], lane == 0);
        ph ^= 1;
        slot += 2;
        if (slot >= kY1) { slot -= kY1; slot_phase ^= 1; }
      }
      pos = next;
    }
    if (has_rel) cp_async_wait();     // (a give-up leaves copies under way)
  }

  tc::fence_before_sync();
  __syncthreads();
  if (threadIdx.x == 0 && *abort_flag != 0 && p.status != nullptr) atomicExch(p.status, 3);
  if (warp == 1) {
    tc::fence_after_sync();
    tc::tmem_dealloc(tmem_base, kTmemCols);
  }
}

// One pass.
template <int D, bool kKeys, bool kGeneral, bool kDrop, typename T>
__global__ void __launch_bounds__(kBwdThreads, 1)
flash_bwd_kernel(const __grid_constant__ CUtensorMap tm_x1, const __grid_constant__ CUtensorMap tm_x2,
                 const __grid_constant__ CUtensorMap tm_y1, const __grid_constant__ CUtensorMap tm_y2,
                 const __grid_constant__ FlashBwdParams p) {
  bwd_pass<D, kKeys, kGeneral, kDrop, false, T>(tm_x1, tm_x2, tm_y1, tm_y2, p, blockIdx.x, gridDim.x);
}

// Both passes side by side, the dQ pass on the first `q_ctas` CTAs.
template <int D, bool kGeneral, bool kDrop, typename T>
__global__ void __launch_bounds__(kBwdThreads, 1)
flash_bwd_both_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                      const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_do,
                      const __grid_constant__ FlashBwdParams pq,
                      const __grid_constant__ FlashBwdParams pk, const int q_ctas) {
  const int cta = blockIdx.x;
  if (cta < q_ctas)
    bwd_pass<D, false, kGeneral, kDrop, true, T>(tm_q, tm_do, tm_k, tm_v, pq, cta, q_ctas);
  else
    bwd_pass<D, true, kGeneral, kDrop, true, T>(tm_k, tm_v, tm_q, tm_do, pk, cta - q_ctas,
                                         gridDim.x - q_ctas);
}

// dQ of rows whose keys were split over work items: the shares added in their order
template <typename T>
__global__ void __launch_bounds__(256) flash_dq_combine_kernel(const float* __restrict__ part,
                                                               T* __restrict__ dq, int splits,
                                                               int64_t n, float scale) {
  const int64_t at = (static_cast<int64_t>(blockIdx.x) * 256 + threadIdx.x) * 8;
  if (at >= n) return;
  float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  for (int s = 0; s < splits; ++s) {
    float x[8];
    Vec8<float>::load(part + s * n + at, x);
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] += x[k];
  }
#pragma unroll
  for (int k = 0; k < 8; ++k) v[k] *= scale;
  Vec8<T>::store(dq + at, v);
}

// A kernel's shared memory, allowed once per kernel
template <typename K>
static bool allow_smem(K kernel, int bytes, bool& configured) {
  if (!configured)
    configured = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) ==
                 cudaSuccess;
  return configured;
}

// `early`: the kernel's prologue may run under the end of the kernel before it (it waits in
// pdl_wait), which saves up to 2 us of a short backward (late -> early: 1 x 512 x 16 x 64: 18.2 -> 17.5 us, 1 x 1024 x 12 x
// 64: 30.7 -> 28.7, 4 x 512 x 16 x 64 in two launches: 40.4 -> 38.8).  CTAs that go round several times are
// slower for it where their items differ or both passes are at work: 4 x 1024 x 12 x 64 causal, side by
// side: 63.9 -> 75.4; 64 x 128 x 12 x 64, p 0.1, side by side: 53.3 -> 66.7; 32 x 512 x 16 x 64 causal, one after the
// other: 172.8 -> 178.1 (without a mask 203.3 -> 200.7).
template <typename... P, typename... A>
static int launch_bwd(void (*kernel)(P...), int ctas, int smem, bool early, cudaStream_t stream,
                      const A&... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(ctas);
  cfg.blockDim = dim3(kBwdThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = early ? 1 : 0;
  count_launch();
  if (cudaLaunchKernelEx(&cfg, kernel, args...) == cudaSuccess) return 0;
  (void)cudaGetLastError();
  return 4;
}

template <int D, bool kKeys, bool kGeneral, bool kDrop, typename T>
static int launch_pass(const CUtensorMap& x1, const CUtensorMap& x2, const CUtensorMap& y1,
                       const CUtensorMap& y2, const FlashBwdParams& p, cudaStream_t stream) {
  constexpr int kSmem = BwdSmem<D, kKeys>::kTotal;
  static_assert(kSmem <= 227 * 1024, "flash backward: shared memory over the per-CTA limit");
  auto kernel = flash_bwd_kernel<D, kKeys, kGeneral, kDrop, T>;
  static bool configured = false;
  if (!allow_smem(kernel, kSmem, configured)) return 3;
  const int64_t items = static_cast<int64_t>(p.walk.row_tiles) * p.walk.nbh * p.splits;
  const int64_t cap = sm_count();
  return launch_bwd(kernel, static_cast<int>(items < cap ? items : cap), kSmem, items <= 3 * cap, stream,
                    x1, x2, y1, y2, p);
}

// The passes of `pq` (dQ) and `pk` (dK / dV), side by side or one after the other
template <int D, bool kGeneral, bool kDrop, typename T>
static int launch_passes(const CUtensorMap& q, const CUtensorMap& k, const CUtensorMap& v,
                         const CUtensorMap& dout, const FlashBwdParams& pq, const FlashBwdParams& pk,
                         int q_ctas, cudaStream_t stream) {
  if (q_ctas == 0) {
    // dQ first: with dropout it leaves the keep bits that the dK / dV pass reads
    const int rc = launch_pass<D, false, kGeneral, kDrop, T>(q, dout, k, v, pq, stream);
    return rc != 0 ? rc : launch_pass<D, true, kGeneral, kDrop, T>(k, v, q, dout, pk, stream);
  }
  constexpr int kSmemQ = BwdSmem<D, false>::kTotal, kSmemK = BwdSmem<D, true>::kTotal;
  constexpr int kSmem = kSmemQ > kSmemK ? kSmemQ : kSmemK;
  auto kernel = flash_bwd_both_kernel<D, kGeneral, kDrop, T>;
  static bool configured = false;
  if (!allow_smem(kernel, kSmem, configured)) return 3;
  const int64_t items = static_cast<int64_t>(pk.walk.row_tiles) * pk.walk.nbh;
  const int64_t k_cap = sm_count() - q_ctas;
  const int64_t q_items = static_cast<int64_t>(pq.walk.row_tiles) * pq.walk.nbh * pq.splits;
  const bool early = q_items + items <= 2 * sm_count();
  return launch_bwd(kernel, q_ctas + static_cast<int>(items < k_cap ? items : k_cap), kSmem, early, stream,
                    q, k, v, dout, pq, pk, q_ctas);
}

template <bool kDrop, typename T>
static int launch_typed(const CUtensorMap& q, const CUtensorMap& k, const CUtensorMap& v,
                        const CUtensorMap& dout, const FlashBwdParams& pq, const FlashBwdParams& pk,
                        int q_ctas, bool general, cudaStream_t stream) {
  if (pq.Dr <= 64)
    return general ? launch_passes<64, true, kDrop, T>(q, k, v, dout, pq, pk, q_ctas, stream)
                   : launch_passes<64, false, kDrop, T>(q, k, v, dout, pq, pk, q_ctas, stream);
  return general ? launch_passes<128, true, kDrop, T>(q, k, v, dout, pq, pk, q_ctas, stream)
                 : launch_passes<128, false, kDrop, T>(q, k, v, dout, pq, pk, q_ctas, stream);
}

static int round128(int n) { return (n + 127) / 128 * 128; }

// One launch or two, and how many CTAs of one launch take the dQ pass (0: two launches).  Side by
// side the passes fill the waves that each alone would leave partly empty and save a launch; one
// after the other the dK / dV pass reads the keep bits that the dQ pass drew instead of drawing them
// again, and each pass has its tensors in L2 to itself.  Weighed as rounds of work items, in tiles
// of the dQ pass: a tile of dK / dV takes 1.4 of them (1.37 for D = 128; with dropout, which costs the dQ pass more,
// 1.05 and 1.27, and 0.5 more drawing), an item a quarter more (D = 128: one, its dK has no second set of
// accumulators to go on with), a launch 2; both in one came out a tenth under that.  Under a causal mask without
// dropout items differ and the heaviest go first, so that no whole rounds are lost in two launches or one: side by
// side up to 5 waves of each.  (With dropout, where drawing counts, causal calls are weighed as the others.)
// Measured, two launches -> one (us).  Taken side by side: 1 x 512 x 16 x 64: 23.3 -> 15.0; 1 x 2048 x 12 x 64 causal: 86
// -> 54; 4 x 512 x 16 x 64: 38.5 -> 28.4; 2 x 1024 x 16 x 128, p 0.1: 94 -> 77; 3 x 1820 x 8 x 128 causal, p 0.1: 162 -> 113; 27
// x 245 x 8 x 64 causal, p 0.1: 44 -> 36; 7 x 1496 x 16 x 64: 331 -> 305; 4 x 1024 x 16 x 128: 122 -> 112; 32 x 256 x 16 x
// 128: 94 -> 87.  Not: 16 x 512 x 16 x 64, p 0.1: 113 -> 137; 20 x 172 x 32 x 64, p 0.1: 83 -> 89; 19 x 378 x 12 x 64, p 0.1: 1.18
// times as long; 32 x 493 x 8 x 128, p 0.1: 155 -> 164.  Over 60 shapes, half of them drawn, the rule is 1.6 % over the
// better of all that was tried (4.1 % with the weights of earlier kernels, 25 % with two launches always), at
// worst 20 % (12 x 684 x 4 x 80, p 0.1: 80, not 67).
static int both_q_ctas(int64_t q_items, int64_t k_items, int64_t q_item_tiles, int64_t q_tiles, int D,
                       bool causal, bool rel, bool drop) {
  const int64_t sms = sm_count();
  const double item = D <= 64 ? 0.25 : 1.0;
  const double k_tile = rel ? 1.4 : (D <= 64 ? (drop ? 1.05 : 1.4) : (drop ? 1.27 : 1.37));
  const double q_item = q_item_tiles + item, k_item = q_tiles * k_tile + item;
  const double k_item_draws = q_tiles * (k_tile + (drop ? 0.5 : 0.0)) + item;
  if (q_items + k_items <= sms) return static_cast<int>(q_items);
  auto rounds = [](int64_t items, int64_t ctas) { return (items + ctas - 1) / ctas; };
  double best = (rounds(q_items, sms) * q_item + rounds(k_items, sms) * k_item + 2.0) / 0.9;
  if (causal && !drop) best = q_items + k_items > 10 * sms ? 0.0 : 1e30;
  int best_n = 0;
  for (int64_t r = rounds(q_items, sms - 1); r * q_item < best; ++r) {
    const int64_t n = rounds(q_items, r);       // the fewest CTAs with r rounds
    const double k_time = rounds(k_items, sms - n) * k_item_draws;
    const double t = r * q_item > k_time ? r * q_item : k_time;
    if (t < best) { best = t; best_n = static_cast<int>(n); }
    if (n == 1) break;
  }
  return best_n;
}

FlashBwdPlan flash_bwd_plan(int B, int H, int Sq, int Sk, int D, bool packed, bool causal,
                            bool key_bias, bool rel, float p_drop, int64_t keep_words) {
  FlashBwdPlan s;
  const int64_t rq = round128(Sq), rk = round128(Sk), bh = static_cast<int64_t>(B) * H;
  const int64_t q_tiles = rq / 128, k_tiles = rk / 128;
  const bool drop = dropout_thr7(p_drop) != 0;
  // Few queries, many keys: the keys of a dQ item are split over idle SMs, down to the other pass's
  // chain of tiles, where that takes four tiles off its own.  (2 x 60 queries x 2000 keys x 8 x 128:
  // 72 -> 48 us for the whole backward.)
  s.splits = 1;
  if (!packed && bh > 0 && q_tiles > 0 && k_tiles > q_tiles) {
    int64_t n = sm_count() / (q_tiles * bh);
    const int64_t most = (k_tiles + q_tiles - 1) / q_tiles;
    if (n > most) n = most;
    if (n >= 2) {
      const int64_t per = (k_tiles + n - 1) / n;
      if (k_tiles - per >= 4) s.splits = static_cast<int>((k_tiles + per - 1) / per);
    }
  }
  s.q_ctas = bh == 0 || keep_words > 0 ? 0
                     : both_q_ctas(q_tiles * bh * s.splits, k_tiles * bh,
                                   (k_tiles + s.splits - 1) / s.splits, q_tiles, D, causal, rel, drop);
  s.stats = 2 * bh * rq;
  s.bias = key_bias ? B * rk : 0;
  const bool keep = drop && s.q_ctas == 0;
  const int64_t words = rk / 32 * rq;
  if (keep_words <= 0) keep_words = int64_t(1) << 28;
  int64_t pairs = keep && words > 0 ? keep_words / words : bh;
  if (pairs < 1) pairs = 1;
  if (pairs > bh) pairs = bh;
  s.pairs = static_cast<int>(pairs);
  s.keep = keep ? s.pairs * words : 0;
  s.part = s.splits > 1 ? s.splits * bh * Sq * D : 0;
  return s;
}

int launch_flash_bwd(const void* q, const void* k, const void* v, const void* o, const void* dout,
                     const float* lse, const FlashBwdPlan& plan, float* scratch, void* dq, void* dk,
                     void* dv, int64_t dq_row_stride, int64_t dkv_row_stride, const float* kbias,
                     const float* rel, float* drel, int B, int H, int Sq, int Sk, int D,
                     const int64_t* q_strides, const int64_t* k_strides, const int64_t* v_strides,
                     float scale, int causal, float p_drop, PhiloxArgs rng, bool bf16, int* status,
                     cudaStream_t stream) {
  if (D < 8 || D > 128 || D % 8 != 0 || B > 65535) return 1;
  if (B <= 0 || H <= 0 || Sq <= 0 || Sk <= 0) return 1;
  CUtensorMap tq, tk, tv, tdo;
  const int64_t do_strides[3] = {static_cast<int64_t>(Sq) * H * D, static_cast<int64_t>(H) * D, D};
  if (!make_tmap_bshd(&tq, q, B, Sq, H, D, q_strides[0], q_strides[1], q_strides[2], 64, bf16) ||
      !make_tmap_bshd(&tk, k, B, Sk, H, D, k_strides[0], k_strides[1], k_strides[2], 64, bf16) ||
      !make_tmap_bshd(&tv, v, B, Sk, H, D, v_strides[0], v_strides[1], v_strides[2], 64, bf16) ||
      !make_tmap_bshd(&tdo, dout, B, Sq, H, D, do_strides[0], do_strides[1], do_strides[2], 64, bf16))
    return 2;
  FlashBwdParams p;
  p.Sq = Sq; p.Sk = Sk; p.H = H; p.Dr = D;
  p.k_steps = (D + 15) / 16;
  p.Rq = round128(Sq); p.Rk = round128(Sk);
  p.thr7 = dropout_thr7(p_drop);   // same quantisation as the forward kernel
  const float keep_prob = 1.f - p.thr7 / 128.f;
  // scratch: nlse | ndelta | key bias | keep bits | shares of dQ, each a multiple of 4 words (the
  // first four of 128)
  float* nlse = scratch;
  float* ndelta = nlse + plan.stats / 2;
  float* kb2 = ndelta + plan.stats / 2;
  p.nlse = nlse; p.ndelta = ndelta;
  p.kb2 = kbias != nullptr ? kb2 : nullptr;
  p.keep = plan.keep != 0 ? reinterpret_cast<uint32_t*>(kb2 + plan.bias) : nullptr;
  p.part = kb2 + plan.bias + plan.keep;
  p.part_rows = static_cast<int64_t>(B) * Sq * H;
  p.rel = rel; p.drel = drel;
  p.scale = scale; p.scale_log2 = scale * kLog2e; p.inv_keep = 1.f / keep_prob;
  p.causal = causal; p.rng = rng; p.status = status;
  p.idesc_s = tc::instr_desc_f16(128, 64, bf16 ? 1 : 0, false, false);
  p.idesc_acc = tc::instr_desc_f16(128, p.k_steps * 16, bf16 ? 1 : 0, false, true);
  {
    const int lanes = D <= 64 ? 8 : 16;
    const dim3 grid((p.Rq + 31) / 32, (H + 7) / 8, B);
    count_launch();
    if (bf16)
      flash_bwd_stats_kernel<__nv_bfloat16><<<grid, 256, 0, stream>>>(
          static_cast<const __nv_bfloat16*>(dout), static_cast<const __nv_bfloat16*>(o), lse, nlse,
          ndelta, kbias, kb2, H, Sq, p.Rq, Sk, p.Rk, D, lanes, keep_prob);
    else
      flash_bwd_stats_kernel<__half><<<grid, 256, 0, stream>>>(
          static_cast<const __half*>(dout), static_cast<const __half*>(o), lse, nlse, ndelta, kbias,
          kb2, H, Sq, p.Rq, Sk, p.Rk, D, lanes, keep_prob);
    if (cudaGetLastError() != cudaSuccess) return 4;
  }
  const bool general = kbias != nullptr || rel != nullptr || causal || Sk % 128 != 0;
  const int bh = B * H;
  FlashBwdParams pq = p, pk = p;
  pq.splits = plan.splits;
  pq.tiles_per_split = (p.Rk / 128 + plan.splits - 1) / plan.splits;
  pq.out1 = dq; pq.row_stride1 = dq_row_stride;
  pq.out2 = nullptr; pq.row_stride2 = 0;
  pk.splits = 1;
  pk.tiles_per_split = p.Rq / 128;
  pk.out1 = dk; pk.row_stride1 = dkv_row_stride;
  pk.out2 = dv; pk.row_stride2 = dkv_row_stride;
  for (int at = 0; at < bh; at += plan.pairs) {
    const int pairs = bh - at < plan.pairs ? bh - at : plan.pairs;
    pq.walk.set(p.Rq / 128, at, pairs, causal ? 2 : 0);
    pk.walk.set(p.Rk / 128, at, pairs, causal ? 1 : 0);
#define FLASH_BWD_CASE(T_)                                                                          \
  p.thr7 != 0 ? launch_typed<true, T_>(tq, tk, tv, tdo, pq, pk, plan.q_ctas, general, stream)       \
              : launch_typed<false, T_>(tq, tk, tv, tdo, pq, pk, plan.q_ctas, general, stream)
    const int rc = bf16 ? (FLASH_BWD_CASE(__nv_bfloat16)) : (FLASH_BWD_CASE(__half));
#undef FLASH_BWD_CASE
    if (rc != 0) return rc;
  }
  if (plan.splits > 1) {
    const int64_t n = p.part_rows * D;
    const unsigned blocks = static_cast<unsigned>((n / 8 + 255) / 256);
    const float f = p.scale * p.inv_keep;
    count_launch();
    if (bf16)
      flash_dq_combine_kernel<__nv_bfloat16><<<blocks, 256, 0, stream>>>(
          p.part, static_cast<__nv_bfloat16*>(dq), plan.splits, n, f);
    else
      flash_dq_combine_kernel<__half><<<blocks, 256, 0, stream>>>(p.part, static_cast<__half*>(dq),
                                                                  plan.splits, n, f);
    if (cudaGetLastError() != cudaSuccess) return 4;
  }
  return 0;
}

}  // namespace slapo
