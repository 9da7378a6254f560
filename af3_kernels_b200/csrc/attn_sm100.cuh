// Biased, key-masked flash attention for sm_100a:  out = softmax(scale * Q K^T + bias, masked) V
//
// Replaces the per-(batch, head, 128-query block) TPP sequence of the reference
// (src/csrc/dot_product_attention.cpp:88-122: scale -> BRGEMM -> add bias -> add mask ->
// softmax -> BRGEMM) with one persistent warp-specialised kernel:
//
//   warp 0      TMA producer: Q tiles, K/V ring, bias ring (cp.async.bulk.tensor, each CTA loads its own tiles)
//   warp 1      tcgen05.mma issuer for the logits (smem x smem -> TMEM)
//   warp 2      TMEM allocator, then tcgen05.mma issuer for O += P V (TMEM x smem -> TMEM)
//   warp 3      key-mask writer (see below)
//   warps 4-7   softmax warpgroup 0 (owns S / P buffer 0 and the even streams of a work item)
//   warps 8-11  softmax warpgroup 1 (owns S / P buffer 1 and the odd streams); or, where items have one stream and the bias
//               is converted here, warps 8-15 that make the bias tiles
//
// A work item is (head, 128-query tile, group of G pair rows).  The G "streams" of an item use
// the same bias tiles, so one staged bias tile serves G logits tiles; each stream has its own
// Q tile, K/V tiles, fp32 running max / sum and O accumulator in TMEM.  One softmax thread owns
// one query row (TMEM lane), so row max / row sum need no cross-thread traffic.
//
// The softmax threads are the bottleneck of this operator (one exponential per logit on the
// 16-lane XU, every other instruction competing for the same issue slots), so everything that
// can be an MMA is one.  With bf16 q/k the whole logit comes out of the tensor core:
//
//   * scale: the softmax warps multiply each Q tile by the softmax scale in shared memory, an item ahead, and round it
//     back to bf16 - the reference's own first step (q = q * scaling, in bf16);
//   * bias: eight small MMAs per tile (M = 128, N = 16, K = 16) whose A operand is a 16-key
//     slice of the staged bf16 bias tile and whose B operand is a 16 x 16 identity, each adding
//     its slice into 16 columns of the accumulator - exact, the products are bias x 1;
//   * key mask: one more K step whose A operand is a column of ones and whose B operand holds,
//     per key, 0 (attend), -2^47 (masked) or -inf (beyond the sequence).  A masked key ends up
//     with weight exactly 0, a row whose keys are all masked with uniform weights over its real
//     keys (what "fill with -1e9, then softmax" gives), a key that does not exist with weight 0.
//
// What is left per logit is a maximum, one fused multiply-add, the exponential, the row sum and
// the bf16 rounding of P.  With fp8 q/k the logit scale t = softmax scale x the two
// de-quantisation factors cannot be folded into Q; there the bias staging pass divides the bias
// by t, the tensor core adds it to the raw fp8 products, the masked-key value is enlarged by 1/t,
// and t rides on the fused multiply-add.  When the caller gives no room for that staging copy
// the second instantiation of the kernel runs, in which the softmax threads apply t and add the
// bias in fp32 from the staged tile in shared memory; the mask column is used either way.
//
// Logits stay fp32 from the tensor core to the exponential; P is rounded to bf16 once, when it
// is written to TMEM as the A operand of the second GEMM.  S and P live in separate TMEM columns:
// a warpgroup releases its S buffer as soon as the logits are in registers, so the next logits
// tile of that buffer is computed under the softmax of the current one.  O is rescaled lazily:
// only when a row maximum grows by more than 2^8 (exact, because l is scaled with it).
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <cstdint>
#include <type_traits>

#include "ptx_sm100.cuh"

namespace af3k {

constexpr int kTile = 128;         // query rows per tile, and the most keys
constexpr int kThreads = 384;      // 12 warps
constexpr int kConvertThreads = 512;   // kConvert: one softmax warpgroup, eight warps that make bias tiles
// 65536 registers per SM: launched at 168 per thread, then 128 x 72 + 256 x 216 = 64512
constexpr int kRegsMisc = 72, kRegsSoftmax = 216;
// kConvert: launched at 128 per thread, then 128 x 72 + 128 x 216 + 256 x 104 = 63488 of 65536
constexpr int kRegsConvert = 104;
constexpr int kMaxStreams = 4;     // pair rows per work item (two per softmax warpgroup; TMEM: kOCol + G * nv <= 512 columns)
// TMEM columns: two fp32 logits buffers, two bf16 P buffers (two keys per column), then O.
constexpr uint32_t kSCol = 0, kPCol = 2 * 128, kOCol = 2 * 128 + 2 * 64;
constexpr float kLazyRescaleLog2 = 8.0f;   // keep a stale row max while exp2 arguments stay <= 8
constexpr int kTailRows = 2;       // pair rows of an item behind the last full round: both softmax warpgroups have work
constexpr int kMaxBiasStages = 3;
constexpr int kBiasTileBytes = kTile * kTile * 2;  // bf16, two 128B-swizzled boxes of 64 columns
constexpr int kMaxKvStages = 6;
constexpr uint32_t kNarrowOff = kTile * 64;        // qk_narrow: channels 32 .. 47 behind the first 32
constexpr uint32_t kTmemCols = 512;
// bf16 bit patterns of the mask column.  -2^47 stands in for the reference's "-1e9" fill: added
// in fp32 to any logit below 2^23 in magnitude it gives exactly -2^47, so all masked keys of a
// row are equal (uniform weights when nothing else is left) and vanish next to any real key.
constexpr uint16_t kMaskColKeep = 0x0000, kMaskColMasked = 0xD700, kMaskColAbsent = 0xFF80;
constexpr uint32_t kMaskPanelBytes = 2048;   // 128 keys x one 16-byte core-matrix row
constexpr uint32_t kBarrierBlockBytes = 512;
constexpr uint32_t kIdentBytes = 512;        // 16 x 16 bf16 identity, K-major core matrices
constexpr float kLog2e = 1.4426950408889634f;

// Exponentials: every weight is one ex2.approx.f32 on the XU (16 lanes per SM and clock: 4 results per
// clock and scheduler).  Measured alternatives that do not beat it here: ex2.approx.f16x2 / .bf16x2 take
// 16 XU cycles per warp instruction (the same 4 results per clock), kind::f16 MMAs take no f16 A with a
// bf16 B, and a degree-3 polynomial on the FMA pipe costs more issue slots than the ex2 it replaces.

enum StatusBits : int {
  kStatusOk = 0,
  kStatusWaitTimeout = 1,   // a bounded mbarrier wait ran out
};

// x / d for 0 <= x < 2^31 by a multiplication (d == 1: mul == 0).  Every role decodes every item, and a division is some
// forty instructions, several times over in each role's loop.
struct Divisor {
  uint32_t d, mul, shift;
};
inline Divisor make_divisor(uint32_t d) {
  Divisor r{d, 0, 0};
  if (d > 1) {
    uint32_t l = 1;
    while ((1ull << l) < d) ++l;
    r.mul = (uint32_t)(((1ull << (31 + l)) + d - 1) / d);
    r.shift = l - 1;
  }
  return r;
}
__device__ __forceinline__ uint32_t divide(uint32_t x, const Divisor& v) { return v.mul != 0 ? __umulhi(x, v.mul) >> v.shift : x; }

struct AttnParams {
  int B1, B2, Sq, Sk, D;
  int n_qt, n_kt;
  int kw;                // keys per key tile (the kernel's kW; its kLast: of the last one)
  int G;                 // pair rows per work item
  int q_split;           // 1: the streams of an item are two neighbouring query tiles of ONE pair row (G == 1)
  int n_streams;         // streams per work item: G, or 2 with q_split
  int n_items;
  int mixed;             // 1: the kernel's kMixed
  int n_main, tail_row;  // the items behind the first n_main are smaller: kTailRows rows each, of the rows from tail_row on
  Divisor div_q, div_h;  // query tiles (or pairs of them) per row and head, heads
  int qk_row_bytes;      // smem bytes per Q / K tile row: 32, 64 or 128 (= swizzle span)
  // 1: bf16 heads of 33 to 48 channels.  A Q / K tile is 32 channels in rows of 64 bytes, then 16 in rows of 32 bytes: 12 KB
  // instead of the 16 KB of 128-byte rows, which makes room for a fourth K/V stage beside two streams' Q tiles (three stages
  // do not cover the loads' latency; 5 x 16 heads x 1536 tokens x 48 channels: 112 -> 99 us a call).  V keeps its
  // 128-byte rows: it is an MN-major operand, whose columns one MMA reads in one swizzle.
  int qk_narrow;
  int v_row_bytes;       // same for V
  int qk_ksteps;         // number of 32-byte K steps of the first GEMM
  int nv;                // N of the second GEMM: D rounded up to 16
  int kv_stages;
  int bias_stages;
  int q_buffers;         // 2: Q tiles double-buffered by item (the next item's land while this one runs); 1: single
  int scale_q;           // 1: bf16 q/k, the Q tiles are multiplied by `scale` in shared memory
  float scale;           // softmax scale; multiplied by q_scale[h] * k_scale[h] when those are set
  const float* q_scale;
  const float* k_scale;
  const uint8_t* mask;   // 1 = attend; nullptr = no mask
  long long mask_row_stride;
  __nv_bfloat16* out;
  long long out_stride_b1, out_stride_b2, out_stride_s;
  const __nv_bfloat16* gate;   // null, or [B1, B2, Sq, D]: the result is multiplied by sigmoid(gate) before it is rounded
  long long gate_stride_b1, gate_stride_b2, gate_stride_s;
  int* status;           // int[4]: {status bits, 1 + first barrier slot that timed out, block, warp}
  long long wait_limit;  // SM clocks a single wait may take before the kernel gives up
  float* debug;          // diagnostic dump of block 0's first logits tile (debug build of the kernel)
  uint32_t q_tile_bytes, k_tile_bytes, v_tile_bytes;   // in shared memory: 128 rows each
  uint32_t kv_load_bytes;                              // what a K and V tile's loads bring
  uint32_t off_q, off_kv, off_bias, off_bar;   // from the 1024-aligned smem base
  // mask-column operands of the extra K step (all no-swizzle, K-major, 16-byte rows):
  //   off_ones: A operand, element (row, 0) = 1;  off_mcol: ring of per-tile B operands, element
  //   (key, 0) = mask value;  off_zero: the all-zero second half of K shared by both.
  uint32_t off_ones, off_mcol, off_zero;
  uint32_t off_ident;    // 16 x 16 identity (B operand of the bias MMAs)
  // kConvert: the bias as the caller holds it
  const void* bias_src;
  long long bias_stride_h, bias_stride_r;
  int bias_f32, bias_wide;   // bias_wide: rows start on boundaries of four keys and end there
  int mask_col;          // 1: the extra K step runs (a mask was given or Sk is not a tile multiple)
};

// Barrier slots inside the barrier block (8 bytes each, kBarrierBlockBytes in all).
struct BarIdx {
  static constexpr int s_full = 0;      // [2]  logits of a tile finished
  static constexpr int s_free = 2;      // [2]  softmax warpgroup has the logits in registers
  static constexpr int p_ready = 4;     // [2]  P written (and O rescaled if needed)
  static constexpr int pv_done = 6;     // [2]  the warpgroup's last P V has finished: its P buffer and that O are free
  static constexpr int bias_full = 8;   // [kMaxBiasStages]
  static constexpr int bias_empty = bias_full + kMaxBiasStages;
  static constexpr int kv_full = bias_empty + kMaxBiasStages;   // [kMaxKvStages]
  static constexpr int kv_empty = kv_full + kMaxKvStages;       // P V of the stage's tile finished
  // Q tiles: slot = (Q buffer) * kMaxStreams + stream
  static constexpr int q_full = kv_empty + kMaxKvStages;       // [2 * kMaxStreams]  Q tile landed
  static constexpr int q_empty = q_full + 2 * kMaxStreams;   // [2 * kMaxStreams]  last Q K^T of the stream finished
  static constexpr int q_scaled = q_empty + 2 * kMaxStreams; // [2 * kMaxStreams]  the softmax warpgroup's warps have scaled the Q tile
  static constexpr int count = q_scaled + 2 * kMaxStreams;
};
constexpr uint32_t kWaitBlockOff = kBarrierBlockBytes - 32;
static_assert(BarIdx::count * 8 <= (int)kWaitBlockOff, "barrier block too small");

// Diagnostic dump: four [128][128] float sections, row = query row of block 0's first stream: raw logits and packed P words (64
// used) of its first key tile, un-normalised O (nv used) and {unused, sum} behind its last.
constexpr int kDbgTimelineTiles = 256;   // per warpgroup; 8 clock values each, after kDbgFloats floats
constexpr int kDbgS = 0, kDbgP = kTile * kTile, kDbgO = 2 * kTile * kTile, kDbgML = 3 * kTile * kTile,
              kDbgFloats = 4 * kTile * kTile;

struct Ctx {
  const AttnParams* p;
  uint32_t smem;       // 1024-aligned shared base (shared-window address)
  uint32_t bars;       // shared address of barrier block
  volatile int* abort_flag;
  uint32_t tmem;       // TMEM base address
};

__device__ __forceinline__ uint32_t bar_addr(const Ctx& c, int idx) { return c.bars + 8u * idx; }

// Behind the barriers, for waits that take long: what the waiting loop needs, so that a call of it carries three words.
struct WaitBlock {
  long long limit;     // AttnParams::wait_limit
  int* status;         // AttnParams::status
  int* abort_flag;
};

__device__ __forceinline__ const WaitBlock* wait_block_of(uint32_t bars) {
  return reinterpret_cast<const WaitBlock*>(__cvta_shared_to_generic(bars + kWaitBlockOff));
}

__device__ __noinline__ void report_timeout_at(int* status, volatile int* abort_flag, int bar_idx) {
  *abort_flag = 1;
  if (status != nullptr) {
    atomicOr(status, kStatusWaitTimeout);
    if (atomicCAS(status + 1, 0, bar_idx + 1) == 0) {
      status[2] = blockIdx.x;
      status[3] = threadIdx.x >> 5;
    }
  }
}
__device__ __forceinline__ void report_timeout(const Ctx& c, int bar_idx) { report_timeout_at(c.p->status, c.abort_flag, bar_idx); }

// The waiting loop of the single-warp roles, out of line, with the report of a wait that ran out.
__device__ __noinline__ bool wait_slow(uint32_t bar, uint32_t parity, const WaitBlock* w) {
  if (mbar_wait_bounded(bar, parity, w->limit, w->abort_flag)) return true;
  report_timeout_at(w->status, w->abort_flag, (int)((bar - smem_u32(w) + kWaitBlockOff) >> 3));
  return false;
}

// One thread (the producer).
#define AF3K_WAIT(ctx, idx, parity)                                                                     \
  do {                                                                                                  \
    const uint32_t bar_ = bar_addr(ctx, idx), par_ = (parity);                                          \
    if (!mbar_try_wait_park(bar_, par_, 2000u) && !wait_slow(bar_, par_, wait_block)) return;           \
  } while (0)

// A whole warp: every lane leaves together, so no .sync.aligned instruction is ever executed by part of a warp after a
// timeout.  One parked attempt, in which most real waits end; the rest is out of line, because the single-warp roles' loops are
// fetched again for every tile, beside warps that stream through long unrolled code.
#define AF3K_WAIT_WARP_C(ctx, idx, parity)                                                              \
  do {                                                                                                  \
    const uint32_t bar_ = bar_addr(ctx, idx), par_ = (parity);                                          \
    if (!__all_sync(0xffffffffu, mbar_try_wait_park(bar_, par_, 2000u)))                                \
      if (!__all_sync(0xffffffffu, wait_slow(bar_, par_, wait_block))) return;                          \
  } while (0)
// The softmax warps keep the waiting loop inline: a call would have to save their registers.
#define AF3K_WAIT_WARP(ctx, idx, parity)                                                     \
  do {                                                                                       \
    const bool ok_ = mbar_wait_bounded(bar_addr(ctx, idx), (parity), (ctx).p->wait_limit,    \
                                       (ctx).abort_flag);                                    \
    if (!__all_sync(0xffffffffu, ok_)) {                                                     \
      report_timeout(ctx, idx);                                                              \
      return;                                                                                \
    }                                                                                        \
  } while (0)

__device__ __forceinline__ uint32_t swizzle_layout_code(int row_bytes) {
  return row_bytes == 128 ? 2u : (row_bytes == 64 ? 4u : 6u);
}

// A work item: head h, first query tile qt, first pair row r0, gv streams.  Normally the streams
// are gv pair rows sharing one query tile index (and therefore one bias tile per key tile).  With
// q_split (chosen when there is a single pair row per item, so that the second softmax warpgroup
// is not left idle) they are gv neighbouring query tiles of pair row r0, each with its own bias
// tiles.
struct Item {
  int qt, h, r0, gv;
};
template <bool kMixed>
__device__ __forceinline__ Item decode_item(const AttnParams& p, int item) {
  Item it;
  if (!kMixed) {
    const uint32_t t = divide((uint32_t)item, p.div_q), rg = divide(t, p.div_h);
    it.qt = (int)((uint32_t)item - t * p.div_q.d) << p.q_split;
    it.h = (int)(t - rg * p.div_h.d);
    it.r0 = (int)rg * p.G;
    it.gv = p.n_streams;
    return it;
  }
  const bool tail = item >= p.n_main;
  const uint32_t i = (uint32_t)(tail ? item - p.n_main : item);
  const int g = tail ? kTailRows : p.G, row = tail ? p.tail_row : 0, end = tail ? p.B1 : p.tail_row;
  const uint32_t t = divide(i, p.div_q), rg = divide(t, p.div_h);
  it.qt = (int)(i - t * p.div_q.d) << p.q_split;
  it.h = (int)(t - rg * p.div_h.d);
  it.r0 = row + (int)rg * g;
  it.gv = p.q_split ? min(2, p.n_qt - it.qt) : min(g, end - it.r0);
  return it;
}
__device__ __forceinline__ int stream_row(const AttnParams& p, const Item& it, int s) { return p.q_split ? it.r0 : it.r0 + s; }
__device__ __forceinline__ int stream_qt(const AttnParams& p, const Item& it, int s) { return p.q_split ? it.qt + s : it.qt; }

// Q buffer of the CTA's j-th item and how often that buffer was used before.  (kMixed) An item with fewer streams than the Q
// buffers hold takes the slots of the others through their phases all the same, so that one count serves all slots: counting
// every slot's own uses in the issuer's loop cost 2 - 5 %.  Each role does there what it does for a slot in use, less the copy,
// the scaling and the MMAs: a wait by parity cannot tell a phase from the one two before it, so whoever waits on a slot's barriers
// at all must wait for every phase of theirs and must itself be waited for before the phase after the next can end.  The producer
// arrives (q_full), the softmax warps wait for that and arrive (q_scaled; nobody does where Q is not scaled), the issuer waits for that and
// arrives (q_empty), the producer waits for that.  A warpgroup without a stream in an item (a lone query tile) is held by nothing else.
__device__ __forceinline__ uint32_t q_buf(const AttnParams& p, uint32_t j) { return p.q_buffers == 2 ? (j & 1u) : 0u; }
__device__ __forceinline__ uint32_t q_use(const AttnParams& p, uint32_t j) { return p.q_buffers == 2 ? (j >> 1) : j; }

// ------------------------------------------------------------------ producer (one thread)
template <bool kMixed, bool kConvert, int kW, int kLast>
__device__ void producer_role(const Ctx& c, const CUtensorMap* tm_q, const CUtensorMap* tm_k,
                              const CUtensorMap* tm_v, const CUtensorMap* tm_bias, const CUtensorMap* tm_q2, const CUtensorMap* tm_k2) {
  const AttnParams& p = *c.p;
  const WaitBlock* wait_block = wait_block_of(c.bars);
  uint32_t icount = 0;
  uint32_t st = 0, lap = 0, bst = 0, blap = 0;     // K/V and bias ring: stage, laps before
  const uint32_t nkv = p.kv_stages, n_bias = p.bias_stages;
  // With two Q buffers the tiles of the next item are requested while the current item runs, so
  // that they are in place (and scaled) when it ends; with one (tiles too large for two), as
  // soon as the current item's K/V loads are all issued.  When a K/V stage of this item has come free, the last item's Q K^T have
  // finished, which the loads wait for (5 x 1536 tokens of 48 channels 86.9 us, 87.5 behind the first key tile; others the same), but where they
  // are scaled in front of the last key tile, so that this is not left over (256 rows of two key tiles, 16 channels: 29.5 us, 30.7 behind it).
  const int q_at = p.q_buffers == 2 ? min((int)(nkv / (uint32_t)p.n_streams) + 1, max(p.n_kt - p.scale_q, 1)) : p.n_kt;
#pragma unroll 1
  for (int item = blockIdx.x; item < p.n_items; item += gridDim.x, ++icount) {
    const Item it = decode_item<kMixed>(p, item);
#pragma unroll 1
    for (int kt = 0; kt <= p.n_kt; ++kt) {
      const bool own = kt == 0 && icount == 0;
      const int q_item = own ? item : item + (int)gridDim.x;
      if ((own || kt == q_at) && q_item < p.n_items) {
        const uint32_t j = own ? 0 : icount + 1, buf = q_buf(p, j), use = q_use(p, j);
        const Item qi = decode_item<kMixed>(p, q_item);
#pragma unroll 1
        for (int s = 0; s < p.n_streams; ++s) {
          const int slot = (int)buf * kMaxStreams + s;
          // the buffer's previous user must have finished its last Q K^T of this stream
          if (use >= 1) AF3K_WAIT(c, BarIdx::q_empty + slot, (use - 1) & 1);
          const uint32_t full = bar_addr(c, BarIdx::q_full + slot);
          if (own && s == 0) {       // (a CTA's first item has a first stream)
            grid_wait_previous();
            grid_release_next();
          }
          if (kMixed && s >= qi.gv) {
            mbar_arrive(full);
            continue;
          }
          mbar_arrive_expect_tx(full, p.q_tile_bytes);
          const uint32_t qdst = c.smem + p.off_q + (buf * p.n_streams + s) * p.q_tile_bytes;
          tma_load_4d(qdst, tm_q, full, 0, stream_qt(p, qi, s) * kTile, qi.h, stream_row(p, qi, s));
          if (p.qk_narrow) tma_load_4d(qdst + kNarrowOff, tm_q2, full, 32, stream_qt(p, qi, s) * kTile, qi.h, stream_row(p, qi, s));
        }
      }
      if (kt == p.n_kt) break;
#pragma unroll 1
      for (int s = 0; s < it.gv; ++s) {
        if (!kConvert && (s == 0 || p.q_split)) {   // one bias tile per key tile, or per stream when the streams are query tiles
          if (blap != 0) AF3K_WAIT(c, BarIdx::bias_empty + bst, (blap - 1) & 1);
          const uint32_t bfull = bar_addr(c, BarIdx::bias_full + bst);
          const uint32_t bdst = c.smem + p.off_bias + bst * kBiasTileBytes;
          const bool both = kW > 64 && (kLast == kW || kLast > 64 || kt != p.n_kt - 1);      // boxes of 64 keys
          mbar_arrive_expect_tx(bfull, both ? kBiasTileBytes : kBiasTileBytes / 2);
          tma_load_3d(bdst, tm_bias, bfull, kt * kW, stream_qt(p, it, s) * kTile, it.h);
          if (both) tma_load_3d(bdst + kBiasTileBytes / 2, tm_bias, bfull, kt * kW + 64, stream_qt(p, it, s) * kTile, it.h);
          if (++bst == n_bias) { bst = 0; ++blap; }
        }
        if (lap != 0) AF3K_WAIT(c, BarIdx::kv_empty + st, (lap - 1) & 1);
        const uint32_t full = bar_addr(c, BarIdx::kv_full + st);
        const uint32_t kdst = c.smem + p.off_kv + st * (p.k_tile_bytes + p.v_tile_bytes);
        mbar_arrive_expect_tx(full, p.kv_load_bytes);
        tma_load_4d(kdst, tm_k, full, 0, kt * kW, it.h, stream_row(p, it, s));
        if (p.qk_narrow) tma_load_4d(kdst + kNarrowOff, tm_k2, full, 32, kt * kW, it.h, stream_row(p, it, s));
        tma_load_4d(kdst + p.k_tile_bytes, tm_v, full, 0, kt * kW, it.h, stream_row(p, it, s));
        if (++st == nkv) { st = 0; ++lap; }
      }
    }
  }
}

// ------------------------------------------------------------------ Q scaling and key-mask column
// q <- bf16(q * scale) for some KB of a Q tile in shared memory, 32 bytes per lane and KB (any swizzle: the operation is
// elementwise), then one arrival per warp.  (Out of line: two callers, once per item each.)
__device__ __noinline__ void scale_q(uint32_t addr, uint32_t bytes, float scale, int lane, uint32_t bar) {
  const uint64_t scale2 = pack_f32x2(scale, scale);
#pragma unroll 1
  for (uint32_t a = addr + lane * 16, end = a + bytes; a < end; a += 1024) {
    uint32_t w[8];
#pragma unroll
    for (int i = 0; i < 2; ++i)
      asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                   : "=r"(w[4 * i]), "=r"(w[4 * i + 1]), "=r"(w[4 * i + 2]), "=r"(w[4 * i + 3]) : "r"(a + 512 * i));
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      float q0, q1;
      unpack_f32x2(mul_f32x2(pack_f32x2(__uint_as_float(w[e] << 16), __uint_as_float(w[e] & 0xffff0000u)), scale2), q0, q1);
      w[e] = pack_bf16x2(q0, q1);
    }
#pragma unroll
    for (int i = 0; i < 2; ++i)
      asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(a + 512 * i), "r"(w[4 * i]), "r"(w[4 * i + 1]), "r"(w[4 * i + 2]),
                   "r"(w[4 * i + 3]) : "memory");
  }
  fence_proxy_async_smem();    // make the generic-proxy stores visible to the tensor core
  __syncwarp();
  if (lane == 0) mbar_arrive(bar);
}

// The mask-column values (bf16) of one logits tile, four per lane (those behind its last key are not read).
template <int kW>
__device__ __forceinline__ void mask_values(const AttnParams& p, const Item& it, int kt, int s, int lane,
                                            uint16_t masked, uint16_t (&val)[4]) {
  const uint8_t* mrow = p.mask != nullptr ? p.mask + (long long)stream_row(p, it, s) * p.mask_row_stride : nullptr;
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    const int key = kt * kW + 32 * g + lane;
    val[g] = key >= p.Sk ? kMaskColAbsent : ((mrow == nullptr || mrow[key] != 0) ? kMaskColKeep : masked);
  }
}

// bf16 bits of the value a masked key gets for head h.  The tensor core's logits are multiplied
// by the head's logit scale t afterwards when that scale is not folded into Q (fp8 q/k), so the
// value is -2^(47 + ceil(-log2 t)) there: still -2^47 or beyond after the multiplication.
__device__ __forceinline__ uint16_t masked_value_bits(const AttnParams& p, int h) {
  if (p.q_scale == nullptr) return kMaskColMasked;
  const float t = p.scale * p.q_scale[h] * p.k_scale[h];
  int e = 47 - min(0, ilogbf(t));
  e = min(e, 120);
  return (uint16_t)(0x8000u | ((uint32_t)(e + 127) << 7));
}

// Key-mask writer (one warp).  For every logits tile, in the producer's order: write the tile's
// mask values into its slot of the mask-column ring.  The slot is the B operand of the extra
// K step; only element 0 of each key's 16-byte row changes, the rest stays zero.  Arrives on the
// tile's kv_full barrier (which then counts two arrivals: this one and the producer's).  The mask
// bytes of a tile are requested one tile ahead, so their latency is not on the path.
template <bool kMixed, int kW>
__device__ void mask_writer_role(const Ctx& c, int lane) {
  const AttnParams& p = *c.p;
  const WaitBlock* wait_block = wait_block_of(c.bars);
  const uint32_t nkv = p.kv_stages;
  uint32_t st = 0, round = 0;      // ring slot, how many times the ring wrapped
  grid_wait_previous();
#pragma unroll 1
  for (int item = blockIdx.x; item < p.n_items; item += gridDim.x) {
    const Item it = decode_item<kMixed>(p, item);
    uint16_t val[4] = {};
    const uint16_t masked = masked_value_bits(p, it.h);
    // step i writes the values of tile i (key tiles outermost, then streams) and requests those of tile i + 1
    const int tiles = p.n_kt * it.gv;
    int nkt = 0, ns = 0;           // the tile requested next
#pragma unroll 1
    for (int i = -1; i < tiles; ++i) {
      const uint16_t cur[4] = {val[0], val[1], val[2], val[3]};
      if (i + 1 < tiles) {
        mask_values<kW>(p, it, nkt, ns, lane, masked, val);
        if (++ns == it.gv) { ns = 0; ++nkt; }
      }
      if (i >= 0) {
        if (round > 0) AF3K_WAIT_WARP_C(c, BarIdx::kv_empty + st, (round - 1) & 1);
        const uint32_t slot = c.smem + p.off_mcol + st * kMaskPanelBytes;
#pragma unroll
        for (int g = 0; g < 4; ++g)
          asm volatile("st.shared.u16 [%0], %1;" ::"r"(slot + (32 * g + lane) * 16), "h"(cur[g]) : "memory");
        fence_proxy_async_smem();    // make the generic-proxy stores visible to the tensor core
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_addr(c, BarIdx::kv_full + st));
        if (++st == nkv) { st = 0; ++round; }
      }
    }
  }
}

// ------------------------------------------------------------------ MMA issuers (two warps)
// The tiles here are small (N = 128, K = 16 and N = D, K = 16), so the cost of issuing an MMA
// matters: one thread issuing both GEMMs of every tile was the limiter of the whole kernel, and
// so was issuing from one lane of a diverged warp (about 150 cycles per tcgen05.mma, because the
// descriptors then travel through per-lane registers).  The two GEMMs are therefore issued by two
// warps, each running its control flow and its waits as a whole warp so that addresses and
// descriptors stay warp-uniform; one elected lane issues.  The two warps touch different TMEM
// columns and every hand-over between them goes through an mbarrier, so no ordering between the
// two instruction streams is assumed.

// Logits of every tile, in order: Q K^T, then the mask column, then (bf16 q/k) the bias slices.
// (The MMA loops are real loops and the fp8 / bf16 choice is a template argument: the warp pays an
// instruction-cache miss for most lines of this loop on every pass, so the loop is kept small.)
template <bool kDebug, bool kTcBias, bool kFp8, bool kMixed, int kW, int kLast>
__device__ void qk_issuer_role(const Ctx& c) {
  const AttnParams& p = *c.p;
  const WaitBlock* wait_block = wait_block_of(c.bars);
  const bool leader = elect_one();
  const uint32_t nkv = p.kv_stages;
  const uint32_t qk_layout = swizzle_layout_code(p.qk_row_bytes);
  constexpr bool fp8 = kFp8;
  const uint32_t idesc_qk = make_idesc(fp8 ? 0u : 1u, fp8 ? 0u : 1u, 0u, 0u, kW);
  const uint32_t kv_stage_bytes = p.k_tile_bytes + p.v_tile_bytes;
  // descriptor words for tile 0 / stage 0; later tiles only move the start-address field
  const uint64_t qd0 = make_smem_desc(c.smem + p.off_q, 16, 8 * p.qk_row_bytes, qk_layout);
  const uint64_t kd0 = make_smem_desc(c.smem + p.off_kv, 16, 8 * p.qk_row_bytes, qk_layout);
  const uint32_t qd_lo = (uint32_t)qd0, qd_hi = (uint32_t)(qd0 >> 32);
  const uint32_t kd_lo = (uint32_t)kd0;
  const uint32_t narrow_hi = (uint32_t)(make_smem_desc(0, 16, 8 * 32, swizzle_layout_code(32)) >> 32);
  const int wide_ksteps = p.qk_narrow ? 2 : p.qk_ksteps;
  const uint32_t q_step = p.q_tile_bytes >> 4, stage_step = kv_stage_bytes >> 4;
  const int ksteps = p.qk_ksteps;
  // extra K step: ones column x mask column, both K-major without swizzle (8-row groups 128 bytes
  // apart, the second 16-byte half of K in the shared zero block)
  const uint64_t od0 = make_smem_desc(c.smem + p.off_ones, p.off_zero - p.off_ones, 128, 0);
  const uint64_t md0 = make_smem_desc(c.smem + p.off_mcol, p.off_zero - p.off_mcol, 128, 0);
  const uint32_t od_lo = (uint32_t)od0, od_hi = (uint32_t)(od0 >> 32);
  const uint32_t md_lo = (uint32_t)md0, md_hi = (uint32_t)(md0 >> 32);
  const uint32_t idesc_mask = make_idesc(1u, 1u, 0u, 0u, kW);
  constexpr uint32_t idesc_short = make_idesc(0u, 0u, 0u, 0u, kW) - make_idesc(0u, 0u, 0u, 0u, kLast);
  const bool mask_col = p.mask_col != 0;
  // bias slices: A = 16 keys of the staged bias tile (K-major, 128-byte swizzled rows, two boxes
  // of 64 keys), B = the 16 x 16 identity (K-major, no swizzle: 8-key halves 256 bytes apart,
  // 8-row groups 128 bytes apart), D = 16 columns of the logits tile
  const uint64_t bd0 = make_smem_desc(c.smem + p.off_bias, 16, 8 * 128, 2);
  const uint64_t id0 = make_smem_desc(c.smem + p.off_ident, 256, 128, 0);
  const uint32_t bd_lo = (uint32_t)bd0, bd_hi = (uint32_t)(bd0 >> 32);
  const uint32_t id_lo = (uint32_t)id0, id_hi = (uint32_t)(id0 >> 32);
  const uint32_t idesc_bias = make_idesc(1u, 1u, 0u, 0u, 16);
  long long* tl = (kDebug && p.debug != nullptr && blockIdx.x == 0)
                      ? reinterpret_cast<long long*>(p.debug + kDbgFloats) + 2 * kDbgTimelineTiles * 8
                      : nullptr;
  uint32_t tl_n = 0;
  // ring positions / barrier parities are carried incrementally: no division on this warp
  uint32_t st = 0, kv_par = 0, icount = 0, bst = 0, b_par = 0;
  uint32_t sfree_par = 0, used = 0;   // bit b: parity of buffer b's next release; buffer b has held a tile
  grid_wait_previous();            // (nothing is there before; a wait's limit counts from here)
#pragma unroll 1
  for (int item = blockIdx.x; item < p.n_items; item += gridDim.x, ++icount) {
    const Item it = decode_item<kMixed>(p, item);
    const int gv = it.gv;
#pragma unroll 1
    for (int kt = 0; kt < p.n_kt; ++kt) {
#pragma unroll 1
      for (int s = 0; s < gv; ++s) {
        const int b = s & 1;
        const int qslot = (int)q_buf(p, icount) * kMaxStreams + s;
        const int q_bar = (p.scale_q ? BarIdx::q_scaled : BarIdx::q_full) + qslot;
        const bool need_bias = kTcBias && (s == 0 || p.q_split);
        const bool need_sfree = (used >> b) & 1u;
        const uint32_t sf_par = (sfree_par >> b) & 1u;
        {
          // everything the tile needs is normally there already: test all its barriers, vote once
          bool ok = mbar_test_wait(bar_addr(c, BarIdx::kv_full + st), kv_par);
          if (need_sfree) ok = mbar_test_wait(bar_addr(c, BarIdx::s_free + b), sf_par) && ok;
          if (need_bias) ok = mbar_test_wait(bar_addr(c, BarIdx::bias_full + bst), b_par) && ok;
          if (kt == 0) ok = mbar_test_wait(bar_addr(c, q_bar), q_use(p, icount) & 1) && ok;
          if (!__all_sync(0xffffffffu, ok)) {
            // (the softmax warpgroup of this buffer must have read the previous logits tile)
            if (need_sfree) AF3K_WAIT_WARP_C(c, BarIdx::s_free + b, sf_par);
            if (need_bias) AF3K_WAIT_WARP_C(c, BarIdx::bias_full + bst, b_par);
            if (kt == 0) AF3K_WAIT_WARP_C(c, q_bar, q_use(p, icount) & 1);
            AF3K_WAIT_WARP_C(c, BarIdx::kv_full + st, kv_par);
          }
        }
        if (need_sfree) sfree_par ^= 1u << b;
        used |= 1u << b;
        tc_fence_after();
        const uint32_t a_lo = qd_lo + (q_buf(p, icount) * p.n_streams + s) * q_step;
        const uint32_t b_lo = kd_lo + st * stage_step;
        const uint32_t s_tmem = c.tmem + kSCol + b * kTile;
        const uint32_t slot16 = st * (kMaskPanelBytes >> 4);
        const uint32_t bias_lo = bd_lo + bst * (kBiasTileBytes >> 4);
        if (leader) {
          const long long t0 = kDebug && tl != nullptr ? clock64() : 0;
          const bool narrow = kLast != kW && kt == p.n_kt - 1;
          const uint32_t fewer = narrow ? idesc_short : 0u;
#pragma unroll 1
          for (int k = 0; k < ksteps; ++k) {     // one K step = 32 bytes of a tile row
            // (Q and K tiles have one layout, so one high descriptor word)
            const bool last16 = !fp8 && k >= wide_ksteps;
            const uint32_t off = last16 ? kNarrowOff >> 4 : 2 * k, hi = last16 ? narrow_hi : qd_hi;
            if (fp8) mma_ss_f8(s_tmem, a_lo + off, hi, b_lo + off, hi, idesc_qk - fewer, k > 0 ? 1u : 0u);
            else     mma_ss_f16(s_tmem, a_lo + off, hi, b_lo + off, hi, idesc_qk - fewer, k > 0 ? 1u : 0u);
          }
          // mask column: start address and leading offset both move with the ring slot (the
          // zero block stays put)
          if (mask_col)
            mma_ss_f16(s_tmem, od_lo, od_hi, md_lo + slot16 - (slot16 << 16), md_hi, idesc_mask - fewer, 1u);
          if (kTcBias) {
#pragma unroll 1
            for (int k = 0; k < (narrow ? kLast : kW) / 16; ++k)   // keys 16k .. 16k + 15: box k / 4, 32 bytes per step
              mma_ss_f16(s_tmem + 16 * k, bias_lo + (k >> 2) * (kBiasTileBytes >> 5) + 2 * (k & 3), bd_hi,
                         id_lo, id_hi, idesc_bias, 1u);
          }
          tc_commit(bar_addr(c, BarIdx::s_full + b));
          if (kt == p.n_kt - 1) tc_commit(bar_addr(c, BarIdx::q_empty + qslot));
          if (kDebug && tl != nullptr && tl_n + 2 <= 2 * kDbgTimelineTiles) { tl[tl_n++] = t0; tl[tl_n++] = clock64(); }
        }
        __syncwarp();
        if (++st == nkv) { st = 0; kv_par ^= 1; }
        if (kTcBias && (s == gv - 1 || p.q_split)) {
          // every bias MMA that reads this stage is issued: the stage is free when they finish
          if (leader) tc_commit(bar_addr(c, BarIdx::bias_empty + bst));
          __syncwarp();
          if (++bst == (uint32_t)p.bias_stages) { bst = 0; b_par ^= 1; }
        }
      }
    }
    // the slots that this item does not use (where Q is not scaled, the producer's arrival on q_full came before the K/V loads that
    // were waited for above)
    if (kMixed) {
#pragma unroll 1
      for (int s = gv; s < p.n_streams; ++s) {
        const int qslot = (int)q_buf(p, icount) * kMaxStreams + s;
        if (p.scale_q) AF3K_WAIT_WARP_C(c, BarIdx::q_scaled + qslot, q_use(p, icount) & 1);
        if (leader) mbar_arrive(bar_addr(c, BarIdx::q_empty + qslot));
        __syncwarp();
      }
    }
  }
}

// O += P V for every tile, in order.
template <bool kDebug, bool kMixed, int kW, int kLast>
__device__ void pv_issuer_role(const Ctx& c) {
  const AttnParams& p = *c.p;
  const WaitBlock* wait_block = wait_block_of(c.bars);
  const bool leader = elect_one();
  const uint32_t nkv = p.kv_stages;
  const uint32_t v_layout = swizzle_layout_code(p.v_row_bytes);
  const uint32_t idesc_pv = make_idesc(1u, 1u, 0u, 1u, (uint32_t)p.nv);   // A = P and B = V, both bf16 (kind::f16 takes no mixed pair)
  const uint32_t kv_stage_bytes = p.k_tile_bytes + p.v_tile_bytes;
  const uint64_t vd0 = make_smem_desc(c.smem + p.off_kv + p.k_tile_bytes, p.v_tile_bytes,
                                      8 * p.v_row_bytes, v_layout);
  const uint32_t vd_lo = (uint32_t)vd0, vd_hi = (uint32_t)(vd0 >> 32);
  const uint32_t stage_step = kv_stage_bytes >> 4;
  const uint32_t v_kstep = (16u * p.v_row_bytes) >> 4;
  long long* tl = (kDebug && p.debug != nullptr && blockIdx.x == 0)
                      ? reinterpret_cast<long long*>(p.debug + kDbgFloats) + 2 * kDbgTimelineTiles * 8 +
                            2 * kDbgTimelineTiles
                      : nullptr;
  uint32_t tl_n = 0;
  uint32_t st = 0;
  uint32_t pready_par = 0;         // bit b: of warpgroup b's next P
  grid_wait_previous();            // (a wait's limit counts from here)
#pragma unroll 1
  for (int item = blockIdx.x; item < p.n_items; item += gridDim.x) {
    const Item it = decode_item<kMixed>(p, item);
    const int gv = it.gv;
#pragma unroll 1
    for (int kt = 0; kt < p.n_kt; ++kt) {
#pragma unroll 1
      for (int s = 0; s < gv; ++s) {
        const int b = s & 1;
        AF3K_WAIT_WARP_C(c, BarIdx::p_ready + b, (pready_par >> b) & 1u);
        pready_par ^= 1u << b;
        tc_fence_after();
        const uint32_t b_lo = vd_lo + st * stage_step;
        const uint32_t o_tmem = c.tmem + kOCol + s * p.nv;
        const uint32_t p_tmem = c.tmem + kPCol + b * 64;
        if (leader) {
          const long long t0 = kDebug && tl != nullptr ? clock64() : 0;
          mma_ts_f16(o_tmem, p_tmem, b_lo, vd_hi, idesc_pv, kt > 0 ? 1u : 0u);
#pragma unroll 1
          for (int k = 1; k < (kLast != kW && kt == p.n_kt - 1 ? kLast : kW) / 16; ++k)   // 16 keys per step: 8 TMEM columns of P
            mma_ts_f16(o_tmem, p_tmem + k * 8, b_lo + k * v_kstep, vd_hi, idesc_pv, 1u);
          tc_commit(bar_addr(c, BarIdx::pv_done + b));
          tc_commit(bar_addr(c, BarIdx::kv_empty + st));
          if (kDebug && tl != nullptr && tl_n + 2 <= 2 * kDbgTimelineTiles) { tl[tl_n++] = t0; tl[tl_n++] = clock64(); }
        }
        __syncwarp();
        if (++st == nkv) st = 0;
      }
    }
  }
}

// ------------------------------------------------------------------ softmax
__device__ __forceinline__ uint4 lds128(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "r"(addr));
  return v;
}



// x = s * scale + bias for the 64 columns [kCol0, kCol0 + 64) of the thread's row, row maximum
// updated.  xr holds the raw logits on entry and x on exit.  Masked and absent keys arrive from
// the tensor core as -2^47 and -inf and need no handling here.
template <int kCol0>
__device__ __forceinline__ void logits_half(uint32_t (&xr)[kTile], uint32_t bias_row, uint32_t row7,
                                            uint64_t scale2, float& mxa, float& mxb) {
#pragma unroll
  for (int j = kCol0 / 8; j < kCol0 / 8 + 8; ++j) {
    const uint4 bv = lds128(bias_row + (j >> 3) * (kBiasTileBytes / 2) + (((j & 7) ^ row7) << 4));
    const uint32_t w[4] = {bv.x, bv.y, bv.z, bv.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int col = j * 8 + 2 * e;
      // bf16 pair -> two fp32: low half shifted up, high half masked in place
      const uint64_t b2 = pack_f32x2(__uint_as_float(w[e] << 16), __uint_as_float(w[e] & 0xffff0000u));
      const uint64_t s2 = pack_f32x2(__uint_as_float(xr[col]), __uint_as_float(xr[col + 1]));
      float x0, x1;
      unpack_f32x2(fma_f32x2(s2, scale2, b2), x0, x1);
      xr[col] = __float_as_uint(x0);
      xr[col + 1] = __float_as_uint(x1);
      if (e & 1) mxb = max3(mxb, x0, x1); else mxa = max3(mxa, x0, x1);
    }
  }
}

// Row maximum over finished logits (bf16 q/k: the tensor core has already applied scale, bias and mask).
template <int kCol0, int kCol1, int kW>
__device__ __forceinline__ void row_max(const uint32_t (&xr)[kW], float& mxa, float& mxb) {
#pragma unroll
  for (int i = kCol0; i < kCol1; i += 4) {
    mxa = max3(mxa, __uint_as_float(xr[i]), __uint_as_float(xr[i + 1]));
    mxb = max3(mxb, __uint_as_float(xr[i + 2]), __uint_as_float(xr[i + 3]));
  }
}

// Weights are exp2(x * f + c), one fused multiply-add, with constants that go with the row's reference m: f = ef, the factor
// from logits to exponents of 2, and c = -m * ef rounded.  The rounding leaves up to 2^-24 |m * ef| in every exponent of the
// row, a factor that the division by their sum takes out again - as long as it is a number.  From |m * ef| = 2^31 on (biases
// of -1e10, masked rows) it need not be: there f is a power of two, so that x * f + c is (x - m) * f exactly, 0 for x == m.
// Other logits of that size are at least 2^31 / 2^24 of the exponent's units away and weigh nothing with either factor; half
// of ef's power of two keeps m * f finite for any finite m.
__device__ __forceinline__ void exponent_terms(float m, float ef, float& f, float& c) {
  f = fabsf(m * ef) < 2147483648.0f ? ef : 0.5f * __uint_as_float(__float_as_uint(ef) & 0x7f800000u);
  c = -m * f;
}

// O accumulator of this thread's row times alpha.
__device__ __forceinline__ void rescale_output(uint32_t o_taddr, int nv, float alpha) {
#pragma unroll 1
  for (int c0 = 0; c0 < nv; c0 += 16) {
    uint32_t o[16];
    tmem_ld_x16(o_taddr + c0, o);
    tc_wait_ld();
#pragma unroll
    for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
    tmem_st_x16(o_taddr + c0, o);
  }
}

// A softmax warp's wait, after a test that came too early (the loop is inline: a call would have to save the registers).
__device__ __forceinline__ bool softmax_wait(const Ctx& c, int idx, uint32_t parity) {
  const bool ok = mbar_wait_bounded(bar_addr(c, idx), parity, c.p->wait_limit, c.abort_flag);
  if (__all_sync(0xffffffffu, ok)) return true;
  report_timeout(c, idx);
  return false;
}

// What a softmax thread carries from tile to tile.  A stream's result is stored at the end of its warpgroup's next tile, before
// that tile's P is handed over (the next P V may write the same accumulator): its last P V has been waited for by then, which a
// warpgroup that stored it at once spent 700 - 1 400 cycles on, and as much again on the way to its next tile.  With Q scaled by these warps, the
// wider stores of P and the other changes of the hand-over, us a call on changing inputs: 768 rows 649 -> 628, 389 rows (grid module)
// 248 -> 236, 2048 fp8 rows 10 900 -> 9 845, 5 x 1536 tokens of 48 channels 97.9 -> 93.7.
struct SoftmaxState {
  float m[2], l[2];          // reference maximum and sum of its streams: [0] the stream whose turn it is, [1] the other one
  uint64_t sum_a, sum_b;     // the last tile's weights, not yet in its stream's sum
  uint32_t s_par, pv_par;    // parities of the next logits tile and of the last P V
  bool s_ready;              // the next logits tile was seen complete already
  bool started;              // there is a last P V
  bool swap;                 // the last tile's stream has another one beside it, whose turn it is now
  // A stream that has had its last key tile: its result is still in TMEM (0: none).
  uint32_t done_o;
  float done_l;
  __nv_bfloat16* done_row;   // where this thread's row goes (null: beyond the matrix)
  const __nv_bfloat16* done_gate;
  float* done_dbg;           // (debug build) its row of the dump: block 0's first stream only
};

// The last tile's weights enter its stream's sum and the turn passes to the other stream.
__device__ __forceinline__ void close_tile(SoftmaxState& st) {
  float s0, s1, s2, s3;
  unpack_f32x2(st.sum_a, s0, s1);
  unpack_f32x2(st.sum_b, s2, s3);
  st.l[0] += (s0 + s1) + (s2 + s3);
  st.done_l = st.l[0];
  if (st.swap) {
    const float m = st.m[0], l = st.l[0];
    st.m[0] = st.m[1]; st.l[0] = st.l[1];
    st.m[1] = m; st.l[1] = l;
  }
}

// O / l -> bf16 -> global for the stream that is done.
template <bool kDebug, bool kGate>
__device__ __forceinline__ void store_result(const Ctx& c, const SoftmaxState& st) {
  const AttnParams& p = *c.p;
  const float inv = __frcp_rn(st.done_l);
#pragma unroll 1
  for (int c0 = 0; c0 < p.nv; c0 += 16) {
    uint32_t o[16];
    tmem_ld_x16(st.done_o + c0, o);
    tc_wait_ld();
    if (kDebug && st.done_dbg != nullptr) {
#pragma unroll
      for (int i = 0; i < 16; ++i) st.done_dbg[kDbgO + c0 + i] = __uint_as_float(o[i]);
      st.done_dbg[kDbgML + 1] = st.done_l;
    }
    if (st.done_row != nullptr) {
#pragma unroll
      for (int hseg = 0; hseg < 2; ++hseg) {
        if (c0 + hseg * 8 + 8 <= p.D) {
          if constexpr (kGate) {
            const uint4 gv = *reinterpret_cast<const uint4*>(st.done_gate + c0 + hseg * 8);
            const uint32_t gw[4] = {gv.x, gv.y, gv.z, gv.w};
#pragma unroll
            for (int e = 0; e < 8; ++e) {
              const float g = __uint_as_float((e & 1) ? gw[e >> 1] & 0xffff0000u : gw[e >> 1] << 16);
              o[hseg * 8 + e] = __float_as_uint(__uint_as_float(o[hseg * 8 + e]) * sigmoid_f32(g));
            }
          }
          uint4 v;
          v.x = pack_bf16x2(__uint_as_float(o[hseg * 8 + 0]) * inv, __uint_as_float(o[hseg * 8 + 1]) * inv);
          v.y = pack_bf16x2(__uint_as_float(o[hseg * 8 + 2]) * inv, __uint_as_float(o[hseg * 8 + 3]) * inv);
          v.z = pack_bf16x2(__uint_as_float(o[hseg * 8 + 4]) * inv, __uint_as_float(o[hseg * 8 + 5]) * inv);
          v.w = pack_bf16x2(__uint_as_float(o[hseg * 8 + 6]) * inv, __uint_as_float(o[hseg * 8 + 7]) * inv);
          *reinterpret_cast<uint4*>(st.done_row + c0 + hseg * 8) = v;
        }
      }
    }
  }
}

// One logits tile of 128 rows and kW keys of one stream; the thread owns row `row` (TMEM lane).
// st.m[0] is the reference maximum the running sums are scaled by (it may lag the true maximum by
// up to kLazyRescaleLog2 bits), st.l[0] the running sum of the fp32 weights.
template <bool kDebug, bool kTcBias, bool kGate, int kW>
__device__ __forceinline__ bool softmax_tile(const Ctx& c, SoftmaxState& st, float* dbg, int wg, int lane,
                                             uint32_t s_taddr, uint32_t p_taddr, uint32_t o_taddr,
                                             uint32_t bias_row, uint32_t row7, float scale, bool first_kt, long long* ts) {
  if (kDebug && ts != nullptr) ts[0] = clock64();
  if (!st.s_ready && !softmax_wait(c, BarIdx::s_full + wg, st.s_par)) return false;
  st.s_par ^= 1;
  tc_fence_after();
  if (kDebug && ts != nullptr) ts[1] = clock64();
  static_assert(kW % 16 == 0 && kW >= 32 && kW <= kTile && (kTcBias || kW == kTile), "key tiles of 32 to 128 keys");
  uint32_t xr[kW];
  tmem_ld_x32(s_taddr, &xr[0]);
  // Under the load: what is left of the tile before, and a look whether its P V has finished.
  close_tile(st);
  if (first_kt) { st.m[0] = -INFINITY; st.l[0] = 0.f; }
  const bool pv_ok = mbar_test_wait(bar_addr(c, BarIdx::pv_done + wg), st.pv_par) || !st.started;
  const float m_run = st.m[0];
  float mt;
  {
    tc_wait_ld();
#pragma unroll
    for (int i = 32; i + 32 <= kW; i += 32) tmem_ld_x32(s_taddr + i, &xr[i]);
    if constexpr (kW % 32 != 0) tmem_ld_x16(s_taddr + kW - 16, &xr[kW - 16]);
    float mxa = -INFINITY, mxb = -INFINITY;
    if (kTcBias) row_max<0, 32>(xr, mxa, mxb);
    tc_wait_ld();
    // the logits are in registers: hand the S buffer back so that the next Q K^T can start
    tc_fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive(bar_addr(c, BarIdx::s_free + wg));
    if (kDebug && dbg != nullptr) {
#pragma unroll
      for (int i = 0; i < kW; ++i) dbg[kDbgS + i] = __uint_as_float(xr[i]);
    }
    if constexpr (kTcBias) {
      row_max<32, kW>(xr, mxa, mxb);
    } else {
      const uint64_t scale2 = pack_f32x2(scale, scale);
      logits_half<0>(xr, bias_row, row7, scale2, mxa, mxb);
      logits_half<64>(xr, bias_row, row7, scale2, mxa, mxb);
    }
    mt = fmaxf(mxa, mxb);
  }
  if (kDebug && ts != nullptr) ts[2] = clock64() + (long long)(mt == 123.456f);   // logits and row maximum in registers
  // factor between a logit difference and the exponent of 2: log2(e), times the logit scale when
  // the tensor core's logits still lack it (fp8 q/k with tensor-core bias: `scale` carries it)
  const float ef = kTcBias ? scale : kLog2e;
  // (m_run is -inf in front of the first key tile)
  const bool grown = (mt - m_run) * ef > kLazyRescaleLog2;
  const float m_use = first_kt || grown ? mt : m_run;
  const bool need = grown && !first_kt;
  float f = ef, nml = 0.f;
  if (kTcBias) exponent_terms(m_use, ef, f, nml);
  // The P buffer and the O accumulators are this warpgroup's again when its last P V has finished.  Waited for in front of
  // the pass, because a branch within it drains the exponentials in flight.
  if (!__all_sync(0xffffffffu, pv_ok) && !softmax_wait(c, BarIdx::pv_done + wg, st.pv_par)) return false;
  st.pv_par ^= st.started ? 1u : 0u;
  st.started = true;
  tc_fence_after();
  if (kDebug && ts != nullptr) ts[3] = clock64();   // last P V awaited, exponential pass starts
  // p = exp2((x - m) * log2e).  fp8 path: the subtraction comes first so that x == m gives
  // exactly 0 even for the huge negative values of masked keys (a row with no attended key: all
  // weights 1).  bf16 path: one fused multiply-add (exponent_terms).
  // The pass is one ex2 per logit on the XU (a warp-wide ex2 every 8 cycles per scheduler, shared
  // by the scheduler's two softmax warps) with one packed FMA, one packed add and one bf16 pack per
  // pair of logits around it.  Two warps alone on a scheduler take 2 230 cycles for a tile each, 2 048 of them the XU's; the kernel
  // takes 2 590 with fp8 and 2 950 - 2 990 with bf16, for what a warp runs between two passes: some 110 instructions in one chain, six cycles each.  (Tried
  // and slower: the maximum searched along with the pass and the pass repeated where a row has grown, 768 rows 636 -> 690 us, for the
  // logits that stay live; the wait for P and O after one or two column groups, 2048 fp8 rows 10 300 -> 11 700.)
  const uint64_t l2e2 = pack_f32x2(f, f);
  const uint64_t nm2 = pack_f32x2(-m_use, -m_use);
  const uint64_t nml2 = pack_f32x2(nml, nml);
  uint64_t suma = pack_f32x2(0.f, 0.f), sumb = suma;
  uint32_t pk[kW / 2];           // P as bf16, two keys per 32-bit TMEM column: the A operand of the second GEMM
#pragma unroll
  for (int i = 0; i < kW / 2; ++i) {
    float y0, y1;
    const uint64_t x2 = pack_f32x2(__uint_as_float(xr[2 * i]), __uint_as_float(xr[2 * i + 1]));
    if (kTcBias) unpack_f32x2(fma_f32x2(x2, l2e2, nml2), y0, y1);
    else         unpack_f32x2(mul_f32x2(add_f32x2(x2, nm2), l2e2), y0, y1);
    const float p0 = ex2_approx(y0);
    const float p1 = ex2_approx(y1);
    // (two chains: one takes 9 % longer, 2048 fp8 rows 9 970 -> 10 840 us, four 1 %)
    if (i & 1) sumb = add_f32x2(sumb, pack_f32x2(p0, p1));
    else       suma = add_f32x2(suma, pack_f32x2(p0, p1));
    pk[i] = pack_bf16x2(p0, p1);
    // Few and wide stores: 2048 fp8 rows, eight of 8 columns 10 370 us, four of 16 10 050, 32 and twice 16 9 900, two of 32 10 040.
    constexpr int kWide = kW >= 80 ? 32 : 16;          // columns of the first store; 16 after that, 8 at the end of an odd multiple
    if (i + 1 == kWide) {
      if constexpr (kWide == 32) tmem_st_x32(p_taddr, pk); else tmem_st_x16(p_taddr, pk);
    } else if (i + 1 > kWide && (i + 1 - kWide) % 16 == 0) {
      tmem_st_x16(p_taddr + i - 15, pk + i - 15);
    } else if (i + 1 == kW / 2) {
      tmem_st_x8(p_taddr + i - 7, pk + i - 7);
    }
  }
  if (kDebug && dbg != nullptr) {
#pragma unroll
    for (int i = 0; i < kW / 2; ++i) dbg[kDbgP + i] = __uint_as_float(pk[i]);
  }
  if (kDebug && ts != nullptr) ts[6] = clock64();     // last exponential issued
  // What else has to be done with the accumulators before the next P V may write one.
  if (__any_sync(0xffffffffu, need)) {
    float alpha = 1.0f;
    if (need) {
      if (kTcBias) {
        // what a key at the old reference weighs under the new one, over what it was counted with
        float f_run, nml_run;
        exponent_terms(m_run, ef, f_run, nml_run);
        alpha = ex2_approx(__fmaf_rn(m_run, f, nml) - __fmaf_rn(m_run, f_run, nml_run));
      } else {
        alpha = ex2_approx((m_run - mt) * ef);
      }
    }
    st.l[0] *= alpha;
    rescale_output(o_taddr, c.p->nv, alpha);
  }
  if (st.done_o != 0) {
    store_result<kDebug, kGate>(c, st);
    st.done_o = 0;
  }
  st.m[0] = m_use;
  st.sum_a = suma;
  st.sum_b = sumb;
  // The next tile's logits are normally finished by now: ask while the P stores drain, so that the
  // barrier's round trip is not paid between two tiles.
  st.s_ready = __all_sync(0xffffffffu, mbar_test_wait(bar_addr(c, BarIdx::s_full + wg), st.s_par));
  tc_wait_st();
  tc_fence_before();
  __syncwarp();
  if (lane == 0) mbar_arrive(bar_addr(c, BarIdx::p_ready + wg));
  if (kDebug && ts != nullptr) ts[4] = clock64();   // P handed over
  return true;
}

// (bf16 q/k) A softmax warp scales its quarter of its warpgroup's Q tiles of the CTA's j-th item.  Eight warps do in 300 cycles
// what took a single-warp role several thousand, and 12 instructions a tile are little beside the softmax's own 450: 768 rows
// 617 us (kernel alone, as it then was), with the P V issuer scaling 616 - 666, with the mask writer 641 - 676, with q scaled by its producer 596.
template <bool kMixed>
__device__ __forceinline__ bool scale_own_q(const Ctx& c, int item, uint32_t j, int wg, int wq, int lane) {
  const AttnParams& p = *c.p;
  const Item it = decode_item<kMixed>(p, item);
  const uint32_t buf = q_buf(p, j), par = q_use(p, j) & 1, bytes = p.q_tile_bytes >> 2;
#pragma unroll 1
  for (int s = wg; s < (kMixed ? p.n_streams : it.gv); s += 2) {
    const int slot = (int)buf * kMaxStreams + s;
    if (!softmax_wait(c, BarIdx::q_full + slot, par)) return false;
    // (nothing is in a slot that the item does not use: an arrival only)
    scale_q(c.smem + p.off_q + (buf * p.n_streams + s) * p.q_tile_bytes + wq * bytes, kMixed && s >= it.gv ? 0u : bytes, p.scale, lane,
            bar_addr(c, BarIdx::q_scaled + slot));
  }
  return true;
}

template <bool kDebug, bool kTcBias, bool kGate, bool kMixed, bool kScalesQ, int kW, int kLast>
__device__ void softmax_role(const Ctx& c, int wg, int wq, int lane) {
  const AttnParams& p = *c.p;
  const int row = wq * 32 + lane;                    // row of the 128-query tile == TMEM lane
  const uint32_t lane_sel = (uint32_t)(wq * 32) << 16;
  const uint32_t s_taddr = c.tmem + lane_sel + kSCol + wg * kTile;
  const uint32_t p_taddr = c.tmem + lane_sel + kPCol + wg * 64;
  SoftmaxState st;
  st.m[0] = st.m[1] = -INFINITY;
  st.l[0] = st.l[1] = 0.f;
  st.sum_a = st.sum_b = 0;
  st.s_par = st.pv_par = 0;
  st.s_ready = st.started = st.swap = false;
  st.done_o = 0;
  st.done_gate = nullptr;
  st.done_dbg = nullptr;
  uint32_t bst = 0, b_par = 0;                       // (fp8 without tensor-core bias) bias ring
  uint32_t n_tiles = 0;                              // (debug build)
  // The next item's Q tiles are scaled behind the last key tile but one (with a single Q buffer they come later), the first item's here.
  const bool scales = kScalesQ && p.scale_q;
  const int scale_kt = !scales ? -1 : (p.q_buffers == 2 ? max(p.n_kt - 2, 0) : p.n_kt - 1);
  uint32_t icount = 0;
  grid_wait_previous();
  if (scales && (int)blockIdx.x < p.n_items && !scale_own_q<kMixed>(c, blockIdx.x, 0, wg, wq, lane)) return;

#pragma unroll 1
  for (int item = blockIdx.x; item < p.n_items; item += gridDim.x, ++icount) {
    const Item it = decode_item<kMixed>(p, item);
    // fp32 path: the logit scale the softmax threads apply themselves.  Tensor-core path: the
    // factor from logit differences to exponents of 2 (the scale is in Q already for bf16 q/k)
    float scale = p.scale;
    if (p.q_scale != nullptr) scale *= p.q_scale[it.h] * p.k_scale[it.h];
    if (kTcBias) scale = (p.scale_q ? 1.0f : scale) * kLog2e;

    // A narrower last tile is taken behind the loop, so that the loop's code is as without: with the choice inside it, or inside the tile,
    // 389 rows took longer than with four tiles of 128 (module call 216 us; inside 222 - 229, here 206).
#pragma unroll 1
    for (int kt = 0; kt < p.n_kt - (kLast != kW); ++kt) {
      // fp8 q/k: this thread adds the bias itself, from its row of the staged tile
      if (!kTcBias) AF3K_WAIT_WARP(c, BarIdx::bias_full + bst, b_par);
      const uint32_t bias_row = c.smem + p.off_bias + bst * kBiasTileBytes + row * 128;

#pragma unroll 1
      for (int s = wg; s < it.gv; s += 2) {
        // diagnostic timeline (debug build only): SM clock at the phase boundaries of every tile
        // this warp processes, 8 slots per tile, behind the tile dump
        long long* ts = nullptr;
        float* dbg = nullptr;
        if (kDebug && p.debug != nullptr && blockIdx.x == 0) {
          if (wq == 0 && lane == 0 && n_tiles < kDbgTimelineTiles)
            ts = reinterpret_cast<long long*>(p.debug + kDbgFloats) + ((size_t)wg * kDbgTimelineTiles + n_tiles) * 8;
          if (item == 0 && s == 0 && kt == 0) dbg = p.debug + (size_t)row * kTile;
          ++n_tiles;
        }
        if (!softmax_tile<kDebug, kTcBias, kGate, kW>(c, st, dbg, wg, lane, s_taddr, p_taddr, c.tmem + lane_sel + kOCol + s * p.nv, bias_row, row & 7, scale,
                                                  kt == 0, ts))
          return;
        st.swap = it.gv > wg + 2;
        if (kLast == kW && kt == p.n_kt - 1) {
          const int qrow = stream_qt(p, it, s) * kTile + row;
          st.done_o = c.tmem + lane_sel + kOCol + s * p.nv;
          st.done_row = qrow < p.Sq ? p.out + (long long)stream_row(p, it, s) * p.out_stride_b1 + (long long)it.h * p.out_stride_b2 +
                                          (long long)qrow * p.out_stride_s
                                    : nullptr;
          if (kDebug) st.done_dbg = p.debug != nullptr && item == 0 && s == 0 ? p.debug + (size_t)row * kTile : nullptr;
          if constexpr (kGate)
            st.done_gate = p.gate + (long long)stream_row(p, it, s) * p.gate_stride_b1 + (long long)it.h * p.gate_stride_b2 +
                           (long long)qrow * p.gate_stride_s;
        }
      }
      if (!kTcBias) {
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_addr(c, BarIdx::bias_empty + bst));
        if (++bst == (uint32_t)p.bias_stages) { bst = 0; b_par ^= 1; }
      }
      if (kScalesQ && kt == scale_kt && item + (int)gridDim.x < p.n_items &&
          !scale_own_q<kMixed>(c, item + gridDim.x, icount + 1, wg, wq, lane))
        return;
    }
    if constexpr (kLast != kW) {
#pragma unroll 1
      for (int s = wg; s < it.gv; s += 2) {
        if (!softmax_tile<kDebug, kTcBias, kGate, kLast>(c, st, nullptr, wg, lane, s_taddr, p_taddr, c.tmem + lane_sel + kOCol + s * p.nv, 0, 0, scale, false,
                                                     nullptr))
          return;
        st.swap = it.gv > wg + 2;
        const int qrow = stream_qt(p, it, s) * kTile + row;
        st.done_o = c.tmem + lane_sel + kOCol + s * p.nv;
        st.done_row = qrow < p.Sq ? p.out + (long long)stream_row(p, it, s) * p.out_stride_b1 + (long long)it.h * p.out_stride_b2 +
                                        (long long)qrow * p.out_stride_s
                                  : nullptr;
        if (kDebug) st.done_dbg = p.debug != nullptr && item == 0 && s == 0 ? p.debug + (size_t)row * kTile : nullptr;
        if constexpr (kGate)
          st.done_gate = p.gate + (long long)stream_row(p, it, s) * p.gate_stride_b1 + (long long)it.h * p.gate_stride_b2 +
                         (long long)qrow * p.gate_stride_s;
      }
      if (kScalesQ && scale_kt == p.n_kt - 1 && item + (int)gridDim.x < p.n_items &&
          !scale_own_q<kMixed>(c, item + gridDim.x, icount + 1, wg, wq, lane))
        return;
    }
  }
  // the last stream's result
  if (st.done_o != 0) {
    close_tile(st);
    AF3K_WAIT_WARP(c, BarIdx::pv_done + wg, st.pv_par);
    tc_fence_after();
    store_result<kDebug, kGate>(c, st);
  }
}

// ------------------------------------------------------------------ bias converted in the kernel
// Two keys' bias in bf16.  What bf16 cannot hold (fp32's lowest value, a quotient, an infinity) becomes its largest value of
// that sign: the tensor core adds a slice of the bias by products with 1 and 0, and an infinity times 0 would make NaN of the 15
// keys beside it.  NaN stays.
__device__ __forceinline__ uint32_t staged_pair(float a, float b) {
  uint32_t w = pack_bf16x2(a, b);
  asm("max.NaN.bf16x2 %0, %0, %1;" : "+r"(w) : "r"(0xff7fff7fu));
  asm("min.NaN.bf16x2 %0, %0, %1;" : "+r"(w) : "r"(0x7f7f7f7fu));
  return w;
}

// The same for two that are bf16 already.
__device__ __forceinline__ uint32_t clamped_pair(uint32_t w) {
  asm("max.NaN.bf16x2 %0, %0, %1;" : "+r"(w) : "r"(0xff7fff7fu));
  asm("min.NaN.bf16x2 %0, %0, %1;" : "+r"(w) : "r"(0x7f7f7f7fu));
  return w;
}

constexpr int kConvertWarps = 8, kConvertRows = 8;   // each warp makes 16 rows of a tile (two rounds of loads)

// One row's keys 4 lane .. 4 lane + 3 into a staged tile: two boxes of 64 keys, rows of 128 bytes, 128-byte swizzle.
__device__ __forceinline__ void store_bias4(uint32_t tile, int row, int lane, uint32_t w0, uint32_t w1) {
  const uint32_t at = tile + row * 128 + (lane >> 4) * (kBiasTileBytes / 2) + (lane & 1) * 8 + ((((lane >> 1) & 7) ^ (row & 7)) << 4);
  asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(at), "r"(w0), "r"(w1) : "memory");
}

// kConvert: eight warps in place of the second softmax warpgroup, which has no stream in items of one, make the bias tiles, from fp32 or
// from bf16 rows that TMA cannot address, in place of the producer's loads.  Otherwise such a call takes a launch more, and for a
// short call that is a good part of it.  us, converted here / in a pass before, 16 heads, fp32 on vectors: 100 tokens 4.7 / 6.3, 512 9.3 / 12.9,
// 1152 20.4 / 33.2 (512 in place 8.2).  A warp takes 16 rows of a tile, a lane four keys of each.  What does
// not exist takes the bias of a row or key that does, or anything: of such rows nothing is stored, such keys are at -inf.
//
// Rows that start on vectors (bias_wide): 8 rows' loads for the next tile follow directly on their store for this one, so that
// 16 rows' are out nearly all the time.  Two such warps share a scheduler with a softmax warp that streams through its code, so the
// loop is kept short: with a test for infinities and a second pass behind it 512 tokens took 11.4 us.
template <bool kF32, int kW>
__device__ void bias_convert_role(const Ctx& c, int cw, int lane) {
  const AttnParams& p = *c.p;
  constexpr int es = kF32 ? 4 : 2;
  using Vec = typename std::conditional<kF32, float4, uint2>::type;
  const int row0 = cw * 2 * kConvertRows;
  const long long step = p.bias_stride_r * es;
  Vec x[2][kConvertRows];
  auto load = [&](const Item& it, int kt, int half) {
    const int first = it.qt * kTile + row0, last = min(2 * kConvertRows - 1, p.Sq - 1 - first);
    if (last < 0) return;
    const char* src = static_cast<const char*>(p.bias_src) + (it.h * p.bias_stride_h + first * p.bias_stride_r + min(kt * kW + 4 * lane, p.Sk - 4)) * es;
#pragma unroll
    for (int r = 0; r < kConvertRows; ++r) x[half][r] = *reinterpret_cast<const Vec*>(src + min(half * kConvertRows + r, last) * step);
  };
  auto store = [&](uint32_t tile, int half) {
#pragma unroll
    for (int r = 0; r < kConvertRows; ++r) {
      uint32_t w0, w1;
      if constexpr (kF32) {
        w0 = staged_pair(x[half][r].x, x[half][r].y);
        w1 = staged_pair(x[half][r].z, x[half][r].w);
      } else {
        w0 = staged_pair(__uint_as_float(x[half][r].x << 16), __uint_as_float(x[half][r].x & 0xffff0000u));
        w1 = staged_pair(__uint_as_float(x[half][r].y << 16), __uint_as_float(x[half][r].y & 0xffff0000u));
      }
      store_bias4(tile, row0 + half * kConvertRows + r, lane, w0, w1);
    }
  };
  int item = blockIdx.x, kt = 0;
  Item it = decode_item<false>(p, item);     // (the grid has no more blocks than items)
  grid_wait_previous();
#pragma unroll
  for (int half = 0; half < 2; ++half) load(it, 0, half);
#pragma unroll 1
  for (uint32_t bst = 0, lap = 0; item < p.n_items;) {
    const uint32_t tile = c.smem + p.off_bias + bst * kBiasTileBytes;
    // the bias MMAs of the stage's tile before must have finished
    if (lap != 0) AF3K_WAIT_WARP(c, BarIdx::bias_empty + bst, (lap - 1) & 1);
    if (++kt == p.n_kt) {                    // the tile after this one
      kt = 0;
      item += gridDim.x;
      if (item < p.n_items) it = decode_item<false>(p, item);
    }
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      store(tile, half);
      if (item < p.n_items) load(it, kt, half);
    }
    fence_proxy_async_smem();    // make the generic-proxy stores visible to the tensor core
    __syncwarp();
    if (lane == 0) mbar_arrive(bar_addr(c, BarIdx::bias_full + bst));
    if (++bst == (uint32_t)p.bias_stages) { bst = 0; ++lap; }
  }
}

// Rows that start anywhere: a lane takes keys 32 apart, element by element, so that a warp's loads are whole pieces of the row
// wherever it starts; a row is requested again, for the next tile, as soon as it has been stored, so that a whole tile is under way.
// Keys that do not exist get 0.  The fetch of instructions is what this kernel is short of, so the code is kept short.  Tried for 1001
// tokens, us a tile (in place 1.4): aligned vectors of four elements stored in pieces that depend on where the row starts 8, put
// together by shuffles 3.9, the same with eight warps 2.5, copied through shared memory in a rolled loop 3.3 - 3.9; this 2.2.
// us, 16 heads, here / pass before: 129 tokens 6.7 / 7.2, 389 bf16 10.6 / 12.1, 1001 fp32 22.7 / 28.4.
template <bool kF32, int kW>
__device__ void bias_convert_ragged_role(const Ctx& c, int cw, int lane) {
  const AttnParams& p = *c.p;
  using T = typename std::conditional<kF32, float, uint16_t>::type;
  constexpr int kRows = 2 * kConvertRows;
  const int row0 = cw * kRows;
  T x[kRows][4];
  struct Rows { const T* src; int last; };      // of this warp in an item, from this lane's first key on
  auto rows_of = [&](const Item& it) {
    const int first = it.qt * kTile + row0, last = min(kRows - 1, p.Sq - 1 - first);
    return Rows{static_cast<const T*>(p.bias_src) + it.h * p.bias_stride_h + (last >= 0 ? first : p.Sq - 1) * p.bias_stride_r + lane, max(last, 0)};
  };
  auto load_row = [&](const Rows& w, int kt, int r) {
    const T* src = w.src + min(r, w.last) * p.bias_stride_r + kt * kW;
    const int n = p.Sk - kt * kW - lane;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      x[r][j] = T(0);
      if (32 * j < kW && n > 32 * j) x[r][j] = src[32 * j];
    }
  };
  auto clamped = [&](T a, T b) {
    if constexpr (kF32) return staged_pair(a, b); else return clamped_pair((uint32_t)a | (uint32_t)b << 16);
  };
  auto write = [&](uint32_t addr, uint32_t w) { asm volatile("st.shared.u16 [%0], %1;" ::"r"(addr), "h"((uint16_t)w) : "memory"); };
  int item = blockIdx.x, kt = 0;
  Rows w = rows_of(decode_item<false>(p, item));     // (the grid has no more blocks than items)
  grid_wait_previous();
#pragma unroll
  for (int r = 0; r < kRows; ++r) load_row(w, 0, r);
#pragma unroll 1
  for (uint32_t bst = 0, lap = 0; item < p.n_items;) {
    const uint32_t tile = c.smem + p.off_bias + bst * kBiasTileBytes + row0 * 128 + (lane & 7) * 2;
    // the bias MMAs of the stage's tile before must have finished
    if (lap != 0) AF3K_WAIT_WARP(c, BarIdx::bias_empty + bst, (lap - 1) & 1);
    if (++kt == p.n_kt) {                    // the tile after this one
      kt = 0;
      item += gridDim.x;
      if (item < p.n_items) w = rows_of(decode_item<false>(p, item));
    }
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
      const uint32_t to = tile + r * 128 + (((lane >> 3) ^ (r & 7)) << 4);
      const uint32_t w0 = clamped(x[r][0], x[r][1]);
      write(to, w0);
      write(to ^ 64u, w0 >> 16);
      if (kW > 64) {
        const uint32_t w1 = clamped(x[r][2], x[r][3]);
        write(to + kBiasTileBytes / 2, w1);
        if (kW > 96) write((to ^ 64u) + kBiasTileBytes / 2, w1 >> 16);
      }
      if (item < p.n_items) load_row(w, kt, r);
    }
    fence_proxy_async_smem();    // make the generic-proxy stores visible to the tensor core
    __syncwarp();
    if (lane == 0) mbar_arrive(bar_addr(c, BarIdx::bias_full + bst));
    if (++bst == (uint32_t)p.bias_stages) { bst = 0; ++lap; }
  }
}

// ------------------------------------------------------------------ kernel
// kGate: the result is multiplied by sigmoid(gate).  A template argument, because a run-time test of the pointer
// cost calls without a gate 0.9 % (768 rows of 768 keys: 671 -> 677 us).
// kFp8 likewise, and for the same reason no debug stamps, divisions, second copies of a waiting loop or of a loop body
// are left in the production kernel (389 rows 261 -> 253.5 us a module call, 256 rows of 64 channels 58.2 -> 57.5; 768 rows
// and 1536 tokens unchanged).  The roles' loops come from the SM's instruction cache, 440 requests and 10 misses a logits
// tile, which is what it was with more code as well; four copies of the softmax tile beside them took 43 misses and 192 -> 222 us
// on 192 rows of 768.
// kMixed: some items have fewer streams than the others (smaller ones behind the last full round, rows or pairs of query
// tiles that leave a remainder), which takes slots and barriers that an item does not use through their phases and two sets
// of constants to decode an item.  A plan of equal items runs without: 768 rows 645 -> 636 us.
// kConvert: plans of one stream per item, bf16 q and k; see bias_convert_role.
// kW: keys per key tile, 32 to 128, kLast: of the last one, where it is narrower (chosen by key_widths in the C API).
template <bool kDebug, bool kTcBias, bool kFp8, bool kGate, bool kMixed, bool kConvert = false, int kW = kTile, int kLast = kW>
__global__ void __launch_bounds__(kConvert ? kConvertThreads : kThreads, 1)
attention_kernel(const __grid_constant__ AttnParams p, const __grid_constant__ CUtensorMap tm_q,
                 const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v,
                 const __grid_constant__ CUtensorMap tm_bias, const __grid_constant__ CUtensorMap tm_q2,
                 const __grid_constant__ CUtensorMap tm_k2) {
  static_assert(!kConvert || (kTcBias && !kFp8 && !kMixed), "the bias is converted for bf16 q and k and equal items only");
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  __shared__ uint32_t tmem_base_slot;
  __shared__ int abort_flag;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;

  Ctx c;
  c.p = &p;
  c.smem = smem_u32(smem_raw);
  c.bars = c.smem + p.off_bar;
  c.abort_flag = &abort_flag;

  if (threadIdx.x == 0) {
    abort_flag = 0;
    *const_cast<WaitBlock*>(wait_block_of(c.bars)) = WaitBlock{p.wait_limit, p.status, &abort_flag};
    prefetch_tensormap(&tm_q);
    prefetch_tensormap(&tm_k);
    prefetch_tensormap(&tm_v);
    if (!kConvert) prefetch_tensormap(&tm_bias);
    for (int i = 0; i < 2 * kMaxStreams; ++i) {
      mbar_init(bar_addr(c, BarIdx::q_full + i), 1);
      mbar_init(bar_addr(c, BarIdx::q_empty + i), 1);
      mbar_init(bar_addr(c, BarIdx::q_scaled + i), 4);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(bar_addr(c, BarIdx::pv_done + i), 1);
      mbar_init(bar_addr(c, BarIdx::s_full + i), 1);
      mbar_init(bar_addr(c, BarIdx::s_free + i), 4);
      mbar_init(bar_addr(c, BarIdx::p_ready + i), 4);
    }
    for (int i = 0; i < kMaxBiasStages; ++i) {
      mbar_init(bar_addr(c, BarIdx::bias_full + i), kConvert ? kConvertWarps : 1);
      // freed by the bias MMAs' completion (bf16 q/k) or by the eight softmax warps (fp8 q/k)
      mbar_init(bar_addr(c, BarIdx::bias_empty + i), kTcBias ? 1 : 8);
    }
    for (int i = 0; i < kMaxKvStages; ++i) {
      mbar_init(bar_addr(c, BarIdx::kv_full + i), p.mask_col ? 2 : 1);
      mbar_init(bar_addr(c, BarIdx::kv_empty + i), 1);
    }
    fence_barrier_init();
  }
  if (warp == 2) {
    tmem_alloc(smem_u32(&tmem_base_slot), kTmemCols);
    tmem_relinquish();
  }
  if (warp == 3) {
    // ones column, mask-column ring, zero block and identity are contiguous: clear them, then set
    // element (row, 0) of the ones operand and the identity's diagonal to bf16 1.0
    const uint32_t base = c.smem + p.off_ones;
    const uint32_t bytes = p.off_ident + kIdentBytes - p.off_ones;
    for (uint32_t o = lane * 16; o < bytes; o += 32 * 16)
      asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};" ::"r"(base + o), "r"(0u) : "memory");
    __syncwarp();
    for (int r = lane; r < kTile; r += 32)
      asm volatile("st.shared.u16 [%0], %1;" ::"r"(base + r * 16), "h"((uint16_t)0x3F80) : "memory");
    // identity element (i, i): 8-row group i / 8 (128 bytes apart), 8-key half i / 8 (256 bytes
    // apart), row i % 8 (16 bytes), key i % 8 (2 bytes)
    if (lane < 16)
      asm volatile("st.shared.u16 [%0], %1;" ::"r"(c.smem + p.off_ident + (lane >> 3) * 384 + (lane & 7) * 18),
                   "h"((uint16_t)0x3F80) : "memory");
    fence_proxy_async_smem();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  c.tmem = tmem_base_slot;

  if (warp < 4) {
    // warps 0-3 need few registers; the two softmax warpgroups take what they give up
    setmaxnreg_dec<kRegsMisc>();
    if (warp == 0) {
      if (lane == 0) producer_role<kMixed, kConvert, kW, kLast>(c, &tm_q, &tm_k, &tm_v, &tm_bias, &tm_q2, &tm_k2);
    } else if (warp == 1) {
      qk_issuer_role<kDebug, kTcBias, kFp8, kMixed, kW, kLast>(c);
    } else if (warp == 2) {
      pv_issuer_role<kDebug, kMixed, kW, kLast>(c);
    } else if (warp == 3) {
      if (p.mask_col) mask_writer_role<kMixed, kW>(c, lane);
    }
  } else if (kConvert && warp >= 8) {
    if constexpr (kConvert) {
      setmaxnreg_dec<kRegsConvert>();
      if (p.bias_wide) {
        if (p.bias_f32) bias_convert_role<true, kW>(c, warp - 8, lane);
        else            bias_convert_role<false, kW>(c, warp - 8, lane);
      } else {
        if (p.bias_f32) bias_convert_ragged_role<true, kW>(c, warp - 8, lane);
        else            bias_convert_ragged_role<false, kW>(c, warp - 8, lane);
      }
    }
  } else {
    setmaxnreg_inc<kRegsSoftmax>();
    softmax_role<kDebug, kTcBias, kGate, kMixed, !kFp8, kW, kLast>(c, (warp - 4) >> 2, warp & 3, lane);
  }

  tc_fence_before();
  __syncthreads();
  if (abort_flag != 0) {
    // a wait ran out: give loads and MMAs still in flight time to land before smem / TMEM go away
    for (int i = 0; i < 200; ++i) __nanosleep(10000);
    __syncthreads();
  }
  if (warp == 2) {
    tc_fence_after();
    tmem_dealloc(c.tmem, kTmemCols);
  }
}

// ------------------------------------------------------------------ operands and results of fp32 callers
// Up to three arrays fp32 -> bf16 (or one bf16 -> fp32) in one launch, a slice of the grid each, eight elements a thread and step.
// Short calls are bound by their launches: with torch's conversions, one kernel for each operand and none of them started under
// the one before, 16 heads of 300 tokens in fp32 took
// 32.4 us a call (16.2 on the device), so 15.1 (10.8); the single block of 512 fp32 tokens 31.1 -> 20.9.
constexpr int kCastThreads = 256, kMaxCasts = 3;
struct CastParams {
  const void* src[kMaxCasts];
  void* dst[kMaxCasts];
  long long n[kMaxCasts];        // elements
};
template <bool kToBf16>
__global__ void __launch_bounds__(kCastThreads) cast_kernel(const __grid_constant__ CastParams p) {
  const int a = blockIdx.y;
  const float* f32 = static_cast<const float*>(kToBf16 ? p.src[a] : p.dst[a]);
  const __nv_bfloat16* bf16 = static_cast<const __nv_bfloat16*>(kToBf16 ? p.dst[a] : p.src[a]);
  const long long n = p.n[a], whole = n / 8, step = (long long)gridDim.x * kCastThreads;
  grid_wait_previous();
  grid_release_next();
  for (long long i = (long long)blockIdx.x * kCastThreads + threadIdx.x; i <= whole; i += step) {
    if (i == whole) {            // the last few
      for (long long e = 8 * whole; e < n; ++e) {
        if constexpr (kToBf16) const_cast<__nv_bfloat16*>(bf16)[e] = __float2bfloat16_rn(f32[e]);
        else                   const_cast<float*>(f32)[e] = __bfloat162float(bf16[e]);
      }
      return;
    }
    if constexpr (kToBf16) {
      const float4 x = reinterpret_cast<const float4*>(f32)[2 * i], y = reinterpret_cast<const float4*>(f32)[2 * i + 1];
      const_cast<uint4*>(reinterpret_cast<const uint4*>(bf16))[i] = make_uint4(pack_bf16x2(x.x, x.y), pack_bf16x2(x.z, x.w), pack_bf16x2(y.x, y.y), pack_bf16x2(y.z, y.w));
    } else {
      const uint4 w = reinterpret_cast<const uint4*>(bf16)[i];
      float4* d = const_cast<float4*>(reinterpret_cast<const float4*>(f32)) + 2 * i;
      d[0] = make_float4(__uint_as_float(w.x << 16), __uint_as_float(w.x & 0xffff0000u), __uint_as_float(w.y << 16), __uint_as_float(w.y & 0xffff0000u));
      d[1] = make_float4(__uint_as_float(w.z << 16), __uint_as_float(w.z & 0xffff0000u), __uint_as_float(w.w << 16), __uint_as_float(w.w & 0xffff0000u));
    }
  }
}

// ------------------------------------------------------------------ bias staging pre-pass
// bias (fp32 or bf16, arbitrary row pitch) -> bf16 [B2, Sq, pitch] with a TMA-legal pitch.
// With fp8 q/k (q_scale / k_scale given) every value is divided by the head's logit scale
// softmax_scale * q_scale[h] * k_scale[h]: the tensor core then adds it to the raw fp8 products
// and the softmax threads apply that scale to the sum.
// (staged_pair says what becomes of values that bf16 cannot hold.)
// One thread converts eight columns, two 16-byte loads where every row starts on a 16-byte boundary (else one by one) and one
// 16-byte store, as many blocks as stay resident: it is bound by memory, and a call that converts pays it in full.  fp32 rows that
// start anywhere (kPieces): a warp converts 256 columns of a row, a lane two next to one another in every 64, so that its loads are
// whole pieces of the row and its stores whole lines (a thread's eight columns one by one touch every sector eight times).
// Two columns a thread, with two 64-bit divisions for each pair, against eight, us: 16 heads of 512 x 512 fp32 11.3 -> 4.9 (5.2
// TB/s), of 1536 x 1536 76.2 -> 35.2 (6.4 TB/s), 4 heads of 768 x 768 6.9 -> 3.0, of 2048 x 2048 bf16 with scales 40.9 -> 14.0.
// Rows anywhere, eight columns one by one -> two in 64, 16 heads: fp32 389 tokens 4.4 -> 3.5, 1001 19.8 -> 13.4, 1537 43.1 -> 36.5, 2047 76.1
// -> 62.4; but bf16 389 3.2 -> 3.8, 1301 23.1 -> 25.0, so that stays as it was.
constexpr int kBiasThreads = 256;
template <typename T, bool kPieces>
__global__ void __launch_bounds__(kBiasThreads, 8)
bias_to_bf16_kernel(const T* src, __nv_bfloat16* dst, int B2, int Sq, int Sk, long long src_stride_h, long long src_stride_r, int pitch,
                    const float* q_scale, const float* k_scale, float softmax_scale) {
  // (no __restrict__: it would allow loads of the read-only kind, which need not stay behind the wait)
  grid_wait_previous();
  grid_release_next();
  // a thread's eight columns, or a warp's 256
  constexpr int kColumns = kPieces ? 256 : 8;
  const uint32_t chunks = (uint32_t)(pitch + kColumns - 1) / kColumns;
  const long long total = (long long)B2 * Sq * chunks;
  const int lane = threadIdx.x & 31, threads = kPieces ? kBiasThreads / 32 : kBiasThreads;
  const bool wide = ((reinterpret_cast<uintptr_t>(src) | (uintptr_t)(src_stride_h * sizeof(T)) | (uintptr_t)(src_stride_r * sizeof(T))) & 15u) == 0;
  for (long long i = (long long)blockIdx.x * threads + (kPieces ? threadIdx.x >> 5 : threadIdx.x); i < total; i += (long long)gridDim.x * threads) {
    long long t;             // row among all heads'
    if (total <= 0x7fffffff) t = (uint32_t)i / chunks; else t = i / chunks;
    const int col = (int)(i - t * chunks) * kColumns;
    int h, r;
    if (t <= 0x7fffffff) { h = (int)((uint32_t)t / (uint32_t)Sq); r = (int)((uint32_t)t % (uint32_t)Sq); }
    else                 { h = (int)(t / Sq); r = (int)(t % Sq); }
    const T* s = src + h * src_stride_h + r * src_stride_r + col;
    const float mul = q_scale != nullptr ? 1.0f / (softmax_scale * q_scale[h] * k_scale[h]) : 1.0f;
    float x[8];
    if constexpr (kPieces) {
      const int left = Sk - col - 2 * lane;
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const int at = (e >> 1) * 64 + (e & 1);
        x[e] = at < left ? (float)s[2 * lane + at] : 0.f;
      }
      uint32_t* d = reinterpret_cast<uint32_t*>(dst + t * pitch + col) + lane;
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (col + 64 * e + 2 * lane < pitch) d[32 * e] = staged_pair(x[2 * e] * mul, x[2 * e + 1] * mul);
      continue;
    }
    if (wide && col + 8 <= Sk) {
      if constexpr (sizeof(T) == 4) {
        const float4 a = *reinterpret_cast<const float4*>(s), b = *reinterpret_cast<const float4*>(s + 4);
        x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w; x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
      } else {
        const uint4 a = *reinterpret_cast<const uint4*>(s);
        const uint32_t w[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
        for (int e = 0; e < 8; ++e) x[e] = __uint_as_float((e & 1) ? w[e >> 1] & 0xffff0000u : w[e >> 1] << 16);
      }
    } else {
#pragma unroll
      for (int e = 0; e < 8; ++e) x[e] = col + e < Sk ? (float)s[e] : 0.f;
    }
    uint32_t o[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) o[e] = staged_pair(x[2 * e] * mul, x[2 * e + 1] * mul);
    reinterpret_cast<uint4*>(dst)[i] = make_uint4(o[0], o[1], o[2], o[3]);
  }
}

}  // namespace af3k
