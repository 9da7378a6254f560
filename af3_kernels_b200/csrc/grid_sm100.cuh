// The two GEMM-shaped passes around the attention core of the grid / triangle attention block, for sm_100a.
//
//   grid_front_kernel   x = LayerNorm(pair);  bias = (x Wb^T) permuted to [Hb, R, N];
//                       [q | k | v | gate] = x [Wq; Wk; Wv; Wg]^T          (or x = pair as it is)
//   grid_out_kernel     out = (weighted * sigmoid(gate)) Wo^T
//
// They stand in for the statements in front of the core in the reference's modules
// (src/af3_kernels/Attention.py:51-52, :152-153) and for the projection BRGEMMs, the SigmoidFwdTPP + MulTPP
// pair and the output BRGEMM inside its fused block (src/csrc/dot_product_attention.cpp:285-345, :347-372).
//
// Both are the same machine: persistent CTAs over tiles of 128 rows, the weights resident in shared memory,
//
//   warps 12-    row producers: global -> registers -> (LayerNorm | gate product) -> bf16 ->
//                shared memory in the layout of a tcgen05.mma A operand (K-major, 128-byte swizzle,
//                panels of 64 channels).  A row is spread over C / 8 lanes, 8 channels each, so global
//                reads are full 16-byte pieces of consecutive lanes, the LayerNorm reductions are four
//                (C = 64: three) shuffles and its parameters stay in registers.  The next rows are
//                requested before the current ones are worked on.
//   warp 0       TMEM allocation, the weights' TMA loads (fp32 weights: converted by the epilogue warps), the MMAs (fp32
//                accumulators in TMEM)
//   warps 4-11   epilogue, one TMEM lane quarter each, the two warpgroups taking the accumulators in turn: TMEM ->
//                registers -> bf16 or fp32 -> a private XOR-swizzled patch of shared memory -> 16-byte stores
//                in runs of 128 bytes
//   warps 1-3    unused (they give their registers to the other roles)
//
// What bounds them is HBM: per row of a bf16 pair with C = 128 the front reads 256 bytes and writes 1 024
// (+ 2 Hb), the output pass reads 512 and writes 256.  The normalised pair and the gated product never
// reach HBM.  The pair bias is part of the GEMM: as arithmetic of the row producers (32 FMAs and five
// shuffles per row piece) it made their chain the limit, 185 us against 148 (768 x 768 x 128 bf16; a bare kernel
// that reads and writes as much takes 144).  The output pass takes 86 us there (69 at the copy rate).
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <cstdint>
#include <type_traits>

#include "pair_bias_sm100.cuh"
#include "ptx_sm100.cuh"

namespace af3k {

// Twelve warps and the row producers, of which the front has 8 and the output pass 16: its rows carry two exponentials and
// divisions per element in one chain, and two such warps per scheduler left it half idle (us, 8 -> 16 warps: 768 rows 90.5 -> 85.8,
// 389 rows bf16 26.1 -> 24.1, fp32 29.8 -> 28.5, 256 rows of 64 channels 7.4 -> 7.1).  The front is bound by its writes: 768 rows
// 149.7 -> 152.4 with 16, where reading 151 MB and writing 604 takes a bare kernel 144.
// Registers: launched with kLaunch per thread (the pool setmaxnreg works in), then 128 x kMisc (warps 0-3) + 256 x kEpi (epilogue)
// + 32 kRowWarps x kRow (row producers).
template <int kRowWarpsT> struct GridRoles {
  static constexpr int kRowWarps = kRowWarpsT, kThreads = 32 * (12 + kRowWarps), kRowsPerWarp = 128 / kRowWarps;
  static constexpr int kBatch = 32 / kRowWarps;      // steps of rows in flight (and worked on together) per warp
  static constexpr int kLaunch = kRowWarps == 8 ? 96 : 72, kMisc = kRowWarps == 8 ? 48 : 40, kEpi = kRowWarps == 8 ? 96 : 88, kRow = kRowWarps == 8 ? 120 : 72;
  static_assert(128 * kMisc + 256 * kEpi + 32 * kRowWarps * kRow <= kLaunch * kThreads, "setmaxnreg totals exceed the launch allocation");
};

// Shared memory: kRows weight rows per panel of 64 channels, the A tiles, the epilogue patches, barriers.
template <int C, int kRowsT, int kStagesT, int kRowWarpsT, bool kLowT = false>
struct GridTile : GridRoles<kRowWarpsT> {
  static constexpr int kStages = kStagesT, kRows = kRowsT;
  static constexpr bool kLow = kLowT;                      // a second A tile per stage for what bf16 leaves over of x
  static constexpr uint32_t kX = 128 * C * 2;              // one A tile: C / 64 panels of 128 rows x 128 bytes
  static constexpr uint32_t kW = kRows * C * 2;            // weights: C / 64 panels of kRows rows x 128 bytes
  static constexpr uint32_t kPatch = 8 * 32 * 128;         // per epilogue warp: 32 rows x 128 bytes
  static constexpr uint32_t off_x = kW, off_low = off_x + kStages * kX, off_patch = off_low + (kLow ? kStages * kX : 0);
  static constexpr uint32_t off_bar = off_patch + kPatch;
  static constexpr uint32_t off_slot = off_bar + 120;      // TMEM address, abort flag
  static constexpr uint32_t kSmem = off_bar + 128;
};
// Front: the q rows, then kBiasRows rows of the bias projection (each fp32 weight as a bf16 high part, rows
// 0-3, plus a bf16 low part, rows 4-7, so that it is not rounded to bf16), then the k, v and gate rows: the
// bias comes out of the q rows' MMAs as 16 more columns (the upper eight read k rows and are not used).
constexpr int kBiasRows = 8;
// fp32 pairs of 64 channels: x goes to the bias rows' MMAs in two parts as well, so that the bias is that of the fp32
// normalised pair, as torch's LayerNorm and Linear compute it for other widths (at 128 channels af3k_pair_bias rounds x
// first, and so does this).
template <int C, typename T> using FrontTile = GridTile<C, 4 * C + kBiasRows, C == 128 ? 2 : 4, 8, C == 64 && sizeof(T) == 4>;
template <int C> using OutTile = GridTile<C, C, 4, 16>;
constexpr int kFrontAcc = 3;     // accumulators of C + 16 (rounded up to C + 32) TMEM columns, taken in turn

struct GridBar {
  static constexpr int w_full = 0, x_ready = 1 /*[4]*/, x_empty = 5 /*[4]*/, acc_full = 9 /*[3]*/, acc_empty = 12 /*[3]*/, count = 15;
};

struct GridParams {
  long long M;             // rows (= R * N)
  int R, N;                // the pair is [R, N, C]
  int H, D;                // heads and head width, H * D == C
  int transpose;           // 1: q, k, v are those of the pair with its two positions exchanged: [N, H, R, D]
  int split;               // front: CTAs that share a tile's four outputs (small problems): 1, 2 or 4
  float q_scale;
  const void* w[4];        // fp32 weight matrices [C, C] (front: q, k, v, gate; out: output projection), if w_f32
  int w_f32;               // 0: bf16, read through the tensor maps
  const void* pair;        // front: input rows
  const void* gamma;       // front with LayerNorm: [C], bf16 or fp32
  const void* beta;
  const void* bias_w;      // [Hb, C], bf16 or fp32
  int ln_f32, bias_w_f32;
  float eps;
  int Hb;
  __nv_bfloat16* bias;     // [Hb, R, bias_pitch]
  long long bias_pitch;
  __nv_bfloat16 *q, *k, *v, *g;   // front: outputs; g [M, C]
  const __nv_bfloat16* weighted;  // out: attention result [M, C]
  const __nv_bfloat16* gate;      // out: gate [M, C]
  void* out;               // out: [M, C] bf16 or fp32
  int* status;
  long long wait_limit;
};

#define AF3K_GRID_WAIT(idx, parity)                                                              \
  do {                                                                                           \
    const bool ok_ = mbar_wait_bounded(bars + 8u * (idx), (parity), p.wait_limit, abort_flag);    \
    if (!__all_sync(0xffffffffu, ok_)) {                                                         \
      grid_timeout(p, abort_flag, (idx));                                                        \
      goto done;                                                                                 \
    }                                                                                            \
  } while (0)

__device__ __forceinline__ void grid_timeout(const GridParams& p, volatile int* abort_flag, int bar) {
  *abort_flag = 1;
  if (p.status != nullptr) {
    atomicOr(p.status, 1 /* wait timeout */);
    if (atomicCAS(p.status + 1, 0, 2000 + bar + 1) == 0) {
      p.status[2] = blockIdx.x;
      p.status[3] = threadIdx.x >> 5;
    }
  }
}

// eight channels of one row as they sit in memory
template <typename T> struct Raw8 { uint4 v[sizeof(T) / 2]; };
template <typename T>
__device__ __forceinline__ Raw8<T> load_raw8(const T* src, bool live) {
  Raw8<T> r;
#pragma unroll
  for (int i = 0; i < (int)sizeof(T) / 2; ++i)
    r.v[i] = live ? reinterpret_cast<const uint4*>(src)[i] : make_uint4(0u, 0u, 0u, 0u);
  return r;
}
template <typename T>
__device__ __forceinline__ void unpack_raw8(const Raw8<T>& r, float (&x)[8]) {
  if constexpr (sizeof(T) == 4) pb_unpack8<T>(r.v[0], r.v[1], x);
  else                          pb_unpack8<T>(r.v[0], r.v[0], x);
}

__device__ __forceinline__ void sts128(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

// Position of the 16-byte piece c8 (channels 8 c8 ..) of a row in an A tile.
__device__ __forceinline__ uint32_t grid_piece(uint32_t tile, int row, int c8) {
  return tile + (uint32_t)((c8 >> 3) * (128 * 128) + row * 128 + (((c8 & 7) ^ (row & 7)) << 4));
}

// The front's four weight matrices [C, C] (output rows), each where its owner keeps it: a call reads the parameters
// as they are then, and there is no copy that could be out of date.
struct FrontMaps { CUtensorMap w[4]; };

// elements i .. i + n - 1 of a parameter in the type it is kept in, all loads in flight at once (with the type looked at
// per element they wait for one another)
template <int n>
__device__ __forceinline__ void params_at(const void* src, long long i, int f32, float (&x)[n]) {
  if (f32) {
#pragma unroll
    for (int e = 0; e < n; ++e) x[e] = static_cast<const float*>(src)[i + e];
  } else {
#pragma unroll
    for (int e = 0; e < n; ++e) x[e] = __bfloat162float(static_cast<const __nv_bfloat16*>(src)[i + e]);
  }
}

// One fp32 weight matrix [C, C] as rows row0 .. of the B operand, rounded to bf16 on the way (the 256 threads of the epilogue
// warps).  A packing pass in front of the block took 5 us: 389 fp32 rows 264 us a call, with this 261.
template <int C>
__device__ __forceinline__ void grid_convert_weights(uint32_t smem, int rows, const void* src, int row0) {
  constexpr int kItems = C * C / 8 / 256;      // 8 channels of a row each, all in flight at once
  static_assert(kItems * 8 * 256 == C * C, "whole items per thread");
  uint4 v[kItems][2];
  const int k0 = threadIdx.x - 128;
#pragma unroll
  for (int i = 0; i < kItems; ++i) {
    const uint4* s = static_cast<const uint4*>(src) + 2 * (k0 + i * 256);
    v[i][0] = s[0];
    v[i][1] = s[1];
  }
#pragma unroll
  for (int i = 0; i < kItems; ++i) {
    const int k = k0 + i * 256, r = row0 + k / (C / 8), c8 = k % (C / 8);
    sts128(smem + (c8 >> 3) * (rows * 128) + r * 128 + (((c8 & 7) ^ (r & 7)) << 4),
           pack_bf16x2(__uint_as_float(v[i][0].x), __uint_as_float(v[i][0].y)), pack_bf16x2(__uint_as_float(v[i][0].z), __uint_as_float(v[i][0].w)),
           pack_bf16x2(__uint_as_float(v[i][1].x), __uint_as_float(v[i][1].y)), pack_bf16x2(__uint_as_float(v[i][1].z), __uint_as_float(v[i][1].w)));
  }
}

// Barrier set-up and TMEM allocation shared by both kernels (all threads; ends with a block barrier).  Nothing here touches
// global memory: each role waits for the kernel before (grid_wait_previous) where it first does, with its set-up behind it.
template <class Tile>
__device__ __forceinline__ uint32_t grid_prologue(const GridParams& p, uint32_t bars, volatile uint32_t* slot, volatile int* abort_flag, uint32_t tmem_cols,
                                                  const CUtensorMap* tm_w, int chunks) {
  const int warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) {
    *abort_flag = 0;
    if (!p.w_f32)
      for (int c = 0; c < chunks; ++c) prefetch_tensormap(tm_w + c);
    mbar_init(bars + 8u * GridBar::w_full, 1 + 8);           // the loading thread, the epilogue warps
    for (int i = 0; i < Tile::kStages; ++i) {
      mbar_init(bars + 8u * (GridBar::x_ready + i), Tile::kRowWarps);
      mbar_init(bars + 8u * (GridBar::x_empty + i), 1);
    }
    for (int i = 0; i < 3; ++i) {
      mbar_init(bars + 8u * (GridBar::acc_full + i), 1);
      mbar_init(bars + 8u * (GridBar::acc_empty + i), 4);
    }
    fence_barrier_init();
  }
  if (warp == 0) {
    __syncwarp();
    tmem_alloc(smem_u32(const_cast<uint32_t*>(slot)), tmem_cols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  return *slot;
}

// The weights, `chunks` matrices of C rows from p.w[chunk0] on, one tensor map each; `gap` rows are left free behind the first one.
// One thread requests bf16 ones ...
template <class Tile, int C>
__device__ __forceinline__ void grid_load_weights(const GridParams& p, uint32_t smem, uint32_t bars, const CUtensorMap* tm_w, int chunk0, int chunks, int gap) {
  grid_wait_previous();
  if (p.w_f32) {
    mbar_arrive(bars + 8u * GridBar::w_full);
    return;
  }
  mbar_arrive_expect_tx(bars + 8u * GridBar::w_full, (uint32_t)chunks * C * C * 2);
  for (int c = 0; c < chunks; ++c)
    for (int kb = 0; kb < C / 64; ++kb)
      for (int r = 0; r < C; r += 64)
        tma_load_2d(smem + kb * (Tile::kRows * 128) + (c * C + (c > 0 ? gap : 0) + r) * 128, tm_w + chunk0 + c, bars + 8u * GridBar::w_full, kb * 64, r);
}
// ... the epilogue warps convert fp32 ones while there is nothing to store yet (and the front's write its bias rows), then arrive.
template <class Tile, int C>
__device__ __forceinline__ void grid_convert_all(const GridParams& p, uint32_t smem, int chunk0, int chunks, int gap) {
  if (p.w_f32)
    for (int c = 0; c < chunks; ++c) grid_convert_weights<C>(smem, Tile::kRows, p.w[chunk0 + c], c * C + (c > 0 ? gap : 0));
}
__device__ __forceinline__ void grid_weights_written(uint32_t bars, int lane) {
  fence_proxy_async_smem();
  __syncwarp();
  if (lane == 0) mbar_arrive(bars + 8u * GridBar::w_full);
}

// Block-wide end of both kernels.
__device__ __forceinline__ void grid_epilogue_common(volatile int* abort_flag, uint32_t tmem, uint32_t tmem_cols) {
  tc_fence_before();
  __syncthreads();
  if (*abort_flag != 0) {
    for (int i = 0; i < 200; ++i) __nanosleep(10000);
    __syncthreads();
  }
  if ((threadIdx.x >> 5) == 0) {
    tc_fence_after();
    tmem_dealloc(tmem, tmem_cols);
  }
}

template <int C, typename T, bool kLn>
__global__ void __launch_bounds__(FrontTile<C, T>::kThreads, 1)
grid_front_kernel(const __grid_constant__ GridParams p, const __grid_constant__ FrontMaps maps) {
  using Tile = FrontTile<C, T>;
  extern __shared__ __align__(1024) uint8_t grid_smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t smem = smem_u32(grid_smem);
  const uint32_t bars = smem + Tile::off_bar;
  volatile uint32_t* slot = reinterpret_cast<volatile uint32_t*>(grid_smem + Tile::off_slot);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(grid_smem + Tile::off_slot + 4);
  constexpr uint32_t kAccCols = C + 32, kTmem = 512;
  static_assert(kFrontAcc * kAccCols <= kTmem, "accumulators exceed TMEM");
  // this CTA's outputs out of {q + bias, k, v, gate}: all of them unless split
  const int part = blockIdx.x % p.split, first = blockIdx.x / p.split, step = gridDim.x / p.split;
  const int chunks = 4 / p.split, chunk0 = part * chunks;
  const bool with_bias = kLn && p.Hb > 0 && part == 0;
  const long long n_tiles = (p.M + 127) / 128;
  const uint32_t tmem = grid_prologue<Tile>(p, bars, slot, abort_flag, kTmem, maps.w + chunk0, chunks);

  if (warp < 4) {
    setmaxnreg_dec<Tile::kMisc>();
    if (warp == 0) {
      // ---- MMA issuer: the tile's outputs one after the other, into the accumulators in turn
      const bool leader = elect_one();
      const uint32_t idesc = make_idesc(1u, 1u, 0u, 0u, C), idesc_q = make_idesc(1u, 1u, 0u, 0u, C + 16);
      const uint64_t ad0 = make_smem_desc(smem + Tile::off_x, 16, 8 * 128, 2), bd0 = make_smem_desc(smem, 16, 8 * 128, 2);
      const uint32_t ad_lo = (uint32_t)ad0, ad_hi = (uint32_t)(ad0 >> 32), bd_lo = (uint32_t)bd0, bd_hi = (uint32_t)(bd0 >> 32);
      if (leader) grid_load_weights<Tile, C>(p, smem, bars, maps.w, chunk0, chunks, kBiasRows);
      __syncwarp();
      AF3K_GRID_WAIT(GridBar::w_full, 0);
      uint32_t n = 0, buf = 0, lap = 0;
      for (long long tile = first; tile < n_tiles; tile += step, ++n) {
        const uint32_t st = n % Tile::kStages;
        // The next kernel's blocks may come in from each CTA's last tile on: they set themselves up as SMs become free.  (From the
        // prologue on they were in the way, 389 rows 255 -> 257 us a module call; as blocks end, 192 rows 48.5 us on the device,
        // 256 rows of 64 channels 50.9, here 46.5 and 49.9.)
        if (tile + step >= n_tiles) grid_release_next();
        AF3K_GRID_WAIT(GridBar::x_ready + st, (n / Tile::kStages) & 1);
        for (int c = 0; c < chunks; ++c) {
          // the epilogue warps must have read this accumulator's previous columns
          if (lap > 0) AF3K_GRID_WAIT(GridBar::acc_empty + buf, (lap - 1) & 1);
          tc_fence_after();
          if (leader) {
            const uint32_t id = c == 0 && with_bias ? idesc_q : idesc;
            const uint32_t row = (uint32_t)(c * C + (c > 0 ? kBiasRows : 0));
#pragma unroll
            for (int ks = 0; ks < C / 16; ++ks) {   // 16 channels = 32 bytes of a 128-byte panel row; panel ks / 4
              const uint32_t a = ad_lo + ((st * Tile::kX + (ks >> 2) * (128 * 128)) >> 4) + 2 * (ks & 3);
              const uint32_t b = bd_lo + (((ks >> 2) * (Tile::kRows * 128) + row * 128) >> 4) + 2 * (ks & 3);
              mma_ss_f16(tmem + buf * kAccCols, a, ad_hi, b, bd_hi, id, ks > 0 ? 1u : 0u);
            }
            if (Tile::kLow && c == 0 && with_bias) {
              // onto the bias columns alone (N = 16: the eight bias rows and eight that are not used)
              constexpr uint32_t idesc_low = make_idesc(1u, 1u, 0u, 0u, 16);
#pragma unroll
              for (int ks = 0; ks < C / 16; ++ks) {
                const uint32_t a = ad_lo + ((Tile::off_low - Tile::off_x + st * Tile::kX + (ks >> 2) * (128 * 128)) >> 4) + 2 * (ks & 3);
                const uint32_t b = bd_lo + (((ks >> 2) * (Tile::kRows * 128) + C * 128) >> 4) + 2 * (ks & 3);
                mma_ss_f16(tmem + buf * kAccCols + C, a, ad_hi, b, bd_hi, idesc_low, 1u);
              }
            }
            tc_commit(bars + 8u * (GridBar::acc_full + buf));
            if (c == chunks - 1) tc_commit(bars + 8u * (GridBar::x_empty + st));
          }
          __syncwarp();
          if (++buf == kFrontAcc) { buf = 0; ++lap; }
        }
      }
    }
  } else if (warp < 12) {
    // ---- epilogue: TMEM lane quarter; warps 4-7 take the CTA's even outputs, 8-11 the odd ones
    grid_wait_previous();
    if (with_bias) {
      // bias projection rows, 16 bytes (8 channels) per thread
      for (int k = threadIdx.x - 128; k < kBiasRows * (C / 8); k += 256) {
        const int r = k / (C / 8), c8 = k % (C / 8), h = r & 3;
        uint32_t w[4] = {0u, 0u, 0u, 0u};
        if (h < p.Hb) {
          float v[8];
          params_at(p.bias_w, h * C + c8 * 8, p.bias_w_f32, v);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            float x = v[2 * e], y = v[2 * e + 1];
            if (r >= 4) {   // what the bf16 high part leaves over
              x -= __bfloat162float(__float2bfloat16_rn(x));
              y -= __bfloat162float(__float2bfloat16_rn(y));
            }
            w[e] = pack_bf16x2(x, y);
          }
        }
        sts128(smem + (c8 >> 3) * (Tile::kRows * 128) + (C + r) * 128 + (((c8 & 7) ^ (r & 7)) << 4), w[0], w[1], w[2], w[3]);
      }
    }
    grid_convert_all<Tile, C>(p, smem, chunk0, chunks, kBiasRows);
    grid_weights_written(bars, lane);
    const int quarter = warp & 3, wg = (warp - 4) >> 2;
    const uint32_t t_lane = tmem + ((uint32_t)(quarter * 32) << 16);
    const uint32_t patch = smem + Tile::off_patch + (uint32_t)(warp - 4) * (32 * 128);
    const int log2d = 31 - __clz(p.D);
    const int tokens = p.transpose ? p.R : p.N;
    uint32_t count = 0, buf = 0, lap = 0;            // outputs of this CTA so far, their accumulator
    for (long long tile = first; tile < n_tiles; tile += step) {
      const long long m0 = tile * 128 + quarter * 32;                 // the warp's first row
      const int i0 = (int)(m0 / p.N), j0 = (int)(m0 - (long long)i0 * p.N);
      // Element offsets of the eight rows this lane stores in every 64-column piece (rows (lane >> 3)
      // + 4 it), worked out once per tile: into [rows, H, tokens, D] at head 0.
      uint32_t off_qkv[8], row_ok = 0;
#pragma unroll
      for (int it = 0; it < 8; ++it) {
        const int row = it * 4 + (lane >> 3);
        int i = i0, j = j0 + row;
        while (j >= p.N) { j -= p.N; ++i; }
        off_qkv[it] = (uint32_t)(p.transpose ? (long long)j * p.H * p.R + i : (long long)i * p.H * p.N + j) << log2d;
        if (m0 + row < p.M) row_ok |= 1u << it;
      }
      for (int c = 0; c < chunks; ++c, ++count) {
        const uint32_t b = buf, l = lap;
        if (++buf == kFrontAcc) { buf = 0; ++lap; }
        if ((count & 1u) != (uint32_t)wg) continue;
        const int which = chunk0 + c;                                   // 0 q, 1 k, 2 v, 3 gate
        const uint32_t t_base = t_lane + b * kAccCols;
        const float mul = which == 0 ? p.q_scale : 1.0f;
        AF3K_GRID_WAIT(GridBar::acc_full + b, l & 1);
        tc_fence_after();
        if (c == 0 && with_bias) {
          // lane = row: consecutive lanes are consecutive j of one pair row (or the next one)
          uint32_t acc[16];
          tmem_ld_x16(t_base + C, acc);
          tc_wait_ld();
          int i = i0, j = j0 + lane;
          while (j >= p.N) { j -= p.N; ++i; }
          if (m0 + lane < p.M) {
#pragma unroll
            for (int h = 0; h < 4; ++h)
              if (h < p.Hb)
                p.bias[((long long)h * p.R + i) * p.bias_pitch + j] =
                    __float2bfloat16_rn(__uint_as_float(acc[h]) + __uint_as_float(acc[4 + h]));
          }
        }
#pragma unroll 1
        for (int c0 = 0; c0 < C; c0 += 64) {
#pragma unroll
          for (int hc = 0; hc < 2; ++hc) {
            uint32_t acc[32];
            tmem_ld_x32(t_base + c0 + 32 * hc, acc);
            tc_wait_ld();
            // own row -> shared, piece at position piece ^ (row & 7): conflict-free both ways
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              float f[8];
#pragma unroll
              for (int e = 0; e < 8; ++e) f[e] = __uint_as_float(acc[8 * j + e]) * mul;
              sts128(patch + lane * 128 + (((4 * hc + j) ^ (lane & 7)) << 4), pack_bf16x2(f[0], f[1]), pack_bf16x2(f[2], f[3]),
                     pack_bf16x2(f[4], f[5]), pack_bf16x2(f[6], f[7]));
            }
          }
          if (c0 + 64 >= C) {
            // the last columns are in registers: the next MMAs may overwrite this accumulator
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bars + 8u * (GridBar::acc_empty + b));
          } else {
            __syncwarp();
          }
          // shared -> global: lane l takes piece l & 7 of rows (l >> 3) + 4 it
          const int ch = c0 + 8 * (lane & 7);
          __nv_bfloat16* dst;
          if (which == 3) dst = p.g + (m0 + (lane >> 3)) * C + ch;
          else dst = (which == 0 ? p.q : (which == 1 ? p.k : p.v)) + (((long long)(ch >> log2d) * tokens) << log2d) + (ch & (p.D - 1));
#pragma unroll
          for (int it = 0; it < 8; ++it) {
            const int row = it * 4 + (lane >> 3);
            uint4 o;
            asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                         : "=r"(o.x), "=r"(o.y), "=r"(o.z), "=r"(o.w)
                         : "r"(patch + row * 128 + (((lane & 7) ^ (row & 7)) << 4)));
            if ((row_ok >> it) & 1u) *reinterpret_cast<uint4*>(dst + (which == 3 ? (uint32_t)(it * 4 * C) : off_qkv[it])) = o;
          }
          __syncwarp();      // the patch is rewritten by the next 64 columns
        }
      }
    }
  } else {
    // ---- row producers: warp w normalises its rows of every tile
    setmaxnreg_inc<Tile::kRow>();
    const int w = warp - 12;
    constexpr int kLanes = C / 8;                       // lanes per row
    constexpr int kRowsIt = 32 / kLanes;                // rows per step of the warp
    constexpr int kIts = Tile::kRowsPerWarp / kRowsIt;    // steps per tile
    constexpr int kBatch = sizeof(T) == 2 ? Tile::kBatch : Tile::kBatch / 2;
    static_assert(kIts % kBatch == 0, "whole batches per tile");
    const int c8 = lane % kLanes, sub = lane / kLanes;  // channels 8 c8 .., row within the step
    const T* src = static_cast<const T*>(p.pair) + 8 * c8;
    Raw8<T> next[kBatch];
    auto request = [&](long long tile, int it0) {
#pragma unroll
      for (int u = 0; u < kBatch; ++u) {
        const long long m = tile * 128 + w * Tile::kRowsPerWarp + (it0 + u) * kRowsIt + sub;
        next[u] = load_raw8<T>(src + m * C, m < p.M);
      }
    };
    float g[8], b[8];
    grid_wait_previous();
    if (first < n_tiles) request(first, 0);
    if (kLn) {
      params_at(p.gamma, 8 * c8, p.ln_f32, g);
      params_at(p.beta, 8 * c8, p.ln_f32, b);
    }
    uint32_t n = 0;
    for (long long tile = first; tile < n_tiles; tile += step, ++n) {
      const uint32_t st = n % Tile::kStages;
      const uint32_t x_tile = smem + Tile::off_x + st * Tile::kX;
      if (n >= (uint32_t)Tile::kStages) AF3K_GRID_WAIT(GridBar::x_empty + st, ((n / Tile::kStages) - 1) & 1);
#pragma unroll
      for (int it0 = 0; it0 < kIts; it0 += kBatch) {
        Raw8<T> cur[kBatch];
#pragma unroll
        for (int u = 0; u < kBatch; ++u) cur[u] = next[u];
        if (it0 + kBatch < kIts) request(tile, it0 + kBatch);
        else if (tile + step < n_tiles) request(tile + step, 0);
        float y[kBatch][8];
#pragma unroll
        for (int u = 0; u < kBatch; ++u) unpack_raw8<T>(cur[u], y[u]);
        if (kLn) {
          // mean, then the (biased) variance of the deviations, over the row's kLanes lanes
          float s[kBatch];
#pragma unroll
          for (int u = 0; u < kBatch; ++u) s[u] = ((y[u][0] + y[u][1]) + (y[u][2] + y[u][3])) + ((y[u][4] + y[u][5]) + (y[u][6] + y[u][7]));
#pragma unroll
          for (int o = kLanes / 2; o > 0; o >>= 1)
#pragma unroll
            for (int u = 0; u < kBatch; ++u) s[u] += __shfl_xor_sync(0xffffffffu, s[u], o);
#pragma unroll
          for (int u = 0; u < kBatch; ++u) {
            const float mean = s[u] * (1.0f / C);
            float q = 0.f;
#pragma unroll
            for (int e = 0; e < 8; ++e) { y[u][e] -= mean; q = fmaf(y[u][e], y[u][e], q); }
            s[u] = q;
          }
#pragma unroll
          for (int o = kLanes / 2; o > 0; o >>= 1)
#pragma unroll
            for (int u = 0; u < kBatch; ++u) s[u] += __shfl_xor_sync(0xffffffffu, s[u], o);
#pragma unroll
          for (int u = 0; u < kBatch; ++u) {
            const float rstd = rsqrtf(s[u] * (1.0f / C) + p.eps);
#pragma unroll
            for (int e = 0; e < 8; ++e) y[u][e] = fmaf(y[u][e] * rstd, g[e], b[e]);
          }
        }
        uint32_t yw[kBatch][4];
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
#pragma unroll
          for (int e = 0; e < 4; ++e) yw[u][e] = pack_bf16x2(y[u][2 * e], y[u][2 * e + 1]);
          const int row = w * Tile::kRowsPerWarp + (it0 + u) * kRowsIt + sub;
          sts128(grid_piece(x_tile, row, c8), yw[u][0], yw[u][1], yw[u][2], yw[u][3]);
          if (Tile::kLow && with_bias) {
            uint32_t lw[4];
#pragma unroll
            for (int e = 0; e < 4; ++e)
              lw[e] = pack_bf16x2(y[u][2 * e] - __uint_as_float(yw[u][e] << 16), y[u][2 * e + 1] - __uint_as_float(yw[u][e] & 0xffff0000u));
            sts128(grid_piece(x_tile + Tile::off_low - Tile::off_x, row, c8), lw[0], lw[1], lw[2], lw[3]);
          }
        }
      }
      fence_proxy_async_smem();     // the tile was written through the generic proxy; the tensor core reads it
      __syncwarp();
      if (lane == 0) mbar_arrive(bars + 8u * (GridBar::x_ready + st));
    }
  }

done:
  grid_epilogue_common(abort_flag, tmem, kTmem);
}

template <int C, typename TOut>
__global__ void __launch_bounds__(OutTile<C>::kThreads, 1)
grid_out_kernel(const __grid_constant__ GridParams p, const __grid_constant__ CUtensorMap tm_w) {
  using Tile = OutTile<C>;
  extern __shared__ __align__(1024) uint8_t grid_smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t smem = smem_u32(grid_smem);
  const uint32_t bars = smem + Tile::off_bar;
  volatile uint32_t* slot = reinterpret_cast<volatile uint32_t*>(grid_smem + Tile::off_slot);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(grid_smem + Tile::off_slot + 4);
  constexpr uint32_t kTmem = 2 * C;               // two accumulators, taken in turn
  const long long n_tiles = (p.M + 127) / 128;
  const uint32_t tmem = grid_prologue<Tile>(p, bars, slot, abort_flag, kTmem, &tm_w, 1);

  if (warp < 4) {
    setmaxnreg_dec<Tile::kMisc>();
    if (warp == 0) {
      const bool leader = elect_one();
      const uint32_t idesc = make_idesc(1u, 1u, 0u, 0u, (uint32_t)C);
      const uint64_t ad0 = make_smem_desc(smem + Tile::off_x, 16, 8 * 128, 2), bd0 = make_smem_desc(smem, 16, 8 * 128, 2);
      const uint32_t ad_lo = (uint32_t)ad0, ad_hi = (uint32_t)(ad0 >> 32), bd_lo = (uint32_t)bd0, bd_hi = (uint32_t)(bd0 >> 32);
      if (leader) grid_load_weights<Tile, C>(p, smem, bars, &tm_w, 0, 1, 0);
      __syncwarp();
      AF3K_GRID_WAIT(GridBar::w_full, 0);
      uint32_t n = 0;
      for (long long tile = blockIdx.x; tile < n_tiles; tile += gridDim.x, ++n) {
        const uint32_t st = n % Tile::kStages, buf = n & 1;
        if (tile + gridDim.x >= n_tiles) grid_release_next();
        AF3K_GRID_WAIT(GridBar::x_ready + st, (n / Tile::kStages) & 1);
        if (n >= 2) AF3K_GRID_WAIT(GridBar::acc_empty + buf, ((n >> 1) - 1) & 1);
        tc_fence_after();
        if (leader) {
#pragma unroll
          for (int ks = 0; ks < C / 16; ++ks) {
            const uint32_t a = ad_lo + ((st * Tile::kX + (ks >> 2) * (128 * 128)) >> 4) + 2 * (ks & 3);
            const uint32_t b = bd_lo + (((ks >> 2) * (C * 128)) >> 4) + 2 * (ks & 3);
            mma_ss_f16(tmem + buf * C, a, ad_hi, b, bd_hi, idesc, ks > 0 ? 1u : 0u);
          }
          tc_commit(bars + 8u * (GridBar::acc_full + buf));
          tc_commit(bars + 8u * (GridBar::x_empty + st));
        }
        __syncwarp();
      }
    }
  } else if (warp < 12) {
    // ---- epilogue: warps 4-7 take the even tiles (accumulator 0), warps 8-11 the odd ones
    setmaxnreg_inc<Tile::kEpi>();
    const int quarter = warp & 3, buf = (warp - 4) >> 2;
    const uint32_t t_base = tmem + ((uint32_t)(quarter * 32) << 16) + buf * C;
    const uint32_t patch = smem + Tile::off_patch + (uint32_t)(warp - 4) * (32 * 128);
    constexpr int kCols = 128 / (int)sizeof(TOut);      // columns per 128-byte piece of a row
    grid_wait_previous();
    grid_convert_all<Tile, C>(p, smem, 0, 1, 0);
    grid_weights_written(bars, lane);
    uint32_t n = (uint32_t)buf;
    for (long long tile = blockIdx.x + (long long)buf * gridDim.x; tile < n_tiles; tile += 2LL * gridDim.x, n += 2) {
      const long long m0 = tile * 128 + quarter * 32;
      AF3K_GRID_WAIT(GridBar::acc_full + buf, (n >> 1) & 1);
      tc_fence_after();
#pragma unroll 1
      for (int c0 = 0; c0 < C; c0 += kCols) {
#pragma unroll
        for (int hc = 0; hc < kCols / 32; ++hc) {
          uint32_t acc[32];
          tmem_ld_x32(t_base + c0 + 32 * hc, acc);
          tc_wait_ld();
          if constexpr (sizeof(TOut) == 2) {
#pragma unroll
            for (int j = 0; j < 4; ++j)
              sts128(patch + lane * 128 + (((4 * hc + j) ^ (lane & 7)) << 4),
                     pack_bf16x2(__uint_as_float(acc[8 * j]), __uint_as_float(acc[8 * j + 1])),
                     pack_bf16x2(__uint_as_float(acc[8 * j + 2]), __uint_as_float(acc[8 * j + 3])),
                     pack_bf16x2(__uint_as_float(acc[8 * j + 4]), __uint_as_float(acc[8 * j + 5])),
                     pack_bf16x2(__uint_as_float(acc[8 * j + 6]), __uint_as_float(acc[8 * j + 7])));
          } else {
#pragma unroll
            for (int j = 0; j < 8; ++j)
              sts128(patch + lane * 128 + ((j ^ (lane & 7)) << 4), acc[4 * j], acc[4 * j + 1], acc[4 * j + 2], acc[4 * j + 3]);
          }
        }
        if (c0 + kCols >= C) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(bars + 8u * (GridBar::acc_empty + buf));
        } else {
          __syncwarp();
        }
        TOut* dst = static_cast<TOut*>(p.out) + m0 * C + c0 + (lane & 7) * (16 / (int)sizeof(TOut));
#pragma unroll
        for (int it = 0; it < 8; ++it) {
          const int row = it * 4 + (lane >> 3);
          uint4 o;
          asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                       : "=r"(o.x), "=r"(o.y), "=r"(o.z), "=r"(o.w)
                       : "r"(patch + row * 128 + (((lane & 7) ^ (row & 7)) << 4)));
          if (m0 + row < p.M) *reinterpret_cast<uint4*>(dst + row * C) = o;
        }
        __syncwarp();
      }
    }
  } else {
    // ---- row producers: weighted * sigmoid(gate), sigmoid in fp32, rounded once
    const int w = warp - 12;
    constexpr int kLanes = C / 8, kRowsIt = 32 / kLanes, kIts = Tile::kRowsPerWarp / kRowsIt, kBatch = Tile::kBatch;
    static_assert(kIts % kBatch == 0, "whole batches per tile");
    const int c8 = lane % kLanes, sub = lane / kLanes;
    uint4 na[kBatch], ng[kBatch];
    auto request = [&](long long tile, int it0) {
#pragma unroll
      for (int u = 0; u < kBatch; ++u) {
        const long long m = tile * 128 + w * Tile::kRowsPerWarp + (it0 + u) * kRowsIt + sub;
        na[u] = load_raw8<__nv_bfloat16>(p.weighted + m * C + 8 * c8, m < p.M).v[0];
        ng[u] = load_raw8<__nv_bfloat16>(p.gate + m * C + 8 * c8, m < p.M).v[0];
      }
    };
    grid_wait_previous();
    if ((long long)blockIdx.x < n_tiles) request(blockIdx.x, 0);
    uint32_t n = 0;
    for (long long tile = blockIdx.x; tile < n_tiles; tile += gridDim.x, ++n) {
      const uint32_t st = n % Tile::kStages;
      const uint32_t x_tile = smem + Tile::off_x + st * Tile::kX;
      if (n >= (uint32_t)Tile::kStages) AF3K_GRID_WAIT(GridBar::x_empty + st, ((n / Tile::kStages) - 1) & 1);
#pragma unroll
      for (int it0 = 0; it0 < kIts; it0 += kBatch) {
        uint4 ca[kBatch], cg[kBatch];
#pragma unroll
        for (int u = 0; u < kBatch; ++u) { ca[u] = na[u]; cg[u] = ng[u]; }
        if (it0 + kBatch < kIts) request(tile, it0 + kBatch);
        else if (tile + gridDim.x < n_tiles) request(tile + gridDim.x, 0);
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
          const uint32_t aw[4] = {ca[u].x, ca[u].y, ca[u].z, ca[u].w}, gw[4] = {cg[u].x, cg[u].y, cg[u].z, cg[u].w};
          uint32_t r[4];
#pragma unroll
          for (int e = 0; e < 4; ++e)
            r[e] = pack_bf16x2(__uint_as_float(aw[e] << 16) * sigmoid_f32(__uint_as_float(gw[e] << 16)),
                               __uint_as_float(aw[e] & 0xffff0000u) * sigmoid_f32(__uint_as_float(gw[e] & 0xffff0000u)));
          const int row = w * Tile::kRowsPerWarp + (it0 + u) * kRowsIt + sub;
          sts128(grid_piece(x_tile, row, c8), r[0], r[1], r[2], r[3]);
        }
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(bars + 8u * (GridBar::x_ready + st));
    }
  }

done:
  grid_epilogue_common(abort_flag, tmem, kTmem);
}

// ------------------------------------------------------------------ packed weights
// Parameters the kernels cannot read where they are ([in, out] in the grid block, fp32 in the single block, any other
// strides), laid out for one call:
// W4 [4 C, C] = q, k, v, gate rows, Wo [C, C] (rows = output channels, bf16), gamma, beta, bias projection (fp32).
// Latency-bound (C = 384: 1.2 MB in and out), so one tile of 64 x 64 per block, read along the source's unit stride
// and turned in shared memory: `[in, out]` weights read along `in` would touch a sector per element.
struct PackMatrix { const void* src; long long so, si; int f32; };   // element (out, in) at so * out + si * in
struct PackParams {
  PackMatrix w[5];         // q, k, v, gate, output projection (src == nullptr: absent)
  PackMatrix bias_w;       // [Hb, C]; src == nullptr: absent
  const void* gamma; const void* beta; int ln_f32;
  int C, Hb;
  __nv_bfloat16* w4; __nv_bfloat16* wo; float* vec;    // vec: gamma [C], beta [C], bias_w [Hb, C]; null: none
  const float4* x; uint2* x_bf16; long long x_n4;      // activations to round in the same launch, in pieces of four; null: none
};
constexpr int kPackTile = 64, kPackThreads = 256, kPackSlices = 6, kPackXEach = 4;
// blockIdx = (tile along in, tile along out, matrix); blockIdx.z == 5: the vectors, from kPackSlices on: the activations
__global__ void __launch_bounds__(kPackThreads) grid_pack_kernel(const __grid_constant__ PackParams p) {
  __shared__ __nv_bfloat16 tile[kPackTile][kPackTile + 2];
  const int C = p.C, m = blockIdx.z;
  grid_wait_previous();
  grid_release_next();
  if (m >= kPackSlices) {
    const long long first = (((long long)(m - kPackSlices) * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x) * (kPackThreads * kPackXEach) + threadIdx.x;
    float4 v[kPackXEach];
#pragma unroll
    for (int i = 0; i < kPackXEach; ++i)
      if (first + i * kPackThreads < p.x_n4) v[i] = p.x[first + i * kPackThreads];
#pragma unroll
    for (int i = 0; i < kPackXEach; ++i)
      if (first + i * kPackThreads < p.x_n4) p.x_bf16[first + i * kPackThreads] = make_uint2(pack_bf16x2(v[i].x, v[i].y), pack_bf16x2(v[i].z, v[i].w));
    return;
  }
  if (m == 5) {
    if (p.vec == nullptr) return;
    if (blockIdx.x != 0 || blockIdx.y != 0) return;
    for (int e = threadIdx.x; e < (2 + p.Hb) * C; e += kPackThreads) {
      const int v = e / C, c = e % C;
      const void* src = v == 0 ? p.gamma : (v == 1 ? p.beta : p.bias_w.src);
      if (src == nullptr) continue;
      float x[1];
      params_at(src, v < 2 ? c : p.bias_w.so * (v - 2) + p.bias_w.si * c, v < 2 ? p.ln_f32 : p.bias_w.f32, x);
      p.vec[e] = x[0];
    }
    return;
  }
  const PackMatrix w = p.w[m];
  if (w.src == nullptr) return;
  const int r0 = blockIdx.y * kPackTile, c0 = blockIdx.x * kPackTile;
  const bool along_out = w.so == 1 && w.si != 1;
  const int fast = threadIdx.x % kPackTile, slow = threadIdx.x / kPackTile;
  constexpr int kStep = kPackThreads / kPackTile, kEach = kPackTile / kStep;
  // all of a thread's loads in flight at once: the type is looked at outside the loop
  auto load = [&](const auto* src) {
    std::remove_const_t<std::remove_reference_t<decltype(*src)>> v[kEach];
#pragma unroll
    for (int i = 0; i < kEach; ++i) {
      const int r = r0 + (along_out ? fast : slow + i * kStep), c = c0 + (along_out ? slow + i * kStep : fast);
      if (r < C && c < C) v[i] = src[w.so * r + w.si * c];
    }
#pragma unroll
    for (int i = 0; i < kEach; ++i) {
      const int r = along_out ? fast : slow + i * kStep, c = along_out ? slow + i * kStep : fast;
      tile[r][c] = (__nv_bfloat16)v[i];     // rounded to nearest
    }
  };
  if (w.f32) load(static_cast<const float*>(w.src));
  else       load(static_cast<const __nv_bfloat16*>(w.src));
  __syncthreads();
  __nv_bfloat16* dst = m < 4 ? p.w4 + (long long)m * C * C : p.wo;
#pragma unroll
  for (int i = 0; i < kPackTile; i += kStep) {
    const int r = slow + i;
    if (r0 + r < C && c0 + fast < C) dst[(long long)(r0 + r) * C + c0 + fast] = tile[r][fast];
  }
}

}  // namespace af3k
