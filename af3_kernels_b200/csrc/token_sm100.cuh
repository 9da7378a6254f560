// The four projections of the single / diffusion attention block in one GEMM, for sm_100a:
//
//     [q | k | v | gate] = x [M, C] * [Wq; Wk; Wv; Wg]^T,   q <- (q + q_bias) * q_scale
//
// The weights are read where their owner keeps them, `[out, in]` as a K-major B operand or `[in, out]` as an MN-major
// one (64-column blocks of 64 K rows, so that either fills a stage): laying them out in a pass of its own took 4.5 us of
// the 49 of a call at 1536 tokens and C = 384, and a copy kept between calls could be out of date.
//
// Stands in for the projection BRGEMMs of the reference's fused block
// (src/csrc/dot_product_attention.cpp:425-480).  M is a token count (tens to a few thousand), C 384 or 768
// in practice: a few GFLOP, so what bounds it is latency - one tile of 128 rows x kN columns per CTA, the
// K blocks of 64 channels streamed through six stages that hold all of K at C = 384, one warp each for the
// TMA and the MMAs, four for the epilogue.  kN is 64, 128 or 256, so that
// few rounds of CTAs do and few SMs are idle.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <cstdint>

#include "ptx_sm100.cuh"

namespace af3k {

constexpr int kTokThreads = 192;
template <int kN> struct TokTile {
  static constexpr int kStages = kN == 256 ? 4 : 6;
  static constexpr uint32_t kA = 128 * 128, kB = kN * 128, kStage = kA + kB;
  static constexpr uint32_t off_bar = kStages * kStage, off_bias = off_bar + 128, kSmem = off_bias + kN * 4;   // off_bias: query bias, fp32
};

struct TokMaps { CUtensorMap w[4]; };
struct TokParams {
  int M, C;
  int tiles_n;               // column tiles of one matrix; a tile never straddles two
  int mn_mask;               // bit i: matrix i is kept [in, out]
  const void* q_bias;        // [C] bf16 or fp32, may be null
  int q_bias_f32;
  float q_scale;
  __nv_bfloat16* out;        // [4, M, C]
  int* status;
  long long wait_limit;
};

template <int kN>
__global__ void __launch_bounds__(kTokThreads, 1)
token_proj_kernel(const __grid_constant__ TokParams p, const __grid_constant__ CUtensorMap tm_x,
                  const __grid_constant__ TokMaps maps) {
  using Tile = TokTile<kN>;
  extern __shared__ __align__(1024) uint8_t tok_smem[];
  const uint32_t smem = smem_u32(tok_smem), bars = smem + Tile::off_bar;   // full [kStages], empty [kStages], acc
  volatile uint32_t* slot = reinterpret_cast<volatile uint32_t*>(tok_smem + Tile::off_bar + 112);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tok_smem + Tile::off_bar + 116);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int which = blockIdx.y / p.tiles_n;                    // 0 q, 1 k, 2 v, 3 gate
  const int m0 = blockIdx.x * 128, n0 = (blockIdx.y - which * p.tiles_n) * kN, kblocks = (p.C + 63) / 64;
  const bool mn = (p.mn_mask >> which) & 1;
  const CUtensorMap* tm_w = maps.w + which;
  auto timeout = [&](int bar) {
    *abort_flag = 1;
    if (p.status != nullptr) {
      atomicOr(p.status, 1 /* wait timeout */);
      if (atomicCAS(p.status + 1, 0, 3000 + bar + 1) == 0) { p.status[2] = blockIdx.x; p.status[3] = warp; }
    }
  };
  if (threadIdx.x == 0) {
    *abort_flag = 0;
    prefetch_tensormap(&tm_x);
    prefetch_tensormap(tm_w);
    for (int i = 0; i < 2 * Tile::kStages + 1; ++i) mbar_init(bars + 8u * i, 1);
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(const_cast<uint32_t*>(slot)), kN);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *slot;

  if (warp == 0) {
    if (lane == 0) {
      for (int kb = 0; kb < kblocks; ++kb) {
        const int st = kb % Tile::kStages;
        if (kb >= Tile::kStages && !mbar_wait_bounded(bars + 8u * (Tile::kStages + st), ((kb / Tile::kStages) - 1) & 1, p.wait_limit, const_cast<volatile int*>(abort_flag))) {
          timeout(Tile::kStages + st);
          break;
        }
        const uint32_t full = bars + 8u * st, dst = smem + st * Tile::kStage;
        if (kb == 0) {
          grid_wait_previous();
          grid_release_next();
        }
        mbar_arrive_expect_tx(full, Tile::kStage);
        tma_load_2d(dst, &tm_x, full, kb * 64, m0);
        if (!mn) {
          tma_load_2d(dst + Tile::kA, tm_w, full, kb * 64, n0);
        } else {
          for (int j = 0; j < kN; j += 64) tma_load_2d(dst + Tile::kA + j * 128, tm_w, full, n0 + j, kb * 64);
        }
      }
    }
  } else if (warp == 1) {
    const bool leader = elect_one();
    const uint32_t idesc = make_idesc(1u, 1u, 0u, mn ? 1u : 0u, kN);
    // B: K-major, 16 channels = 32 bytes along the 128-byte rows; MN-major, 16 rows of 128 bytes (64 columns), the next
    // 64 columns 64 rows on
    const uint64_t d0 = make_smem_desc(smem, 16, 8 * 128, 2), b0 = make_smem_desc(smem, mn ? 64 * 128 : 16, 8 * 128, 2);
    const uint32_t lo = (uint32_t)d0, hi = (uint32_t)(d0 >> 32), b_lo = (uint32_t)b0, b_hi = (uint32_t)(b0 >> 32);
    const uint32_t b_step = mn ? (16 * 128) >> 4 : 2;
    bool ok = true;
    grid_wait_previous();      // (a wait's limit counts from here)
    for (int kb = 0; kb < kblocks && ok; ++kb) {
      const int st = kb % Tile::kStages;
      ok = mbar_wait_bounded(bars + 8u * st, (kb / Tile::kStages) & 1, p.wait_limit, const_cast<volatile int*>(abort_flag));
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) { timeout(st); break; }
      tc_fence_after();
      if (leader) {
        const uint32_t a = lo + ((st * Tile::kStage) >> 4), b = b_lo + ((st * Tile::kStage + Tile::kA) >> 4);
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) mma_ss_f16(tmem, a + 2 * ks, hi, b + b_step * ks, b_hi, idesc, kb + ks > 0 ? 1u : 0u);
        tc_commit(bars + 8u * (Tile::kStages + st));
        if (kb == kblocks - 1) tc_commit(bars + 8u * (2 * Tile::kStages));
      }
      __syncwarp();
    }
  } else {
    // ---- epilogue: TMEM lane quarter; the stages are free when the accumulator is complete
    const int quarter = warp & 3;
    grid_wait_previous();
    // The query bias lands in shared memory while the GEMM runs.  Read in the epilogue, element by element in the type it is kept in,
    // it was most of the kernel, each load behind the one before: 1536 tokens of 384 channels 13.7 -> 5.1 us, of 768 18.4 -> 12.5,
    // 128 tokens of 384 9.4 -> 4.0.
    if (which == 0) {
      for (int e = threadIdx.x - 64; e < kN; e += 128) {
        float bq = 0.f;
        if (p.q_bias != nullptr && n0 + e < p.C)
          bq = p.q_bias_f32 ? static_cast<const float*>(p.q_bias)[n0 + e] : __bfloat162float(static_cast<const __nv_bfloat16*>(p.q_bias)[n0 + e]);
        asm volatile("st.shared.f32 [%0], %1;" ::"r"(smem + Tile::off_bias + 4u * e), "f"(bq) : "memory");
      }
      asm volatile("bar.sync 1, 128;" ::: "memory");      // the four epilogue warps
    }
    const bool ok = mbar_wait_bounded(bars + 8u * (2 * Tile::kStages), 0, p.wait_limit, const_cast<volatile int*>(abort_flag));
    if (__all_sync(0xffffffffu, ok)) {
      tc_fence_after();
      const uint32_t t_base = tmem + ((uint32_t)(quarter * 32) << 16);
      const uint32_t patch = smem + quarter * (32 * 128);
#pragma unroll 1
      for (int c0 = 0; c0 < kN; c0 += 64) {
#pragma unroll
        for (int hc = 0; hc < 2; ++hc) {
          uint32_t acc[32];
          tmem_ld_x32(t_base + c0 + 32 * hc, acc);
          tc_wait_ld();
          if (which == 0) {
#pragma unroll
            for (int e = 0; e < 32; e += 4) {
              float bq[4];      // all lanes read the same words
              asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                           : "=f"(bq[0]), "=f"(bq[1]), "=f"(bq[2]), "=f"(bq[3]) : "r"(smem + Tile::off_bias + 4u * (c0 + 32 * hc + e)));
#pragma unroll
              for (int u = 0; u < 4; ++u) acc[e + u] = __float_as_uint((__uint_as_float(acc[e + u]) + bq[u]) * p.q_scale);
            }
          }
          // own row -> shared, piece at position piece ^ (row & 7): conflict-free both ways
#pragma unroll
          for (int j = 0; j < 4; ++j)
            asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(patch + lane * 128 + (((4 * hc + j) ^ (lane & 7)) << 4)),
                         "r"(pack_bf16x2(__uint_as_float(acc[8 * j]), __uint_as_float(acc[8 * j + 1]))),
                         "r"(pack_bf16x2(__uint_as_float(acc[8 * j + 2]), __uint_as_float(acc[8 * j + 3]))),
                         "r"(pack_bf16x2(__uint_as_float(acc[8 * j + 4]), __uint_as_float(acc[8 * j + 5]))),
                         "r"(pack_bf16x2(__uint_as_float(acc[8 * j + 6]), __uint_as_float(acc[8 * j + 7]))) : "memory");
        }
        __syncwarp();
        // shared -> global: lane l takes piece l & 7 of rows (l >> 3) + 4 it; C is a multiple of eight
        const int col = n0 + c0 + 8 * (lane & 7);
        if (col < p.C) {
          __nv_bfloat16* dst = p.out + ((long long)which * p.M) * p.C + col;
#pragma unroll
          for (int it = 0; it < 8; ++it) {
            const int row = it * 4 + (lane >> 3), m = m0 + quarter * 32 + row;
            uint4 o;
            asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                         : "=r"(o.x), "=r"(o.y), "=r"(o.z), "=r"(o.w)
                         : "r"(patch + row * 128 + (((lane & 7) ^ (row & 7)) << 4)));
            if (m < p.M) *reinterpret_cast<uint4*>(dst + (long long)m * p.C) = o;
          }
        }
        __syncwarp();      // the patch is rewritten by the next 64 columns
      }
    } else {
      timeout(2 * Tile::kStages);
    }
  }

  tc_fence_before();
  __syncthreads();
  if (*abort_flag != 0) {
    for (int i = 0; i < 200; ++i) __nanosleep(10000);
    __syncthreads();
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, kN);
  }
}

}  // namespace af3k
