// C ABI of libaf3k.so (declared in include/af3k.h): argument validation, launch planning,
// TMA descriptor encoding and kernel launches.  No torch types cross this boundary.
#include "../../include/af3k.h"

#include <algorithm>
#include <atomic>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <utility>
#include <vector>

#include <cuda.h>
#include <cuda_runtime.h>
#include <cudaTypedefs.h>

#include "attn_sm100.cuh"
#include "grid_sm100.cuh"
#include "pair_bias_sm100.cuh"
#include "token_sm100.cuh"

namespace {

using namespace af3k;

std::atomic<long long> g_wait_limit{-1};
thread_local int t_last_launches = 0;
std::atomic<float*> g_debug_dump{nullptr};
thread_local char t_detail[256] = "";

// Records which CUDA call failed (text returned by af3k_last_error_detail) and clears the
// runtime's sticky-until-read error so that it does not surface in the caller's next CUDA call.
int cuda_fail(const char* what, cudaError_t e) {
  std::snprintf(t_detail, sizeof(t_detail), "%s: %s", what, cudaGetErrorString(e));
  (void)cudaGetLastError();
  return AF3K_ERR_CUDA;
}
int driver_fail(const char* what, int r) {
  std::snprintf(t_detail, sizeof(t_detail), "%s: CUresult %d", what, r);
  return AF3K_ERR_CUDA;
}

long long wait_limit_cycles() {
  long long v = g_wait_limit.load();
  if (v > 0) return v;
  const char* e = std::getenv("AF3K_WAIT_LIMIT_CYCLES");
  v = e ? std::atoll(e) : 0;
  if (v <= 0) v = 2000000000LL;
  g_wait_limit.store(v);
  return v;
}

PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  });
  return fn;
}

constexpr int kStaticSmemReserve = 1024;   // the kernels' few static bytes, padded to the dynamic part's alignment

// Single key tiles come in these widths (48 was not tried: 33 to 48 keys run as 64); every width is a kernel of its own, whose softmax
// warps have that many logits in registers.
constexpr int kKeyWidths[] = {32, 64, 80, 96, 112, 128};

// f(kernel) for the kernel of key tiles of kw keys, the last of last_w.
template <bool kFp8, bool kGate, bool kMixed, bool kConvert, typename F>
void with_width(int kw, int last_w, F&& f) {
  if (last_w != kw) {
    switch (last_w) {
      case 32: return f(attention_kernel<false, true, kFp8, kGate, kMixed, kConvert, 128, 32>);
      case 64: return f(attention_kernel<false, true, kFp8, kGate, kMixed, kConvert, 128, 64>);
      default: return f(attention_kernel<false, true, kFp8, kGate, kMixed, kConvert, 128, 96>);
    }
  }
  switch (kw) {
    case 32: return f(attention_kernel<false, true, kFp8, kGate, kMixed, kConvert, 32>);
    case 64: return f(attention_kernel<false, true, kFp8, kGate, kMixed, kConvert, 64>);
    case 80: return f(attention_kernel<false, true, kFp8, kGate, kMixed, kConvert, 80>);
    case 96: return f(attention_kernel<false, true, kFp8, kGate, kMixed, kConvert, 96>);
    case 112: return f(attention_kernel<false, true, kFp8, kGate, kMixed, kConvert, 112>);
    default: return f(attention_kernel<false, true, kFp8, kGate, kMixed, kConvert, 128>);
  }
}

struct DeviceInfo {
  int sm_count = 0;
  int cc_major = 0;
  int max_smem_optin = 0;
  bool attr_set = false;
};

int device_info(DeviceInfo** out) {
  static DeviceInfo infos[64];
  static std::mutex mu;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || dev < 0 || dev >= 64) return cuda_fail("cudaGetDevice", e);
  std::lock_guard<std::mutex> lock(mu);
  DeviceInfo& d = infos[dev];
  if (d.sm_count == 0) {
    cudaDeviceProp prop;
    if ((e = cudaGetDeviceProperties(&prop, dev)) != cudaSuccess)
      return cuda_fail("cudaGetDeviceProperties", e);
    d.sm_count = prop.multiProcessorCount;
    d.cc_major = prop.major;
    d.max_smem_optin = (int)prop.sharedMemPerBlockOptin;
  }
  if (d.cc_major != 10) return AF3K_ERR_UNSUPPORTED_DEVICE;
  if (!d.attr_set) {
    // the opt-in limit covers static + dynamic shared memory; the kernel has a few static bytes
    const int dyn = d.max_smem_optin - kStaticSmemReserve;
    const cudaFuncAttribute attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
    std::vector<const void*> kernels = {
        (const void*)attention_kernel<false, true, true, true, false>,   (const void*)attention_kernel<false, true, true, true, true>,
        (const void*)attention_kernel<false, false, true, false, false>, (const void*)attention_kernel<false, false, true, true, false>,
        (const void*)attention_kernel<false, false, true, false, true>,  (const void*)attention_kernel<false, false, true, true, true>,
        (const void*)attention_kernel<true, true, false, false, true>,   (const void*)attention_kernel<true, true, true, false, true>,
        (const void*)attention_kernel<true, false, true, false, true>,
    };
    const auto add = [&](auto kernel) { kernels.push_back((const void*)kernel); };
    const auto add_width = [&](int kw, int last_w) {
      with_width<false, false, false, false>(kw, last_w, add); with_width<false, false, true, false>(kw, last_w, add);
      with_width<false, true, false, false>(kw, last_w, add);  with_width<false, true, true, false>(kw, last_w, add);
      with_width<false, false, false, true>(kw, last_w, add);  with_width<false, true, false, true>(kw, last_w, add);
      with_width<true, false, false, false>(kw, last_w, add);  with_width<true, false, true, false>(kw, last_w, add);
    };
    for (int kw : kKeyWidths) add_width(kw, kw);
    for (int last_w : {32, 64, 96}) add_width(kTile, last_w);
    e = cudaSuccess;
    for (const void* kfn : kernels)
      if (e == cudaSuccess) e = cudaFuncSetAttribute(kfn, attr, dyn);
    if (e != cudaSuccess)
      return cuda_fail("cudaFuncSetAttribute(MaxDynamicSharedMemorySize)", e);
    if ((e = cudaFuncSetAttribute(pair_bias_kernel_t<float>, attr, PbTile<float>::kSmemBytes)) != cudaSuccess ||
        (e = cudaFuncSetAttribute(pair_bias_kernel_t<__nv_bfloat16>, attr, PbTile<__nv_bfloat16>::kSmemBytes)) !=
            cudaSuccess)
      return cuda_fail("cudaFuncSetAttribute(MaxDynamicSharedMemorySize, pair_bias)", e);
    if ((e = cudaFuncSetAttribute(pair_bias_mma_kernel, attr, kPbmSmemBytes)) != cudaSuccess)
      return cuda_fail("cudaFuncSetAttribute(MaxDynamicSharedMemorySize, pair_bias_mma)", e);
    const std::pair<const void*, uint32_t> gemm_kernels[] = {
        {(const void*)grid_front_kernel<128, __nv_bfloat16, true>, FrontTile<128, __nv_bfloat16>::kSmem}, {(const void*)grid_front_kernel<128, float, true>, FrontTile<128, float>::kSmem},
        {(const void*)grid_front_kernel<128, __nv_bfloat16, false>, FrontTile<128, __nv_bfloat16>::kSmem}, {(const void*)grid_front_kernel<64, __nv_bfloat16, true>, FrontTile<64, __nv_bfloat16>::kSmem},
        {(const void*)grid_front_kernel<64, float, true>, FrontTile<64, float>::kSmem}, {(const void*)grid_front_kernel<64, __nv_bfloat16, false>, FrontTile<64, __nv_bfloat16>::kSmem},
        {(const void*)grid_out_kernel<128, __nv_bfloat16>, OutTile<128>::kSmem}, {(const void*)grid_out_kernel<128, float>, OutTile<128>::kSmem},
        {(const void*)grid_out_kernel<64, __nv_bfloat16>, OutTile<64>::kSmem}, {(const void*)grid_out_kernel<64, float>, OutTile<64>::kSmem},
        {(const void*)token_proj_kernel<64>, TokTile<64>::kSmem}, {(const void*)token_proj_kernel<128>, TokTile<128>::kSmem}, {(const void*)token_proj_kernel<256>, TokTile<256>::kSmem},
    };
    for (const auto& k : gemm_kernels)
      if ((e = cudaFuncSetAttribute(k.first, attr, (int)k.second)) != cudaSuccess)
        return cuda_fail("cudaFuncSetAttribute(MaxDynamicSharedMemorySize, projections)", e);
    d.attr_set = true;
  }
  *out = &d;
  return AF3K_OK;
}

int row_bytes_for(int64_t bytes) { return bytes <= 32 ? 32 : (bytes <= 64 ? 64 : 128); }
CUtensorMapSwizzle swizzle_for(int row_bytes) {
  return row_bytes == 128 ? CU_TENSOR_MAP_SWIZZLE_128B
                          : (row_bytes == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B);
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// Does the bias need the bf16 staging copy?
bool bias_needs_staging(const af3k_attention_desc& d, const void* bias) {
  if (d.bias_dtype != AF3K_BF16) return true;
  if ((d.bias_stride[0] * 2) % 16 != 0 || (d.bias_stride[1] * 2) % 16 != 0) return true;
  if (bias != nullptr && !aligned16(bias)) return true;
  return false;
}
int64_t staged_bias_pitch(int64_t Sk) { return (Sk + 7) / 8 * 8; }

int validate(const af3k_attention_desc& d) {
  if (d.qk_dtype != AF3K_BF16 && d.qk_dtype != AF3K_FP8_E4M3) return AF3K_ERR_BAD_DTYPE;
  if (d.bias_dtype != AF3K_BF16 && d.bias_dtype != AF3K_F32) return AF3K_ERR_BAD_DTYPE;
  if (d.B1 < 0 || d.B2 < 0 || d.Sq < 0 || d.Sk <= 0 || d.D <= 0) return AF3K_ERR_BAD_SHAPE;
  if (d.D % 8 != 0 || d.D > 64) return AF3K_ERR_BAD_SHAPE;
  if (d.qk_dtype == AF3K_FP8_E4M3 && d.D % 16 != 0) return AF3K_ERR_BAD_SHAPE;
  if (d.B1 > 0x7fffffff || d.B2 > 0x7fffffff || d.Sq > 0x7fffff00 || d.Sk > 0x7fffff00)
    return AF3K_ERR_BAD_SHAPE;
  if (d.rows_per_item < 0 || d.rows_per_item > 8) return AF3K_ERR_BAD_SHAPE;   // a request, clamped by the plan
  if (d.bias_prescaled != 0 && (d.bias_prescaled != 1 || d.qk_dtype != AF3K_FP8_E4M3 || d.bias_dtype != AF3K_BF16))
    return AF3K_ERR_BAD_DTYPE;
  if (d.max_ctas < 0) return AF3K_ERR_BAD_SHAPE;
  if (d.gate != nullptr) {
    if (!aligned16(d.gate)) return AF3K_ERR_BAD_ALIGNMENT;
    for (int i = 0; i < 3; ++i)
      if (d.gate_stride[i] < 0 || (d.gate_stride[i] * 2) % 16) return AF3K_ERR_BAD_STRIDE;
  }
  const int64_t es = d.qk_dtype == AF3K_FP8_E4M3 ? 1 : 2;
  for (int i = 0; i < 3; ++i) {
    if (d.q_stride[i] < 0 || d.k_stride[i] < 0 || d.v_stride[i] < 0 || d.out_stride[i] < 0)
      return AF3K_ERR_BAD_STRIDE;
    if ((d.q_stride[i] * es) % 16 || (d.k_stride[i] * es) % 16 || (d.v_stride[i] * 2) % 16 ||
        (d.out_stride[i] * 2) % 16)
      return AF3K_ERR_BAD_STRIDE;
  }
  if (d.q_stride[2] < d.D || d.k_stride[2] < d.D || d.v_stride[2] < d.D || d.out_stride[2] < d.D)
    return AF3K_ERR_BAD_STRIDE;
  if (d.bias_stride[0] < 0 || d.bias_stride[1] < d.Sk || d.mask_row_stride < 0)
    return AF3K_ERR_BAD_STRIDE;
  // A zero stride (a broadcast view) is only meaningful on a dimension of extent 1: TMA cannot
  // express it, and a zero output stride would make rows overwrite each other.
  const int64_t ext_q[3] = {d.B1, d.B2, d.Sq}, ext_k[3] = {d.B1, d.B2, d.Sk};
  for (int i = 0; i < 3; ++i) {
    if (ext_q[i] > 1 && (d.q_stride[i] == 0 || d.out_stride[i] == 0)) return AF3K_ERR_BAD_STRIDE;
    if (ext_k[i] > 1 && (d.k_stride[i] == 0 || d.v_stride[i] == 0)) return AF3K_ERR_BAD_STRIDE;
  }
  if (d.B2 > 1 && d.bias_stride[0] == 0) return AF3K_ERR_BAD_STRIDE;
  return AF3K_OK;
}

// Launches a kernel whose blocks may become resident under the tail of the kernel before it on the stream; the
// kernel itself waits for that one (grid_wait_previous) before it touches global memory.  Not with a block limit
// (max_ctas): the SMs it leaves free are another stream's, and blocks that wait there would take them.
template <typename... KArgs, typename... Args>
void launch_overlapped(void (*kernel)(KArgs...), dim3 grid, int threads, size_t smem, cudaStream_t stream, bool overlap, const Args&... args) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = &attr;
  cfg.numAttrs = overlap ? 1 : 0;
  (void)cudaLaunchKernelEx(&cfg, kernel, args...);   // the caller reads cudaGetLastError
}

struct Plan {
  AttnParams p;
  int last_w;      // keys of the last key tile
  size_t smem_bytes;
  int grid;
  double cost;     // of the longest CTA, in logits-tile times of one warpgroup
};

// The longest CTA's time when n_main items of cost c_main and then n_tail of cost c_tail are dealt out round-robin.
double dealt_cost(long long n_main, double c_main, long long n_tail, double c_tail, long long ctas) {
  const long long n = n_main + n_tail, cuts[] = {0, n_main % ctas - 1, n_main % ctas, n % ctas - 1, n % ctas, ctas - 1};
  double most = 0;
  for (long long b : cuts) {
    if (b < 0 || b >= ctas) continue;
    const long long m = n_main / ctas + (b < n_main % ctas), all = n / ctas + (b < n % ctas);
    const double cost = m * c_main + (all - m) * c_tail;
    if (cost > most) most = cost;
  }
  return most;
}

// A logits tile of an item with one stream against one of an item with two: the warpgroup has the XU, the MMA
// issuers and the instruction fetch to itself.  So where twice the CTAs are free, two query tiles take two of them:
// 16 heads, us a call, two tiles per CTA -> one: 300 tokens 10.2 -> 8.5, 512 11.7 -> 9.6, 700 15.1 -> 13.0, 1152 (144
// CTAs) 21.4 -> 16.8; 2 x 512 tokens 15.1 -> 11.9.  From there on the CTAs would take two rounds.
constexpr double kLoneTile = 0.75;

// Smaller items behind the last full round have to promise this much: the model is no better than that.
constexpr double kTailGain = 0.98;

// Keys per key tile, and of the last one.  A tile's loads from TMEM, maximum, exponentials, stores and MMAs go with its width
// while its waits and hand-overs do not, so a single tile is the narrowest that holds the call's keys, and the last of several, behind
// tiles of 128, the narrowest in steps of 32 where that leaves out at least a twelfth of the call's columns.  Its code beside the loop's costs
// about what less than that gains: time with it over time without, 5 x 16 heads, rows of the operator, converted bias: 2 tiles, the last of 32 0.93
// 0.88 0.92, of 96 0.97 0.93 1.00; 3 tiles, 96 0.97 0.97 1.01; 4 tiles, 32 0.98 0.93 0.94, 96 1.01 1.00 1.01; 6 tiles, 64 1.00 0.96 0.99; 8 tiles, 32
// 0.99 0.96 0.98, 64 1.00 0.97 0.99; 13 tiles, 32 1.02 - 0.99, 64 1.01 - 1.01.
// Where the borders between tiles lie is part of the result: they decide which key a row's weights are rounded against.  Tiles of one
// width each (389 keys as four of 112) left results up to 1.5 % farther from 64 bits (192 rows of 192 keys 2.632e-3 -> 2.673e-3).
// (Depends on nothing but the keys and the kind of kernel, so that all plans of a call add up the same tiles.)  Device time, us, all tiles
// of 128 -> so: module call of 150 rows 46.2 -> 39.0, 192 48.9 -> 43.3, 389 216 -> 206; operator on 392 rows 151 -> 138, fp8 140 -> 131, on 77 keys
// 5.6 -> 5.3.  With the width as a run-time value in the issuers' loops 1536 tokens took 25.2 instead of 24.5, so the widths
// are template arguments of every role.
void key_widths(const af3k_attention_desc& d, bool tc_bias, bool debug, Plan* plan) {
  AttnParams* const p = &plan->p;
  const bool fp8 = d.qk_dtype == AF3K_FP8_E4M3;
  p->n_kt = (p->Sk + kTile - 1) / kTile;
  p->kw = plan->last_w = kTile;
  if (!tc_bias || (fp8 && d.gate != nullptr) || debug) return;   // kernels of one width
  const int rest = p->Sk - (p->n_kt - 1) * kTile;
  if (p->n_kt > 1) {
    const int w = (rest + 31) / 32 * 32;
    if (12 * (kTile - w) >= kTile * p->n_kt) plan->last_w = w;
    return;
  }
  for (int kw : kKeyWidths)
    if (kw >= rest) { p->kw = plan->last_w = kw; return; }
}

// Picks rows-per-item G and the K/V ring depth from a cost model of one CTA's time (below).
// allow_q_split: the kernel variant that will run supports query-tile streams (every variant in
// which the tensor core adds the bias).
// lone: one query tile of one pair row per item.
int make_plan(const af3k_attention_desc& d, const DeviceInfo& dev, Plan* plan, bool allow_q_split = true, bool lone = false) {
  AttnParams& p = plan->p;
  std::memset(&p, 0, sizeof(p));
  const int es = d.qk_dtype == AF3K_FP8_E4M3 ? 1 : 2;
  p.B1 = (int)d.B1; p.B2 = (int)d.B2; p.Sq = (int)d.Sq; p.Sk = (int)d.Sk; p.D = (int)d.D;
  p.n_qt = (p.Sq + kTile - 1) / kTile;
  p.debug = g_debug_dump.load();
  key_widths(d, allow_q_split, p.debug != nullptr, plan);
  p.qk_row_bytes = row_bytes_for(d.D * es);
  p.v_row_bytes = row_bytes_for(d.D * 2);
  p.qk_ksteps = (int)((d.D * es + 31) / 32);
  p.nv = (int)((d.D + 15) / 16 * 16);
  p.q_tile_bytes = kTile * p.qk_row_bytes;
  if (es == 2 && d.D > 32 && d.D <= 48) {
    p.qk_narrow = 1;
    p.qk_row_bytes = 64;
    p.q_tile_bytes = kTile * (64 + 32);
  }
  p.k_tile_bytes = p.q_tile_bytes;
  p.v_tile_bytes = kTile * p.v_row_bytes;
  p.kv_load_bytes = p.kw * (p.k_tile_bytes / kTile + p.v_row_bytes);
  p.scale = d.softmax_scale;

  const int budget = dev.max_smem_optin - kStaticSmemReserve;
  p.mask_col = 1;   // set for real in the launch path once the mask pointer is known
  constexpr int kSharedBiasStages = 2;
  const int fixed = kSharedBiasStages * kBiasTileBytes + (int)kBarrierBlockBytes +
                    (kMaxKvStages + 2) * (int)kMaskPanelBytes /*ones column, mask ring, zero block*/ +
                    (int)kIdentBytes;
  const int kv_stage = (int)(p.k_tile_bytes + p.v_tile_bytes);
  const int g_tmem = (int)((kTmemCols - kOCol) / p.nv);
  int g_max = kMaxStreams < g_tmem ? kMaxStreams : g_tmem;
  if (g_max > p.B1) g_max = p.B1 > 0 ? p.B1 : 1;
  if (lone) g_max = 1;

  int best_g = 0, best_stages = 0, best_qbuf = 0;
  bool best_split = false;
  long long best_rows = 0;     // pair rows taken by the main items
  double best_cost = 0;
  const int ctas = (d.max_ctas > 0 && d.max_ctas < dev.sm_count) ? d.max_ctas : dev.sm_count;
  // rows_per_item is a request: it is honoured up to what TMEM and the batch allow
  const int g_req = d.rows_per_item > g_max ? g_max : d.rows_per_item;
  auto tiles_of = [&](bool split) { return (long long)(split ? (p.n_qt + 1) / 2 : p.n_qt); };
  // An item's time, in logits-tile times of one warpgroup: streams alternate between the two softmax warpgroups (an odd
  // count leaves one idle slot), n_kt tiles for each of a warpgroup's slots, plus about 0.8 for the epilogue and the
  // hand-over to the next item; with a single Q buffer the next item's Q tiles are loaded and scaled at the hand-over
  // (about 0.5: each stream's tile is replaced as soon as its last Q K^T has finished).  These figures, kLoneTile and kRingPenalty are
  // from when results were stored at the item's end and the P V issuer scaled Q; they were not measured again since.
  auto item_cost = [&](int g, bool split, int qbuf) {
    const int streams = split ? 2 : g;
    return p.n_kt * ((streams + 1) / 2) * (streams == 1 ? kLoneTile : 1.0) + 0.8 + (qbuf == 1 ? 0.5 : 0.0);
  };
  for (int g = 1; g <= g_max; ++g) {
    if (g_req != 0 && g != g_req) continue;
    // one pair row per item: the two softmax warpgroups take two neighbouring query tiles, or one of them idles
    const bool may_split = g == 1 && allow_q_split && p.n_qt >= 2 && !lone;
    for (int form = may_split ? 0 : 2; form < 4; ++form) {
      const bool split = form < 2;
      const int qbuf = 2 - (form & 1);
      const int streams = split ? 2 : g;
      int stages = (budget - fixed - qbuf * streams * (int)p.q_tile_bytes) / kv_stage;
      if (stages > kMaxKvStages) stages = kMaxKvStages;
      if (stages < 2) continue;
      // a K/V tile takes about two thousand cycles to arrive, most of a logits tile's time: with a
      // short ring the MMAs wait for their operands (measured: 4 stages cost about 3 %)
      static const double kRingPenalty[7] = {0, 0, 1.4, 1.15, 1.03, 1.0, 1.0};
      double weight = kRingPenalty[stages];
      if (split) weight *= 1.02;   // query-tile streams share no bias tile: pair rows win a tie
      const double main_cost = item_cost(g, split, qbuf);
      const long long per_group = (long long)p.B2 * tiles_of(split), groups = (p.B1 + g - 1) / g;
      auto offer = [&](double cost, long long rows) {
        cost *= weight;
        if (best_g != 0 && cost >= (rows < p.B1 ? kTailGain : 1.0) * best_cost) return;
        best_g = g; best_cost = cost; best_stages = stages; best_qbuf = qbuf; best_split = split;
        best_rows = rows;
      };
      offer(dealt_cost(groups * per_group, main_cost, 0, 0.0, ctas), p.B1);
      // A last round that is not full: the rows from some row on go to items of two rows (256 rows of 64 channels, 512 items
      // of four rows in four rounds -> 440 and 144 of two: 57.9 -> 54.5 us a module call).  One row would leave a warpgroup
      // without work, three take as long as four.
      const long long rounds = groups * per_group / ctas;
      for (long long r = rounds; r >= 1 && r >= rounds - 1 && g_req == 0 && g > kTailRows; --r) {
        const long long main_groups = r * ctas / per_group, rows = main_groups * g;
        if (main_groups < 1 || rows >= p.B1) continue;
        const long long tail = (p.B1 - rows + kTailRows - 1) / kTailRows * per_group;
        offer(dealt_cost(main_groups * per_group, main_cost, tail, item_cost(kTailRows, false, qbuf), ctas), rows);
      }
    }
  }
  if (best_g == 0) return AF3K_ERR_BAD_SHAPE;
  plan->cost = best_cost;
  p.G = best_g;
  p.q_split = best_split ? 1 : 0;
  p.n_streams = p.q_split ? 2 : p.G;
  p.kv_stages = best_stages;
  p.q_buffers = best_qbuf;
  p.tail_row = (int)best_rows;
  const long long per_group = (long long)p.B2 * tiles_of(best_split);
  const long long n_main = (best_rows + p.G - 1) / p.G * per_group, n_tail = (p.B1 - best_rows + kTailRows - 1) / kTailRows * per_group;
  if (n_main + n_tail > 0x7fffffff) return AF3K_ERR_BAD_SHAPE;
  p.n_main = (int)n_main;
  p.mixed = (n_tail != 0 || (p.q_split ? p.n_qt % 2 : p.B1 % p.G) != 0) ? 1 : 0;
  p.n_items = (int)(n_main + n_tail);
  p.div_q = make_divisor((uint32_t)tiles_of(best_split));
  p.div_h = make_divisor((uint32_t)p.B2);

  // (After the choice: the cost model compares such plans with two bias stages and the Q buffers it asked for.)
  // Streams that are query tiles bring a bias tile for each of their logits tiles (32 KB beside 16 KB of K and V), and with
  // two stages a load's latency was the time between two tiles: a third stage where K and V keep one more than that.  (Nothing
  // is gained where a lone query tile uses them, and the warps that convert an fp32 bias get slower: 512 tokens 10.7 -> 12.7 us.)
  // The Q tiles of a CTA's only item need no second buffer.  16 heads, bf16 bias, us, two stages -> three -> four: 1536 tokens
  // 29.1 -> 24.5 -> 26.0, 2048 tokens 35.0 -> 30.5 -> 31.4.
  p.bias_stages = kSharedBiasStages;
  if (p.q_split) {
    if (p.n_items <= ctas) p.q_buffers = 1;
    int lead = 0;
    for (int nb = kSharedBiasStages; nb <= kMaxBiasStages; ++nb) {
      int stages = (budget - fixed - (nb - kSharedBiasStages) * kBiasTileBytes - p.q_buffers * p.n_streams * (int)p.q_tile_bytes) / kv_stage;
      if (stages > kMaxKvStages) stages = kMaxKvStages;
      if (stages < 2) break;
      const int l = nb < stages - 1 ? nb : stages - 1;     // logits tiles whose operands can be under way
      if (l > lead) { lead = l; p.bias_stages = nb; p.kv_stages = stages; }
    }
  }

  uint32_t off = 0;
  p.off_q = off;      off += p.q_buffers * p.n_streams * p.q_tile_bytes;
  p.off_kv = off;     off += p.kv_stages * kv_stage;
  p.off_bias = off;   off += p.bias_stages * kBiasTileBytes;
  p.off_bar = off;    off += kBarrierBlockBytes;
  p.off_ones = off;   off += kMaskPanelBytes;
  p.off_mcol = off;   off += kMaxKvStages * kMaskPanelBytes;
  p.off_zero = off;   off += kMaskPanelBytes;
  p.off_ident = off;  off += kIdentBytes;
  size_t smem = off;
  // One CTA per SM is required (each CTA allocates all of TMEM): ask for more than half the SM's
  // shared memory even when the tiles need less.
  if (smem < 120 * 1024) smem = 120 * 1024;
  plan->smem_bytes = smem;
  plan->grid = p.n_items < ctas ? p.n_items : ctas;
  return AF3K_OK;
}

// Whether the attention kernel is to convert the bias itself (then *plan is one that can: one query tile of one pair row per item).
// It is where that is no slower on the device by these estimates, in us: the pass 1.6 and, for fp32 whose copy stays in L2, 8 TB/s,
// else 5; a lone tile of 128 keys 1.45, converted in place 1.65 (rows on vectors) or 2.2 (rows that start anywhere), and 1.2 for each such
// item; a tile of a pair of streams 1.6, at least 1.1.  A single key tile or rows on vectors cost a lone item less than any pass.
// Measured on the device, us, the way that is taken (the other); 16 heads, fp32 rows that start anywhere, unless said:
//   one query tile per item   here 129 tokens 6.7 (7.2), 389 10.4 (12.1), 1001 22.7 (28.4), bf16 22.2 (27.5); 8 heads of 700 14.0 (15.0); 4 heads
//                             of 129 6.5 (7.0), of 200 7.1 (7.5); the pass 4 heads of 1001 17.2 (18.2), 6 of 389 10.0 (10.3)
//   pairs of query tiles      here on vectors 1200 39.6 (43.1), 1536 46.5 (60.7), 2048 66 (96), anywhere 1301 52.7 (54.0), 2047 81 (106), bf16
//                             78 (89); the pass 1200 46.7 (48.3), 1301 bf16 43.7 (52.3), 1536 bf16 55.4 (57.5)
//   several pair rows         nearly always the pass: 4 heads of 100 rows 9.5 (11.8), of 140 rows of 32 keys 7.8 (10.6), 3 rows of 1000 tokens on vectors
//                             43.5 (46.3); in a graph 62 rows 6.7 (7.6)
// Several pair rows to an item: a short call is bound by its launches, which take the host 8.6 us with the pass and 5.9 without, so
// there up to kLaunchWorth us of the device's time are given for the one launch less (4 heads, 45 rows 8.7 -> 7.4 us a call, 62 rows 8.7 -> 7.7,
// 40 rows of 100 on vectors 8.7 -> 7.7; most on the device: 74 rows of 64 keys 6.7 -> 8.0), and nothing is under capture, where launches are the graph's.
// Below kFewItems ragged items the pass stays, although here would be faster up to 200 tokens (3 heads of 131: 7.0, here 6.5): no call in
// use has fewer than four heads.
constexpr int kFewItems = 8;
constexpr double kLaunchWorth = 1.2, kShortCall = 5.5;
constexpr double kL2Bytes = 126e6;
bool convert_in_kernel(const af3k_attention_desc& d, const DeviceInfo& dev, Plan* plan, bool wide, cudaStream_t stream) {
  const AttnParams& p = plan->p;
  const bool lone = p.n_streams == 1 && !p.mixed;
  if (lone && (wide || p.n_kt == 1)) return true;
  if (lone && p.n_items < kFewItems) return false;
  Plan other;
  if (!lone && (d.rows_per_item > 1 || make_plan(d, dev, &other, true, true) != AF3K_OK || other.p.mixed)) return false;
  const Plan& l = lone ? *plan : other;
  const double es = d.bias_dtype == AF3K_F32 ? 4 : 2, elements = (double)d.B2 * d.Sq * d.Sk, bytes = elements * (es + 2);
  const double pass = 1.6 + bytes / (es == 4 && bytes < kL2Bytes ? 8e6 : 5e6);
  const double tiles = std::max(((p.n_kt - 1) * p.kw + plan->last_w) / (double)kTile, 0.5), width = tiles / p.n_kt;     // key tiles of 128
  const auto lone_items = [&](double tile) { return ((l.p.n_items + l.grid - 1) / l.grid) * (tiles * tile + 1.2); };
  const double reads = d.B1 * elements * es / 5e6;      // each pair row reads the whole bias
  const double here = std::max(lone_items(wide ? 1.65 : 2.2), reads);
  const double there = pass + (lone ? lone_items(1.45) : plan->cost * std::max(1.6 * width, 1.1));
  bool convert = here < (lone ? 1.0 : 0.98) * there;      // (plans that are given up have to be beaten by this much)
  if (!convert && p.G > 1 && there < kShortCall && here - there <= kLaunchWorth) {
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(stream, &capture) != cudaSuccess) (void)cudaGetLastError();
    convert = capture == cudaStreamCaptureStatusNone;
  }
  if (convert && !lone) *plan = other;
  return convert;
}

int encode_qkv_map(CUtensorMap* tm, const void* base, bool fp8, int64_t D, int64_t S, int64_t B2,
                   int64_t B1, const int64_t* stride, int row_bytes, int rows) {   // row_bytes, rows: of the box
  auto enc = tensor_map_encoder();
  if (!enc) return driver_fail("cuTensorMapEncodeTiled entry point", -1);
  const uint64_t es = fp8 ? 1 : 2;
  cuuint64_t dims[4] = {(cuuint64_t)D, (cuuint64_t)S, (cuuint64_t)B2, (cuuint64_t)B1};
  cuuint64_t strides[3] = {(cuuint64_t)stride[2] * es, (cuuint64_t)stride[1] * es,
                           (cuuint64_t)stride[0] * es};
  // a dimension of extent 1 may carry any stride; TMA still wants it non-zero and 16-aligned
  for (int i = 0; i < 3; ++i)
    if (strides[i] == 0) strides[i] = 16;
  cuuint32_t box[4] = {(cuuint32_t)(row_bytes / es), (cuuint32_t)rows, 1, 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  CUresult r = enc(tm, fp8 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4,
                   const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                   swizzle_for(row_bytes), CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? AF3K_OK : driver_fail("cuTensorMapEncodeTiled(q/k/v)", (int)r);
}

int encode_bias_map(CUtensorMap* tm, const void* base, int64_t Sk, int64_t Sq, int64_t B2,
                    int64_t stride_h, int64_t stride_r) {
  auto enc = tensor_map_encoder();
  if (!enc) return driver_fail("cuTensorMapEncodeTiled entry point", -1);
  cuuint64_t dims[3] = {(cuuint64_t)Sk, (cuuint64_t)Sq, (cuuint64_t)B2};
  cuuint64_t strides[2] = {(cuuint64_t)stride_r * 2, (cuuint64_t)stride_h * 2};
  for (int i = 0; i < 2; ++i)
    if (strides[i] == 0) strides[i] = 16;
  cuuint32_t box[3] = {64, (cuuint32_t)kTile, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = enc(tm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides,
                   box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? AF3K_OK : driver_fail("cuTensorMapEncodeTiled(bias)", (int)r);
}

__global__ void wait_timeout_selftest_kernel(long long limit, int* status) {
  __shared__ __align__(8) unsigned long long bar;
  __shared__ int abort_flag;
  if (threadIdx.x == 0) {
    abort_flag = 0;
    af3k::mbar_init(af3k::smem_u32(&bar), 1);
    af3k::fence_barrier_init();
    // nothing ever arrives on `bar`: the bounded wait must give up and report
    const bool ok = af3k::mbar_wait_bounded(af3k::smem_u32(&bar), 0, limit, &abort_flag);
    if (!ok && status != nullptr) atomicOr(status, (int)af3k::kStatusWaitTimeout);
    af3k::mbar_inval(af3k::smem_u32(&bar));
  }
}

// ---------------------------------------------------------------------------------------------
// Variant for callers that have no way to hand us scratch memory.
//
// The bf16 staging copy of the bias normally lives in a caller-provided workspace.  Some hosts
// cannot provide one: a serving process that gave every byte of device memory to its own arena
// at start-up, a plug-in interface that only passes inputs and outputs through, or a
// latency-critical loop in which cudaMalloc (which synchronises the device) is forbidden.  For
// them the staging copy goes into a fixed array that is part of this library's device image.
// The array is reserved on every GPU that loads the library, for the life of the process, so
// its size is kept modest.
constexpr size_t kStaticScratchBytes = 16u << 20;   // 16 MiB: B2 * Sq * round_up(Sk, 8) <= 8 Mi entries
static __device__ __align__(256) unsigned char g_static_bias_scratch[kStaticScratchBytes];

// In host code the name of a __device__ array is only a handle for the runtime, not an address
// the GPU can use; the real device address has to be asked for, per device.
int static_scratch_address(void** out) {
  static void* addr[64] = {nullptr};
  static std::mutex mu;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || dev < 0 || dev >= 64) return cuda_fail("cudaGetDevice", e);
  std::lock_guard<std::mutex> lock(mu);
  if (addr[dev] == nullptr) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_static_bias_scratch);   // resolves for the current device
    if (e != cudaSuccess || p == nullptr) return cuda_fail("cudaGetSymbolAddress(static scratch)", e);
    addr[dev] = p;
  }
  *out = addr[dev];
  return AF3K_OK;
}

}  // namespace

extern "C" {

int af3k_version(void) { return 1006; }

const char* af3k_strerror(int code) {
  switch (code) {
    case AF3K_OK: return "ok";
    case AF3K_ERR_BAD_DTYPE: return "unsupported element type";
    case AF3K_ERR_BAD_SHAPE: return "unsupported shape (D must be a multiple of 8 and <= 64; Sk > 0)";
    case AF3K_ERR_BAD_STRIDE: return "unsupported stride (innermost must be 1, others 16-byte multiples)";
    case AF3K_ERR_BAD_ALIGNMENT: return "pointer is not 16-byte aligned";
    case AF3K_ERR_WORKSPACE: return "workspace missing or too small";
    case AF3K_ERR_NULL_POINTER: return "null pointer";
    case AF3K_ERR_CUDA: return "CUDA runtime or driver call failed";
    case AF3K_ERR_UNSUPPORTED_DEVICE: return "device is not compute capability 10.x (B200)";
    case AF3K_ERR_SCRATCH_LIMIT: return "problem needs more scratch than the built-in array holds";
    default: return "unknown error code";
  }
}

size_t af3k_dot_product_attention_workspace(const af3k_attention_desc* desc, const void* bias) {
  if (desc == nullptr || validate(*desc) != AF3K_OK) return 0;
  // fp8 q/k: the staging copy is what lets the tensor core add the bias (optional, see the entry)
  if (!bias_needs_staging(*desc, bias) && (desc->qk_dtype != AF3K_FP8_E4M3 || desc->bias_prescaled)) return 0;
  return (size_t)desc->B2 * desc->Sq * staged_bias_pitch(desc->Sk) * 2;
}

int af3k_last_launch_count(void) { return t_last_launches; }

const char* af3k_last_error_detail(void) { return t_detail; }

void af3k_set_wait_limit_cycles(long long cycles) { g_wait_limit.store(cycles > 0 ? cycles : -1); }

namespace {
int launch_bias_staging(const af3k_attention_desc& d, const DeviceInfo& dev, const void* bias, const float* sq,
                        const float* sk, void* staged, cudaStream_t stream) {
  const int64_t pitch = staged_bias_pitch(d.Sk);
  const bool f32 = d.bias_dtype == AF3K_F32;
  const bool pieces = f32 && ((reinterpret_cast<uintptr_t>(bias) | (uintptr_t)d.bias_stride[0] * 4 | (uintptr_t)d.bias_stride[1] * 4) & 15u) != 0;
  const long long total = (long long)d.B2 * d.Sq * (pieces ? (pitch + 255) / 256 * 32 : pitch / 8);      // threads
  long long blocks = (total + kBiasThreads - 1) / kBiasThreads;
  if (blocks > dev.sm_count * 8) blocks = dev.sm_count * 8;
  const auto launch = [&](auto kernel, auto* src) {
    launch_overlapped(kernel, dim3((unsigned)blocks), kBiasThreads, 0, stream, d.max_ctas <= 0, src, static_cast<__nv_bfloat16*>(staged), (int)d.B2,
                      (int)d.Sq, (int)d.Sk, (long long)d.bias_stride[0], (long long)d.bias_stride[1], (int)pitch, sq, sk, d.softmax_scale);
  };
  if (!f32)        launch(bias_to_bf16_kernel<__nv_bfloat16, false>, static_cast<const __nv_bfloat16*>(bias));
  else if (pieces) launch(bias_to_bf16_kernel<float, true>, static_cast<const float*>(bias));
  else             launch(bias_to_bf16_kernel<float, false>, static_cast<const float*>(bias));
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? AF3K_OK : cuda_fail("launch bias_to_bf16_kernel", e);
}
}  // namespace

int af3k_stage_bias(const af3k_attention_desc* desc, const void* bias, const float* q_scale,
                    const float* k_scale, void* staged, size_t staged_bytes, void* stream_v) {
  t_last_launches = 0;
  if (desc == nullptr) return AF3K_ERR_NULL_POINTER;
  af3k_attention_desc d = *desc;
  d.bias_prescaled = 0;      // describes the input bias here
  int rc = validate(d);
  if (rc != AF3K_OK) return rc;
  if (d.B2 == 0 || d.Sq == 0) return AF3K_OK;
  if (!bias || !staged) return AF3K_ERR_NULL_POINTER;
  if ((q_scale != nullptr) != (k_scale != nullptr)) return AF3K_ERR_BAD_DTYPE;
  if (q_scale != nullptr && d.qk_dtype != AF3K_FP8_E4M3) return AF3K_ERR_BAD_DTYPE;
  if (!aligned16(staged)) return AF3K_ERR_BAD_ALIGNMENT;
  if (staged_bytes < (size_t)d.B2 * d.Sq * staged_bias_pitch(d.Sk) * 2) return AF3K_ERR_WORKSPACE;
  DeviceInfo* dev = nullptr;
  if ((rc = device_info(&dev)) != AF3K_OK) return rc;
  rc = launch_bias_staging(d, *dev, bias, q_scale, k_scale, staged, reinterpret_cast<cudaStream_t>(stream_v));
  if (rc == AF3K_OK) t_last_launches = 1;
  return rc;
}

namespace {
// convert: the kernel itself may convert the bias
int attention_call(const af3k_attention_desc* desc, const void* q, const void* k, const void* v, const void* bias, const uint8_t* mask, void* out,
                   const float* q_scale, const float* k_scale, void* workspace, size_t workspace_bytes, int* status_dev, void* stream_v, bool convert) {
  t_last_launches = 0;
  if (desc == nullptr) return AF3K_ERR_NULL_POINTER;
  const af3k_attention_desc& d = *desc;
  int rc = validate(d);
  if (rc != AF3K_OK) return rc;
  if (d.B1 == 0 || d.B2 == 0 || d.Sq == 0) return AF3K_OK;  // empty output
  if (!q || !k || !v || !bias || !out) return AF3K_ERR_NULL_POINTER;
  const bool fp8 = d.qk_dtype == AF3K_FP8_E4M3;
  if (fp8 != (q_scale != nullptr) || fp8 != (k_scale != nullptr)) return AF3K_ERR_BAD_DTYPE;
  if (!aligned16(q) || !aligned16(k) || !aligned16(v) || !aligned16(out)) return AF3K_ERR_BAD_ALIGNMENT;

  DeviceInfo* dev = nullptr;
  rc = device_info(&dev);
  if (rc != AF3K_OK) return rc;
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_v);

  // fp8 q/k run the tensor-core-bias kernel when the bias is (or can be) staged pre-divided by
  // the logit scale; bf16 q/k always do
  const bool fp8_with_tc_bias = fp8 && (d.bias_prescaled ||
      (workspace != nullptr && aligned16(workspace) &&
       workspace_bytes >= (size_t)d.B2 * d.Sq * staged_bias_pitch(d.Sk) * 2));
  Plan plan;
  rc = make_plan(d, *dev, &plan, !fp8 || fp8_with_tc_bias);
  if (rc != AF3K_OK) return rc;
  AttnParams& p = plan.p;
  if (plan.smem_bytes > (size_t)(dev->max_smem_optin - kStaticSmemReserve)) return AF3K_ERR_BAD_SHAPE;

  // bias: use in place when TMA can address it, else stage a bf16 copy in the workspace
  const void* bias_base = bias;
  int64_t bias_sh = d.bias_stride[0], bias_sr = d.bias_stride[1];
  int launches = 0;
  // fp8 q/k: with a staging copy divided by the head's logit scale the tensor core adds the bias
  // to the raw fp8 products (the fast kernel); without room for one the softmax threads add the
  // bias in fp32 as before
  const size_t stage_bytes = (size_t)d.B2 * d.Sq * staged_bias_pitch(d.Sk) * 2;
  const bool must_stage = bias_needs_staging(d, bias);
  if (d.bias_prescaled && must_stage) return AF3K_ERR_BAD_STRIDE;   // a staged copy is TMA-addressable by construction
  const bool stage_fp8 = fp8 && !d.bias_prescaled && workspace != nullptr && workspace_bytes >= stage_bytes &&
                         aligned16(workspace);
  const bool fp8_tc = fp8 && (d.bias_prescaled || stage_fp8);
  // the kernel converts the bias itself: items of one query tile
  const uintptr_t bias_es = d.bias_dtype == AF3K_F32 ? 4 : 2;
  const bool wide = d.Sk % 4 == 0 && (reinterpret_cast<uintptr_t>(bias) | (uintptr_t)bias_sh * bias_es | (uintptr_t)bias_sr * bias_es) % (4 * bias_es) == 0;
  const bool in_kernel = convert && must_stage && !fp8 && p.debug == nullptr && convert_in_kernel(d, *dev, &plan, wide, stream);
  p.bias_wide = wide ? 1 : 0;
  if ((must_stage && !in_kernel) || stage_fp8) {
    if (workspace == nullptr || workspace_bytes < stage_bytes) return AF3K_ERR_WORKSPACE;
    if (!aligned16(workspace)) return AF3K_ERR_BAD_ALIGNMENT;
    const int64_t pitch = staged_bias_pitch(d.Sk);
    if ((rc = launch_bias_staging(d, *dev, bias, stage_fp8 ? q_scale : nullptr, stage_fp8 ? k_scale : nullptr,
                                  workspace, stream)) != AF3K_OK)
      return rc;
    ++launches;
    bias_base = workspace;
    bias_sr = pitch;
    bias_sh = pitch * d.Sq;
  }

  CUtensorMap tm_q, tm_k, tm_v, tm_b{};
  if ((rc = encode_qkv_map(&tm_q, q, fp8, d.D, d.Sq, d.B2, d.B1, d.q_stride, p.qk_row_bytes, kTile))) return rc;
  if ((rc = encode_qkv_map(&tm_k, k, fp8, d.D, d.Sk, d.B2, d.B1, d.k_stride, p.qk_row_bytes, p.kw))) return rc;
  if ((rc = encode_qkv_map(&tm_v, v, false, d.D, d.Sk, d.B2, d.B1, d.v_stride, p.v_row_bytes, p.kw))) return rc;
  CUtensorMap tm_q2{}, tm_k2{};
  if (p.qk_narrow && ((rc = encode_qkv_map(&tm_q2, q, fp8, d.D, d.Sq, d.B2, d.B1, d.q_stride, 32, kTile)) ||
                      (rc = encode_qkv_map(&tm_k2, k, fp8, d.D, d.Sk, d.B2, d.B1, d.k_stride, 32, p.kw))))
    return rc;
  if (in_kernel) {
    p.bias_src = bias;
    p.bias_stride_h = bias_sh;
    p.bias_stride_r = bias_sr;
    p.bias_f32 = bias_es == 4 ? 1 : 0;
  } else if ((rc = encode_bias_map(&tm_b, bias_base, d.Sk, d.Sq, d.B2, bias_sh, bias_sr))) return rc;

  p.q_scale = q_scale;
  p.k_scale = k_scale;
  p.mask = mask;
  p.mask_row_stride = d.mask_row_stride;
  p.mask_col = (mask != nullptr || d.Sk != (int64_t)(p.n_kt - 1) * p.kw + plan.last_w) ? 1 : 0;
  p.out = static_cast<__nv_bfloat16*>(out);
  p.out_stride_b1 = d.out_stride[0];
  p.out_stride_b2 = d.out_stride[1];
  p.out_stride_s = d.out_stride[2];
  p.gate = static_cast<const __nv_bfloat16*>(d.gate);
  p.gate_stride_b1 = d.gate_stride[0];
  p.gate_stride_b2 = d.gate_stride[1];
  p.gate_stride_s = d.gate_stride[2];
  p.status = status_dev;
  p.wait_limit = wait_limit_cycles();

  // scale, bias and mask all come out of the tensor core, except for fp8 q/k without a staging
  // copy of the bias: there the softmax threads apply scale and bias in fp32
  const bool tc_bias = !fp8 || fp8_tc;
  p.scale_q = (fp8 || d.softmax_scale == 1.0f) ? 0 : 1;   // a scale of exactly 1 (q already scaled by its producer) needs no pass over Q
  const bool dbg = p.debug != nullptr;
  const auto launch = [&](auto kernel) {
    launch_overlapped(kernel, dim3(plan.grid), in_kernel ? kConvertThreads : kThreads, plan.smem_bytes, stream, d.max_ctas <= 0, p, tm_q, tm_k, tm_v, tm_b, tm_q2, tm_k2);
  };
  if (in_kernel) {
    if (p.gate != nullptr) with_width<false, true, false, true>(p.kw, plan.last_w, launch);
    else                   with_width<false, false, false, true>(p.kw, plan.last_w, launch);
  } else if (dbg && p.gate == nullptr) {
    if (!fp8)         launch(attention_kernel<true, true, false, false, true>);
    else if (tc_bias) launch(attention_kernel<true, true, true, false, true>);
    else              launch(attention_kernel<true, false, true, false, true>);
  } else if (!fp8) {
    if (p.gate != nullptr) { if (p.mixed) with_width<false, true, true, false>(p.kw, plan.last_w, launch);  else with_width<false, true, false, false>(p.kw, plan.last_w, launch); }
    else                   { if (p.mixed) with_width<false, false, true, false>(p.kw, plan.last_w, launch); else with_width<false, false, false, false>(p.kw, plan.last_w, launch); }
  } else if (p.gate != nullptr) {
    if (tc_bias) { if (p.mixed) launch(attention_kernel<false, true, true, true, true>);  else launch(attention_kernel<false, true, true, true, false>); }
    else         { if (p.mixed) launch(attention_kernel<false, false, true, true, true>); else launch(attention_kernel<false, false, true, true, false>); }
  } else if (tc_bias) {
    if (p.mixed) with_width<true, false, true, false>(p.kw, plan.last_w, launch); else with_width<true, false, false, false>(p.kw, plan.last_w, launch);
  } else {
    if (p.mixed) launch(attention_kernel<false, false, true, false, true>); else launch(attention_kernel<false, false, true, false, false>);
  }
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail("launch attention_kernel", e);
  ++launches;
  t_last_launches = launches;
  return AF3K_OK;
}

}  // namespace

int af3k_dot_product_attention(const af3k_attention_desc* desc, const void* q, const void* k,
                               const void* v, const void* bias, const uint8_t* mask, void* out,
                               const float* q_scale, const float* k_scale, void* workspace,
                               size_t workspace_bytes, int* status_dev, void* stream) {
  return attention_call(desc, q, k, v, bias, mask, out, q_scale, k_scale, workspace, workspace_bytes, status_dev, stream, false);
}

int af3k_dot_product_attention_convert(const af3k_attention_desc* desc, const void* q, const void* k, const void* v, const void* bias,
                                       const uint8_t* mask, void* out, int* status_dev, void* stream) {
  return attention_call(desc, q, k, v, bias, mask, out, nullptr, nullptr, nullptr, 0, status_dev, stream, true);
}

void af3k_debug_set_dump(float* dump_dev) { g_debug_dump.store(dump_dev); }

static int describe(const af3k_attention_desc* desc, Plan* plan) {
  if (desc == nullptr) return AF3K_ERR_NULL_POINTER;
  int rc = validate(*desc);
  if (rc != AF3K_OK) return rc;
  DeviceInfo dev;
  dev.sm_count = 148;
  dev.cc_major = 10;
  dev.max_smem_optin = 232448;
  int cur = 0;
  cudaDeviceProp prop;
  if (cudaGetDevice(&cur) == cudaSuccess && cudaGetDeviceProperties(&prop, cur) == cudaSuccess &&
      prop.major == 10) {
    dev.sm_count = prop.multiProcessorCount;
    dev.max_smem_optin = (int)prop.sharedMemPerBlockOptin;
  }
  return make_plan(*desc, dev, plan);
}

int af3k_describe_plan(const af3k_attention_desc* desc, int32_t* out6) {
  Plan plan;
  int rc = out6 == nullptr ? AF3K_ERR_NULL_POINTER : describe(desc, &plan);
  if (rc != AF3K_OK) return rc;
  out6[0] = plan.p.G;
  out6[1] = plan.p.kv_stages;
  out6[2] = plan.p.n_items;
  out6[3] = plan.grid;
  out6[4] = (int32_t)plan.smem_bytes;
  out6[5] = (int32_t)kOCol + plan.p.n_streams * plan.p.nv;
  return AF3K_OK;
}

int af3k_describe_plan_streams(const af3k_attention_desc* desc, int32_t* out4) {
  Plan plan;
  int rc = out4 == nullptr ? AF3K_ERR_NULL_POINTER : describe(desc, &plan);
  if (rc != AF3K_OK) return rc;
  out4[0] = plan.p.n_streams;
  out4[1] = plan.p.q_split;
  out4[2] = plan.p.q_buffers;
  out4[3] = plan.p.bias_stages;
  return AF3K_OK;
}

size_t af3k_static_scratch_bytes(void) { return kStaticScratchBytes; }

int af3k_dot_product_attention_noalloc(const af3k_attention_desc* desc, const void* q,
                                       const void* k, const void* v, const void* bias,
                                       const uint8_t* mask, void* out, const float* q_scale,
                                       const float* k_scale, int* status_dev, void* stream) {
  if (desc == nullptr) return AF3K_ERR_NULL_POINTER;
  int rc = validate(*desc);
  if (rc != AF3K_OK) return rc;
  // the staging copy is required for a bias TMA cannot read in place, optional (faster kernel)
  // for fp8 q/k: an optional copy that does not fit is simply not made
  size_t need = af3k_dot_product_attention_workspace(desc, bias);
  if (need > kStaticScratchBytes && !bias_needs_staging(*desc, bias)) need = 0;
  if (need > kStaticScratchBytes) {
    std::snprintf(t_detail, sizeof(t_detail),
                  "bias staging copy needs %zu bytes, the built-in scratch holds %zu", need,
                  kStaticScratchBytes);
    return AF3K_ERR_SCRATCH_LIMIT;
  }
  // the device check comes first, so that a GPU this library has no code for is reported as
  // such and not as a failed symbol lookup
  DeviceInfo* dev = nullptr;
  if ((rc = device_info(&dev)) != AF3K_OK) return rc;
  void* scratch = nullptr;
  if (need != 0 && (rc = static_scratch_address(&scratch)) != AF3K_OK) return rc;
  // From here on this is the ordinary call with the built-in array as its workspace.  The
  // staging pre-pass rewrites every entry it later reads (pad columns included), so nothing of a
  // previous call's contents needs clearing.
  return af3k_dot_product_attention(desc, q, k, v, bias, mask, out, q_scale, k_scale, scratch,
                                    need != 0 ? kStaticScratchBytes : 0, status_dev, stream);
}

int af3k_pair_bias(const void* pair, int32_t pair_dtype, int64_t R, int64_t N, int64_t C, int64_t H,
                   const float* gamma, const float* beta, const float* proj, float eps, void* normed,
                   void* bias, int64_t bias_pitch, void* stream_v) {
  t_last_launches = 0;
  if (pair_dtype != AF3K_BF16 && pair_dtype != AF3K_F32) return AF3K_ERR_BAD_DTYPE;
  if (C != kPbChannels || H < 1 || H > kPbMaxHeads || R < 0 || N < 0 || R > 0x7fffffff || N > 0x7fffffff)
    return AF3K_ERR_BAD_SHAPE;
  if (bias_pitch < N || (bias_pitch & 7) != 0) return AF3K_ERR_BAD_STRIDE;
  if (R == 0 || N == 0) return AF3K_OK;
  if (!pair || !gamma || !beta || !proj || !normed || !bias) return AF3K_ERR_NULL_POINTER;
  if (!aligned16(pair) || !aligned16(normed) || !aligned16(bias)) return AF3K_ERR_BAD_ALIGNMENT;
  DeviceInfo* dev = nullptr;
  int rc = device_info(&dev);
  if (rc != AF3K_OK) return rc;
  PairBiasParams p;
  p.pair = pair; p.normed = static_cast<__nv_bfloat16*>(normed); p.bias = static_cast<__nv_bfloat16*>(bias);
  p.gamma = gamma; p.beta = beta; p.proj = proj;
  p.R = (int)R; p.N = (int)N; p.H = (int)H; p.bias_pitch = bias_pitch; p.eps = eps;
  // persistent CTAs (two per SM for the 4-head kernel, one for the wide ones) over R * ceil(N / 128) tiles
  const long long n_tiles = R * ((N + kPbTileJ - 1) / kPbTileJ);
  const long long max_ctas = (long long)dev->sm_count * (H <= 4 ? 2 : 1);
  const unsigned grid = (unsigned)(n_tiles < max_ctas ? n_tiles : max_ctas);
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_v);
  const bool f32 = pair_dtype == AF3K_F32;
#ifndef AF3K_PB_MMA_MIN_HEADS
#define AF3K_PB_MMA_MIN_HEADS 5
#endif
  if (!f32 && H >= AF3K_PB_MMA_MIN_HEADS) {
    // bf16 pair, more than four heads: moments and normalisation per thread, the head projection on
    // the tensor core (its time does not depend on the head count)
    const long long cap = (long long)dev->sm_count * 5;
    const unsigned grid_m = (unsigned)(n_tiles < cap ? n_tiles : cap);
    pair_bias_mma_kernel<<<grid_m, kPbmRows, kPbmSmemBytes, stream>>>(p, wait_limit_cycles());
  } else if (H <= 4) {
    // one thread per vector, tiles transposed through shared memory; five CTAs fit an SM
    const long long tiles_t = R * ((N + (f32 ? 64 : 128) - 1) / (f32 ? 64 : 128));
    const long long cap = (long long)dev->sm_count * 5;
    const unsigned grid_t = (unsigned)(tiles_t < cap ? tiles_t : cap);
    if (f32) pair_bias_kernel_t<float><<<grid_t, PbTile<float>::kRows, PbTile<float>::kSmemBytes, stream>>>(p);
    else     pair_bias_kernel_t<__nv_bfloat16><<<grid_t, PbTile<__nv_bfloat16>::kRows,
                                                PbTile<__nv_bfloat16>::kSmemBytes, stream>>>(p);
  } else if (H <= 8) {
    if (f32) pair_bias_kernel<float, 8><<<grid, kPbThreads, 0, stream>>>(p);
    else     pair_bias_kernel<__nv_bfloat16, 8><<<grid, kPbThreads, 0, stream>>>(p);
  } else {
    if (f32) pair_bias_kernel<float, 16><<<grid, kPbThreads, 0, stream>>>(p);
    else     pair_bias_kernel<__nv_bfloat16, 16><<<grid, kPbThreads, 0, stream>>>(p);
  }
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail("launch pair_bias_kernel", e);
  t_last_launches = 1;
  return AF3K_OK;
}

int af3k_pair_bias_status(int32_t* out4) {
  if (out4 == nullptr) return AF3K_ERR_NULL_POINTER;
  int host[4] = {0, 0, 0, 0};
  cudaError_t e = cudaMemcpyFromSymbol(host, g_pair_bias_status, sizeof(host));
  if (e != cudaSuccess) return cuda_fail("cudaMemcpyFromSymbol(pair-bias status)", e);
  for (int i = 0; i < 4; ++i) out4[i] = host[i];
  if (host[0] != 0) {
    const int zero[4] = {0, 0, 0, 0};
    if ((e = cudaMemcpyToSymbol(g_pair_bias_status, zero, sizeof(zero))) != cudaSuccess)
      return cuda_fail("cudaMemcpyToSymbol(pair-bias status)", e);
  }
  return AF3K_OK;
}

}  // extern "C"

namespace {
int encode_weight_map(CUtensorMap* tm, const void* w, int64_t C, int64_t rows) {
  auto enc = tensor_map_encoder();
  if (!enc) return driver_fail("cuTensorMapEncodeTiled entry point", -1);
  cuuint64_t dims[2] = {(cuuint64_t)C, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)C * 2};
  cuuint32_t box[2] = {64, 64};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = enc(tm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(w), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? AF3K_OK : driver_fail("cuTensorMapEncodeTiled(weights)", (int)r);
}

template <int C>
void launch_front(const GridParams& p, const FrontMaps& tm, unsigned grid, bool f32, bool ln, cudaStream_t stream) {
  const uint32_t smem = f32 ? FrontTile<C, float>::kSmem : FrontTile<C, __nv_bfloat16>::kSmem;
  constexpr int kThreads = FrontTile<C, float>::kThreads;
  if (!ln)      launch_overlapped(grid_front_kernel<C, __nv_bfloat16, false>, dim3(grid), kThreads, smem, stream, true, p, tm);
  else if (f32) launch_overlapped(grid_front_kernel<C, float, true>, dim3(grid), kThreads, smem, stream, true, p, tm);
  else          launch_overlapped(grid_front_kernel<C, __nv_bfloat16, true>, dim3(grid), kThreads, smem, stream, true, p, tm);
}
}  // namespace

extern "C" {

int af3k_grid_front_weights(const void* pair, int32_t pair_dtype, const af3k_front_weights* weights, float eps, int64_t Hb, int64_t R,
                            int64_t N, int64_t C, int64_t H, float q_scale, int32_t transpose, void* bias, int64_t bias_pitch, void* q,
                            void* k, void* v, void* gate, int* status_dev, void* stream_v) {
  t_last_launches = 0;
  if (weights == nullptr) return AF3K_ERR_NULL_POINTER;
  const af3k_front_weights& w = *weights;
  const bool ln = w.gamma != nullptr;
  if (pair_dtype != AF3K_BF16 && !(pair_dtype == AF3K_F32 && ln)) return AF3K_ERR_BAD_DTYPE;
  for (int32_t t : {w.w_dtype, w.ln_dtype, w.bias_w_dtype})
    if (t != AF3K_BF16 && t != AF3K_F32) return AF3K_ERR_BAD_DTYPE;
  if (C != 64 && C != 128) return AF3K_ERR_BAD_SHAPE;
  if (R < 0 || N < 0 || H < 1 || C % H != 0 || (C / H) % 8 != 0 || Hb < 0 || Hb > 4 || (Hb > 0 && !ln)) return AF3K_ERR_BAD_SHAPE;
  if (R > 0x7fffffff || N > 0x7fffffff || (R > 0 && N > 0x7fffffffLL / C / R)) return AF3K_ERR_BAD_SHAPE;   // 32-bit element offsets
  if (Hb > 0 && (bias_pitch < N || (bias_pitch & 7) != 0)) return AF3K_ERR_BAD_STRIDE;
  if (R == 0 || N == 0) return AF3K_OK;
  if (!pair || !q || !k || !v || !gate || (ln && !w.beta) || (Hb > 0 && (!w.bias_w || !bias))) return AF3K_ERR_NULL_POINTER;
  for (const void* m : w.w)
    if (!m) return AF3K_ERR_NULL_POINTER;
  for (const void* ptr : {pair, w.w[0], w.w[1], w.w[2], w.w[3], (const void*)q, (const void*)k, (const void*)v, (const void*)gate})
    if (!aligned16(ptr)) return AF3K_ERR_BAD_ALIGNMENT;
  if (Hb > 0 && !aligned16(bias)) return AF3K_ERR_BAD_ALIGNMENT;
  DeviceInfo* dev = nullptr;
  int rc = device_info(&dev);
  if (rc != AF3K_OK) return rc;
  FrontMaps tm{};
  for (int i = 0; i < 4 && w.w_dtype == AF3K_BF16; ++i)
    if ((rc = encode_weight_map(&tm.w[i], w.w[i], C, C)) != AF3K_OK) return rc;
  GridParams p;
  std::memset(&p, 0, sizeof(p));
  p.M = R * N; p.R = (int)R; p.N = (int)N; p.H = (int)H; p.D = (int)(C / H); p.transpose = transpose ? 1 : 0;
  for (int i = 0; i < 4; ++i) p.w[i] = w.w[i];
  p.w_f32 = w.w_dtype == AF3K_F32 ? 1 : 0;
  p.q_scale = q_scale; p.pair = pair; p.gamma = w.gamma; p.beta = w.beta; p.ln_f32 = w.ln_dtype == AF3K_F32 ? 1 : 0;
  p.bias_w = w.bias_w; p.bias_w_f32 = w.bias_w_dtype == AF3K_F32 ? 1 : 0; p.eps = eps; p.Hb = (int)Hb;
  p.bias = static_cast<__nv_bfloat16*>(bias); p.bias_pitch = bias_pitch;
  p.q = static_cast<__nv_bfloat16*>(q); p.k = static_cast<__nv_bfloat16*>(k);
  p.v = static_cast<__nv_bfloat16*>(v); p.g = static_cast<__nv_bfloat16*>(gate);
  p.status = status_dev; p.wait_limit = wait_limit_cycles();
  // Few tiles: several CTAs take a tile, each a part of the output columns (and the weights' rows).  They
  // repeat the row work, which costs less than the part of the epilogue and of the weights' load it saves.
  const long long n_tiles = (p.M + 127) / 128;
  p.split = 1;
  while (p.split < (C == 128 ? 4 : 2) && n_tiles * p.split * 2 <= dev->sm_count) p.split *= 2;
  const long long ctas = n_tiles * p.split, most = dev->sm_count / p.split * p.split;
  const unsigned grid = (unsigned)(ctas < most ? ctas : most);
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_v);
  if (C == 128) launch_front<128>(p, tm, grid, pair_dtype == AF3K_F32, ln, stream);
  else          launch_front<64>(p, tm, grid, pair_dtype == AF3K_F32, ln, stream);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail("launch grid_front_kernel", e);
  t_last_launches = 1;
  return AF3K_OK;
}

int af3k_grid_front(const void* pair, int32_t pair_dtype, const float* gamma, const float* beta, float eps, const float* bias_w,
                    int64_t Hb, const void* w4, int64_t R, int64_t N, int64_t C, int64_t H, float q_scale, int32_t transpose,
                    void* bias, int64_t bias_pitch, void* q, void* k, void* v, void* gate, int* status_dev, void* stream_v) {
  if (Hb > 0 && bias_w && !aligned16(bias_w)) { t_last_launches = 0; return AF3K_ERR_BAD_ALIGNMENT; }
  af3k_front_weights w{};
  for (int i = 0; i < 4; ++i) w.w[i] = w4 ? static_cast<const char*>(w4) + (size_t)i * C * C * 2 : nullptr;
  w.gamma = gamma; w.beta = beta; w.bias_w = bias_w;
  w.w_dtype = AF3K_BF16;
  w.ln_dtype = w.bias_w_dtype = AF3K_F32;
  return af3k_grid_front_weights(pair, pair_dtype, &w, eps, Hb, R, N, C, H, q_scale, transpose, bias, bias_pitch, q, k, v, gate,
                                 status_dev, stream_v);
}

int af3k_grid_out_weights(const void* weighted, const void* gate, const void* wo, int32_t wo_dtype, void* out, int32_t out_dtype, int64_t M,
                          int64_t C, int* status_dev, void* stream_v) {
  t_last_launches = 0;
  for (int32_t t : {wo_dtype, out_dtype})
    if (t != AF3K_BF16 && t != AF3K_F32) return AF3K_ERR_BAD_DTYPE;
  if ((C != 64 && C != 128) || M < 0 || M > 0x7fffffff) return AF3K_ERR_BAD_SHAPE;
  if (M == 0) return AF3K_OK;
  if (!weighted || !gate || !wo || !out) return AF3K_ERR_NULL_POINTER;
  if (!aligned16(weighted) || !aligned16(gate) || !aligned16(wo) || !aligned16(out)) return AF3K_ERR_BAD_ALIGNMENT;
  DeviceInfo* dev = nullptr;
  int rc = device_info(&dev);
  if (rc != AF3K_OK) return rc;
  CUtensorMap tm{};
  if (wo_dtype == AF3K_BF16 && (rc = encode_weight_map(&tm, wo, C, C)) != AF3K_OK) return rc;
  GridParams p;
  std::memset(&p, 0, sizeof(p));
  p.w[0] = wo; p.w_f32 = wo_dtype == AF3K_F32 ? 1 : 0;
  p.M = M; p.weighted = static_cast<const __nv_bfloat16*>(weighted); p.gate = static_cast<const __nv_bfloat16*>(gate);
  p.out = out; p.status = status_dev; p.wait_limit = wait_limit_cycles();
  const long long n_tiles = (M + 127) / 128;
  const unsigned grid = (unsigned)(n_tiles < dev->sm_count ? n_tiles : dev->sm_count);
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_v);
  const bool f32 = out_dtype == AF3K_F32;
  if (C == 128) {
    if (f32) launch_overlapped(grid_out_kernel<128, float>, dim3(grid), OutTile<128>::kThreads, OutTile<128>::kSmem, stream, true, p, tm);
    else     launch_overlapped(grid_out_kernel<128, __nv_bfloat16>, dim3(grid), OutTile<128>::kThreads, OutTile<128>::kSmem, stream, true, p, tm);
  } else {
    if (f32) launch_overlapped(grid_out_kernel<64, float>, dim3(grid), OutTile<64>::kThreads, OutTile<64>::kSmem, stream, true, p, tm);
    else     launch_overlapped(grid_out_kernel<64, __nv_bfloat16>, dim3(grid), OutTile<64>::kThreads, OutTile<64>::kSmem, stream, true, p, tm);
  }
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail("launch grid_out_kernel", e);
  t_last_launches = 1;
  return AF3K_OK;
}

int af3k_grid_out(const void* weighted, const void* gate, const void* wo, void* out, int32_t out_dtype, int64_t M, int64_t C,
                  int* status_dev, void* stream_v) {
  return af3k_grid_out_weights(weighted, gate, wo, AF3K_BF16, out, out_dtype, M, C, status_dev, stream_v);
}

namespace {
int launch_pack(const af3k_matrix* w5, const af3k_matrix* bias_w, const void* gamma, const void* beta, int32_t ln_dtype, int64_t C,
                int64_t Hb, void* w4, void* wo, float* vec, const float* x, void* x_bf16, int64_t x_n, void* stream_v) {
  t_last_launches = 0;
  if (C < 1 || C > 1024 || Hb < 0 || Hb > 1024 || (Hb > 0 && bias_w == nullptr)) return AF3K_ERR_BAD_SHAPE;
  if (!w5 || !w4 || (w5[4].data && !wo) || ((gamma || beta || Hb > 0) && !vec)) return AF3K_ERR_NULL_POINTER;
  PackParams p;
  std::memset(&p, 0, sizeof(p));
  auto matrix = [](const af3k_matrix& m) { return PackMatrix{m.data, m.stride_out, m.stride_in, m.dtype == AF3K_F32 ? 1 : 0}; };
  for (int i = 0; i < 5; ++i) {
    if (!w5[i].data && i == 4) continue;           // a block without an output projection
    if (!w5[i].data) return AF3K_ERR_NULL_POINTER;
    if (w5[i].dtype != AF3K_F32 && w5[i].dtype != AF3K_BF16) return AF3K_ERR_BAD_DTYPE;
    p.w[i] = matrix(w5[i]);
  }
  if (Hb > 0) {
    if (bias_w->dtype != AF3K_F32 && bias_w->dtype != AF3K_BF16) return AF3K_ERR_BAD_DTYPE;
    p.bias_w = matrix(*bias_w);
  }
  p.gamma = gamma; p.beta = beta; p.ln_f32 = ln_dtype == AF3K_F32 ? 1 : 0;
  p.C = (int)C; p.Hb = (int)Hb;
  p.w4 = static_cast<__nv_bfloat16*>(w4); p.wo = static_cast<__nv_bfloat16*>(wo); p.vec = vec;
  const unsigned tiles = (unsigned)((C + kPackTile - 1) / kPackTile);
  unsigned slices = vec != nullptr ? 6 : (w5[4].data ? 5 : 4);
  if (x_n > 0) {
    p.x = reinterpret_cast<const float4*>(x); p.x_bf16 = static_cast<uint2*>(x_bf16); p.x_n4 = x_n / 4;
    const long long per_slice = (long long)tiles * tiles * kPackThreads * kPackXEach, more = (p.x_n4 + per_slice - 1) / per_slice;
    if (more > 65535 - kPackSlices) return AF3K_ERR_BAD_SHAPE;
    slices = kPackSlices + (unsigned)more;
  }
  launch_overlapped(grid_pack_kernel, dim3(tiles, tiles, slices), kPackThreads, 0, reinterpret_cast<cudaStream_t>(stream_v), true, p);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail("launch grid_pack_kernel", e);
  t_last_launches = 1;
  return AF3K_OK;
}
}  // namespace

int af3k_grid_pack(const af3k_matrix* w5, const af3k_matrix* bias_w, const void* gamma, const void* beta, int32_t ln_dtype,
                   int64_t C, int64_t Hb, void* w4, void* wo, float* vec, void* stream_v) {
  return launch_pack(w5, bias_w, gamma, beta, ln_dtype, C, Hb, w4, wo, vec, nullptr, nullptr, 0, stream_v);
}

int af3k_token_pack(const af3k_matrix* w4, int64_t C, void* w4_bf16, const float* x, int64_t M, void* x_bf16, void* stream_v) {
  t_last_launches = 0;
  if (!w4) return AF3K_ERR_NULL_POINTER;
  if (C < 4 || C % 4 != 0 || M < 0 || M > 0x7fffff00LL) return AF3K_ERR_BAD_SHAPE;
  if (M > 0 && (!x || !x_bf16)) return AF3K_ERR_NULL_POINTER;
  if (!aligned16(x) || !aligned16(x_bf16)) return AF3K_ERR_BAD_ALIGNMENT;
  af3k_matrix w5[5] = {w4[0], w4[1], w4[2], w4[3], {}};
  return launch_pack(w5, nullptr, nullptr, nullptr, AF3K_F32, C, 0, w4_bf16, nullptr, nullptr, x, x_bf16, M * C, stream_v);
}

int af3k_token_projection_weights(const void* x, const af3k_matrix* w4, const void* q_bias, int32_t q_bias_dtype, int64_t M, int64_t C,
                                  float q_scale, void* out, int* status_dev, void* stream_v) {
  t_last_launches = 0;
  if (q_bias && q_bias_dtype != AF3K_BF16 && q_bias_dtype != AF3K_F32) return AF3K_ERR_BAD_DTYPE;
  if (M < 0 || C < 8 || C % 8 != 0 || C > (1 << 20) || M > 0x7fffff00LL) return AF3K_ERR_BAD_SHAPE;
  if (M == 0) return AF3K_OK;
  if (!x || !w4 || !out) return AF3K_ERR_NULL_POINTER;
  if (!aligned16(x) || !aligned16(out)) return AF3K_ERR_BAD_ALIGNMENT;
  int mn_mask = 0;
  for (int i = 0; i < 4; ++i) {
    if (!w4[i].data) return AF3K_ERR_NULL_POINTER;
    if (w4[i].dtype != AF3K_BF16) return AF3K_ERR_BAD_DTYPE;
    if (!aligned16(w4[i].data)) return AF3K_ERR_BAD_ALIGNMENT;
    const bool mn = w4[i].stride_in != 1;
    const int64_t pitch = mn ? w4[i].stride_in : w4[i].stride_out;
    if ((mn && w4[i].stride_out != 1) || pitch < C || pitch % 8 != 0 || pitch >= (1LL << 38)) return AF3K_ERR_BAD_STRIDE;
    mn_mask |= mn << i;
  }
  DeviceInfo* dev = nullptr;
  int rc = device_info(&dev);
  if (rc != AF3K_OK) return rc;
  const int64_t m_tiles = (M + 127) / 128;
  // Columns of a tile: the narrowest that takes fewest rounds of one CTA per SM (64 with some SMs to spare).  Single block, us on the
  // device, 64 / 128 / 256: 384 channels 256 tokens 10.5 / 11.0 / 12.4, 1024 21.9 / 20.5 / 21.0, 2048 44.5 / 41.3 / 39.5; 768 channels
  // 384 tokens 15.9 / 15.1 / 17.0, 512 20.1 / 17.2 / 18.4, 1536 49.4 / 41.8 / 38.3.
  const auto tiles = [&](int64_t n) { return m_tiles * 4 * ((C + n - 1) / n); };
  const auto rounds = [&](int64_t n) { return (tiles(n) + dev->sm_count - 1) / dev->sm_count; };
  const int kn = tiles(64) <= dev->sm_count * 3 / 4 ? 64 : (rounds(128) <= rounds(256) ? 128 : 256);
  const int64_t tiles_n = (C + kn - 1) / kn;
  if (4 * tiles_n > 65535) return AF3K_ERR_BAD_SHAPE;
  auto enc = tensor_map_encoder();
  if (!enc) return driver_fail("cuTensorMapEncodeTiled entry point", -1);
  CUtensorMap tm_x;
  TokMaps maps;
  auto map = [&](CUtensorMap* tm, const void* base, int64_t rows, int64_t pitch, int box_rows) {
    cuuint64_t dims[2] = {(cuuint64_t)C, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)pitch * 2};
    cuuint32_t box[2] = {64, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    return enc(tm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  };
  CUresult r = map(&tm_x, x, M, C, 128);
  for (int i = 0; i < 4 && r == CUDA_SUCCESS; ++i) {
    const bool mn = (mn_mask >> i) & 1;
    r = map(&maps.w[i], w4[i].data, C, mn ? w4[i].stride_in : w4[i].stride_out, mn ? 64 : kn);
  }
  if (r != CUDA_SUCCESS) return driver_fail("cuTensorMapEncodeTiled(token projection)", (int)r);
  TokParams p;
  std::memset(&p, 0, sizeof(p));
  p.M = (int)M; p.C = (int)C; p.tiles_n = (int)tiles_n; p.mn_mask = mn_mask;
  p.q_bias = q_bias; p.q_bias_f32 = q_bias_dtype == AF3K_F32 ? 1 : 0; p.q_scale = q_scale;
  p.out = static_cast<__nv_bfloat16*>(out); p.status = status_dev; p.wait_limit = wait_limit_cycles();
  const dim3 grid((unsigned)m_tiles, (unsigned)(4 * tiles_n));
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_v);
  if (kn == 256) launch_overlapped(token_proj_kernel<256>, grid, kTokThreads, TokTile<256>::kSmem, stream, true, p, tm_x, maps);
  else if (kn == 128) launch_overlapped(token_proj_kernel<128>, grid, kTokThreads, TokTile<128>::kSmem, stream, true, p, tm_x, maps);
  else           launch_overlapped(token_proj_kernel<64>, grid, kTokThreads, TokTile<64>::kSmem, stream, true, p, tm_x, maps);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail("launch token_proj_kernel", e);
  t_last_launches = 1;
  return AF3K_OK;
}

int af3k_token_projection(const void* x, const void* w4, const void* q_bias, int32_t q_bias_dtype, int64_t M, int64_t C, float q_scale,
                          void* out, int* status_dev, void* stream_v) {
  af3k_matrix w[4];
  for (int i = 0; i < 4; ++i) w[i] = af3k_matrix{w4 ? static_cast<const char*>(w4) + (size_t)i * C * C * 2 : nullptr, C, 1, AF3K_BF16};
  return af3k_token_projection_weights(x, w, q_bias, q_bias_dtype, M, C, q_scale, out, status_dev, stream_v);
}

int af3k_qkvg_projection(const void* x, const void* w4, int64_t R, int64_t N, int64_t H, float q_scale,
                         void* q, void* k, void* v, void* gate, int* status_dev, void* stream_v) {
  return af3k_grid_front(x, AF3K_BF16, nullptr, nullptr, 0.f, nullptr, 0, w4, R, N, 128, H, q_scale, 0, nullptr, 0, q, k, v, gate,
                         status_dev, stream_v);
}

int af3k_pair_front(const void* pair, const float* gamma, const float* beta, float eps, const float* bias_w,
                    int64_t Hb, const void* w4, int64_t R, int64_t N, int64_t H, float q_scale, void* bias,
                    int64_t bias_pitch, void* q, void* k, void* v, void* gate, int* status_dev, void* stream_v) {
  if (Hb < 1) return AF3K_ERR_BAD_SHAPE;
  if (!gamma) return AF3K_ERR_NULL_POINTER;
  return af3k_grid_front(pair, AF3K_BF16, gamma, beta, eps, bias_w, Hb, w4, R, N, 128, H, q_scale, 0, bias, bias_pitch, q, k, v, gate,
                         status_dev, stream_v);
}

int af3k_cast(const void* const* src, void* const* dst, const int64_t* n, int32_t count, int32_t to_dtype, void* stream_v) {
  t_last_launches = 0;
  if (to_dtype != AF3K_BF16 && to_dtype != AF3K_F32) return AF3K_ERR_BAD_DTYPE;
  if (count < 0 || count > kMaxCasts) return AF3K_ERR_BAD_SHAPE;
  if (count > 0 && (!src || !dst || !n)) return AF3K_ERR_NULL_POINTER;
  CastParams p{};
  long long most = 0;
  for (int i = 0; i < count; ++i) {
    if (n[i] < 0) return AF3K_ERR_BAD_SHAPE;
    if (n[i] > 0 && (!src[i] || !dst[i])) return AF3K_ERR_NULL_POINTER;
    if (!aligned16(src[i]) || !aligned16(dst[i])) return AF3K_ERR_BAD_ALIGNMENT;
    p.src[i] = src[i]; p.dst[i] = dst[i]; p.n[i] = n[i];
    if (n[i] > most) most = n[i];
  }
  if (most == 0) return AF3K_OK;
  DeviceInfo* dev = nullptr;
  int rc = device_info(&dev);
  if (rc != AF3K_OK) return rc;
  long long blocks = (most / 8 + kCastThreads) / kCastThreads;
  if (blocks > dev->sm_count * 8) blocks = dev->sm_count * 8;
  const dim3 grid((unsigned)blocks, (unsigned)count);
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_v);
  if (to_dtype == AF3K_BF16) launch_overlapped(cast_kernel<true>, grid, kCastThreads, 0, stream, true, p);
  else                       launch_overlapped(cast_kernel<false>, grid, kCastThreads, 0, stream, true, p);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail("launch cast_kernel", e);
  t_last_launches = 1;
  return AF3K_OK;
}

int af3k_sigmoid_gate(const void* weighted, const void* gate, void* out, int64_t n, void* stream_v) {
  t_last_launches = 0;
  if (n < 0 || (n & 7) != 0) return AF3K_ERR_BAD_SHAPE;
  if (n == 0) return AF3K_OK;
  if (!weighted || !gate || !out) return AF3K_ERR_NULL_POINTER;
  if (!aligned16(weighted) || !aligned16(gate) || !aligned16(out)) return AF3K_ERR_BAD_ALIGNMENT;
  DeviceInfo* dev = nullptr;
  int rc = device_info(&dev);
  if (rc != AF3K_OK) return rc;
  const long long n8 = n / 8;
  long long blocks = (n8 + 255) / 256;
  const long long cap = (long long)dev->sm_count * 8;
  if (blocks > cap) blocks = cap;
  sigmoid_gate_kernel<<<(unsigned)blocks, 256, 0, reinterpret_cast<cudaStream_t>(stream_v)>>>(
      static_cast<const uint4*>(weighted), static_cast<const uint4*>(gate), static_cast<uint4*>(out), n8);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail("launch sigmoid_gate_kernel", e);
  t_last_launches = 1;
  return AF3K_OK;
}

int af3k_selftest_wait_timeout(long long limit_cycles, int* status_dev, void* stream_v) {
  if (limit_cycles <= 0) return AF3K_ERR_BAD_SHAPE;
  wait_timeout_selftest_kernel<<<1, 32, 0, reinterpret_cast<cudaStream_t>(stream_v)>>>(limit_cycles,
                                                                                      status_dev);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? AF3K_OK : cuda_fail("launch wait_timeout_selftest_kernel", e);
}

}  // extern "C"
