// Native host path: what a call of the operator does between Python and the C ABI - argument checks,
// dtype and layout conversions, output allocation, the cache of staged biases, stream look-up - on
// at::Tensor, without the interpreter.  A small attention call is bound by its host time: through
// Python and ctypes it took 37 - 44 us on the host whatever the size (kernel: 5 - 20 us), through this
// file about 7 us, of which the launch itself is 3.
//
// Nothing here computes: every result comes from a kernel of libaf3k.so, whose entry points are looked
// up in the library the Python binding loaded (bind_library).
#include <ATen/cuda/CUDAEvent.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <dlfcn.h>
#include <torch/extension.h>

#include <cmath>
#include <cstring>
#include <list>
#include <map>
#include <mutex>

#include "../../include/af3k.h"

namespace {

using at::Tensor;
using OptTensor = std::optional<Tensor>;

// ------------------------------------------------------------------ library and errors
struct Library {
  decltype(&af3k_dot_product_attention) attention = nullptr;
  decltype(&af3k_dot_product_attention_convert) attention_convert = nullptr;
  decltype(&af3k_dot_product_attention_workspace) workspace = nullptr;
  decltype(&af3k_stage_bias) stage_bias = nullptr;
  decltype(&af3k_grid_front_weights) grid_front = nullptr;
  decltype(&af3k_grid_out_weights) grid_out = nullptr;
  decltype(&af3k_sigmoid_gate) sigmoid_gate = nullptr;
  decltype(&af3k_cast) cast = nullptr;
  decltype(&af3k_grid_pack) grid_pack = nullptr;
  decltype(&af3k_token_pack) token_pack = nullptr;
  decltype(&af3k_token_projection_weights) token_projection = nullptr;
};
Library g_lib;

void bind_library(const std::string& path) {
  void* h = dlopen(path.c_str(), RTLD_NOW | RTLD_LOCAL);
  TORCH_CHECK(h != nullptr, "cannot load ", path, ": ", dlerror());
  auto find = [&](const char* name) {
    void* p = dlsym(h, name);
    TORCH_CHECK(p != nullptr, path, " does not export ", name);
    return p;
  };
#define AF3K_BIND(field, name) g_lib.field = reinterpret_cast<decltype(g_lib.field)>(find(#name))
  AF3K_BIND(attention, af3k_dot_product_attention);
  AF3K_BIND(attention_convert, af3k_dot_product_attention_convert);
  AF3K_BIND(workspace, af3k_dot_product_attention_workspace);
  AF3K_BIND(stage_bias, af3k_stage_bias);
  AF3K_BIND(grid_front, af3k_grid_front_weights);
  AF3K_BIND(grid_out, af3k_grid_out_weights);
  AF3K_BIND(sigmoid_gate, af3k_sigmoid_gate);
  AF3K_BIND(cast, af3k_cast);
  AF3K_BIND(grid_pack, af3k_grid_pack);
  AF3K_BIND(token_pack, af3k_token_pack);
  AF3K_BIND(token_projection, af3k_token_projection_weights);
#undef AF3K_BIND
}

// Return codes become the Python binding's Af3kError.
void check(int code) {
  if (code == AF3K_OK) return;
  py::gil_scoped_acquire gil;
  py::module_::import("af3_kernels_b200._capi").attr("check")(code);
}

[[noreturn]] void value_error(const std::string& what) { throw py::value_error(what); }
[[noreturn]] void type_error(const std::string& what) { throw py::type_error(what); }

// An uninitialised tensor, straight from the caching allocator of the current stream: at::empty goes through the dispatcher
// first, half of its 1.2 us.
Tensor new_tensor(at::IntArrayRef sizes, at::ScalarType type, const at::Device& dev) { return at::detail::empty_cuda(sizes, type, dev, std::nullopt); }

// Status words {bits, 1 + barrier, block, warp} of a device, shared by all calls on it; kept for the
// life of the process.
Tensor status_buffer(int64_t device) {
  static std::mutex mu;
  static std::vector<Tensor>* bufs = new std::vector<Tensor>(64);
  std::lock_guard<std::mutex> lock(mu);
  Tensor& t = bufs->at(device);
  if (!t.defined()) t = at::zeros({4}, at::TensorOptions().dtype(at::kInt).device(at::kCUDA, device));
  return t;
}

// ------------------------------------------------------------------ conversions
// Each of up to three tensors as bf16: those that are fp32, contiguous, aligned and not lazily negated in one launch of the library's,
// others by torch.
// block_limit: the call leaves SMs to another stream.  The library's conversions may be resident, waiting, while the kernel before
// still runs, on those SMs too; torch's come in when it has ended, so they are taken there.
void to_bf16(std::initializer_list<Tensor*> tensors, cudaStream_t stream, bool block_limit = false) {
  const void* src[3];
  void* dst[3];
  int64_t n[3];
  int32_t count = 0;
  std::vector<std::pair<Tensor*, Tensor>> made;
  for (Tensor* t : tensors) {
    if (t->scalar_type() == at::kBFloat16) continue;
    if (block_limit || t->scalar_type() != at::kFloat || t->is_neg() || !t->is_contiguous() || !t->is_cuda() || reinterpret_cast<uintptr_t>(t->data_ptr()) % 16 != 0) {
      *t = t->to(at::kBFloat16);
      continue;
    }
    Tensor b = new_tensor(t->sizes(), at::kBFloat16, t->device());
    src[count] = t->data_ptr(); dst[count] = b.data_ptr(); n[count++] = t->numel();
    made.emplace_back(t, std::move(b));
  }
  if (count != 0) check(g_lib.cast(src, dst, n, count, AF3K_BF16, stream));
  for (auto& [t, b] : made) *t = std::move(b);
}

// A contiguous bf16 result as fp32.
Tensor to_float(const Tensor& t, cudaStream_t stream, bool block_limit = false) {
  if (block_limit) return t.to(at::kFloat);
  Tensor f = new_tensor(t.sizes(), at::kFloat, t.device());
  const void* src = t.data_ptr();
  void* dst = f.data_ptr();
  const int64_t n = t.numel();
  check(g_lib.cast(&src, &dst, &n, 1, AF3K_F32, stream));
  return f;
}

// ------------------------------------------------------------------ staged biases
// A bias the kernel cannot read in place (fp32, rows that are not 16-byte multiples) or, with fp8 q/k,
// not before it was divided by each head's logit scale, is converted once; the copy is used again
// while the very same tensor object is alive and unmodified (its version counter) and, for fp8, the
// scales are the same.  Four copies are kept; copies of dead tensors are dropped when another is made.
// Only for dot_product_attention(cache_bias=True): a write that bumps no counter (.data, a collective) is missed, so the
// entry points with the reference's signatures and the blocks convert in every call.
// A stream that is being captured never gets one of them: the graph would go on reading the copy after the
// list gave it up, and would not see a later write to the bias.  It converts inside the graph.
struct TensorId {
  c10::weak_intrusive_ptr<c10::TensorImpl> impl;
  int64_t version = -1;
  explicit TensorId(const Tensor& t) : impl(t.getIntrusivePtr()), version(t._version()) {}
  bool is(const Tensor& t) const { return !impl.expired() && impl._unsafe_get_target() == t.unsafeGetTensorImpl() && version == (int64_t)t._version(); }
};

struct Staged {
  TensorId bias;
  std::vector<int64_t> sizes, strides;
  const void* data;
  int64_t B2, Sq, Sk;
  std::optional<TensorId> q_scale, k_scale;
  float scale;
  Tensor copy;
  at::cuda::CUDAEvent made;                 // behind the conversion kernel
  std::vector<c10::StreamId> ordered;       // streams that are behind it already
};

std::mutex g_staged_mu;
std::list<Staged>* g_staged = new std::list<Staged>();
constexpr size_t kStagedMost = 4;

// The bias as [B2, Sq, Sk]; another shape with as many elements (four dimensions, or three others) is reshaped.
Tensor bias_3d(const Tensor& bias, int64_t B2, int64_t Sq, int64_t Sk) {
  const int64_t sizes[3] = {B2, Sq, Sk};
  return bias.sizes() == at::IntArrayRef(sizes, 3) ? bias : bias.reshape(sizes);
}

// The bias as the library takes it: bf16 or fp32, [B2, Sq, Sk], rows of any pitch.
Tensor plain_bias(Tensor bias, int64_t B2, int64_t Sq, int64_t Sk) {
  if (bias.scalar_type() != at::kBFloat16 && bias.scalar_type() != at::kFloat) bias = bias.to(at::kFloat);
  bias = bias_3d(bias, B2, Sq, Sk);
  return (Sk > 1 && bias.stride(2) != 1) || (B2 > 1 && bias.stride(0) == 0) || (Sq > 1 && bias.stride(1) == 0) ? bias.contiguous() : bias;
}

Tensor make_staged(const Tensor& bias_in, int64_t B2, int64_t Sq, int64_t Sk, int64_t D, const float* q_scale,
                   const float* k_scale, float scale, cudaStream_t stream) {
  const Tensor bias = plain_bias(bias_in, B2, Sq, Sk);
  af3k_attention_desc d{};
  d.B1 = 1; d.B2 = B2; d.Sq = Sq; d.Sk = Sk; d.D = (D + 15) / 16 * 16;
  const int64_t most = std::max(Sq, Sk) * 64;
  for (int64_t* s : {d.q_stride, d.k_stride, d.v_stride, d.out_stride}) { s[0] = B2 * most; s[1] = most; s[2] = 64; }
  d.bias_stride[0] = bias.stride(0); d.bias_stride[1] = bias.stride(1);
  d.qk_dtype = q_scale != nullptr ? AF3K_FP8_E4M3 : AF3K_BF16;
  d.bias_dtype = bias.scalar_type() == at::kBFloat16 ? AF3K_BF16 : AF3K_F32;
  d.softmax_scale = scale;
  Tensor staged = at::empty({B2, Sq, (Sk + 7) / 8 * 8}, bias.options().dtype(at::kBFloat16));
  check(g_lib.stage_bias(&d, bias.data_ptr(), q_scale, k_scale, staged.data_ptr(), staged.numel() * 2, stream));
  return staged;
}

Tensor staged_bias(const Tensor& bias, int64_t B2, int64_t Sq, int64_t Sk, int64_t D, const OptTensor& qs_id,
                   const OptTensor& ks_id, const float* q_scale, const float* k_scale, float scale) {
  const auto stream = c10::cuda::getCurrentCUDAStream(bias.device().index());
  const bool capturing = c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None;
  const bool cacheable = !capturing && !bias.is_inference() && !(qs_id && (qs_id->is_inference() || ks_id->is_inference()));
  std::lock_guard<std::mutex> lock(g_staged_mu);
  if (cacheable) {
    for (auto it = g_staged->begin(); it != g_staged->end(); ++it) {
      Staged& e = *it;
      if (!e.bias.is(bias) || e.B2 != B2 || e.Sq != Sq || e.Sk != Sk || e.data != bias.data_ptr() || bias.sizes() != e.sizes ||
          bias.strides() != e.strides || e.q_scale.has_value() != qs_id.has_value())
        continue;
      if (qs_id && (!e.q_scale->is(*qs_id) || !e.k_scale->is(*ks_id) || e.scale != scale)) continue;
      if (std::find(e.ordered.begin(), e.ordered.end(), stream.id()) == e.ordered.end()) {
        e.made.block(stream);
        c10::cuda::CUDACachingAllocator::recordStream(e.copy.storage().data_ptr(), stream);
        e.ordered.push_back(stream.id());
      }
      if (it != g_staged->begin()) g_staged->splice(g_staged->begin(), *g_staged, it);
      return e.copy;
    }
  }
  Tensor copy = make_staged(bias, B2, Sq, Sk, D, q_scale, k_scale, scale, stream);
  if (!cacheable) return copy;
  g_staged->remove_if([&](const Staged& e) { return e.bias.impl.expired() || e.bias.impl._unsafe_get_target() == bias.unsafeGetTensorImpl(); });
  while (g_staged->size() >= kStagedMost) g_staged->pop_back();
  Staged e{TensorId(bias), bias.sizes().vec(), bias.strides().vec(), bias.data_ptr(), B2, Sq, Sk, std::nullopt, std::nullopt, scale, copy,
           at::cuda::CUDAEvent(), {stream.id()}};
  if (qs_id) { e.q_scale.emplace(*qs_id); e.k_scale.emplace(*ks_id); }
  e.made.record(stream);
  g_staged->push_front(std::move(e));
  return copy;
}

// ------------------------------------------------------------------ the operator
// unit innermost stride; a broadcast (zero-stride) view cannot be described to TMA
Tensor inner_contiguous(const Tensor& t) {
  bool bad = t.size(3) != 1 && t.stride(3) != 1;
  for (int i = 0; i < 3; ++i) bad = bad || (t.stride(i) == 0 && t.size(i) > 1);
  return bad ? t.contiguous() : t;
}

std::string shape_text(const Tensor& t) {
  std::ostringstream s;
  s << t.sizes();
  return s.str();
}

// mask: bool, [Sk] or [1 | B1, Sk] (the Python side brings other forms to this one)
void check_mask(const Tensor& mask, int64_t B1, int64_t Sk) {
  if (mask.dim() < 1 || mask.dim() > 2 || mask.size(-1) != Sk || (mask.dim() == 2 && mask.size(0) != 1 && mask.size(0) != B1))
    value_error("mask of shape " + shape_text(mask) + " does not match B1=" + std::to_string(B1) + ", Sk=" + std::to_string(Sk));
}

// bias_form: 0 an ordinary bias tensor, 1 the copy of a StagedBias, 2 the same divided by fp8 scales, 3 an ordinary one that
// the kernel may convert itself
Tensor attention(Tensor q, Tensor k, Tensor v, const OptTensor& mask_in, Tensor bias, const OptTensor& q_scale_in,
                 const OptTensor& k_scale_in, std::optional<double> softmax_scale, int64_t rows_per_item, const OptTensor& out_in,
                 bool use_workspace, bool cache_bias, int64_t max_ctas, int64_t bias_form, int* status = nullptr) {
  if (q.dim() != 4 || k.dim() != 4 || v.dim() != 4) value_error("q, k, v must be 4-D [B1, B2, S, D]");
  if (!q.is_cuda()) throw std::runtime_error("af3_kernels_b200 runs on CUDA tensors only (no CPU fallback)");
  const auto dev = q.device();
  if (k.device() != dev || v.device() != dev || bias.device() != dev) value_error("q, k, v, bias must live on the same device");
  const int64_t B1 = q.size(0), B2 = q.size(1), Sq = q.size(2), D = q.size(3), Sk = k.size(2);
  for (const Tensor* t : {&k, &v})
    if (t->size(0) != B1 || t->size(1) != B2 || t->size(2) != Sk || t->size(3) != D) value_error("k and v must be [B1, B2, Sk, D] matching q");
  const c10::cuda::CUDAGuard guard(dev);
  const bool fp8 = q.scalar_type() == at::kFloat8_e4m3fn;
  bool f32_result = false;
  Tensor q_scale, k_scale;
  if (fp8) {
    if (k.scalar_type() != at::kFloat8_e4m3fn || !q_scale_in || !k_scale_in) type_error("fp8 q needs fp8 k and q_scale / k_scale");
    q_scale = q_scale_in->to(dev, at::kFloat).contiguous();
    k_scale = k_scale_in->to(dev, at::kFloat).contiguous();
    if (q_scale.numel() != B2 || k_scale.numel() != B2) value_error("q_scale / k_scale must have one entry per head");
  } else {
    if (q.scalar_type() == at::kFloat) {
      // the reference has an fp32 instantiation (src/csrc/dot_product_attention.cpp:554-558); here fp32
      // callers get the bf16 kernel (operands rounded once) and an fp32 result
      if (out_in) value_error("`out` must be omitted with fp32 q (the result is converted from the kernel's bf16 output)");
      f32_result = true;
    }
    if (q.scalar_type() != at::kBFloat16 && !f32_result) type_error(std::string("q must be bfloat16, float32 or float8_e4m3fn, got ") + c10::toString(q.scalar_type()));
    if ((q_scale_in || k_scale_in) && !f32_result) type_error("q_scale / k_scale are only valid with fp8 q and k");
    to_bf16({&q, &k, &v}, c10::cuda::getCurrentCUDAStream(dev.index()), max_ctas > 0);
  }
  if (v.scalar_type() != at::kBFloat16) v = v.to(at::kBFloat16);
  const float scale = softmax_scale ? (float)*softmax_scale : (float)(1.0 / std::sqrt((double)D));

  bool prescaled = bias_form == 2;
  if (bias_form == 0 || bias_form == 3) {
    if (bias.numel() != B2 * Sq * Sk) {
      value_error("bias must have B2*Sq*Sk = " + std::to_string(B2 * Sq * Sk) + " elements, got " + std::to_string(bias.numel()));
    }
    const bool as_is = bias.dim() == 3 && bias.size(0) == B2 && bias.size(1) == Sq && bias.size(2) == Sk;
    const bool needs_copy = bias.scalar_type() != at::kBFloat16 || !as_is || bias.stride(2) != 1 || (bias.stride(1) * 2) % 16 != 0 || (bias.stride(0) * 2) % 16 != 0 ||
                            reinterpret_cast<uintptr_t>(bias.data_ptr()) % 16 != 0;
    if (use_workspace && cache_bias && (needs_copy || fp8) && bias.numel() != 0) {
      bias = staged_bias(bias, B2, Sq, Sk, D, fp8 ? q_scale_in : std::nullopt, fp8 ? k_scale_in : std::nullopt,
                         fp8 ? q_scale.data_ptr<float>() : nullptr, fp8 ? k_scale.data_ptr<float>() : nullptr, scale);
      prescaled = fp8;
    } else {
      bias = plain_bias(bias, B2, Sq, Sk);
    }
  }
  q = inner_contiguous(q); k = inner_contiguous(k); v = inner_contiguous(v);

  Tensor mask;
  int64_t mask_stride = 0;
  if (mask_in) {
    mask = *mask_in;
    check_mask(mask, B1, Sk);
    mask = mask.contiguous();
    if (mask.device() != dev) mask = mask.to(dev);
    mask_stride = mask.dim() == 2 && !(mask.size(0) == 1 && B1 != 1) ? Sk : 0;
  }

  Tensor out;
  if (!out_in) {
    out = new_tensor({B1, B2, Sq, D}, at::kBFloat16, dev);
  } else {
    out = *out_in;
    if (out.dim() != 4 || out.size(0) != B1 || out.size(1) != B2 || out.size(2) != Sq || out.size(3) != D ||
        out.scalar_type() != at::kBFloat16 || out.stride(3) != 1)
      value_error("out must be a bf16 [B1, B2, Sq, D] tensor with unit inner stride");
    if (out.device() != dev) value_error("out must live on the device of q, k, v, bias");
  }
  if (out.numel() == 0) return f32_result ? out.to(at::kFloat) : out;
  if (out_in && !out.is_inference()) out.unsafeGetTensorImpl()->bump_version();   // written in place, as by any torch operator

  af3k_attention_desc d{};
  d.B1 = B1; d.B2 = B2; d.Sq = Sq; d.Sk = Sk; d.D = D;
  for (int i = 0; i < 3; ++i) {
    d.q_stride[i] = q.stride(i); d.k_stride[i] = k.stride(i); d.v_stride[i] = v.stride(i); d.out_stride[i] = out.stride(i);
  }
  d.bias_stride[0] = bias.stride(0); d.bias_stride[1] = bias.stride(1);
  d.mask_row_stride = mask_stride;
  d.qk_dtype = fp8 ? AF3K_FP8_E4M3 : AF3K_BF16;
  d.bias_dtype = bias.scalar_type() == at::kBFloat16 ? AF3K_BF16 : AF3K_F32;
  d.softmax_scale = scale;
  d.rows_per_item = (int32_t)rows_per_item;
  d.bias_prescaled = prescaled ? 1 : 0;
  d.max_ctas = (int32_t)max_ctas;
  const uint8_t* mask_data = mask.defined() ? static_cast<const uint8_t*>(mask.data_ptr()) : nullptr;
  int* const status_data = status != nullptr ? status : status_buffer(dev.index()).data_ptr<int>();
  const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(dev.index());
  if (bias_form == 3 && !fp8) {
    const int rc = g_lib.attention_convert(&d, q.data_ptr(), k.data_ptr(), v.data_ptr(), bias.data_ptr(), mask_data, out.data_ptr(), status_data, stream);
    if (rc != AF3K_ERR_WORKSPACE) {
      check(rc);
      return f32_result ? to_float(out, stream, max_ctas > 0) : out;
    }
  }
  Tensor ws;
  if (use_workspace) {
    const size_t bytes = g_lib.workspace(&d, bias.data_ptr());
    if (bytes != 0) ws = new_tensor({(int64_t)bytes}, at::kByte, dev);
  }
  check(g_lib.attention(&d, q.data_ptr(), k.data_ptr(), v.data_ptr(), bias.data_ptr(), mask_data, out.data_ptr(), fp8 ? q_scale.data_ptr<float>() : nullptr, fp8 ? k_scale.data_ptr<float>() : nullptr,
                        ws.defined() ? ws.data_ptr() : nullptr, ws.defined() ? (size_t)ws.numel() : 0,
                        status_data, stream));
  return f32_result ? to_float(out, stream, max_ctas > 0) : out;
}

// ------------------------------------------------------------------ block parameters
// Every call reads the parameters as they are then.  Nothing made from them is kept between calls: a copy found again
// by storage and version misses writes that bump no counter (p.data.copy_(), a collective or a kernel on the raw
// pointer), and a captured graph would replay it after it was given up or had become old.
int32_t dtype_code(const Tensor& t) { return t.scalar_type() == at::kFloat ? AF3K_F32 : AF3K_BF16; }

Tensor kernel_dtype(const Tensor& t) {      // bf16 or fp32
  return t.scalar_type() == at::kFloat || t.scalar_type() == at::kBFloat16 ? t : t.detach().to(at::kFloat);
}

// The first n parameters are [C, C]; all are where the activations are (a kernel handed the address of a module that was
// left on the host would fault).
void check_parameters(const std::vector<Tensor>& params, size_t n, int64_t C, const at::Device& dev) {
  for (size_t i = 0; i < params.size(); ++i) {
    const Tensor& t = params[i];
    if (t.device() != dev) value_error("parameters must live on the device of the activations, " + dev.str() + ", got " + t.device().str());
    if (i < n && (t.dim() != 2 || t.size(0) != C || t.size(1) != C)) value_error("projection weights must be [C, C]");
  }
}

// q, k, v, gate and perhaps output projection [C, C] as (out, in) matrices (in_out: as (in, out) ones), in the kernels'
// layout: one launch -> [4 C or 5 C, C] bf16.  tokens: fp32 activations of the single block that the same launch rounds to bf16, in place of
// which their bf16 form is left.
Tensor packed_matrices(const std::vector<Tensor>& w, int64_t C, cudaStream_t stream, bool in_out = false, Tensor* tokens = nullptr) {
  std::vector<Tensor> src;
  af3k_matrix w5[5] = {};
  for (size_t i = 0; i < w.size(); ++i) {
    src.push_back(kernel_dtype(w[i]));
    w5[i] = af3k_matrix{src[i].data_ptr(), src[i].stride(in_out ? 1 : 0), src[i].stride(in_out ? 0 : 1), dtype_code(src[i])};
  }
  Tensor packed = at::empty({(int64_t)w.size() * C, C}, src[0].options().dtype(at::kBFloat16));
  char* p = static_cast<char*>(packed.data_ptr());
  if (tokens != nullptr) {
    const Tensor x = *tokens;
    *tokens = at::empty(x.sizes(), x.options().dtype(at::kBFloat16));
    check(g_lib.token_pack(w5, C, p, x.data_ptr<float>(), x.size(0), tokens->data_ptr(), stream));
    return packed;
  }
  check(g_lib.grid_pack(w5, nullptr, nullptr, nullptr, AF3K_F32, C, 0, p, w.size() > 4 ? p + 4 * C * C * 2 : nullptr, nullptr, stream));
  return packed;
}

// The grid block's parameters: matrices q, k, v, gate, output as [out, in], read where they are if the kernels can
// (nn.Linear.weight, bf16 or fp32), else packed for this call; then (all or none) LayerNorm weight and bias, bias projection.
struct GridParameters {
  af3k_front_weights front{};
  const void* wo = nullptr;
  std::vector<Tensor> keep;
};
GridParameters grid_parameters(const std::vector<Tensor>& params, int64_t C, cudaStream_t stream) {
  GridParameters r;
  r.front.ln_dtype = r.front.bias_w_dtype = AF3K_F32;
  const void* m[5];
  const at::ScalarType type = params[0].scalar_type();
  bool in_place = type == at::kBFloat16 || type == at::kFloat;
  for (int i = 0; i < 5; ++i) {
    m[i] = params[i].data_ptr();
    in_place = in_place && params[i].scalar_type() == type && params[i].is_contiguous() && reinterpret_cast<uintptr_t>(m[i]) % 16 == 0;
  }
  r.front.w_dtype = in_place ? dtype_code(params[0]) : AF3K_BF16;
  if (!in_place) {
    r.keep.push_back(packed_matrices({params.begin(), params.begin() + 5}, C, stream));
    for (int i = 0; i < 5; ++i) m[i] = static_cast<char*>(r.keep[0].data_ptr()) + i * C * C * 2;
  }
  for (int i = 0; i < 4; ++i) r.front.w[i] = m[i];
  r.wo = m[4];
  if (params.size() > 5) {
    Tensor gamma = kernel_dtype(params[5]), beta = kernel_dtype(params[6]);
    const Tensor bw = kernel_dtype(params[7]).contiguous();
    if (gamma.scalar_type() != beta.scalar_type()) { gamma = gamma.detach().to(at::kFloat); beta = beta.detach().to(at::kFloat); }
    gamma = gamma.contiguous(); beta = beta.contiguous();
    r.front.gamma = gamma.data_ptr(); r.front.beta = beta.data_ptr(); r.front.bias_w = bw.data_ptr();
    r.front.ln_dtype = dtype_code(gamma); r.front.bias_w_dtype = dtype_code(bw);
    r.keep.insert(r.keep.end(), {gamma, beta, bw});
  }
  return r;
}

// ------------------------------------------------------------------ the grid attention block
// The sizes all three kernels take: widths 64 and 128, heads of 8 to 64 channels (the attention kernel's), up to four
// bias heads and 32-bit element offsets (the front's).  Others go through torch's projections.
bool grid_sizes_fused(int64_t R, int64_t N, int64_t C, int64_t head, int64_t bias_heads) {
  if ((C != 64 && C != 128) || head < 1 || C % head != 0 || bias_heads > 4) return false;
  const int64_t D = C / head, most = 0x7fffffffLL / C;
  return D % 8 == 0 && D <= 64 && R > 0 && N > 0 && R <= most && N <= most / R;
}

bool grid_fused(const Tensor& pair, int64_t head, int64_t bias_heads) {
  return pair.is_cuda() && pair.dim() == 3 && grid_sizes_fused(pair.size(0), pair.size(1), pair.size(2), head, bias_heads) &&
         (pair.scalar_type() == at::kBFloat16 || pair.scalar_type() == at::kFloat);
}

// The whole module: raw pair [N, N, C] -> front (LayerNorm, bias, q / k / v / gate) -> attention -> gate and output
// projection, three launches.  weights: nn.Linear.weight of q, k, v, gate, output; then LayerNorm weight and bias,
// bias projection.  transpose: attention along the columns of the pair; q, k, v are written, and the result is
// read back, in the exchanged order, so nothing is permuted in memory.  project false: up to the gated result (bf16),
// for an output projection that torch differentiates.
Tensor grid_module(Tensor pair, const Tensor& mask_in, const std::vector<Tensor>& params, double eps, int64_t head, bool transpose, bool project) {
  const at::Device dev = pair.device();
  const c10::cuda::CUDAGuard guard(dev);
  const int64_t R = pair.size(0), N = pair.size(1), C = pair.size(2), D = C / head, M = R * N;
  if (R != N) value_error("pair must be [N, N, c_pair]");
  check_parameters(params, 5, C, dev);
  if (params[7].dim() != 2 || params[7].size(0) != head || params[7].size(1) != C || params[5].numel() != C || params[6].numel() != C)
    value_error("LayerNorm and bias projection do not match the pair");
  pair = pair.contiguous();
  if (reinterpret_cast<uintptr_t>(pair.data_ptr()) % 16 != 0) pair = pair.clone();
  Tensor mask = mask_in.device() == dev ? mask_in.contiguous() : mask_in.to(dev).contiguous();
  check_mask(mask, N, N);
  const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(dev.index());
  const GridParameters w = grid_parameters(params, C, stream);
  const int64_t pitch = (N + 7) / 8 * 8;
  Tensor buf = new_tensor({5 * M * C + head * N * pitch}, at::kBFloat16, dev);           // q, k, v, gate, attention result, bias
  Tensor out = new_tensor({R, N, C}, project ? pair.scalar_type() : at::kBFloat16, dev);
  char* b = static_cast<char*>(buf.data_ptr());
  const size_t part = (size_t)M * C * 2;             // (a multiple of 128 bytes)
  void* const bias = b + 5 * part;
  void *q = b, *k = b + part, *v = b + 2 * part, *gate = b + 3 * part, *weighted = b + 4 * part;
  const bool f32 = pair.scalar_type() == at::kFloat;
  int* status = status_buffer(dev.index()).data_ptr<int>();
  check(g_lib.grid_front(pair.data_ptr(), f32 ? AF3K_F32 : AF3K_BF16, &w.front, (float)eps, head, R, N, C, head,
                         1.0f / std::sqrt((float)D), transpose, bias, pitch, q, k, v, gate, status, stream));
  af3k_attention_desc d{};
  d.B1 = N; d.B2 = head; d.Sq = N; d.Sk = N; d.D = D;
  for (int64_t* st : {d.q_stride, d.k_stride, d.v_stride}) { st[0] = head * N * D; st[1] = N * D; st[2] = D; }
  d.out_stride[0] = transpose ? C : N * C; d.out_stride[1] = D; d.out_stride[2] = transpose ? N * C : C;
  d.bias_stride[0] = N * pitch; d.bias_stride[1] = pitch;
  d.mask_row_stride = mask.dim() == 2 && mask.size(0) == N ? N : 0;
  d.qk_dtype = AF3K_BF16; d.bias_dtype = AF3K_BF16;
  d.softmax_scale = 1.0f;                            // q left the projection scaled
  check(g_lib.attention(&d, q, k, v, bias, static_cast<const uint8_t*>(mask.data_ptr()), weighted, nullptr, nullptr, nullptr, 0,
                        status, stream));
  if (!project) check(g_lib.sigmoid_gate(weighted, gate, out.data_ptr(), M * C, stream));
  else check(g_lib.grid_out(weighted, gate, w.wo, w.front.w_dtype, out.data_ptr(), f32 ? AF3K_F32 : AF3K_BF16, M, C, status, stream));
  return out;
}

// The block on an already normalised pair [R, N, C] with a bias of the caller's.  weights: q, k, v, gate, output as
// [out, in].
Tensor grid_block(const Tensor& pair, const OptTensor& mask, const Tensor& bias, const std::vector<Tensor>& weights, int64_t head, bool project) {
  const at::Device dev = pair.device();
  const c10::cuda::CUDAGuard guard(dev);
  const int64_t R = pair.size(0), N = pair.size(1), C = pair.size(2), D = C / head, M = R * N;
  check_parameters(weights, 5, C, dev);
  Tensor x = pair.to(at::kBFloat16).contiguous();
  if (reinterpret_cast<uintptr_t>(x.data_ptr()) % 16 != 0) x = x.clone();
  const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(dev.index());
  const GridParameters w = grid_parameters(weights, C, stream);
  Tensor buf = at::empty({5, M, C}, x.options());
  auto at_part = [&](int i, at::IntArrayRef sizes) { return buf.select(0, i).view(sizes); };
  Tensor q = at_part(0, {R, head, N, D}), k = at_part(1, {R, head, N, D}), v = at_part(2, {R, head, N, D});
  Tensor gate = at_part(3, {M, C}), weighted = at_part(4, {R, N, head, D});
  Tensor out = at::empty({R, N, C}, project ? x.options().dtype(pair.scalar_type()) : x.options());
  int* status = status_buffer(dev.index()).data_ptr<int>();
  check(g_lib.grid_front(x.data_ptr(), AF3K_BF16, &w.front, 0.f, 0, R, N, C, head, 1.0f / std::sqrt((float)D), 0, nullptr, 0, q.data_ptr(),
                         k.data_ptr(), v.data_ptr(), gate.data_ptr(), status, stream));
  attention(q, k, v, mask, bias, std::nullopt, std::nullopt, 1.0, 0, weighted.permute({0, 2, 1, 3}), true, false, 0, 3);
  if (!project) check(g_lib.sigmoid_gate(weighted.data_ptr(), gate.data_ptr(), out.data_ptr(), M * C, stream));
  else check(g_lib.grid_out(weighted.data_ptr(), gate.data_ptr(), w.wo, w.front.w_dtype, out.data_ptr(), pair.scalar_type() == at::kFloat ? AF3K_F32 : AF3K_BF16,
                       M, C, status, stream));
  return out;
}

// ------------------------------------------------------------------ the single / diffusion attention block
// x [N, C] -> the four projections in one GEMM (query bias and softmax scale folded in) -> attention, gated as it
// leaves the kernel: two launches.  weights: q, k, v, gate as [in, out].
Tensor self_block(const Tensor& x_in, const OptTensor& mask_in, Tensor bias, const std::vector<Tensor>& weights, Tensor q_bias, int64_t head) {
  const at::Device dev = x_in.device();
  const c10::cuda::CUDAGuard guard(dev);
  const int64_t N = x_in.size(0), C = x_in.size(1), D = C / head;
  check_parameters(weights, 4, C, dev);
  check_parameters({q_bias}, 0, C, dev);
  if (q_bias.numel() != C) value_error("q_bias must have one entry per channel");
  if (bias.numel() != head * N * N) value_error("bias must have B2*Sq*Sk = " + std::to_string(head * N * N) + " elements, got " + std::to_string(bias.numel()));
  if (bias.device() != dev) value_error("q, k, v, bias must live on the same device");
  if (N == 0) return at::empty({N, C}, x_in.options());
  q_bias = kernel_dtype(q_bias).contiguous();
  const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(dev.index());
  // weights the kernel can read where they are: bf16, [out, in] or [in, out], rows of 16-byte multiples
  af3k_matrix w4[4];
  bool in_place_w = true;
  for (int i = 0; i < 4; ++i) {
    const int64_t so = weights[i].stride(1), si = weights[i].stride(0);
    w4[i] = af3k_matrix{weights[i].data_ptr(), so, si, AF3K_BF16};
    in_place_w = in_place_w && weights[i].scalar_type() == at::kBFloat16 && reinterpret_cast<uintptr_t>(w4[i].data) % 16 == 0 &&
                 (so == 1 || si == 1) && std::max(so, si) >= C && std::max(so, si) % 8 == 0;
  }
  // fp32 tokens are rounded in the same launch as weights that are packed
  const bool with_tokens = !in_place_w && x_in.scalar_type() == at::kFloat && !x_in.is_neg() && x_in.is_contiguous() && reinterpret_cast<uintptr_t>(x_in.data_ptr()) % 16 == 0;
  Tensor packed, x = x_in;
  if (!with_tokens) {
    to_bf16({&x}, stream);
    x = x.contiguous();
    if (reinterpret_cast<uintptr_t>(x.data_ptr()) % 16 != 0) x = x.clone();
  }
  if (!in_place_w) {
    packed = packed_matrices(weights, C, stream, true, with_tokens ? &x : nullptr);
    for (int i = 0; i < 4; ++i) w4[i] = af3k_matrix{static_cast<char*>(packed.data_ptr()) + i * C * C * 2, C, 1, AF3K_BF16};
  }
  const float scale = 1.0f / std::sqrt((float)D);
  const bool in_place = bias.scalar_type() == at::kBFloat16 && bias.dim() == 3 && bias.size(0) == head && bias.size(1) == N && bias.stride(2) == 1 && (bias.stride(1) * 2) % 16 == 0 &&
                        (bias.stride(0) * 2) % 16 == 0 && (bias.stride(0) != 0 || head == 1) && (bias.stride(1) != 0 || N == 1) &&
                        reinterpret_cast<uintptr_t>(bias.data_ptr()) % 16 == 0;
  if (!in_place) bias = plain_bias(bias, head, N, N);
  Tensor mask;
  if (mask_in) {
    if (mask_in->numel() != N) value_error("mask of shape " + shape_text(*mask_in) + " does not match B1=1, Sk=" + std::to_string(N));
    mask = mask_in->device() == dev ? mask_in->contiguous() : mask_in->to(dev).contiguous();
  }
  Tensor qkvg = new_tensor({4, N, C}, at::kBFloat16, dev), out = new_tensor({N, C}, at::kBFloat16, dev);
  char* b = static_cast<char*>(qkvg.data_ptr());
  const size_t part = (size_t)N * C * 2;
  int* status = status_buffer(dev.index()).data_ptr<int>();
  check(g_lib.token_projection(x.data_ptr(), w4, q_bias.data_ptr(), q_bias.scalar_type() == at::kFloat ? AF3K_F32 : AF3K_BF16, N, C,
                               scale, b, status, stream));
  af3k_attention_desc d{};
  d.B1 = 1; d.B2 = head; d.Sq = N; d.Sk = N; d.D = D;
  for (int64_t* st : {d.q_stride, d.k_stride, d.v_stride, d.out_stride, d.gate_stride}) { st[0] = N * C; st[1] = D; st[2] = C; }
  d.qk_dtype = AF3K_BF16;
  d.softmax_scale = 1.0f;                            // q left the projection scaled
  d.gate = b + 3 * part;
  const auto call = [&] {
    d.bias_stride[0] = bias.stride(0); d.bias_stride[1] = bias.stride(1);
    d.bias_dtype = dtype_code(bias);
    return g_lib.attention_convert(&d, b, b + part, b + 2 * part, bias.data_ptr(), mask.defined() ? static_cast<const uint8_t*>(mask.data_ptr()) : nullptr,
                                   out.data_ptr(), status, stream);
  };
  int rc = call();
  if (rc == AF3K_ERR_WORKSPACE) {
    bias = make_staged(bias, head, N, N, D, nullptr, nullptr, scale, stream);
    rc = call();
  }
  check(rc);
  if (x_in.scalar_type() == at::kFloat) return to_float(out, stream);
  return x_in.scalar_type() == at::kBFloat16 ? out : out.to(x_in.scalar_type());
}

// ------------------------------------------------------------------ the operator on host tensors
// The batch rows are independent problems, so the call is a pipeline over row blocks on three streams:
// host-to-device copies of block i + 1, the kernel on block i, the device-to-host copy of block i - 1
// (the link carries both directions at once).  Bias, mask and scales go over once, first.  What bounds it
// is the link: at 256 rows of 256 keys 51 MB in at 55 GB/s is 0.93 ms.  Only the last block's kernel and
// copy back stick out behind the input copies, while every block costs three more copies (4 us each on the
// copy engine) and about 20 us of host time, so each block takes half of the rows that are left, down to
// kHostBlockBytes of input; a call that small runs on the caller's stream alone.  (Eight equal blocks
// at this size: 1.34 ms, this schedule: 1.20, eight blocks issued from Python: 1.40; 64 rows of 64 keys:
// 1.05 -> 0.15 ms.  A kernel that stores straight into the pinned result, without the copy back, was
// slower, 2.1 ms: such stores reach 16 GB/s.)
constexpr int64_t kHostBlockBytes = 2 << 20;

#define AF3K_CUDA_CHECK(call)                                                                  \
  do {                                                                                         \
    const cudaError_t e_ = (call);                                                             \
    if (e_ != cudaSuccess) {                                                                   \
      (void)cudaGetLastError();                                                                \
      throw std::runtime_error(std::string(#call) + ": " + cudaGetErrorString(e_));            \
    }                                                                                          \
  } while (0)

// The two copy streams of a thread on a device, the same in every call: streams taken anew from torch's pool would be
// other ones each time.
struct CopyStreams { c10::cuda::CUDAStream in, out; };
const CopyStreams& copy_streams(c10::DeviceIndex device) {
  static thread_local std::map<int, CopyStreams> kept;
  auto it = kept.find(device);
  if (it == kept.end())
    it = kept.emplace(device, CopyStreams{c10::cuda::getStreamFromPool(false, device), c10::cuda::getStreamFromPool(false, device)}).first;
  return it->second;
}

void host_attention(Tensor q, Tensor k, Tensor v, const OptTensor& mask_in, Tensor bias, const OptTensor& q_scale,
                    const OptTensor& k_scale, std::optional<double> softmax_scale, Tensor out, int64_t device, int64_t chunks) {
  const int64_t B1 = q.size(0), B2 = q.size(1), Sq = q.size(2), D = q.size(3), Sk = k.dim() == 4 ? k.size(2) : 0;
  for (const Tensor* t : {&k, &v})
    if (t->dim() != 4 || t->size(0) != B1 || t->size(1) != B2 || t->size(2) != Sk || t->size(3) != D)
      value_error("k and v must be [B1, B2, Sk, D] matching q");
  if (bias.numel() != B2 * Sq * Sk)
    value_error("bias must have B2*Sq*Sk = " + std::to_string(B2 * Sq * Sk) + " elements, got " + std::to_string(bias.numel()));
  if (mask_in) check_mask(*mask_in, B1, Sk);
  const at::Device dev(at::kCUDA, (c10::DeviceIndex)device);
  const c10::cuda::CUDAGuard guard(dev);
  q = q.contiguous(); k = k.contiguous(); v = v.contiguous();
  const int64_t row_bytes = (int64_t)((q.nbytes() + k.nbytes() + v.nbytes()) / B1);
  std::vector<int64_t> bounds{0};
  while ((int64_t)bounds.size() < chunks && (B1 - bounds.back()) * row_bytes >= 2 * kHostBlockBytes && B1 - bounds.back() >= 2)
    bounds.push_back(bounds.back() + (B1 - bounds.back() + 1) / 2);
  bounds.push_back(B1);
  const int64_t blocks = (int64_t)bounds.size() - 1;
  const auto main = c10::cuda::getCurrentCUDAStream(dev.index());
  const auto s_in = blocks > 1 ? copy_streams(dev.index()).in : main;
  const auto s_out = blocks > 1 ? copy_streams(dev.index()).out : main;

  auto on_device = [&](const Tensor& t) { return at::empty(t.sizes(), t.options().device(dev).pinned_memory(false)); };
  auto copy = [&](void* dst, const void* src, size_t bytes, cudaMemcpyKind kind, cudaStream_t s) {
    if (bytes != 0) AF3K_CUDA_CHECK(cudaMemcpyAsync(dst, src, bytes, kind, s));
  };
  // a small operand, sent whole: its host form, and where it goes
  struct Sent { Tensor host, device; };
  auto place = [&](const Tensor& t) {
    const Tensor c = t.contiguous();
    return t.is_cuda() ? Sent{Tensor(), c.to(dev)} : Sent{c, on_device(c)};
  };
  // the call may only return (or throw) once nothing on the device touches the host tensors or the
  // buffers below any more
  struct Drain {
    cudaStream_t s[3];
    bool done = false;
    ~Drain() {
      if (!done)
        for (cudaStream_t t : s) (void)cudaStreamSynchronize(t);
    }
  };
  // all buffers come from the caller's stream: what used their memory before is ordered ahead of that stream, and the
  // copy streams wait for a point on it behind the last allocation
  Tensor dq = on_device(q), dk = on_device(k), dv = on_device(v), dout = on_device(out);
  Sent bias_s = place(bias), mask_s, qs_s, ks_s;
  if (mask_in) mask_s = place(*mask_in);
  if (q_scale) qs_s = place(q_scale->to(at::kFloat));
  if (k_scale) ks_s = place(k_scale->to(at::kFloat));
  Tensor bias_d = bias_s.device, mask_d = mask_s.device;
  // the kernels' status words live in pinned host memory here: only a wait that ran out writes them, and
  // reading them after the call's own synchronisation costs no copy
  Tensor status = at::empty({4}, at::TensorOptions().dtype(at::kInt).pinned_memory(true));
  int* st = status.data_ptr<int>();
  std::memset(st, 0, 16);
  OptTensor qs, ks;
  if (q_scale) qs = qs_s.device;
  if (k_scale) ks = ks_s.device;
  const bool fp8 = q.scalar_type() == at::kFloat8_e4m3fn;
  {
    Drain drain{{s_in, main, s_out}};
    std::vector<at::cuda::CUDAEvent> ev(2 * blocks + 2);
    if (blocks > 1) {
      ev[2 * blocks].record(main);
      ev[2 * blocks].block(s_in);
      ev[2 * blocks].block(s_out);
    }
    int64_t form = 0;
    for (const Sent* t : {&qs_s, &ks_s, &bias_s, &mask_s})
      if (t->host.defined()) copy(t->device.data_ptr(), t->host.data_ptr(), t->host.nbytes(), cudaMemcpyHostToDevice, s_in);
    const bool aligned = bias_d.scalar_type() == at::kBFloat16 && Sk % 8 == 0;
    if (fp8 ? (qs && ks && qs->numel() == B2 && ks->numel() == B2) : !aligned) {
      // converted on the caller's stream, under the copies of the first block
      if (blocks > 1) {
        ev[2 * blocks + 1].record(s_in);
        ev[2 * blocks + 1].block(main);
      }
      const float scale = softmax_scale ? (float)*softmax_scale : (float)(1.0 / std::sqrt((double)D));
      bias_d = make_staged(bias_d, B2, Sq, Sk, D, fp8 ? qs->data_ptr<float>() : nullptr, fp8 ? ks->data_ptr<float>() : nullptr, scale, main)
                   .slice(2, 0, Sk);
      form = fp8 ? 2 : 1;
    }
    const bool row_mask = mask_d.defined() && mask_d.dim() == 2 && mask_d.size(0) == B1 && B1 != 1;
    for (int64_t i = 0; i < blocks; ++i) {
      const int64_t lo = bounds[i], hi = bounds[i + 1];
      auto part = [&](const Tensor& t) { return t.slice(0, lo, hi); };
      for (auto [d, h] : {std::pair<Tensor*, Tensor*>{&dq, &q}, {&dk, &k}, {&dv, &v}}) {
        const size_t row = h->nbytes() / B1;
        copy(static_cast<char*>(d->data_ptr()) + lo * row, static_cast<const char*>(h->data_ptr()) + lo * row, (hi - lo) * row,
             cudaMemcpyHostToDevice, s_in);
      }
      if (blocks > 1) {
        ev[2 * i].record(s_in);
        ev[2 * i].block(main);
      }
      attention(part(dq), part(dk), part(dv), row_mask ? OptTensor(part(mask_d)) : (mask_d.defined() ? OptTensor(mask_d) : std::nullopt),
                bias_d, qs, ks, softmax_scale, 0, part(dout), true, false, 0, form, st);
      if (blocks > 1) {
        ev[2 * i + 1].record(main);
        ev[2 * i + 1].block(s_out);
      }
      const size_t row = out.nbytes() / B1;
      copy(static_cast<char*>(out.data_ptr()) + lo * row, static_cast<const char*>(dout.data_ptr()) + lo * row, (hi - lo) * row,
           cudaMemcpyDeviceToHost, s_out);
    }
    AF3K_CUDA_CHECK(cudaStreamSynchronize(s_out));     // behind the last kernel and, through it, the last copy in
    drain.done = true;
  }
  if (st[0] != 0) {
    throw std::runtime_error("af3k kernel reported status " + std::to_string(st[0]) + " (wait timeout: barrier slot " +
                             std::to_string(st[1] - 1) + ", block " + std::to_string(st[2]) + ", warp " + std::to_string(st[3]) +
                             "); the output is not valid");
  }
}

// ------------------------------------------------------------------ the ordinary calls, straight from Python
// Each returns None for what is not ordinary; the Python function then takes its general way.  Attribute look-ups, transposed
// views and checks in Python were most of the host time of a small call.  Host time of a call, us, before -> after:
// operator 8.0 -> 7.4, grid module 21.4 -> 15.2, single block 17.5 -> 11.5.
bool plain_mask(py::handle mask, int most_dims) {
  if (mask.is_none()) return true;
  if (!THPVariable_Check(mask.ptr())) return false;
  const Tensor& t = THPVariable_Unpack(mask.ptr());
  return t.scalar_type() == at::kBool && t.dim() >= 1 && t.dim() <= most_dims;
}
OptTensor mask_of(py::handle mask) { return mask.is_none() ? OptTensor() : OptTensor(THPVariable_Unpack(mask.ptr())); }

py::object operator_call(const Tensor& q, const Tensor& k, const Tensor& v, py::handle mask, py::handle bias, const OptTensor& q_scale, const OptTensor& k_scale) {
  if (!q.is_cuda() || !plain_mask(mask, 2) || !THPVariable_Check(bias.ptr())) return py::none();
  Tensor out;
  {
    const OptTensor m = mask_of(mask);
    const Tensor b = THPVariable_Unpack(bias.ptr());
    const py::gil_scoped_release nogil;
    out = attention(q, k, v, m, b, q_scale, k_scale, std::nullopt, 0, std::nullopt, true, false, 0, 3);
  }
  return py::cast(std::move(out));
}

// What attribute access finds in an instance's own dictionary (borrowed, null if nothing).
py::object own_dict(py::handle object) {
  py::object d = py::reinterpret_steal<py::object>(PyObject_GenericGetDict(object.ptr(), nullptr));
  if (!d) PyErr_Clear();
  return d;
}
PyObject* own(py::handle object, PyObject* name) {
  const py::object d = own_dict(object);
  return d && PyDict_Check(d.ptr()) ? PyDict_GetItemWithError(d.ptr(), name) : nullptr;
}
PyObject* entry(PyObject* dict, PyObject* name) { return dict != nullptr && PyDict_Check(dict) ? PyDict_GetItemWithError(dict, name) : nullptr; }

// GridSelfAttentionCpp.forward where its layers are torch's own, their parameters plain tensors and nothing is differentiated.
py::object grid_forward(py::handle module, const Tensor& pair, py::handle mask, py::handle linear, py::handle layer_norm) {
  static PyObject* const names[8] = {PyUnicode_InternFromString("q_projection"), PyUnicode_InternFromString("k_projection"),
                                     PyUnicode_InternFromString("v_projection"), PyUnicode_InternFromString("gating_query"),
                                     PyUnicode_InternFromString("output_projection"), PyUnicode_InternFromString("act_norm"),
                                     PyUnicode_InternFromString("act_norm"), PyUnicode_InternFromString("pair_bias_projection")};
  static PyObject* const modules = PyUnicode_InternFromString("_modules"), *const parameters = PyUnicode_InternFromString("_parameters"),
                  *const weight = PyUnicode_InternFromString("weight"), *const bias = PyUnicode_InternFromString("bias"),
                  *const heads = PyUnicode_InternFromString("num_head"), *const transposed = PyUnicode_InternFromString("transpose"),
                  *const epsilon = PyUnicode_InternFromString("eps"), *const hooks = PyUnicode_InternFromString("_forward_hooks"),
                  *const pre_hooks = PyUnicode_InternFromString("_forward_pre_hooks");
  PyObject* const head = own(module, heads);
  PyObject* const transpose = own(module, transposed);
  if (head == nullptr || !PyLong_Check(head) || transpose == nullptr || !PyBool_Check(transpose) || mask.is_none() || !plain_mask(mask, 2)) return py::none();
  const int64_t H = PyLong_AsLongLong(head);
  if (!grid_fused(pair, H, H)) return py::none();
  const py::object of_module = own_dict(module);
  PyObject* const layers = entry(of_module.ptr(), modules);
  std::vector<Tensor> params;
  params.reserve(8);
  double eps = 0;
  for (int i = 0; i < 8; ++i) {
    if (entry(of_module.ptr(), names[i]) != nullptr) return py::none();                       // set past the module's layers
    PyObject* const layer = entry(layers, names[i]);
    const bool norm = i == 5 || i == 6;
    if (layer == nullptr || Py_TYPE(layer) != (PyTypeObject*)(norm ? layer_norm : linear).ptr()) return py::none();
    if (own(layer, weight) != nullptr || own(layer, bias) != nullptr) return py::none();        // set past its parameters
    PyObject* const own_params = own(layer, parameters);
    PyObject* const p = entry(own_params, i == 6 ? bias : weight);
    if (p == nullptr || !THPVariable_Check(p)) return py::none();
    if (i >= 5 && pair.size(2) != 128) {
      // other widths call LayerNorm and bias projection as modules
      PyObject *const h = own(layer, hooks), *const ph = own(layer, pre_hooks), *const b = entry(own_params, bias);
      if (h == nullptr || ph == nullptr || PyObject_Size(h) != 0 || PyObject_Size(ph) != 0 || (i == 7 && (b == nullptr || b != Py_None))) return py::none();
    }
    if (i == 5) {
      PyObject* const e = own(layer, epsilon);
      if (e == nullptr || !PyFloat_Check(e)) return py::none();
      eps = PyFloat_AsDouble(e);
    }
    params.push_back(THPVariable_Unpack(p));
  }
  if (at::GradMode::is_enabled() && params[4].requires_grad()) return py::none();
  Tensor out;
  {
    const Tensor m = THPVariable_Unpack(mask.ptr());
    const py::gil_scoped_release nogil;
    out = grid_module(pair, m, params, eps, H, transpose == Py_True, true);
  }
  return py::cast(std::move(out));
}

py::object self_forward(const Tensor& x, py::handle mask, const Tensor& bias, const Tensor& q, const Tensor& q_bias, const Tensor& k, const Tensor& v,
                        const Tensor& gate, int64_t head) {
  if (x.dim() != 2 || !x.is_cuda() || head < 1 || !plain_mask(mask, 1)) return py::none();
  const int64_t C = x.size(1), D = C / head;
  if (C % head != 0 || D % 8 != 0 || D < 8 || D > 64 || C > 1024) return py::none();
  Tensor out;
  {
    const OptTensor m = mask_of(mask);
    const py::gil_scoped_release nogil;
    out = self_block(x, m, bias, {q, k, v, gate}, q_bias, head);
  }
  return py::cast(std::move(out));
}

}  // namespace

PYBIND11_MODULE(_host, m) {
  m.def("grid_fused", &grid_fused);
  m.def("grid_sizes_fused", &grid_sizes_fused);
  m.def("grid_module", &grid_module, py::call_guard<py::gil_scoped_release>());
  m.def("grid_block", &grid_block, py::call_guard<py::gil_scoped_release>());
  m.def("self_block", &self_block, py::call_guard<py::gil_scoped_release>());
  m.def("operator_call", &operator_call);
  m.def("grid_forward", &grid_forward);
  m.def("self_forward", &self_forward);
  m.def("stage_bias", [](const Tensor& bias, int64_t B2, int64_t Sq, int64_t Sk, int64_t D, const OptTensor& q_scale, const OptTensor& k_scale,
                         double scale) {
    const c10::cuda::CUDAGuard guard(bias.device());
    return make_staged(bias, B2, Sq, Sk, D, q_scale ? q_scale->data_ptr<float>() : nullptr, k_scale ? k_scale->data_ptr<float>() : nullptr,
                       (float)scale, c10::cuda::getCurrentCUDAStream(bias.device().index()));
  }, py::call_guard<py::gil_scoped_release>());
  m.def("host_attention", &host_attention, py::call_guard<py::gil_scoped_release>());
  m.def("bind_library", &bind_library);
  m.def("status_buffer", &status_buffer);
  m.def("attention", [](const Tensor& q, const Tensor& k, const Tensor& v, const OptTensor& mask, const Tensor& bias, const OptTensor& q_scale,
                        const OptTensor& k_scale, std::optional<double> softmax_scale, int64_t rows_per_item, const OptTensor& out,
                        bool use_workspace, bool cache_bias, int64_t max_ctas, int64_t bias_form) {
    return attention(q, k, v, mask, bias, q_scale, k_scale, softmax_scale, rows_per_item, out, use_workspace, cache_bias, max_ctas, bias_form);
  }, py::call_guard<py::gil_scoped_release>());
}
