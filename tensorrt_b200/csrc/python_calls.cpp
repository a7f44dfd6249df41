// Whole calls of the Python modules (quantize -> GEMM, the gated MLP, FP8 attention, a forward of the decoder stack) as one
// native function each.
//
// A decode step's linear runs for ten to twenty microseconds on the device; the same steps issued one by one from
// Python (argument checks, two to six tensors, a ctypes call per kernel) take longer than that on the host.  The
// functions here issue the same b200q_* calls on the current stream with the scratch of a call in one allocation.
//
// The GEMMs of the linears and the MLP stand directly behind a kernel that quantizes their activation and lets its dependents
// go late (common.cuh::pdl_enter; tests/test_late_quantizers.py), so they may request weight tiles before that kernel ends:
// static_weights without a promise from the caller.  Those of the stack rest on its constructor, which waits for its weights.
//
// They take the plain case only (strided CUDA tensors of the exact Python type, matching sizes, fp32 scales, no
// dispatch or function mode active) and return None for anything else, before anything is launched: the caller then
// takes the general path in capi.py, which converts, or raises the error that belongs to the input.  From the first
// launch on, and for a failure of the device or the driver, a status raises the error that capi.py raises for it.
#include <ATen/ATen.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/TensorSubclassLikeUtils.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAGuard.h>
#include <cuda_runtime_api.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/utils/pybind.h>

#include <array>
#include <cmath>
#include <optional>
#include <vector>

#include "b200q.h"
#include "internal.h"

namespace {

using at::Tensor;

bool plain(PyObject* o) {
  if (!THPVariable_CheckExact(o)) return false;
  const Tensor& t = THPVariable_Unpack(o);
  return t.is_cuda() && t.layout() == at::kStrided && !at::isTensorSubclassLike(t) && !t.is_neg() && !t.is_conj();
}

bool modes_active() { return c10::impl::dispatch_mode_enabled() || at::impl::torch_function_mode_enabled(); }

int dtype_code(const Tensor& t) {
  switch (t.scalar_type()) {
    case at::kFloat: return B200Q_F32;
    case at::kHalf: return B200Q_F16;
    case at::kBFloat16: return B200Q_BF16;
    default: return -1;
  }
}

b200q_stream_t current_stream() { return static_cast<b200q_stream_t>(at::cuda::getCurrentCUDAStream().stream()); }

int64_t up16(int64_t n) { return (n + 15) / 16 * 16; }

// A tensor argument that may be None; `ok` turns false when it is something else than a plain tensor.
const Tensor* optional_arg(PyObject* o, bool& ok) {
  if (o == Py_None) return nullptr;
  if (!plain(o)) {
    ok = false;
    return nullptr;
  }
  return &THPVariable_Unpack(o);
}

// fp32 contiguous tensor of n1 or n2 values on `dev`
bool f32_of(const Tensor& t, int64_t n1, int64_t n2, at::Device dev) {
  return t.scalar_type() == at::kFloat && t.is_contiguous() && t.device() == dev && (t.numel() == n1 || t.numel() == n2);
}

bool codes_of(const Tensor& w, at::Device dev) { return w.scalar_type() == at::kByte && w.dim() == 2 && w.is_contiguous() && w.device() == dev; }

bool bias_of(const Tensor* b, int64_t n, at::Device dev) {
  return b == nullptr || (b->scalar_type() == at::kBFloat16 && b->is_contiguous() && b->numel() == n && b->device() == dev);
}

Tensor bf16_like(const Tensor& x, int64_t n) {
  auto shape = x.sizes().vec();
  shape.back() = n;
  return at::empty(shape, x.options().dtype(at::kBFloat16));
}

const float* f32(const Tensor* t) { return t == nullptr ? nullptr : static_cast<const float*>(t->data_ptr()); }

struct Operand {   // FP8 operand: codes and scales inside a scratch buffer
  uint8_t* codes;
  float* scales;
  int64_t n_scales;
};

// A status that ends the call: raised by `finish` as the B200QError of _lib.check.
struct CallError {
  int status;
  const char* what;
};

void must(int status, const char* what) {
  if (status != B200Q_OK) throw CallError{status, what};
}

// Status of the first launch of a call: false = the arguments were refused, nothing has run.
bool taken(int status, const char* what) {
  if (status == B200Q_ERR_INVALID || status == B200Q_ERR_ALIGN) return false;
  must(status, what);
  return true;
}

// ---------------------------------------------------------------- fp8_linear
std::optional<Tensor> fp8_linear(const Tensor& x_in, const Tensor& w, const Tensor& ws, const Tensor* bias, const Tensor* amax,
                                 const b200q_cfg& cfg) {
  const auto dev = x_in.device();
  const int dt = dtype_code(x_in);
  if (dt < 0 || x_in.dim() < 1 || x_in.numel() == 0 || !codes_of(w, dev)) return std::nullopt;
  const int64_t K = w.size(1), N = w.size(0);
  if (K % 16 != 0 || N == 0 || x_in.size(-1) != K || !f32_of(ws, 1, N, dev) || !bias_of(bias, N, dev)) return std::nullopt;
  const int64_t M = x_in.numel() / K;
  if (amax != nullptr && !f32_of(*amax, 1, M, dev)) return std::nullopt;
  c10::cuda::CUDAGuard guard(dev);
  const Tensor x = x_in.contiguous();
  const int64_t n = amax == nullptr ? 0 : amax->numel(), n_scales = n == 1 ? 1 : M;
  Tensor out = bf16_like(x, N);
  if (cfg.tile_n == 0) {
    const int rc = b200q::fp8_linear_small(x.data_ptr(), dt, f32(amax), n, static_cast<const uint8_t*>(w.data_ptr()), f32(&ws), ws.numel(),
                                           bias == nullptr ? nullptr : bias->data_ptr(), out.data_ptr(), M, N, K, current_stream());
    if (rc != 1) {
      must(rc, "b200q_fp8_gemm");
      return out;
    }
  }
  Tensor scratch = at::empty({up16(M * K) + 4 * n_scales}, x.options().dtype(at::kByte));
  auto* codes = static_cast<uint8_t*>(scratch.data_ptr());
  auto* scales = reinterpret_cast<float*>(codes + up16(M * K));
  const auto st = current_stream();
  if (!taken(b200q::fp8_quantize(x.data_ptr(), dt, M, K, f32(amax), n, codes, scales, st, true), "b200q_fp8_quantize")) return std::nullopt;
  must(b200q_fp8_gemm(codes, scales, n_scales, static_cast<const uint8_t*>(w.data_ptr()), f32(&ws), ws.numel(),
                      bias == nullptr ? nullptr : bias->data_ptr(), out.data_ptr(), M, N, K, st, &cfg),
       "b200q_fp8_gemm");
  return out;
}

// ---------------------------------------------------------------- nvfp4_linear
std::optional<Tensor> nvfp4_linear(const Tensor& x_in, const Tensor& w, const Tensor& wsf, const Tensor& wg, const Tensor* bias,
                                   const Tensor* amax, const b200q_cfg& cfg) {
  const auto dev = x_in.device();
  const int dt = dtype_code(x_in);
  if (dt < 0 || x_in.dim() < 1 || x_in.numel() == 0 || !codes_of(w, dev)) return std::nullopt;
  const int64_t K = w.size(1) * 2, N = w.size(0);
  if (K % 32 != 0 || N == 0 || x_in.size(-1) != K || !f32_of(wg, 1, 1, dev) || !bias_of(bias, N, dev)) return std::nullopt;
  if (wsf.scalar_type() != at::kByte || !wsf.is_contiguous() || wsf.device() != dev ||
      wsf.numel() < static_cast<int64_t>(b200q_nvfp4_scale_bytes(N, K)))
    return std::nullopt;
  if (amax != nullptr && !f32_of(*amax, 1, 1, dev)) return std::nullopt;
  c10::cuda::CUDAGuard guard(dev);
  const Tensor x = x_in.contiguous();
  if (reinterpret_cast<uintptr_t>(x.data_ptr()) % 32 != 0) return std::nullopt;
  const int64_t M = x.numel() / K, sf_bytes = static_cast<int64_t>(b200q_nvfp4_scale_bytes(M, K));
  const int64_t ws_bytes = amax == nullptr ? static_cast<int64_t>(b200q::nvfp4_dynamic_workspace_bytes(dt, M, K)) : 0;
  const int64_t code_bytes = up16(M * K / 2);
  Tensor scratch = at::empty({code_bytes + sf_bytes + 16 + ws_bytes}, x.options().dtype(at::kByte));
  auto* codes = static_cast<uint8_t*>(scratch.data_ptr());
  uint8_t* sf = codes + code_bytes;
  auto* g = reinterpret_cast<float*>(sf + sf_bytes);
  void* workspace = sf + sf_bytes + 16;
  Tensor out = bf16_like(x, N);
  const auto st = current_stream();
  int rc;
  if (amax != nullptr) {
    rc = b200q::nvfp4_quantize(x.data_ptr(), dt, M, K, f32(amax), codes, sf, g, st, true);
  } else {
    // the two words that the abs-max of a large tensor counts in start at zero
    if (ws_bytes > 0 && cudaMemsetAsync(workspace, 0, 16, static_cast<cudaStream_t>(st)) != cudaSuccess) must(B200Q_ERR_CUDA, "b200q_amax");
    rc = b200q::nvfp4_quantize_dynamic(x.data_ptr(), dt, M, K, codes, sf, g, workspace, static_cast<size_t>(ws_bytes), st, true);
  }
  if (!taken(rc, "b200q_nvfp4_quantize")) return std::nullopt;
  must(b200q_nvfp4_gemm(codes, sf, g, static_cast<const uint8_t*>(w.data_ptr()), static_cast<const uint8_t*>(wsf.data_ptr()), f32(&wg),
                        bias == nullptr ? nullptr : bias->data_ptr(), out.data_ptr(), M, N, K, st, &cfg),
       "b200q_nvfp4_gemm");
  return out;
}

// ---------------------------------------------------------------- Fp8GatedMlp.forward
// The kernel choice of Fp8GatedMlp.forward in linear.py, step for step.
std::optional<Tensor> fp8_gated_mlp(const Tensor& x_in, const Tensor& gu, const Tensor& gus, const Tensor& dn, const Tensor& dns,
                                    const Tensor* in_amax, const Tensor* act_amax, const b200q_cfg& cfg) {
  const auto dev = x_in.device();
  const int dt = dtype_code(x_in);
  if (dt < 0 || x_in.dim() < 1 || x_in.numel() == 0 || !codes_of(gu, dev) || !codes_of(dn, dev)) return std::nullopt;
  const int64_t K = gu.size(1), F = gu.size(0) / 2, H = dn.size(0);
  if (K % 16 != 0 || F == 0 || F % 128 != 0 || F > 32768 || gu.size(0) != 2 * F || dn.size(1) != F || H == 0 || x_in.size(-1) != K)
    return std::nullopt;
  if (!f32_of(gus, 1, 2 * F, dev) || !f32_of(dns, 1, H, dev)) return std::nullopt;
  const int64_t M = x_in.numel() / K;
  if ((in_amax != nullptr && !f32_of(*in_amax, 1, M, dev)) || (act_amax != nullptr && !f32_of(*act_amax, 1, M, dev))) return std::nullopt;
  if (cfg.tile_n != 0) return std::nullopt;          // a forced tile shape: the general path hands it to each GEMM
  c10::cuda::CUDAGuard guard(dev);
  const Tensor x = x_in.contiguous();
  const auto st = current_stream();
  const auto bytes = x.options().dtype(at::kByte);
  const int64_t n_in = in_amax == nullptr ? 0 : in_amax->numel(), n_act = act_amax == nullptr ? 0 : act_amax->numel();
  const int64_t in_scales = n_in == 1 ? 1 : M, act_scales = n_act == 1 ? 1 : M;
  // scratch: input codes, activation codes, both scales, and whatever bf16 tensor stands between the GEMMs
  const bool fused = M >= 256, fused_quant = fused && n_act == 1;
  const int64_t mid = fused_quant ? 0 : (fused ? M * F * 2 : M * F * 4 + (n_act ? M * F * 2 : 0));
  const int64_t o_act = up16(M * K), o_s1 = o_act + up16(M * F), o_s2 = o_s1 + up16(4 * in_scales), o_mid = o_s2 + up16(4 * act_scales);
  Tensor scratch = at::empty({o_mid + mid}, bytes);
  auto* base = static_cast<uint8_t*>(scratch.data_ptr());
  auto *xc = base, *ac = base + o_act;
  auto *xs = reinterpret_cast<float*>(base + o_s1), *as = reinterpret_cast<float*>(base + o_s2);
  uint8_t* m1 = base + o_mid;
  const auto* guc = static_cast<const uint8_t*>(gu.data_ptr());
  Tensor out = bf16_like(x, H);
  if (!taken(b200q::fp8_quantize(x.data_ptr(), dt, M, K, f32(in_amax), n_in, xc, xs, st, true), "b200q_fp8_quantize")) return std::nullopt;
  if (fused_quant) {
    must(b200q_fp8_gemm_silu_mul_quantize(xc, xs, in_scales, guc, f32(&gus), gus.numel(), nullptr, f32(act_amax), ac, as, M, 2 * F, K, st, nullptr),
         "b200q_fp8_gemm_silu_mul_quantize");
  } else if (fused) {
    must(b200q_fp8_gemm_silu_mul(xc, xs, in_scales, guc, f32(&gus), gus.numel(), nullptr, m1, M, 2 * F, K, st, nullptr),
         "b200q_fp8_gemm_silu_mul");
    must(b200q::fp8_quantize(m1, B200Q_BF16, M, F, f32(act_amax), n_act, ac, as, st, true), "b200q_fp8_quantize");
  } else {
    must(b200q_fp8_gemm(xc, xs, in_scales, guc, f32(&gus), gus.numel(), nullptr, m1, M, 2 * F, K, st, &cfg), "b200q_fp8_gemm");
    if (n_act) {
      uint8_t* act = m1 + M * F * 4;
      must(b200q_silu_mul(m1, act, M, F, st), "b200q_silu_mul");
      must(b200q::fp8_quantize(act, B200Q_BF16, M, F, f32(act_amax), n_act, ac, as, st, true), "b200q_fp8_quantize");
    } else {
      must(b200q::silu_mul_fp8_quantize(m1, ac, as, M, F, st, true), "b200q_silu_mul_fp8_quantize");
    }
  }
  must(b200q_fp8_gemm(ac, as, act_scales, static_cast<const uint8_t*>(dn.data_ptr()), f32(&dns), dns.numel(), nullptr, out.data_ptr(), M, H, F, st,
                      &cfg),
       "b200q_fp8_gemm");
  return out;
}

// ---------------------------------------------------------------- fp8_sdpa
bool head_strides(const Tensor& t, int64_t* s) {   // 16-byte rows of D contiguous elements; 0 where there is one only
  const int64_t unit = 16 / t.element_size();
  for (int i = 0; i < 3; ++i) {
    s[i] = t.size(i) > 1 ? t.stride(i) : 0;
    if (s[i] < 0 || s[i] % unit != 0) return false;
  }
  return t.stride(3) == 1 && reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0;
}

std::optional<Tensor> fp8_sdpa(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& aq, const Tensor& ak, const Tensor& av, bool causal,
                               double scale) {
  const auto dev = q.device();
  const int dt = dtype_code(q);
  if (dt < 0 || q.dim() != 4 || k.dim() != 4 || k.sizes() != v.sizes() || k.device() != dev || v.device() != dev ||
      k.scalar_type() != q.scalar_type() || v.scalar_type() != q.scalar_type())
    return std::nullopt;
  const int64_t B = q.size(0), Hq = q.size(1), Sq = q.size(2), D = q.size(3), Hkv = k.size(1), Sk = k.size(2);
  if (k.size(0) != B || k.size(3) != D || q.numel() == 0 || k.numel() == 0 || Hq % Hkv != 0 || D % 16 != 0 || D > 128) return std::nullopt;
  if (!f32_of(aq, 1, 1, dev) || !f32_of(ak, 1, 1, dev) || !f32_of(av, 1, 1, dev)) return std::nullopt;
  int64_t strides[9];
  if (!head_strides(q, strides) || !head_strides(k, strides + 3) || !head_strides(v, strides + 6)) return std::nullopt;
  c10::cuda::CUDAGuard guard(dev);
  Tensor out = at::empty(q.sizes(), q.options());
  const int64_t out_strides[3] = {Hq * Sq * D, Sq * D, D};
  Tensor scratch = at::empty({static_cast<int64_t>(b200q_fp8_attention_workspace_bytes(B, Hkv, Sk, D))}, q.options().dtype(at::kByte));
  must(b200q_fp8_attention(q.data_ptr(), k.data_ptr(), v.data_ptr(), dt, strides, f32(&aq), f32(&ak), f32(&av), out.data_ptr(), out_strides,
                           scratch.data_ptr(), static_cast<size_t>(scratch.numel()), B, Hq, Hkv, Sq, Sk, D, static_cast<float>(scale),
                           causal ? 1 : 0, current_stream()),
       "b200q_fp8_sdpa");
  return out;
}

// ---------------------------------------------------------------- DecoderStack.forward on one rank
// The layers of stack.py::DecoderLayer.forward with CudaBackend's kernels, step for step: same calls, same bits.  Issued from
// Python a layer takes 150 to 250 us of host time (nine to eleven calls, two to six tensors each), which is longer than its
// kernels run below about a thousand tokens: three layers of hidden 2048 over 300 tokens 450 us eager, 203 in a graph.
struct QuantizedWeight {
  const Tensor *codes, *scales, *global;   // global: NVFP4
  int64_t n() const { return codes->size(0); }
};
struct StackLayer {
  const Tensor *norm1, *norm2;
  QuantizedWeight qkv, o, gate_up, down;
  const Tensor* amax[4];                   // NVFP4: calibrated ranges of the inputs of qkv, o, gate_up, down
};
struct StackShape {
  int64_t n_q, n_kv, head_dim, seq_len;    // seq_len 0: every kv head repeated in place of attention
  float eps;
  bool fp8, fuse_gate_up;
};

bool weight_of(const QuantizedWeight& w, int64_t n, int64_t k, bool fp8, at::Device dev) {
  if (!codes_of(*w.codes, dev) || w.codes->size(1) != (fp8 ? k : k / 2) || (n > 0 && w.n() != n)) return false;
  if (fp8) return f32_of(*w.scales, 1, w.n(), dev);
  return w.scales->scalar_type() == at::kByte && w.scales->is_contiguous() && w.scales->device() == dev &&
         w.scales->numel() >= static_cast<int64_t>(b200q_nvfp4_scale_bytes(w.n(), k)) && f32_of(*w.global, 1, 1, dev);
}

bool norm_of(const Tensor& w, int64_t n, at::Device dev) {
  return w.scalar_type() == at::kBFloat16 && w.is_contiguous() && w.numel() == n && w.device() == dev;
}

std::optional<Tensor> decoder_stack(const Tensor& h_in, const std::vector<StackLayer>& layers, const StackShape& s) {
  const auto dev = h_in.device();
  if (layers.empty() || h_in.dim() != 2 || h_in.scalar_type() != at::kBFloat16 || !h_in.is_contiguous() || h_in.numel() == 0) return std::nullopt;
  const int64_t T = h_in.size(0), H = h_in.size(1), Q = s.n_q * s.head_dim, KV = s.n_kv * s.head_dim, W = Q + 2 * KV;
  if (s.n_q <= 0 || s.n_kv <= 0 || s.head_dim <= 0 || s.n_q % s.n_kv != 0 || H % 32 != 0 || H > 16384 || s.head_dim % 16 != 0 || s.head_dim > 128 || Q % 32 != 0)
    return std::nullopt;
  if (s.seq_len < 0 || (s.seq_len > 0 && T % s.seq_len != 0)) return std::nullopt;
  if (reinterpret_cast<uintptr_t>(h_in.data_ptr()) % 32 != 0) return std::nullopt;
  const int64_t F = layers[0].gate_up.codes->dim() == 2 ? layers[0].gate_up.n() / 2 : 0;
  if (F <= 0 || F % 32 != 0 || F > 32768) return std::nullopt;
  for (const StackLayer& l : layers) {
    if (!norm_of(*l.norm1, H, dev) || !norm_of(*l.norm2, H, dev) || !weight_of(l.qkv, W, H, s.fp8, dev) || !weight_of(l.o, H, Q, s.fp8, dev) ||
        !weight_of(l.gate_up, 2 * F, H, s.fp8, dev) || !weight_of(l.down, H, F, s.fp8, dev))
      return std::nullopt;
    for (const Tensor* a : l.amax)
      if (!s.fp8 && !f32_of(*a, 1, 1, dev)) return std::nullopt;
  }
  c10::cuda::CUDAGuard guard(dev);
  const auto st = current_stream();
  b200q_cfg cfg{};
  cfg.static_weights = 1;                          // complete since the stack's constructor synchronised
  // the same choices as CudaBackend.gate_up_activation, gate_up_quantize_static and expand_heads_quantize
  const bool fused = s.fuse_gate_up && 2 * F % 256 == 0 && (s.fp8 ? T >= 256 : b200q_nvfp4_gemm_tile(T, 2 * F) == 512);
  const bool attention = s.seq_len > 0, expand_quant = !s.fp8 || KV <= 2048;
  // scratch: an operand (codes, then its scales), what stands between QKV and O or between gate/up and down, the residual stream
  // twice, the output of a row-parallel linear
  const int64_t widest = std::max(H, std::max(Q, F));
  const int64_t code_bytes = up16(s.fp8 ? T * widest : T * widest / 2);
  const int64_t scale_bytes = up16(s.fp8 ? 4 * T : static_cast<int64_t>(b200q_nvfp4_scale_bytes(T, widest)) + 16);
  const int64_t ws_bytes = attention ? up16(static_cast<int64_t>(b200q_fp8_attention_workspace_bytes(T / s.seq_len, s.n_kv, s.seq_len, s.head_dim)) + 16) : 0;
  const bool bf16_heads = attention || !expand_quant;
  const auto up32 = [](int64_t n) { return (n + 31) / 32 * 32; };
  const int64_t qkv_bytes = up32(T * W * 2), head_bytes = bf16_heads ? up32(T * Q * 2) : 0;
  // (NVFP4 with the activation in the GEMM's epilogue: the down projection's operand itself)
  const int64_t ffn_bytes = !fused ? T * F * 4 : (s.fp8 ? T * F * 2 : code_bytes + scale_bytes);
  const int64_t mid_bytes = std::max(qkv_bytes + head_bytes + ws_bytes, ffn_bytes);
  const int64_t row_bytes = up32(T * H * 2);
  const int64_t o_codes = 3 * row_bytes + up32(mid_bytes), o_scales = o_codes + code_bytes;
  Tensor scratch = at::empty({o_scales + scale_bytes}, h_in.options().dtype(at::kByte));
  auto* base = static_cast<uint8_t*>(scratch.data_ptr());
  uint8_t *rows[2] = {base, base + row_bytes}, *delta = base + 2 * row_bytes, *mid = base + 3 * row_bytes;
  uint8_t *qkv = mid, *heads = mid + qkv_bytes, *ws = heads + head_bytes;
  struct Quantized {
    uint8_t *codes, *sf;
    float *scales, *global;
  };
  const auto operand = [&](uint8_t* c) {           // NVFP4: the global scale behind the block scales
    uint8_t* sf = c + code_bytes;
    return Quantized{c, sf, reinterpret_cast<float*>(sf), reinterpret_cast<float*>(sf + scale_bytes - 16)};
  };
  const Quantized x = operand(base + o_codes), act = operand(mid);
  Tensor out = at::empty(h_in.sizes(), h_in.options());
  const auto gemm = [&](const Quantized& a, const QuantizedWeight& w, int64_t k, void* y) {
    const auto* c = static_cast<const uint8_t*>(w.codes->data_ptr());
    if (s.fp8)
      must(b200q_fp8_gemm(a.codes, a.scales, T, c, f32(w.scales), w.scales->numel(), nullptr, y, T, w.n(), k, st, &cfg), "b200q_fp8_gemm");
    else
      must(b200q_nvfp4_gemm(a.codes, a.sf, a.global, c, static_cast<const uint8_t*>(w.scales->data_ptr()), f32(w.global), nullptr, y, T, w.n(), k, st, &cfg),
           "b200q_nvfp4_gemm");
  };
  const auto quantize = [&](const void* y, int64_t k, const Tensor* amax) {
    if (s.fp8) must(b200q_fp8_quantize(y, B200Q_BF16, T, k, nullptr, 0, x.codes, x.scales, st), "b200q_fp8_quantize");
    else must(b200q_nvfp4_quantize(y, B200Q_BF16, T, k, f32(amax), x.codes, x.sf, x.global, st), "b200q_nvfp4_quantize");
  };
  const void* h = h_in.data_ptr();
  const void* d = nullptr;
  int turn = 0;
  bool first = true;
  const auto norm = [&](const Tensor* w, const Tensor* amax) -> bool {
    void* h_out = d == nullptr ? const_cast<void*>(h) : rows[turn];
    const int rc = s.fp8 ? b200q_add_rms_norm_fp8_quantize(h, d, w->data_ptr(), h_out, x.codes, x.scales, T, H, s.eps, st)
                         : b200q_add_rms_norm_nvfp4_quantize(h, d, w->data_ptr(), h_out, f32(amax), x.codes, x.sf, x.global, T, H, s.eps, st);
    const char* what = s.fp8 ? "b200q_add_rms_norm_fp8_quantize" : "b200q_add_rms_norm_nvfp4_quantize";
    if (first && !taken(rc, what)) return false;
    must(rc, what);
    first = false;
    if (d != nullptr) h = h_out, turn ^= 1;
    return true;
  };
  for (const StackLayer& l : layers) {
    if (!norm(l.norm1, l.amax[0])) return std::nullopt;
    gemm(x, l.qkv, H, qkv);
    if (attention) {
      const int64_t B = T / s.seq_len, S = s.seq_len;
      const auto many = [](int64_t n, int64_t stride) { return n > 1 ? stride : int64_t{0}; };
      const int64_t in[3] = {many(B, S * W), 0, many(S, W)};
      const int64_t strides[9] = {in[0], many(s.n_q, s.head_dim), in[2], in[0], many(s.n_kv, s.head_dim), in[2],
                                  in[0], many(s.n_kv, s.head_dim), in[2]};
      const int64_t out_strides[3] = {many(B, S * Q), many(s.n_q, s.head_dim), many(S, Q)};
      auto* amax = reinterpret_cast<float*>(ws + ws_bytes - 16);
      must(b200q_amax_columns(qkv, B200Q_BF16, T, Q, KV, KV, amax, st), "b200q_amax_columns");
      must(b200q_fp8_attention(qkv, qkv + Q * 2, qkv + (Q + KV) * 2, B200Q_BF16, strides, amax, amax + 1, amax + 2, heads, out_strides, ws,
                               static_cast<size_t>(ws_bytes - 16), B, s.n_q, s.n_kv, S, S, s.head_dim,
                               static_cast<float>(1.0 / std::sqrt(static_cast<double>(s.head_dim))), 1, st),
           "b200q_fp8_sdpa");
      quantize(heads, Q, l.amax[1]);
    } else {
      const int rep = static_cast<int>(s.n_q / s.n_kv), n_q = static_cast<int>(s.n_q), hd = static_cast<int>(s.head_dim);
      if (!s.fp8) {
        must(b200q_expand_heads_nvfp4_quantize(qkv, W, Q + KV, f32(l.amax[1]), x.codes, x.sf, x.global, T, n_q, rep, hd, st), "b200q_expand_heads_nvfp4_quantize");
      } else if (expand_quant) {
        must(b200q_expand_heads_fp8_quantize(qkv, W, Q + KV, x.codes, x.scales, T, n_q, rep, hd, st), "b200q_expand_heads_fp8_quantize");
      } else {
        must(b200q_expand_heads(qkv, W, Q + KV, heads, T, n_q, rep, hd, st), "b200q_expand_heads");
        quantize(heads, Q, nullptr);
      }
    }
    gemm(x, l.o, Q, delta);
    d = delta;
    norm(l.norm2, l.amax[2]);
    const auto* gu = static_cast<const uint8_t*>(l.gate_up.codes->data_ptr());
    if (s.fp8 && fused) {
      must(b200q_fp8_gemm_silu_mul(x.codes, x.scales, T, gu, f32(l.gate_up.scales), l.gate_up.scales->numel(), nullptr, mid, T, 2 * F, H, st, nullptr),
           "b200q_fp8_gemm_silu_mul");
      quantize(mid, F, nullptr);
    } else if (fused) {
      must(b200q_nvfp4_gemm_silu_mul_quantize(x.codes, x.sf, x.global, gu, static_cast<const uint8_t*>(l.gate_up.scales->data_ptr()),
                                              f32(l.gate_up.global), f32(l.amax[3]), act.codes, act.sf, act.global, T, 2 * F, H, st),
           "b200q_nvfp4_gemm_silu_mul_quantize");
    } else {
      gemm(x, l.gate_up, H, mid);
      if (s.fp8) must(b200q_silu_mul_fp8_quantize(mid, x.codes, x.scales, T, F, st), "b200q_silu_mul_fp8_quantize");
      else must(b200q_silu_mul_nvfp4_quantize(mid, f32(l.amax[3]), x.codes, x.sf, x.global, T, F, st), "b200q_silu_mul_nvfp4_quantize");
    }
    gemm(fused && !s.fp8 ? act : x, l.down, F, delta);
  }
  must(b200q_add(h, delta, out.data_ptr(), T * H, st), "b200q_add");
  return out;
}

// ---------------------------------------------------------------- Python side
// Runs `fn` without the GIL (allocations and launches) and hands its result over; None = not taken.
template <typename F>
PyObject* finish(F&& fn) {
  std::optional<Tensor> out;
  try {
    pybind11::gil_scoped_release no_gil;
    out = fn();
  } catch (const CallError& e) {
    pybind11::module_::import("tensorrt_b200._lib").attr("check")(e.status, e.what);
  }
  if (!out.has_value()) Py_RETURN_NONE;
  return THPVariable_Wrap(std::move(*out));
}

// tile_n of capi.gemm_config
bool read_cfg(PyObject* tile_n, b200q_cfg& cfg) {
  cfg = b200q_cfg{};
  const long t = PyLong_AsLong(tile_n);
  if (t == -1 && PyErr_Occurred()) return false;
  cfg.tile_n = static_cast<int32_t>(t);
  cfg.static_weights = 1;     // holds behind a late quantize kernel
  return true;
}

PyObject* py_fp8_linear(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  b200q_cfg cfg;
  TORCH_CHECK_VALUE(n == 6, "fp8_linear: 6 arguments expected");
  if (!read_cfg(a[5], cfg)) return nullptr;
  bool ok = plain(a[0]) && plain(a[1]) && plain(a[2]) && !modes_active();
  const Tensor *bias = optional_arg(a[3], ok), *amax = optional_arg(a[4], ok);
  if (!ok) Py_RETURN_NONE;
  return finish([&] { return fp8_linear(THPVariable_Unpack(a[0]), THPVariable_Unpack(a[1]), THPVariable_Unpack(a[2]), bias, amax, cfg); });
  END_HANDLE_TH_ERRORS
}

PyObject* py_nvfp4_linear(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  b200q_cfg cfg;
  TORCH_CHECK_VALUE(n == 7, "nvfp4_linear: 7 arguments expected");
  if (!read_cfg(a[6], cfg)) return nullptr;
  bool ok = plain(a[0]) && plain(a[1]) && plain(a[2]) && plain(a[3]) && !modes_active();
  const Tensor *bias = optional_arg(a[4], ok), *amax = optional_arg(a[5], ok);
  if (!ok) Py_RETURN_NONE;
  return finish([&] {
    return nvfp4_linear(THPVariable_Unpack(a[0]), THPVariable_Unpack(a[1]), THPVariable_Unpack(a[2]), THPVariable_Unpack(a[3]), bias, amax, cfg);
  });
  END_HANDLE_TH_ERRORS
}

PyObject* py_fp8_gated_mlp(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  b200q_cfg cfg;
  TORCH_CHECK_VALUE(n == 8, "fp8_gated_mlp: 8 arguments expected");
  if (!read_cfg(a[7], cfg)) return nullptr;
  bool ok = plain(a[0]) && plain(a[1]) && plain(a[2]) && plain(a[3]) && plain(a[4]) && !modes_active();
  const Tensor *in_amax = optional_arg(a[5], ok), *act_amax = optional_arg(a[6], ok);
  if (!ok) Py_RETURN_NONE;
  return finish([&] {
    return fp8_gated_mlp(THPVariable_Unpack(a[0]), THPVariable_Unpack(a[1]), THPVariable_Unpack(a[2]), THPVariable_Unpack(a[3]),
                         THPVariable_Unpack(a[4]), in_amax, act_amax, cfg);
  });
  END_HANDLE_TH_ERRORS
}

PyObject* py_fp8_sdpa(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  TORCH_CHECK_VALUE(n == 8, "fp8_sdpa: 8 arguments expected");
  const int causal = PyObject_IsTrue(a[6]);
  if (causal < 0) return nullptr;
  for (int i = 0; i < 6; ++i)
    if (!plain(a[i])) Py_RETURN_NONE;
  if (modes_active()) Py_RETURN_NONE;
  const Tensor& q = THPVariable_Unpack(a[0]);
  double scale = 0.0;
  if (a[7] != Py_None) {
    scale = PyFloat_AsDouble(a[7]);
    if (scale == -1.0 && PyErr_Occurred()) return nullptr;
  } else if (q.dim() == 4 && q.size(3) > 0) {
    scale = 1.0 / std::sqrt(static_cast<double>(q.size(3)));
  }
  return finish([&] {
    return fp8_sdpa(q, THPVariable_Unpack(a[1]), THPVariable_Unpack(a[2]), THPVariable_Unpack(a[3]), THPVariable_Unpack(a[4]),
                    THPVariable_Unpack(a[5]), causal != 0, scale);
  });
  END_HANDLE_TH_ERRORS
}

// One layer as a tuple of tensors: norm1, norm2, then codes and scales (NVFP4: and global scale) of qkv, o, gate/up and down,
// NVFP4: then the four ranges.
bool read_layer(PyObject* t, bool fp8, StackLayer& l) {
  const Py_ssize_t n = fp8 ? 10 : 18;
  if (!PyTuple_CheckExact(t) || PyTuple_GET_SIZE(t) != n) return false;
  std::array<const Tensor*, 18> a{};
  for (Py_ssize_t i = 0; i < n; ++i) {
    PyObject* o = PyTuple_GET_ITEM(t, i);
    if (!plain(o)) return false;
    a[i] = &THPVariable_Unpack(o);
  }
  l = StackLayer{};
  l.norm1 = a[0], l.norm2 = a[1];
  int i = 2;
  for (QuantizedWeight* w : {&l.qkv, &l.o, &l.gate_up, &l.down}) {
    w->codes = a[i++], w->scales = a[i++];
    if (!fp8) w->global = a[i++];
  }
  if (!fp8)
    for (int k = 0; k < 4; ++k) l.amax[k] = a[i++];
  return true;
}

PyObject* py_decoder_stack(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  TORCH_CHECK_VALUE(n == 9 && PyList_Check(a[1]), "decoder_stack: 9 arguments expected, the second a list");
  StackShape s{PyLong_AsLongLong(a[2]), PyLong_AsLongLong(a[3]), PyLong_AsLongLong(a[4]), PyLong_AsLongLong(a[5]),
               static_cast<float>(PyFloat_AsDouble(a[6])), PyObject_IsTrue(a[7]) == 1, PyObject_IsTrue(a[8]) == 1};
  if (PyErr_Occurred()) return nullptr;
  if (!plain(a[0]) || modes_active()) Py_RETURN_NONE;
  std::vector<StackLayer> layers(static_cast<size_t>(PyList_GET_SIZE(a[1])));
  for (size_t i = 0; i < layers.size(); ++i)
    if (!read_layer(PyList_GET_ITEM(a[1], static_cast<Py_ssize_t>(i)), s.fp8, layers[i])) Py_RETURN_NONE;
  return finish([&] { return decoder_stack(THPVariable_Unpack(a[0]), layers, s); });
  END_HANDLE_TH_ERRORS
}

PyMethodDef methods[] = {
    {"fp8_linear", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_fp8_linear)), METH_FASTCALL,
     "x, w_codes, w_scales, bias, x_amax, tile_n -> bf16 tensor, or None: take the general path"},
    {"nvfp4_linear", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_nvfp4_linear)), METH_FASTCALL,
     "x, w_codes, w_scales, w_global, bias, x_amax, tile_n -> bf16 tensor or None"},
    {"fp8_gated_mlp", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_fp8_gated_mlp)), METH_FASTCALL,
     "x, gu_codes, gu_scales, down_codes, down_scales, input_amax, act_amax, tile_n -> bf16 tensor or None"},
    {"fp8_sdpa", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_fp8_sdpa)), METH_FASTCALL,
     "q, k, v, amax_q, amax_k, amax_v, is_causal, scale -> tensor like q or None"},
    {"decoder_stack", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_decoder_stack)), METH_FASTCALL,
     "h, layers, n_q, n_kv, head_dim, seq_len, eps, fp8, fuse_gate_up -> tensor like h or None"},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "b200q_native", "Whole calls of the b200q modules", -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_b200q_native() { return PyModule_Create(&module_def); }
