// Whole calls of the Python modules (quantize -> GEMM, the gated MLP, FP8 attention) as one native function each.
//
// A decode step's linear runs for ten to twenty microseconds on the device; the same steps issued one by one from
// Python (argument checks, two to six tensors, a ctypes call per kernel) take longer than that on the host.  The
// functions here issue the same b200q_* calls on the current stream with the scratch of a call in one allocation.
//
// Every GEMM here stands directly behind a kernel that quantizes its activation and lets its dependents go late
// (common.cuh::pdl_enter), so it may request weight tiles before that kernel ends: static_weights without a promise
// from the caller.
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

#include <cmath>
#include <optional>

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

PyMethodDef methods[] = {
    {"fp8_linear", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_fp8_linear)), METH_FASTCALL,
     "x, w_codes, w_scales, bias, x_amax, tile_n -> bf16 tensor, or None: take the general path"},
    {"nvfp4_linear", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_nvfp4_linear)), METH_FASTCALL,
     "x, w_codes, w_scales, w_global, bias, x_amax, tile_n -> bf16 tensor or None"},
    {"fp8_gated_mlp", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_fp8_gated_mlp)), METH_FASTCALL,
     "x, gu_codes, gu_scales, down_codes, down_scales, input_amax, act_amax, tile_n -> bf16 tensor or None"},
    {"fp8_sdpa", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_fp8_sdpa)), METH_FASTCALL,
     "q, k, v, amax_q, amax_k, amax_v, is_causal, scale -> tensor like q or None"},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "b200q_native", "Whole calls of the b200q modules", -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_b200q_native() { return PyModule_Create(&module_def); }
