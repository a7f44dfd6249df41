// Calls inside the library that the public header does not carry: the quantize entry points with `late` (see
// common.cuh::pdl_enter), used where a GEMM on the same stream follows directly.
#pragma once

#include <stdint.h>

#include "b200q.h"

namespace b200q {
int fp8_quantize(const void* x, int dtype, int64_t rows, int64_t cols, const float* amax, int64_t amax_numel, uint8_t* codes_out,
                 float* scales_out, b200q_stream_t stream, bool late);
int silu_mul_fp8_quantize(const void* gate_up, uint8_t* codes_out, float* scales_out, int64_t rows, int64_t f, b200q_stream_t stream,
                          bool late);
int nvfp4_quantize(const void* x, int dtype, int64_t rows, int64_t cols, const float* amax, uint8_t* codes_out, uint8_t* scales_out,
                   float* global_scale_out, b200q_stream_t stream, bool late);
int nvfp4_quantize_dynamic(const void* x, int dtype, int64_t rows, int64_t cols, uint8_t* codes_out, uint8_t* scales_out,
                           float* global_scale_out, void* workspace, size_t workspace_bytes, b200q_stream_t stream, bool late);
size_t nvfp4_dynamic_workspace_bytes(int dtype, int64_t rows, int64_t cols);   // 0: one launch
// bf16 out [M, N] = fp8(x [M, K]) @ dequant(w [N, K])^T + bias in one launch, or 1: not one of the
// sizes where that is faster (gemm_fp8.cu), take fp8_quantize and the GEMM
int fp8_linear_small(const void* x, int dtype, const float* amax, int64_t amax_numel, const uint8_t* w, const float* w_scales,
                     int64_t w_scales_numel, const void* bias, void* out, int64_t M, int64_t N, int64_t K, b200q_stream_t stream);
}  // namespace b200q
