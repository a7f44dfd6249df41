// NVFP4 block arithmetic shared by the quantize kernels and the kernels that quantize what they produce.
//   global = (amax / 6) / 448, 0 -> 1
//   s_blk  = e4m3_rne(min((amax_blk / 6) / global, 448));  d = fp32(s_blk) * global
//   code   = e2m1_rne_sat(x_fp32 / d); all codes of a block with s_blk == 0 are 0
#pragma once

#include "common.cuh"

namespace b200q {
namespace {

// byte offset of the 4-byte scale word holding scale columns [4*(c/4), 4*(c/4)+4) of row r
__device__ __forceinline__ int64_t swizzled_word_offset(int64_t r, int64_t c, int64_t col_tiles) {
  const int64_t tile = (r >> 7) * col_tiles + (c >> 2);
  return tile * 512 + (r & 31) * 16 + ((r >> 5) & 3) * 4;
}

// eight fp32 -> eight E2M1 nibbles in one word (RNE, saturating), element 0 in the lowest nibble
__device__ __forceinline__ uint32_t pack8_e2m1(float a0, float a1, float a2, float a3, float a4, float a5, float a6, float a7) {
  uint32_t r;
  asm("{\n\t.reg .b8 b0, b1, b2, b3;\n\t"
      "cvt.rn.satfinite.e2m1x2.f32 b0, %2, %1;\n\t"
      "cvt.rn.satfinite.e2m1x2.f32 b1, %4, %3;\n\t"
      "cvt.rn.satfinite.e2m1x2.f32 b2, %6, %5;\n\t"
      "cvt.rn.satfinite.e2m1x2.f32 b3, %8, %7;\n\t"
      "mov.b32 %0, {b0, b1, b2, b3};\n\t}"
      : "=r"(r)
      : "f"(a0), "f"(a1), "f"(a2), "f"(a3), "f"(a4), "f"(a5), "f"(a6), "f"(a7));
  return r;
}

constexpr float kRcp6 = 0.16666667163372039794921875f;   // RN(1/6)
constexpr float kRcp448 = 0.002232142956927418708801269531f;  // RN(1/448)

// Per-launch constants of the scale computation: global scale, its reciprocal, and whether
// the shared-divisor sequence may be used for divisions by it.
struct GlobalScale {
  float g, yg;
  bool fast;
  __device__ __forceinline__ explicit GlobalScale(float amax) {
    // (amax / 6) / 448 as exact IEEE quotients; the shared-divisor sequence is exact for a
    // numerator in the normal range away from its ends, anything else takes true divisions
    const uint32_t e = (__float_as_uint(amax) >> 23) & 0xffu;
    if (e >= 64u && e <= 190u) {
      g = b200q_div_by_shared(b200q_div_by_shared(amax, kE2M1Max, kRcp6), kE4M3Max, kRcp448);
    } else {
      g = nvfp4_global_from_amax(amax);
    }
    yg = b200q_rcp_rn(g);
    fast = b200q_div_fast_ok(g);
  }
};


// Codes of N values (8 or 16) of a block whose abs-max is `a`: returns the 8-bit scale, writes the codes as N / 8 words and
// the effective divisor d = fp32(scale) * global.  `a` is NaN when every value of the block is, and only then; its scale is
// then NaN too (0x7f).  So the maximum has to be folded from the values themselves: fmaxf from a zero drops it.
template <int N>
__device__ __forceinline__ uint32_t quantize_values(const float* f, float a, const GlobalScale& gs, uint32_t* codes, float& d_out) {
  // s = (a / 6) / g, both as exact IEEE quotients
  float s;
  if (gs.fast) {
    s = b200q_div_by_shared(b200q_div_by_shared(a, kE2M1Max, kRcp6), gs.g, gs.yg);
  } else {
    s = __fdiv_rn(__fdiv_rn(a, kE2M1Max), gs.g);
  }
  const bool clamped = s > kE4M3Max;
  const uint32_t sb = f32x2_to_e4m3x2(s, 0.0f) & 0xffu;  // saturates to 448
  const float d = __fmul_rn(e4m3_to_f32(sb), gs.g);
  d_out = d;
  float q[N];
  if (sb != 0u && !clamped && b200q_div_fast_ok(d)) {
    // common case: |x| <= 6.5 d, so the quotient can neither overflow nor need a clamp
    const float y = b200q_rcp_rn(d);
#pragma unroll
    for (int i = 0; i < N; ++i) q[i] = b200q_div_by_shared(f[i], d, y);
  } else if (sb != 0u) {
    // stored scale saturated at 448 (amax input below the data) or an extreme divisor:
    // true division on a numerator clamped to 8 d, which still saturates to +-6
    const float lim = __fmul_rn(d, 8.0f);
#pragma unroll
    for (int i = 0; i < N; ++i) q[i] = with_sign_of(__fdiv_rn(fminf(fabsf(f[i]), lim), d), f[i]);
  } else {
#pragma unroll
    for (int i = 0; i < N / 8; ++i) codes[i] = 0u;
    return sb;
  }
#pragma unroll
  for (int i = 0; i < N; i += 8) codes[i / 8] = pack8_e2m1(q[i], q[i + 1], q[i + 2], q[i + 3], q[i + 4], q[i + 5], q[i + 6], q[i + 7]);
  return sb;
}

// The same with the block's values negated (nf = -f): the quotients of two values at a time (div2_by_shared_negated).
template <int N>
__device__ __forceinline__ uint32_t quantize_negated(const float* nf, float a, const GlobalScale& gs, uint32_t* codes) {
  float s;
  if (gs.fast) {
    s = b200q_div_by_shared(b200q_div_by_shared(a, kE2M1Max, kRcp6), gs.g, gs.yg);
  } else {
    s = __fdiv_rn(__fdiv_rn(a, kE2M1Max), gs.g);
  }
  const bool clamped = s > kE4M3Max;
  const uint32_t sb = f32x2_to_e4m3x2(s, 0.0f) & 0xffu;  // saturates to 448
  const float d = __fmul_rn(e4m3_to_f32(sb), gs.g);
  float q[N];
  if (sb != 0u && !clamped && b200q_div_fast_ok(d)) {
    const float y = b200q_rcp_rn(d);
    const uint64_t dd = pack2(d, d), ny = pack2(-y, -y);
#pragma unroll
    for (int i = 0; i < N; i += 2) {
      const float2 t = unpack2(div2_by_shared_negated(pack2(nf[i], nf[i + 1]), dd, ny));
      q[i] = t.x, q[i + 1] = t.y;
    }
  } else if (sb != 0u) {
    const float lim = __fmul_rn(d, 8.0f);
#pragma unroll
    for (int i = 0; i < N; ++i) q[i] = with_sign_of(__fdiv_rn(fminf(fabsf(nf[i]), lim), d), -nf[i]);
  } else {
#pragma unroll
    for (int i = 0; i < N / 8; ++i) codes[i] = 0u;
    return sb;
  }
#pragma unroll
  for (int i = 0; i < N; i += 8) codes[i / 8] = pack8_e2m1(q[i], q[i + 1], q[i + 2], q[i + 3], q[i + 4], q[i + 5], q[i + 6], q[i + 7]);
  return sb;
}

// Quantize one block held in f[16].
__device__ __forceinline__ uint32_t quantize_block(const float* f, const GlobalScale& gs, uint32_t& c_lo, uint32_t& c_hi,
                                                   float& d_out) {
  float m[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) m[i] = fmaxf(fabsf(f[2 * i]), fabsf(f[2 * i + 1]));
  const float a = fmaxf(fmaxf(fmaxf(m[0], m[1]), fmaxf(m[2], m[3])), fmaxf(fmaxf(m[4], m[5]), fmaxf(m[6], m[7])));
  uint32_t codes[2];
  const uint32_t sb = quantize_values<16>(f, a, gs, codes, d_out);
  c_lo = codes[0];
  c_hi = codes[1];
  return sb;
}

// Where the NVFP4 form of a fused kernel puts its result.
struct Nvfp4Out {
  const float* amax;     // tensor amax (calibrated)
  uint8_t* codes;        // [rows, cols / 2]
  uint8_t* sf;           // swizzled block scales
  float* gout;           // global scale, may be null
  uint32_t col_tiles;    // scale tiles per 128 rows
};

// Scale words of row `row` >= rows of the last 128-row tile: zero (padding the GEMM may read).  All threads of a CTA.
__device__ __forceinline__ void zero_scale_row(uint8_t* sf, int64_t row, uint32_t col_tiles) {
  uint8_t* p = sf + (row >> 7) * static_cast<int64_t>(col_tiles) * 512 + (row & 31) * 16 + ((row >> 5) & 3) * 4;
  for (uint32_t c = threadIdx.x; c < col_tiles; c += blockDim.x) *reinterpret_cast<uint32_t*>(p + c * 512u) = 0u;
}

}  // namespace
}  // namespace b200q
