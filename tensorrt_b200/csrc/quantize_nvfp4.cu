// NVFP4 dynamic block quantize: E2M1 codes (two per byte), E4M3 block scales written
// straight into the 128x4 swizzled layout the block-scaled tensor-core MMA reads, fp32
// global scale.  Fake-quantize and dequantize share the arithmetic.
//
// HBM-bound streaming kernel.  One thread owns one 16-element block: a single 256-bit
// load (bf16/fp16) brings it in, the block abs-max needs no cross-lane traffic, the 16
// codes leave as one 64-bit store, and four neighbouring lanes (four consecutive blocks
// of one row = one 4-byte word of the swizzled scale layout) merge their scale bytes with
// two shuffles into one 32-bit store.  A warp therefore reads 1 KiB and writes 256 B of
// codes + 32 B of scales per step, all fully coalesced.  The kernel is only HBM-bound if
// it issues few instructions per element (~14 issue slots per element are available at
// full bandwidth): divisions go through the shared-divisor sequence of exact_div.h, the
// grid is (row, chunk) so no index division is needed, and each lane has two loads in
// flight before it starts computing.
//
// Arithmetic contract (identical to the CPU restatement the tests compare against):
//   global = (amax / 6) / 448, 0 -> 1
//   s_blk  = e4m3_rne(min((amax_blk / 6) / global, 448));  d = fp32(s_blk) * global
//   code   = e2m1_rne_sat(x_fp32 / d); all codes of a block with s_blk == 0 are 0
//   x_hat  = e2m1 * d, rounded (RNE) to the input dtype.
#include "internal.h"
#include "nvfp4_block.cuh"

namespace b200q {
namespace {

constexpr int kThreads = 256;

// Block16<T>: one 16-element block.  `Raw` is what a lane keeps in registers while its loads
// are in flight; `widen` turns it into 16 fp32 values.
template <typename T>
struct Block16;

template <>
struct Block16<__nv_bfloat16> {
  struct Raw { U32x8 w; };
  __device__ static __forceinline__ Raw load_raw(const __nv_bfloat16* p) { return Raw{ld_nc_256(p)}; }
  __device__ static __forceinline__ void widen(const Raw& r, float* f) {
    Elem<__nv_bfloat16>::unpack(make_uint4(r.w.v[0], r.w.v[1], r.w.v[2], r.w.v[3]), f);
    Elem<__nv_bfloat16>::unpack(make_uint4(r.w.v[4], r.w.v[5], r.w.v[6], r.w.v[7]), f + 8);
  }
  __device__ static __forceinline__ void store(__nv_bfloat16* p, const float* f) {
    U32x8 w;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      __nv_bfloat162 h = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
      w.v[i] = *reinterpret_cast<uint32_t*>(&h);
    }
    st_256(p, w);
  }
};

template <>
struct Block16<__half> {
  struct Raw { U32x8 w; };
  __device__ static __forceinline__ Raw load_raw(const __half* p) { return Raw{ld_nc_256(p)}; }
  __device__ static __forceinline__ void widen(const Raw& r, float* f) {
    Elem<__half>::unpack(make_uint4(r.w.v[0], r.w.v[1], r.w.v[2], r.w.v[3]), f);
    Elem<__half>::unpack(make_uint4(r.w.v[4], r.w.v[5], r.w.v[6], r.w.v[7]), f + 8);
  }
  __device__ static __forceinline__ void store(__half* p, const float* f) {
    U32x8 w;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      __half2 h = __floats2half2_rn(f[2 * i], f[2 * i + 1]);
      w.v[i] = *reinterpret_cast<uint32_t*>(&h);
    }
    st_256(p, w);
  }
};

template <>
struct Block16<float> {
  struct Raw { U32x8 a, b; };
  __device__ static __forceinline__ Raw load_raw(const float* p) { return Raw{ld_nc_256(p), ld_nc_256(p + 8)}; }
  __device__ static __forceinline__ void widen(const Raw& r, float* f) {
#pragma unroll
    for (int i = 0; i < 8; ++i) f[i] = __uint_as_float(r.a.v[i]), f[8 + i] = __uint_as_float(r.b.v[i]);
  }
  __device__ static __forceinline__ void store(float* p, const float* f) {
    U32x8 a, b;
#pragma unroll
    for (int i = 0; i < 8; ++i) a.v[i] = __float_as_uint(f[i]), b.v[i] = __float_as_uint(f[8 + i]);
    st_256(p, a);
    st_256(p + 8, b);
  }
};

// Where a block's 16 values come from.
//   Src::kPlain     row-major [rows, cols]
//   Src::kSiluMul   silu(gate) * up of a [rows, 2 cols] gate/up projection (gate columns first), rounded to bf16 as
//                   silu_mul_kernel stores it: the activation in front of the down projection is never written
//   Src::kExpand    column c of the output is column src_col0 + (c / hd / rep) * hd + c % hd of a row of src_stride
//                   elements (every kv head repeated `rep` times): the expanded tensor is never written
// Measured at [8192, 14336] bf16: kSiluMul 146 us (3.7 TB/s; issue slots: about 17 instructions an element) against 114 for
// silu_mul_kernel and 55 for the plain form behind it.
enum class Src { kPlain, kSiluMul, kExpand };
struct ExpandMap {
  int64_t src_stride, src_col0;
  uint32_t head_dim, rep;
};

// FAKE = false: codes + swizzled scales.  FAKE = true: dequantized values in T.
// Grid: x = row, y = chunk of the row, the last row first: a tensor that a kernel before this one read or wrote from the first row
// on and that does not fit L2 is there from its end only (8191 x 5120 bf16, FP8 and NVFP4 fake-quantize of one tensor behind each
// other 57.9 -> 56.0 us).  Codes in front of a GEMM, which takes the first rows first: 0.991 of the time of whole linears (119 sizes of 1 to
// 8192 rows; nothing beyond the spread at 8192 x 14336 -> 4096).  Behind itself, with nothing else in between, a few us at some hundred
// rows go either way with the place of the padding rows (700 x 2048 3.5 -> 2.8, 1184 x 4096 5.1 -> 5.8).  A warp covers U spans of 32
// consecutive blocks
// (512 elements each); all U 256-bit loads of a lane are issued before any arithmetic.
// Rows from `rows` to the end of the last 128-row scale tile (FAKE = false) only clear their scale words.
template <typename T, bool FAKE, int U, Src SRC>
__global__ void __launch_bounds__(kThreads)
nvfp4_quantize_kernel(const T* __restrict__ x, const float* __restrict__ amax, uint8_t* __restrict__ codes,
                      uint8_t* __restrict__ sf, T* __restrict__ fake, float* __restrict__ gout, uint32_t rows, uint32_t cols,
                      uint32_t blocks_per_row, uint32_t col_tiles, const ExpandMap map, bool late) {
  pdl_enter(late);
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const int64_t row = static_cast<int64_t>(gridDim.x) - 1 - blockIdx.x;
  if constexpr (!FAKE) {
    if (row >= rows) {
      if (blockIdx.y == 0) zero_scale_row(sf, row, col_tiles);
      return;
    }
  }
  const uint32_t blk0 = ((blockIdx.y * (blockDim.x >> 5) + warp) * U) * 32u + lane;
  const T* xr = SRC == Src::kSiluMul ? x + row * 2 * cols : (SRC == Src::kExpand ? x + row * map.src_stride + map.src_col0 : x + row * cols);
  typename Block16<T>::Raw raw[U], up[SRC == Src::kSiluMul ? U : 1];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const uint32_t blk = blk0 + u * 32u;
    if (blk < blocks_per_row) {
      uint32_t col = blk * 16u;
      if constexpr (SRC == Src::kExpand) {
        const uint32_t head = col / map.head_dim;
        col = (head / map.rep) * map.head_dim + (col - head * map.head_dim);
      }
      raw[u] = Block16<T>::load_raw(xr + col);
      if constexpr (SRC == Src::kSiluMul) up[u] = Block16<T>::load_raw(xr + cols + col);
    }
  }
  const GlobalScale gs(ld_dependent(amax));
  if (gout != nullptr && row == 0 && blockIdx.y == 0 && threadIdx.x == 0) *gout = gs.g;
  uint8_t* code_row = codes + row * (cols >> 1);
  uint8_t* sf_row = sf + ((row >> 7) * col_tiles) * 512 + (row & 31) * 16 + ((row >> 5) & 3) * 4;
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const uint32_t blk = blk0 + u * 32u;
    const bool live = blk < blocks_per_row;
    uint32_t sb = 0u, c_lo = 0u, c_hi = 0u;
    float d = 0.0f;
    if (live) {
      float f[16];
      Block16<T>::widen(raw[u], f);
      if constexpr (SRC == Src::kSiluMul) {
        float b[16];
        Block16<T>::widen(up[u], b);
#pragma unroll
        for (int i = 0; i < 16; ++i) f[i] = __bfloat162float(__float2bfloat16_rn(silu_mul_f32(f[i], b[i])));
      }
      sb = quantize_block(f, gs, c_lo, c_hi, d);
    }
    if constexpr (!FAKE) {
      if (live) *reinterpret_cast<uint2*>(code_row + blk * 8u) = make_uint2(c_lo, c_hi);
      uint32_t w = sb << (8u * (lane & 3u));
      w |= __shfl_xor_sync(0xffffffffu, w, 1);
      w |= __shfl_xor_sync(0xffffffffu, w, 2);
      if ((lane & 3u) == 0u && live) *reinterpret_cast<uint32_t*>(sf_row + (blk >> 2) * 512u) = w;
    } else {
      if (live) {
        float o[16];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          float2 p = e2m1x2_to_f32x2((c_lo >> (8 * i)) & 0xffu);
          o[2 * i] = __fmul_rn(p.x, d), o[2 * i + 1] = __fmul_rn(p.y, d);
          p = e2m1x2_to_f32x2((c_hi >> (8 * i)) & 0xffu);
          o[8 + 2 * i] = __fmul_rn(p.x, d), o[8 + 2 * i + 1] = __fmul_rn(p.y, d);
        }
        Block16<T>::store(fake + row * cols + blk * 16u, o);
      }
    }
  }
}

// Quantize of a small tensor under its own abs-max, measured in the same launch: every CTA that has blocks of its own
// reads the whole tensor (from L2 after the first) for the maximum and quantizes its share; three launches in a row (a
// cleared result, the abs-max, the quantize) cost more.  A thread owns one block; rows take a multiple of four blocks (one
// scale word), the rows that pad the last 128-row scale tile only clear their words.
// Taken up to 256 KB (8 to 64 CTAs read them, 128 at 16 columns) and 2048 CTAs.  Measured against abs-max and quantize in
// a graph, 1 to 4096 rows: at most 128 KB 0.43 to 0.80 of their time in 16 bits, 0.53 to 0.69 in fp32; at 256 KB 0.65 to 1.05
// and 0.60 to 1.00; fp32 of 384 to 512 KB 0.97 to 1.74 (16 x 8192: 8.2 us against 5.2); a single row of 98304, whose
// padding is 3072 CTAs, 7.9 against 6.9.
constexpr int64_t kDynamicMaxBytes = 1 << 18, kDynamicMaxCtas = 2048;
bool dynamic_in_one_launch(int dtype, int64_t rows, int64_t cols) {
  if (rows <= 0 || cols <= 0) return true;
  if (rows > kDynamicMaxBytes / (dtype == B200Q_F32 ? 4 : 2) / cols) return false;
  return (rows + 127) / 128 * 128 * ((cols / 16 + 3) / 4 * 4) <= kDynamicMaxCtas * kThreads;
}

template <typename T>
__global__ void __launch_bounds__(kThreads)
nvfp4_quantize_dynamic_kernel(const T* __restrict__ x, uint8_t* __restrict__ codes, uint8_t* __restrict__ sf, float* __restrict__ gout,
                              uint32_t rows, uint32_t blocks_per_row, uint32_t col_tiles, uint32_t units, bool late) {
  __shared__ float red[kThreads / 32];
  pdl_enter(late);
  const uint32_t unit = blockIdx.x * kThreads + threadIdx.x;
  const uint32_t row = unit / (col_tiles * 4u), blk = unit - row * (col_tiles * 4u);
  const bool live = row < rows && blk < blocks_per_row;
  float amax = 0.0f;
  if ((blockIdx.x * kThreads) / (col_tiles * 4u) < rows) {    // the CTA has blocks of its own
    constexpr int U = sizeof(T) == 4 ? 4 : 8;                 // 256 bytes of loads in flight per lane
    const uint32_t total = rows * blocks_per_row;
    for (uint32_t b0 = threadIdx.x; b0 < total; b0 += U * kThreads) {
      typename Block16<T>::Raw raw[U];
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (b0 + u * kThreads < total) raw[u] = Block16<T>::load_raw(x + static_cast<int64_t>(b0 + u * kThreads) * 16);
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (b0 + u * kThreads < total) {
          float f[16];
          Block16<T>::widen(raw[u], f);
#pragma unroll
          for (int i = 0; i < 16; ++i) amax = fmaxf(amax, fabsf(f[i]));
        }
    }
    amax = warp_max(amax);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = amax;
    __syncthreads();
    amax = warp_max((threadIdx.x & 31) < kThreads / 32 ? red[threadIdx.x & 31] : 0.0f);
  }
  const GlobalScale gs(amax);
  if (unit == 0 && gout != nullptr) *gout = gs.g;
  uint32_t sb = 0u;
  if (live) {
    float f[16], d;
    uint32_t c_lo, c_hi;
    Block16<T>::widen(Block16<T>::load_raw(x + (static_cast<int64_t>(row) * blocks_per_row + blk) * 16), f);
    sb = quantize_block(f, gs, c_lo, c_hi, d);
    *reinterpret_cast<uint2*>(codes + (static_cast<int64_t>(row) * blocks_per_row + blk) * 8) = make_uint2(c_lo, c_hi);
  }
  uint32_t w = sb << (8u * (threadIdx.x & 3u));
  w |= __shfl_xor_sync(0xffffffffu, w, 1);
  w |= __shfl_xor_sync(0xffffffffu, w, 2);
  if ((threadIdx.x & 3u) == 0u && unit < units)
    *reinterpret_cast<uint32_t*>(sf + ((row >> 7) * col_tiles + (blk >> 2)) * 512u + (row & 31u) * 16u + ((row >> 5) & 3u) * 4u) = w;
}

template <typename T>
int launch_dynamic(const void* x, uint8_t* codes, uint8_t* sf, float* gout, int64_t rows, int64_t cols, cudaStream_t st, bool late) {
  const uint32_t bpr = static_cast<uint32_t>(cols >> 4), col_tiles = (bpr + 3u) >> 2;
  const uint32_t units = static_cast<uint32_t>((rows + 127) / 128 * 128) * col_tiles * 4u;   // at most kDynamicMaxCtas * kThreads
  launch_pdl(nvfp4_quantize_dynamic_kernel<T>, dim3((units + kThreads - 1) / kThreads), dim3(kThreads), 0, st, static_cast<const T*>(x), codes,
             sf, gout, static_cast<uint32_t>(rows), bpr, col_tiles, units, late);
  return check_launch();
}

template <typename T>
__global__ void __launch_bounds__(kThreads)
nvfp4_dequantize_kernel(const uint8_t* __restrict__ codes, const uint8_t* __restrict__ sf, const float* __restrict__ gptr,
                        T* __restrict__ out, int64_t rows, int64_t cols) {
  const float g = __ldg(gptr);
  const int64_t blocks_per_row = cols >> 4;
  const int64_t col_tiles = (blocks_per_row + 3) >> 2;
  const int64_t total = rows * blocks_per_row;
  for (int64_t b = blockIdx.x * (int64_t)kThreads + threadIdx.x; b < total; b += (int64_t)gridDim.x * kThreads) {
    const int64_t row = b / blocks_per_row, blk = b - row * blocks_per_row;
    const uint32_t sb = sf[swizzled_word_offset(row, blk, col_tiles) + (blk & 3)];
    const float d = __fmul_rn(e4m3_to_f32(sb), g);
    const uint2 c = *reinterpret_cast<const uint2*>(codes + b * 8);
    float o[16];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float2 p = e2m1x2_to_f32x2((c.x >> (8 * i)) & 0xffu);
      o[2 * i] = __fmul_rn(p.x, d), o[2 * i + 1] = __fmul_rn(p.y, d);
      p = e2m1x2_to_f32x2((c.y >> (8 * i)) & 0xffu);
      o[8 + 2 * i] = __fmul_rn(p.x, d), o[8 + 2 * i + 1] = __fmul_rn(p.y, d);
    }
    Block16<T>::store(out + b * 16, o);
  }
}

template <typename T, bool FAKE, Src SRC = Src::kPlain>
int launch(const void* x, const float* amax, uint8_t* codes, uint8_t* sf, void* fake, float* gout, int64_t rows,
           int64_t cols, cudaStream_t st, const ExpandMap& map = ExpandMap{}, bool late = false) {
  constexpr int U = sizeof(T) == 4 || SRC == Src::kSiluMul ? 2 : 4;  // 128 bytes of loads in flight per lane
  const uint32_t blocks_per_row = static_cast<uint32_t>(cols >> 4);
  const uint32_t spans_per_row = (blocks_per_row + 31u) >> 5;
  const uint32_t warps_needed = (spans_per_row + U - 1) / U;
  // up to 8 warps per CTA; short rows get smaller CTAs instead of idle warps
  const uint32_t warps = warps_needed < 8u ? warps_needed : 8u;
  const uint32_t chunks = (warps_needed + warps - 1) / warps;
  if (chunks > 65535u) return B200Q_ERR_INVALID;
  // real quantize: the padding rows of the last 128-row scale tile are CTAs of the same launch (a memset in front of
  // it cost a launch of its own)
  int64_t grid_rows = FAKE ? rows : (rows + 127) / 128 * 128;
  if (grid_rows > 0x7fffffffLL) {   // beyond the grid limit: clear the last tile in front
    const int64_t ct = (cols / 16 + 3) / 4;
    if (cudaMemsetAsync(sf + (rows / 128) * ct * 512, 0, static_cast<size_t>(ct * 512), st) != cudaSuccess) return B200Q_ERR_CUDA;
    grid_rows = rows;
  }
  dim3 grid(static_cast<unsigned>(grid_rows), chunks), block(warps * 32u);
  launch_pdl(nvfp4_quantize_kernel<T, FAKE, U, SRC>, grid, block, 0, st, static_cast<const T*>(x), amax, codes, sf, static_cast<T*>(fake),
             gout, static_cast<uint32_t>(rows), static_cast<uint32_t>(cols), blocks_per_row, (blocks_per_row + 3u) >> 2, map, late);
  return check_launch();
}

int validate(const void* x, int dtype, int64_t rows, int64_t cols, const float* amax) {
  if (rows < 0 || cols < 0) return B200Q_ERR_INVALID;
  if (rows == 0 || cols == 0) return B200Q_OK;  // empty tensors are a valid no-op, whatever the pointers
  if (x == nullptr || amax == nullptr) return B200Q_ERR_INVALID;
  if (dtype != B200Q_F32 && dtype != B200Q_F16 && dtype != B200Q_BF16) return B200Q_ERR_INVALID;
  if (cols % 16 != 0 || rows > 0x7fffffffLL || cols > 0x7fffffffLL) return B200Q_ERR_INVALID;
  if (!aligned(x, 32)) return B200Q_ERR_ALIGN;
  return B200Q_OK;
}

}  // namespace

int nvfp4_quantize(const void* x, int dtype, int64_t rows, int64_t cols, const float* amax, uint8_t* codes_out, uint8_t* scales_out,
                   float* global_scale_out, b200q_stream_t stream, bool late) {
  if (int rc = validate(x, dtype, rows, cols, amax)) return rc;
  if (rows == 0 || cols == 0) return B200Q_OK;
  if (codes_out == nullptr || scales_out == nullptr) return B200Q_ERR_INVALID;
  if (!aligned(codes_out, 8) || !aligned(scales_out, 16)) return B200Q_ERR_ALIGN;
  if (int rc = check_arch()) return rc;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  switch (dtype) {
    case B200Q_BF16: return launch<__nv_bfloat16, false>(x, amax, codes_out, scales_out, nullptr, global_scale_out, rows, cols, st, ExpandMap{}, late);
    case B200Q_F16: return launch<__half, false>(x, amax, codes_out, scales_out, nullptr, global_scale_out, rows, cols, st, ExpandMap{}, late);
    default: return launch<float, false>(x, amax, codes_out, scales_out, nullptr, global_scale_out, rows, cols, st, ExpandMap{}, late);
  }
}

size_t nvfp4_dynamic_workspace_bytes(int dtype, int64_t rows, int64_t cols) {
  return dynamic_in_one_launch(dtype, rows, cols) ? 0 : b200q_amax_workspace_bytes();
}

int nvfp4_quantize_dynamic(const void* x, int dtype, int64_t rows, int64_t cols, uint8_t* codes_out, uint8_t* scales_out,
                                 float* global_scale_out, void* workspace, size_t workspace_bytes, b200q_stream_t stream, bool late) {
  if (int rc = validate(x, dtype, rows, cols, reinterpret_cast<const float*>(x))) return rc;
  if (rows == 0 || cols == 0) return B200Q_OK;
  if (codes_out == nullptr || scales_out == nullptr) return B200Q_ERR_INVALID;
  if (!aligned(codes_out, 8) || !aligned(scales_out, 16)) return B200Q_ERR_ALIGN;
  const size_t need = nvfp4_dynamic_workspace_bytes(dtype, rows, cols);
  if (need > 0 && (workspace == nullptr || workspace_bytes < need)) return B200Q_ERR_WORKSPACE;
  if (int rc = check_arch()) return rc;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (need == 0) {
    switch (dtype) {
      case B200Q_BF16: return launch_dynamic<__nv_bfloat16>(x, codes_out, scales_out, global_scale_out, rows, cols, st, late);
      case B200Q_F16: return launch_dynamic<__half>(x, codes_out, scales_out, global_scale_out, rows, cols, st, late);
      default: return launch_dynamic<float>(x, codes_out, scales_out, global_scale_out, rows, cols, st, late);
    }
  }
  float* amax = static_cast<float*>(workspace) + 2;      // behind the two words that the abs-max kernel keeps
  if (int rc = b200q_amax(x, dtype, rows * cols, amax, workspace, workspace_bytes, stream)) return rc;
  return nvfp4_quantize(x, dtype, rows, cols, amax, codes_out, scales_out, global_scale_out, stream, late);
}

}  // namespace b200q

using namespace b200q;

extern "C" {

size_t b200q_nvfp4_scale_bytes(int64_t rows, int64_t cols) {
  if (rows <= 0 || cols <= 0) return 0;
  const int64_t rt = (rows + 127) / 128, ct = (cols / 16 + 3) / 4;
  return static_cast<size_t>(rt * ct * 512);
}

int b200q_nvfp4_quantize(const void* x, int dtype, int64_t rows, int64_t cols, const float* amax, uint8_t* codes_out,
                         uint8_t* scales_out, float* global_scale_out, b200q_stream_t stream) {
  return nvfp4_quantize(x, dtype, rows, cols, amax, codes_out, scales_out, global_scale_out, stream, false);
}

size_t b200q_nvfp4_quantize_dynamic_workspace_bytes(int64_t rows, int64_t cols) {
  return nvfp4_dynamic_workspace_bytes(B200Q_F32, rows, cols);     // enough for every type
}

int b200q_nvfp4_quantize_dynamic(const void* x, int dtype, int64_t rows, int64_t cols, uint8_t* codes_out, uint8_t* scales_out,
                                 float* global_scale_out, void* workspace, size_t workspace_bytes, b200q_stream_t stream) {
  return nvfp4_quantize_dynamic(x, dtype, rows, cols, codes_out, scales_out, global_scale_out, workspace, workspace_bytes, stream, false);
}

int b200q_silu_mul_nvfp4_quantize(const void* gate_up, const float* amax, uint8_t* codes_out, uint8_t* scales_out, float* global_scale_out,
                                  int64_t rows, int64_t f, b200q_stream_t stream) {
  if (int rc = validate(gate_up, B200Q_BF16, rows, f, amax)) return rc;
  if (rows == 0 || f == 0) return B200Q_OK;
  if (codes_out == nullptr || scales_out == nullptr) return B200Q_ERR_INVALID;
  if (!aligned(codes_out, 8) || !aligned(scales_out, 16)) return B200Q_ERR_ALIGN;
  if (int rc = check_arch()) return rc;
  return launch<__nv_bfloat16, false, Src::kSiluMul>(gate_up, amax, codes_out, scales_out, nullptr, global_scale_out, rows, f,
                                                     static_cast<cudaStream_t>(stream));
}

int b200q_expand_heads_nvfp4_quantize(const void* src, int64_t src_stride, int64_t src_col0, const float* amax, uint8_t* codes_out,
                                      uint8_t* scales_out, float* global_scale_out, int64_t rows, int heads_out, int rep, int head_dim,
                                      b200q_stream_t stream) {
  if (heads_out <= 0 || rep <= 0 || head_dim <= 0 || head_dim % 16 != 0 || heads_out % rep != 0 || src_stride < 0 || src_col0 < 0 ||
      src_stride % 16 != 0 || src_col0 % 16 != 0)
    return B200Q_ERR_INVALID;
  const int64_t cols = static_cast<int64_t>(heads_out) * head_dim;
  if (rows > 1 && src_col0 + cols / rep > src_stride) return B200Q_ERR_INVALID;      // beyond the row
  if (int rc = validate(src, B200Q_BF16, rows, cols, amax)) return rc;
  if (rows == 0) return B200Q_OK;
  if (codes_out == nullptr || scales_out == nullptr) return B200Q_ERR_INVALID;
  if (!aligned(codes_out, 8) || !aligned(scales_out, 16)) return B200Q_ERR_ALIGN;
  if (int rc = check_arch()) return rc;
  return launch<__nv_bfloat16, false, Src::kExpand>(src, amax, codes_out, scales_out, nullptr, global_scale_out, rows, cols,
                                                    static_cast<cudaStream_t>(stream),
                                                    ExpandMap{src_stride, src_col0, static_cast<uint32_t>(head_dim), static_cast<uint32_t>(rep)});
}

int b200q_nvfp4_fake_quantize(const void* x, int dtype, int64_t rows, int64_t cols, const float* amax, void* out,
                              b200q_stream_t stream) {
  if (int rc = validate(x, dtype, rows, cols, amax)) return rc;
  if (rows == 0 || cols == 0) return B200Q_OK;
  if (out == nullptr) return B200Q_ERR_INVALID;
  if (!aligned(out, 32)) return B200Q_ERR_ALIGN;
  if (int rc = check_arch()) return rc;
  if (rows == 0 || cols == 0) return B200Q_OK;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  switch (dtype) {
    case B200Q_BF16: return launch<__nv_bfloat16, true>(x, amax, nullptr, nullptr, out, nullptr, rows, cols, st);
    case B200Q_F16: return launch<__half, true>(x, amax, nullptr, nullptr, out, nullptr, rows, cols, st);
    default: return launch<float, true>(x, amax, nullptr, nullptr, out, nullptr, rows, cols, st);
  }
}

int b200q_nvfp4_dequantize(const uint8_t* codes, const uint8_t* scales_swizzled, const float* global_scale, int64_t rows,
                           int64_t cols, void* out, int dtype, b200q_stream_t stream) {
  if (codes == nullptr || scales_swizzled == nullptr || global_scale == nullptr || out == nullptr || rows < 0 || cols < 0 ||
      cols % 16 != 0)
    return B200Q_ERR_INVALID;
  if (!aligned(codes, 8) || !aligned(out, 32)) return B200Q_ERR_ALIGN;
  if (int rc = check_arch()) return rc;
  if (rows == 0 || cols == 0) return B200Q_OK;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int64_t total = rows * (cols >> 4);
  int64_t ctas = (total + kThreads - 1) / kThreads;
  const int64_t cap = (int64_t)sm_count() * 16;
  if (ctas > cap) ctas = cap;
  const unsigned grid = static_cast<unsigned>(ctas);
  switch (dtype) {
    case B200Q_BF16: nvfp4_dequantize_kernel<<<grid, kThreads, 0, st>>>(codes, scales_swizzled, global_scale, static_cast<__nv_bfloat16*>(out), rows, cols); break;
    case B200Q_F16: nvfp4_dequantize_kernel<<<grid, kThreads, 0, st>>>(codes, scales_swizzled, global_scale, static_cast<__half*>(out), rows, cols); break;
    case B200Q_F32: nvfp4_dequantize_kernel<<<grid, kThreads, 0, st>>>(codes, scales_swizzled, global_scale, static_cast<float*>(out), rows, cols); break;
    default: return B200Q_ERR_INVALID;
  }
  return check_launch();
}

}  // extern "C"
