// Elementwise / row-wise kernels either side of the quantized linears in the decoder
// linear stack: RMSNorm, silu(gate) * up, residual add, and the "attention = identity on V"
// head expansion.  All are HBM-bound streaming kernels over bf16 with 128-bit accesses.
#include <cstdlib>
#include <type_traits>

#include "internal.h"
#include "nvfp4_block.cuh"
#include "tcgen05.cuh"

namespace b200q {
namespace gemm {
int* device_status_word();
}
namespace {

constexpr int kThreads = 256;

__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// float at the same shared-memory address in CTA `rank` of the cluster
__device__ __forceinline__ float ld_cluster_f32(const float* p, int rank) {
  uint32_t local = static_cast<uint32_t>(__cvta_generic_to_shared(p)), remote;
  float v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(rank));
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(remote) : "memory");
  return v;
}

// Eight normalised values per thread (bf16-rounded), one group g of 8 per lane, the two halves of a 16-element block
// in neighbouring lanes -> NVFP4 codes and swizzled block scales of row `row`.  All 32 lanes take part; lanes whose g
// lies beyond the row pass zeros.  The warp's first g is a multiple of 8, so that 8 lanes hold one scale word.
__device__ __forceinline__ void store_nvfp4_group(const float* v, int g, int groups, int64_t row, int64_t cols, const GlobalScale& gs,
                                                  const Nvfp4Out& o) {
  float a = fabsf(v[0]);
#pragma unroll
  for (int j = 1; j < 8; ++j) a = fmaxf(a, fabsf(v[j]));
  a = fmaxf(a, __shfl_xor_sync(0xffffffffu, a, 1));
  uint32_t codes, sb = 0u;
  if (g < groups) {
    float d;
    sb = quantize_values<8>(v, a, gs, &codes, d);
    *reinterpret_cast<uint32_t*>(o.codes + row * (cols >> 1) + static_cast<int64_t>(g) * 4) = codes;
  }
  uint32_t w = (g & 1) == 0 ? sb << (8 * ((g >> 1) & 3)) : 0u;
  w |= __shfl_xor_sync(0xffffffffu, w, 2);
  w |= __shfl_xor_sync(0xffffffffu, w, 4);
  if ((g & 7) == 0 && g < groups)
    *reinterpret_cast<uint32_t*>(o.sf + ((row >> 7) * o.col_tiles + (g >> 3)) * 512 + (row & 31) * 16 + ((row >> 5) & 3) * 4) = w;
}

// y = x * rsqrt(mean(x^2) + eps) * w, fp32 math, bf16 in/out; one CTA per row, the row stays
// in registers (ITEMS groups of 8 per thread) or is re-read (ITEMS == 0).
template <int ITEMS>
__global__ void __launch_bounds__(kThreads)
rms_norm_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w, __nv_bfloat16* __restrict__ y,
                int64_t cols, float eps) {
  pdl_launch_dependents();
  pdl_wait();
  __shared__ float red[kThreads / 32];
  const int64_t row = blockIdx.x;
  const __nv_bfloat16* xr = x + row * cols;
  __nv_bfloat16* yr = y + row * cols;
  const int groups = static_cast<int>(cols >> 3);
  float v[ITEMS > 0 ? ITEMS : 1][8];
  float ss = 0.0f;
  if constexpr (ITEMS > 0) {
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
      const int g = threadIdx.x + i * kThreads;
      if (g < groups) {
        Elem<__nv_bfloat16>::load8(xr + (int64_t)g * 8, v[i]);
#pragma unroll
        for (int j = 0; j < 8; ++j) ss = fmaf(v[i][j], v[i][j], ss);
      }
    }
  } else {
    for (int g = threadIdx.x; g < groups; g += kThreads) {
      float t[8];
      Elem<__nv_bfloat16>::load8(xr + (int64_t)g * 8, t);
#pragma unroll
      for (int j = 0; j < 8; ++j) ss = fmaf(t[j], t[j], ss);
    }
  }
  const float total = block_sum<kThreads>(ss, red);
  const float inv = rsqrtf(total / static_cast<float>(cols) + eps);
  auto emit = [&](int g, const float* t) {
    float wv[8], o[8];
    Elem<__nv_bfloat16>::load8(w + (int64_t)g * 8, wv);
#pragma unroll
    for (int j = 0; j < 8; ++j) o[j] = t[j] * inv * wv[j];
    Elem<__nv_bfloat16>::store8(yr + (int64_t)g * 8, o);
  };
  if constexpr (ITEMS > 0) {
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
      const int g = threadIdx.x + i * kThreads;
      if (g < groups) emit(g, v[i]);
    }
  } else {
    for (int g = threadIdx.x; g < groups; g += kThreads) {
      float t[8];
      Elem<__nv_bfloat16>::load8(xr + (int64_t)g * 8, t);
      emit(g, t);
    }
  }
}

// Residual add + RMSNorm + per-token FP8 quantize of one row per CTA, the row held in registers:
//   h_new = bf16(h + delta)            (delta may be null: h_new = h, nothing is written back)
//   x     = bf16(h_new * rsqrt(mean(h_new^2) + eps) * w)
//   scale = max|x| / 448 (0 -> 1);  code = e4m3(x / scale)
// Same arithmetic and rounding points as add -> rms_norm -> fp8 quantize run one after the
// other, with 1.75 bytes of traffic per element and step instead of 3.25.
// PARTS > 1: a cluster of PARTS CTAs shares one token (few tokens that add_norm_quant_row_kernel does not take: bases that are
// not 32-byte aligned, columns that are no multiple of 16, and up to 16 rows of more than 8192 columns); the slices'
// sums of squares and maxima meet through distributed shared memory, summed in rank order.
// NVF4: the normalised row leaves as NVFP4 codes and block scales under a calibrated tensor amax (`nv`) instead of
// per-token FP8; no row maximum is needed.
// CTAs of the rows that only pad the last 128-row scale tile clear theirs.
template <int ITEMS, int PARTS, bool NVF4>
__global__ void __launch_bounds__(kThreads)
add_norm_quant_kernel(const __nv_bfloat16* __restrict__ h, const __nv_bfloat16* __restrict__ delta,
                      const __nv_bfloat16* __restrict__ w, __nv_bfloat16* __restrict__ h_out, uint8_t* __restrict__ codes,
                      float* __restrict__ scales, int64_t rows, int64_t cols, float eps, const Nvfp4Out nv) {
  pdl_launch_dependents();
  pdl_wait();
  __shared__ float red[kThreads / 32];
  __shared__ float part_val[2];
  const int64_t row = blockIdx.x / PARTS;
  if constexpr (NVF4) {
    if (row >= rows) {                       // whole clusters: no CTA of this token waits for another
      if (blockIdx.x % PARTS == 0) zero_scale_row(nv.sf, row, nv.col_tiles);
      return;
    }
  }
  const int part = PARTS > 1 ? static_cast<int>(blockIdx.x % PARTS) : 0;   // == rank in the cluster
  const int groups = static_cast<int>(cols >> 3);
  int per_part = (groups + PARTS - 1) / PARTS;
  if constexpr (NVF4) per_part = (per_part + 7) / 8 * 8;   // whole scale words
  const int g_begin = min(groups, part * per_part), g_end = min(groups, g_begin + per_part);
  // few-token form: the norm weights are requested together with the row, ahead of the first
  // reduction; many-token form: loaded after it (fewer live registers, more CTAs per SM)
  constexpr bool kEarlyW = PARTS > 1;
  float v[ITEMS][8];
  float wv[kEarlyW ? ITEMS : 1][8];
  float ss = 0.0f;
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) {
    const int g = g_begin + threadIdx.x + i * kThreads;
    if (g < g_end) {
      Elem<__nv_bfloat16>::load8(h + row * cols + (int64_t)g * 8, v[i]);
      if constexpr (kEarlyW) Elem<__nv_bfloat16>::load8(w + (int64_t)g * 8, wv[i]);
      if (delta != nullptr) {
        float d[8];
        Elem<__nv_bfloat16>::load8(delta + row * cols + (int64_t)g * 8, d);
#pragma unroll
        for (int j = 0; j < 8; ++j) v[i][j] = __bfloat162float(__float2bfloat16_rn(v[i][j] + d[j]));
        Elem<__nv_bfloat16>::store8(h_out + row * cols + (int64_t)g * 8, v[i]);
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) ss = fmaf(v[i][j], v[i][j], ss);
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) v[i][j] = 0.0f;
    }
  }
  float total = block_sum<kThreads>(ss, red);
  if constexpr (PARTS > 1) {
    if (threadIdx.x == 0) part_val[0] = total;
    cluster_barrier();
    total = 0.0f;
#pragma unroll
    for (int r = 0; r < PARTS; ++r) total += ld_cluster_f32(&part_val[0], r);
  }
  const float inv = rsqrtf(total / static_cast<float>(cols) + eps);
  float amax = 0.0f;
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) {
    const int g = g_begin + threadIdx.x + i * kThreads;
    if (g < g_end) {
      float wl[8];
      if constexpr (!kEarlyW) Elem<__nv_bfloat16>::load8(w + (int64_t)g * 8, wl);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float wj = kEarlyW ? wv[kEarlyW ? i : 0][j] : wl[j];
        v[i][j] = __bfloat162float(__float2bfloat16_rn(v[i][j] * inv * wj));
        amax = fmaxf(amax, fabsf(v[i][j]));
      }
    }
  }
  if constexpr (NVF4) {
    const GlobalScale gs(ld_dependent(nv.amax));
    if (blockIdx.x == 0 && threadIdx.x == 0 && nv.gout != nullptr) *nv.gout = gs.g;
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) store_nvfp4_group(v[i], g_begin + threadIdx.x + i * kThreads, g_end, row, cols, gs, nv);
    if constexpr (PARTS > 1) cluster_barrier();  // nobody leaves while a peer may still read its shared memory
    return;
  }
  // block max (values are >= 0): reuse the sum scratch
  amax = warp_max(amax);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = amax;
  __syncthreads();
  amax = (threadIdx.x & 31) < kThreads / 32 ? red[threadIdx.x & 31] : 0.0f;
  amax = warp_max(amax);
  if constexpr (PARTS > 1) {
    if (threadIdx.x == 0) part_val[1] = amax;
    cluster_barrier();
    float other = 0.0f;
    if ((threadIdx.x & 31) < PARTS) other = ld_cluster_f32(&part_val[1], threadIdx.x & 31);
    amax = warp_max(other);
    cluster_barrier();  // nobody leaves while a peer may still read its shared memory
  }
  const float scale = fp8_scale_from_amax(amax);
  if (threadIdx.x == 0 && part == 0) scales[row] = scale;
  const float y = b200q_rcp_rn(scale);
  const bool fast = b200q_div_fast_ok(scale);
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) {
    const int g = g_begin + threadIdx.x + i * kThreads;
    if (g < g_end) {
      float q[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) q[j] = fast ? b200q_div_by_shared(v[i][j], scale, y) : __fdiv_rn(v[i][j], scale);
      const uint32_t lo = f32x2_to_e4m3x2(q[0], q[1]) | (f32x2_to_e4m3x2(q[2], q[3]) << 16);
      const uint32_t hi = f32x2_to_e4m3x2(q[4], q[5]) | (f32x2_to_e4m3x2(q[6], q[7]) << 16);
      *reinterpret_cast<uint2*>(codes + row * cols + (int64_t)g * 8) = make_uint2(lo, hi);
    }
  }
}

// Form of add_norm_quant_kernel for many long rows that add_norm_quant_warp_kernel does not take (FP8 with a delta and more
// than 4096 columns, inputs that are not 32-byte aligned): persistent CTAs (two per SM) walk the rows with a stride
// of the grid, and the rows of h and delta arrive through a ring of shared-memory stages filled by
// bulk asynchronous copies that one thread issues `stages` rows ahead.  One CTA per row keeps too few
// bytes in flight to cover the HBM latency (its loads stop while it reduces and stores); here the
// copies of the next rows run during all of that.  What is left is the chain of a row, about 2 us with its barriers: rows
// of 4096 columns and less are bound by it.  Thread-to-element mapping, arithmetic and
// reduction order are those of add_norm_quant_kernel, so the results are bit-identical.
constexpr int kStreamStagesMax = 8;
constexpr int kStreamRingBytes = 96 * 1024;

template <int ITEMS, bool HAS_DELTA, bool NVF4>
__global__ void __launch_bounds__(kThreads, 2)
add_norm_quant_stream_kernel(const __nv_bfloat16* __restrict__ h, const __nv_bfloat16* __restrict__ delta,
                             const __nv_bfloat16* __restrict__ w, __nv_bfloat16* __restrict__ h_out, uint8_t* __restrict__ codes,
                             float* __restrict__ scales, int rows, int cols, float eps, int stages, int* __restrict__ status,
                             const Nvfp4Out nv) {
  pdl_launch_dependents();
  pdl_wait();
  extern __shared__ __align__(128) unsigned char ring[];
  __shared__ uint64_t full[kStreamStagesMax];
  __shared__ float red[kThreads / 32];
  const uint32_t row_bytes = static_cast<uint32_t>(cols) * 2u;
  const uint32_t stage_bytes = row_bytes * (HAS_DELTA ? 2u : 1u);
  const int groups = cols >> 3;
  const int step = static_cast<int>(gridDim.x);
  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) ptx::mbar_init(&full[s], 1);
    ptx::fence_barrier_init();
  }
  __syncthreads();
  auto issue = [&](int row, int s) {
    ptx::mbar_arrive_expect_tx(&full[s], stage_bytes);
    ptx::bulk_load(ring + (size_t)s * stage_bytes, h + (int64_t)row * cols, row_bytes, &full[s]);
    if constexpr (HAS_DELTA) ptx::bulk_load(ring + (size_t)s * stage_bytes + row_bytes, delta + (int64_t)row * cols, row_bytes, &full[s]);
  };
  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) {
      const int64_t row = (int64_t)blockIdx.x + (int64_t)s * step;
      if (row < rows) issue(static_cast<int>(row), s);
    }
  }
  // the norm weights of this thread's groups are the same for every row
  uint4 wp[ITEMS];
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) {
    const int g = threadIdx.x + i * kThreads;
    wp[i] = g < groups ? ld_nc_128(w + (int64_t)g * 8) : make_uint4(0u, 0u, 0u, 0u);
  }
  const GlobalScale gs(NVF4 ? ld_dependent(nv.amax) : 1.0f);
  if constexpr (NVF4) {
    if (blockIdx.x == 0 && threadIdx.x == 0 && nv.gout != nullptr) *nv.gout = gs.g;
    for (int64_t row = rows + blockIdx.x; row < (rows + 127) / 128 * 128; row += step) zero_scale_row(nv.sf, row, nv.col_tiles);
  }
  int k = 0;
  for (int64_t row = blockIdx.x; row < rows; row += step, ++k) {
    const int s = k % stages;
    const bool arrived = ptx::mbar_wait(&full[s], static_cast<uint32_t>(k / stages) & 1u);
    // also separates this row's use of `red` from the previous row's last read of it
    if (__syncthreads_or(!arrived)) {
      if (threadIdx.x == 0) atomicCAS(status, 0, 81);
      break;
    }
    const unsigned char* st = ring + (size_t)s * stage_bytes;
    float v[ITEMS][8];
    float ss = 0.0f;
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
      const int g = threadIdx.x + i * kThreads;
      if (g < groups) {
        Elem<__nv_bfloat16>::unpack(*reinterpret_cast<const uint4*>(st + (size_t)g * 16), v[i]);
        if constexpr (HAS_DELTA) {
          float d[8];
          Elem<__nv_bfloat16>::unpack(*reinterpret_cast<const uint4*>(st + row_bytes + (size_t)g * 16), d);
#pragma unroll
          for (int j = 0; j < 8; ++j) v[i][j] = __bfloat162float(__float2bfloat16_rn(v[i][j] + d[j]));
          Elem<__nv_bfloat16>::store8(h_out + row * cols + (int64_t)g * 8, v[i]);
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) ss = fmaf(v[i][j], v[i][j], ss);
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) v[i][j] = 0.0f;
      }
    }
    const float total = block_sum<kThreads>(ss, red);
    // every thread has taken its part of the stage: refill it with the row `stages` steps ahead
    if (threadIdx.x == 0) {
      const int64_t next = row + (int64_t)stages * step;
      if (next < rows) issue(static_cast<int>(next), s);
    }
    const float inv = rsqrtf(total / static_cast<float>(cols) + eps);
    float amax = 0.0f;
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
      const int g = threadIdx.x + i * kThreads;
      if (g < groups) {
        float wl[8];
        Elem<__nv_bfloat16>::unpack(wp[i], wl);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          v[i][j] = __bfloat162float(__float2bfloat16_rn(v[i][j] * inv * wl[j]));
          amax = fmaxf(amax, fabsf(v[i][j]));
        }
      }
    }
    if constexpr (NVF4) {
#pragma unroll
      for (int i = 0; i < ITEMS; ++i) store_nvfp4_group(v[i], threadIdx.x + i * kThreads, groups, row, cols, gs, nv);
      continue;
    }
    amax = warp_max(amax);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = amax;
    __syncthreads();
    amax = (threadIdx.x & 31) < kThreads / 32 ? red[threadIdx.x & 31] : 0.0f;
    amax = warp_max(amax);
    const float scale = fp8_scale_from_amax(amax);
    if (threadIdx.x == 0) scales[row] = scale;
    const float y = b200q_rcp_rn(scale);
    auto emit = [&](auto fast_tag) {
      constexpr bool kFast = decltype(fast_tag)::value;
#pragma unroll
      for (int i = 0; i < ITEMS; ++i) {
        const int g = threadIdx.x + i * kThreads;
        if (g < groups) {
          float q[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) q[j] = kFast ? b200q_div_by_shared(v[i][j], scale, y) : __fdiv_rn(v[i][j], scale);
          const uint32_t lo = f32x2_to_e4m3x2(q[0], q[1]) | (f32x2_to_e4m3x2(q[2], q[3]) << 16);
          const uint32_t hi = f32x2_to_e4m3x2(q[4], q[5]) | (f32x2_to_e4m3x2(q[6], q[7]) << 16);
          *reinterpret_cast<uint2*>(codes + row * cols + (int64_t)g * 8) = make_uint2(lo, hi);
        }
      }
    };
    if (b200q_div_fast_ok(scale)) emit(std::true_type{});   // one branch per row, not one select per element
    else emit(std::false_type{});
  }
}

// ---- add + RMSNorm + quantize on pieces of 16 elements, packed as bf16

// x + delta.  One bf16 pair addition rounds the exact sum once, and an fp32 addition in front of that rounding changes
// nothing: the sum of two bf16 values that needs more than 24 bits lies next to the larger one.
__device__ __forceinline__ void piece_add(U32x8& x, const U32x8& d) {
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const __nv_bfloat162 t = __hadd2(*reinterpret_cast<const __nv_bfloat162*>(&x.v[j]), *reinterpret_cast<const __nv_bfloat162*>(&d.v[j]));
    x.v[j] = *reinterpret_cast<const uint32_t*>(&t);
  }
}

// Squares of a piece added to `ss`: its low half takes the first 8 elements, the high half the others, each in order.
__device__ __forceinline__ uint64_t piece_squares(const U32x8& x, uint64_t ss) {
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const uint64_t lo = pack2(__uint_as_float(x.v[j] << 16), __uint_as_float(x.v[4 + j] << 16));
    const uint64_t hi = pack2(__uint_as_float(x.v[j] & 0xffff0000u), __uint_as_float(x.v[4 + j] & 0xffff0000u));
    ss = fma2(lo, lo, ss);
    ss = fma2(hi, hi, ss);
  }
  return ss;
}

// -(x * inv * w) rounded to bf16 (ninv = (-inv, -inv)): negated for the divisions of the quantizers, where the signs cancel.
__device__ __forceinline__ void piece_norm_negated(U32x8& x, const uint4& w0, const uint4& w1, uint64_t ninv) {
  const uint32_t w[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const uint64_t xv = pack2(__uint_as_float(x.v[j] << 16), __uint_as_float(x.v[j] & 0xffff0000u));
    const uint64_t wj = pack2(__uint_as_float(w[j] << 16), __uint_as_float(w[j] & 0xffff0000u));
    const float2 t = unpack2(mul2(mul2(xv, ninv), wj));
    const __nv_bfloat162 b = __floats2bfloat162_rn(t.x, t.y);
    x.v[j] = *reinterpret_cast<const uint32_t*>(&b);
  }
}

// abs-max of a piece; NaN only when all its values are
__device__ __forceinline__ float piece_abs_max(const U32x8& x) {
  __nv_bfloat162 m = __habs2(*reinterpret_cast<const __nv_bfloat162*>(&x.v[0]));
#pragma unroll
  for (int j = 1; j < 8; ++j) m = __hmax2(m, __habs2(*reinterpret_cast<const __nv_bfloat162*>(&x.v[j])));
  return fmaxf(__low2float(m), __high2float(m));
}

__device__ __forceinline__ void piece_values(const U32x8& x, float* f) {
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    f[2 * j] = __uint_as_float(x.v[j] << 16);
    f[2 * j + 1] = __uint_as_float(x.v[j] & 0xffff0000u);
  }
}

// E4M3 codes of a negated piece under `scale` (dd = (scale, scale), ny = -(1 / scale) twice; FAST: b200q_div_fast_ok(scale)).
template <bool FAST>
__device__ __forceinline__ uint4 piece_fp8(const U32x8& x, float scale, uint64_t dd, uint64_t ny) {
  float f[16];
  piece_values(x, f);
#pragma unroll
  for (int j = 0; j < 16; j += 2) {
    if constexpr (FAST) {
      const float2 q = unpack2(div2_by_shared_negated(pack2(f[j], f[j + 1]), dd, ny));
      f[j] = q.x, f[j + 1] = q.y;
    } else {
      f[j] = __fdiv_rn(-f[j], scale), f[j + 1] = __fdiv_rn(-f[j + 1], scale);
    }
  }
  uint4 c;
  uint32_t* o = &c.x;
#pragma unroll
  for (int j = 0; j < 4; ++j) o[j] = f32x2_to_e4m3x2(f[4 * j], f[4 * j + 1]) | (f32x2_to_e4m3x2(f[4 * j + 2], f[4 * j + 3]) << 16);
  return c;
}

// Place of the first scale word of a row.
__device__ __forceinline__ uint8_t* nvfp4_scale_row(const Nvfp4Out& nv, int64_t row) {
  return nv.sf + (row >> 7) * static_cast<int64_t>(nv.col_tiles) * 512 + (row & 31) * 16 + ((row >> 5) & 3) * 4;
}

// NVFP4 codes and scale word of negated piece p of a row; all 32 lanes, the warp's pieces in order (p % 4 == lane % 4): four
// lanes hold one scale word.
__device__ __forceinline__ void piece_nvfp4_store(const U32x8& x, int p, int pieces, const GlobalScale& gs, uint8_t* code_row, uint8_t* sf_row) {
  uint32_t sb = 0u;
  if (p < pieces) {
    float f[16];
    uint32_t c[2];
    piece_values(x, f);
    sb = quantize_negated<16>(f, piece_abs_max(x), gs, c);
    *reinterpret_cast<uint2*>(code_row + p * 8) = make_uint2(c[0], c[1]);
  }
  uint32_t word = sb << (8 * (p & 3));
  word |= __shfl_xor_sync(0xffffffffu, word, 1);
  word |= __shfl_xor_sync(0xffffffffu, word, 2);
  if ((p & 3) == 0 && p < pieces) *reinterpret_cast<uint32_t*>(sf_row + static_cast<uint32_t>(p >> 2) * 512u) = word;
}

// Form for many tokens with rows of up to 8192 elements (a multiple of 16, 32-byte aligned): WPR warps (1, 2, 4 for rows of
// up to 2048, 4096, 8192 elements) hold a row in registers, packed as bf16, four pieces of 16 elements per lane, and reduce
// it with shuffles and one barrier between those warps.  No CTA-wide barrier stands between loading, reducing and storing,
// so the rows of an SM stream independently.  What bounds it is issue slots beside HBM: hence bf16 pair additions for
// h + delta, fp32 pairs for the squares, the products and the quotients (about 10 instructions an element, half of what the
// scalar form takes).  The squares are added in the order of add_norm_quant_kernel, whose thread t sums groups t, t + 256, ... of 8 elements and
// whose 8 warps of 32 threads are added by a tree: lane l of a warp here plays threads 2l and 2l + 1 of two of them.
template <int ITEMS, int WPR, bool HAS_DELTA, bool NVF4>
__global__ void __launch_bounds__(kThreads, 2)
add_norm_quant_warp_kernel(const __nv_bfloat16* __restrict__ h, const __nv_bfloat16* __restrict__ delta,
                           const __nv_bfloat16* __restrict__ w, __nv_bfloat16* __restrict__ h_out, uint8_t* __restrict__ codes,
                           float* __restrict__ scales, int64_t rows, int64_t cols, float eps, const Nvfp4Out nv) {
  constexpr int kSlots = kThreads / 32 / WPR;     // rows per CTA
  constexpr int VP = 4 / WPR;                     // pairs of warps of the one-CTA form that this warp stands for
  constexpr int N = ITEMS * VP;                   // pieces of 16 elements per lane
  pdl_launch_dependents();
  pdl_wait();
  __shared__ float part[kSlots][8];
  __shared__ float part_max[kSlots][WPR];
  const int lane = threadIdx.x & 31, slot = (threadIdx.x >> 5) / WPR, sub = (threadIdx.x >> 5) % WPR;
  const int64_t row = static_cast<int64_t>(blockIdx.x) * kSlots + slot;
  const int pieces = static_cast<int>(cols >> 4);
  if (row >= rows) {                              // the warps of a row leave together
    if constexpr (NVF4) {
      if (sub == 0 && row < (rows + 127) / 128 * 128) {
        uint8_t* sf = nvfp4_scale_row(nv, row);
        for (uint32_t c = lane; c < nv.col_tiles; c += 32) *reinterpret_cast<uint32_t*>(sf + c * 512u) = 0u;
      }
    }
    return;
  }
  const auto piece_of = [&](int k) { return (sub * VP + k / ITEMS) * 32 + lane + (k % ITEMS) * (kThreads / 2); };
  const __nv_bfloat16* hr = h + row * cols;
  U32x8 x[N];
#pragma unroll
  for (int k = 0; k < N; ++k) {
    const int p = piece_of(k);
    if (p < pieces) x[k] = ld_nc_256(hr + p * 16);
    else x[k] = U32x8{};
  }
  if constexpr (HAS_DELTA) {
    const __nv_bfloat16* dr = delta + row * cols;
    U32x8 d[N];
#pragma unroll
    for (int k = 0; k < N; ++k)
      if (piece_of(k) < pieces) d[k] = ld_nc_256(dr + piece_of(k) * 16);
#pragma unroll
    for (int k = 0; k < N; ++k) {
      if (piece_of(k) < pieces) {
        piece_add(x[k], d[k]);
        st_256(h_out + row * cols + piece_of(k) * 16, x[k]);
      }
    }
  }
  // sums of squares of the even and the odd group of 8 (low and high half of a pair)
  float sums[8];
#pragma unroll
  for (int v = 0; v < VP; ++v) {
    uint64_t ss = 0ull;
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) ss = piece_squares(x[v * ITEMS + i], ss);
    float2 s = unpack2(ss);
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) {
      s.x += __shfl_xor_sync(0xffffffffu, s.x, o);
      s.y += __shfl_xor_sync(0xffffffffu, s.y, o);
    }
    sums[v] = s.x + s.y;                          // lanes 0-15: warp 2 (sub VP + v) of the one-CTA form, lanes 16-31: the next
  }
  if constexpr (WPR > 1) {
    if ((lane & 15) == 0) {
#pragma unroll
      for (int v = 0; v < VP; ++v) part[slot][(sub * VP + v) * 2 + (lane >> 4)] = sums[v];
    }
    asm volatile("bar.sync %0, %1;" ::"r"(1 + slot), "n"(32 * WPR) : "memory");
#pragma unroll
    for (int v = 0; v < 8; ++v) sums[v] = part[slot][v];
  } else {
    float t[4];
#pragma unroll
    for (int v = 0; v < 4; ++v) t[v] = sums[v];
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      sums[2 * v] = __shfl_sync(0xffffffffu, t[v], 0);
      sums[2 * v + 1] = __shfl_sync(0xffffffffu, t[v], 16);
    }
  }
  const float total = ((sums[0] + sums[4]) + (sums[2] + sums[6])) + ((sums[1] + sums[5]) + (sums[3] + sums[7]));
  const float inv = rsqrtf(total / static_cast<float>(cols) + eps);
  // the normalised values, negated for the divisions below (the signs cancel there; magnitudes are the same)
  const uint64_t ninv = pack2(-inv, -inv);
#pragma unroll
  for (int k = 0; k < N; ++k) {
    const int p = piece_of(k);
    if (p < pieces) {
      piece_norm_negated(x[k], ld_128(w + p * 16), ld_128(w + p * 16 + 8), ninv);
    }
  }
  if constexpr (NVF4) {
    const GlobalScale gs(ld_dependent(nv.amax));
    if (blockIdx.x == 0 && threadIdx.x == 0 && nv.gout != nullptr) *nv.gout = gs.g;
#pragma unroll
    for (int k = 0; k < N; ++k) piece_nvfp4_store(x[k], piece_of(k), pieces, gs, nv.codes + row * (cols >> 1), nvfp4_scale_row(nv, row));
    return;
  }
  float amax = 0.0f;
#pragma unroll
  for (int k = 0; k < N; ++k) amax = fmaxf(amax, piece_abs_max(x[k]));   // pieces beyond the row hold zeros
  amax = warp_max(amax);
  if constexpr (WPR > 1) {
    if (lane == 0) part_max[slot][sub] = amax;
    asm volatile("bar.sync %0, %1;" ::"r"(1 + slot), "n"(32 * WPR) : "memory");
#pragma unroll
    for (int v = 0; v < WPR; ++v) amax = fmaxf(amax, part_max[slot][v]);
  }
  const float scale = fp8_scale_from_amax(amax);
  if (lane == 0 && sub == 0) scales[row] = scale;
  const float y = b200q_rcp_rn(scale);
  const uint64_t dd = pack2(scale, scale), ny = pack2(-y, -y);
  auto emit = [&](auto fast_tag) {
#pragma unroll
    for (int k = 0; k < N; ++k) {
      const int p = piece_of(k);
      if (p < pieces) *reinterpret_cast<uint4*>(codes + row * cols + p * 16) = piece_fp8<decltype(fast_tag)::value>(x[k], scale, dd, ny);
    }
  };
  if (b200q_div_fast_ok(scale)) emit(std::true_type{});   // one branch per row, not one select per element
  else emit(std::false_type{});
}

// Form for few tokens (a decode step) with rows of 2048 to 16384 elements (a multiple of 16, 32-byte aligned): one CTA per
// row with one piece of 16 elements per thread, so that what a launch takes is one round trip to L2 (row, delta and norm
// weights at once) and two reductions over at most 32 warps.  A cluster of CTAs per row took longer for its barriers than
// it saved: with delta, FP8 / NVFP4, 64 x 8192 6.4 / 5.3 us there, 3.2 / 3.9 here; 8 x 4096 3.4 / 3.4, 2.1 / 2.3; 128 x 2048 4.2 /
// 4.0, 2.0 / 2.3.  The squares are added in another order than in the other forms (a piece per thread, then a tree).
template <bool HAS_DELTA, bool NVF4>
__global__ void __launch_bounds__(1024, 1)
add_norm_quant_row_kernel(const __nv_bfloat16* __restrict__ h, const __nv_bfloat16* __restrict__ delta,
                          const __nv_bfloat16* __restrict__ w, __nv_bfloat16* __restrict__ h_out, uint8_t* __restrict__ codes,
                          float* __restrict__ scales, int64_t rows, int64_t cols, float eps, const Nvfp4Out nv) {
  pdl_launch_dependents();
  pdl_wait();
  __shared__ float part[32], part_max[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const int64_t row = blockIdx.x;
  const int pieces = static_cast<int>(cols >> 4), p = threadIdx.x;
  if constexpr (NVF4) {
    if (row >= rows) {
      zero_scale_row(nv.sf, row, nv.col_tiles);
      return;
    }
  }
  const bool live = p < pieces;
  U32x8 x{};
  uint4 w0{}, w1{};
  if (live) {
    x = ld_nc_256(h + row * cols + p * 16);
    U32x8 d;
    if constexpr (HAS_DELTA) d = ld_nc_256(delta + row * cols + p * 16);
    w0 = ld_nc_128(w + p * 16), w1 = ld_nc_128(w + p * 16 + 8);
    if constexpr (HAS_DELTA) {
      piece_add(x, d);
      st_256(h_out + row * cols + p * 16, x);
    }
  }
  const float2 s2 = unpack2(piece_squares(x, 0ull));
  float ss = s2.x + s2.y;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
  if (lane == 0) part[warp] = ss;
  __syncthreads();
  float total = lane < warps ? part[lane] : 0.0f;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) total += __shfl_xor_sync(0xffffffffu, total, o);
  const float inv = rsqrtf(total / static_cast<float>(cols) + eps);
  if (live) piece_norm_negated(x, w0, w1, pack2(-inv, -inv));
  if constexpr (NVF4) {
    const GlobalScale gs(ld_dependent(nv.amax));
    if (blockIdx.x == 0 && threadIdx.x == 0 && nv.gout != nullptr) *nv.gout = gs.g;
    piece_nvfp4_store(x, p, pieces, gs, nv.codes + row * (cols >> 1), nvfp4_scale_row(nv, row));
    return;
  }
  const float mine = warp_max(fmaxf(0.0f, piece_abs_max(x)));
  if (lane == 0) part_max[warp] = mine;
  __syncthreads();
  const float scale = fp8_scale_from_amax(warp_max(lane < warps ? part_max[lane] : 0.0f));
  if (threadIdx.x == 0) scales[row] = scale;
  const float y = b200q_rcp_rn(scale);
  if (live)
    *reinterpret_cast<uint4*>(codes + row * cols + p * 16) =
        b200q_div_fast_ok(scale) ? piece_fp8<true>(x, scale, pack2(scale, scale), pack2(-y, -y)) : piece_fp8<false>(x, scale, 0ull, 0ull);
}

// act[t, j] = silu(gu[t, j]) * gu[t, F + j], gu is [T, 2F] (gate columns first)
__global__ void __launch_bounds__(kThreads)
silu_mul_kernel(const __nv_bfloat16* __restrict__ gu, __nv_bfloat16* __restrict__ act, int64_t rows, int64_t f) {
  pdl_launch_dependents();
  pdl_wait();
  const int64_t groups_per_row = f >> 3;
  const int64_t total = rows * groups_per_row;
  for (int64_t g = blockIdx.x * (int64_t)kThreads + threadIdx.x; g < total; g += (int64_t)gridDim.x * kThreads) {
    const int64_t row = g / groups_per_row, c = (g - row * groups_per_row) * 8;
    float a[8], b[8], o[8];
    Elem<__nv_bfloat16>::load8(gu + row * 2 * f + c, a);
    Elem<__nv_bfloat16>::load8(gu + row * 2 * f + f + c, b);
#pragma unroll
    for (int j = 0; j < 8; ++j) o[j] = silu_mul_f32(a[j], b[j]);
    Elem<__nv_bfloat16>::store8(act + row * f + c, o);
  }
}

// silu(gate) * up fused with the per-token FP8 quantize that feeds the down projection: the
// bf16 activation [T, F] is never written.  One CTA per token; the row stays in registers as
// packed bf16 (ITEMS groups of 8 per thread), rounded exactly as silu_mul_kernel stores it, so
// codes and scales equal those of the two separate kernels.
// PARTS > 1: a cluster of PARTS CTAs shares one token (few tokens, long rows: a decode step would
// otherwise run on a handful of SMs); each CTA takes a contiguous slice of the row and the slice
// maxima meet through distributed shared memory.
template <int ITEMS, int PARTS>
__global__ void __launch_bounds__(kThreads)
silu_mul_quant_kernel(const __nv_bfloat16* __restrict__ gu, uint8_t* __restrict__ codes, float* __restrict__ scales, int64_t f, bool late) {
  pdl_enter(late);
  __shared__ float red[kThreads / 32];
  __shared__ float part_max;
  const int64_t row = blockIdx.x / PARTS;
  const int part = PARTS > 1 ? static_cast<int>(blockIdx.x % PARTS) : 0;   // == rank in the cluster
  const int groups = static_cast<int>(f >> 3);
  const int per_part = (groups + PARTS - 1) / PARTS;
  const int g_begin = part * per_part, g_end = min(groups, g_begin + per_part);
  uint4 y[ITEMS];
  __nv_bfloat162 m2 = __floats2bfloat162_rn(0.0f, 0.0f);   // running max |.| of the packed results (exact in bf16)
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) {
    const int g = g_begin + threadIdx.x + i * kThreads;
    y[i] = make_uint4(0u, 0u, 0u, 0u);
    if (g < g_end) {
      float a[8], b[8];
      Elem<__nv_bfloat16>::load8(gu + row * 2 * f + (int64_t)g * 8, a);
      Elem<__nv_bfloat16>::load8(gu + row * 2 * f + f + (int64_t)g * 8, b);
      uint32_t* u = &y[i].x;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const __nv_bfloat162 h = __floats2bfloat162_rn(silu_mul_f32(a[2 * j], b[2 * j]), silu_mul_f32(a[2 * j + 1], b[2 * j + 1]));
        u[j] = *reinterpret_cast<const uint32_t*>(&h);
        m2 = __hmax2(m2, __habs2(h));
      }
    }
  }
  float amax = fmaxf(__low2float(m2), __high2float(m2));
  amax = warp_max(amax);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = amax;
  __syncthreads();
  amax = (threadIdx.x & 31) < kThreads / 32 ? red[threadIdx.x & 31] : 0.0f;
  amax = warp_max(amax);
  if constexpr (PARTS > 1) {
    if (threadIdx.x == 0) part_max = amax;
    cluster_barrier();
    float other = 0.0f;
    if ((threadIdx.x & 31) < PARTS) other = ld_cluster_f32(&part_max, threadIdx.x & 31);
    amax = warp_max(other);
    cluster_barrier();  // nobody leaves (or rewrites part_max) while a peer may still read it
  }
  const float scale = fp8_scale_from_amax(amax);
  if (threadIdx.x == 0 && part == 0) scales[row] = scale;
  const float rcp = b200q_rcp_rn(scale);
  auto emit = [&](auto fast_tag) {
    constexpr bool kFast = decltype(fast_tag)::value;
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
      const int g = g_begin + threadIdx.x + i * kThreads;
      if (g < g_end) {
        float v[8], q[8];
        Elem<__nv_bfloat16>::unpack(y[i], v);
#pragma unroll
        for (int j = 0; j < 8; ++j) q[j] = kFast ? b200q_div_by_shared(v[j], scale, rcp) : __fdiv_rn(v[j], scale);
        const uint32_t lo = f32x2_to_e4m3x2(q[0], q[1]) | (f32x2_to_e4m3x2(q[2], q[3]) << 16);
        const uint32_t hi = f32x2_to_e4m3x2(q[4], q[5]) | (f32x2_to_e4m3x2(q[6], q[7]) << 16);
        *reinterpret_cast<uint2*>(codes + row * f + (int64_t)g * 8) = make_uint2(lo, hi);
      }
    }
  };
  // one branch per row, not one select per element: the true division is an order of magnitude longer
  if (b200q_div_fast_ok(scale)) emit(std::true_type{});
  else emit(std::false_type{});
}

// Many-token form of silu_mul_quant_kernel: persistent CTAs (two per SM), one row per iteration, the
// gate and up halves of the row arriving in chunks of 2 * kThreads groups (8 KB each) through a ring of
// shared-memory stages that one thread keeps filled with bulk asynchronous copies, across rows.  The
// row's results wait in registers, packed as bf16, for the row maximum.  Same expression, rounding
// points and thread-to-element mapping per chunk as the per-row kernels: same codes and scales.
constexpr int kSiluChunkGroups = 2 * kThreads;                // groups of 8 elements per chunk and half
constexpr int kSiluChunkBytes = kSiluChunkGroups * 16;        // per half
constexpr int kSiluStages = 6;                                // 6 x 16 KB

// GATED = false: the same machine as a plain per-token FP8 quantize of bf16 rows [rows, f] (one source, chunks of
// 8 KB): rows too long to stay in registers with one CTA per row would otherwise be read twice.
template <int CHUNKS, bool GATED>
__global__ void __launch_bounds__(kThreads, 2)
silu_mul_quant_stream_kernel(const __nv_bfloat16* __restrict__ gu, uint8_t* __restrict__ codes, float* __restrict__ scales, int rows,
                             int f, int* __restrict__ status, bool late) {
  constexpr int kStageBytes = (GATED ? 2 : 1) * kSiluChunkBytes;
  pdl_enter(late);
  extern __shared__ __align__(128) unsigned char ring[];
  __shared__ uint64_t full[kSiluStages];
  __shared__ float red[kThreads / 32];
  const int groups = f >> 3;
  const int nch = (groups + kSiluChunkGroups - 1) / kSiluChunkGroups;    // chunks per row (<= CHUNKS)
  const int step = static_cast<int>(gridDim.x);
  const int my_rows = (rows - static_cast<int>(blockIdx.x) + step - 1) / step;
  const int total = my_rows * nch;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kSiluStages; ++s) ptx::mbar_init(&full[s], 1);
    ptx::fence_barrier_init();
  }
  __syncthreads();
  // copy number q of this CTA: chunk q % nch of its row number q / nch; gate half first, up half behind it
  auto issue = [&](int q) {
    const int64_t row = static_cast<int64_t>(blockIdx.x) + static_cast<int64_t>(q / nch) * step;
    const int c = q % nch;
    const int g0 = c * kSiluChunkGroups;
    const uint32_t bytes = static_cast<uint32_t>(min(kSiluChunkGroups, groups - g0)) * 16u;
    const __nv_bfloat16* gate = gu + row * (GATED ? 2 : 1) * f + static_cast<int64_t>(g0) * 8;
    const int s = q % kSiluStages;
    unsigned char* dst = ring + static_cast<size_t>(s) * kStageBytes;
    ptx::mbar_arrive_expect_tx(&full[s], (GATED ? 2u : 1u) * bytes);
    ptx::bulk_load(dst, gate, bytes, &full[s]);
    if constexpr (GATED) ptx::bulk_load(dst + kSiluChunkBytes, gate + f, bytes, &full[s]);
  };
  if (threadIdx.x == 0)
    for (int q = 0; q < kSiluStages && q < total; ++q) issue(q);
  bool arrived = true;   // after one wait gave up the rest are not waited for: the status word says the result is void
  int q = 0;
  for (int64_t row = blockIdx.x; row < rows; row += step) {
    uint4 y[CHUNKS][2];
    __nv_bfloat162 m2 = __floats2bfloat162_rn(0.0f, 0.0f);
#pragma unroll
    for (int c = 0; c < CHUNKS; ++c) {
      if (c < nch) {
        const int s = q % kSiluStages;
        if (arrived && !ptx::mbar_wait(&full[s], static_cast<uint32_t>(q / kSiluStages) & 1u)) {
          arrived = false;
          atomicCAS(status, 0, 82);
        }
        const unsigned char* st = ring + static_cast<size_t>(s) * kStageBytes;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int gl = threadIdx.x + i * kThreads;              // group inside the chunk
          y[c][i] = make_uint4(0u, 0u, 0u, 0u);
          if (c * kSiluChunkGroups + gl < groups) {
            if constexpr (!GATED) {
              y[c][i] = *reinterpret_cast<const uint4*>(st + static_cast<size_t>(gl) * 16);
              const uint32_t* u = &y[c][i].x;
#pragma unroll
              for (int j = 0; j < 4; ++j) m2 = __hmax2(m2, __habs2(*reinterpret_cast<const __nv_bfloat162*>(&u[j])));
              continue;
            }
            float a[8], b[8];
            Elem<__nv_bfloat16>::unpack(*reinterpret_cast<const uint4*>(st + static_cast<size_t>(gl) * 16), a);
            Elem<__nv_bfloat16>::unpack(*reinterpret_cast<const uint4*>(st + kSiluChunkBytes + static_cast<size_t>(gl) * 16), b);
            uint32_t* u = &y[c][i].x;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const __nv_bfloat162 hh = __floats2bfloat162_rn(silu_mul_f32(a[2 * j], b[2 * j]), silu_mul_f32(a[2 * j + 1], b[2 * j + 1]));
              u[j] = *reinterpret_cast<const uint32_t*>(&hh);
              m2 = __hmax2(m2, __habs2(hh));
            }
          }
        }
        __syncthreads();                                           // the whole CTA has taken its part of the stage
        if (threadIdx.x == 0 && q + kSiluStages < total) issue(q + kSiluStages);
        ++q;
      }
    }
    float amax = fmaxf(__low2float(m2), __high2float(m2));
    amax = warp_max(amax);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = amax;
    __syncthreads();
    amax = (threadIdx.x & 31) < kThreads / 32 ? red[threadIdx.x & 31] : 0.0f;
    amax = warp_max(amax);
    const float scale = fp8_scale_from_amax(amax);
    if (threadIdx.x == 0) scales[row] = scale;
    const float rcp = b200q_rcp_rn(scale);
    auto emit = [&](auto fast_tag) {
      constexpr bool kFast = decltype(fast_tag)::value;
#pragma unroll
      for (int c = 0; c < CHUNKS; ++c) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int g = c * kSiluChunkGroups + threadIdx.x + i * kThreads;
          if (c < nch && g < groups) {
            float v[8], qv[8];
            Elem<__nv_bfloat16>::unpack(y[c][i], v);
#pragma unroll
            for (int j = 0; j < 8; ++j) qv[j] = kFast ? b200q_div_by_shared(v[j], scale, rcp) : __fdiv_rn(v[j], scale);
            const uint32_t lo = f32x2_to_e4m3x2(qv[0], qv[1]) | (f32x2_to_e4m3x2(qv[2], qv[3]) << 16);
            const uint32_t hi = f32x2_to_e4m3x2(qv[4], qv[5]) | (f32x2_to_e4m3x2(qv[6], qv[7]) << 16);
            *reinterpret_cast<uint2*>(codes + row * f + static_cast<int64_t>(g) * 8) = make_uint2(lo, hi);
          }
        }
      }
    };
    if (b200q_div_fast_ok(scale)) emit(std::true_type{});
    else emit(std::false_type{});
    // `red` is written again only after the next row's chunk barriers
  }
}

// out = a + b (bf16, fp32 add)
__global__ void __launch_bounds__(kThreads)
add_kernel(const __nv_bfloat16* __restrict__ a, const __nv_bfloat16* __restrict__ b, __nv_bfloat16* __restrict__ out, int64_t n) {
  pdl_launch_dependents();
  pdl_wait();
  const int64_t groups = n >> 3;
  for (int64_t g = blockIdx.x * (int64_t)kThreads + threadIdx.x; g < groups; g += (int64_t)gridDim.x * kThreads) {
    float x[8], y[8];
    Elem<__nv_bfloat16>::load8(a + g * 8, x);
    Elem<__nv_bfloat16>::load8(b + g * 8, y);
#pragma unroll
    for (int j = 0; j < 8; ++j) x[j] += y[j];
    Elem<__nv_bfloat16>::store8(out + g * 8, x);
  }
}

// out[t, h * hd + d] = src[t, src_col0 + (h / rep) * hd + d]: every kv head repeated `rep` times
__global__ void __launch_bounds__(kThreads)
expand_heads_kernel(const __nv_bfloat16* __restrict__ src, int64_t src_stride, int64_t src_col0, __nv_bfloat16* __restrict__ out,
                    int64_t rows, int heads_out, int rep, int head_dim) {
  pdl_launch_dependents();
  pdl_wait();
  const int64_t groups_per_head = head_dim >> 3;
  const int64_t groups_per_row = heads_out * groups_per_head;
  const int64_t total = rows * groups_per_row;
  for (int64_t g = blockIdx.x * (int64_t)kThreads + threadIdx.x; g < total; g += (int64_t)gridDim.x * kThreads) {
    const int64_t row = g / groups_per_row, r = g - row * groups_per_row;
    const int64_t h = r / groups_per_head, d = (r - h * groups_per_head) * 8;
    const uint4 v = *reinterpret_cast<const uint4*>(src + row * src_stride + src_col0 + (h / rep) * head_dim + d);
    *reinterpret_cast<uint4*>(out + row * groups_per_row * 8 + h * head_dim + d) = v;
  }
}

// expand_heads followed by the per-token FP8 quantize, in one pass over the kv slice: a repeated head does
// not change the token's abs-max, so the token is quantized once (one warp per token, its slice in
// registers) and every code group is stored `rep` times.  The same codes and scales as
// b200q_expand_heads + b200q_fp8_quantize with dynamic per-row amax; the expanded bf16 tensor is never written.
template <int ITEMS>
__global__ void __launch_bounds__(kThreads)
expand_heads_quant_kernel(const __nv_bfloat16* __restrict__ src, int64_t src_stride, int64_t src_col0, uint8_t* __restrict__ codes,
                          float* __restrict__ scales, int64_t rows, int heads_out, int rep, int head_dim) {
  pdl_launch_dependents();
  pdl_wait();
  const int lane = threadIdx.x & 31;
  const int64_t row = blockIdx.x * (int64_t)(kThreads / 32) + (threadIdx.x >> 5);
  if (row >= rows) return;
  const int kv_heads = heads_out / rep;
  const int groups = (kv_heads * head_dim) >> 3;            // groups of 8 elements in the token's kv slice
  const int64_t out_cols = static_cast<int64_t>(heads_out) * head_dim;
  float v[ITEMS][8];
  float amax = 0.0f;
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) {
    const int g = lane + i * 32;
    if (g < groups) {
      Elem<__nv_bfloat16>::load8(src + row * src_stride + src_col0 + (int64_t)g * 8, v[i]);
#pragma unroll
      for (int j = 0; j < 8; ++j) amax = fmaxf(amax, fabsf(v[i][j]));
    }
  }
  amax = warp_max(amax);
  const float scale = fp8_scale_from_amax(amax);
  if (lane == 0) scales[row] = scale;
  const float y = b200q_rcp_rn(scale);
  const bool fast = b200q_div_fast_ok(scale);
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) {
    const int g = lane + i * 32;
    if (g < groups) {
      float q[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) q[j] = fast ? b200q_div_by_shared(v[i][j], scale, y) : __fdiv_rn(v[i][j], scale);
      const uint2 packed = make_uint2(f32x2_to_e4m3x2(q[0], q[1]) | (f32x2_to_e4m3x2(q[2], q[3]) << 16),
                                      f32x2_to_e4m3x2(q[4], q[5]) | (f32x2_to_e4m3x2(q[6], q[7]) << 16));
      const int e = g * 8, kvh = e / head_dim, d = e - kvh * head_dim;
      uint8_t* dst = codes + row * out_cols + static_cast<int64_t>(kvh) * rep * head_dim + d;
      for (int r = 0; r < rep; ++r) *reinterpret_cast<uint2*>(dst + static_cast<int64_t>(r) * head_dim) = packed;
    }
  }
}

int grid_for(int64_t work_items) {
  int64_t ctas = (work_items + kThreads - 1) / kThreads;
  const int64_t cap = (int64_t)sm_count() * 16;
  return static_cast<int>(ctas < 1 ? 1 : (ctas > cap ? cap : ctas));
}

// Whether the rows of add_norm_quant go to warps instead of CTAs.  Measured (us; CTA forms -> warps): 8192 x 4096 with delta
// 55.5 -> 47.8 FP8 and 60.0 -> 43.3 NVFP4, without 52.6 -> 25.6 and 57.4 -> 28.0; 1200 x 512 7.2 -> 2.7; 300 x 8192 7.8 -> 5.1.
// Not faster: few short rows (300 x 2048 2.9 -> 3.8, 600 x 4096 NVFP4 6.1 -> 6.2), where a CTA per row has more threads on the
// device, and many long rows with a delta in FP8 (8192 x 8192 78.7 -> 81.1), which the ring-fed form streams.
bool warp_rows(int64_t rows, int64_t cols, bool has_delta, bool nvf4) {
  if (cols > 8192) return false;
  const bool many = rows >= 8 * sm_count();
  if (cols > 4096 && has_delta && !nvf4 && many) return false;
  return many || rows * cols >= (cols > 4096 || !nvf4 ? int64_t{1} << 21 : int64_t{3} << 20);
}

// Launch of the add + RMSNorm + quantize kernels (checked arguments).  NVF4: result into `nv`, else per-token FP8.
template <bool NVF4>
int launch_add_norm_quant(const void* h, const void* delta, const void* weight, void* h_out, uint8_t* codes_out, float* scales_out,
                          int64_t rows, int64_t cols, float eps, const Nvfp4Out& nv, cudaStream_t st) {
  const auto* hp = static_cast<const __nv_bfloat16*>(h);
  const auto* dp = static_cast<const __nv_bfloat16*>(delta);
  const auto* wp = static_cast<const __nv_bfloat16*>(weight);
  auto* op = static_cast<__nv_bfloat16*>(h_out);
  const int64_t groups = cols >> 3;
  int parts = 1;   // few tokens: split every row over a cluster so that the launch covers more SMs
  while (parts < 8 && rows * parts < 2 * sm_count() && groups / (parts * 2) >= kThreads / 2) parts *= 2;
  int64_t per_part = (groups + parts - 1) / parts;
  if (NVF4) per_part = (per_part + 7) / 8 * 8;
  const int items = static_cast<int>((per_part + kThreads - 1) / kThreads);
  const int64_t grid_rows = NVF4 ? (rows + 127) / 128 * 128 : rows;
  const bool by_pieces = cols % 16 == 0 && aligned(h, 32) && aligned(delta, 32) && (delta == nullptr || aligned(h_out, 32)) &&
                         (NVF4 ? aligned(nv.codes, 8) : aligned(codes_out, 16));
  // (a CTA of 1024 threads starts later than a cluster where there are hardly any rows: 8 x 16384 NVFP4 4.2 us, 4.0)
  if (by_pieces && parts > 1 && (cols <= 8192 || rows > 16)) {
    const dim3 grid(static_cast<unsigned>(grid_rows)), block(static_cast<unsigned>((cols / 16 + 31) / 32 * 32));
    if (delta != nullptr) launch_pdl(add_norm_quant_row_kernel<true, NVF4>, grid, block, 0, st, hp, dp, wp, op, codes_out, scales_out, rows, cols, eps, nv);
    else launch_pdl(add_norm_quant_row_kernel<false, NVF4>, grid, block, 0, st, hp, dp, wp, op, codes_out, scales_out, rows, cols, eps, nv);
    return check_launch();
  }
  if (by_pieces && parts == 1 && warp_rows(rows, cols, delta != nullptr, NVF4)) {
    const int per_cta = items <= 1 ? 8 : (items <= 2 ? 4 : 2);
    const dim3 grid(static_cast<unsigned>((grid_rows + per_cta - 1) / per_cta));
#define B200Q_ANQW(I, W)                                                                                                                   \
  do {                                                                                                                                     \
    if (delta != nullptr) launch_pdl(add_norm_quant_warp_kernel<I, W, true, NVF4>, grid, dim3(kThreads), 0, st, hp, dp, wp, op, codes_out, \
                                     scales_out, rows, cols, eps, nv);                                                                     \
    else launch_pdl(add_norm_quant_warp_kernel<I, W, false, NVF4>, grid, dim3(kThreads), 0, st, hp, dp, wp, op, codes_out, scales_out,     \
                    rows, cols, eps, nv);                                                                                                  \
  } while (0)
    if (items <= 1) B200Q_ANQW(1, 1);
    else if (items <= 2) B200Q_ANQW(2, 2);
    else B200Q_ANQW(4, 4);
#undef B200Q_ANQW
    return check_launch();
  }
  // many tokens that the warps do not take: persistent CTAs fed through a shared-memory ring of rows
  const int64_t stage_bytes = cols * 2 * (delta != nullptr ? 2 : 1);
  if (parts == 1 && items <= 4 && rows >= 8 * sm_count() && kStreamRingBytes / stage_bytes >= 2) {
    int stages = static_cast<int>(kStreamRingBytes / stage_bytes);
    if (stages > kStreamStagesMax) stages = kStreamStagesMax;
    int* status = gemm::device_status_word();
    if (status == nullptr) return B200Q_ERR_CUDA;
    const size_t smem = static_cast<size_t>(stages) * static_cast<size_t>(stage_bytes);
    const dim3 grid(static_cast<unsigned>(2 * sm_count()));
    const int r32 = static_cast<int>(rows), c32 = static_cast<int>(cols);
#define B200Q_ANQS(I, D)                                                                                                     \
  do {                                                                                                                        \
    cudaFuncSetAttribute(add_norm_quant_stream_kernel<I, D, NVF4>, cudaFuncAttributeMaxDynamicSharedMemorySize, kStreamRingBytes); \
    launch_pdl(add_norm_quant_stream_kernel<I, D, NVF4>, grid, dim3(kThreads), smem, st, hp, dp, wp, op, codes_out, scales_out,     \
               r32, c32, eps, stages, status, nv);                                                                                \
  } while (0)
    if (delta != nullptr) {
      if (items <= 1) B200Q_ANQS(1, true);
      else if (items <= 2) B200Q_ANQS(2, true);
      else B200Q_ANQS(4, true);
    } else {
      if (items <= 1) B200Q_ANQS(1, false);
      else if (items <= 2) B200Q_ANQS(2, false);
      else B200Q_ANQS(4, false);
    }
#undef B200Q_ANQS
    return check_launch();
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(grid_rows * parts));
  cfg.blockDim = dim3(kThreads);
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = static_cast<unsigned>(parts);
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_enabled() ? 2 : 1;
#define B200Q_ANQ(I, P) cudaLaunchKernelEx(&cfg, add_norm_quant_kernel<I, P, NVF4>, hp, dp, wp, op, codes_out, scales_out, rows, cols, eps, nv)
  if (parts == 1) {
    if (items <= 1) B200Q_ANQ(1, 1);
    else if (items <= 2) B200Q_ANQ(2, 1);
    else if (items <= 4) B200Q_ANQ(4, 1);
    else B200Q_ANQ(8, 1);
  } else if (parts == 2) {
    if (items <= 1) B200Q_ANQ(1, 2);
    else if (items <= 2) B200Q_ANQ(2, 2);
    else B200Q_ANQ(4, 2);
  } else if (parts == 4) {
    if (items <= 1) B200Q_ANQ(1, 4);
    else B200Q_ANQ(2, 4);
  } else {
    B200Q_ANQ(1, 8);
  }
#undef B200Q_ANQ
  return check_launch();
}

int check_add_norm(const void* h, const void* delta, const void* weight, const void* h_out) {
  if (h == nullptr || weight == nullptr) return B200Q_ERR_INVALID;
  if (delta != nullptr && h_out == nullptr) return B200Q_ERR_INVALID;
  if (!aligned(h, 16) || !aligned(weight, 16) || (delta != nullptr && (!aligned(delta, 16) || !aligned(h_out, 16)))) return B200Q_ERR_ALIGN;
  return B200Q_OK;
}

}  // namespace

// Dynamic per-token FP8 quantize of many long bf16 rows through the ring-fed persistent kernel
// (silu_mul_quant_stream_kernel<.., false>).  Returns 1 when the shape does not qualify (the caller
// then takes its one-CTA-per-row kernels), else the launch status.
int launch_fp8_rows_stream(const __nv_bfloat16* x, uint8_t* codes, float* scales, int64_t rows, int64_t cols, cudaStream_t st, bool late) {
  static const bool enabled = [] {
    const char* e = std::getenv("B200Q_ROWS_STREAM");   // 0 = always one CTA per row (A/B measurements)
    return e == nullptr || e[0] != '0';
  }();
  if (!enabled) return 1;
  const int64_t groups = cols >> 3;
  // rows of up to 16384 elements stay in registers with one CTA per row, which is faster (0.82-0.91 of HBM against
  // 0.54-0.72 here); beyond that the one-CTA form reads the row twice and this one wins (0.81)
  if (cols % 8 != 0 || rows < 8 * sm_count() || rows > 0x7fffffffLL || cols <= 16384 || groups > 8 * kSiluChunkGroups) return 1;
  if (!aligned(x, 16) || !aligned(codes, 8)) return 1;
  int* status = gemm::device_status_word();
  if (status == nullptr) return B200Q_ERR_CUDA;
  const int nch = static_cast<int>((groups + kSiluChunkGroups - 1) / kSiluChunkGroups);
  const size_t smem = static_cast<size_t>(kSiluStages) * kSiluChunkBytes;
  const dim3 grid(static_cast<unsigned>(2 * sm_count()));
  const int r32 = static_cast<int>(rows), f32 = static_cast<int>(cols);
#define B200Q_ROWS_STREAM(C)                                                                                                 \
  do {                                                                                                                        \
    cudaFuncSetAttribute(silu_mul_quant_stream_kernel<C, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)); \
    launch_pdl(silu_mul_quant_stream_kernel<C, false>, grid, dim3(kThreads), smem, st, x, codes, scales, r32, f32, status, late);     \
  } while (0)
  if (nch <= 2) B200Q_ROWS_STREAM(2);
  else if (nch <= 4) B200Q_ROWS_STREAM(4);
  else B200Q_ROWS_STREAM(8);
#undef B200Q_ROWS_STREAM
  return check_launch();
}

int silu_mul_fp8_quantize(const void* gate_up, uint8_t* codes_out, float* scales_out, int64_t rows, int64_t f,
                                b200q_stream_t stream, bool late) {
  if (rows < 0 || f < 0 || f % 8 != 0 || rows > 0x7fffffffLL || f > kThreads * 8 * 16) return B200Q_ERR_INVALID;
  if (rows == 0 || f == 0) return B200Q_OK;
  if (gate_up == nullptr || codes_out == nullptr || scales_out == nullptr) return B200Q_ERR_INVALID;
  if (!aligned(gate_up, 16) || !aligned(codes_out, 8)) return B200Q_ERR_ALIGN;
  if (int rc = check_arch()) return rc;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const auto* gp = static_cast<const __nv_bfloat16*>(gate_up);
  const int64_t groups = f >> 3;
  // many tokens, rows of at least one chunk: persistent CTAs fed through a shared-memory ring
  if (rows >= 8 * sm_count() && groups >= kSiluChunkGroups) {
    int* status = gemm::device_status_word();
    if (status == nullptr) return B200Q_ERR_CUDA;
    const int nch = static_cast<int>((groups + kSiluChunkGroups - 1) / kSiluChunkGroups);
    const size_t smem = static_cast<size_t>(kSiluStages) * 2 * kSiluChunkBytes;
    const dim3 grid(static_cast<unsigned>(2 * sm_count()));
    const int r32 = static_cast<int>(rows), f32 = static_cast<int>(f);
#define B200Q_SILUS(C)                                                                                              \
  do {                                                                                                               \
    cudaFuncSetAttribute(silu_mul_quant_stream_kernel<C, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)); \
    launch_pdl(silu_mul_quant_stream_kernel<C, true>, grid, dim3(kThreads), smem, st, gp, codes_out, scales_out, r32, f32, status, late); \
  } while (0)
    if (nch <= 2) B200Q_SILUS(2);
    else if (nch <= 4) B200Q_SILUS(4);
    else B200Q_SILUS(8);
#undef B200Q_SILUS
    return check_launch();
  }
  // few tokens: split every row over a cluster so that the launch covers the SMs
  int parts = 1;
  while (parts < 8 && rows * parts < 2 * sm_count() && groups / (parts * 2) >= kThreads / 2) parts *= 2;
  // long rows: 16 groups per thread cost 92 registers (two CTAs per SM) and the kernel turns
  // compute-bound on the exponentials; two CTAs per row at 8 groups per thread double the warps per SM
  if (parts == 1 && groups > 8 * kThreads) parts = 2;
  const int items = static_cast<int>(((groups + parts - 1) / parts + kThreads - 1) / kThreads);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(rows * parts));
  cfg.blockDim = dim3(kThreads);
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = static_cast<unsigned>(parts);
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_enabled() ? 2 : 1;
#define B200Q_SILU(I, P) cudaLaunchKernelEx(&cfg, silu_mul_quant_kernel<I, P>, gp, codes_out, scales_out, f, late)
  if (parts == 1) {
    if (items <= 1) B200Q_SILU(1, 1);
    else if (items <= 2) B200Q_SILU(2, 1);
    else if (items <= 4) B200Q_SILU(4, 1);
    else if (items <= 8) B200Q_SILU(8, 1);
    else B200Q_SILU(16, 1);
  } else if (parts == 2) {
    if (items <= 1) B200Q_SILU(1, 2);
    else if (items <= 2) B200Q_SILU(2, 2);
    else if (items <= 4) B200Q_SILU(4, 2);
    else B200Q_SILU(8, 2);
  } else if (parts == 4) {
    if (items <= 1) B200Q_SILU(1, 4);
    else if (items <= 2) B200Q_SILU(2, 4);
    else B200Q_SILU(4, 4);
  } else {
    if (items <= 1) B200Q_SILU(1, 8);
    else B200Q_SILU(2, 8);
  }
#undef B200Q_SILU
  return check_launch();
}

}  // namespace b200q

using namespace b200q;

extern "C" {

int b200q_rms_norm(const void* x, const void* weight, void* out, int64_t rows, int64_t cols, float eps, b200q_stream_t stream) {
  if (rows < 0 || cols < 0 || cols % 8 != 0 || rows > 0x7fffffffLL) return B200Q_ERR_INVALID;
  if (rows == 0 || cols == 0) return B200Q_OK;
  if (x == nullptr || weight == nullptr || out == nullptr) return B200Q_ERR_INVALID;
  if (!aligned(x, 16) || !aligned(weight, 16) || !aligned(out, 16)) return B200Q_ERR_ALIGN;
  if (int rc = check_arch()) return rc;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const auto* xp = static_cast<const __nv_bfloat16*>(x);
  const auto* wp = static_cast<const __nv_bfloat16*>(weight);
  auto* yp = static_cast<__nv_bfloat16*>(out);
  const int items = static_cast<int>(((cols >> 3) + kThreads - 1) / kThreads);
  dim3 grid(static_cast<unsigned>(rows));
  if (items <= 1) launch_pdl(rms_norm_kernel<1>, dim3(grid), dim3(kThreads), 0, st, xp, wp, yp, cols, eps);
  else if (items <= 2) launch_pdl(rms_norm_kernel<2>, dim3(grid), dim3(kThreads), 0, st, xp, wp, yp, cols, eps);
  else if (items <= 4) launch_pdl(rms_norm_kernel<4>, dim3(grid), dim3(kThreads), 0, st, xp, wp, yp, cols, eps);
  else launch_pdl(rms_norm_kernel<0>, dim3(grid), dim3(kThreads), 0, st, xp, wp, yp, cols, eps);
  return check_launch();
}

int b200q_add_rms_norm_fp8_quantize(const void* h, const void* delta, const void* weight, void* h_out, uint8_t* codes_out,
                                    float* scales_out, int64_t rows, int64_t cols, float eps, b200q_stream_t stream) {
  if (rows < 0 || cols < 0 || cols % 16 != 0 || rows > 0x7fffffffLL || cols > kThreads * 8 * 8) return B200Q_ERR_INVALID;
  if (rows == 0 || cols == 0) return B200Q_OK;
  if (codes_out == nullptr || scales_out == nullptr) return B200Q_ERR_INVALID;
  if (int rc = check_add_norm(h, delta, weight, h_out)) return rc;
  if (!aligned(codes_out, 8)) return B200Q_ERR_ALIGN;
  if (int rc = check_arch()) return rc;
  return launch_add_norm_quant<false>(h, delta, weight, h_out, codes_out, scales_out, rows, cols, eps, Nvfp4Out{}, static_cast<cudaStream_t>(stream));
}

int b200q_add_rms_norm_nvfp4_quantize(const void* h, const void* delta, const void* weight, void* h_out, const float* amax,
                                      uint8_t* codes_out, uint8_t* scales_out, float* global_scale_out, int64_t rows, int64_t cols,
                                      float eps, b200q_stream_t stream) {
  if (rows < 0 || cols < 0 || cols % 16 != 0 || rows > 0x7fffff80LL || cols > kThreads * 8 * 8) return B200Q_ERR_INVALID;
  if (rows == 0 || cols == 0) return B200Q_OK;
  if (amax == nullptr || codes_out == nullptr || scales_out == nullptr) return B200Q_ERR_INVALID;
  if (int rc = check_add_norm(h, delta, weight, h_out)) return rc;
  if (!aligned(codes_out, 8) || !aligned(scales_out, 16)) return B200Q_ERR_ALIGN;
  if (int rc = check_arch()) return rc;
  const Nvfp4Out nv{amax, codes_out, scales_out, global_scale_out, static_cast<uint32_t>((cols / 16 + 3) / 4)};
  return launch_add_norm_quant<true>(h, delta, weight, h_out, nullptr, nullptr, rows, cols, eps, nv, static_cast<cudaStream_t>(stream));
}

int b200q_silu_mul(const void* gate_up, void* out, int64_t rows, int64_t f, b200q_stream_t stream) {
  if (rows < 0 || f < 0 || f % 8 != 0) return B200Q_ERR_INVALID;
  if (rows == 0 || f == 0) return B200Q_OK;
  if (gate_up == nullptr || out == nullptr) return B200Q_ERR_INVALID;
  if (!aligned(gate_up, 16) || !aligned(out, 16)) return B200Q_ERR_ALIGN;
  if (int rc = check_arch()) return rc;
  launch_pdl(silu_mul_kernel, dim3(grid_for(rows * (f >> 3))), dim3(kThreads), 0, static_cast<cudaStream_t>(stream),
             static_cast<const __nv_bfloat16*>(gate_up), static_cast<__nv_bfloat16*>(out), rows, f);
  return check_launch();
}

int b200q_silu_mul_fp8_quantize(const void* gate_up, uint8_t* codes_out, float* scales_out, int64_t rows, int64_t f,
                                b200q_stream_t stream) {
  return silu_mul_fp8_quantize(gate_up, codes_out, scales_out, rows, f, stream, false);
}

int b200q_add(const void* a, const void* b, void* out, int64_t n, b200q_stream_t stream) {
  if (n < 0 || n % 8 != 0) return B200Q_ERR_INVALID;
  if (n == 0) return B200Q_OK;
  if (a == nullptr || b == nullptr || out == nullptr) return B200Q_ERR_INVALID;
  if (!aligned(a, 16) || !aligned(b, 16) || !aligned(out, 16)) return B200Q_ERR_ALIGN;
  if (int rc = check_arch()) return rc;
  launch_pdl(add_kernel, dim3(grid_for(n >> 3)), dim3(kThreads), 0, static_cast<cudaStream_t>(stream),
             static_cast<const __nv_bfloat16*>(a), static_cast<const __nv_bfloat16*>(b), static_cast<__nv_bfloat16*>(out), n);
  return check_launch();
}

int b200q_expand_heads(const void* src, int64_t src_stride, int64_t src_col0, void* out, int64_t rows, int heads_out, int rep,
                       int head_dim, b200q_stream_t stream) {
  if (rows < 0 || heads_out <= 0 || rep <= 0 || head_dim <= 0 || head_dim % 8 != 0 || heads_out % rep != 0 || src_stride % 8 != 0 ||
      src_col0 % 8 != 0)
    return B200Q_ERR_INVALID;
  if (rows == 0) return B200Q_OK;
  if (src == nullptr || out == nullptr) return B200Q_ERR_INVALID;
  if (!aligned(src, 16) || !aligned(out, 16)) return B200Q_ERR_ALIGN;
  if (int rc = check_arch()) return rc;
  launch_pdl(expand_heads_kernel, dim3(grid_for(rows * heads_out * (head_dim >> 3))), dim3(kThreads), 0, static_cast<cudaStream_t>(stream),
             static_cast<const __nv_bfloat16*>(src), src_stride, src_col0, static_cast<__nv_bfloat16*>(out), rows, heads_out, rep, head_dim);
  return check_launch();
}

int b200q_expand_heads_fp8_quantize(const void* src, int64_t src_stride, int64_t src_col0, uint8_t* codes_out, float* scales_out,
                                    int64_t rows, int heads_out, int rep, int head_dim, b200q_stream_t stream) {
  if (rows < 0 || heads_out <= 0 || rep <= 0 || head_dim <= 0 || head_dim % 8 != 0 || heads_out % rep != 0 || src_stride % 8 != 0 ||
      src_col0 % 8 != 0 || rows > 0x7fffffffLL)
    return B200Q_ERR_INVALID;
  const int64_t kv_width = static_cast<int64_t>(heads_out / rep) * head_dim;
  if (kv_width > 32 * 8 * 8) return B200Q_ERR_INVALID;       // the slice of a token stays in one warp's registers
  if (rows == 0) return B200Q_OK;
  if (src == nullptr || codes_out == nullptr || scales_out == nullptr) return B200Q_ERR_INVALID;
  if (!aligned(src, 16) || !aligned(codes_out, 8)) return B200Q_ERR_ALIGN;
  if (int rc = check_arch()) return rc;
  const int items = static_cast<int>(((kv_width >> 3) + 31) / 32);
  const dim3 grid(static_cast<unsigned>((rows + kThreads / 32 - 1) / (kThreads / 32)));
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const auto* sp = static_cast<const __nv_bfloat16*>(src);
#define B200Q_EHQ(I) launch_pdl(expand_heads_quant_kernel<I>, grid, dim3(kThreads), 0, st, sp, src_stride, src_col0, codes_out, scales_out, rows, heads_out, rep, head_dim)
  if (items <= 1) B200Q_EHQ(1);
  else if (items <= 2) B200Q_EHQ(2);
  else if (items <= 4) B200Q_EHQ(4);
  else B200Q_EHQ(8);
#undef B200Q_EHQ
  return check_launch();
}

}  // extern "C"
