// FP8 scaled-dot-product attention for Q, K, V that come out of `tensorrt::quantize_op(.., 8, 4, ..)`.
//
// The reference marks an SDPA whose three inputs are FP8 fake-quantized
// (py/torch_tensorrt/dynamo/lowering/passes/annotate_fp8_sdpa.py:34-76) and builds a TensorRT attention
// layer whose softmax output is quantized to FP8 with the data-independent scale 1/448, with a static
// 1/sqrt(D) factor on the query (py/torch_tensorrt/dynamo/conversion/impl/attention.py:272-283).  Here:
//
//   S = (Q_hat K_hat^T) * scale            Q_hat, K_hat, V_hat: E4M3 codes x per-tensor scale
//   P = softmax(S)  (optionally causal, lower-right aligned)
//   P_hat = e4m3(P * 448) / 448            exactly the normalized probabilities, quantized
//   O = P_hat V_hat
//
// Both contractions run on the tensor cores (tcgen05.mma kind::f8f6f4, accumulators in tensor memory).
// P_hat is the quantization of the NORMALIZED probabilities, so the row maximum and the row sum must be
// known before the first probability is quantized: the kernel makes two passes over the keys.  Pass 1
// computes Q K^T tile by tile and keeps the running maximum and sum per query row in registers; pass 2
// computes Q K^T again (the last key tile's exponentials are kept), turns every score into its final probability, quantizes it, writes the 128 x 128
// tile of codes to shared memory in the operand layout and multiplies it with the V tile.  The attention
// core is a few per cent of a decoder layer's arithmetic, so the repeated Q K^T is cheaper than a
// rescaling scheme whose quantization points would differ from the definition above.
//
// What bounds it: the chain of a key tile, and beside it (special-function pipe 62 % and issue slots 55 % of active cycles at
// [4, 32 / 8, 2048, 128] causal) the exponentials, two per score at 16 per clock and SM: 1024 clocks per 128 x 128 tile and pass, and
// two warps per scheduler and CTA reach 0.93 of that rate in a loop of their own.  An eighth of them runs on the FMA pipe instead
// (ex2_poly2, more exact than the unit).  What it loses beside them is warps that wait for scores: without any arithmetic in the
// softmax warps the kernel still takes 0.58 of its time, the chain of loads, MMAs and barriers of a tile.  Shared-memory addresses
// that are compile-time constants shorten that chain (203 -> 190 us at [4, 32 / 8, 2048, 128] causal); a second V stage or a third K
// stage lengthens it (193), scores in buffers of 64 keys too (223).  So a softmax thread takes its 64 scores of a tile into registers and hands the tensor-memory
// buffer back before it computes (the tensor core fills it under the exponentials); in pass 2 the scores of tile j + 2
// are issued in front of the product of tile j (wait for scores per tile 819 -> 171 clocks of about 2500); edge tiles
// have their own copy of the loop; query tiles with the most keys start first (head_group).  Order and roundings per row are those
// of a loop over 32-column pieces for fp16 and fp32 results; bf16 results see FREE.  [4, 32 / 8, 2048, 128] causal, the whole call in
// turn with others: 300 -> 246 us, 208 with the exponentials on both pipes, constant addresses, queries quantized here and the last
// tile raised once.
//
// One CTA per (batch, head, 128 queries): warp 0 = TMA producer, warp 1 = MMA issue + tensor-memory
// allocation, warps 2-9 = softmax (two threads per query row, each half of the columns; lane quarter = warp & 3).  K and Q tiles are
// [rows, D] with D bytes per row (K-major), V is supplied TRANSPOSED per head ([D, keys], produced by
// b200q_fp8_quantize_transpose) so that the second contraction is K-major too.  D <= 128 (a multiple of
// 16); rows are zero-filled to 128 bytes by the TMA loads.  No TMA multicast; every wait is bounded.
#include "common.cuh"
#include "tcgen05.cuh"

#include <cuda.h>

#include <type_traits>

namespace b200q {
namespace gemm {
int* device_status_word();
using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                   const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                   CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn encode_tiled();
}  // namespace gemm

namespace {

constexpr int kAttThreads = 320;          // producer warp, MMA warp, 8 softmax warps
constexpr int kTile = 128;                 // queries per CTA, keys per step, padded head dimension
constexpr int kTileBytes = kTile * 128;    // one operand tile: 128 rows x 128 bytes
// Two CTAs per SM: while one waits for its tensor-core results the other's softmax warps have the issue
// slots.  Per CTA that leaves 6 operand tiles of shared memory (Q, 2 K stages, 1 V stage, 2 P tiles) and
// 256 columns of tensor memory.  Columns 0-127 hold a score tile; columns 128-255 a second one in pass 1
// and the output accumulator in pass 2.
constexpr int kKStages = 2, kVStages = 1;
constexpr int kChunk = 32;                 // score columns of one step of a softmax thread
constexpr int kTmemCols = 256;
constexpr int kAttSmem = kTileBytes * (1 + kKStages + kVStages + 2) + 512;   // tail: barriers
constexpr int kAttSmemAlone = 114 * 1024;  // with the 1 KB that each CTA costs, more than half of an SM's 228 KB
static_assert(kAttSmemAlone >= kAttSmem, "");
// Of the 16 pairs of a chunk, those whose exponentials run on the FMA pipe (ex2_poly2), us of this kernel with 0 / 2 / 3 / 4 of them:
// [4, 32 / 8, 2048, 128] causal 190 / 180 / 181 / 185; [3, 16, 577 x 1500, 64] 41.8 / 40.0 / 39.5 / 40.5; [8, 32 / 8, 1024, 128] causal
// 119 / 115 / 117 / 118; [1, 74, 4096, 128] 740 / 703 / 700 / 732.  Beyond four the issue slots bind.
constexpr int kPolyPairs = 2;

struct AttParams {
  const float* q_scale;     // per-tensor scales (device scalars)
  const float* k_scale;
  const float* v_scale;
  const void* q;            // queries that the kernel quantizes itself: [B, Hq, Sq, D] at these strides (elements), under q_amax
  const float* q_amax;
  int64_t q_sb, q_sh, q_ss;
  void* out;                // [B, Hq, Sq, D] at these strides (elements, multiples of 8; D contiguous)
  int64_t out_sb, out_sh, out_ss;
  int out_dtype;
  int Hq, Hkv, Sq, Sk, D;
  int BH, q_tiles;          // B * Hq, tiles of 128 queries
  int group;                // heads whose query tiles are walked together
  float softmax_scale;
  int causal;
  int* status;
};

__device__ __forceinline__ void att_timeout(int* status, int where) { atomicCAS(status, 0, where); }

// 2^x on the special-function unit (about 2 ulp; -inf -> 0, subnormal results flushed)
__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// maximum that keeps a NaN
__device__ __forceinline__ float max_nan(float a, float b) {
  float r;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}

// 2^x of a pair on the FMA pipe, x < 128: x = n + f with n the nearest integer (Cody and Waite's reduction; the rounding constant
// 1.5 * 2^23 is raised by 127, so that the low bits of the sum are the biased exponent of 2^n), 2^f by the polynomial of degree 6
// with constant term 1 of the smallest largest relative error on [-1/2, 1/2] (2.0e-9, from a weighted least-squares exchange).  With
// the fp32 roundings of Horner's scheme: largest relative error 7.9e-8, root mean square 2.7e-8, mean 9e-10; ex2.approx over the same
// range [-20, 9]: 1.4e-7, 5.5e-8, -2.4e-8.  Below -126.5 the result is 0; NaN stays NaN.
__device__ __forceinline__ uint64_t ex2_poly2(uint64_t x) {
  constexpr float kRound = 12582912.0f + 127.0f;
  const auto both = [](float c) { return pack2(c, c); };
  const float2 a = unpack2(x);
  x = pack2(max_nan(a.x, -127.0f), max_nan(a.y, -127.0f));
  const uint64_t t = add2(x, both(kRound));
  const uint64_t f = add2(x, fma2(t, both(-1.0f), both(kRound)));
  uint64_t y = fma2(f, both(0x1.41fbbcp-13f), both(0x1.5f3e54p-10f));
  y = fma2(y, f, both(0x1.3b2d4cp-7f));
  y = fma2(y, f, both(0x1.c6aee8p-5f));
  y = fma2(y, f, both(0x1.ebfbdcp-3f));
  y = fma2(y, f, both(0x1.62e430p-1f));
  y = fma2(y, f, both(1.0f));
  const float2 n = unpack2(t);
  return mul2(y, pack2(__uint_as_float(__float_as_uint(n.x) << 23), __uint_as_float(__float_as_uint(n.y) << 23)));
}

// 2^x of pair k of a chunk
template <bool BOTH_PIPES>
__device__ __forceinline__ uint64_t ex2_pair(uint64_t x, int k) {
  constexpr int kPairs = kChunk / 2;
  if (BOTH_PIPES && (k + 1) * kPolyPairs / kPairs != k * kPolyPairs / kPairs) return ex2_poly2(x);
  const float2 a = unpack2(x);
  return pack2(ex2_approx(a.x), ex2_approx(a.y));
}

// four fp32 -> four E4M3 bytes in one register
__device__ __forceinline__ uint32_t f32x4_to_e4m3x4(float a, float b, float c, float d) {
  uint32_t r;
  asm("{\n\t.reg .b16 lo, hi;\n\tcvt.rn.satfinite.e4m3x2.f32 lo, %2, %1;\n\tcvt.rn.satfinite.e4m3x2.f32 hi, %4, %3;\n\t"
      "mov.b32 %0, {lo, hi};\n\t}"
      : "=r"(r)
      : "f"(a), "f"(b), "f"(c), "f"(d));
  return r;
}

// QT: type of the queries, uint8_t = E4M3 codes (tmap_q); WIDE: their rows start on 32-byte boundaries.
// Queries that are not codes yet are quantized here, by the softmax warps while K is on its way and the kernel in front still writes the
// operands of K and V: each is read by one CTA only, so a pass of its own would write and read their codes for nothing.  Both launches,
// us, operand pass for all three / this: [4, 32 / 8, 2048, 128] causal 212 / 202; [3, 16, 577 x 1500, 64] 51 / 47.7; [8, 32 / 8, 1024,
// 128] causal 147 / 137; [8, 12, 200, 128] causal 21.2 / 18.9; [1, 8, 64, 64] 13.1 / 11.2.
// FREE: bf16 results.  There an eighth of the exponentials runs on the FMA pipe and the last key tile keeps its own.  Neither holds
// anything in fewer bits, but both change roundings, and a probability as near to a boundary of E4M3 as fp32 resolves it may take the
// code on the other side.  How near, in both forms and for rows of up to 200 keys: within 2^-24 ln 2 (8 s + 16) + 2^-21 of it, s the
// row's largest score in powers of two; a few of 100 000 probabilities.  (Distance to 64 bits at [4, 32 / 8, 2048, 128] causal
// 1.678e-3 -> 1.656e-3.)  Such a probability changes by one step, at most an eighth.  In a row of few keys that is several steps of a
// bf16 result; in rows of many, single values moved by up to 0.12 against the other form, 3.5e-4 of the norm.  The line lies at the
// type because the same change is eight times as many steps of an fp16 result, which callers compare to 1e-3: fp16 and fp32 keep every
// operation and its order.
template <typename QT, bool WIDE, bool FREE>
__global__ void __launch_bounds__(kAttThreads, 2)
fp8_sdpa_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                const __grid_constant__ CUtensorMap tmap_vt, const AttParams p) {
  // the 128-byte swizzle counts from 1024-byte boundaries; addresses that are constants keep the single-thread roles short
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* sq = smem;
  uint8_t* sk = sq + kTileBytes;
  uint8_t* sv = sk + kKStages * kTileBytes;
  uint8_t* sp = sv + kVStages * kTileBytes;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sp + 2 * kTileBytes);
  uint64_t* q_full = bars;
  uint64_t* k_full = q_full + 1;
  uint64_t* k_empty = k_full + kKStages;
  uint64_t* v_full = k_empty + kKStages;
  uint64_t* v_empty = v_full + kVStages;
  uint64_t* s_full = v_empty + kVStages;     // score buffers in tensor memory
  uint64_t* s_empty = s_full + 2;
  uint64_t* p_full = s_empty + 2;            // 2 probability tiles in shared memory
  uint64_t* p_empty = p_full + 2;
  uint64_t* o_full = p_empty + 2;
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(o_full + 1);

  if ((ptx::smem_u32(smem) & 1023u) != 0) {                   // cannot be: no static shared memory stands in front
    if (threadIdx.x == 0) att_timeout(p.status, 60);
    return;
  }
  constexpr bool kCodes = std::is_same<QT, uint8_t>::value;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // CTAs walk the heads in groups (head_group), in a group the query tiles with the most keys first: a causal launch then
  // ends on its shortest CTAs
  int head0 = 0, heads = p.BH, place = static_cast<int>(blockIdx.x);
  if (p.group < p.BH) {
    head0 = place / (p.group * p.q_tiles) * p.group;
    heads = min(p.group, p.BH - head0);
    place -= head0 * p.q_tiles;
  }
  const int q_tile = place / heads;
  const int q0 = (p.q_tiles - 1 - q_tile) * kTile;
  const int bh = head0 + place - q_tile * heads;              // b * Hq + h
  const int b = bh / p.Hq, h = bh - b * p.Hq;
  const int bhkv = b * p.Hkv + h / (p.Hq / p.Hkv);
  const int shift = p.Sk - p.Sq;                              // causal: key j visible to query i when j <= i + shift
  int k_end = p.Sk;
  if (p.causal) k_end = max(0, min(p.Sk, q0 + kTile + shift));
  const int n_tiles = (k_end + kTile - 1) / kTile;

  if (threadIdx.x == 0) {
    ptx::mbar_init(q_full, 1);
    for (int s = 0; s < kKStages; ++s) ptx::mbar_init(k_full + s, 1), ptx::mbar_init(k_empty + s, 1);
    for (int s = 0; s < kVStages; ++s) ptx::mbar_init(v_full + s, 1), ptx::mbar_init(v_empty + s, 1);
    for (int s = 0; s < 2; ++s) {
      ptx::mbar_init(s_full + s, 1);
      ptx::mbar_init(s_empty + s, 8);   // one arrival per softmax warp
      ptx::mbar_init(p_full + s, 8);
      ptx::mbar_init(p_empty + s, 1);
    }
    ptx::mbar_init(o_full, 1);
    ptx::fence_barrier_init();
    ptx::prefetch_tmap(&tmap_vt);
    // this thread is the producer: the first tiles are requested in front of the tensor-memory allocation, once the kernel that
    // writes the operands is complete (it may still run under a programmatic launch)
    pdl_wait();
    ptx::fence_proxy_async_all();
    if constexpr (kCodes) {
      ptx::mbar_arrive_expect_tx(q_full, kTileBytes);
      ptx::tma_load_3d(sq, &tmap_q, q_full, 0, q0, bh);
    }
    if (n_tiles > 0) {
      ptx::mbar_arrive_expect_tx(k_full, kTileBytes);
      ptx::tma_load_3d(sk, &tmap_k, k_full, 0, 0, bhkv);
    }
  }
  if (warp == 1) {
    ptx::tmem_alloc<1>(tmem_holder, kTmemCols);
    ptx::tmem_relinquish<1>();
  }
  float q_scale = 0.0f;
  if constexpr (!kCodes) {
    if (warp >= 2) {
      // 128 rows in pieces of 16 elements, 8 to a row, 4 to a thread.  Queries and their range are older than the kernel in front
      // of this one, so nothing waits for that.
      const int g = threadIdx.x & 7, row0 = (static_cast<int>(threadIdx.x) - 64) >> 3;
      const QT* src = static_cast<const QT*>(p.q) + b * p.q_sb + h * p.q_sh + static_cast<int64_t>(q0 + row0) * p.q_ss + g * 16;
      Raw16<QT, WIDE> raw[4];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (g * 16 < p.D && q0 + row0 + u * 32 < p.Sq) raw[u].load(src + static_cast<int64_t>(u * 32) * p.q_ss);
      q_scale = fp8_scale_from_amax(ld_dependent(p.q_amax));
      const float y = b200q_rcp_rn(q_scale), lim = __fmul_rn(q_scale, 512.0f);
      const bool fast = b200q_div_fast_ok(q_scale) != 0;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int row = row0 + u * 32;
        uint4 c = make_uint4(0u, 0u, 0u, 0u);     // rows past the end, and columns D..: the contraction takes 32 at a time
        if (g * 16 < p.D && q0 + row < p.Sq) c = e4m3_of_16(raw[u], q_scale, y, lim, fast);
        *reinterpret_cast<uint4*>(sq + row * 128 + ((g ^ (row & 7)) * 16)) = c;
      }
      ptx::fence_proxy_async();                   // the tensor core reads this tile through the async proxy
    }
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem_base = *tmem_holder;
  const uint32_t tmem_o = tmem_base + kTile;

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer
    if (lane == 0) {
      int ks = n_tiles > 0 ? 1 : 0, vs = 0;       // the first K tile is on its way (above)
      uint32_t kph = 0, vph = 0;
      bool ok = true;
      // the order of the loads is the order in which the MMA thread uses them: pass 1 all K tiles; pass 2, which begins with
      // the last key tile and needs no scores for it, K 0, K 1, V last, K 2, V 0, K 3, V 1, ...
      auto load_k = [&](int j) -> bool {
        if (!ptx::mbar_wait(k_empty + ks, kph ^ 1u)) {
          att_timeout(p.status, 61);
          return false;
        }
        ptx::mbar_arrive_expect_tx(k_full + ks, kTileBytes);
        ptx::tma_load_3d(sk + ks * kTileBytes, &tmap_k, k_full + ks, 0, j * kTile, bhkv);
        if (++ks == kKStages) ks = 0, kph ^= 1u;
        return true;
      };
      auto load_v = [&](int j) -> bool {
        if (!ptx::mbar_wait(v_empty + vs, vph ^ 1u)) {
          att_timeout(p.status, 62);
          return false;
        }
        ptx::mbar_arrive_expect_tx(v_full + vs, kTileBytes);
        ptx::tma_load_3d(sv + vs * kTileBytes, &tmap_vt, v_full + vs, j * kTile, 0, bhkv);
        if (++vs == kVStages) vs = 0, vph ^= 1u;
        return true;
      };
      for (int j = 1; j < n_tiles && ok; ++j) ok = load_k(j);
      // (FREE; otherwise from the first tile on: K 0, K 1, K 2, V 0, ...)
      for (int i = FREE ? 1 : 0; i < n_tiles + 2 && ok; ++i) {
        if (i < n_tiles) ok = load_k(FREE ? i - 1 : i);
        if (ok && i >= 2) ok = load_v(!FREE ? i - 2 : (i == 2 ? n_tiles - 1 : i - 3));
      }
      // drain: every load issued above has landed and was consumed before shared memory is released
      for (int s = 0; s < kKStages && ok; ++s) {
        const int st = (ks + s) % kKStages;
        const uint32_t ph = (st >= ks) ? kph : (kph ^ 1u);
        if (!ptx::mbar_wait(k_empty + st, ph ^ 1u)) att_timeout(p.status, 63), ok = false;
      }
      for (int s = 0; s < kVStages && ok; ++s) {
        const int st = (vs + s) % kVStages;
        const uint32_t ph = (st >= vs) ? vph : (vph ^ 1u);
        if (!ptx::mbar_wait(v_empty + st, ph ^ 1u)) att_timeout(p.status, 64), ok = false;
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer
    if (lane == 0) {
      constexpr uint32_t idesc_s = ptx::idesc_f8(kTile, kTile);
      const uint32_t idesc_o = ptx::idesc_f8(kTile, p.D);       // only the head's own columns
      const int kb_scores = (p.D + 31) / 32;                    // 32 bytes of the head dimension per MMA
      const uint32_t q_lo = ptx::desc_lo_sw128(ptx::smem_u32(sq));
      const uint32_t k_lo0 = ptx::desc_lo_sw128(ptx::smem_u32(sk));
      const uint32_t v_lo0 = ptx::desc_lo_sw128(ptx::smem_u32(sv));
      const uint32_t p_lo0 = ptx::desc_lo_sw128(ptx::smem_u32(sp));
      int ks = 0, vs = 0, pb = 0;
      uint32_t kph = 0, vph = 0, pph = 0;
      uint32_t sph0 = 0, sph1 = 0;                              // score buffers: parity of their next use
      bool ok = true;
      if constexpr (kCodes) ok = ptx::mbar_wait(q_full, 0);     // else written in front of the barrier above
      if (!ok) att_timeout(p.status, 65);
      // scores of the next key tile in ring order into score buffer `sb`
      auto issue_scores = [&](int sb) -> bool {
        const uint32_t sph = sb == 0 ? sph0 : sph1;
        if (!ptx::mbar_wait(k_full + ks, kph) || !ptx::mbar_wait(s_empty + sb, sph ^ 1u)) {
          att_timeout(p.status, 66);
          return false;
        }
        ptx::tc_fence_after();
        const uint32_t k_lo = k_lo0 + ks * (kTileBytes >> 4);
#pragma unroll
        for (int kb = 0; kb < 4; ++kb)
          if (kb < kb_scores)
            ptx::mma_f8<1>(tmem_base + sb * kTile, ptx::desc_join(q_lo + kb * 2, ptx::kDescHiSw128),
                           ptx::desc_join(k_lo + kb * 2, ptx::kDescHiSw128), idesc_s, kb > 0 ? 1u : 0u);
        ptx::tc_commit<1>(s_full + sb);
        ptx::tc_commit<1>(k_empty + ks);
        if (sb == 0) sph0 ^= 1u;
        else sph1 ^= 1u;
        if (++ks == kKStages) ks = 0, kph ^= 1u;
        return true;
      };
      for (int j = 0; j < n_tiles && ok; ++j) ok = issue_scores(j & 1);    // pass 1: scores only, two buffers
      // pass 2, the last key tile (no scores) and then 0, 1, ..: the scores of the tile after next are issued in front of the
      // product of a tile.  Their buffer is free once every warp has taken the next tile, which it does right after writing its
      // part of P: the warps wait for scores, nobody waits for the product yet.
      // (Without FREE tile 0 is the first and has scores as well.)
      for (int j = FREE ? 1 : 0; j < min(2, n_tiles) && ok; ++j) ok = issue_scores(0);
      for (int j = 0; j < n_tiles && ok; ++j) {
        if (j + 2 < n_tiles) ok = issue_scores(0);
        if (!ok) break;
        if (!ptx::mbar_wait(p_full + pb, pph) || !ptx::mbar_wait(v_full + vs, vph)) {
          att_timeout(p.status, 67);
          ok = false;
          break;
        }
        ptx::tc_fence_after();
        const uint32_t p_lo = p_lo0 + pb * (kTileBytes >> 4);
        const uint32_t v_lo = v_lo0 + vs * (kTileBytes >> 4);
#pragma unroll
        for (int kb = 0; kb < 4; ++kb)
          ptx::mma_f8<1>(tmem_o, ptx::desc_join(p_lo + kb * 2, ptx::kDescHiSw128), ptx::desc_join(v_lo + kb * 2, ptx::kDescHiSw128),
                         idesc_o, (j > 0 || kb > 0) ? 1u : 0u);
        ptx::tc_commit<1>(p_empty + pb);
        ptx::tc_commit<1>(v_empty + vs);
        if (++vs == kVStages) vs = 0, vph ^= 1u;
        if (++pb == 2) pb = 0, pph ^= 1u;
      }
      if (ok) ptx::tc_commit<1>(o_full);
    }
  } else {
    // ------------------------------------------------------------ softmax (warps 2..9): two threads per query row.
    // A warp reaches the 32 tensor-memory lanes of its quarter (warp & 3); the two warps of a quarter split
    // the columns: warp set `ch` takes the 32-column chunks ch and ch + 2 of every score tile (columns 32 ch .. and
    // 64 + 32 ch ..).  A thread takes both into registers and hands the buffer back before it computes, so the
    // tensor core fills the next tile under the exponentials of this one.
    const int q = warp & 3;
    const int ch = (warp - 2) >> 2;
    const int r = q * 32 + lane;                  // row inside the tile
    const int qi = q0 + r;                        // query index inside the head
    const uint32_t lane_addr = static_cast<uint32_t>(q * 32) << 16;
    // scores in the base-2 exponent domain: s2 = acc * c2, c2 = q_scale * k_scale * softmax_scale * log2(e) > 0,
    // so the running maximum is kept on the raw accumulators and the scaling rides in the FMA in front of ex2
    pdl_wait();                                   // the other scales come from the kernel in front; results are stored behind it
    if constexpr (kCodes) q_scale = ld_dependent(p.q_scale);
    const float c2 = q_scale * ld_dependent(p.k_scale) * p.softmax_scale * 1.4426950408889634f;
    const uint64_t c2c2 = pack2(c2, c2);
    const int last_key = p.causal ? min(k_end - 1, qi + shift) : k_end - 1;   // keys beyond it are masked for this row
    // key tiles below this index are visible to every row of the CTA in full: no per-element mask there
    const int full_tiles = (p.causal ? max(0, min(k_end, q0 + shift + 1)) : k_end) / kTile;
    int pb = 0;
    uint32_t sph0 = 0, sph1 = 0, pph = 0;
    float m = -INFINITY, l = 0.0f;                // raw-accumulator maximum, sum of 2^(s2 - m * c2)
    bool ok = true;
    // scores of key tile j (buffer sb) into v (chunk ch, then chunk ch + 2), masked; false when the wait gave up
    auto take_scores = [&](auto masked, int j, int sb, uint32_t* v) -> bool {
      if (!ptx::mbar_wait(s_full + sb, sb == 0 ? sph0 : sph1)) return false;
      if (sb == 0) sph0 ^= 1u;
      else sph1 ^= 1u;
      ptx::tc_fence_after();
      const uint32_t taddr = tmem_base + lane_addr + sb * kTile + ch * kChunk;
      ptx::tmem_ld_32x32(taddr, v);
      ptx::tmem_ld_32x32(taddr + 2 * kChunk, v + kChunk);
      ptx::tmem_ld_wait();
      ptx::tc_fence_before();
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(s_empty + sb);
      if constexpr (decltype(masked)::value) {
        const int visible = last_key - (j * kTile + ch * kChunk);      // index of the last visible column, from the first chunk's start
#pragma unroll
        for (int i = 0; i < kChunk; ++i) {
          if (i > visible) v[i] = 0xff800000u;   // -inf
          if (i + 2 * kChunk > visible) v[kChunk + i] = 0xff800000u;
        }
      }
      return true;
    };
    // ---- pass 1: running maximum and sum
    auto pass1 = [&](auto masked, int j) -> bool {
      uint32_t vv[2 * kChunk];
      if (!take_scores(masked, j, j & 1, vv)) {
        att_timeout(p.status, 68);
        return false;
      }
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const uint32_t* v = vv + c * kChunk;
        // four independent chains each for the maximum and the sum: a warp has few neighbours on its scheduler
        // here, so the length of a dependent chain is what it waits for
        float x0 = __uint_as_float(v[0]), x1 = __uint_as_float(v[1]), x2 = __uint_as_float(v[2]), x3 = __uint_as_float(v[3]);
#pragma unroll
        for (int i = 4; i < kChunk; i += 4) {
          x0 = fmaxf(x0, __uint_as_float(v[i]));
          x1 = fmaxf(x1, __uint_as_float(v[i + 1]));
          x2 = fmaxf(x2, __uint_as_float(v[i + 2]));
          x3 = fmaxf(x3, __uint_as_float(v[i + 3]));
        }
        const float cm = fmaxf(fmaxf(x0, x1), fmaxf(x2, x3));
        if (cm > m) {
          l *= ex2_approx((m - cm) * c2);         // m = -inf: l is 0 and stays 0
          m = cm;
        }
        // nothing visible yet (m = -inf): offset 0, every exponential of -inf adds 0
        const float off = m > -INFINITY ? -m * c2 : 0.0f;
        const uint64_t offoff = pack2(off, off);
        uint64_t l01 = 0ull, l23 = 0ull;          // pairs of zeros
#pragma unroll
        for (int i = 0; i < kChunk; i += 4) {
          l01 = add2(l01, ex2_pair<FREE>(fma2(pack2(__uint_as_float(v[i]), __uint_as_float(v[i + 1])), c2c2, offoff), i / 2));
          l23 = add2(l23, ex2_pair<FREE>(fma2(pack2(__uint_as_float(v[i + 2]), __uint_as_float(v[i + 3])), c2c2, offoff), i / 2 + 1));
        }
        const float2 s0 = unpack2(l01), s1 = unpack2(l23);
        l += (s0.x + s0.y) + (s1.x + s1.y);
      }
      return true;
    };
    // The last key tile keeps its exponentials: pass 2 begins with them and scales them, so that this tile's scores are computed and
    // raised once.  One maximum over both chunks, so that they all have one reference.  Whole calls, us, without / with it: causal
    // [8, 12, 200, 128] 18.8 / 16.9, [8, 48 / 12, 300, 128] 57.9 / 54.2, [8, 32 / 8, 1024, 128] 137.3 / 133.7, [4, 32 / 8, 2048, 128]
    // 202.9 / 199.1; [4, 12, 3000 x 300, 80] 59.9 / 57.8, [3, 16, 577 x 1500, 64] 48.2 / 48.0.  The probabilities of that tile lose two
    // roundings (distance to 64 bits at the fourth of these 1.678e-3 -> 1.656e-3).
    uint32_t e[2 * kChunk];
    auto pass1_last = [&]() -> bool {
      if (!take_scores(std::true_type{}, n_tiles - 1, (n_tiles - 1) & 1, e)) {
        att_timeout(p.status, 68);
        return false;
      }
      float x0 = __uint_as_float(e[0]), x1 = __uint_as_float(e[1]), x2 = __uint_as_float(e[2]), x3 = __uint_as_float(e[3]);
#pragma unroll
      for (int i = 4; i < 2 * kChunk; i += 4) {
        x0 = fmaxf(x0, __uint_as_float(e[i]));
        x1 = fmaxf(x1, __uint_as_float(e[i + 1]));
        x2 = fmaxf(x2, __uint_as_float(e[i + 2]));
        x3 = fmaxf(x3, __uint_as_float(e[i + 3]));
      }
      const float cm = fmaxf(fmaxf(x0, x1), fmaxf(x2, x3));
      if (cm > m) {
        l *= ex2_approx((m - cm) * c2);
        m = cm;
      }
      const float off = m > -INFINITY ? -m * c2 : 0.0f;
      const uint64_t offoff = pack2(off, off);
      uint64_t l01 = 0ull, l23 = 0ull;
#pragma unroll
      for (int i = 0; i < 2 * kChunk; i += 4) {
        const uint64_t a = ex2_pair<FREE>(fma2(pack2(__uint_as_float(e[i]), __uint_as_float(e[i + 1])), c2c2, offoff), (i / 2) & 15);
        const uint64_t b = ex2_pair<FREE>(fma2(pack2(__uint_as_float(e[i + 2]), __uint_as_float(e[i + 3])), c2c2, offoff), (i / 2 + 1) & 15);
        l01 = add2(l01, a);
        l23 = add2(l23, b);
        const float2 ua = unpack2(a), ub = unpack2(b);
        e[i] = __float_as_uint(ua.x), e[i + 1] = __float_as_uint(ua.y), e[i + 2] = __float_as_uint(ub.x), e[i + 3] = __float_as_uint(ub.y);
      }
      const float2 s0 = unpack2(l01), s1 = unpack2(l23);
      l += (s0.x + s0.y) + (s1.x + s1.y);
      return true;
    };
    const int rest = FREE ? n_tiles - 1 : n_tiles, first_edge = min(full_tiles, rest);
    for (int j = 0; j < first_edge && ok; ++j) ok = pass1(std::false_type{}, j);
    for (int j = max(first_edge, 0); j < rest && ok; ++j) ok = pass1(std::true_type{}, j);
    if (FREE && n_tiles > 0 && ok) ok = pass1_last();
    // The two threads of a row each hold the statistics of their columns: merge (every softmax thread gets here).  They pass them
    // on through the first probability tile, each in a piece of this row that the other one alone writes later, behind its read.
    uint8_t* srow = sp + r * 128;
    *reinterpret_cast<float2*>(srow + (((2 * (ch ^ 1)) ^ (r & 7)) * 16)) = make_float2(m, l);
    asm volatile("bar.sync 1, 256;" ::: "memory");
    const float m_own = m;
    {
      const float2 o = *reinterpret_cast<const float2*>(srow + (((2 * ch) ^ (r & 7)) * 16));
      const float mm = fmaxf(m, o.x);
      const float mine = m > -INFINITY ? l * ex2_approx((m - mm) * c2) : 0.0f;
      const float theirs = o.x > -INFINITY ? o.y * ex2_approx((o.x - mm) * c2) : 0.0f;
      l = mine + theirs;
      m = mm;
    }
    // ---- pass 2: final probabilities, quantized with scale 1/448, written as the A operand of P V:
    // 448 * 2^(s2 - m2) / l = 2^(acc * c2 + off2) with the normaliser folded into the exponent
    const float off2 = l > 0.0f ? -m * c2 + __log2f(kE4M3Max / l) : -INFINITY;
    const uint64_t off22 = pack2(off2, off2);
    // 16 columns = one 16-byte piece of the operand row; 128-byte swizzle: the piece i of row r lives at piece i ^ (r & 7)
    auto put_piece = [&](uint8_t* prow, int g, const uint32_t* w) {
      const int piece = 2 * ch + (g & 1) + 4 * (g >> 1);
      *reinterpret_cast<uint4*>(prow + ((piece ^ (r & 7)) * 16)) = make_uint4(w[0], w[1], w[2], w[3]);
    };
    auto tile_written = [&]() {
      ptx::fence_proxy_async();                   // the tensor core reads this tile through the async proxy
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(p_full + pb);
      if (++pb == 2) pb = 0, pph ^= 1u;
    };
    if (FREE && n_tiles > 0 && ok) {              // the last key tile: 448 * e / l, e referred from this thread's maximum to the row's
      const float f = l > 0.0f ? kE4M3Max / l * ex2_approx((m_own - m) * c2) : 0.0f;
      const uint64_t ff = pack2(f, f);
#pragma unroll
      for (int g = 0; g < 4; ++g) {
        uint32_t w[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const uint32_t* t = e + g * 16 + i * 4;
          const float2 a = unpack2(mul2(pack2(__uint_as_float(t[0]), __uint_as_float(t[1])), ff));
          const float2 b = unpack2(mul2(pack2(__uint_as_float(t[2]), __uint_as_float(t[3])), ff));
          w[i] = f32x4_to_e4m3x4(a.x, a.y, b.x, b.y);
        }
        put_piece(sp + r * 128, g, w);
      }
      tile_written();
    }
    auto pass2 = [&](auto masked, int j) -> bool {
      uint32_t v[2 * kChunk];
      if (!take_scores(masked, j, 0, v) || !ptx::mbar_wait(p_empty + pb, pph ^ 1u)) {
        att_timeout(p.status, 69);
        return false;
      }
      uint8_t* prow = sp + pb * kTileBytes + r * 128;
#pragma unroll
      for (int g = 0; g < 4; ++g) {               // 16 columns = one 16-byte piece of the operand row
        uint32_t w[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const uint32_t* e = v + g * 16 + i * 4;
          const int k = (g & 1) * 8 + i * 2;
          const float2 a = unpack2(ex2_pair<FREE>(fma2(pack2(__uint_as_float(e[0]), __uint_as_float(e[1])), c2c2, off22), k));
          const float2 b = unpack2(ex2_pair<FREE>(fma2(pack2(__uint_as_float(e[2]), __uint_as_float(e[3])), c2c2, off22), k + 1));
          w[i] = f32x4_to_e4m3x4(a.x, a.y, b.x, b.y);
        }
        put_piece(prow, g, w);
      }
      tile_written();
      return true;
    };
    for (int j = 0; j < first_edge && ok; ++j) ok = pass2(std::false_type{}, j);
    for (int j = max(first_edge, 0); j < rest && ok; ++j) ok = pass2(std::true_type{}, j);
    // ---- output: O * (v_scale / 448) -> out dtype
    if (ok && n_tiles > 0 && !ptx::mbar_wait(o_full, 0)) {
      att_timeout(p.status, 70);
      ok = false;
    }
    // tcgen05.ld is a warp-wide instruction: every lane of the warp takes part in the loads, rows past the
    // end of the sequence only skip their stores
    if (ok && q0 + q * 32 < p.Sq) {
      ptx::tc_fence_after();
      const float oscale = n_tiles > 0 ? ld_dependent(p.v_scale) / kE4M3Max : 0.0f;
      const int64_t row_off = b * p.out_sb + h * p.out_sh + qi * p.out_ss;
#pragma unroll 1
      for (int c = 2 * ch; c < 2 * ch + 2; ++c) {
        if (c * 32 >= p.D) break;
        uint32_t v[32];
        if (n_tiles > 0) {
          ptx::tmem_ld_32x32(tmem_o + lane_addr + c * 32, v);
          ptx::tmem_ld_wait();
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] = 0u;
        }
#pragma unroll
        for (int g = 0; g < 4; ++g) {             // 8 columns per store
          const int col = c * 32 + g * 8;
          if (col >= p.D || qi >= p.Sq) break;
          float x[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) x[i] = __uint_as_float(v[g * 8 + i]) * oscale;
          if (p.out_dtype == B200Q_BF16) Elem<__nv_bfloat16>::store8(static_cast<__nv_bfloat16*>(p.out) + row_off + col, x);
          else if (p.out_dtype == B200Q_F16) Elem<__half>::store8(static_cast<__half*>(p.out) + row_off + col, x);
          else Elem<float>::store8(static_cast<float*>(p.out) + row_off + col, x);
        }
      }
    }
  }

  ptx::tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc<1>(tmem_base, kTmemCols);
  }
}

// ---------------------------------------------------------------- Q, K, V -> operands
// One launch quantizes Q and K to E4M3 codes [B, H, S, D] and V to codes transposed per head [B, H, D, vt_stride]
// (keys contiguous, zero beyond S).  The inputs may be strided (D contiguous): a token-major [tokens, heads * D] slice
// of a QKV projection is read where it lies.  HBM-bound (3 bytes per 16-bit element); a CTA takes 128 rows of one
// head, 16 elements per thread and step with four steps of loads in flight.  Before, Q and K went through the
// row kernels, one CTA per row of D elements (at [4, 32, 2048, 128] 262144 CTAs of which 16 threads had work), and V through a
// byte-wise transpose: 355 us for the three operands of [4, 32 / 8, 2048, 128] bf16.  With a division per element and its choice of
// path inside the loop, 60 % of the issue slots were taken at 36 % of the memory's rate: 42 us; two quotients at a time where a piece
// lies within the range (e4m3_of_16): 31.6 us (4.8 TB/s), 12.7 for K and V alone (b200q_fp8_attention).
struct QkvPart {
  const void* x;
  int64_t sb, sh, ss;        // strides of batch, head, row in elements
  const float* amax;
  uint8_t* out;
  float* scale_out;
  int H, S;
  int tiles;                 // tiles of 128 rows per head
};
struct QkvParts {
  QkvPart part[3];
  int first[3];              // first CTA of each part
  int D;
  int inv_pieces;            // 65536 / (D / 16), rounded up: t / pieces = t * inv_pieces >> 16 for t < 2048
  int64_t vt_stride;
};

template <typename T, bool WIDE>
__global__ void __launch_bounds__(256)
fp8_attention_quantize_kernel(const __grid_constant__ QkvParts p) {
  __shared__ uint32_t tile[kTile * 32];           // V: 128 keys x 128 bytes
  const int cta = static_cast<int>(blockIdx.x);
  const int which = cta >= p.first[2] ? 2 : (cta >= p.first[1] ? 1 : 0);
  const QkvPart& part = p.part[which];
  pdl_launch_dependents();   // the attention kernel behind it may quantize its first queries meanwhile
  if (cta == 0 && threadIdx.x < 3 && p.part[threadIdx.x].scale_out != nullptr)
    *p.part[threadIdx.x].scale_out = fp8_scale_from_amax(__ldg(p.part[threadIdx.x].amax));
  const int local = cta - p.first[which];
  const int head = local / part.tiles;            // b * H + h
  const int r0 = (local - head * part.tiles) * kTile;
  const int b = head / part.H, h = head - b * part.H;
  const T* x = static_cast<const T*>(part.x) + b * part.sb + h * part.sh;
  const float scale = fp8_scale_from_amax(__ldg(part.amax));
  const float y = b200q_rcp_rn(scale);
  const bool fast = b200q_div_fast_ok(scale) != 0;
  const float lim = __fmul_rn(scale, 512.0f);     // |x| >= 512 * scale saturates to 448 anyway
  const int pieces = p.D >> 4;                    // 16-element pieces of a row
  constexpr int U = sizeof(T) == 4 ? 2 : 4;
  const int rows = min(kTile, part.S - r0);       // V: rows beyond S up to the tile's end are zero codes
  for (int t0 = threadIdx.x; t0 < kTile * pieces; t0 += 256 * U) {
    Raw16<T, WIDE> raw[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int t = t0 + u * 256, row = t * p.inv_pieces >> 16, g = t - row * pieces;
      if (row < rows) raw[u].load(x + static_cast<int64_t>(r0 + row) * part.ss + g * 16);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int t = t0 + u * 256, row = t * p.inv_pieces >> 16, g = t - row * pieces;
      uint4 c = make_uint4(0u, 0u, 0u, 0u);
      if (row < rows) {
        c = e4m3_of_16(raw[u], scale, y, lim, fast);
        if (which != 2)
          *reinterpret_cast<uint4*>(part.out + (static_cast<int64_t>(head) * part.S + r0 + row) * p.D + g * 16) = c;
      }
      // 16-byte pieces of a key row are swizzled by the key's group of 16, so that the transposing reads below
      // (8 key groups x 4 words) hit 32 different banks
      if (which == 2 && row < kTile) *reinterpret_cast<uint4*>(&tile[row * 32 + ((g ^ ((row >> 4) & 7)) << 2)]) = c;
    }
  }
  if (which != 2) return;
  __syncthreads();
  // item: 4 columns (one word) of 16 keys, transposed in 4 x 4 byte blocks -> four 16-byte stores
  for (int t = threadIdx.x; t < pieces * 4 * 8; t += 256) {
    const int kg = t & 7, d4 = t >> 3;
    if (r0 + kg * 16 >= p.vt_stride) continue;
    uint32_t o[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint32_t* src = &tile[(kg * 16 + i * 4) * 32 + (d4 ^ (kg << 2))];
      const uint32_t k0 = src[0], k1 = src[32], k2 = src[64], k3 = src[96];
      const uint32_t a01 = __byte_perm(k0, k1, 0x5140), a23 = __byte_perm(k2, k3, 0x5140);
      const uint32_t b01 = __byte_perm(k0, k1, 0x7362), b23 = __byte_perm(k2, k3, 0x7362);
      o[0][i] = __byte_perm(a01, a23, 0x5410);
      o[1][i] = __byte_perm(a01, a23, 0x7632);
      o[2][i] = __byte_perm(b01, b23, 0x5410);
      o[3][i] = __byte_perm(b01, b23, 0x7632);
    }
    uint8_t* dst = part.out + (static_cast<int64_t>(head) * p.D + d4 * 4) * p.vt_stride + r0 + kg * 16;
#pragma unroll
    for (int i = 0; i < 4; ++i) *reinterpret_cast<uint4*>(dst + i * p.vt_stride) = make_uint4(o[i][0], o[i][1], o[i][2], o[i][3]);
  }
}

// `first` and the grid of the parts filled in; 0 CTAs = nothing to do.
int launch_attention_quantize(QkvParts& p, int B, int dtype, cudaStream_t st) {
  int64_t ctas = 0;
  p.inv_pieces = 65536 / (p.D / 16) + 1;
  for (int i = 0; i < 3; ++i) {
    p.first[i] = static_cast<int>(ctas);
    // V: the zero columns between S and the row stride are written too
    const int64_t extent = i < 2 ? p.part[i].S : (p.part[i].S > 0 ? p.vt_stride : 0);
    p.part[i].tiles = static_cast<int>((extent + kTile - 1) / kTile);
    ctas += static_cast<int64_t>(p.part[i].tiles) * p.part[i].H * B;
    if (ctas > 0x7fffffffLL) return B200Q_ERR_INVALID;
  }
  if (ctas == 0) return B200Q_OK;
  // 256-bit loads when every row starts on a 32-byte boundary
  const int64_t unit = dtype == B200Q_F32 ? 8 : 16;
  bool wide = true;
  for (int i = 0; i < 3; ++i) {
    const QkvPart& a = p.part[i];
    wide = wide && (a.tiles == 0 || (aligned(a.x, 32) && a.sb % unit == 0 && a.sh % unit == 0 && a.ss % unit == 0));
  }
  const dim3 grid(static_cast<unsigned>(ctas));
#define B200Q_AQ(T)                                                                  \
  do {                                                                               \
    if (wide) fp8_attention_quantize_kernel<T, true><<<grid, 256, 0, st>>>(p);       \
    else fp8_attention_quantize_kernel<T, false><<<grid, 256, 0, st>>>(p);           \
  } while (0)
  switch (dtype) {
    case B200Q_BF16: B200Q_AQ(__nv_bfloat16); break;
    case B200Q_F16: B200Q_AQ(__half); break;
    case B200Q_F32: B200Q_AQ(float); break;
    default: return B200Q_ERR_INVALID;
  }
#undef B200Q_AQ
  return check_launch();
}

// [inner bytes, rows, heads] byte tensor -> boxes of 128 x 128 x 1, 128-byte swizzle, zero fill out of bounds
int make_head_map(CUtensorMap* map, const void* base, int64_t inner, int64_t rows, int64_t heads, int64_t row_stride) {
  gemm::EncodeTiledFn fn = gemm::encode_tiled();
  if (fn == nullptr) return B200Q_ERR_CUDA;
  const cuuint64_t dims[3] = {static_cast<cuuint64_t>(inner), static_cast<cuuint64_t>(rows), static_cast<cuuint64_t>(heads)};
  const cuuint64_t strides[2] = {static_cast<cuuint64_t>(row_stride), static_cast<cuuint64_t>(row_stride * rows)};
  const cuuint32_t box[3] = {128, 128, 1};
  const cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? B200Q_OK : B200Q_ERR_CUDA;
}

// Heads whose query tiles are walked together, longest first.  All heads, where their K and V codes stay in L2: a causal launch
// then ends on its shortest tiles whatever its heads.  Where they do not, all running CTAs would stream keys of their own from
// HBM, so only as many heads as have 32 MB of codes (at least the query heads of one kv head).  Measured, us a call, head by
// head in order of the queries / all heads at once / this: causal [4, 64, 8192, 128] 6580 / 6440 to 7320 / 5845, [8, 32, 4096,
// 128] 1918 / 1860 to 2055 / 1720; [8, 32, 2048 x 4096, 128] without a mask 1738 / 1734 to 1930 / 1576, [2, 128, 1024 x 16384,
// 128] 3875 / 3980 / 3436; groups of 16 to 64 MB within 2 % of each other.  Causal [4, 32 / 8, 2048, 128], 17 MB: 246 with all
// heads, 272 with 8.
int head_group(const AttParams& p) {
  const int rep = p.Hq / p.Hkv;
  const int64_t kv_bytes = 2LL * p.Sk * p.D;
  const int64_t kv_heads = kv_bytes > 0 ? (int64_t{32} << 20) / kv_bytes : p.BH;
  const int64_t heads = (kv_heads > 1 ? kv_heads : 1) * rep;
  return heads < p.BH ? static_cast<int>(heads) : p.BH;
}

// Sizes and pointers that both entry points of the attention kernel ask for.
int check_attention(const void* q, const void* k, const void* v, const void* out, const int64_t* out_strides, int dtype, int64_t B,
                           int64_t Hq, int64_t Hkv, int64_t Sq, int64_t Sk, int64_t D, float softmax_scale) {
  if (B < 0 || Hq <= 0 || Hkv <= 0 || Hq % Hkv != 0 || Sq < 0 || Sk < 0 || D <= 0 || D > 128 || D % 16 != 0) return B200Q_ERR_INVALID;
  if (B * Hq > 65535 || Sq > 0x7fffffffLL || Sk > 0x7fffffffLL) return B200Q_ERR_INVALID;
  if (dtype != B200Q_BF16 && dtype != B200Q_F16 && dtype != B200Q_F32) return B200Q_ERR_INVALID;
  if (!(softmax_scale > 0.0f)) return B200Q_ERR_INVALID;
  if (B == 0 || Sq == 0) return B200Q_OK;
  if (q == nullptr || out == nullptr) return B200Q_ERR_INVALID;
  if (Sk > 0 && (k == nullptr || v == nullptr)) return B200Q_ERR_INVALID;
  if (!aligned(q, 16) || !aligned(k, 16) || !aligned(v, 16) || !aligned(out, 32)) return B200Q_ERR_ALIGN;
  if (out_strides == nullptr) return B200Q_ERR_INVALID;
  for (int i = 0; i < 3; ++i)
    if (out_strides[i] < 0 || out_strides[i] % 8 != 0) return B200Q_ERR_ALIGN;   // 8-element stores
  return B200Q_OK;
}

// Under a programmatic launch CTAs are placed while the kernel in front still holds SMs: two on an SM that is free, none on one that is
// free a little later.  With no more CTAs than SMs each therefore asks for so much shared memory that it has its SM alone.  With up to
// two per SM and causal, where the longest query tiles start first so as to share an SM with short ones, the launch is a plain one.
// Otherwise the fullest SM has two either way, and calls of up to five key tiles gain more from the early start.  Whole calls in a
// graph, us, three operands and a plain launch / programmatic as it comes / this rule: bf16 [1, 4, 4096, 128] 72.7 / 93.7 / 58.6, [1, 16 / 4,
// 909, 64] 24.4 / 28.1 / 20.3; causal [1, 16 / 4, 2048, 128] 46.4 / 50.0 / 39.5, fp16 [1, 15 / 5, 1300, 128] 32.2 / 36.8 / 28.4.  Over 900
// shapes never slower than the first (0.96 at most; programmatic as it comes 1.55), up to 1.08 of the second where that happens to
// spread ([4, 5, 1000, 64] causal 26.9 / 21.4 / 22.8).
template <typename QT, bool WIDE, bool FREE>
int launch_sdpa_form(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const AttParams& p, unsigned ctas, bool behind,
                          cudaStream_t st) {
  const unsigned sms = static_cast<unsigned>(sm_count());
  const int smem = behind && ctas <= sms ? kAttSmemAlone : kAttSmem;
  if (ctas > sms && ctas <= 2 * sms && p.causal && p.Sk > 5 * kTile) behind = false;
  static bool configured[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return B200Q_ERR_CUDA;
  if (!configured[dev]) {
    if (cudaFuncSetAttribute(fp8_sdpa_kernel<QT, WIDE, FREE>, cudaFuncAttributeMaxDynamicSharedMemorySize, kAttSmemAlone) != cudaSuccess) return B200Q_ERR_CUDA;
    configured[dev] = true;
  }
  if (behind) {
    if (launch_pdl(fp8_sdpa_kernel<QT, WIDE, FREE>, dim3(ctas), dim3(kAttThreads), smem, st, tq, tk, tv, p) != cudaSuccess) return B200Q_ERR_CUDA;
  } else {
    fp8_sdpa_kernel<QT, WIDE, FREE><<<ctas, kAttThreads, smem, st>>>(tq, tk, tv, p);
  }
  return check_launch();
}

// p: scales, queries (q_amax == nullptr: codes, at `q_codes`) and the result filled in.  `behind`: the kernel that writes the K and
// V operands was launched directly in front.
int launch_sdpa(AttParams& p, const uint8_t* q_codes, const uint8_t* k_codes, const uint8_t* vt_codes, const int64_t* out_strides,
                       int q_dtype, int64_t B, int64_t Hq, int64_t Hkv, int64_t Sq, int64_t Sk, int64_t vt_stride, int64_t D,
                       float softmax_scale, int causal, bool behind, b200q_stream_t stream) {
  p.out_sb = out_strides[0];
  p.out_sh = out_strides[1];
  p.out_ss = out_strides[2];
  p.status = gemm::device_status_word();
  if (p.status == nullptr) return B200Q_ERR_CUDA;
  const bool codes = p.q_amax == nullptr;
  CUtensorMap tq, tk, tv;
  // a zero-length key axis still needs valid maps: the kernel then loads nothing and writes zeros
  const int64_t sk_map = Sk > 0 ? Sk : 1;
  const void* any = codes ? static_cast<const void*>(q_codes) : p.q;
  const void* kbase = Sk > 0 ? static_cast<const void*>(k_codes) : any;
  const void* vbase = Sk > 0 ? static_cast<const void*>(vt_codes) : any;
  if (int rc = make_head_map(&tk, kbase, D, sk_map, B * Hkv, D)) return rc;
  if (int rc = make_head_map(&tv, vbase, Sk > 0 ? Sk : 16, D, B * Hkv, Sk > 0 ? vt_stride : 16)) return rc;
  if (codes) {
    if (int rc = make_head_map(&tq, q_codes, D, Sq, B * Hq, D)) return rc;
  } else {
    tq = tk;                                     // not read
  }
  p.Hq = static_cast<int>(Hq);
  p.Hkv = static_cast<int>(Hkv);
  p.Sq = static_cast<int>(Sq);
  p.Sk = static_cast<int>(Sk);
  p.D = static_cast<int>(D);
  p.softmax_scale = softmax_scale;
  p.causal = causal ? 1 : 0;
  p.BH = static_cast<int>(B * Hq);
  p.q_tiles = static_cast<int>((Sq + kTile - 1) / kTile);
  const int64_t ctas = static_cast<int64_t>(p.q_tiles) * p.BH;
  if (ctas > 0x7fffffffLL) return B200Q_ERR_INVALID;
  p.group = head_group(p);
  const unsigned n = static_cast<unsigned>(ctas);
  const auto st = static_cast<cudaStream_t>(stream);
  if (codes)
    return p.out_dtype == B200Q_BF16 ? launch_sdpa_form<uint8_t, true, true>(tq, tk, tv, p, n, behind, st)
                                     : launch_sdpa_form<uint8_t, true, false>(tq, tk, tv, p, n, behind, st);
  const int64_t unit = q_dtype == B200Q_F32 ? 8 : 16;
  const bool wide = aligned(p.q, 32) && p.q_sb % unit == 0 && p.q_sh % unit == 0 && p.q_ss % unit == 0;
  // queries and result have one type here
#define B200Q_SDPA(T, FREE) (wide ? launch_sdpa_form<T, true, FREE>(tq, tk, tv, p, n, behind, st) : launch_sdpa_form<T, false, FREE>(tq, tk, tv, p, n, behind, st))
  switch (q_dtype) {
    case B200Q_BF16: return B200Q_SDPA(__nv_bfloat16, true);
    case B200Q_F16: return B200Q_SDPA(__half, false);
    case B200Q_F32: return B200Q_SDPA(float, false);
    default: return B200Q_ERR_INVALID;
  }
#undef B200Q_SDPA
}

}  // namespace
}  // namespace b200q

using namespace b200q;

extern "C" {

int b200q_fp8_quantize_transpose(const void* x, int dtype, int64_t heads, int64_t S, int64_t D, const float* amax, uint8_t* out_t,
                                 int64_t s_stride, float* scale_out, b200q_stream_t stream) {
  if (heads < 0 || S < 0 || D <= 0 || D > 128 || D % 16 != 0 || s_stride < S || s_stride % 16 != 0 || heads > 65535) return B200Q_ERR_INVALID;
  if (heads == 0 || S == 0) return B200Q_OK;
  if (x == nullptr || amax == nullptr || out_t == nullptr) return B200Q_ERR_INVALID;
  if (!aligned(x, 16) || !aligned(out_t, 16) || (dtype == B200Q_F32 && !aligned(x, 32))) return B200Q_ERR_ALIGN;
  if (int rc = check_arch()) return rc;
  if (dtype != B200Q_BF16 && dtype != B200Q_F16 && dtype != B200Q_F32) return B200Q_ERR_INVALID;
  if (s_stride > 0x7fffff00LL) return B200Q_ERR_INVALID;
  QkvParts p{};
  p.D = static_cast<int>(D);
  p.vt_stride = s_stride;
  p.part[0].H = p.part[1].H = 1;
  p.part[2] = QkvPart{x, S * D, 0, D, amax, out_t, scale_out, 1, static_cast<int>(S), 0};
  return launch_attention_quantize(p, static_cast<int>(heads), dtype, static_cast<cudaStream_t>(stream));
}

// Host-side check of one strided input of b200q_fp8_attention_quantize.
static int check_strided(const void* x, const int64_t* strides, int dtype) {
  const int64_t unit = dtype == B200Q_F32 ? 4 : 8;     // elements in 16 bytes
  if (x == nullptr) return B200Q_ERR_INVALID;
  if (!aligned(x, 16)) return B200Q_ERR_ALIGN;
  for (int i = 0; i < 3; ++i)
    if (strides[i] < 0 || strides[i] % unit != 0) return B200Q_ERR_ALIGN;
  return B200Q_OK;
}

int b200q_fp8_attention_quantize(const void* q, const void* k, const void* v, int dtype, const int64_t* strides, const float* amax_q,
                                 const float* amax_k, const float* amax_v, uint8_t* q_codes, uint8_t* k_codes, uint8_t* vt_codes,
                                 float* scales, int64_t B, int64_t Hq, int64_t Hkv, int64_t Sq, int64_t Sk, int64_t vt_stride, int64_t D,
                                 b200q_stream_t stream) {
  if (B < 0 || Hq <= 0 || Hkv <= 0 || Sq < 0 || Sk < 0 || D <= 0 || D > 128 || D % 16 != 0) return B200Q_ERR_INVALID;
  if (vt_stride < Sk || vt_stride % 16 != 0 || vt_stride > 0x7fffff00LL || B > 0x7fffffffLL || Hq > 0x7fffffffLL || Hkv > 0x7fffffffLL || Sq > 0x7fffff00LL || Sk > 0x7fffff00LL)
    return B200Q_ERR_INVALID;
  if (dtype != B200Q_BF16 && dtype != B200Q_F16 && dtype != B200Q_F32) return B200Q_ERR_INVALID;
  if (B == 0 || (Sq == 0 && Sk == 0)) return B200Q_OK;
  if (strides == nullptr || amax_q == nullptr || amax_k == nullptr || amax_v == nullptr || scales == nullptr) return B200Q_ERR_INVALID;
  if (Sq > 0) {
    if (int rc = check_strided(q, strides, dtype)) return rc;
    if (q_codes == nullptr) return B200Q_ERR_INVALID;
  }
  if (Sk > 0) {
    if (int rc = check_strided(k, strides + 3, dtype)) return rc;
    if (int rc = check_strided(v, strides + 6, dtype)) return rc;
    if (k_codes == nullptr || vt_codes == nullptr) return B200Q_ERR_INVALID;
  }
  if (!aligned(q_codes, 16) || !aligned(k_codes, 16) || !aligned(vt_codes, 16)) return B200Q_ERR_ALIGN;
  if (int rc = check_arch()) return rc;
  QkvParts p{};
  p.D = static_cast<int>(D);
  p.vt_stride = vt_stride;
  p.part[0] = QkvPart{q, strides[0], strides[1], strides[2], amax_q, q_codes, scales, static_cast<int>(Hq), static_cast<int>(Sq), 0};
  p.part[1] = QkvPart{k, strides[3], strides[4], strides[5], amax_k, k_codes, scales + 1, static_cast<int>(Hkv), static_cast<int>(Sk), 0};
  p.part[2] = QkvPart{v, strides[6], strides[7], strides[8], amax_v, vt_codes, scales + 2, static_cast<int>(Hkv), static_cast<int>(Sk), 0};
  return launch_attention_quantize(p, static_cast<int>(B), dtype, static_cast<cudaStream_t>(stream));
}

int b200q_fp8_sdpa(const uint8_t* q_codes, const uint8_t* k_codes, const uint8_t* vt_codes, const float* q_scale, const float* k_scale,
                   const float* v_scale, void* out, int out_dtype, int64_t B, int64_t Hq, int64_t Hkv, int64_t Sq, int64_t Sk,
                   int64_t vt_stride, int64_t D, float softmax_scale, int causal, b200q_stream_t stream) {
  const int64_t strides[3] = {Hq * Sq * D, Sq * D, D};
  return b200q_fp8_sdpa_strided(q_codes, k_codes, vt_codes, q_scale, k_scale, v_scale, out, strides, out_dtype, B, Hq, Hkv, Sq, Sk, vt_stride,
                                D, softmax_scale, causal, stream);
}

int b200q_fp8_sdpa_strided(const uint8_t* q_codes, const uint8_t* k_codes, const uint8_t* vt_codes, const float* q_scale,
                           const float* k_scale, const float* v_scale, void* out, const int64_t* out_strides, int out_dtype, int64_t B,
                           int64_t Hq, int64_t Hkv, int64_t Sq, int64_t Sk, int64_t vt_stride, int64_t D, float softmax_scale, int causal,
                           b200q_stream_t stream) {
  if (vt_stride < Sk || vt_stride % 16 != 0) return B200Q_ERR_INVALID;
  if (int rc = check_attention(q_codes, k_codes, vt_codes, out, out_strides, out_dtype, B, Hq, Hkv, Sq, Sk, D, softmax_scale)) return rc;
  if (B == 0 || Sq == 0) return B200Q_OK;
  if (q_scale == nullptr || k_scale == nullptr || v_scale == nullptr) return B200Q_ERR_INVALID;
  if (int rc = check_arch()) return rc;
  AttParams p{};
  p.q_scale = q_scale;
  p.k_scale = k_scale;
  p.v_scale = v_scale;
  p.out = out;
  p.out_dtype = out_dtype;
  return launch_sdpa(p, q_codes, k_codes, vt_codes, out_strides, out_dtype, B, Hq, Hkv, Sq, Sk, vt_stride, D, softmax_scale, causal, false, stream);
}

static int64_t round16(int64_t n) { return (n + 15) / 16 * 16; }

size_t b200q_fp8_attention_workspace_bytes(int64_t B, int64_t Hkv, int64_t Sk, int64_t D) {
  if (B <= 0 || Hkv <= 0 || Sk < 0 || D <= 0) return 16;
  return static_cast<size_t>(B * Hkv * Sk * D + B * Hkv * D * round16(Sk) + 16);   // D is a multiple of 16
}

int b200q_fp8_attention(const void* q, const void* k, const void* v, int dtype, const int64_t* strides, const float* amax_q,
                        const float* amax_k, const float* amax_v, void* out, const int64_t* out_strides, void* workspace,
                        size_t workspace_bytes, int64_t B, int64_t Hq, int64_t Hkv, int64_t Sq, int64_t Sk, int64_t D, float softmax_scale,
                        int causal, b200q_stream_t stream) {
  if (int rc = check_attention(q, k, v, out, out_strides, dtype, B, Hq, Hkv, Sq, Sk, D, softmax_scale)) return rc;
  if (B == 0 || Sq == 0) return B200Q_OK;
  if (Sq > 0x7fffff00LL || Sk > 0x7fffff00LL || strides == nullptr || amax_q == nullptr || amax_k == nullptr || amax_v == nullptr)
    return B200Q_ERR_INVALID;
  if (workspace == nullptr || workspace_bytes < b200q_fp8_attention_workspace_bytes(B, Hkv, Sk, D)) return B200Q_ERR_INVALID;
  if (int rc = check_strided(q, strides, dtype)) return rc;
  if (!aligned(workspace, 16)) return B200Q_ERR_ALIGN;
  const int64_t vt_stride = round16(Sk);
  auto* k_codes = static_cast<uint8_t*>(workspace);
  uint8_t* vt_codes = k_codes + B * Hkv * Sk * D;
  auto* scales = reinterpret_cast<float*>(vt_codes + B * Hkv * D * vt_stride);
  if (Sk > 0) {
    if (int rc = b200q_fp8_attention_quantize(nullptr, k, v, dtype, strides, amax_q, amax_k, amax_v, nullptr, k_codes, vt_codes, scales, B, Hq, Hkv,
                                              0, Sk, vt_stride, D, stream))
      return rc;
  } else if (int rc = check_arch()) {
    return rc;
  }
  AttParams p{};
  p.q = q;
  p.q_amax = amax_q;
  p.q_sb = strides[0];
  p.q_sh = strides[1];
  p.q_ss = strides[2];
  p.k_scale = scales + 1;
  p.v_scale = scales + 2;
  p.out = out;
  p.out_dtype = dtype;
  return launch_sdpa(p, nullptr, k_codes, vt_codes, out_strides, dtype, B, Hq, Hkv, Sq, Sk, vt_stride, D, softmax_scale, causal, Sk > 0, stream);
}

}  // extern "C"
