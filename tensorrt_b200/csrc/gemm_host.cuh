// Host side of the tcgen05 GEMMs: TMA tensor maps, tile-shape choice, launch.
#pragma once

#include <cuda.h>

#include <algorithm>

#include "gemm_kernel_2cta.cuh"
#include "gemm_kernel_nvf4_pair.cuh"
#include "gemm_kernel_splitk.cuh"

namespace b200q {
namespace gemm {

using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                   const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                   CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// cuTensorMapEncodeTiled resolved through the runtime, so the library has no link-time
// dependency on libcuda.
EncodeTiledFn encode_tiled();

// Device status word shared by all GEMM launches of this process on the current device.
int* device_status_word();

// Row-major byte matrix [rows, row_bytes] -> tiles of box_rows x 128 bytes, 128-byte swizzle,
// out-of-bounds bytes read as zero.
inline int make_operand_map(CUtensorMap* map, const void* base, int64_t rows, int64_t row_bytes, int box_rows) {
  EncodeTiledFn fn = encode_tiled();
  if (fn == nullptr) return B200Q_ERR_CUDA;
  const cuuint64_t dims[2] = {static_cast<cuuint64_t>(row_bytes), static_cast<cuuint64_t>(rows)};
  const cuuint64_t strides[1] = {static_cast<cuuint64_t>(row_bytes)};
  const cuuint32_t box[2] = {static_cast<cuuint32_t>(kBKBytes), static_cast<cuuint32_t>(box_rows)};
  const cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? B200Q_OK : B200Q_ERR_CUDA;
}

// bf16 output [M, N] -> boxes of 32 rows x 64 columns (128 bytes), 128-byte swizzle.
inline int make_output_map(CUtensorMap* map, const void* base, int64_t M, int64_t N) {
  EncodeTiledFn fn = encode_tiled();
  if (fn == nullptr) return B200Q_ERR_CUDA;
  const cuuint64_t dims[2] = {static_cast<cuuint64_t>(N), static_cast<cuuint64_t>(M)};
  const cuuint64_t strides[1] = {static_cast<cuuint64_t>(N) * 2};
  const cuuint32_t box[2] = {64, 32};
  const cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? B200Q_OK : B200Q_ERR_CUDA;
}

// Receive buffers of the reduce-scatter epilogue: recv[r] is rank r's buffer
// [world][rows_per_rank][N] bf16, mapped into this process (peer memory).
struct RsTargets {
  void* recv[8];
};

// Output maps of a launch: the local output, or one map per destination rank.
inline int build_out_maps(OutMaps* maps, Params& p, const RsTargets* rs) {
  p.tma_store = (p.N % 8 == 0) ? 1 : 0;
  if (p.rs_world > 1) {
    if (rs == nullptr || !p.tma_store || p.rs_world > 8 || p.rs_rows % 128 != 0 || p.rs_rows * p.rs_world != p.M)
      return B200Q_ERR_INVALID;
    for (int r = 0; r < p.rs_world; ++r)
      if (int rc = make_output_map(&maps->m[r], rs->recv[r], static_cast<int64_t>(p.rs_world) * p.rs_rows, p.N)) return rc;
    return B200Q_OK;
  }
  if (p.tma_store) return make_output_map(&maps->m[0], p.out, p.M, p.N);
  return B200Q_OK;
}

template <bool NVF4, int BN>
int launch_tile(const uint8_t* a, const uint8_t* b, Params p, cudaStream_t st, const RsTargets* rs = nullptr) {
  using C = Cfg<NVF4, BN>;
  static bool configured[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return B200Q_ERR_CUDA;
  if (!configured[dev]) {
    if (cudaFuncSetAttribute(gemm_kernel<NVF4, BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmemBytes) != cudaSuccess)
      return B200Q_ERR_CUDA;
    configured[dev] = true;
  }
  CUtensorMap ta, tb;
  OutMaps tout = {};
  if (int rc = make_operand_map(&ta, a, p.M, p.k_bytes, kBM)) return rc;
  if (int rc = make_operand_map(&tb, b, p.N, p.k_bytes, BN)) return rc;
  if (int rc = build_out_maps(&tout, p, rs)) return rc;
  const int tiles = ((p.M + kBM - 1) / kBM) * ((p.N + BN - 1) / BN);
  const int grid = tiles < sm_count() ? tiles : sm_count();
  const int threads = (NVF4 && p.sf_copier) ? kThreads + 32 : kThreads;   // optional scale-copier warp
  gemm_kernel<NVF4, BN><<<grid, threads, C::kSmemBytes, st>>>(ta, tb, tout, p);
  return check_launch();
}

// Swizzled block-scale buffer as a 3-D tensor [128 u32 = one 512-byte tile, column tile, row tile].
inline int make_scale_map(CUtensorMap* map, const void* base, int64_t row_tiles, int64_t col_tiles, int box_row_tiles) {
  EncodeTiledFn fn = encode_tiled();
  if (fn == nullptr) return B200Q_ERR_CUDA;
  const cuuint64_t dims[3] = {128, static_cast<cuuint64_t>(col_tiles), static_cast<cuuint64_t>(row_tiles)};
  const cuuint64_t strides[2] = {512, static_cast<cuuint64_t>(col_tiles) * 512};
  const cuuint32_t box[3] = {128, 4, static_cast<cuuint32_t>(box_row_tiles)};
  const cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT32, 3, const_cast<void*>(base), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? B200Q_OK : B200Q_ERR_CUDA;
}

// CTA-pair kernel: clusters of two CTAs, one cluster per 256 x 256 output tile.
template <bool NVF4, int SILU = 0, int BN = kPairN>
int launch_pair(const uint8_t* a, const uint8_t* b, Params p, cudaStream_t st, const RsTargets* rs = nullptr) {
  using C = Cfg2<NVF4, BN>;
  static bool configured[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return B200Q_ERR_CUDA;
  if (!configured[dev]) {
    if (cudaFuncSetAttribute(gemm_pair_kernel<NVF4, SILU, BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmemBytes) != cudaSuccess)
      return B200Q_ERR_CUDA;
    configured[dev] = true;
  }
  CUtensorMap ta, tb, tsfa, tsfb;
  OutMaps tout = {};
  if (int rc = make_operand_map(&ta, a, p.M, p.k_bytes, 128)) return rc;
  if (int rc = make_operand_map(&tb, b, p.N, p.k_bytes, BN / 2)) return rc;
  if constexpr (SILU == 2) {
    // E4M3 codes [M, F] leave through plain stores: no output map
    p.tma_store = 0;
    if (rs != nullptr || p.rs_world > 1) return B200Q_ERR_INVALID;
  } else if constexpr (SILU == 1) {
    // out is [M, F]: TMA stores only (F is a multiple of 128)
    p.tma_store = 1;
    if (rs != nullptr || p.rs_world > 1) return B200Q_ERR_INVALID;
    if (int rc = make_output_map(&tout.m[0], p.out, p.M, p.silu_f)) return rc;
  } else {
    if (int rc = build_out_maps(&tout, p, rs)) return rc;
  }
  if constexpr (NVF4) {
    if (int rc = make_scale_map(&tsfa, p.sfa, (p.M + 127) / 128, p.sf_col_tiles, 1)) return rc;
    if (int rc = make_scale_map(&tsfb, p.sfb, (p.N + 127) / 128, p.sf_col_tiles, 2)) return rc;
  } else {
    tsfa = ta;
    tsfb = ta;
  }
  const int tiles = ((p.M + kPairM - 1) / kPairM) * (SILU ? (p.silu_f + BN / 2 - 1) / (BN / 2) : (p.N + BN - 1) / BN);
  const int max_pairs = sm_count() / 2;
  const int pairs = tiles < max_pairs ? tiles : max_pairs;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(pairs * 2));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = C::kSmemBytes;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (cudaLaunchKernelEx(&cfg, gemm_pair_kernel<NVF4, SILU, BN>, ta, tb, tout, tsfa, tsfb, p) != cudaSuccess) {
    cudaGetLastError();
    return B200Q_ERR_CUDA;
  }
  return B200Q_OK;
}

// NVFP4 CTA-pair kernel with the scales stored to tensor memory by warps (gemm_kernel_nvf4_pair.cuh).
template <bool SILU = false>
int launch_nvf4_pair(const uint8_t* a, const uint8_t* b, Params p, cudaStream_t st) {
  using C = CfgNvPair;
  static bool configured[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return B200Q_ERR_CUDA;
  if (!configured[dev]) {
    if (cudaFuncSetAttribute(gemm_nvf4_pair_kernel<SILU>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmemBytes) != cudaSuccess)
      return B200Q_ERR_CUDA;
    configured[dev] = true;
  }
  CUtensorMap ta, tb, tsfa, tsfb;
  if (int rc = make_operand_map(&ta, a, p.M, p.k_bytes, 128)) return rc;
  if (int rc = make_operand_map(&tb, b, p.N, p.k_bytes, 128)) return rc;
  if (int rc = make_scale_map(&tsfa, p.sfa, (p.M + 127) / 128, p.sf_col_tiles, 1)) return rc;
  if (int rc = make_scale_map(&tsfb, p.sfb, (p.N + 127) / 128, p.sf_col_tiles, SILU ? 1 : 2)) return rc;
  const int tiles = ((p.M + kPairM - 1) / kPairM) * ((p.N + kPairN - 1) / kPairN);   // SILU: N = 2 F, F / 128 tiles of columns
  const int max_pairs = sm_count() / 2;
  const int pairs = tiles < max_pairs ? tiles : max_pairs;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(pairs * 2));
  cfg.blockDim = dim3(kNvPairThreads);
  cfg.dynamicSmemBytes = C::kSmemBytes;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (cudaLaunchKernelEx(&cfg, gemm_nvf4_pair_kernel<SILU>, ta, tb, tsfa, tsfb, p) != cudaSuccess) {
    cudaGetLastError();
    return B200Q_ERR_CUDA;
  }
  return B200Q_OK;
}

// Dynamic shared memory that `kernel` may be launched with, set once per device (`configured`: one flag per device).
template <typename Kernel>
int allow_smem(Kernel* kernel, int bytes, bool* configured) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return B200Q_ERR_CUDA;
  if (!configured[dev]) {
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess) return B200Q_ERR_CUDA;
    configured[dev] = true;
  }
  return B200Q_OK;
}

// One launch of a small-M kernel: `tiles` clusters of `splits` CTAs.
template <typename Kernel>
int launch_clusters(Kernel* kernel, int tiles, int splits, int smem_bytes, cudaStream_t st, const CUtensorMap& tw, const CUtensorMap& tx,
                    const Params& p, int stages, int bt, int blocks) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(tiles * blocks * splits));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = static_cast<size_t>(smem_bytes);
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = static_cast<unsigned>(splits);
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;   // see common.cuh: pdl_wait in the kernel
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_enabled() ? 2 : 1;
  if (cudaLaunchKernelEx(&cfg, kernel, tw, tx, p, splits, stages, bt, blocks) != cudaSuccess) {
    cudaGetLastError();
    return B200Q_ERR_CUDA;
  }
  return B200Q_OK;
}

// Blocks of tokens of the small-M kernel.
inline int smallm_blocks(int M, bool nvf4) {
  const int most = nvf4 ? 128 : 256;
  return M <= 128 ? 1 : (M + most - 1) / most;
}

// Tokens of a block: a multiple of 16; NVFP4 in several blocks the 128 rows of a scale tile.
inline int smallm_block_tokens(int M, int blocks, bool nvf4) {
  return nvf4 && blocks > 1 ? 128 : ((M + blocks - 1) / blocks + 15) / 16 * 16;
}

// Small-M kernel: operands swapped, one cluster of `splits` CTAs per tile of 128 weight rows and block of tokens (one block of
// up to 128; above, FP8 blocks of up to 256, NVFP4 of 128).  Up to one CTA per SM the operand ring takes all of shared memory; beyond that
// the ring is sized so that two CTAs share an SM, which lets one CTA's prologue and cluster
// reduction overlap the other's weight stream and fits twice as many CTAs into a wave.
// `stages` > 0 overrides the ring depth.
template <bool NVF4, bool BLOCKS>
int launch_smallm(const uint8_t* a, const uint8_t* b, Params p, cudaStream_t st, int splits, int stages) {
  using C = SmallCfg<NVF4>;
  static bool configured[64] = {};
  if (int rc = allow_smem(gemm_smallm_kernel<NVF4, void, BLOCKS>, kSmemLimit, configured)) return rc;
  const int blocks = BLOCKS ? smallm_blocks(p.M, NVF4) : 1;
  const int bt = smallm_block_tokens(p.M, blocks, NVF4);
  const int tiles = (p.N + kSmallWRows - 1) / kSmallWRows;
  if (static_cast<int64_t>(tiles) * blocks * splits > 0x7fffffffLL) return B200Q_ERR_INVALID;
  const int most = C::max_stages(bt, kSmemLimit);
  if (stages <= 0) {
    stages = most;
    if (tiles * blocks * splits > sm_count() && C::max_stages(bt, kSmallHalfSmem) >= C::min_stages(bt)) {
      // two CTAs per SM: half of the SM's 228 KiB (1 KiB reserved per CTA) and, for NVFP4,
      // half of the 512 tensor-memory columns (128 accumulator + 32 scale columns per stage)
      stages = C::max_stages(bt, kSmallHalfSmem);
      if (NVF4 && stages > 4) stages = 4;
    }
  }
  if (stages > most) stages = most;
  if (stages < C::min_stages(bt)) stages = C::min_stages(bt);
  CUtensorMap tw, tx;
  if (int rc = make_operand_map(&tw, b, p.N, p.k_bytes, kSmallWRows)) return rc;
  if (int rc = make_operand_map(&tx, a, p.M, p.k_bytes, bt)) return rc;
  return launch_clusters(gemm_smallm_kernel<NVF4, void, BLOCKS>, tiles, splits, C::smem_bytes(bt, stages), st, tw, tx, p, stages, bt, blocks);
}

// The small-M kernel that quantizes its activation (FP8; p.x, p.x_amax set; limits kOwnXTiles, kOwnXSlice).
template <typename XT>
int launch_smallm_own_x(const uint8_t* b, const Params& p, cudaStream_t st, int splits, int tiles_per_cta) {
  const int stages = tiles_per_cta < 2 ? 2 : tiles_per_cta;      // the whole K slice at once
  constexpr int kMostBytes = 1024 + kSmallTailBytes + kOwnXTiles * (SmallCfg<false>::kWBytes + 2048);
  static_assert(kMostBytes <= kSmallHalfSmem, "two CTAs share an SM");
  const int bytes = 1024 + kSmallTailBytes + stages * SmallCfg<false>::kWBytes + tiles_per_cta * 2048;
  static bool configured[64] = {};
  if (int rc = allow_smem(gemm_smallm_kernel<false, XT>, kMostBytes, configured)) return rc;
  CUtensorMap tw;
  if (int rc = make_operand_map(&tw, b, p.N, p.k_bytes, kSmallWRows)) return rc;
  return launch_clusters(gemm_smallm_kernel<false, XT>, (p.N + kSmallWRows - 1) / kSmallWRows, splits, bytes, st, tw, tw, p, stages, 16, 1);
}

// Cluster size of the small-M kernel.  Measured: one SM pulls about 60 bytes per nanosecond
// through TMA whatever the ring depth, so about 110 streaming SMs are needed to saturate HBM;
// the smallest power of two that reaches that many CTAs wins, larger clusters only add
// reduction cost.  With at most 32 tokens the partial tiles are small enough that two CTAs per SM
// pay (one's prologue and cluster reduction under the other's weight stream: 10-25 % faster at
// 16 tokens, neutral at 64, slower at 128), so the target there is one and a half CTAs per SM, as long
// as all CTAs are resident at once: 80 tiles x 4 = 320 CTAs on 296 places cost a second round (10240 x 8192
// at 1 / 16 tokens: FP8 23.0 / 24.4 us against 17.4 / 18.4 with 2 CTAs per tile, NVFP4 16.2 / 17.6 against 12.4 / 13.2).
inline int smallm_most_splits(int n_tiles, int k_tiles, int sms, int tokens) {
  const int want = tokens <= 32 ? (sms * 3) / 2 : (sms * 3) / 4;
  int s = 1;
  while (s < 8 && n_tiles * s < want && n_tiles * s * 2 <= 2 * sms && s * 2 <= k_tiles) s <<= 1;
  return s;
}

// Clusters of 2, 4 or 8 CTAs, one per SM, that are resident at once on the current device.  A cluster does not cross a GPC, and
// how many SMs a GPC has differs from part to part, so the occupancy API is asked, once per device.  `sms`: SMs of the device.
struct ActiveClusters {
  int sms, of2, of4, of8;
};
ActiveClusters active_clusters(int sms);

// Clusters of `s` CTAs of a small-M kernel that are resident at once, two CTAs per SM where `shared_sm`.  Seen as the jump to a
// second round on a part where the API gives 74, 33 and 15 clusters of 2, 4 and 8 (FP8 at 16 tokens, K 4096): alone 15 of 8
// (5.98 us, 16 take 10.2) and 33 of 4 (8.1, 34 take 12.3); two CTAs per SM have the places of clusters of half the size: 33 of 8
// (7.3, 34 take 11.3), 148 of 2 (14.9, 149 take 21.1), and of 4 nearly, 71 (9.4, 72 take 14.1).
inline int smallm_resident(int s, const ActiveClusters& c, bool shared_sm) {
  if (!shared_sm) return s == 1 ? c.sms : (s == 2 ? c.of2 : (s == 4 ? c.of4 : c.of8));
  return s == 1 ? 2 * c.sms : (s == 2 ? c.sms : (s == 4 ? (c.of2 * 71 + 73) / 74 : c.of4));
}

// Time of the small-M kernel with clusters of `s` CTAs in ns, good enough to compare cluster sizes: a launch, the K tiles of a
// CTA, and what the cluster adds (every token's partial sums, twice from eight CTAs); dearer where CTAs share an SM; once more
// for every further round of clusters.  Clusters of eight count as one round up to four fifths of those that fit: with 13 to 15
// tiles clusters of four take 0.87 to 0.97 of their time (NVFP4 1920 x 2048 at 8 tokens 4.5 us against 5.1, FP8 1920 x 4096 at 64
// tokens 7.65 against 8.4; only 1664 x 4096 at one token is 2 % slower).
inline int64_t smallm_cost(int n_tiles, int k_tiles, const ActiveClusters& c, int tokens, int s) {
  const bool shared_sm = n_tiles * s > c.sms;
  const int log2s = s == 1 ? 0 : (s == 2 ? 1 : (s == 4 ? 2 : 3));
  int resident = smallm_resident(s, c, shared_sm);
  if (s == 8 && !shared_sm) resident = (resident * 4 + 4) / 5;
  const int64_t rounds = (n_tiles + resident - 1) / resident, per = (k_tiles + s - 1) / s;
  const int64_t stream = per * (1800 + 3 * tokens) * (shared_sm ? 13 : 10) / 100;
  const int64_t reduce = tokens * 3 * log2s * (shared_sm ? 3 : 1) + (s == 8 ? 9 * tokens : 0);
  return rounds * (4900 + stream) + reduce;
}

// Fewer CTAs per tile than that where they are cheaper by more than 3 %: short K slices and many tokens (the reduction), and
// cluster counts just above what is resident.  Measured at 37 weight shapes (1024 x 1024 to 57344 x 8192), 10 token counts and
// both formats: 1.011 of the best cluster size's time on average (1.170 without this step, 2.3 times at worst: FP8 2048 x 2048
// at 16 / 64 / 128 tokens 9.1 / 13.5 / 17.9 us on 8 CTAs, 5.0 / 6.7 / 8.7 on 4; 6144 x 4096 at 128 tokens 16.3 on 4, 12.3 on
// 2), and nowhere more than 2 % slower than without.  At worst 1.23 of the best: FP8 5120 x 5120 at 96 tokens 14.8 us on 4
// CTAs, 12.1 on 2; 4096 x 1024 in both formats 1.08 to 1.21, where 2 CTAs would win at every token count.
inline int smallm_splits(int n_tiles, int k_tiles, int sms, int tokens) {
  const int most = smallm_most_splits(n_tiles, k_tiles, sms, tokens);
  if (most == 1) return 1;
  const ActiveClusters clusters = active_clusters(sms);
  const int64_t cost = smallm_cost(n_tiles, k_tiles, clusters, tokens, most);
  int best = most;
  int64_t least = cost * 97 / 100;
  for (int s = most >> 1; s >= 1; s >>= 1) {
    const int64_t c = smallm_cost(n_tiles, k_tiles, clusters, tokens, s);
    if (c < least) least = c, best = s;
  }
  return best;
}

bool valid_tile_n(int bn);    // values b200q_cfg::tile_n accepts
int sf_copier_enabled();     // environment variable B200Q_SF_COPIER (default in gemm_fp8.cu)
int forced_smallm_stages();  // from the environment variable B200Q_SMALLM_STAGES (0 when unset)

// Kernel of a problem with more than 128 rows: 512 / 448 = CTA pair with 256 x 256 / 256 x 192 tiles, 256 / 128 = one CTA with 128 x 256 /
// 128 x 128 tiles.  A launch takes as long as its rounds: tiles over SMs (SM pairs), rounded up, times the time of one
// tile, in units of a pair's 256 x 256 tile.  Large problems (many rounds) go to the pair kernels; a problem just above
// a whole number of rounds, or with few rows, to the finer tiles (333 x 10240 x 8192 FP8: 80 pair tiles on 74 pairs are
// two rounds, 48.0 us; 120 tiles of 128 x 256 are one, 32.6).  A single round of the small tile is not half of the big one's:
// both wait for the same K loop.  The percentages are from a sweep of the three kernels over 14 row counts (129 to 4096)
// and seven weight shapes in each format.  Over these 196 points the rule takes 1.003 of the fastest kernel's time on
// average; at worst 1.09, FP8 with K = 4096 and a single round of either tile, where 128 x 256 would win (4096 x 4096 at 600
// rows 17.7 us against 16.3; at K = 14336 the pair does, 42.9 against 47.5).  The choice by tile counts before it was 14 %
// slower on average and 2.2 times at worst (NVFP4 4096 x 14336 at 600 to 1000 rows: 48 to 64 pair tiles, 57 to 59 us on
// 128 x 128 tiles, 28.7 to 29.3 on pairs).  The reduce-scatter epilogue keeps the choice by tile counts that its NVLink
// overlap was measured with.
// FP8 pairs also take tiles of 256 x 192, 0.88 of the time of the wide ones: where rounds of those are cheaper, 0.99 of the time
// on average over 295 points (18 weight shapes, 129 to 6000 rows), 0.88 at best and nowhere more: 10240 x 8192 at 200 rows 30.6 ->
// 27.4 us, at 512 49.9 -> 44.9; 20480 x 5120 at 256 38.2 -> 33.8; 8192 x 28672 at 600 168.8 -> 148.2.  (Tiles of 256 x 128, 0.83,
// are never the best by more than 1 %.)
constexpr int kTile256Fp8 = 110, kTile128Fp8 = 85, kTile192Pair = 90, kTile256Nv = 145, kTile128Nv = 110;   // per cent of a pair tile
inline int large_tile(int M, int N, int sms, bool nvf4, bool rs) {
  const int64_t pair = static_cast<int64_t>((M + kPairM - 1) / kPairM) * ((N + kPairN - 1) / kPairN);
  const int64_t t256 = static_cast<int64_t>((M + kBM - 1) / kBM) * ((N + 255) / 256);
  const int64_t t128 = static_cast<int64_t>((M + kBM - 1) / kBM) * ((N + 127) / 128);
  if (rs) {
    if (!nvf4 && pair >= sms / 2) return 512;
    return t256 >= sms ? 256 : 128;
  }
  const auto cost = [](int64_t tiles, int units, int each) { return (tiles + units - 1) / units * each; };
  const int64_t c512 = cost(pair, sms / 2, 100), c256 = cost(t256, sms, nvf4 ? kTile256Nv : kTile256Fp8),
                c128 = cost(t128, sms, nvf4 ? kTile128Nv : kTile128Fp8);
  if (!nvf4) {
    const int64_t pair192 = static_cast<int64_t>((M + kPairM - 1) / kPairM) * ((N + 191) / 192), c448 = cost(pair192, sms / 2, kTile192Pair);
    if (c448 < c512 && c448 < c256 && c448 < c128) return 448;
  }
  if (c512 <= c256 && c512 <= c128) return 512;
  return c256 <= c128 ? 256 : 128;
}

// Above 128 rows: cluster size of the small-M kernel over blocks of tokens, 0 = the tile kernel that `large_tile` takes.  With few
// weight rows and some hundred tokens the tiles leave SMs idle, each of which walks all of K (4096 x 14336 FP8 at 129 to 512 rows:
// 64 to 128 tiles of 128 x 128, 112 K tiles of 0.28 us each); blocks of tokens whose K is split over a cluster use them.  Both sides
// are estimated in ns from a sweep of all kernels over 12 weight shapes and 129 to 1024 rows in each format (180 points, standard
// deviation 3 to 6 %): the tile kernels as rounds times (start + K tiles), the small-M kernel as K tiles of a CTA, the parked
// partial tile (every token, more the larger the cluster) and the traffic of all clusters together; only where all clusters are
// resident at once, one CTA per SM (asked of the kernel for one block, which fills an SM as well).  Taken where it is cheaper by 3 %
// and by 1 us (NVFP4 1.6): a launch of clusters behind a quantize kernel costs more than one of tiles.  Whole calls in a graph, 1530
// sizes where this holds (129 to 4000 rows): FP8 0.75 of the time on average, 2 of 808 slower by 2.5 to 2.8 %; NVFP4 0.83, none of 722
// by more than 1 %.  With 3 % alone, 73 more FP8 sizes, 0.90 to 1.08 of the time, and 370 more NVFP4 sizes, 0.89 to 1.12.  It leaves
// points behind: FP8 4096 x 4096 at 333 rows 14.3 us on tiles, 13.3 on clusters of two.  FP8, the GEMM alone, us, tile kernel / this:
// 4096 x 14336 at 129 rows 35.6 / 19.2, at 256 35.6 / 25.2, at 384 36.2 / 26.7; 2048 x 8192 at 256 22.2 / 17.3; 8192 x 28672 at 129 69.2
// / 48.6; 4096 x 4096 at 129 14.0 / 11.4; NVFP4 4096 x 14336 at 256 27.4 / 20.0.
constexpr int64_t kBlocksGainFp8 = 1000, kBlocksGainNv = 1600;   // ns
inline int block_splits(int M, int N, int k_tiles, int sms, bool nvf4, int tile) {
  const int blocks = smallm_blocks(M, nvf4), n_tiles = (N + kSmallWRows - 1) / kSmallWRows;
  const int64_t clusters = static_cast<int64_t>(n_tiles) * blocks;
  if (clusters > sms) return 0;
  const bool pairs = tile == 512 || tile == 448;
  const int bm = pairs ? kPairM : kBM, bn = tile == 128 ? 128 : (tile == 448 ? 192 : 256), units = pairs ? sms / 2 : sms;
  const int64_t tiles = static_cast<int64_t>((M + bm - 1) / bm) * ((N + bn - 1) / bn), rounds = (tiles + units - 1) / units;
  int64_t least;
  if (nvf4) {
    least = tile == 512 ? 4490 + rounds * (1840 + 394 * k_tiles)
                        : (tile == 256 ? 3290 + rounds * (2550 + 684 * k_tiles) : 4480 + rounds * (290 + 484 * k_tiles));
  } else {
    least = tile == 512   ? 5000 + rounds * (1770 + 334 * k_tiles)
            : tile == 448 ? 5000 + rounds * (1300 + 300 * k_tiles)
                          : (tile == 256 ? 3600 + rounds * (1640 + 391 * k_tiles) : 4100 + rounds * (510 + 289 * k_tiles));
  }
  least = std::min(least * 97 / 100, least - (nvf4 ? kBlocksGainNv : kBlocksGainFp8));
  const int64_t bt = smallm_block_tokens(M, blocks, nvf4);
  const ActiveClusters active = active_clusters(sms);
  int best = 0;
  for (int s = 1, log2s = 0; s <= 8 && s <= k_tiles; s <<= 1, ++log2s) {
    if (clusters * s > sms || clusters > smallm_resident(s, active, false)) break;
    const int64_t per = (k_tiles + s - 1) / s, all = clusters * s * per;
    const int64_t cost = nvf4 ? 6260 + per * 390 + 620 * log2s + all * 66 / 100
                              : 3500 + per * (180 + bt * 48 / 100) + bt * (18 + 6 * log2s + (s == 8 ? 4 : 0)) + all * 77 / 100;
    if (cost < least) least = cost, best = s;
  }
  return best;
}

// `cfg->tile_n` (128 / 256 / 448 / 512; up to 128 rows 1001 to 1008) overrides the choice of kernel (used by tests to cover the
// instantiations).  M <= 128 goes to the small-M kernel unless a tile width is forced.
template <bool NVF4>
int launch(const uint8_t* a, const uint8_t* b, Params p, cudaStream_t st, const b200q_cfg* cfg, const RsTargets* rs = nullptr) {
  p.status = device_status_word();
  if (p.status == nullptr) return B200Q_ERR_CUDA;
  p.sf_copier = NVF4 ? sf_copier_enabled() : 0;
  p.static_weights = (cfg != nullptr && cfg->static_weights != 0) ? 1 : 0;
  int bn = cfg != nullptr ? cfg->tile_n : 0;
  // A cluster size forced for a decode step must not reach the prompt passes of the same program: FP8 2048 x 8192 at 512 rows 22.4 us
  // on tiles, 48.0 on clusters of eight.
  if (bn > 1000 && p.M > kBM) bn = 0;
  const int k_tiles = (p.k_bytes + kBKBytes - 1) / kBKBytes;
  const int tile = p.M > kBM || rs != nullptr ? large_tile(p.M, p.N, sm_count(), NVF4, rs != nullptr) : 0;
  if (rs == nullptr) {
    // small M: weights are streamed once; the swapped-operand cluster kernel handles it
    // (1001 / 1002 / 1004 / 1008 force 1 / 2 / 4 / 8 CTAs per tile)
    int splits = 0;
    if (bn == 1001 || bn == 1002 || bn == 1004 || bn == 1008) splits = bn - 1000;
    else if (bn == 0 && p.M <= kBM) splits = smallm_splits((p.N + kSmallWRows - 1) / kSmallWRows, k_tiles, sm_count(), p.M);
    else if (bn == 0) splits = block_splits(p.M, p.N, k_tiles, sm_count(), NVF4, tile);
    if (splits >= 1 && splits <= k_tiles)
      return p.M <= kBM ? launch_smallm<NVF4, false>(a, b, p, st, splits, forced_smallm_stages())
                        : launch_smallm<NVF4, true>(a, b, p, st, splits, forced_smallm_stages());
  }
  if (bn >= 1000) bn = 0;
  if (bn == 0) bn = tile != 0 ? tile : large_tile(p.M, p.N, sm_count(), NVF4, false);
  // The NVFP4 pair kernel with the scale warps writes local output only; the reduce-scatter epilogue keeps the
  // generic kernels.
  if constexpr (!NVF4) {
    if (bn == 448) return launch_pair<false, 0, 192>(a, b, p, st, rs);
  }
  if (bn == 512 || bn == 448) {
    if constexpr (NVF4) {
      if (rs == nullptr) return launch_nvf4_pair(a, b, p, st);
      return launch_pair<NVF4>(a, b, p, st, rs);
    } else {
      return launch_pair<NVF4>(a, b, p, st, rs);
    }
  }
  return bn == 256 ? launch_tile<NVF4, 256>(a, b, p, st, rs) : launch_tile<NVF4, 128>(a, b, p, st, rs);
}

}  // namespace gemm
}  // namespace b200q
