// FP8 E4M3 x E4M3 GEMM entry point (tcgen05 kind::f8f6f4) and the pieces shared by both
// quantized GEMMs: the TMA descriptor encoder lookup and the device status word.
#include <atomic>
#include <cstdlib>
#include <mutex>

#include "gemm_host.cuh"
#include "internal.h"

namespace b200q {
namespace gemm {

namespace {
__device__ int g_device_status = 0;
std::mutex g_mu;
int* g_status_addr[64] = {};
}  // namespace

EncodeTiledFn encode_tiled() {
  static EncodeTiledFn fn = []() -> EncodeTiledFn {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess)
      return nullptr;
    return reinterpret_cast<EncodeTiledFn>(p);
  }();
  return fn;
}

int* device_status_word() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
  std::lock_guard<std::mutex> lk(g_mu);
  if (g_status_addr[dev] == nullptr) {
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_device_status) != cudaSuccess) return nullptr;
    g_status_addr[dev] = static_cast<int*>(p);
  }
  return g_status_addr[dev];
}

namespace {
int ask_active_clusters(int size, int sms) {
  using C = SmallCfg<false>;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(size * sms));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = static_cast<size_t>(C::smem_bytes(16, C::max_stages(16, kSmemLimit)));
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = static_cast<unsigned>(size);
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaFuncSetAttribute(gemm_smallm_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemLimit) != cudaSuccess ||
      cudaOccupancyMaxActiveClusters(&n, gemm_smallm_kernel<false>, &cfg) != cudaSuccess || n <= 0) {
    cudaGetLastError();
    n = sms > size ? sms / size : 1;                       // as if no GPC had SMs left over
  }
  return n;
}
}  // namespace

ActiveClusters active_clusters(int sms) {
  static std::atomic<uint64_t> known[64] = {};             // by device: three counts of 16 bits, 0 = not asked yet
  int dev = 0;
  const bool keep = cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < 64;
  uint64_t v = keep ? known[dev].load(std::memory_order_relaxed) : 0u;
  if (v == 0) {
    for (int size = 8; size >= 2; size >>= 1) v = v << 16 | static_cast<uint64_t>(ask_active_clusters(size, sms));
    if (keep) known[dev].store(v, std::memory_order_relaxed);
  }
  return {sms, static_cast<int>(v & 0xffffu), static_cast<int>(v >> 16 & 0xffffu), static_cast<int>(v >> 32)};
}

bool valid_tile_n(int bn) {
  return bn == 0 || bn == 128 || bn == 256 || bn == 448 || bn == 512 || bn == 1001 || bn == 1002 || bn == 1004 || bn == 1008;
}

int sf_copier_enabled() {
  static const int v = [] {
    const char* e = std::getenv("B200Q_SF_COPIER");   // measured 3-4 % faster with the copier warp: on unless set to 0
    return e != nullptr ? std::atoi(e) : 1;
  }();
  return v;
}

int forced_smallm_stages() {
  static const int v = [] {
    const char* e = std::getenv("B200Q_SMALLM_STAGES");
    return e != nullptr ? std::atoi(e) : 0;
  }();
  return v;
}

}  // namespace gemm
}  // namespace b200q

namespace b200q {

// One launch where every CTA can quantize its slice of the activation while its weights arrive: at most 16 KB of
// activation (read by every CTA for the abs-max), at most kOwnXTiles K tiles per CTA, at most kOwnXSlice tokens x K tiles,
// and 16 tiles of weight rows.  Clusters as large as they may be, which keeps the slices short, but no more than are resident at
// once: 34 tiles on clusters of eight and 72 on clusters of four would take two rounds, which the plain GEMM avoids (8 x 4608 x
// 1024 12.0 us against 6.5; such sizes then take smaller clusters or two launches).  Measured against the quantize launch and the
// GEMM behind it at 776 points inside (1 to 8 tokens, N 1920 to 28672, K 256 to 8192, bf16 and fp32, weights rotating through more
// than L2 where they are that large): 0.78 of the time of an eager call, which a launch less decides (at worst 1.05, fp32
// 1.18).  In a replayed graph 0.91 where the range is given (at worst 1.04); where it is measured 1.03 for bf16 and 1.08 for
// fp32 (at worst 1.18 and 1.38), whose elements every CTA reads twice.  Outside, with the same kernel: 4 x 10240 x 4096 16.0 us
// against 12.6, 1 x 10240 x 8192 27.2 against 18.5, 16 x 4096 x 4096 14.7 against 9.1 (the quantizer's work in every CTA), 1 x
// 1024 x 1024 5.3 against 5.1 (too few CTAs to gain).
int fp8_linear_small(const void* x, int dtype, const float* amax, int64_t amax_numel, const uint8_t* w, const float* w_scales,
                     int64_t w_scales_numel, const void* bias, void* out, int64_t M, int64_t N, int64_t K, b200q_stream_t stream) {
  const int64_t width = dtype == B200Q_F32 ? 4 : 2;
  if (M <= 0 || M > gemm::kOwnXSlice || K <= 0 || K > 16384 || M * K * width > 16384 || K % 16 != 0 || N > 0x7fffffffLL) return 1;
  const int tiles = static_cast<int>((N + gemm::kSmallWRows - 1) / gemm::kSmallWRows);
  const int k_tiles = static_cast<int>((K + gemm::kBKBytes - 1) / gemm::kBKBytes);
  if (tiles < 16) return 1;
  const int sms = sm_count();
  int splits = gemm::smallm_most_splits(tiles, k_tiles, sms, static_cast<int>(M));
  if (splits > 1) {
    const gemm::ActiveClusters clusters = gemm::active_clusters(sms);
    while (splits > 1 && tiles > gemm::smallm_resident(splits, clusters, true)) splits >>= 1;      // its CTAs share SMs
  }
  const int per_cta = (k_tiles + splits - 1) / splits;
  if (per_cta > gemm::kOwnXTiles || per_cta * M > gemm::kOwnXSlice) return 1;
  if (!aligned(x, 16) || !aligned(w, 16) || !aligned(out, 16)) return 1;
  if (int rc = check_arch()) return rc;
  gemm::Params p{};
  p.status = gemm::device_status_word();
  if (p.status == nullptr) return B200Q_ERR_CUDA;
  p.x = x;
  p.x_amax = amax;
  p.x_amax_numel = static_cast<int>(amax_numel);
  p.b_scales = w_scales;
  p.b_scale_stride = w_scales_numel == 1 ? 0 : 1;
  p.bias = static_cast<const __nv_bfloat16*>(bias);
  p.out = static_cast<__nv_bfloat16*>(out);
  p.M = static_cast<int>(M);
  p.N = static_cast<int>(N);
  p.k_bytes = static_cast<int>(K);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  switch (dtype) {
    case B200Q_BF16: return gemm::launch_smallm_own_x<__nv_bfloat16>(w, p, st, splits, per_cta);
    case B200Q_F16: return gemm::launch_smallm_own_x<__half>(w, p, st, splits, per_cta);
    case B200Q_F32: return gemm::launch_smallm_own_x<float>(w, p, st, splits, per_cta);
    default: return 1;
  }
}

}  // namespace b200q

using namespace b200q;

extern "C" {

int b200q_device_status(int reset) {
  int* w = gemm::device_status_word();
  if (w == nullptr) return B200Q_ERR_CUDA;
  int v = 0;
  if (cudaMemcpy(&v, w, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess) return B200Q_ERR_CUDA;
  if (reset && v != 0) {
    const int zero = 0;
    if (cudaMemcpy(w, &zero, sizeof(int), cudaMemcpyHostToDevice) != cudaSuccess) return B200Q_ERR_CUDA;
  }
  return v == 0 ? B200Q_OK : B200Q_ERR_TIMEOUT;
}

int b200q_fp8_gemm(const uint8_t* a_codes, const float* a_scales, int64_t a_scales_numel, const uint8_t* b_codes,
                   const float* b_scales, int64_t b_scales_numel, const void* bias, void* out, int64_t M, int64_t N,
                   int64_t K, b200q_stream_t stream, const b200q_cfg* cfg) {
  if (a_codes == nullptr || b_codes == nullptr || a_scales == nullptr || b_scales == nullptr || out == nullptr)
    return B200Q_ERR_INVALID;
  if (cfg != nullptr && (!gemm::valid_tile_n(cfg->tile_n) || cfg->reserved != 0)) return B200Q_ERR_INVALID;
  if (M < 0 || N < 0 || K <= 0 || M > 0x7fffffffLL || N > 0x7fffffffLL || K > 0x7fffffffLL) return B200Q_ERR_INVALID;
  if (K % 16 != 0) return B200Q_ERR_INVALID;
  if ((a_scales_numel != 1 && a_scales_numel != M) || (b_scales_numel != 1 && b_scales_numel != N)) return B200Q_ERR_INVALID;
  if (!aligned(a_codes, 16) || !aligned(b_codes, 16) || !aligned(out, 16)) return B200Q_ERR_ALIGN;
  if (int rc = check_arch()) return rc;
  if (M == 0 || N == 0) return B200Q_OK;
  gemm::Params p{};
  p.a_scales = a_scales;
  p.b_scales = b_scales;
  p.a_scale_stride = a_scales_numel == 1 ? 0 : 1;
  p.b_scale_stride = b_scales_numel == 1 ? 0 : 1;
  p.bias = static_cast<const __nv_bfloat16*>(bias);
  p.out = static_cast<__nv_bfloat16*>(out);
  p.M = static_cast<int>(M);
  p.N = static_cast<int>(N);
  p.k_bytes = static_cast<int>(K);
  return gemm::launch<false>(a_codes, b_codes, p, static_cast<cudaStream_t>(stream), cfg);
}

int b200q_fp8_gemm_silu_mul(const uint8_t* a_codes, const float* a_scales, int64_t a_scales_numel, const uint8_t* b_codes,
                            const float* b_scales, int64_t b_scales_numel, const void* bias, void* out, int64_t M, int64_t N,
                            int64_t K, b200q_stream_t stream, const b200q_cfg* cfg) {
  if (a_codes == nullptr || b_codes == nullptr || a_scales == nullptr || b_scales == nullptr || out == nullptr)
    return B200Q_ERR_INVALID;
  if (cfg != nullptr && (cfg->tile_n != 0 || cfg->reserved != 0)) return B200Q_ERR_INVALID;   // one kernel serves this entry
  if (M < 0 || N < 0 || K <= 0 || M > 0x7fffffffLL || N > 0x7fffffffLL || K > 0x7fffffffLL) return B200Q_ERR_INVALID;
  if (K % 16 != 0 || N % 256 != 0) return B200Q_ERR_INVALID;                                   // F = N / 2 in whole 128-column tiles
  if ((a_scales_numel != 1 && a_scales_numel != M) || (b_scales_numel != 1 && b_scales_numel != N)) return B200Q_ERR_INVALID;
  if (!aligned(a_codes, 16) || !aligned(b_codes, 16) || !aligned(out, 16)) return B200Q_ERR_ALIGN;
  if (int rc = check_arch()) return rc;
  if (M == 0 || N == 0) return B200Q_OK;
  gemm::Params p{};
  p.a_scales = a_scales;
  p.b_scales = b_scales;
  p.a_scale_stride = a_scales_numel == 1 ? 0 : 1;
  p.b_scale_stride = b_scales_numel == 1 ? 0 : 1;
  p.bias = static_cast<const __nv_bfloat16*>(bias);
  p.out = static_cast<__nv_bfloat16*>(out);
  p.M = static_cast<int>(M);
  p.N = static_cast<int>(N);
  p.k_bytes = static_cast<int>(K);
  p.silu_f = static_cast<int>(N / 2);
  p.status = gemm::device_status_word();
  if (p.status == nullptr) return B200Q_ERR_CUDA;
  return gemm::launch_pair<false, 1>(a_codes, b_codes, p, static_cast<cudaStream_t>(stream));
}

int b200q_fp8_gemm_silu_mul_quantize(const uint8_t* a_codes, const float* a_scales, int64_t a_scales_numel, const uint8_t* b_codes,
                                     const float* b_scales, int64_t b_scales_numel, const void* bias, const float* act_amax,
                                     uint8_t* codes_out, float* scale_out, int64_t M, int64_t N, int64_t K, b200q_stream_t stream,
                                     const b200q_cfg* cfg) {
  if (a_codes == nullptr || b_codes == nullptr || a_scales == nullptr || b_scales == nullptr || codes_out == nullptr || act_amax == nullptr)
    return B200Q_ERR_INVALID;
  if (cfg != nullptr && (cfg->tile_n != 0 || cfg->reserved != 0)) return B200Q_ERR_INVALID;
  if (M < 0 || N < 0 || K <= 0 || M > 0x7fffffffLL || N > 0x7fffffffLL || K > 0x7fffffffLL) return B200Q_ERR_INVALID;
  if (K % 16 != 0 || N % 256 != 0) return B200Q_ERR_INVALID;
  if ((a_scales_numel != 1 && a_scales_numel != M) || (b_scales_numel != 1 && b_scales_numel != N)) return B200Q_ERR_INVALID;
  if (!aligned(a_codes, 16) || !aligned(b_codes, 16) || !aligned(codes_out, 16)) return B200Q_ERR_ALIGN;
  if (int rc = check_arch()) return rc;
  if (M == 0 || N == 0) return B200Q_OK;
  gemm::Params p{};
  p.a_scales = a_scales;
  p.b_scales = b_scales;
  p.a_scale_stride = a_scales_numel == 1 ? 0 : 1;
  p.b_scale_stride = b_scales_numel == 1 ? 0 : 1;
  p.bias = static_cast<const __nv_bfloat16*>(bias);
  p.out = reinterpret_cast<__nv_bfloat16*>(codes_out);
  p.M = static_cast<int>(M);
  p.N = static_cast<int>(N);
  p.k_bytes = static_cast<int>(K);
  p.silu_f = static_cast<int>(N / 2);
  p.act_amax = act_amax;
  p.act_scale_out = scale_out;
  p.status = gemm::device_status_word();
  if (p.status == nullptr) return B200Q_ERR_CUDA;
  return gemm::launch_pair<false, 2>(a_codes, b_codes, p, static_cast<cudaStream_t>(stream));
}

static int fill_rs(gemm::Params& p, gemm::RsTargets& rs, const b200q_peers* peers, int64_t M) {
  if (peers == nullptr || peers->world < 2 || peers->world > 8 || peers->rank < 0 || peers->rank >= peers->world) return B200Q_ERR_INVALID;
  if (M % (static_cast<int64_t>(peers->world) * 128) != 0) return B200Q_ERR_INVALID;
  p.rs_world = peers->world;
  p.rs_rank = peers->rank;
  p.rs_rows = static_cast<int>(M / peers->world);
  for (int r = 0; r < peers->world; ++r) {
    if (peers->recv[r] == nullptr) return B200Q_ERR_INVALID;
    if (!aligned(peers->recv[r], 16)) return B200Q_ERR_ALIGN;
    rs.recv[r] = peers->recv[r];
  }
  return B200Q_OK;
}

int b200q_fp8_gemm_reduce_scatter(const uint8_t* a_codes, const float* a_scales, int64_t a_scales_numel, const uint8_t* b_codes,
                                  const float* b_scales, int64_t b_scales_numel, const b200q_peers* peers, int64_t M, int64_t N,
                                  int64_t K, b200q_stream_t stream, const b200q_cfg* cfg) {
  if (a_codes == nullptr || b_codes == nullptr || a_scales == nullptr || b_scales == nullptr) return B200Q_ERR_INVALID;
  if (cfg != nullptr && (!gemm::valid_tile_n(cfg->tile_n) || cfg->reserved != 0)) return B200Q_ERR_INVALID;
  if (M <= 0 || N <= 0 || K <= 0 || M > 0x7fffffffLL || N > 0x7fffffffLL || K > 0x7fffffffLL) return B200Q_ERR_INVALID;
  if (K % 16 != 0 || N % 8 != 0) return B200Q_ERR_INVALID;
  if ((a_scales_numel != 1 && a_scales_numel != M) || (b_scales_numel != 1 && b_scales_numel != N)) return B200Q_ERR_INVALID;
  if (!aligned(a_codes, 16) || !aligned(b_codes, 16)) return B200Q_ERR_ALIGN;
  gemm::Params p{};
  gemm::RsTargets rs{};
  if (int rc = fill_rs(p, rs, peers, M)) return rc;
  if (int rc = check_arch()) return rc;
  p.a_scales = a_scales;
  p.b_scales = b_scales;
  p.a_scale_stride = a_scales_numel == 1 ? 0 : 1;
  p.b_scale_stride = b_scales_numel == 1 ? 0 : 1;
  p.out = static_cast<__nv_bfloat16*>(peers->recv[peers->rank]);
  p.M = static_cast<int>(M);
  p.N = static_cast<int>(N);
  p.k_bytes = static_cast<int>(K);
  return gemm::launch<false>(a_codes, b_codes, p, static_cast<cudaStream_t>(stream), cfg, &rs);
}

}  // extern "C"
