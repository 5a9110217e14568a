// Host launchers of the tcgen05 GEMM (kernel template in pkb/gemm_umma.cuh).
#include <array>
#include <cstdlib>

#include "pkb/api.h"
#include "pkb/gemm_split.cuh"
#include "pkb/gemm_umma2.cuh"
#include "pkb/host.h"

namespace pkb {

template <int BN, int EPI, bool OUT_F32>
static int launch_plain(const CUtensorMap& ta, const CUtensorMap& tb, const GemmParams& p,
                        int num_ctas, cudaStream_t stream) {
  auto kern = gemm_umma_kernel<BN, EPI, OUT_F32, false, false>;
  constexpr int smem = GemmSmem<BN>::kTotal;
  static bool configured = false;  // per instantiation; attribute is per device but idempotent
  if (!configured) {
    PKB_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    configured = true;
  }
  kern<<<num_ctas, kGemmThreads, smem, stream>>>(ta, tb, p);
  PKB_CHECK_CUDA(cudaGetLastError());
  return kApiOk;
}

template <int BN, bool OUT_F32>
static int dispatch_epi(int epi, const CUtensorMap& ta, const CUtensorMap& tb, const GemmParams& p,
                        int num_ctas, cudaStream_t stream) {
  switch (epi) {
    case kEpiNone: return launch_plain<BN, kEpiNone, OUT_F32>(ta, tb, p, num_ctas, stream);
    case kEpiSilu: return launch_plain<BN, kEpiSilu, OUT_F32>(ta, tb, p, num_ctas, stream);
    case kEpiBias: return launch_plain<BN, kEpiBias, OUT_F32>(ta, tb, p, num_ctas, stream);
    case kEpiBiasSilu: return launch_plain<BN, kEpiBiasSilu, OUT_F32>(ta, tb, p, num_ctas, stream);
  }
  set_last_error("unknown epilogue");
  return kApiBadArgument;
}

// The backward layouts on CTA pairs: PKB_GEMM_PAIR_MN=0 keeps the one-CTA-per-tile kernels.
static bool pair_mn_enabled() {
  static const bool on = [] { const char* e = getenv("PKB_GEMM_PAIR_MN"); return !(e != nullptr && e[0] == '0'); }();
  return on;
}

// Tile width of the CTA-pair kernel. A wave is sm_count / 2 tiles of 256 x BN, so a problem costs its number of waves times the
// width, times a factor for narrow tiles, which read more operand bytes per flop. The factors are measured (us at 256 / 192 /
// 128): 1333 x 4104 x 4096 (2, 2, 3 waves) 51.9 / 43.8 / 46.0; 4096 x 4096 x 4096 (4, 5, 7) 94.2 / 94.1 / 94.2; 4104 x 4096 x 1336
// (4, 6, 8) 50 / 56 / 64. With an MN-major B what narrow tiles gain does not follow from the waves (256 / 128: 1333 x 4104 x 4096 52.2 /
// 48.1, 1536 x 4096 x 14336 150 / 128, but 1333 x 4096 x 4104 52.2 / 59.4, 1333 x 14336 x 4096 114 / 123), so 128 columns are taken only where
// they save 30 % of the columns computed (512 x 4096 x 4096 29.7 / 23.5, 640 x 2048 x 8192 50.3 / 33.8); 192 columns, of which half a box is
// not used, can never save as many.
static int pair_tile_n(int M, int N, int pairs, bool b_mn) {
  const long long num_m = (M + 255) / 256;
  auto cost = [&](int bn, double per_col) {
    const long long tiles = num_m * ((N + bn - 1) / bn);
    return (double)((tiles + pairs - 1) / pairs) * (bn * per_col);
  };
  int best = 256;
  double c = cost(256, 1.0);
  if (!b_mn && cost(192, 1.09) < c) { best = 192; c = cost(192, 1.09); }
  if (cost(128, b_mn ? 1.4 : 1.16) < c) best = 128;
  return best;
}

template <int EPI, bool OUT_F32, bool A_MN, bool B_MN, int BN>
static int launch_pair_bn(const CUtensorMap& ta, const CUtensorMap& tb, const GemmParams& p, int ctas, cudaStream_t stream) {
  if constexpr (!OUT_F32) {
    if (p.ldc % 8 == 0 && (reinterpret_cast<uintptr_t>(p.C) & 15) == 0) {
      GemmOutMaps om;
      int rc = encode_tmap_2d(&om.m[0], kTmapBf16, p.C, (uint64_t)p.N, (uint64_t)p.M, (uint64_t)p.ldc * 2, 64, 32, kSwizzle128);
      if (rc) return rc;
      auto kern = gemm_umma2_tma_kernel<EPI, A_MN, B_MN, BN>;
      PKB_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kGemm2SmemTotal));
      kern<<<ctas, kGemmThreads, kGemm2SmemTotal, stream>>>(ta, tb, om, p);
      PKB_CHECK_CUDA(cudaGetLastError());
      return kApiOk;
    }
  }
  auto launch = [&](auto kern) -> int {
    PKB_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kGemm2SmemTotal));
    kern<<<ctas, kGemmThreads, kGemm2SmemTotal, stream>>>(ta, tb, p);
    PKB_CHECK_CUDA(cudaGetLastError());
    return kApiOk;
  };
  if constexpr (A_MN || B_MN) return launch(gemm_umma2_mn_kernel<EPI, OUT_F32, A_MN, B_MN, BN>);
  else return launch(gemm_umma2_kernel<EPI, OUT_F32, BN>);
}

// 256 x BN tiles on clusters of two CTAs (every operand byte crosses L2 -> shared memory once per pair). `a` / `b` are K-major
// unless A_MN / B_MN; num_ctas 0 = all SMs, else at least 2 (rounded down to whole pairs).
template <int EPI, bool OUT_F32, bool A_MN, bool B_MN>
static int launch_pair(const CUtensorMap& ta, const void* b, long long ldb, GemmParams p, int num_ctas, cudaStream_t stream) {
  p.group_m = 8;
  int ctas = (num_ctas > 0 ? num_ctas : sm_count()) & ~1;
  const int bn = pair_tile_n(p.M, p.N, ctas / 2, B_MN);
  const int tiles = ((p.M + 255) / 256) * ((p.N + bn - 1) / bn);
  if (ctas > 2 * tiles) ctas = 2 * tiles;
  CUtensorMap tb;
  int rc = B_MN ? encode_tmap_2d(&tb, kTmapBf16, b, (uint64_t)p.N, (uint64_t)p.K, (uint64_t)ldb * 2, 64, kGemmBlockK, kSwizzle128)
                : encode_tmap_2d(&tb, kTmapBf16, b, (uint64_t)p.K, (uint64_t)p.N, (uint64_t)ldb * 2, kGemmBlockK, (uint32_t)bn / 2, kSwizzle128);
  if (rc) return rc;
  if (bn == 128) return launch_pair_bn<EPI, OUT_F32, A_MN, B_MN, 128>(ta, tb, p, ctas, stream);
  if constexpr (!B_MN) {
    if (bn == 192) return launch_pair_bn<EPI, OUT_F32, A_MN, B_MN, 192>(ta, tb, p, ctas, stream);
  }
  return launch_pair_bn<EPI, OUT_F32, A_MN, B_MN, 256>(ta, tb, p, ctas, stream);
}

template <bool OUT_F32>
static int dispatch_pair(int epi, const CUtensorMap& ta, const void* b, long long ldb, const GemmParams& p, int num_ctas,
                         cudaStream_t stream) {
  switch (epi) {
    case kEpiNone: return launch_pair<kEpiNone, OUT_F32, false, false>(ta, b, ldb, p, num_ctas, stream);
    case kEpiSilu: return launch_pair<kEpiSilu, OUT_F32, false, false>(ta, b, ldb, p, num_ctas, stream);
    case kEpiBias: return launch_pair<kEpiBias, OUT_F32, false, false>(ta, b, ldb, p, num_ctas, stream);
    case kEpiBiasSilu: return launch_pair<kEpiBiasSilu, OUT_F32, false, false>(ta, b, ldb, p, num_ctas, stream);
  }
  set_last_error("unknown epilogue");
  return kApiBadArgument;
}

// Up to 64 rows, at most one 128-column tile per SM and at least 24 K blocks: the kernel that shares a tile's K range between the CTAs of
// a cluster (gemm_split.cuh). Measured against one CTA per tile, L2 flushed, us: 1 x 2048 x 2048 12.3 / 14.4, 64 x 2048 x 2048 13.8 / 14.4,
// 33 x 1024 x 8192 14.4 / 32.8, 7 x 264 x 16384 16.2 / 56.6, 64 x 4096 x 4096 18.0 / 22.6; with one CTA per tile, where only the deeper ring
// tells, 1 x 14336 x 4096 34.9 / 43.9, 16 x 14336 x 4096 34.8 / 36.4. Fewer K blocks: 1 x 1024 x 1024 10.3 / 10.3, 64 x 1024 x 1024 12.2 /
// 11.6, 64 x 2048 x 512 12.2 / 10.1, 1 x 256 x 256 9.0 / 8.2. More than one tile per SM: 16 x 20000 x 4096 51.4 / 53.0, 64 x 128256 x 4096
// 192 / 192, 128 rows of it 205 / 198 (1 row 182 / 242). More rows: 80 x 1024 x 8192 16.6 / 33.3 and 80 x 4096 x 4096 18.7 / 23.1, but 128 x
// 2048 x 512 13.9 / 10.5 and 128 x 20000 x 4096 56 / 50.
static bool split_fits(int M, int N, int K) {
  return M <= 64 && (N + 127) / 128 <= sm_count() && K > 23 * kGemmBlockK;
}

// Cluster size: as many CTAs as leave every tile's cluster resident at once (15 clusters of 8 CTAs, 33 of 4, 74 of 2: a cluster stays
// inside a group of 16 to 20 SMs), and at least four K blocks each. One cluster too many is a second wave: 64 x 2048 x 2048 (16 tiles)
// 20.4 us on clusters of 8, 13.8 on 4.
template <int EPI, bool OUT_F32, bool B_MN>
static int split_count(int tiles, int num_k) {
  static const std::array<int, 9> resident = resident_clusters(gemm_split_kernel<EPI, OUT_F32, B_MN>, kGemmThreads, kSplitSmemTotal);
  int s = 8;
  while (s > 1 && (tiles > resident[s] || num_k < 4 * s)) s >>= 1;
  return s;
}

template <int EPI, bool OUT_F32, bool B_MN>
static int launch_split(const void* a, long long lda, const void* b, long long ldb, const GemmParams& p, cudaStream_t stream) {
  const int a_rows = p.M <= 16 ? 16 : p.M <= 32 ? 32 : 64;
  int stages = kSplitRingBytes / (a_rows * 128 + kSplitBN * 128);
  if (stages > kSplitMaxStages) stages = kSplitMaxStages;
  CUtensorMap ta, tb;
  int rc = encode_tmap_2d(&ta, kTmapBf16, a, (uint64_t)p.K, (uint64_t)p.M, (uint64_t)lda * 2, kGemmBlockK, (uint32_t)a_rows, kSwizzle128);
  if (rc) return rc;
  rc = B_MN ? encode_tmap_2d(&tb, kTmapBf16, b, (uint64_t)p.N, (uint64_t)p.K, (uint64_t)ldb * 2, 64, kGemmBlockK, kSwizzle128)
            : encode_tmap_2d(&tb, kTmapBf16, b, (uint64_t)p.K, (uint64_t)p.N, (uint64_t)ldb * 2, kGemmBlockK, kSplitBN, kSwizzle128);
  if (rc) return rc;
  const int tiles = (p.N + kSplitBN - 1) / kSplitBN;
  const int splits = split_count<EPI, OUT_F32, B_MN>(tiles, (p.K + kGemmBlockK - 1) / kGemmBlockK);
  auto kern = gemm_split_kernel<EPI, OUT_F32, B_MN>;
  PKB_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSplitSmemTotal));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(tiles * splits));
  cfg.blockDim = dim3(kGemmThreads);
  cfg.dynamicSmemBytes = kSplitSmemTotal;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)splits;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  PKB_CHECK_CUDA(cudaLaunchKernelEx(&cfg, kern, ta, tb, p, splits, a_rows, stages));
  return kApiOk;
}

template <bool OUT_F32>
static int dispatch_split(int epi, const void* a, long long lda, const void* b, long long ldb, const GemmParams& p, cudaStream_t stream) {
  switch (epi) {
    case kEpiNone: return launch_split<kEpiNone, OUT_F32, false>(a, lda, b, ldb, p, stream);
    case kEpiSilu: return launch_split<kEpiSilu, OUT_F32, false>(a, lda, b, ldb, p, stream);
    case kEpiBias: return launch_split<kEpiBias, OUT_F32, false>(a, lda, b, ldb, p, stream);
    case kEpiBiasSilu: return launch_split<kEpiBiasSilu, OUT_F32, false>(a, lda, b, ldb, p, stream);
  }
  set_last_error("unknown epilogue");
  return kApiBadArgument;
}

}  // namespace pkb

using namespace pkb;

// CTA-pair form: 256 x 256 tiles on clusters of two CTAs (see pkb/gemm_umma2.cuh).
extern "C" int pkb_gemm_bf16_pair(const void* a, long long lda, const void* b, long long ldb,
                                  void* c, long long ldc, int M, int N, int K, const void* bias,
                                  float alpha, int epilogue, int out_f32, int num_ctas,
                                  void* stream) {
  PKB_CHECK_ARG(M > 0 && N > 0 && K > 0, "empty problem");
  PKB_CHECK_ARG(lda % 8 == 0 && ldb % 8 == 0 && K % 8 == 0, "lda, ldb, K must be multiples of 8");
  PKB_CHECK_ARG((epilogue & 2) == 0 || bias != nullptr, "bias epilogue without bias");
  PKB_CHECK_ARG(num_ctas != 1, "num_ctas = 1: the tiles of this form belong to pairs of CTAs");
  CUtensorMap ta;
  int rc = encode_tmap_2d(&ta, kTmapBf16, a, (uint64_t)K, (uint64_t)M, (uint64_t)lda * 2, kGemmBlockK, 128, kSwizzle128);
  if (rc) return rc;
  GemmParams p = {};
  p.M = M; p.N = N; p.K = K;
  p.C = c; p.ldc = ldc;
  p.bias = static_cast<const __nv_bfloat16*>(bias);
  p.alpha = alpha;
  p.status = status_block_device_ptr();
  p.wait_budget_ns = kDefaultWaitBudgetNs;
  p.kernel_id = 101;
  p.world = 1;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  return out_f32 ? dispatch_pair<true>(epilogue, ta, b, ldb, p, num_ctas, s) : dispatch_pair<false>(epilogue, ta, b, ldb, p, num_ctas, s);
}

extern "C" int pkb_gemm_bf16(const void* a, long long lda, const void* b, long long ldb, void* c,
                             long long ldc, int M, int N, int K, const void* bias, float alpha,
                             int epilogue, int out_f32, int block_n, int num_ctas, void* stream) {
  PKB_CHECK_ARG(M > 0 && N > 0 && K > 0, "empty problem");
  PKB_CHECK_ARG(lda % 8 == 0 && ldb % 8 == 0 && K % 8 == 0, "lda, ldb, K must be multiples of 8");
  PKB_CHECK_ARG((epilogue & 2) == 0 || bias != nullptr, "bias epilogue without bias");
  if (block_n == 0) block_n = (N >= 256 && (long long)M * N >= 128ll * 256 * 64) ? 256 : 128;
  PKB_CHECK_ARG(block_n == 128 || block_n == 256, "block_n must be 128 or 256");

  CUtensorMap ta, tb;
  int rc = encode_tmap_2d(&ta, kTmapBf16, a, (uint64_t)K, (uint64_t)M, (uint64_t)lda * 2,
                          kGemmBlockK, kGemmBlockM, kSwizzle128);
  if (rc) return rc;
  rc = encode_tmap_2d(&tb, kTmapBf16, b, (uint64_t)K, (uint64_t)N, (uint64_t)ldb * 2, kGemmBlockK,
                      (uint32_t)block_n, kSwizzle128);
  if (rc) return rc;

  GemmParams p = {};
  p.M = M; p.N = N; p.K = K;
  p.C = c; p.ldc = ldc;
  p.bias = static_cast<const __nv_bfloat16*>(bias);
  p.alpha = alpha;
  p.status = status_block_device_ptr();
  p.wait_budget_ns = kDefaultWaitBudgetNs;
  p.group_m = 16;
  p.kernel_id = 100;
  p.world = 1;

  const int num_m = (M + kGemmBlockM - 1) / kGemmBlockM;
  const int num_n = (N + block_n - 1) / block_n;
  const int tiles = num_m * num_n;
  int ctas = num_ctas > 0 ? num_ctas : sm_count();
  if (ctas > tiles) ctas = tiles;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (block_n == 256)
    return out_f32 ? dispatch_epi<256, true>(epilogue, ta, tb, p, ctas, s)
                   : dispatch_epi<256, false>(epilogue, ta, tb, p, ctas, s);
  return out_f32 ? dispatch_epi<128, true>(epilogue, ta, tb, p, ctas, s)
                 : dispatch_epi<128, false>(epilogue, ta, tb, p, ctas, s);
}

// The form chosen by shape: few rows -> gemm_split.cuh (see split_fits); from 512 x 256 on the CTA pairs; else
// one CTA per tile.
extern "C" int pkb_gemm_bf16_auto(const void* a, long long lda, const void* b, long long ldb, void* c, long long ldc, int M, int N,
                                  int K, const void* bias, float alpha, int epilogue, int out_f32, void* stream) {
  PKB_CHECK_ARG(M > 0 && N > 0 && K > 0, "empty problem");
  if (!split_fits(M, N, K))
    return M >= 512 && N >= 256 ? pkb_gemm_bf16_pair(a, lda, b, ldb, c, ldc, M, N, K, bias, alpha, epilogue, out_f32, 0, stream)
                                : pkb_gemm_bf16(a, lda, b, ldb, c, ldc, M, N, K, bias, alpha, epilogue, out_f32, 0, 0, stream);
  PKB_CHECK_ARG(lda % 8 == 0 && ldb % 8 == 0 && K % 8 == 0, "lda, ldb, K must be multiples of 8");
  PKB_CHECK_ARG((epilogue & 2) == 0 || bias != nullptr, "bias epilogue without bias");
  GemmParams p = {};
  p.M = M; p.N = N; p.K = K;
  p.C = c; p.ldc = ldc;
  p.bias = static_cast<const __nv_bfloat16*>(bias);
  p.alpha = alpha;
  p.status = status_block_device_ptr();
  p.wait_budget_ns = kDefaultWaitBudgetNs;
  p.kernel_id = 108;
  p.world = 1;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  return out_f32 ? dispatch_split<true>(epilogue, a, lda, b, ldb, p, s) : dispatch_split<false>(epilogue, a, lda, b, ldb, p, s);
}

// Grouped (ragged) GEMM: rows of A are grouped back to back, group e = rows
// [offsets[e], offsets[e+1]) (int32 device array of groups + 1 entries, read on the device only) and
// uses the weight block b[e*N : (e+1)*N, :]. C[total_rows, N] (or N/2 columns for the SwiGLU
// epilogue). max_rows bounds offsets[groups]; rows at or beyond it are never touched.
// epilogue: 0 none, 1 SiLU, 4 SwiGLU over interleaved (gate, up) weight rows.
extern "C" int pkb_gemm_bf16_grouped(const void* a, long long lda, const void* b, long long ldb,
                                     void* c, long long ldc, const void* offsets, int groups,
                                     int max_rows, int N, int K, int epilogue, int block_n,
                                     void* stream) {
  PKB_CHECK_ARG(groups >= 1 && groups <= kGemmMaxGroups, "1..256 groups");
  PKB_CHECK_ARG(max_rows > 0 && N > 0 && K > 0, "empty problem");
  PKB_CHECK_ARG(lda % 8 == 0 && ldb % 8 == 0 && K % 8 == 0, "lda, ldb, K must be multiples of 8");
  PKB_CHECK_ARG(epilogue == kEpiNone || epilogue == kEpiSilu || epilogue == kEpiSwiGLU, "unsupported epilogue");
  if (block_n == 0) block_n = N >= 256 ? 256 : 128;
  PKB_CHECK_ARG(block_n == 128 || block_n == 256, "block_n must be 128 or 256");
  CUtensorMap ta, tb;
  int rc = encode_tmap_2d(&ta, kTmapBf16, a, (uint64_t)K, (uint64_t)max_rows, (uint64_t)lda * 2,
                          kGemmBlockK, kGemmBlockM, kSwizzle128);
  if (rc) return rc;
  rc = encode_tmap_2d(&tb, kTmapBf16, b, (uint64_t)K, (uint64_t)groups * N, (uint64_t)ldb * 2,
                      kGemmBlockK, (uint32_t)block_n, kSwizzle128);
  if (rc) return rc;
  GemmParams p = {};
  p.M = max_rows; p.N = N; p.K = K;
  p.C = c; p.ldc = ldc; p.alpha = 1.0f;
  p.status = status_block_device_ptr();
  p.wait_budget_ns = kDefaultWaitBudgetNs;
  p.kernel_id = 102;
  p.world = 1;
  p.grp_offsets = static_cast<const int*>(offsets);
  p.grp_count = groups;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  // CTA pairs (256 x 256 tiles over two SMs, half of the B traffic per SM) when the shape allows; PKB_GROUPED_PAIR=0 keeps
  // the one-CTA-per-tile kernel
  static const bool pair_on = [] { const char* e = getenv("PKB_GROUPED_PAIR"); return !(e != nullptr && e[0] == '0'); }();
  if (pair_on && block_n == 256 && N % 256 == 0 && K % kGemmBlockK == 0 && sm_count() >= 2) {
    CUtensorMap tb2;
    rc = encode_tmap_2d(&tb2, kTmapBf16, b, (uint64_t)K, (uint64_t)groups * N, (uint64_t)ldb * 2, kGemmBlockK, 128, kSwizzle128);
    if (rc) return rc;
    p.kernel_id = 107;
    const int num_ctas = sm_count() & ~1;
#define PKB_GROUPED_PAIR_LAUNCH(EPI)                                                                             \
    {                                                                                                             \
      auto kern = gemm_umma2_grouped_kernel<EPI>;                                                                 \
      PKB_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kGemm2SmemTotal));   \
      kern<<<num_ctas, kGemmThreads, kGemm2SmemTotal, s>>>(ta, tb2, p);                                           \
    }
    if (epilogue == kEpiNone) PKB_GROUPED_PAIR_LAUNCH(kEpiNone)
    else if (epilogue == kEpiSilu) PKB_GROUPED_PAIR_LAUNCH(kEpiSilu)
    else PKB_GROUPED_PAIR_LAUNCH(kEpiSwiGLU)
#undef PKB_GROUPED_PAIR_LAUNCH
    PKB_CHECK_CUDA(cudaGetLastError());
    return kApiOk;
  }
  const int ctas = sm_count();
#define PKB_GROUPED(BN, EPI)                                                                        \
  {                                                                                                 \
    auto kern = gemm_umma_grouped_kernel<BN, EPI>;                                                  \
    PKB_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,          \
                                        GemmSmem<BN>::kTotal));                                     \
    kern<<<ctas, kGemmThreads, GemmSmem<BN>::kTotal, s>>>(ta, tb, p);                               \
  }
  if (block_n == 256) {
    if (epilogue == kEpiNone) PKB_GROUPED(256, kEpiNone)
    else if (epilogue == kEpiSilu) PKB_GROUPED(256, kEpiSilu)
    else PKB_GROUPED(256, kEpiSwiGLU)
  } else {
    if (epilogue == kEpiNone) PKB_GROUPED(128, kEpiNone)
    else if (epilogue == kEpiSilu) PKB_GROUPED(128, kEpiSilu)
    else PKB_GROUPED(128, kEpiSwiGLU)
  }
#undef PKB_GROUPED
  PKB_CHECK_CUDA(cudaGetLastError());
  return kApiOk;
}

// Grouped GEMM whose output rows are scattered: row m of the product is stored as row row_meta[m].y (ldc elements per
// row, bf16) of the buffer dest_ptrs[row_meta[m].x], which may live on another rank. row_meta is an int2 device array with
// one entry per row of A; dest_ptrs is a HOST array of ndest <= 8 device addresses (16-byte aligned).
extern "C" int pkb_gemm_bf16_grouped_scatter(const void* a, long long lda, const void* b, long long ldb, long long ldc,
                                             const void* offsets, int groups, int max_rows, int N, int K, int block_n,
                                             const void* row_meta, const unsigned long long* dest_ptrs, int ndest,
                                             void* stream) {
  PKB_CHECK_ARG(groups >= 1 && groups <= kGemmMaxGroups, "1..256 groups");
  PKB_CHECK_ARG(max_rows > 0 && N > 0 && K > 0, "empty problem");
  PKB_CHECK_ARG(lda % 8 == 0 && ldb % 8 == 0 && K % 8 == 0 && ldc % 8 == 0, "lda, ldb, ldc, K must be multiples of 8");
  PKB_CHECK_ARG(row_meta != nullptr && dest_ptrs != nullptr && ndest >= 1 && ndest <= kGemmMaxWorld,
                "row_meta and 1..8 destination buffers are required");
  if (block_n == 0) block_n = N >= 256 ? 256 : 128;
  PKB_CHECK_ARG(block_n == 128 || block_n == 256, "block_n must be 128 or 256");
  CUtensorMap ta, tb;
  int rc = encode_tmap_2d(&ta, kTmapBf16, a, (uint64_t)K, (uint64_t)max_rows, (uint64_t)lda * 2, kGemmBlockK, kGemmBlockM,
                          kSwizzle128);
  if (rc) return rc;
  rc = encode_tmap_2d(&tb, kTmapBf16, b, (uint64_t)K, (uint64_t)groups * N, (uint64_t)ldb * 2, kGemmBlockK, (uint32_t)block_n,
                      kSwizzle128);
  if (rc) return rc;
  GemmParams p = {};
  p.M = max_rows; p.N = N; p.K = K;
  p.C = nullptr; p.ldc = ldc; p.alpha = 1.0f;
  p.status = status_block_device_ptr();
  p.wait_budget_ns = kDefaultWaitBudgetNs;
  p.kernel_id = 106;
  p.world = 1;
  p.grp_offsets = static_cast<const int*>(offsets);
  p.grp_count = groups;
  p.row_meta = static_cast<const int2*>(row_meta);
  for (int g = 0; g < kGemmMaxWorld; ++g) {
    PKB_CHECK_ARG((dest_ptrs[g < ndest ? g : 0] & 15) == 0, "destination buffers must be 16-byte aligned");
    p.rs_out[g] = reinterpret_cast<void*>(static_cast<uintptr_t>(dest_ptrs[g < ndest ? g : 0]));
  }
  const int ctas = sm_count();
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (block_n == 256) {
    auto kern = gemm_umma_grouped_kernel<256, kEpiRowScatter>;
    PKB_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, GemmSmem<256>::kTotal));
    kern<<<ctas, kGemmThreads, GemmSmem<256>::kTotal, s>>>(ta, tb, p);
  } else {
    auto kern = gemm_umma_grouped_kernel<128, kEpiRowScatter>;
    PKB_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, GemmSmem<128>::kTotal));
    kern<<<ctas, kGemmThreads, GemmSmem<128>::kTotal, s>>>(ta, tb, p);
  }
  PKB_CHECK_CUDA(cudaGetLastError());
  return kApiOk;
}

// C[M,N] = epi(A[M,K] @ B[K,N]) with B row-major [K, N] (ldb elements between K rows, N % 8 == 0).
// epilogue: 0 none, 1 SiLU. out_f32 selects fp32 output.
extern "C" int pkb_gemm_bf16_bkn(const void* a, long long lda, const void* b, long long ldb, void* c,
                                 long long ldc, int M, int N, int K, float alpha, int epilogue,
                                 int out_f32, void* stream) {
  PKB_CHECK_ARG(M > 0 && N > 0 && K > 0, "empty problem");
  PKB_CHECK_ARG(lda % 8 == 0 && ldb % 8 == 0 && K % 8 == 0 && N % 8 == 0, "lda, ldb, K, N must be multiples of 8");
  PKB_CHECK_ARG(epilogue == kEpiNone || epilogue == kEpiSilu, "epilogue must be none or silu");
  CUtensorMap ta, tb;
  int rc = encode_tmap_2d(&ta, kTmapBf16, a, (uint64_t)K, (uint64_t)M, (uint64_t)lda * 2, kGemmBlockK,
                          kGemmBlockM, kSwizzle128);
  if (rc) return rc;
  rc = encode_tmap_2d(&tb, kTmapBf16, b, (uint64_t)N, (uint64_t)K, (uint64_t)ldb * 2, 64, kGemmBlockK,
                      kSwizzle128);
  if (rc) return rc;
  GemmParams p = {};
  p.M = M; p.N = N; p.K = K; p.C = c; p.ldc = ldc; p.alpha = alpha;
  p.status = status_block_device_ptr();
  p.wait_budget_ns = kDefaultWaitBudgetNs;
  p.group_m = 16; p.kernel_id = 103; p.world = 1;
  const int tiles = ((M + 127) / 128) * ((N + 127) / 128);
  int ctas = sm_count();
  if (ctas > tiles) ctas = tiles;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (split_fits(M, N, K)) {
    p.kernel_id = 109;
    if (epilogue == kEpiSilu)
      return out_f32 ? launch_split<kEpiSilu, true, true>(a, lda, b, ldb, p, s) : launch_split<kEpiSilu, false, true>(a, lda, b, ldb, p, s);
    return out_f32 ? launch_split<kEpiNone, true, true>(a, lda, b, ldb, p, s) : launch_split<kEpiNone, false, true>(a, lda, b, ldb, p, s);
  }
  if (pair_mn_enabled() && M >= 256 && N >= 256) {
    if (epilogue == kEpiSilu)
      return out_f32 ? launch_pair<kEpiSilu, true, false, true>(ta, b, ldb, p, 0, s) : launch_pair<kEpiSilu, false, false, true>(ta, b, ldb, p, 0, s);
    return out_f32 ? launch_pair<kEpiNone, true, false, true>(ta, b, ldb, p, 0, s) : launch_pair<kEpiNone, false, false, true>(ta, b, ldb, p, 0, s);
  }
  constexpr int smem = GemmSmem<128>::kTotal;
#define PKB_BKN(EPI, F32)                                                                          \
  {                                                                                                \
    auto kern = gemm_umma_bkn_kernel<128, EPI, F32>;                                               \
    PKB_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem)); \
    kern<<<ctas, kGemmThreads, smem, s>>>(ta, tb, p);                                              \
  }
  if (epilogue == kEpiSilu) { if (out_f32) PKB_BKN(kEpiSilu, true) else PKB_BKN(kEpiSilu, false) }
  else { if (out_f32) PKB_BKN(kEpiNone, true) else PKB_BKN(kEpiNone, false) }
#undef PKB_BKN
  PKB_CHECK_CUDA(cudaGetLastError());
  return kApiOk;
}

// C[M,N] = alpha * A^T B with A [K, M] and B [K, N] row-major (lda, ldb in elements; M, N, K % 8 == 0).
// The natural form of a weight gradient (dW = dY^T X): no transposed copy of either operand.
extern "C" int pkb_gemm_bf16_tn(const void* a, long long lda, const void* b, long long ldb, void* c,
                                long long ldc, int M, int N, int K, float alpha, int out_f32, void* stream) {
  PKB_CHECK_ARG(M > 0 && N > 0 && K > 0, "empty problem");
  PKB_CHECK_ARG(lda % 8 == 0 && ldb % 8 == 0 && M % 8 == 0 && N % 8 == 0, "lda, ldb, M, N must be multiples of 8");
  CUtensorMap ta, tb;
  int rc = encode_tmap_2d(&ta, kTmapBf16, a, (uint64_t)M, (uint64_t)K, (uint64_t)lda * 2, 64, kGemmBlockK, kSwizzle128);
  if (rc) return rc;
  rc = encode_tmap_2d(&tb, kTmapBf16, b, (uint64_t)N, (uint64_t)K, (uint64_t)ldb * 2, 64, kGemmBlockK, kSwizzle128);
  if (rc) return rc;
  GemmParams p = {};
  p.M = M; p.N = N; p.K = K; p.C = c; p.ldc = ldc; p.alpha = alpha;
  p.status = status_block_device_ptr();
  p.wait_budget_ns = kDefaultWaitBudgetNs;
  p.group_m = 16; p.kernel_id = 104; p.world = 1;
  const int tiles = ((M + 127) / 128) * ((N + 255) / 256);
  int ctas = sm_count();
  if (ctas > tiles) ctas = tiles;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (pair_mn_enabled() && M >= 256 && N >= 256)
    return out_f32 ? launch_pair<kEpiNone, true, true, true>(ta, b, ldb, p, 0, s) : launch_pair<kEpiNone, false, true, true>(ta, b, ldb, p, 0, s);
  constexpr int smem = GemmSmem<256>::kTotal;
  if (out_f32) {
    auto kern = gemm_umma_tn_kernel<256, true>;
    PKB_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    kern<<<ctas, kGemmThreads, smem, s>>>(ta, tb, p);
  } else {
    auto kern = gemm_umma_tn_kernel<256, false>;
    PKB_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    kern<<<ctas, kGemmThreads, smem, s>>>(ta, tb, p);
  }
  PKB_CHECK_CUDA(cudaGetLastError());
  return kApiOk;
}
