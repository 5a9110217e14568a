// tcgen05 GEMM for few rows (M <= 64: decoding, small batches):  C[M,N] = epilogue( A[M,K] * B[N,K]^T ).
//
// Bound by reading B: what counts is how many SMs pull it and how many bytes each has in flight, not the tensor pipe. So
//   * a cluster of S CTAs shares a 128-column tile, each takes an S-th of K; the partial sums (fp32) meet in shared memory and
//     every CTA adds up and stores its 128 / S columns, always in the order of the cluster ranks (the result does not depend on
//     timing);
//   * a stage holds only the rows of A that exist (`a_rows` = 16, 32 or 64): the MMA still reads 128 rows, the surplus ones out
//     of whatever follows in the ring, and their rows of the accumulator are never stored. With 16 rows a stage is 18 KiB and
//     the ring eleven deep, 176 KiB of weights in flight per SM instead of 96.
//   warp 0 : TMA producer      warp 1 : MMA issuer      warps 2-5 : accumulator -> shared memory; then all warps reduce and store
// Waits are bounded as in gemm_umma.cuh.
#pragma once
#include "pkb/gemm_umma.cuh"

namespace pkb {

constexpr int kSplitBN = 128;
constexpr int kSplitMaxStages = 11;
constexpr int kSplitRingBytes = kSplitMaxStages * (16 * 128 + kSplitBN * 128);   // 198 KiB; 8 stages with 64 rows of A
constexpr int kSplitSmemTotal = kSplitRingBytes + 256 + 1024;

constexpr int kSplitPitch = kSplitBN * 4 + 16;    // bytes between rows of partial sums: 16-byte accesses of 8 rows hit all banks

// Epilogue and store of NV (a multiple of 4) neighbouring outputs of one row, the first at column `col` (a multiple of 4) of C.
template <int EPI, bool OUT_F32, int NV>
__device__ __forceinline__ void split_store(const GemmParams& p, int row, int col, float (&v)[NV]) {
  if (row >= p.M || col >= p.N) return;
#pragma unroll
  for (int j = 0; j < NV; ++j) {
    v[j] *= p.alpha;
    if constexpr (EPI == kEpiBias || EPI == kEpiBiasSilu) {
      if (col + j < p.N) v[j] += __bfloat162float(p.bias[col + j]);
    }
    if constexpr (EPI == kEpiSilu || EPI == kEpiBiasSilu) v[j] = silu_f(v[j]);
  }
  constexpr int kOutBytes = OUT_F32 ? 4 : 2;
  uint8_t* o = static_cast<uint8_t*>(p.C) + (static_cast<long long>(row) * p.ldc + col) * kOutBytes;
  constexpr int kBytes = NV * kOutBytes;
  if (col + NV <= p.N && (reinterpret_cast<uintptr_t>(o) & (kBytes >= 16 ? 15 : kBytes - 1)) == 0) {
    uint32_t w[kBytes / 4];
#pragma unroll
    for (int j = 0; j < kBytes / 4; ++j) w[j] = OUT_F32 ? __float_as_uint(v[j]) : pack_bf16x2(v[(2 * j) % NV], v[(2 * j + 1) % NV]);
    if constexpr (kBytes == 8) {
      *reinterpret_cast<uint2*>(o) = make_uint2(w[0], w[1]);
    } else {
#pragma unroll
      for (int j = 0; j < kBytes / 4; j += 4) st_global_v4(o + j * 4, U4{w[j], w[j + 1], w[j + 2], w[j + 3]});
    }
  } else {
#pragma unroll
    for (int j = 0; j < NV; ++j)
      if (col + j < p.N) {
        if constexpr (OUT_F32) reinterpret_cast<float*>(o)[j] = v[j];
        else reinterpret_cast<__nv_bfloat16*>(o)[j] = __float2bfloat16_rn(v[j]);
      }
  }
}

// B_MN: B is [K, N] row-major, its tiles come as two boxes of 64 x 64 (see gemm_umma.cuh).
template <int EPI, bool OUT_F32, bool B_MN>
__global__ void __launch_bounds__(kGemmThreads, 1)
gemm_split_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b, const GemmParams p,
                  const int splits, const int a_rows, const int stages) {
  constexpr int BN = kSplitBN;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
  const int a_bytes = a_rows * 128;
  const int stage_bytes = a_bytes + BN * 128;
  const uint32_t bar_base = smem_base + kSplitRingBytes;
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (kSplitMaxStages + s); };
  const uint32_t acc_bar = bar_base + 8u * (2 * kSplitMaxStages);
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(smem_gen + kSplitRingBytes + 8 * (2 * kSplitMaxStages + 1));
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_holder + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int rank = splits > 1 ? (int)cluster_ctarank() : 0;
  const int tile = blockIdx.x / splits;
  const int num_k = (p.K + kGemmBlockK - 1) / kGemmBlockK;
  const int n0 = tile * BN;
  const int kb0 = num_k * rank / splits, kb1 = num_k * (rank + 1) / splits;

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int s = 0; s < stages; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), 1);
    }
    mbar_init(acc_bar, 1);
    fence_mbar_init();
    tma_prefetch_desc(&tmap_a);
    tma_prefetch_desc(&tmap_b);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_holder), BN);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_holder;

  if (warp == 0) {
    const uint32_t lead = elect_one() ? 1u : 0u;   // warp-uniform loop: one elected lane's copies take effect (see umma_f16_ss_p)
    int stage = 0;
    uint32_t phase = 0;
    for (int kb = kb0; kb < kb1; ++kb) {
      if (!mbar_wait(empty_bar(stage), phase ^ 1u, abort_flag, p.wait_budget_ns)) {
        if (lane == 0) record_status(p.status, kStatusMbarTimeout, p.kernel_id, p.rank, stage, 11, tile);
        break;
      }
      mbar_expect_tx_p(full_bar(stage), stage_bytes, lead);
      const uint32_t sa = smem_base + stage * stage_bytes;
      tma_load_2d_p(sa, &tmap_a, full_bar(stage), kb * kGemmBlockK, 0, lead);
      if constexpr (B_MN) {
        tma_load_2d_p(sa + a_bytes, &tmap_b, full_bar(stage), n0, kb * kGemmBlockK, lead);
        tma_load_2d_p(sa + a_bytes + 8192, &tmap_b, full_bar(stage), n0 + 64, kb * kGemmBlockK, lead);
      } else {
        tma_load_2d_p(sa + a_bytes, &tmap_b, full_bar(stage), kb * kGemmBlockK, n0, lead);
      }
      if (++stage == stages) {
        stage = 0;
        phase ^= 1u;
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    const uint32_t lead = elect_one() ? 1u : 0u;
    constexpr uint32_t idesc = make_idesc(kGemmBlockM, BN, 1, 1, 0, B_MN ? 1 : 0);
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int kb = kb0; kb < kb1; ++kb) {
      if (!mbar_wait(full_bar(stage), phase, abort_flag, p.wait_budget_ns)) {
        if (lane == 0) record_status(p.status, kStatusMbarTimeout, p.kernel_id, p.rank, stage, 21, tile);
        ok = false;
        break;
      }
      tc_fence_after_sync();
      const uint32_t sa = smem_base + stage * stage_bytes;
      const uint32_t a_lo = smem_desc_lo_kmajor(sa);
      const uint32_t b_lo = B_MN ? smem_desc_lo_mnmajor(sa + a_bytes, 8192u) : smem_desc_lo_kmajor(sa + a_bytes);
#pragma unroll
      for (int k = 0; k < kGemmBlockK / 16; ++k)
        umma_f16_ss_p(tmem_base, smem_desc_join(a_lo + 2u * k), smem_desc_join(b_lo + (B_MN ? 128u : 2u) * k), idesc,
                      (kb != kb0 || k != 0) ? 1u : 0u, lead);
      umma_commit_p(empty_bar(stage), lead);
      if (++stage == stages) {
        stage = 0;
        phase ^= 1u;
      }
    }
    if (ok) umma_commit_p(acc_bar, lead);
    __syncwarp();
  } else {
    const int q = warp & 3;
    bool ok = mbar_wait(acc_bar, 0, abort_flag, p.wait_budget_ns);
    ok = __all_sync(0xffffffffu, ok);
    if (!ok) {
      if (lane == 0) record_status(p.status, kStatusMbarTimeout, p.kernel_id, p.rank, 0, 30, tile);
    } else if (q * 32 < p.M) {
      tc_fence_after_sync();
      const int r_in_tile = q * 32 + lane;
#pragma unroll 1
      for (int c = 0; c < BN && n0 + c < p.N; c += 32) {
        uint32_t r[32];
        tmem_ld_32x32(tmem_base + (static_cast<uint32_t>(q * 32) << 16) + c, r);
        tmem_ld_wait();
        if (splits == 1) {
#pragma unroll
          for (int j = 0; j < 32; j += 8) {
            float v[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[j + i]);
            split_store<EPI, OUT_F32>(p, r_in_tile, n0 + c + j, v);
          }
        } else {          // a row of partial sums; the ring is free once the last MMA has completed
          const uint32_t dst = smem_base + static_cast<uint32_t>(r_in_tile * kSplitPitch + c * 4);
#pragma unroll
          for (int j = 0; j < 32; j += 4)
            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst + j * 4), "r"(r[j]), "r"(r[j + 1]), "r"(r[j + 2]), "r"(r[j + 3])
                         : "memory");
        }
      }
      tc_fence_before_sync();
    }
  }
  __syncthreads();
  const bool failed = *abort_flag != 0;
  if (splits > 1) {
    cluster_sync_all();                  // every CTA's partial sums are in its shared memory
    // this CTA's columns of the tile, four per thread: 32 / splits threads side by side on a row
    const int per_row = BN / 4 / splits;
    for (int i = threadIdx.x; !failed && i < p.M * per_row; i += kGemmThreads) {
      const int r = i / per_row, c = (rank * per_row + i - r * per_row) * 4;
      const uint32_t src = smem_base + static_cast<uint32_t>(r * kSplitPitch + c * 4);
      float4 part[8];
#pragma unroll
      for (int s = 0; s < 8; ++s)
        if (s < splits) part[s] = ld_shared_cluster_v4(mapa_shared(src, s));
      float v[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int s = 0; s < 8; ++s)
        if (s < splits) { v[0] += part[s].x; v[1] += part[s].y; v[2] += part[s].z; v[3] += part[s].w; }
      split_store<EPI, OUT_F32>(p, r, n0 + c, v);
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (failed) {
    // give copies that are still in flight time to land before the shared memory is released
    const uint64_t t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
    __syncthreads();
  }
  if (splits > 1) cluster_sync_all();    // nobody's shared memory goes away while a peer still reads it
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, BN);
  }
}

}  // namespace pkb
