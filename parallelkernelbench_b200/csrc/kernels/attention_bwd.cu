// Flash-attention backward on tcgen05 / TMEM.
//
// One CTA, or several that share the walk (see fa_bwd_splits), owns one 128-row KV tile of one KV head and walks every (query head
// of the group, 128-row Q tile) pair that can see it. Per pair, from the saved forward (O, log-sum-exp):
//     S  = Q K^T                         (tensor core, TMEM)
//     dP = dO V^T                        (tensor core, TMEM)
//     P  = exp2(S * scale * log2e - lse2)            dS = P * (dP - delta) * scale     (softmax warps, thread = q row)
//     dV += P^T dO     dK += dS^T Q      (tensor core, accumulate in TMEM over the whole walk, GQA summed)
//     dQ_partial = dS K                  (tensor core, into the TMEM columns dP has just left) -> tiled fp32 TMA reduction into dQ
// A step's products run under the computations of the P / dS warps: dP under P, dV and the next step's S under dS, dQ and dK
// under the next P. For that P and dS share one buffer (each waits for the products that read the other), which makes room for
// a second Q stage, and dQ takes the columns of dP instead of those of S. Cycles per step (device-side trace, S = 16384, 32 / 8
// heads): 4440 at d = 128 and 4000 at d = 64; 5890 and 5000 with one buffer of each and S, dP before and dV, dK, dQ behind the
// computation. What is left is the chain of P (1750 cycles), dP, dS (1290); the drain
// of dQ (3500 cycles at d = 128: 64 KiB of fp32 additions per step and SM) comes next.
// Whole backward: S = 16384 d = 128 6.86 -> 5.2 ms (1059 TFLOP/s), d = 64 5.62 -> 4.1 ms, S = 4096 d = 128 742 -> 372 us.
// delta = rowsum(dO * O) and lse2 = lse * log2e come from a small pre-kernel.
//
//   warp 0      TMA producer: K_j, V_j once; Q_i and dO_i per step
//   warp 1      MMA issuer
//   warps 4-11  softmax / dS (thread = q row; warps 4-7 take KV columns 0-63, warps 8-11 columns 64-127): P from S, then dS
//               from dP, written as bf16 into 128-byte-swizzled shared memory; the same [q][kv] tiles serve as K-major A
//               (dS for dQ) and as MN-major A (P^T, dS^T)
//   warps 12-15 dQ drain (thread = q row), and at the end dV, dK (see share_sums where several CTAs share a tile)
// dK and dV are the same bits on every call; dQ is added up in the order in which the KV tiles get there.
// K_j ([kv][d]) is the K-major B operand of S and the MN-major B operand of dQ; Q_i and dO_i are K-major A operands of
// S / dP and MN-major B operands of dK / dV: every tile is loaded once and read through two descriptors.
//
// Positions follow the forward kernel's segment description, so causal masks in context-parallel (zigzag) layouts are
// exact. Reference behaviour replaced: materialised fp32 scores and their softmax per ring step
// (reference: reference/57_ring_attention_backward_dp.py:39-69).
#include <array>
#include <type_traits>

#include "pkb/api.h"
#include "pkb/attention_api.h"
#include "pkb/host.h"
#include "pkb/ptx.cuh"

namespace pkb {

constexpr int kFbThreads = 512;
constexpr int kFbTile = 128;
constexpr float kFbLog2e = 1.4426950408889634f;
// register budgets after the prologue (the kernel is compiled for 128 per thread: 512 x 128 = the whole file)
constexpr int kFbRegsIo = 72, kFbRegsSoftmax = 144, kFbRegsDrain = 152;
static_assert(128 * kFbRegsIo + 256 * kFbRegsSoftmax + 128 * kFbRegsDrain <= 65536, "register budgets exceed the register file");

struct FaBwdParams {
  pkb_attn_desc d;
  const float* lse2;    // [batch, hq, sq]  log-sum-exp in base-2 units
  const float* delta;   // [batch, hq, sq]  rowsum(dO * O)
  float* dk;            // [batch * skv, hkv, D] fp32
  float* dv;            // [batch * skv, hkv, D] fp32
  // Context-parallel form: when seg_scatter != 0 the dK / dV rows of KV segment s are ADDED (fp32 vector reductions) into
  // dk_seg[s] / dv_seg[s], which point at row 0 of that segment inside the accumulator of the rank that owns the rows -
  // peer memory for remote segments, so the partial sums go home from the epilogue instead of through a reduce-scatter.
  int seg_scatter;
  float* dk_seg[16];
  float* dv_seg[16];
  // splits > 1: two clusters of splits / 2 CTAs share the walk of a KV tile. The dK / dV of a cluster meet in shared memory, the two
  // clusters ADD theirs to the zeroed buffers (0 + a + b is the same in either order, so the result does not depend on timing).
  int splits;
  uint32_t* status;
  uint64_t budget_ns;
  long long* trace;     // optional: CTA (0,0,0) stamps clock64 at its hand-overs (see fb_trace)
};

// Device-side trace: a plain store into the slot of (role, step, event); roles 0 issuing warp, 1 P / dS warps (first warp),
// 2 dQ drain warps (first warp). Layout: [3 roles][kFbTraceSteps][8 events] int64.
constexpr int kFbTraceSteps = 160;
__device__ __forceinline__ void fb_trace(const FaBwdParams& p, int role, int event, int step) {
  if (p.trace == nullptr || blockIdx.x != 0 || blockIdx.y != 0 || blockIdx.z != 0 || step >= kFbTraceSteps) return;
  long long t;
  asm volatile("mov.u64 %0, %%clock64;" : "=l"(t)::"memory");
  p.trace[(role * kFbTraceSteps + step) * 8 + event] = t;
}

template <int D>
struct FbSmem {
  static constexpr int kTileBytes = kFbTile * D * 2;
  static constexpr int kPBytes = kFbTile * kFbTile * 2;
  static constexpr int kK = 0;
  static constexpr int kV = kK + kTileBytes;
  static constexpr int kQ = kV + kTileBytes;               // two stages
  static constexpr int kDO = kQ + 2 * kTileBytes;
  static constexpr int kPDS = kDO + kTileBytes;            // P of a step, then its dS
  // dQ staging, 8 KiB per drain warp: two boxes of 32 rows x 32 fp32 columns (128-byte swizzle). A buffer of its own, so that
  // the reductions of step s run under the products and the P / dS computation of step s+1.
  static constexpr int kDqStage = kPDS + kPBytes;
  // a shared tile's partial dV and dK, fp32, over the operand tiles of the finished walk; 16-byte accesses of 8 rows hit all banks
  static constexpr int kPartPitch = D * 4 + 16;
  static constexpr int kPartBytes = kFbTile * kPartPitch;
  static_assert(2 * kPartBytes <= kPDS, "partial sums outgrew the operand tiles");
  static constexpr int kBars = kDqStage + 4 * 8192;
  static constexpr int kTotal = kBars + 320;
  static_assert(kTotal <= 232448, "shared-memory plan exceeds the 227 KiB a CTA may use");
};

// delta[b,h,s] = sum_d dO * O ; lse2 = lse * log2(e); dQ (and, where they are added to or not fully written, dK and dV) are
// zero-filled on the way. Memory bound: D / 8 lanes per (head, position) with 16-byte accesses, positions fastest, so that
// delta, lse and lse2 are runs of memory.
template <int D>
__global__ void __launch_bounds__(256)
fa_bwd_prep_kernel(const __nv_bfloat16* __restrict__ o, const __nv_bfloat16* __restrict__ dout, const float* __restrict__ lse,
                   float* __restrict__ delta, float* __restrict__ lse2, float* __restrict__ dq, float* __restrict__ dk,
                   float* __restrict__ dv, long long kv_elems, int batch, int sq, int hq) {
  constexpr int L = D / 8;
  const int l = threadIdx.x % L;
  const long long first = ((long long)blockIdx.x * blockDim.x + threadIdx.x) / L;
  const long long stride = ((long long)gridDim.x * blockDim.x) / L;
  const long long total = (long long)batch * sq * hq;
  const U4 zero{0u, 0u, 0u, 0u};
  for (long long base = first - (threadIdx.x & 31) / L; base < total; base += stride) {   // the same for all lanes of a warp
    const long long i = base + (threadIdx.x & 31) / L;
    float acc = 0.f;
    if (i < total) {
      const long long bh = i / sq;
      const int s = (int)(i - bh * sq);
      const long long b = bh / hq;
      const long long row = ((b * sq + s) * hq + (bh - b * hq)) * D;
      const U4 x = ld_global_nc_v4(o + row + l * 8), y = ld_global_nc_v4(dout + row + l * 8);
      const uint32_t xw[4] = {x.x, x.y, x.z, x.w}, yw[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 f = unpack_bf16x2(xw[j]), g = unpack_bf16x2(yw[j]);
        acc = fmaf(f.x, g.x, acc);
        acc = fmaf(f.y, g.y, acc);
      }
      st_global_v4(dq + row + l * 4, zero);
      st_global_v4(dq + row + D / 2 + l * 4, zero);
    }
#pragma unroll
    for (int m = L / 2; m > 0; m >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, m);
    if (l == 0 && i < total) {
      delta[i] = acc;
      lse2[i] = lse[i] * kFbLog2e;
    }
  }
  if (kv_elems > 0) {
    const long long n4 = kv_elems / 4;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += (long long)gridDim.x * blockDim.x) {
      st_global_v4(dk + i * 4, zero);
      st_global_v4(dv + i * 4, zero);
    }
  }
}

__device__ __forceinline__ void red_add_v4_f32(float* p, float a, float b, float c, float d) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}

// Position of Q row `row` (inside one batch entry) and whether the 128-row tile starting there can see kv position kp0.
__device__ __forceinline__ int fb_q_pos(const pkb_attn_desc& d, int row) {
  const int seg = row / d.q_seg_rows;
  return d.q_seg_pos[seg] + (row - seg * d.q_seg_rows);
}

template <int D, bool TRACE = false>
__global__ void __launch_bounds__(kFbThreads, 1)
fa_bwd_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
              const __grid_constant__ CUtensorMap tmap_v, const __grid_constant__ CUtensorMap tmap_do,
              const __grid_constant__ CUtensorMap tmap_dq, const FaBwdParams p) {
  using S = FbSmem<D>;
  constexpr int kAtoms = D / 64;
  constexpr int kAtomBytes = kFbTile * 128;
  extern __shared__ __align__(1024) uint8_t smem[];
  const uint32_t sb = smem_u32(smem);
  const pkb_attn_desc& d = p.d;

  const uint32_t bar0 = sb + S::kBars;
  const uint32_t kv_full = bar0;
  auto q_full = [&](int st) { return bar0 + 8u * (1 + st); };
  auto q_empty = [&](int st) { return bar0 + 8u * (3 + st); };   // dK complete: the last reader of Q
  const uint32_t do_full = bar0 + 40;
  const uint32_t do_empty = bar0 + 48;    // dV complete: the last reader of dO and of P
  const uint32_t s_full = bar0 + 56;      // S in TMEM
  const uint32_t dp_full = bar0 + 64;     // dP in TMEM
  const uint32_t p_full = bar0 + 72;      // P in shared memory, S read out of TMEM
  const uint32_t ds_full = bar0 + 80;     // dS in shared memory, dP read out of TMEM
  const uint32_t dq_full = bar0 + 88;     // dQ partial in TMEM
  const uint32_t dq_empty = bar0 + 96;    // dQ partial drained: the dP columns may be overwritten
  const uint32_t acc_full = bar0 + 104;   // dV and dK final
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(smem + S::kBars + 8 * 14);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_holder + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int rep = d.hq / d.hkv;
  // x: (batch, KV head, split), y: KV tile. x runs fastest, so the heavy tiles of all heads are started before any light one. The
  // first and the second half of a tile's splits are a cluster each.
  const int split = blockIdx.x % p.splits;
  const int kv_head = (blockIdx.x / p.splits) % d.hkv;
  const int batch = blockIdx.x / (p.splits * d.hkv);

  // which KV tile: heavy tiles (early positions see the most queries under a causal mask) come first in launch order
  int kv_row0 = 0, kv_pos0 = 0, kv_valid = 0, kv_seg = 0, kv_row_in_seg = 0;
  {
    int t = blockIdx.y;
    bool found = false;
    for (int seg = 0; seg < d.num_kv_segs && !found; ++seg) {
      const int nt = (d.kv_seg_len[seg] + kFbTile - 1) / kFbTile;
      if (t < nt) {
        kv_seg = seg;
        kv_row_in_seg = t * kFbTile;
        kv_row0 = d.kv_seg_row0[seg] + t * kFbTile;
        kv_pos0 = d.kv_seg_pos0[seg] + t * kFbTile;
        kv_valid = min(kFbTile, d.kv_seg_len[seg] - t * kFbTile);
        found = true;
      }
      t -= nt;
    }
    if (!found) return;   // uniform over the CTA: nothing allocated yet
  }
  // Active Q tiles: inside a segment positions grow, so under a causal mask the tiles that can see this KV tile are a
  // suffix of every segment. seg_first / seg_cnt (shared memory, filled below) turn a step index into a tile in O(segments).
  int* seg_first = reinterpret_cast<int*>(smem + S::kBars + 8 * 16);
  int* seg_cnt = seg_first + 16;
  int* n_active_s = seg_cnt + 16;
  const int tiles_per_seg = d.num_q_segs == 1 ? (d.sq + kFbTile - 1) / kFbTile : d.q_seg_rows / kFbTile;
  const int rows_per_seg = d.num_q_segs == 1 ? d.sq : d.q_seg_rows;
  if (threadIdx.x == 0) {
    int total = 0;
    for (int sg = 0; sg < d.num_q_segs; ++sg) {
      int first = 0;
      if (d.causal) {
        while (first < tiles_per_seg && d.q_seg_pos[sg] + min(first * kFbTile + kFbTile, rows_per_seg) - 1 < kv_pos0) ++first;
      }
      seg_first[sg] = first;
      seg_cnt[sg] = tiles_per_seg - first;
      total += tiles_per_seg - first;
    }
    *n_active_s = total;
  }
  if (threadIdx.x == 0) {
    *abort_flag = 0;
    if ((sb & 1023u) != 0) {
      *abort_flag = 1;
      record_status(p.status, kStatusBadArgument, 650, 0, 0, 1, 0);
    }
    mbar_init(kv_full, 1);
    for (int st = 0; st < 2; ++st) {
      mbar_init(q_full(st), 1);
      mbar_init(q_empty(st), 1);
    }
    mbar_init(do_full, 1);
    mbar_init(do_empty, 1);
    mbar_init(s_full, 1);
    mbar_init(dp_full, 1);
    mbar_init(p_full, 8);
    mbar_init(ds_full, 8);
    mbar_init(dq_full, 1);
    mbar_init(dq_empty, 4);
    mbar_init(acc_full, 1);
    fence_mbar_init();
    tma_prefetch_desc(&tmap_q);
    tma_prefetch_desc(&tmap_k);
    tma_prefetch_desc(&tmap_v);
    tma_prefetch_desc(&tmap_do);
    tma_prefetch_desc(&tmap_dq);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_holder), 512);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const int n_active = *n_active_s;
  const int step0 = (int)((long long)n_active * rep * split / p.splits);
  const int n_steps = (int)((long long)n_active * rep * (split + 1) / p.splits) - step0;
  const uint32_t tmem_base = *tmem_holder;
  const uint32_t tmem_s = tmem_base;
  const uint32_t tmem_dp = tmem_base + 128;   // dP, then the dQ partial (D columns)
  const uint32_t tmem_dv = tmem_base + 256;
  const uint32_t tmem_dk = tmem_base + 256 + D;
  const bool bad = *abort_flag != 0;
  const int kv_tok0 = batch * d.skv + kv_row0;

  // the walk over (query head, q tile): heads outer, active tiles inner. A role keeps the index of its next tile and the head.
  struct Walk { int head, k; };
  auto walk_begin = [&]() { return Walk{kv_head * rep + (n_active > 0 ? step0 / n_active : 0), n_active > 0 ? step0 % n_active : 0}; };
  auto walk_next = [&](Walk& w, int& head, int& qt) {
    head = w.head;
    int k = w.k;
    qt = 0;
    for (int sg = 0; sg < d.num_q_segs; ++sg) {
      if (k < seg_cnt[sg]) {
        qt = sg * tiles_per_seg + seg_first[sg] + k;
        break;
      }
      k -= seg_cnt[sg];
    }
    if (++w.k == n_active) {
      w.k = 0;
      ++w.head;
    }
  };

  // Sums of a shared tile: each CTA of the cluster holds the dV and dK of its part of the walk in shared memory, adds up its share of
  // the rows over the CTAs in the order of their ranks and adds the sum to the result. Every thread of the cluster meets at the two
  // barriers, whatever it waited for in vain before; `t`, `threads`: the threads that add.
  const int csize = p.splits > 1 ? p.splits >> 1 : 1;
  auto share_sums = [&](int t, int threads) {
    cluster_sync_all();                  // every CTA's partial sums are in its shared memory
    constexpr int kPerRow = D / 4;
    const int rank = split % csize;
    uint32_t has = 0;                    // ranks whose part of the walk is not empty
    for (int c = 0; c < csize; ++c) {
      const long long total = (long long)n_active * rep, first = split - rank + c;
      if (total * (first + 1) / p.splits > total * first / p.splits) has |= 1u << c;
    }
    const int i_begin = 2 * kv_valid * kPerRow * rank / csize, i_end = 2 * kv_valid * kPerRow * (rank + 1) / csize;
    // ITEMS x RANKS loads of a thread are in flight together
    auto add_up = [&](auto items, auto ranks) {
      constexpr int ITEMS = decltype(items)::value, RANKS = decltype(ranks)::value;
      for (int i0 = i_begin + t; i0 < i_end; i0 += ITEMS * threads) {
        float4 part[ITEMS][RANKS];
#pragma unroll
        for (int u = 0; u < ITEMS; ++u) {
          const int i = i0 + u * threads, row2 = i / kPerRow;
          const uint32_t src = sb + (row2 >= kv_valid ? S::kPartBytes + (row2 - kv_valid) * S::kPartPitch : row2 * S::kPartPitch) + (i % kPerRow) * 16;
#pragma unroll
          for (int c = 0; c < RANKS; ++c)
            part[u][c] = i < i_end && ((has >> c) & 1u) ? ld_shared_cluster_v4(mapa_shared(src, c)) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int u = 0; u < ITEMS; ++u) {
          const int i = i0 + u * threads, row2 = i / kPerRow;
          if (i >= i_end) break;
          float4 v = part[u][0];
#pragma unroll
          for (int c = 1; c < RANKS; ++c) { v.x += part[u][c].x; v.y += part[u][c].y; v.z += part[u][c].z; v.w += part[u][c].w; }
          const bool is_dk = row2 >= kv_valid;
          red_add_v4_f32((is_dk ? p.dk : p.dv) + ((static_cast<long long>(kv_tok0) + (is_dk ? row2 - kv_valid : row2)) * d.hkv + kv_head) * D + (i % kPerRow) * 4,
                         v.x, v.y, v.z, v.w);
        }
      }
    };
    if (has != 0) {
      if (csize <= 4) add_up(std::integral_constant<int, 4>{}, std::integral_constant<int, 4>{});
      else add_up(std::integral_constant<int, 2>{}, std::integral_constant<int, 8>{});
    }
    cluster_sync_all();                  // nobody's shared memory goes away while a peer still reads it
  };

  // `work`: false when no query sees this tile (warps 12-15 then store zeros into its dK / dV rows)
  const bool work = !bad && n_steps != 0;
  if (warp < 4) {
    warpgroup_reg_dec<kFbRegsIo>();
    if (warp == 0 && work) {
    // producer: the whole warp walks the loop, one elected lane's copies take effect. Under `if (lane == 0)` the loop would
    // run in divergent code, where addresses cannot live in uniform registers (see umma_f16_ss_p).
    {
      const uint32_t lead = elect_one() ? 1u : 0u;
      mbar_expect_tx_p(kv_full, 2 * S::kTileBytes, lead);
#pragma unroll
      for (int a = 0; a < kAtoms; ++a) {
        tma_load_3d_p(sb + S::kK + a * kAtomBytes, &tmap_k, kv_full, a * 64, kv_head, kv_tok0, lead);
        tma_load_3d_p(sb + S::kV + a * kAtomBytes, &tmap_v, kv_full, a * 64, kv_head, kv_tok0, lead);
      }
      bool ok = true;
      Walk wq = walk_begin(), wdo = walk_begin();
      auto load_q = [&](int step) {
        int head, qt;
        walk_next(wq, head, qt);
        const int st = step & 1;
        if (!mbar_wait(q_empty(st), ((step >> 1) & 1) ^ 1u, abort_flag, p.budget_ns)) { ok = false; return; }
        mbar_expect_tx_p(q_full(st), S::kTileBytes, lead);
#pragma unroll
        for (int a = 0; a < kAtoms; ++a)
          tma_load_3d_p(sb + S::kQ + st * S::kTileBytes + a * kAtomBytes, &tmap_q, q_full(st), a * 64, head, batch * d.sq + qt * kFbTile, lead);
      };
      load_q(0);
      for (int step = 0; step < n_steps && ok; ++step) {
        int head, qt;
        walk_next(wdo, head, qt);
        if (!mbar_wait(do_empty, (step & 1) ^ 1u, abort_flag, p.budget_ns)) { ok = false; break; }
        mbar_expect_tx_p(do_full, S::kTileBytes, lead);
#pragma unroll
        for (int a = 0; a < kAtoms; ++a)
          tma_load_3d_p(sb + S::kDO + a * kAtomBytes, &tmap_do, do_full, a * 64, head, batch * d.sq + qt * kFbTile, lead);
        if (step + 1 < n_steps) load_q(step + 1);
      }
      if (!ok && lane == 0) record_status(p.status, kStatusMbarTimeout, 650, 0, 0, 11, 0);
    }
    __syncwarp();
    } else if (warp == 1 && work) {
    // issuer: warp-uniform loop with prepared descriptor words; one elected lane's tcgen05 instructions take effect
    {
      const uint32_t lead = elect_one() ? 1u : 0u;
      constexpr uint32_t idesc_s = make_idesc(kFbTile, kFbTile, 1, 1, 0, 0);   // S, dP: both operands K-major
      constexpr uint32_t idesc_acc = make_idesc(kFbTile, D, 1, 1, 1, 1);       // dV, dK: A and B MN-major
      constexpr uint32_t idesc_dq = make_idesc(kFbTile, D, 1, 1, 0, 1);        // dQ: A K-major, B MN-major
      // K-major views step 16 along K by 32 bytes inside a 64-column atom (atoms kAtomBytes apart); MN-major views step 16
      // along K by 16 rows of 128 bytes
      const uint32_t q_k = smem_desc_lo_kmajor(sb + S::kQ), k_k = smem_desc_lo_kmajor(sb + S::kK);
      const uint32_t do_k = smem_desc_lo_kmajor(sb + S::kDO), v_k = smem_desc_lo_kmajor(sb + S::kV);
      const uint32_t ds_k = smem_desc_lo_kmajor(sb + S::kPDS);
      const uint32_t k_mn = smem_desc_lo_mnmajor(sb + S::kK, kAtomBytes), pds_mn = smem_desc_lo_mnmajor(sb + S::kPDS, kAtomBytes);
      const uint32_t do_mn = smem_desc_lo_mnmajor(sb + S::kDO, kAtomBytes);
      const uint32_t q_mn = smem_desc_lo_mnmajor(sb + S::kQ, kAtomBytes);
      constexpr uint32_t kQStep = S::kTileBytes >> 4;
      auto issue_s = [&](int step) {
        const int st = step & 1;
        if (!mbar_wait(q_full(st), (step >> 1) & 1, abort_flag, p.budget_ns)) return false;
        tc_fence_after_sync();
#pragma unroll
        for (int k = 0; k < D / 16; ++k) {
          const uint32_t off = ((k >> 2) * kAtomBytes + (k & 3) * 32) >> 4;
          umma_f16_ss_p(tmem_s, smem_desc_join(q_k + st * kQStep + off), smem_desc_join(k_k + off), idesc_s, k != 0, lead);
        }
        umma_commit_p(s_full, lead);
        return true;
      };
      bool ok = mbar_wait(kv_full, 0, abort_flag, p.budget_ns) && issue_s(0);
      for (int step = 0; step < n_steps && ok; ++step) {
        const uint32_t ph = step & 1;
        if constexpr (TRACE) { if (lane == 0) fb_trace(p, 0, 0, step); }
        // dP, under the computation of P
        if (!mbar_wait(do_full, ph, abort_flag, p.budget_ns)) { ok = false; break; }
        if constexpr (TRACE) { if (lane == 0) fb_trace(p, 0, 1, step); }
        if (!mbar_wait(dq_empty, ph ^ 1u, abort_flag, p.budget_ns)) { ok = false; break; }
        if constexpr (TRACE) { if (lane == 0) fb_trace(p, 0, 2, step); }
        tc_fence_after_sync();
#pragma unroll
        for (int k = 0; k < D / 16; ++k) {
          const uint32_t off = ((k >> 2) * kAtomBytes + (k & 3) * 32) >> 4;
          umma_f16_ss_p(tmem_dp, smem_desc_join(do_k + off), smem_desc_join(v_k + off), idesc_s, k != 0, lead);
        }
        umma_commit_p(dp_full, lead);
        if constexpr (TRACE) { if (lane == 0) fb_trace(p, 0, 3, step); }
        // dV += P^T dO (K dimension = the 128 q rows, 16 per instruction = 2048 bytes of a [row][128 B] atom) and the next step's S,
        // under the computation of dS
        const uint32_t acc0 = step != 0;
        if (!mbar_wait(p_full, ph, abort_flag, p.budget_ns)) { ok = false; break; }
        if constexpr (TRACE) { if (lane == 0) fb_trace(p, 0, 4, step); }
        tc_fence_after_sync();
#pragma unroll
        for (int k = 0; k < kFbTile / 16; ++k)
          umma_f16_ss_p(tmem_dv, smem_desc_join(pds_mn + k * (2048 >> 4)), smem_desc_join(do_mn + k * (2048 >> 4)), idesc_acc,
                        k != 0 ? 1u : acc0, lead);
        umma_commit_p(do_empty, lead);
        if (step + 1 < n_steps && !issue_s(step + 1)) { ok = false; break; }
        if (!mbar_wait(ds_full, ph, abort_flag, p.budget_ns)) { ok = false; break; }
        if constexpr (TRACE) { if (lane == 0) fb_trace(p, 0, 5, step); }
        tc_fence_after_sync();
        // dQ partial = dS K_j (K dimension = the 128 kv rows), into the columns that held dP: first, because its drain has to end
        // before the next dP; then dK += dS^T Q. Both under the computation of the next P.
#pragma unroll
        for (int k = 0; k < kFbTile / 16; ++k) {
          const uint32_t aoff = ((k >> 2) * kAtomBytes + (k & 3) * 32) >> 4;
          umma_f16_ss_p(tmem_dp, smem_desc_join(ds_k + aoff), smem_desc_join(k_mn + k * (2048 >> 4)), idesc_dq, k != 0, lead);
        }
        umma_commit_p(dq_full, lead);
#pragma unroll
        for (int k = 0; k < kFbTile / 16; ++k)
          umma_f16_ss_p(tmem_dk, smem_desc_join(pds_mn + k * (2048 >> 4)), smem_desc_join(q_mn + ph * kQStep + k * (2048 >> 4)), idesc_acc,
                        k != 0 ? 1u : acc0, lead);
        umma_commit_p(q_empty(ph), lead);
        if constexpr (TRACE) { if (lane == 0) fb_trace(p, 0, 6, step); }
      }
      if (ok) umma_commit_p(acc_full, lead);
      else if (lane == 0) record_status(p.status, kStatusMbarTimeout, 650, 0, 0, 20, 0);
    }
    __syncwarp();
    }
    if (csize > 1) {                     // the two barriers of share_sums
      cluster_sync_all();
      cluster_sync_all();
    }
  } else if (warp < 12) {
    warpgroup_reg_inc<kFbRegsSoftmax>();
    // ------------------------------ P and dS (thread = q row, half of the KV columns) ------------------------------
    const int q4 = warp & 3;
    const int c_begin = (warp >= 8) ? 2 : 0;      // 32-column chunks handled by this warpgroup
    const int row = q4 * 32 + lane;
    const float scale2 = d.scale * kFbLog2e;
    bool ok = work;
    // lse2 and delta of the next step are requested in the middle of this one: read at the start of a step they cost it their
    // latency, about 1000 of 4850 cycles
    Walk w = walk_begin();
    int next_row;
    float next_lse2, next_delta;
    auto fetch = [&]() {
      int head, qt;
      walk_next(w, head, qt);
      next_row = qt * kFbTile + row;
      next_lse2 = 0.f;
      next_delta = 0.f;
      if (next_row < d.sq) {
        const long long i = ((long long)batch * d.hq + head) * d.sq + next_row;
        next_lse2 = p.lse2[i];
        next_delta = p.delta[i];
      }
    };
    if (work) fetch();
    for (int step = 0; step < n_steps && ok; ++step) {
      const uint32_t ph = step & 1;
      const int q_row = next_row;
      const float lse2 = next_lse2, delta = next_delta;
      const bool row_ok = q_row < d.sq;
      const int my_pos = row_ok ? fb_q_pos(d, q_row) : -1;
      const bool row_dead = !row_ok || lse2 == -INFINITY;
      const bool need_mask = row_dead || kv_valid < kFbTile || (d.causal && kv_pos0 + kFbTile - 1 > my_pos);
      if constexpr (TRACE) { if (warp == 4 && lane == 0) fb_trace(p, 1, 0, step); }
      // Two halves: P from S, then dS from dP. They share a buffer, so each waits for the products that read the other.
      ok = mbar_wait(s_full, ph, abort_flag, p.budget_ns);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      if constexpr (TRACE) { if (warp == 4 && lane == 0) fb_trace(p, 1, 1, step); }
      tc_fence_after_sync();
      const uint32_t lane_off = static_cast<uint32_t>(q4 * 32) << 16;
      const uint32_t pds_row = sb + S::kPDS + static_cast<uint32_t>(row) * 128u;
      auto store_chunk = [&](int c, const float* v) {     // 32 columns of this row, bf16, 128-byte swizzle
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          const int chunk = c * 4 + g;
          const uint32_t dst = pds_row + (chunk >> 3) * kAtomBytes + (static_cast<uint32_t>((chunk & 7) ^ (row & 7)) << 4);
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst), "r"(pack_bf16x2(v[8 * g], v[8 * g + 1])),
                       "r"(pack_bf16x2(v[8 * g + 2], v[8 * g + 3])), "r"(pack_bf16x2(v[8 * g + 4], v[8 * g + 5])),
                       "r"(pack_bf16x2(v[8 * g + 6], v[8 * g + 7]))
                       : "memory");
        }
      };
      float pv[64];
#pragma unroll
      for (int cc = 0; cc < 2; ++cc) {
        const int c = c_begin + cc;
        uint32_t rs[32];
        tmem_ld_32x32(tmem_s + lane_off + c * 32, rs);
        tmem_ld_wait();
        if (!need_mask) {                 // the whole row of this tile is visible: no per-element tests, packed fp32 pairs
          const float neg_lse2 = -lse2;
#pragma unroll
          for (int i = 0; i < 32; i += 2) {
            float x0, x1;
            fma2_bcast(x0, x1, __uint_as_float(rs[i]), __uint_as_float(rs[i + 1]), scale2, neg_lse2);
            pv[cc * 32 + i] = fast_exp2(x0);
            pv[cc * 32 + i + 1] = fast_exp2(x1);
          }
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            const int col = c * 32 + i;
            const bool masked = row_dead || col >= kv_valid || (d.causal && kv_pos0 + col > my_pos);
            pv[cc * 32 + i] = masked ? 0.f : fast_exp2(fmaf(__uint_as_float(rs[i]), scale2, -lse2));
          }
        }
      }
      // dK of the step before is complete when the Q stage it read is free
      if (step > 0) ok = mbar_wait(q_empty(ph ^ 1u), ((step - 1) >> 1) & 1, abort_flag, p.budget_ns);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
#pragma unroll
      for (int cc = 0; cc < 2; ++cc) store_chunk(c_begin + cc, pv + cc * 32);
      tc_fence_before_sync();
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_full);
      if constexpr (TRACE) { if (warp == 4 && lane == 0) fb_trace(p, 1, 2, step); }
      if (step + 1 < n_steps) fetch();
      ok = mbar_wait(dp_full, ph, abort_flag, p.budget_ns);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      if constexpr (TRACE) { if (warp == 4 && lane == 0) fb_trace(p, 1, 3, step); }
      tc_fence_after_sync();
#pragma unroll
      for (int cc = 0; cc < 2; ++cc) {
        const int c = c_begin + cc;
        uint32_t rd[32];
        tmem_ld_32x32(tmem_dp + lane_off + c * 32, rd);
        tmem_ld_wait();
        float dsv[32];
        if (!need_mask) {
          const float neg_ds = -delta * d.scale;
#pragma unroll
          for (int i = 0; i < 32; i += 2) {
            float t0, t1;
            fma2_bcast(t0, t1, __uint_as_float(rd[i]), __uint_as_float(rd[i + 1]), d.scale, neg_ds);   // (dP - delta) * scale
            mul2(dsv[i], dsv[i + 1], pv[cc * 32 + i], pv[cc * 32 + i + 1], t0, t1);
          }
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) dsv[i] = pv[cc * 32 + i] * (__uint_as_float(rd[i]) - delta) * d.scale;
        }
        if (cc == 0) {
          ok = mbar_wait(do_empty, ph, abort_flag, p.budget_ns);   // dV of this step has read P
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
        }
        store_chunk(c, dsv);
      }
      if (!ok) break;
      tc_fence_before_sync();
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(ds_full);
      if constexpr (TRACE) { if (warp == 4 && lane == 0) fb_trace(p, 1, 4, step); }
    }
    if (!ok && work && lane == 0) record_status(p.status, kStatusMbarTimeout, 650, 0, 0, 30, 0);
    __syncwarp();
    if (csize > 1) share_sums(threadIdx.x - 128, 384);
  } else {
    // ------------------------------ dQ drain, then dV / dK (thread = row) ------------------------------
    warpgroup_reg_inc<kFbRegsDrain>();
    const int q4 = warp & 3;
    const int row = q4 * 32 + lane;
    constexpr int DH = D;
    const int col0 = 0;
    const uint32_t lane_off = static_cast<uint32_t>(q4 * 32) << 16;
    bool ok = !bad;
    Walk w = walk_begin();
    for (int step = 0; step < n_steps && ok; ++step) {
      int head, qt;
      walk_next(w, head, qt);
      if constexpr (TRACE) { if (warp == 12 && lane == 0) fb_trace(p, 2, 0, step); }
      ok = mbar_wait(dq_full, step & 1, abort_flag, p.budget_ns);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      if constexpr (TRACE) { if (warp == 12 && lane == 0) fb_trace(p, 2, 1, step); }
      tc_fence_after_sync();
      // The partial is added to the fp32 dQ in global memory by tiled TMA reductions, a box of 32 x 32 per request. Requests are
      // what a reduction by rows is bound by: 256 of them per step took 4100 to 4700 cycles, with 128 bytes each (d = 64) as with
      // 256 (d = 128). The whole row is read
      // first, so that tensor memory is free for the next dP.
      const uint32_t stg = sb + S::kDqStage + static_cast<uint32_t>(warp - 12) * 8192u;
      const int q_tok = batch * d.sq + qt * kFbTile + q4 * 32;
      const bool any_row = qt * kFbTile + q4 * 32 < d.sq, row_in = qt * kFbTile + row < d.sq;
      auto stage_box = [&](const uint32_t* r, int c) {     // columns 32 c .. of this warp's rows
        const uint32_t row_addr = stg + (c & 1) * 4096u + static_cast<uint32_t>(lane) * 128u;
#pragma unroll
        for (int j = 0; j < 8; ++j)
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(row_addr + (static_cast<uint32_t>(j ^ (lane & 7)) << 4)), "r"(r[4 * j]),
                       "r"(r[4 * j + 1]), "r"(r[4 * j + 2]), "r"(r[4 * j + 3])
                       : "memory");
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          if (any_row) tma_reduce_add_3d(&tmap_dq, stg + (c & 1) * 4096u, c * 32, head, q_tok);
          tma_store_commit();
        }
      };
      uint32_t r[D];
#pragma unroll
      for (int c = 0; c < D; c += 32) tmem_ld_32x32(tmem_dp + lane_off + c, *reinterpret_cast<uint32_t (*)[32]>(&r[c]));
      tmem_ld_wait();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(dq_empty);
      if (!row_in) {       // may be rows of the next sequence of the batch: add zeros, whatever this sequence's K holds
#pragma unroll
        for (int i = 0; i < D; ++i) r[i] = 0u;
      }
#pragma unroll
      for (int h = 0; h < D / 64; ++h) {
        if (lane == 0) tma_store_wait_read<0>();           // the boxes staged before have been read
        __syncwarp();
        stage_box(r + h * 64, 2 * h);
        stage_box(r + h * 64 + 32, 2 * h + 1);
      }
      if constexpr (TRACE) { if (warp == 12 && lane == 0) fb_trace(p, 2, 2, step); }
    }
    if (lane == 0) tma_store_wait_all<0>();   // every reduction of this warp has been performed
    __syncwarp();
    if (ok && n_steps > 0) {
      ok = mbar_wait(acc_full, 0, abort_flag, p.budget_ns);
      ok = __all_sync(0xffffffffu, ok);
      if (ok) tc_fence_after_sync();
    }
    if (ok) {
      // rows of dV / dK are the KV rows of this tile
      const bool add = p.seg_scatter || p.splits > 1;
      const bool row_ok = row < kv_valid && !(add && n_steps == 0);   // nothing to add for a tile no query saw
      float* dvp = p.dv + ((static_cast<long long>(kv_tok0) + row) * d.hkv + kv_head) * D + col0;
      float* dkp = p.dk + ((static_cast<long long>(kv_tok0) + row) * d.hkv + kv_head) * D + col0;
      if (p.seg_scatter) {
        const long long off = (static_cast<long long>(kv_row_in_seg + row) * d.hkv + kv_head) * D + col0;
        dvp = p.dv_seg[kv_seg] + off;
        dkp = p.dk_seg[kv_seg] + off;
      }
      const uint32_t part = sb + static_cast<uint32_t>(row) * S::kPartPitch;
#pragma unroll
      for (int c = 0; c < DH / 32; ++c) {
        uint32_t rv[32], rk[32];
        if (n_steps > 0) {
          tmem_ld_32x32(tmem_dv + lane_off + col0 + c * 32, rv);
          tmem_ld_32x32(tmem_dk + lane_off + col0 + c * 32, rk);
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) { rv[i] = 0u; rk[i] = 0u; }
        }
        if (csize > 1) {                 // for share_sums: the products that read the operand tiles are complete
          if (n_steps > 0) {
#pragma unroll
            for (int i = 0; i < 32; i += 4) {
              asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(part + (c * 32 + i) * 4), "r"(rv[i]), "r"(rv[i + 1]), "r"(rv[i + 2]),
                           "r"(rv[i + 3])
                           : "memory");
              asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(part + S::kPartBytes + (c * 32 + i) * 4), "r"(rk[i]), "r"(rk[i + 1]),
                           "r"(rk[i + 2]), "r"(rk[i + 3])
                           : "memory");
            }
          }
        } else if (row_ok && add) {
#pragma unroll
          for (int i = 0; i < 32; i += 4) {
            red_add_v4_f32(dvp + c * 32 + i, __uint_as_float(rv[i]), __uint_as_float(rv[i + 1]), __uint_as_float(rv[i + 2]),
                           __uint_as_float(rv[i + 3]));
            red_add_v4_f32(dkp + c * 32 + i, __uint_as_float(rk[i]), __uint_as_float(rk[i + 1]), __uint_as_float(rk[i + 2]),
                           __uint_as_float(rk[i + 3]));
          }
        } else if (row_ok) {
#pragma unroll
          for (int i = 0; i < 32; i += 4) {
            st_global_v4(dvp + c * 32 + i, U4{rv[i], rv[i + 1], rv[i + 2], rv[i + 3]});
            st_global_v4(dkp + c * 32 + i, U4{rk[i], rk[i + 1], rk[i + 2], rk[i + 3]});
          }
        }
      }
      // remote additions must have been performed before this rank tells its peers (the barrier launch that follows) that it is done
      if (p.seg_scatter) __threadfence_system();
    } else if (lane == 0 && !bad) {
      record_status(p.status, kStatusMbarTimeout, 650, 0, 0, 40, 0);
    }
    __syncwarp();
    if (csize > 1) share_sums(threadIdx.x - 128, 384);
  }

  tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag) {
    const uint64_t t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, 512);
  }
}

// CTAs per KV tile and head: as many as bring the longest walk (the first KV tile under a causal mask) down to an SM's share of all
// steps; at least two steps each, eight where that makes more CTAs than SMs (a CTA's K and V loads and its dK / dV cost about one
// and a half steps). They are two clusters of at most 8; where all CTAs would fit the SMs, the clusters are made small enough that
// they do so too. d = 128, us on 1 / 2 / 4 / 6 / 8 CTAs per tile: batch 2, S = 1024, 8 / 2 heads, causal (32 tiles) 128 / 66 / 48 / 58 / 58;
// S = 1024, 2 / 1 heads, causal (8 tiles) 87 / 40 / 32 / 30 / 30; S = 1200, 8 / 1 heads, no mask (10 tiles) - / 164 / 95 / 73 / 60 and 52 on
// 12; S = 4096, 16 / 4 heads, causal (128 tiles) 334 / 190. What the fixed order costs: 46 and 44 us for the first and the third
// when every CTA added its sums to memory as it came.
template <int D>
static int fa_bwd_splits(const pkb_attn_desc& d, int kv_tiles) {
  const long long rep = d.hq / d.hkv;
  const long long rows_per_seg = d.num_q_segs == 1 ? d.sq : d.q_seg_rows;
  const long long q_tiles = (rows_per_seg + kFbTile - 1) / kFbTile;
  long long total = 0, longest = 0;          // Q tiles that see a KV tile: all KV tiles of a head, and the most of any one
  for (int s = 0; s < d.num_kv_segs; ++s)
    for (int t = 0; t * kFbTile < d.kv_seg_len[s]; ++t) {
      long long seen = 0;
      for (int q = 0; q < d.num_q_segs; ++q) {
        const long long hidden = d.causal ? ((long long)d.kv_seg_pos0[s] + t * kFbTile - d.q_seg_pos[q]) / kFbTile : 0;
        seen += q_tiles - (hidden < 0 ? 0 : hidden > q_tiles ? q_tiles : hidden);
      }
      total += seen;
      if (seen > longest) longest = seen;
    }
  const long long heads = (long long)d.hkv * d.batch, sms = sm_count();
  if (total == 0) return 1;
  long long s = longest * sms / (total * heads);
  const long long most = longest * rep;
  if (s * kv_tiles * heads > sms && s > most / 8) s = most / 8 > sms / (kv_tiles * heads) ? most / 8 : sms / (kv_tiles * heads);
  if (s > most / 2) s = most / 2;
  if (s < 2) return 1;
  int cluster = s < 16 ? (int)s / 2 : 8;
  static const std::array<int, 9> resident = resident_clusters(fa_bwd_kernel<D, false>, kFbThreads, FbSmem<D>::kTotal);
  if (2 * cluster * kv_tiles * heads <= sms)
    while (cluster > 1 && 2 * kv_tiles * heads > resident[cluster]) --cluster;
  return 2 * cluster;
}

// KV rows of the buffer that lie in a segment (segments may overlap, so their lengths do not add up to it).
static int fa_bwd_covered(const pkb_attn_desc& d) {
  int covered = 0;
  for (int end = 0;;) {                    // `end`: everything below is counted or outside; the next segment piece starts at `from`
    int from = d.skv, to = d.skv;
    for (int s = 0; s < d.num_kv_segs; ++s) {
      const int a = d.kv_seg_row0[s], b = a + d.kv_seg_len[s];
      if (b > end && (a > end ? a : end) < from) { from = a > end ? a : end; to = b; }
    }
    if (from == d.skv) return covered;
    covered += to - from;
    end = to;
  }
}

// Trace buffer of the next backward launches (device memory, 3 * kFbTraceSteps * 8 int64, zeroed by the caller); null = off.
static long long* g_fb_trace = nullptr;

template <int D>
static int launch_fa_bwd(const pkb_attn_desc& d, const void* q, const void* k, const void* v, const void* o, const void* dout,
                         const void* lse, void* delta, void* lse2, void* dq, void* dk, void* dv, cudaStream_t stream,
                         const unsigned long long* dk_seg = nullptr, const unsigned long long* dv_seg = nullptr) {
  CUtensorMap tq, tk, tv, tdo;
  int rc = encode_tmap_3d(&tq, kTmapBf16, q, D, d.hq, (uint64_t)d.batch * d.sq, (uint64_t)D * 2, (uint64_t)d.hq * D * 2, 64, 1,
                          kFbTile, kSwizzle128);
  if (rc) return rc;
  rc = encode_tmap_3d(&tdo, kTmapBf16, dout, D, d.hq, (uint64_t)d.batch * d.sq, (uint64_t)D * 2, (uint64_t)d.hq * D * 2, 64, 1,
                      kFbTile, kSwizzle128);
  if (rc) return rc;
  rc = encode_tmap_3d(&tk, kTmapBf16, k, D, d.hkv, (uint64_t)d.batch * d.skv, (uint64_t)D * 2, (uint64_t)d.hkv * D * 2, 64, 1,
                      kFbTile, kSwizzle128);
  if (rc) return rc;
  rc = encode_tmap_3d(&tv, kTmapBf16, v, D, d.hkv, (uint64_t)d.batch * d.skv, (uint64_t)D * 2, (uint64_t)d.hkv * D * 2, 64, 1,
                      kFbTile, kSwizzle128);
  if (rc) return rc;
  int kv_tiles = 0;
  for (int s = 0; s < d.num_kv_segs; ++s) kv_tiles += (d.kv_seg_len[s] + kFbTile - 1) / kFbTile;
  const bool scatter = dk_seg != nullptr && dv_seg != nullptr;
  const int splits = scatter ? 1 : fa_bwd_splits<D>(d, kv_tiles);
  // every row of dK / dV is written by the main kernel unless rows lie outside all segments or CTAs add to them
  const long long kv_elems = !scatter && (splits > 1 || fa_bwd_covered(d) < d.skv) ? (long long)d.batch * d.skv * d.hkv * D : 0;
  CUtensorMap tdq;
  rc = encode_tmap_3d(&tdq, kTmapFp32, dq, D, d.hq, (uint64_t)d.batch * d.sq, (uint64_t)D * 4, (uint64_t)d.hq * D * 4, 32, 1, 32,
                      kSwizzle128);
  if (rc) return rc;
  const long long rows = (long long)d.batch * d.sq * d.hq;
  long long pblocks = (rows * (D / 8) + 255) / 256;
  if (pblocks > 148 * 16) pblocks = 148 * 16;
  fa_bwd_prep_kernel<D><<<(int)pblocks, 256, 0, stream>>>(static_cast<const __nv_bfloat16*>(o), static_cast<const __nv_bfloat16*>(dout),
                                                          static_cast<const float*>(lse), static_cast<float*>(delta),
                                                          static_cast<float*>(lse2), static_cast<float*>(dq), static_cast<float*>(dk),
                                                          static_cast<float*>(dv), kv_elems, d.batch, d.sq, d.hq);
  PKB_CHECK_CUDA(cudaGetLastError());
  FaBwdParams p;
  p.d = d;
  p.lse2 = static_cast<const float*>(lse2);
  p.delta = static_cast<const float*>(delta);
  p.dk = static_cast<float*>(dk);
  p.dv = static_cast<float*>(dv);
  p.splits = splits;
  p.seg_scatter = scatter ? 1 : 0;
  for (int sg = 0; sg < 16; ++sg) {
    p.dk_seg[sg] = p.seg_scatter && sg < d.num_kv_segs ? reinterpret_cast<float*>(dk_seg[sg]) : nullptr;
    p.dv_seg[sg] = p.seg_scatter && sg < d.num_kv_segs ? reinterpret_cast<float*>(dv_seg[sg]) : nullptr;
  }
  p.status = status_block_device_ptr();
  p.trace = g_fb_trace;
  p.budget_ns = d.budget_ns ? d.budget_ns : kDefaultWaitBudgetNs;
  auto kern = g_fb_trace != nullptr ? fa_bwd_kernel<D, true> : fa_bwd_kernel<D, false>;
  constexpr int smem = FbSmem<D>::kTotal;
  PKB_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  if (kv_tiles == 0) return kApiOk;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(d.hkv * d.batch * splits), (unsigned)kv_tiles);
  cfg.blockDim = dim3(kFbThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)splits / 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = splits > 2 ? 1 : 0;
  PKB_CHECK_CUDA(cudaLaunchKernelEx(&cfg, kern, tq, tk, tv, tdo, tdq, p));
  return kApiOk;
}

}  // namespace pkb

using namespace pkb;

// dq, dk and dv are written whole (rows of dk / dv that no segment covers, or that no query sees, become zero).
extern "C" int pkb_flash_attn_bwd(const pkb_attn_desc* desc, const void* q, const void* k, const void* v, const void* o,
                                  const void* dout, const void* lse, void* delta_scratch, void* lse2_scratch, void* dq,
                                  void* dk, void* dv, void* stream) {
  PKB_CHECK_ARG(desc != nullptr, "null descriptor");
  const pkb_attn_desc& d = *desc;
  PKB_CHECK_ARG(d.head_dim == 64 || d.head_dim == 128, "head_dim must be 64 or 128");
  PKB_CHECK_ARG(d.hq % d.hkv == 0 && d.batch >= 1 && d.sq >= 1 && d.skv >= 1, "bad attention shape");
  PKB_CHECK_ARG(d.num_q_segs >= 1 && d.num_q_segs <= 16 && d.num_kv_segs >= 1 && d.num_kv_segs <= 16, "1..16 segments");
  PKB_CHECK_ARG(d.q_seg_rows % kFbTile == 0 || d.num_q_segs == 1, "q segments must be multiples of 128 rows");
  PKB_CHECK_ARG(d.q_seg_rows >= 1, "q_seg_rows must be positive");
  for (int s = 0; s < d.num_kv_segs; ++s)
    PKB_CHECK_ARG(d.kv_seg_row0[s] >= 0 && d.kv_seg_len[s] >= 0 && d.kv_seg_row0[s] + d.kv_seg_len[s] <= d.skv,
                  "kv segment outside the buffer");
  // the other tensors are held to this by their tensor maps
  PKB_CHECK_ARG((((uintptr_t)o | (uintptr_t)dk | (uintptr_t)dv) & 15) == 0, "o, dk and dv must be 16-byte aligned");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (d.head_dim == 128) return launch_fa_bwd<128>(d, q, k, v, o, dout, lse, delta_scratch, lse2_scratch, dq, dk, dv, s);
  return launch_fa_bwd<64>(d, q, k, v, o, dout, lse, delta_scratch, lse2_scratch, dq, dk, dv, s);
}

// Context-parallel backward: like pkb_flash_attn_bwd, but the dK / dV rows of KV segment s are added into the fp32 buffers at
// addresses dk_seg[s] / dv_seg[s] ([kv_seg_len[s], hkv, d] each, row 0 of the segment first), which may be peers' symmetric
// memory. The caller zero-fills every accumulator and makes all ranks meet (a barrier launch) before this call, and makes
// them meet again after it before anyone reads its accumulator. dq as in pkb_flash_attn_bwd (dk_seg / dv_seg are not zeroed here).
extern "C" int pkb_flash_attn_bwd_scatter(const pkb_attn_desc* desc, const void* q, const void* k, const void* v, const void* o,
                                          const void* dout, const void* lse, void* delta_scratch, void* lse2_scratch, void* dq,
                                          const unsigned long long* dk_seg, const unsigned long long* dv_seg, void* stream) {
  PKB_CHECK_ARG(desc != nullptr && dk_seg != nullptr && dv_seg != nullptr, "null descriptor or destination table");
  const pkb_attn_desc& d = *desc;
  PKB_CHECK_ARG(d.head_dim == 64 || d.head_dim == 128, "head_dim must be 64 or 128");
  PKB_CHECK_ARG(d.hq % d.hkv == 0 && d.batch == 1 && d.sq >= 1 && d.skv >= 1, "bad attention shape (one sequence)");
  PKB_CHECK_ARG(d.num_q_segs >= 1 && d.num_q_segs <= 16 && d.num_kv_segs >= 1 && d.num_kv_segs <= 16, "1..16 segments");
  PKB_CHECK_ARG(d.q_seg_rows % kFbTile == 0 || d.num_q_segs == 1, "q segments must be multiples of 128 rows");
  PKB_CHECK_ARG(d.q_seg_rows >= 1, "q_seg_rows must be positive");
  for (int s = 0; s < d.num_kv_segs; ++s) {
    PKB_CHECK_ARG(d.kv_seg_row0[s] >= 0 && d.kv_seg_len[s] >= 0 && d.kv_seg_row0[s] + d.kv_seg_len[s] <= d.skv,
                  "kv segment outside the buffer");
    PKB_CHECK_ARG(dk_seg[s] != 0 && dv_seg[s] != 0 && ((dk_seg[s] | dv_seg[s]) & 15) == 0, "segment destinations must be 16-byte aligned");
  }
  PKB_CHECK_ARG(((uintptr_t)o & 15) == 0, "o must be 16-byte aligned");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (d.head_dim == 128)
    return launch_fa_bwd<128>(d, q, k, v, o, dout, lse, delta_scratch, lse2_scratch, dq, nullptr, nullptr, s, dk_seg, dv_seg);
  return launch_fa_bwd<64>(d, q, k, v, o, dout, lse, delta_scratch, lse2_scratch, dq, nullptr, nullptr, s, dk_seg, dv_seg);
}

extern "C" int pkb_flash_attn_bwd_set_trace(void* dev_words) {
  pkb::g_fb_trace = static_cast<long long*>(dev_words);
  return pkb::kApiOk;
}
