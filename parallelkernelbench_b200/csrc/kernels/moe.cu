// Expert-parallel MoE data movement over peer memory. No host round trip anywhere: counts, offsets
// and slots stay on the device (the reference pays three host syncs per layer call,
// reference: reference/31_fused_moe_fwd.py:60-101).
//
//  moe_route       one warp per token: router logits (+ bias) -> softmax -> top-k (descending, ties to the lower
//                  expert index) -> gates, expert indices and the per-expert histogram, in one pass over the row
//  moe_histogram   per-expert assignment counts of this rank's tokens
//  moe_plan        from the all-gathered count matrix [W, E]: where each (source, expert) segment starts
//                  in its destination's receive buffer (expert-major, source-minor), this rank's own
//                  expert row offsets for the grouped GEMM, and its total of received rows
//  moe_dispatch    per batch of tokens: claim a slot in the (expert, me) segment for every assignment, then read each
//                  token's row once and write it STRAIGHT into the destination ranks' receive buffers with 16-byte P2P
//                  stores - as it is, or quantised in registers to e4m3 with one fp32 scale per 128 elements. Ends with
//                  the in-kernel cross-rank barrier so that, when the kernel is complete everywhere, every rank holds
//                  all of its tokens
//  moe_dequant     e4m3 rows that arrived from OTHER ranks -> bf16 (the dispatch wrote this rank's own rows as bf16)
//  moe_combine     after a barrier, pull the k expert-output rows of every token from the ranks that computed them
//                  (P2P loads), weight by the gates, add in a fixed order (deterministic) and store bf16
// Reference behaviour replaced: permute + all_to_all_single + chunk sort, and the inverse path with
// scatter_add_ (reference: reference/28_moe_pre_all2all.py, reference/29_moe_post_all2all.py).
#include "pkb/api.h"
#include "pkb/collectives_api.h"
#include "pkb/fp8_block.cuh"
#include "pkb/host.h"
#include "pkb/symm_host.h"

namespace pkb {

__global__ void moe_histogram_kernel(const int* __restrict__ expert_idx, long long n, int num_experts,
                                     int* __restrict__ counts) {
  extern __shared__ int hist[];
  for (int e = threadIdx.x; e < num_experts; e += blockDim.x) hist[e] = 0;
  __syncthreads();
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const int e = expert_idx[i];
    if (e >= 0 && e < num_experts) atomicAdd(&hist[e], 1);
  }
  __syncthreads();
  for (int e = threadIdx.x; e < num_experts; e += blockDim.x)
    if (hist[e]) atomicAdd(&counts[e], hist[e]);
}

// One block. all_counts[s * E + e] = rows source rank s sends to expert e; total: shared memory, [E].
// seg_base[e]   : first slot, in the receive buffer of the rank that owns expert e, of MY segment
// my_offsets[le]: row offsets of my local experts (E_local + 1 entries), my_total = my_offsets[E_local]
__device__ __forceinline__ void moe_plan_block(const int* all_counts, int world, int num_experts, int experts_per_rank, int my_grank,
                                               int* seg_base, int* my_offsets, int* cursor, int* total) {
  for (int e = threadIdx.x; e < num_experts; e += blockDim.x) {
    int t = 0;
    for (int s = 0; s < world; ++s) t += all_counts[s * num_experts + e];
    total[e] = t;
    cursor[e] = 0;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < num_experts; e += blockDim.x) {
    const int first = (e / experts_per_rank) * experts_per_rank;  // first expert of the owning rank
    int base = 0;
    for (int e2 = first; e2 < e; ++e2) base += total[e2];
    for (int s = 0; s < my_grank; ++s) base += all_counts[s * num_experts + e];
    seg_base[e] = base;
  }
  if (threadIdx.x == 0) {
    int acc = 0;
    for (int le = 0; le < experts_per_rank; ++le) {
      my_offsets[le] = acc;
      acc += total[my_grank * experts_per_rank + le];
    }
    my_offsets[experts_per_rank] = acc;
  }
}

__global__ void moe_plan_kernel(const int* __restrict__ all_counts, int world, int num_experts, int experts_per_rank,
                                int my_grank, int* __restrict__ seg_base, int* __restrict__ my_offsets,
                                int* __restrict__ cursor) {
  extern __shared__ int total[];  // [E] rows per expert over all sources
  moe_plan_block(all_counts, world, num_experts, experts_per_rank, my_grank, seg_base, my_offsets, cursor, total);
}

// Softmax over up to 256 experts and top-k selection, one warp per token. Lane l holds experts l, l + 32, ...
// Selection = k rounds of a warp-wide arg-max on (probability, lower index wins ties), so the output is sorted by
// descending probability like torch.topk. A NaN logit has probability 0 (a token with nothing else has gates NaN), so that every round
// finds an expert. The histogram is accumulated per block in shared memory first.
constexpr int kRouteMaxPerLane = 8;

// work: NULL (counts holds zeros and is added to), or int32 [E + 1] that is zero before and after the kernel: counts is then
// written whole, without a launch to clear it. seg_base / offsets / cursor: NULL, or the plan of a group of one rank, which
// needs no counts from elsewhere and so no launch of its own.
struct MoeRoutePlan {
  int* work;
  int* seg_base;
  int* offsets;
  int* cursor;
};

__global__ void __launch_bounds__(256)
moe_route_kernel(const float* __restrict__ logits, long long ld, const float* __restrict__ bias, int num_tokens,
                 int num_experts, int top_k, float* __restrict__ gates, int* __restrict__ idx, int* __restrict__ counts,
                 const MoeRoutePlan plan) {
  extern __shared__ int hist[];
  for (int e = threadIdx.x; e < num_experts; e += blockDim.x) hist[e] = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int warps_per_block = blockDim.x >> 5;
  for (long long t = (long long)blockIdx.x * warps_per_block + (threadIdx.x >> 5); t < num_tokens;
       t += (long long)gridDim.x * warps_per_block) {
    const float* row = logits + t * ld;
    float v[kRouteMaxPerLane];
    float m = -INFINITY;
#pragma unroll
    for (int j = 0; j < kRouteMaxPerLane; ++j) {
      const int e = j * 32 + lane;
      v[j] = e < num_experts ? row[e] + (bias ? bias[e] : 0.f) : -INFINITY;
      m = fmaxf(m, v[j]);
    }
    m = warp_max(m);
    float sum = 0.f;
#pragma unroll
    for (int j = 0; j < kRouteMaxPerLane; ++j) {
      v[j] = (j * 32 + lane) < num_experts ? fmaxf(expf(v[j] - m), 0.f) : -1.f;   // probabilities are >= 0: -1 marks "absent / taken"
      sum += fmaxf(v[j], 0.f);
    }
    sum = warp_sum(sum);
    const float inv = 1.0f / sum;
    for (int r = 0; r < top_k; ++r) {
      float best = -1.f;
      int best_e = 0x7fffffff;
#pragma unroll
      for (int j = 0; j < kRouteMaxPerLane; ++j)
        if (v[j] > best) { best = v[j]; best_e = j * 32 + lane; }   // ascending j: the lower index wins ties
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) {
        const float ob = __shfl_xor_sync(0xffffffffu, best, off);
        const int oe = __shfl_xor_sync(0xffffffffu, best_e, off);
        if (ob > best || (ob == best && oe < best_e)) { best = ob; best_e = oe; }
      }
      if ((best_e & 31) == lane) {
#pragma unroll
        for (int j = 0; j < kRouteMaxPerLane; ++j)
          if (j == (best_e >> 5)) v[j] = -1.f;
      }
      if (lane == 0) {
        gates[t * top_k + r] = best * inv;
        idx[t * top_k + r] = best_e;
        atomicAdd(&hist[best_e], 1);
      }
    }
  }
  __syncthreads();
  int* sums = plan.work != nullptr ? plan.work : counts;
  for (int e = threadIdx.x; e < num_experts; e += blockDim.x)
    if (hist[e]) atomicAdd(&sums[e], hist[e]);
  if (plan.work == nullptr) return;
  // the block that finishes last publishes the histogram, leaves the work words zero for the next call and, for a group of one
  // rank, writes the plan
  __shared__ int s_last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(&plan.work[num_experts], 1) == (int)gridDim.x - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  for (int e = threadIdx.x; e < num_experts; e += blockDim.x) counts[e] = atomicExch(&plan.work[e], 0);
  if (threadIdx.x == 0) plan.work[num_experts] = 0;
  if (plan.seg_base == nullptr) return;
  __syncthreads();
  moe_plan_block(counts, 1, num_experts, num_experts, 0, plan.seg_base, plan.offsets, plan.cursor, hist);
}

constexpr int kMoeMaxBatch = 8;   // tokens a block of the exchange kernels takes per step

struct MoeDispatchArgs {
  const uint8_t* payload;   // [T, row_bytes] rows: bytes to send as they are, or bf16 [T, hidden] to quantise
  const uint8_t* scales;    // raw form: [T, scale_bytes] or nullptr
  int payload_bytes, scale_bytes;   // what arrives per row; multiples of 16
  const int* expert_idx;    // [T * k] global expert per assignment
  long long num_assign;     // T * k
  int top_k;
  int experts_per_rank;
  const int* seg_base;      // [E]
  int* cursor;              // [E] zeroed by the plan kernel
  int* slots;               // [T * k] out: slot on the destination (or -1 if it did not fit)
  uint64_t recv_payload_off, recv_scale_off;   // heap offsets of the receive buffers
  int capacity;             // rows of the receive buffers
  int* overflow;            // incremented when a row does not fit
  uint64_t recv_meta_off;   // 0, or heap offset of int2 [capacity]: (sender's index in the group, assignment index) per row
  __nv_bfloat16* local_rows;  // quantising form: nullptr, or [capacity, hidden] that receives the rows that stay on this rank
                              // as bf16 (the value the e4m3 code stands for) instead of the receive buffers
  int batch;                // tokens per block and step
};

// One block of 32 warps per SM: the cross-GPU block barrier caps the grid at kSymmMaxBlocks blocks, and 240 blocks would load
// 92 SMs twice and 56 once.
constexpr int kMoeXchgThreads = 1024;

// Where assignment i goes. Every lane of a warp has its own claim in flight (one lane per assignment and warp, as before,
// paid the latency of the index, the atomic and the row one after the other for every row).
__device__ __forceinline__ int moe_claim(const SymmCtx& c, const MoeDispatchArgs& a, long long i, int& dest) {
  const int e = a.expert_idx[i];
  int slot = a.seg_base[e] + atomicAdd(&a.cursor[e], 1);
  dest = c.members[e / a.experts_per_rank];
  if (slot >= a.capacity) {
    slot = -1;
    atomicAdd(a.overflow, 1);
  }
  return slot;
}

// One 16-byte chunk (8 bf16) of a 128-element block that 16 neighbouring lanes hold: e4m3 codes, and with `back` the chunk
// replaced by the values of its codes. Returns the block's scale. All lanes call it.
__device__ __forceinline__ float quantise8(U4& x, uint32_t (&codes)[2], bool back) {
  float v[8];
  const uint32_t w[4] = {x.x, x.y, x.z, x.w};
  float amax = 0.f;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 f = unpack_bf16x2(w[j]);
    v[2 * j] = f.x; v[2 * j + 1] = f.y;
    amax = fmaxf(amax, fmaxf(fabsf(f.x), fabsf(f.y)));
  }
#pragma unroll
  for (int off = 1; off < 16; off <<= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, off));
  const float s = fp8_block_scale(amax, 0);
  fp8_encode8(v, s, codes);
  if (back) {
    fp8_decode8(codes, s, v);
    x = U4{pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]), pack_bf16x2(v[4], v[5]), pack_bf16x2(v[6], v[7])};
  }
  return s;
}
__device__ __forceinline__ uint32_t pick(int lane, uint32_t lo, uint32_t hi) { return lane < 16 ? lo : hi; }

// Memory bound: T rows in, k * T rows out. The row is read once for its k copies, and with QUANT it is quantised on the way (a
// warp holds four 128-element blocks at a time), so no e4m3 copy of the tokens is written and read again. The claims of the
// next batch are in flight while this batch's rows are copied. 8192 tokens x 7168, top-8, one rank: e4m3 rows 120 us (587 MB,
// 4.9 TB/s; quantiser 29 + copy of one row per warp and assignment 355 us before), bf16 rows of e4m3 values 236 us (1.06 GB,
// 4.5 TB/s; 29 + 355 + 334 us for the conversion before).
template <bool QUANT>
__global__ void __launch_bounds__(kMoeXchgThreads, 1) moe_dispatch_kernel(const SymmCtx c, const MoeDispatchArgs a) {
  extern __shared__ int s_claim[];            // [2 buffers][slot, destination rank][batch * k]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int per_batch = a.batch * a.top_k;
  const long long tokens = (a.num_assign + a.top_k - 1) / a.top_k;
  const long long batches = (tokens + a.batch - 1) / a.batch;
  // 512 arriving bytes per warp and step
  const int chunks = (max(a.payload_bytes, QUANT ? 0 : a.scale_bytes) + 511) / 512;
  int buf = 0;
  int next_slot = -1, next_dest = 0;
  auto claim_first = [&](long long batch) {   // this thread's assignment of the batch (the rest, if any, follow in publish)
    const long long i = batch * per_batch + threadIdx.x;
    if (batch < batches && (int)threadIdx.x < per_batch && i < a.num_assign) next_slot = moe_claim(c, a, i, next_dest);
    else next_slot = -1;
  };
  auto record = [&](long long i, int slot, int dest, int at) {
    int* s = s_claim + buf * 2 * per_batch;
    s[at] = slot;
    s[per_batch + at] = dest;
    if (i < a.num_assign) {
      a.slots[i] = slot;
      if (slot >= 0 && a.recv_meta_off != 0) symm_ptr<int2>(c, dest, a.recv_meta_off)[slot] = make_int2(c.grank, (int)i);
    }
  };
  claim_first(blockIdx.x);
  for (long long batch = blockIdx.x; batch < batches; batch += gridDim.x) {
    const long long i0 = batch * per_batch;
    if ((int)threadIdx.x < per_batch) record(i0 + threadIdx.x, next_slot, next_dest, threadIdx.x);
    for (int at = threadIdx.x + blockDim.x; at < per_batch; at += blockDim.x) {
      int dest = 0;
      const int slot = i0 + at < a.num_assign ? moe_claim(c, a, i0 + at, dest) : -1;
      record(i0 + at, slot, dest, at);
    }
    __syncthreads();                          // the other buffer is rewritten only after the next of these
    claim_first(batch + gridDim.x);
    const int* s_slot = s_claim + buf * 2 * per_batch;
    const int* s_dest = s_slot + per_batch;
    buf ^= 1;
    const int units = (int)min((long long)a.batch, tokens - batch * a.batch) * chunks;
    for (int u = warp; u < units; u += kMoeXchgThreads / 32) {
      const int tok = u / chunks;
      const int b = (u - tok * chunks) * 512 + lane * 16;      // first arriving byte (QUANT: element) of this lane
      const long long t = batch * a.batch + tok;
      const bool in = b < a.payload_bytes;
      if constexpr (QUANT) {
        // 512 elements per warp and step: lane l holds 16-byte chunks l and 32 + l of the bf16 row piece, so that every access
        // of the warp is one run of memory. 16 lanes share a 128-element block.
        const int col = b - lane * 16;
        const uint8_t* src = a.payload + (t * a.payload_bytes + col) * 2 + lane * 16;
        const bool in0 = col + lane * 8 < a.payload_bytes, in1 = col + 256 + lane * 8 < a.payload_bytes;
        U4 x0{}, x1{};
        if (in0) x0 = ld_global_nc_v4(src);
        if (in1) x1 = ld_global_nc_v4(src + 512);
        uint32_t q0[2], q1[2];
        const float s0 = quantise8(x0, q0, a.local_rows != nullptr), s1 = quantise8(x1, q1, a.local_rows != nullptr);
        // e4m3 row piece, 16 bytes per lane: lane l stores the codes of chunks 2 l and 2 l + 1
        const int from = (lane * 2) & 31;
        U4 codes;
        codes.x = pick(lane, __shfl_sync(0xffffffffu, q0[0], from), __shfl_sync(0xffffffffu, q1[0], from));
        codes.y = pick(lane, __shfl_sync(0xffffffffu, q0[1], from), __shfl_sync(0xffffffffu, q1[1], from));
        codes.z = pick(lane, __shfl_sync(0xffffffffu, q0[0], from + 1), __shfl_sync(0xffffffffu, q1[0], from + 1));
        codes.w = pick(lane, __shfl_sync(0xffffffffu, q0[1], from + 1), __shfl_sync(0xffffffffu, q1[1], from + 1));
        for (int j = 0; j < a.top_k; ++j) {
          const int slot = s_slot[tok * a.top_k + j], dest = s_dest[tok * a.top_k + j];
          if (slot < 0) continue;
          if (a.local_rows != nullptr && dest == c.rank) {
            __nv_bfloat16* o = a.local_rows + (long long)slot * a.payload_bytes + col + lane * 8;
            if (in0) st_global_v4(o, x0);
            if (in1) st_global_v4(o + 256, x1);
          } else {
            if (in) st_global_v4(symm_ptr<uint8_t>(c, dest, a.recv_payload_off) + (long long)slot * a.payload_bytes + b, codes);
            float* sc = reinterpret_cast<float*>(symm_ptr<uint8_t>(c, dest, a.recv_scale_off) + (long long)slot * a.scale_bytes);
            if ((lane & 15) == 0) {
              if (in0) sc[(col >> 7) + (lane >> 4)] = s0;
              if (in1) sc[(col >> 7) + 2 + (lane >> 4)] = s1;
            }
          }
        }
      } else {
        U4 v{}, sc{};
        const bool with_scales = a.scales != nullptr && b < a.scale_bytes;
        if (in) v = ld_global_v4(a.payload + t * a.payload_bytes + b);
        if (with_scales) sc = ld_global_v4(a.scales + t * a.scale_bytes + b);
        for (int j = 0; j < a.top_k; ++j) {
          const int slot = s_slot[tok * a.top_k + j], dest = s_dest[tok * a.top_k + j];
          if (slot < 0) continue;
          if (in) st_global_v4(symm_ptr<uint8_t>(c, dest, a.recv_payload_off) + (long long)slot * a.payload_bytes + b, v);
          if (with_scales) st_global_v4(symm_ptr<uint8_t>(c, dest, a.recv_scale_off) + (long long)slot * a.scale_bytes + b, sc);
        }
      }
    }
  }
  // when this barrier has been crossed by every block of every rank, all rows have landed everywhere; a group of one is
  // done when the kernel is
  if (c.gsize > 1) symm_block_barrier(c, 500, 1);
}

// Rows of the receive buffer that came from other ranks -> bf16. This rank's own rows of local expert le sit in slots
// [seg_base[le], seg_base[le] + counts[le]) and are already in `out`. One warp per row.
__global__ void __launch_bounds__(256)
moe_dequant_kernel(const uint8_t* __restrict__ payload, const uint8_t* __restrict__ scales, int hidden, int scale_bytes,
                   const int* __restrict__ offsets, const int* __restrict__ seg_base, const int* __restrict__ counts,
                   int experts, int capacity, __nv_bfloat16* __restrict__ out) {
  const int lane = threadIdx.x & 31;
  const long long warps = ((long long)gridDim.x * blockDim.x) >> 5;
  const int rows = min(offsets[experts], capacity);
  for (long long row = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; row < rows; row += warps) {
    int lo = 0, hi = experts;                // offsets[lo] <= row < offsets[hi]
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (offsets[mid] <= row) lo = mid; else hi = mid;
    }
    if (row >= seg_base[lo] && row < seg_base[lo] + counts[lo]) continue;
    const float* sc = reinterpret_cast<const float*>(scales + row * scale_bytes);
    for (int b = lane * 8; b < hidden; b += 256) {
      const uint2 u = *reinterpret_cast<const uint2*>(payload + row * hidden + b);
      const uint32_t q[2] = {u.x, u.y};
      float v[8];
      fp8_decode8(q, sc[b >> 7], v);
      st_global_v4(out + row * hidden + b,
                   U4{pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]), pack_bf16x2(v[4], v[5]), pack_bf16x2(v[6], v[7])});
    }
  }
}

struct MoeCombineArgs {
  uint64_t y_off;            // heap offset of the expert outputs [capacity, hidden] bf16 on every rank
  const int* expert_idx;     // [T * k]
  const int* slots;          // [T * k]
  const float* gates;        // [T * k]
  __nv_bfloat16* out;        // [T, hidden]
  long long num_tokens;
  int top_k, hidden, experts_per_rank;
  int local_rows;            // 1: row (t, j) sits at row t * k + j of THIS rank's buffer (the experts pushed it there)
  int batch;                 // tokens per block and step
};

// 16 bytes of a row, or zeros where there is no row: the loads of a token's k rows stay in flight together (behind a branch
// each, the next load waited for the arithmetic of the one before)
__device__ __forceinline__ U4 ld_row_or_zero(const uint8_t* p) {
  U4 v;
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.u64 q, %4, 0;\n\tmov.u32 %0, 0;\n\tmov.u32 %1, 0;\n\tmov.u32 %2, 0;\n\tmov.u32 %3, 0;\n\t"
      "@q ld.relaxed.sys.global.v4.u32 {%0, %1, %2, %3}, [%4];\n\t}"
      : "=&r"(v.x), "=&r"(v.y), "=&r"(v.z), "=&r"(v.w)
      : "l"(p)
      : "memory");
  return v;
}

// Memory bound: k * T rows in, T rows out. A block takes a batch of tokens: row addresses and gates of the batch go to shared
// memory (fetched while the batch before is added up), then the warps share the batch's (token, 256 columns) pieces. 8192 x
// 7168, top-8: 170 us (1.06 GB, 6.2 TB/s); 533 us with one warp per token and a branch around every row's load.
template <int MAXK>
__global__ void __launch_bounds__(kMoeXchgThreads, 1) moe_combine_kernel(const SymmCtx c, const MoeCombineArgs a) {
  __shared__ const uint8_t* s_row[2][kMoeMaxBatch * MAXK];
  __shared__ float s_gate[2][kMoeMaxBatch * MAXK];
  // every rank's expert outputs are complete once all ranks have entered this kernel
  if (c.gsize > 1 && !symm_block_barrier(c, 501, 1)) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long batches = (a.num_tokens + a.batch - 1) / a.batch;
  const int chunks = (a.hidden + 255) / 256;
  const int my_tok = threadIdx.x / MAXK, my_j = threadIdx.x % MAXK;
  int buf = 0;
  const uint8_t* next_row = nullptr;
  float next_gate = 0.f;
  auto fetch = [&](long long batch) {
    const long long t = batch * a.batch + my_tok;
    next_row = nullptr;
    next_gate = 0.f;
    if (batch >= batches || my_tok >= a.batch || my_j >= a.top_k || t >= a.num_tokens) return;
    const long long i = t * a.top_k + my_j;
    const int slot = a.slots[i];
    if (slot < 0) return;
    next_row = a.local_rows ? symm_local<uint8_t>(c, a.y_off) + i * a.hidden * 2
                            : symm_ptr<uint8_t>(c, c.members[a.expert_idx[i] / a.experts_per_rank], a.y_off) + (long long)slot * a.hidden * 2;
    next_gate = a.gates[i];
  };
  fetch(blockIdx.x);
  for (long long batch = blockIdx.x; batch < batches; batch += gridDim.x) {
    if (my_tok < a.batch) {
      s_row[buf][threadIdx.x] = next_row;
      s_gate[buf][threadIdx.x] = next_gate;
    }
    __syncthreads();                          // the other buffer is rewritten only after the next of these
    fetch(batch + gridDim.x);
    const int units = (int)min((long long)a.batch, a.num_tokens - batch * a.batch) * chunks;
    for (int u = warp; u < units; u += kMoeXchgThreads / 32) {
      const int tok = u / chunks;
      const int col = (u - tok * chunks) * 256 + lane * 8;
      if (col >= a.hidden) continue;
      U4 v[MAXK];
#pragma unroll
      for (int j = 0; j < MAXK; ++j) {
        const uint8_t* r = s_row[buf][tok * MAXK + j];
        v[j] = ld_row_or_zero(r == nullptr ? nullptr : r + col * 2);
      }
      float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int j = 0; j < MAXK; ++j) {        // an absent row adds 0 * 0
        const float w = s_gate[buf][tok * MAXK + j];
        const float2 f0 = unpack_bf16x2(v[j].x), f1 = unpack_bf16x2(v[j].y), f2 = unpack_bf16x2(v[j].z), f3 = unpack_bf16x2(v[j].w);
        acc[0] += w * f0.x; acc[1] += w * f0.y; acc[2] += w * f1.x; acc[3] += w * f1.y;
        acc[4] += w * f2.x; acc[5] += w * f2.y; acc[6] += w * f3.x; acc[7] += w * f3.y;
      }
      const U4 o{pack_bf16x2(acc[0], acc[1]), pack_bf16x2(acc[2], acc[3]), pack_bf16x2(acc[4], acc[5]), pack_bf16x2(acc[6], acc[7])};
      st_global_v4(a.out + (batch * a.batch + tok) * a.hidden + col, o);
    }
    buf ^= 1;
  }
  // peers may still be reading my expert outputs: nobody overwrites them before everyone is done
  if (c.gsize > 1) symm_block_barrier(c, 501, 2);
}

// Tokens per block and step: as many blocks as there are SMs get work before a block takes more than one token at a time.
static int moe_batch(long long tokens, int grid) {
  int b = kMoeMaxBatch;
  while (b > 1 && tokens < (long long)b * grid) b >>= 1;
  return b;
}

static int moe_grid() {   // fixed: the same on every rank, the barrier pairs blocks by index
  const int sms = sm_count();
  return sms < kSymmMaxBlocks ? sms : kSymmMaxBlocks;
}

template <bool QUANT>
static int launch_moe_dispatch(const pkb_symm_ctx* h, MoeDispatchArgs a, cudaStream_t s) {
  const int grid = moe_grid();
  a.batch = a.top_k <= 32 ? moe_batch((a.num_assign + a.top_k - 1) / a.top_k, grid) : 1;
  const size_t smem = sizeof(int) * 4 * a.batch * a.top_k;
  PKB_CHECK_ARG(smem <= 48 * 1024, "top_k too large");
  moe_dispatch_kernel<QUANT><<<grid, kMoeXchgThreads, smem, s>>>(symm_ctx_from_api(h), a);
  PKB_CHECK_CUDA(cudaGetLastError());
  return kApiOk;
}

}  // namespace pkb

using namespace pkb;

extern "C" {

int pkb_moe_histogram(const void* expert_idx, long long n, int num_experts, void* counts, void* stream) {
  PKB_CHECK_ARG(num_experts >= 1 && num_experts <= 4096, "1..4096 experts");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  PKB_CHECK_CUDA(cudaMemsetAsync(counts, 0, sizeof(int) * num_experts, s));
  if (n == 0) return kApiOk;
  long long blocks = (n + 255) / 256;
  if (blocks > 148 * 4) blocks = 148 * 4;
  moe_histogram_kernel<<<(int)blocks, 256, num_experts * sizeof(int), s>>>(static_cast<const int*>(expert_idx), n,
                                                                          num_experts, static_cast<int*>(counts));
  PKB_CHECK_CUDA(cudaGetLastError());
  return kApiOk;
}

// logits [T, E] fp32 (row pitch ld elements) + optional fp32 bias [E] -> gates [T, k] fp32 (softmax probabilities of the
// chosen experts, descending), idx [T, k] int32, counts [E] int32 (zeroed here, then accumulated). E <= 256, k <= E.
int pkb_moe_route(const void* logits, long long ld, const void* bias, int num_tokens, int num_experts, int top_k,
                  void* gates, void* idx, void* counts, void* stream) {
  PKB_CHECK_ARG(num_experts >= 1 && num_experts <= 32 * kRouteMaxPerLane, "1..256 experts");
  PKB_CHECK_ARG(top_k >= 1 && top_k <= num_experts, "top_k must be in 1..experts");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  PKB_CHECK_CUDA(cudaMemsetAsync(counts, 0, sizeof(int) * num_experts, s));
  if (num_tokens == 0) return kApiOk;
  long long blocks = ((long long)num_tokens + 7) / 8;
  if (blocks > 148 * 8) blocks = 148 * 8;
  moe_route_kernel<<<(int)blocks, 256, num_experts * sizeof(int), s>>>(
      static_cast<const float*>(logits), ld, static_cast<const float*>(bias), num_tokens, num_experts, top_k,
      static_cast<float*>(gates), static_cast<int*>(idx), static_cast<int*>(counts), MoeRoutePlan{});
  PKB_CHECK_CUDA(cudaGetLastError());
  return kApiOk;
}

// The same without a separate launch to clear counts: work is an int32 [E + 1] scratch that is zero before and after. With
// seg_base, offsets [E + 1] and cursor given, the plan of a group of one rank (pkb_moe_plan with world = 1) is written too.
int pkb_moe_route_plan(const void* logits, long long ld, const void* bias, int num_tokens, int num_experts, int top_k,
                       void* gates, void* idx, void* counts, void* work, void* seg_base, void* offsets, void* cursor,
                       void* stream) {
  PKB_CHECK_ARG(num_experts >= 1 && num_experts <= 32 * kRouteMaxPerLane, "1..256 experts");
  PKB_CHECK_ARG(top_k >= 1 && top_k <= num_experts, "top_k must be in 1..experts");
  PKB_CHECK_ARG(work != nullptr, "work words are required");
  PKB_CHECK_ARG((seg_base == nullptr) == (offsets == nullptr) && (offsets == nullptr) == (cursor == nullptr),
                "seg_base, offsets and cursor go together");
  long long blocks = ((long long)num_tokens + 7) / 8;
  if (blocks > 148 * 8) blocks = 148 * 8;
  if (blocks < 1) blocks = 1;
  moe_route_kernel<<<(int)blocks, 256, num_experts * sizeof(int), static_cast<cudaStream_t>(stream)>>>(
      static_cast<const float*>(logits), ld, static_cast<const float*>(bias), num_tokens, num_experts, top_k,
      static_cast<float*>(gates), static_cast<int*>(idx), static_cast<int*>(counts),
      MoeRoutePlan{static_cast<int*>(work), static_cast<int*>(seg_base), static_cast<int*>(offsets), static_cast<int*>(cursor)});
  PKB_CHECK_CUDA(cudaGetLastError());
  return kApiOk;
}

int pkb_moe_plan(const void* all_counts, int world, int num_experts, int experts_per_rank, int my_grank,
                 void* seg_base, void* my_offsets, void* cursor, void* stream) {
  PKB_CHECK_ARG(num_experts == world * experts_per_rank, "experts must divide evenly over the group");
  PKB_CHECK_ARG(num_experts <= 4096, "at most 4096 experts");
  moe_plan_kernel<<<1, 256, num_experts * sizeof(int), static_cast<cudaStream_t>(stream)>>>(
      static_cast<const int*>(all_counts), world, num_experts, experts_per_rank, my_grank, static_cast<int*>(seg_base),
      static_cast<int*>(my_offsets), static_cast<int*>(cursor));
  PKB_CHECK_CUDA(cudaGetLastError());
  return kApiOk;
}

// recv_meta_off: 0, or the heap offset of an int2 [capacity] array that receives, for every row written, the sender's
// index in the group and the assignment index (token * k + j) - what an expert needs to send the row's result home.
int pkb_moe_dispatch_meta(const pkb_symm_ctx* h, const void* payload, const void* scales, int payload_bytes,
                          int scale_bytes, const void* expert_idx, long long num_assign, int top_k, int experts_per_rank,
                          const void* seg_base, void* cursor, void* slots, unsigned long long recv_payload_off,
                          unsigned long long recv_scale_off, int capacity, void* overflow,
                          unsigned long long recv_meta_off, void* stream) {
  PKB_CHECK_ARG(h && h->base, "symmetric heap not initialised");
  PKB_CHECK_ARG(payload_bytes % 16 == 0 && scale_bytes % 16 == 0, "row sizes must be multiples of 16 bytes");
  PKB_CHECK_ARG((recv_payload_off & 15) == 0 && (recv_scale_off & 15) == 0, "heap offsets misaligned");
  PKB_CHECK_ARG((recv_meta_off & 7) == 0, "heap offsets misaligned");
  PKB_CHECK_ARG(top_k >= 1, "top_k must be positive");
  MoeDispatchArgs a{static_cast<const uint8_t*>(payload), static_cast<const uint8_t*>(scales), payload_bytes, scale_bytes,
                    static_cast<const int*>(expert_idx), num_assign, top_k, experts_per_rank,
                    static_cast<const int*>(seg_base), static_cast<int*>(cursor), static_cast<int*>(slots),
                    recv_payload_off, recv_scale_off, capacity, static_cast<int*>(overflow), recv_meta_off, nullptr, 1};
  return launch_moe_dispatch<false>(h, a, static_cast<cudaStream_t>(stream));
}

// The same from bf16 rows x [T, hidden] (hidden a multiple of 128): the rows travel as e4m3 with one fp32 scale per 128
// elements (scale_bytes per row at the receiver), quantised on the way. local_rows: NULL, or bf16 [capacity, hidden] that
// receives the rows whose expert is on this rank (as the values of their e4m3 codes) in place of the receive buffers.
int pkb_moe_dispatch_quant(const pkb_symm_ctx* h, const void* x, int hidden, int scale_bytes, const void* expert_idx,
                           long long num_assign, int top_k, int experts_per_rank, const void* seg_base, void* cursor,
                           void* slots, unsigned long long recv_payload_off, unsigned long long recv_scale_off, int capacity,
                           void* overflow, unsigned long long recv_meta_off, void* local_rows, void* stream) {
  PKB_CHECK_ARG(h && h->base, "symmetric heap not initialised");
  PKB_CHECK_ARG(hidden > 0 && hidden % 128 == 0 && scale_bytes >= hidden / 128 * 4 && scale_bytes % 16 == 0, "bad row sizes");
  PKB_CHECK_ARG((((uintptr_t)x | (uintptr_t)local_rows) & 15) == 0, "rows must be 16-byte aligned");
  PKB_CHECK_ARG((recv_payload_off & 15) == 0 && (recv_scale_off & 15) == 0 && (recv_meta_off & 7) == 0, "heap offsets misaligned");
  PKB_CHECK_ARG(top_k >= 1, "top_k must be positive");
  MoeDispatchArgs a{static_cast<const uint8_t*>(x), nullptr, hidden, scale_bytes,
                    static_cast<const int*>(expert_idx), num_assign, top_k, experts_per_rank,
                    static_cast<const int*>(seg_base), static_cast<int*>(cursor), static_cast<int*>(slots),
                    recv_payload_off, recv_scale_off, capacity, static_cast<int*>(overflow), recv_meta_off,
                    static_cast<__nv_bfloat16*>(local_rows), 1};
  return launch_moe_dispatch<true>(h, a, static_cast<cudaStream_t>(stream));
}

// e4m3 rows received from other ranks -> rows of out (bf16 [capacity, hidden]). offsets int32 [experts + 1]: rows of each local
// expert; seg_base / counts int32 [experts]: where this rank's own rows of that expert sit (they are left alone).
int pkb_moe_dequant(const void* payload, const void* scales, int hidden, int scale_bytes, const void* offsets,
                    const void* seg_base, const void* counts, int experts, int capacity, void* out, void* stream) {
  PKB_CHECK_ARG(hidden % 128 == 0 && experts >= 1, "hidden must be a multiple of 128");
  PKB_CHECK_ARG((((uintptr_t)payload | (uintptr_t)scales | (uintptr_t)out) & 15) == 0, "buffers must be 16-byte aligned");
  const int grid = sm_count() * 8;
  moe_dequant_kernel<<<grid, 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const uint8_t*>(payload), static_cast<const uint8_t*>(scales), hidden, scale_bytes,
      static_cast<const int*>(offsets), static_cast<const int*>(seg_base), static_cast<const int*>(counts), experts, capacity,
      static_cast<__nv_bfloat16*>(out));
  PKB_CHECK_CUDA(cudaGetLastError());
  return kApiOk;
}

int pkb_moe_dispatch(const pkb_symm_ctx* h, const void* payload, const void* scales, int payload_bytes,
                     int scale_bytes, const void* expert_idx, long long num_assign, int top_k, int experts_per_rank,
                     const void* seg_base, void* cursor, void* slots, unsigned long long recv_payload_off,
                     unsigned long long recv_scale_off, int capacity, void* overflow, void* stream) {
  return pkb_moe_dispatch_meta(h, payload, scales, payload_bytes, scale_bytes, expert_idx, num_assign, top_k, experts_per_rank,
                               seg_base, cursor, slots, recv_payload_off, recv_scale_off, capacity, overflow, 0ull, stream);
}

// local_rows = 0: pull row `slots[t, j]` of the expert outputs at y_off from the rank that owns expert idx[t, j].
// local_rows = 1: the experts already pushed the result of assignment (t, j) to row t * k + j of THIS rank's buffer at y_off.
int pkb_moe_combine_from(const pkb_symm_ctx* h, unsigned long long y_off, const void* expert_idx, const void* slots,
                         const void* gates, void* out, long long num_tokens, int top_k, int hidden, int experts_per_rank,
                         int local_rows, void* stream) {
  PKB_CHECK_ARG(h && h->base, "symmetric heap not initialised");
  PKB_CHECK_ARG(hidden % 8 == 0 && top_k >= 1 && top_k <= 8, "hidden % 8 == 0 and top_k <= 8");
  MoeCombineArgs a{y_off, static_cast<const int*>(expert_idx), static_cast<const int*>(slots),
                   static_cast<const float*>(gates), static_cast<__nv_bfloat16*>(out), num_tokens, top_k, hidden,
                   experts_per_rank, local_rows, 1};
  const int grid = moe_grid();
  a.batch = moe_batch(num_tokens, grid);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (top_k <= 2) moe_combine_kernel<2><<<grid, kMoeXchgThreads, 0, s>>>(symm_ctx_from_api(h), a);
  else if (top_k <= 4) moe_combine_kernel<4><<<grid, kMoeXchgThreads, 0, s>>>(symm_ctx_from_api(h), a);
  else moe_combine_kernel<8><<<grid, kMoeXchgThreads, 0, s>>>(symm_ctx_from_api(h), a);
  PKB_CHECK_CUDA(cudaGetLastError());
  return kApiOk;
}

int pkb_moe_combine(const pkb_symm_ctx* h, unsigned long long y_off, const void* expert_idx, const void* slots,
                    const void* gates, void* out, long long num_tokens, int top_k, int hidden, int experts_per_rank,
                    void* stream) {
  return pkb_moe_combine_from(h, y_off, expert_idx, slots, gates, out, num_tokens, top_k, hidden, experts_per_rank, 0, stream);
}

}  // extern "C"
