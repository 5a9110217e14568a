// Memory-bound kernels around the GEMMs: RoPE, fp8 1x128 block quantise / dequantise, fused
// Adam / AdamW, vocab-parallel cross-entropy statistics, column reductions for the LayerNorm
// backward, and a tensor-parallel RMSNorm whose cross-rank sum runs inside the kernel.
// All use 16-byte global accesses and fp32 arithmetic.
//
// Reference behaviour: reference/17_rope_allgather.py:10-37, reference/19_blocked_fp8_quantize.py:7-23,
// reference/20_blocked_fp8_dequantize.py:6-16, reference/43_fused_adam_grad_unshard_allgather.py:28-40,
// reference/47_fsdp_step_e2e.py:52-65, reference/73_vocab_parallel_cross_entropy_loss.py:21-42,
// reference/9_layernorm_backward.py:6-11, reference/18_tp_rms_norm.py:9-19.
#include <cuda_fp8.h>
#include <math.h>

#include "pkb/api.h"
#include "pkb/collectives_api.h"
#include "pkb/fp8_block.cuh"
#include "pkb/host.h"
#include "pkb/symm.cuh"

namespace pkb {

// ================================================================================================
// RoPE (rotate-half): x is [tokens, heads, dim]; cos/sin are [tokens, dim] (the two halves of a row
// of cos/sin normally repeat). out[.., :d/2] = x1*cos1 - x2*sin1 ; out[.., d/2:] = x2*cos2 + x1*sin2
// ================================================================================================
template <typename T>
__global__ void rope_kernel(const T* __restrict__ x, const T* __restrict__ cs, const T* __restrict__ sn,
                            T* __restrict__ out, long long tokens, int heads, int dim) {
  const int half = dim >> 1;
  const long long total = tokens * heads * half;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const int j = (int)(i % half);
    const long long th = i / half;
    const long long t = th / heads;
    const T* xr = x + th * dim;
    const float x1 = (float)xr[j], x2 = (float)xr[j + half];
    const float c1 = (float)cs[t * dim + j], c2 = (float)cs[t * dim + j + half];
    const float s1 = (float)sn[t * dim + j], s2 = (float)sn[t * dim + j + half];
    out[th * dim + j] = (T)(x1 * c1 - x2 * s1);
    out[th * dim + j + half] = (T)(x2 * c2 + x1 * s2);
  }
}

// ================================================================================================
// fp8 e4m3 quantise with one fp32 scale per 128 consecutive elements: s = amax/448 (1 if amax = 0),
// y = sat(x / s). One warp handles one block: 4 elements per lane.
// ================================================================================================
template <typename T>
__device__ __forceinline__ void load16(const T* p, float (&v)[16]);
template <>
__device__ __forceinline__ void load16<__nv_bfloat16>(const __nv_bfloat16* p, float (&v)[16]) {
  const U4 u0 = ld_global_nc_v4(p), u1 = ld_global_nc_v4(p + 8);
  const uint32_t w[8] = {u0.x, u0.y, u0.z, u0.w, u1.x, u1.y, u1.z, u1.w};
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const float2 f = unpack_bf16x2(w[j]);
    v[2 * j] = f.x; v[2 * j + 1] = f.y;
  }
}
template <>
__device__ __forceinline__ void load16<float>(const float* p, float (&v)[16]) {
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const U4 u = ld_global_nc_v4(p + 4 * q);
    v[4 * q] = __uint_as_float(u.x); v[4 * q + 1] = __uint_as_float(u.y);
    v[4 * q + 2] = __uint_as_float(u.z); v[4 * q + 3] = __uint_as_float(u.w);
  }
}

// A thread owns 16 consecutive elements (32 or 64 bytes in, one 16-byte store out); the 8 lanes of a 128-element block share
// its maximum through three shuffles. Memory bound: what counts is bytes in flight per thread, not arithmetic.
template <typename T>
__global__ void __launch_bounds__(256) fp8_quant_kernel(const T* __restrict__ x, uint8_t* __restrict__ y, float* __restrict__ scales,
                                                        long long nblocks, int pow2_scales) {
  const long long nthr = nblocks * 8;
  for (long long t0 = (long long)blockIdx.x * blockDim.x; t0 < nthr; t0 += (long long)gridDim.x * blockDim.x) {
    const long long t = t0 + threadIdx.x;      // nthr is a multiple of 8: a group of 8 lanes is active or idle as a whole
    float v[16];
    float amax = 0.f;
    if (t < nthr) {
      load16<T>(x + (t << 4), v);
#pragma unroll
      for (int j = 0; j < 16; ++j) amax = fmaxf(amax, fabsf(v[j]));
    }
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 4));
    if (t >= nthr) continue;
    const float s = fp8_block_scale(amax, pow2_scales);
    uint32_t o[4];
    fp8_encode8(v, s, o);
    fp8_encode8(v + 8, s, o + 2);
    st_global_v4(y + (t << 4), U4{o[0], o[1], o[2], o[3]});
    if ((t & 7) == 0) scales[t >> 3] = s;
  }
}

// A thread owns 16 consecutive e4m3 values (one 16-byte load, 32 or 64 bytes out as 16-byte stores); 8 threads share a block's
// scale. `valid_rows` (device, may be null): rows at and beyond *valid_rows of a [rows, blocks_per_row * 128] buffer are left
// alone - a receive buffer sized for the worst case is only dequantised as far as it was filled.
template <typename T>
__global__ void __launch_bounds__(256) fp8_dequant_kernel(const uint8_t* __restrict__ y, const float* __restrict__ scales,
                                                          T* __restrict__ x, long long nblocks, const int* __restrict__ valid_rows,
                                                          long long blocks_per_row) {
  long long nb = nblocks;
  if (valid_rows != nullptr) {
    const long long lim = (long long)(*valid_rows) * blocks_per_row;
    if (lim < nb) nb = lim;
  }
  const long long nthr = nb * 8;
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < nthr; t += (long long)gridDim.x * blockDim.x) {
    const U4 u = ld_global_nc_v4(y + (t << 4));
    const float sc = scales[t >> 3];
    const uint32_t w[4] = {u.x, u.y, u.z, u.w};
    float v[16];
    fp8_decode8(w, sc, v);
    fp8_decode8(w + 2, sc, v + 8);
    T* o = x + (t << 4);
    if constexpr (sizeof(T) == 2) {
      st_global_v4(o, U4{pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]), pack_bf16x2(v[4], v[5]), pack_bf16x2(v[6], v[7])});
      st_global_v4(o + 8, U4{pack_bf16x2(v[8], v[9]), pack_bf16x2(v[10], v[11]), pack_bf16x2(v[12], v[13]), pack_bf16x2(v[14], v[15])});
    } else {
#pragma unroll
      for (int q = 0; q < 4; ++q)
        st_global_v4(o + 4 * q, U4{__float_as_uint(v[4 * q]), __float_as_uint(v[4 * q + 1]), __float_as_uint(v[4 * q + 2]),
                                   __float_as_uint(v[4 * q + 3])});
    }
  }
}

// ================================================================================================
// Adam / AdamW on fp32 master weights. grad is fp32 or bf16 and is multiplied by grad_scale first.
// decoupled = 1: AdamW (p *= 1 - lr*wd before the update); 0: L2 folded into the gradient.
// Optionally writes a bf16 copy of the new parameters (what the next forward consumes).
// ================================================================================================
struct AdamArgs {
  float beta1, beta2, eps, weight_decay, grad_scale;
  float decay;         // 1 - lr * weight_decay
  float step_size;     // lr / (1 - beta1^step)
  float inv_sqrt_c2;   // 1 / sqrt(1 - beta2^step)
  int decoupled;
};

// One element. The bias corrections are folded into two constants, as torch.optim does (step size lr / bias_c1, denominator
// sqrt(v) / sqrt(bias_c2) + eps): one square root and one division remain of one and three.
__device__ __forceinline__ float adam_update(float w, float& m, float& v, float grad, const AdamArgs& a) {
  grad *= a.grad_scale;
  if (a.decoupled) w *= a.decay;
  else grad = fmaf(a.weight_decay, w, grad);
  m = a.beta1 * m + (1.0f - a.beta1) * grad;
  v = a.beta2 * v + (1.0f - a.beta2) * grad * grad;
  return w - a.step_size * m / (sqrtf(v) * a.inv_sqrt_c2 + a.eps);
}

// Memory bound: 28 bytes move per element (bf16 gradient and bf16 copy), 2.25 ms for the 525 M parameters of a 128256 x 4096
// head at the copy bandwidth. VEC: four elements per thread and access (16-byte loads of p, m, v), two accesses in flight; the
// scalar form (any alignment, any count) takes what is left. Measured on that head: 4.11 ms with one element per thread (the
// three divisions and 4-byte accesses bound it), 2.70 ms.
template <typename G, bool VEC>
__global__ void __launch_bounds__(256)
adam_kernel(float* __restrict__ p, float* __restrict__ m, float* __restrict__ v, const G* __restrict__ g,
            __nv_bfloat16* __restrict__ p_bf16, long long n, AdamArgs a) {
  if constexpr (VEC) {
    const long long nv = n >> 2;
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long i0 = (long long)blockIdx.x * blockDim.x + threadIdx.x; i0 < nv; i0 += 2 * stride) {
      float4 pp[2], mm[2], vv[2];
      float gg[2][4];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const long long i = i0 + u * stride;
        if (i < nv) {
          pp[u] = __ldcs(reinterpret_cast<const float4*>(p) + i);
          mm[u] = __ldcs(reinterpret_cast<const float4*>(m) + i);
          vv[u] = __ldcs(reinterpret_cast<const float4*>(v) + i);
          if constexpr (sizeof(G) == 2) {
            const uint2 w = __ldcs(reinterpret_cast<const uint2*>(g) + i);
            const float2 f0 = unpack_bf16x2(w.x), f1 = unpack_bf16x2(w.y);
            gg[u][0] = f0.x; gg[u][1] = f0.y; gg[u][2] = f1.x; gg[u][3] = f1.y;
          } else {
            const float4 w = __ldcs(reinterpret_cast<const float4*>(g) + i);
            gg[u][0] = w.x; gg[u][1] = w.y; gg[u][2] = w.z; gg[u][3] = w.w;
          }
        }
      }
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const long long i = i0 + u * stride;
        if (i >= nv) break;
        pp[u].x = adam_update(pp[u].x, mm[u].x, vv[u].x, gg[u][0], a);
        pp[u].y = adam_update(pp[u].y, mm[u].y, vv[u].y, gg[u][1], a);
        pp[u].z = adam_update(pp[u].z, mm[u].z, vv[u].z, gg[u][2], a);
        pp[u].w = adam_update(pp[u].w, mm[u].w, vv[u].w, gg[u][3], a);
        __stcs(reinterpret_cast<float4*>(p) + i, pp[u]);
        __stcs(reinterpret_cast<float4*>(m) + i, mm[u]);
        __stcs(reinterpret_cast<float4*>(v) + i, vv[u]);
        if (p_bf16) reinterpret_cast<uint2*>(p_bf16)[i] = make_uint2(pack_bf16x2(pp[u].x, pp[u].y), pack_bf16x2(pp[u].z, pp[u].w));
      }
    }
  }
  const long long tail0 = VEC ? (n & ~3ll) : 0;
  for (long long i = tail0 + (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    float mi = m[i], vi = v[i];
    const float w = adam_update(p[i], mi, vi, (float)g[i], a);
    p[i] = w; m[i] = mi; v[i] = vi;
    if (p_bf16) p_bf16[i] = __float2bfloat16_rn(w);
  }
}

// ================================================================================================
// Vocab-parallel cross-entropy, local pass: per row of this rank's logit shard emit
// {local max, sum exp(x - local max), target logit (0 if the target lives on another rank)}.
// The three values of all ranks are then combined (tiny all-gather) by ce_finalize_kernel.
// ================================================================================================
// Memory bound: the logits are read once. A thread keeps a running maximum and a running sum relative to it (rescaled when the
// maximum moves, once per four 16-byte loads at most), so one pass gives both; four loads are in flight per thread. 4096 x 128256
// bf16 (1.05 GB, 160 us at the copy bandwidth): 1843 us with two passes of 2-byte loads, 202 us now. The scalar form takes rows
// whose length or address is not a multiple of 16 bytes. ROW_THREADS: 512 (the block), or 32 for short rows, where most of a block's
// threads would find nothing to load (see pkb_ce_stats).
constexpr int kCeThreads = 512, kCeWarpFormThreads = 128, kCeUnroll = 4;
constexpr float kLog2eCe = 1.4426950408889634f;

template <typename T, bool VEC, int ROW_THREADS>
__global__ void __launch_bounds__(ROW_THREADS == 32 ? kCeWarpFormThreads : ROW_THREADS)
ce_stats_kernel(const T* __restrict__ logits, const long long* __restrict__ target, float* __restrict__ stats, int rows,
                int vocab_local, long long vocab_start) {
  __shared__ float red_m[kCeThreads / 32], red_s[kCeThreads / 32];
  constexpr int kPer = VEC ? 16 / (int)sizeof(T) : 1;   // elements per load
  constexpr int kUnroll = kCeUnroll;
  constexpr bool kWarpRow = ROW_THREADS == 32;
  constexpr int kRows = kWarpRow ? kCeWarpFormThreads / 32 : 1;   // rows a block works on at a time
  for (int row = blockIdx.x * kRows + (kWarpRow ? (int)threadIdx.x >> 5 : 0); row < rows; row += gridDim.x * kRows) {
    const T* lr = logits + (long long)row * vocab_local;
    float m = -INFINITY, sum = 0.f, off = 0.f;
    for (int base = (threadIdx.x & (ROW_THREADS - 1)) * kPer; base < vocab_local; base += ROW_THREADS * kPer * kUnroll) {
      float f[kUnroll * kPer];
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        const int i = base + u * ROW_THREADS * kPer;
        if (i < vocab_local) {
          if constexpr (!VEC) {
            f[u] = (float)lr[i];
          } else {
            const U4 w = ld_global_nc_v4(lr + i);
            if constexpr (sizeof(T) == 2) {
              const float2 a = unpack_bf16x2(w.x), b = unpack_bf16x2(w.y), c = unpack_bf16x2(w.z), d = unpack_bf16x2(w.w);
              f[u * kPer] = a.x; f[u * kPer + 1] = a.y; f[u * kPer + 2] = b.x; f[u * kPer + 3] = b.y;
              f[u * kPer + 4] = c.x; f[u * kPer + 5] = c.y; f[u * kPer + 6] = d.x; f[u * kPer + 7] = d.y;
            } else {
              f[u * kPer] = __uint_as_float(w.x); f[u * kPer + 1] = __uint_as_float(w.y);
              f[u * kPer + 2] = __uint_as_float(w.z); f[u * kPer + 3] = __uint_as_float(w.w);
            }
          }
        } else {
#pragma unroll
          for (int j = 0; j < kPer; ++j) f[u * kPer + j] = -INFINITY;
        }
      }
      float lm = f[0];
#pragma unroll
      for (int j = 1; j < kUnroll * kPer; ++j) lm = fmaxf(lm, f[j]);
      // off = -m * log2(e), rounded. All terms share its rounding (2e-5 of them at m = 400), which is undone at the end.
      if (lm > m) {
        const float next = -lm * kLog2eCe;
        if (m != -INFINITY) sum *= fast_exp2(next - off);
        m = lm;
        off = next;
      }
#pragma unroll
      for (int j = 0; j < kUnroll * kPer; j += 2) {
        float x0, x1;
        fma2_bcast(x0, x1, f[j], f[j + 1], kLog2eCe, off);
        sum += fast_exp2(x0);
        sum += fast_exp2(x1);
      }
    }
    if (m != -INFINITY) sum *= fast_exp2(fmaf(-m, kLog2eCe, -off));
    const float wm = warp_max(m);
    sum = warp_sum(wm == -INFINITY ? sum : sum * fast_exp2((m - wm) * kLog2eCe));
    float mx = wm, tot = sum;
    if constexpr (!kWarpRow) {
      const int warp = threadIdx.x >> 5;
      if ((threadIdx.x & 31) == 0) { red_m[warp] = wm; red_s[warp] = sum; }
      __syncthreads();
      if (threadIdx.x == 0) {
        mx = red_m[0];
        for (int w = 1; w < kCeThreads / 32; ++w) mx = fmaxf(mx, red_m[w]);
        tot = 0.f;
        for (int w = 0; w < kCeThreads / 32; ++w) tot += mx == -INFINITY ? red_s[w] : red_s[w] * fast_exp2((red_m[w] - mx) * kLog2eCe);
      }
    }
    if ((threadIdx.x & (ROW_THREADS - 1)) == 0) {
      const long long t = target[row] - vocab_start;
      stats[(long long)row * 3 + 0] = mx;
      stats[(long long)row * 3 + 1] = tot;
      stats[(long long)row * 3 + 2] = (t >= 0 && t < vocab_local) ? (float)lr[t] : 0.f;
    }
    if constexpr (!kWarpRow) __syncthreads();
  }
}

// stats_all is [W, rows, 3]; loss[row] = log(sum_w se_w * exp(mx_w - gmax)) + gmax - sum_w tgt_w
__global__ void ce_finalize_kernel(const float* __restrict__ stats_all, float* __restrict__ loss, int rows, int world) {
  for (int row = blockIdx.x * blockDim.x + threadIdx.x; row < rows; row += gridDim.x * blockDim.x) {
    float gmax = -INFINITY;
    for (int w = 0; w < world; ++w) gmax = fmaxf(gmax, stats_all[((long long)w * rows + row) * 3]);
    float se = 0.f, tgt = 0.f;
    for (int w = 0; w < world; ++w) {
      const float* s = stats_all + ((long long)w * rows + row) * 3;
      se += s[1] * __expf(s[0] - gmax);
      tgt += s[2];
    }
    loss[row] = logf(se) + gmax - tgt;
  }
}

// ================================================================================================
// Column reductions of the LayerNorm backward: dgamma[c] = sum_r dY[r,c] * Xhat[r,c], dbeta[c] = sum_r dY[r,c]
// One block per 32-column strip; 32 x 8 threads walk the rows, shared-memory finish. fp32 output.
// ================================================================================================
template <typename T>
__global__ void ln_bwd_colreduce_kernel(const T* __restrict__ xhat, const T* __restrict__ dy,
                                        float* __restrict__ dgamma, float* __restrict__ dbeta, int rows, int cols) {
  __shared__ float sg[8][33], sb[8][33];
  const int c = blockIdx.x * 32 + threadIdx.x;
  float g = 0.f, b = 0.f;
  if (c < cols) {
    for (int r = threadIdx.y; r < rows; r += 8) {
      const float d = (float)dy[(long long)r * cols + c];
      g += d * (float)xhat[(long long)r * cols + c];
      b += d;
    }
  }
  sg[threadIdx.y][threadIdx.x] = g;
  sb[threadIdx.y][threadIdx.x] = b;
  __syncthreads();
  if (threadIdx.y == 0 && c < cols) {
    for (int k = 1; k < 8; ++k) { g += sg[k][threadIdx.x]; b += sb[k][threadIdx.x]; }
    dgamma[c] = g;
    dbeta[c] = b;
  }
}

// ================================================================================================
// Tensor-parallel RMSNorm (hidden dimension sharded): every block owns a set of rows on every rank,
// publishes their local sums of squares in the symmetric heap, crosses ONE in-kernel barrier with the
// same-index blocks of the peers, adds the peers' partial sums and normalises. One launch, no NCCL.
// ================================================================================================
struct TpRmsArgs {
  const __nv_bfloat16* x;
  const __nv_bfloat16* gamma;
  __nv_bfloat16* y;
  int rows, cols_local;
  long long cols_total;
  float eps;
  uint64_t sums_off;  // heap offset of fp32 [rows] partial sums
};

__global__ void __launch_bounds__(256) tp_rmsnorm_kernel(const SymmCtx c, const TpRmsArgs a) {
  __shared__ float red[8];
  float* my_sums = symm_local<float>(c, a.sums_off);
  const int rows_per_block = (a.rows + gridDim.x - 1) / gridDim.x;
  const int r0 = blockIdx.x * rows_per_block;
  const int r1 = min(a.rows, r0 + rows_per_block);
  for (int row = r0; row < r1; ++row) {
    const __nv_bfloat16* xr = a.x + (long long)row * a.cols_local;
    float ss = 0.f;
    for (int i = threadIdx.x * 8; i < a.cols_local; i += blockDim.x * 8) {
      U4 u = ld_global_v4(xr + i);
      float2 f0 = unpack_bf16x2(u.x), f1 = unpack_bf16x2(u.y), f2 = unpack_bf16x2(u.z), f3 = unpack_bf16x2(u.w);
      ss += f0.x * f0.x + f0.y * f0.y + f1.x * f1.x + f1.y * f1.y + f2.x * f2.x + f2.y * f2.y + f3.x * f3.x + f3.y * f3.y;
    }
    ss = warp_sum(ss);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
    __syncthreads();
    if (threadIdx.x == 0) {
      float t = 0.f;
      for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += red[w];
      my_sums[row] = t;
    }
    __syncthreads();
  }
  if (!symm_block_barrier(c, 400, 1)) return;
  for (int row = r0; row < r1; ++row) {
    float tot = 0.f;
    for (int g = 0; g < c.gsize; ++g) tot += symm_ptr<float>(c, c.members[g], a.sums_off)[row];
    const float rstd = rsqrtf(tot / (float)a.cols_total + a.eps);
    const __nv_bfloat16* xr = a.x + (long long)row * a.cols_local;
    __nv_bfloat16* yr = a.y + (long long)row * a.cols_local;
    for (int i = threadIdx.x * 8; i < a.cols_local; i += blockDim.x * 8) {
      U4 u = ld_global_v4(xr + i), g = ld_global_v4(a.gamma + i);
      float2 f0 = unpack_bf16x2(u.x), f1 = unpack_bf16x2(u.y), f2 = unpack_bf16x2(u.z), f3 = unpack_bf16x2(u.w);
      float2 g0 = unpack_bf16x2(g.x), g1 = unpack_bf16x2(g.y), g2 = unpack_bf16x2(g.z), g3 = unpack_bf16x2(g.w);
      U4 o{pack_bf16x2(f0.x * rstd * g0.x, f0.y * rstd * g0.y), pack_bf16x2(f1.x * rstd * g1.x, f1.y * rstd * g1.y),
           pack_bf16x2(f2.x * rstd * g2.x, f2.y * rstd * g2.y), pack_bf16x2(f3.x * rstd * g3.x, f3.y * rstd * g3.y)};
      st_global_v4(yr + i, o);
    }
  }
  // the sums buffer is rewritten by the next call: peers must have read it first
  symm_block_barrier(c, 400, 2);
}

static int grid_1d(long long work_items, int threads, int max_blocks = 148 * 8) {
  long long b = (work_items + threads - 1) / threads;
  if (b < 1) b = 1;
  return (int)(b > max_blocks ? max_blocks : b);
}

static SymmCtx ctx_of(const pkb_symm_ctx* h) {
  SymmCtx c;
  c.base = h->base; c.stride = h->stride; c.mc_base = h->mc_base;
  c.rank = h->rank; c.world = h->world; c.gsize = h->gsize; c.grank = h->grank;
  for (int i = 0; i < kSymmMaxWorld; ++i) c.members[i] = h->members[i];
  c.channel = h->channel;
  c.status = status_block_device_ptr();
  c.budget_ns = h->budget_ns ? h->budget_ns : kDefaultWaitBudgetNs;
  return c;
}

}  // namespace pkb

using namespace pkb;

extern "C" {

// dtype: 0 bf16, 1 fp32
int pkb_rope(const void* x, const void* cos_t, const void* sin_t, void* out, long long tokens, int heads,
             int dim, int dtype, void* stream) {
  PKB_CHECK_ARG(dim % 2 == 0 && tokens >= 0 && heads > 0, "bad RoPE shape");
  if (tokens == 0) return kApiOk;
  const long long total = tokens * heads * (dim / 2);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (dtype == 0)
    rope_kernel<__nv_bfloat16><<<grid_1d(total, 256), 256, 0, s>>>(
        static_cast<const __nv_bfloat16*>(x), static_cast<const __nv_bfloat16*>(cos_t),
        static_cast<const __nv_bfloat16*>(sin_t), static_cast<__nv_bfloat16*>(out), tokens, heads, dim);
  else
    rope_kernel<float><<<grid_1d(total, 256), 256, 0, s>>>(static_cast<const float*>(x), static_cast<const float*>(cos_t),
                                                        static_cast<const float*>(sin_t), static_cast<float*>(out),
                                                        tokens, heads, dim);
  PKB_CHECK_CUDA(cudaGetLastError());
  return kApiOk;
}

int pkb_fp8_quant_1x128(const void* x, void* y, void* scales, long long n, int dtype, int pow2_scales, void* stream) {
  PKB_CHECK_ARG(n % 128 == 0, "element count must be a multiple of 128");
  if (n == 0) return kApiOk;
  const long long nb = n / 128;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  PKB_CHECK_ARG(((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y)) & 15) == 0, "input and payload must be 16-byte aligned");
  const int grid = grid_1d(nb * 8, 256);
  if (dtype == 0)
    fp8_quant_kernel<__nv_bfloat16><<<grid, 256, 0, s>>>(static_cast<const __nv_bfloat16*>(x), static_cast<uint8_t*>(y),
                                                        static_cast<float*>(scales), nb, pow2_scales);
  else
    fp8_quant_kernel<float><<<grid, 256, 0, s>>>(static_cast<const float*>(x), static_cast<uint8_t*>(y),
                                                static_cast<float*>(scales), nb, pow2_scales);
  PKB_CHECK_CUDA(cudaGetLastError());
  return kApiOk;
}

static int launch_fp8_dequant(const void* y, const void* scales, void* x, long long n, int dtype, const int* valid_rows,
                              long long blocks_per_row, void* stream) {
  PKB_CHECK_ARG(n % 128 == 0, "element count must be a multiple of 128");
  PKB_CHECK_ARG((((uintptr_t)y | (uintptr_t)x) & 15) == 0, "buffers must be 16-byte aligned");
  if (n == 0) return kApiOk;
  const long long nb = n / 128;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int grid = grid_1d(nb * 8, 256);
  if (dtype == 0)
    fp8_dequant_kernel<__nv_bfloat16><<<grid, 256, 0, s>>>(static_cast<const uint8_t*>(y), static_cast<const float*>(scales),
                                                          static_cast<__nv_bfloat16*>(x), nb, valid_rows, blocks_per_row);
  else
    fp8_dequant_kernel<float><<<grid, 256, 0, s>>>(static_cast<const uint8_t*>(y), static_cast<const float*>(scales),
                                                  static_cast<float*>(x), nb, valid_rows, blocks_per_row);
  PKB_CHECK_CUDA(cudaGetLastError());
  return kApiOk;
}

int pkb_fp8_dequant_1x128(const void* y, const void* scales, void* x, long long n, int dtype, void* stream) {
  return launch_fp8_dequant(y, scales, x, n, dtype, nullptr, 0, stream);
}

// The same for a [rows, cols] buffer of which only the first *valid_rows rows (an int32 in device memory) hold data.
int pkb_fp8_dequant_1x128_rows(const void* y, const void* scales, void* x, long long rows, long long cols, int dtype,
                               const void* valid_rows, void* stream) {
  PKB_CHECK_ARG(cols % 128 == 0 && valid_rows != nullptr, "cols must be a multiple of 128 and valid_rows given");
  return launch_fp8_dequant(y, scales, x, rows * cols, dtype, static_cast<const int*>(valid_rows), cols / 128, stream);
}

int pkb_adam(void* p, void* m, void* v, const void* g, void* p_bf16, long long n, int grad_dtype, float lr,
             float beta1, float beta2, float eps, float weight_decay, float grad_scale, int step, int decoupled,
             void* stream) {
  PKB_CHECK_ARG(step >= 1, "step counts from 1");
  if (n == 0) return kApiOk;
  AdamArgs a{beta1, beta2, eps, weight_decay, grad_scale, 1.0f - lr * weight_decay,
             (float)(lr / (1.0 - pow((double)beta1, (double)step))), (float)(1.0 / sqrt(1.0 - pow((double)beta2, (double)step))), decoupled};
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const uintptr_t gmask = grad_dtype == 0 ? 7 : 15;
  const bool vec = (((uintptr_t)p | (uintptr_t)m | (uintptr_t)v) & 15) == 0 && ((uintptr_t)g & gmask) == 0 && ((uintptr_t)p_bf16 & 7) == 0;
  const int grid = vec ? grid_1d((n + 7) / 8, 256, 148 * 16) : grid_1d(n, 256);
#define PKB_ADAM(G, V)                                                                                                       \
  adam_kernel<G, V><<<grid, 256, 0, s>>>(static_cast<float*>(p), static_cast<float*>(m), static_cast<float*>(v),             \
                                         static_cast<const G*>(g), static_cast<__nv_bfloat16*>(p_bf16), n, a)
  if (grad_dtype == 0) {
    if (vec) PKB_ADAM(__nv_bfloat16, true); else PKB_ADAM(__nv_bfloat16, false);
  } else {
    if (vec) PKB_ADAM(float, true); else PKB_ADAM(float, false);
  }
#undef PKB_ADAM
  PKB_CHECK_CUDA(cudaGetLastError());
  return kApiOk;
}

int pkb_ce_stats(const void* logits, const void* target, void* stats, int rows, int vocab_local,
                 long long vocab_start, int dtype, void* stream) {
  if (rows == 0) return kApiOk;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int per = dtype == 0 ? 8 : 4;
  const bool vec = vocab_local % per == 0 && ((uintptr_t)logits & 15) == 0;
  // A warp per row up to two of its passes (2048 bf16 elements), and up to eight where the rows fill the GPU. Us, warp / block per
  // row: 8192 x 64 10.2 / 51.2, 8192 x 1000 12.3 / 55.3, 64 x 2048 8.2 / 8.1, 4096 x 8192 20.5 / 45.1; scalar form 8192 x 1001 16.2 / 30.7,
  // 1024 x 4001 20.5 / 12.2.
  const int pass = 32 * kCeUnroll * (vec ? per : 1);
  const bool warp_row = vocab_local <= 2 * pass || (vocab_local <= 8 * pass && rows >= 16 * sm_count());
  const int blocks = warp_row ? (rows + kCeWarpFormThreads / 32 - 1) / (kCeWarpFormThreads / 32) : rows;
  const int grid = blocks < 148 * 8 ? blocks : 148 * 8;
#define PKB_CE2(T, V, R)                                                                                                       \
  ce_stats_kernel<T, V, R><<<grid, R == 32 ? kCeWarpFormThreads : R, 0, s>>>(static_cast<const T*>(logits),                      \
                                                                           static_cast<const long long*>(target),              \
                                                                           static_cast<float*>(stats), rows, vocab_local, vocab_start)
#define PKB_CE(T, V) \
  if (warp_row) PKB_CE2(T, V, 32); else PKB_CE2(T, V, kCeThreads)
  if (dtype == 0) {
    if (vec) { PKB_CE(__nv_bfloat16, true); } else { PKB_CE(__nv_bfloat16, false); }
  } else {
    if (vec) { PKB_CE(float, true); } else { PKB_CE(float, false); }
  }
#undef PKB_CE2
#undef PKB_CE
  PKB_CHECK_CUDA(cudaGetLastError());
  return kApiOk;
}

int pkb_ce_finalize(const void* stats_all, void* loss, int rows, int world, void* stream) {
  if (rows == 0) return kApiOk;
  ce_finalize_kernel<<<grid_1d(rows, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const float*>(stats_all), static_cast<float*>(loss), rows, world);
  PKB_CHECK_CUDA(cudaGetLastError());
  return kApiOk;
}

int pkb_ln_bwd_colreduce(const void* xhat, const void* dy, void* dgamma, void* dbeta, int rows, int cols,
                         int dtype, void* stream) {
  if (cols == 0) return kApiOk;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  dim3 block(32, 8);
  const int grid = (cols + 31) / 32;
  if (dtype == 0)
    ln_bwd_colreduce_kernel<__nv_bfloat16><<<grid, block, 0, s>>>(static_cast<const __nv_bfloat16*>(xhat),
                                                                 static_cast<const __nv_bfloat16*>(dy),
                                                                 static_cast<float*>(dgamma), static_cast<float*>(dbeta),
                                                                 rows, cols);
  else
    ln_bwd_colreduce_kernel<float><<<grid, block, 0, s>>>(static_cast<const float*>(xhat), static_cast<const float*>(dy),
                                                         static_cast<float*>(dgamma), static_cast<float*>(dbeta), rows, cols);
  PKB_CHECK_CUDA(cudaGetLastError());
  return kApiOk;
}

int pkb_tp_rmsnorm(const pkb_symm_ctx* h, const void* x, const void* gamma, void* y, int rows, int cols_local,
                   long long cols_total, float eps, unsigned long long sums_off, void* stream) {
  PKB_CHECK_ARG(h && h->base, "symmetric heap not initialised");
  PKB_CHECK_ARG(cols_local % 8 == 0 && rows > 0, "cols_local must be a multiple of 8");
  TpRmsArgs a{static_cast<const __nv_bfloat16*>(x), static_cast<const __nv_bfloat16*>(gamma),
              static_cast<__nv_bfloat16*>(y), rows, cols_local, cols_total, eps, sums_off};
  int grid = rows < 148 ? rows : 148;
  tp_rmsnorm_kernel<<<grid, 256, 0, static_cast<cudaStream_t>(stream)>>>(ctx_of(h), a);
  PKB_CHECK_CUDA(cudaGetLastError());
  return kApiOk;
}

}  // extern "C"
