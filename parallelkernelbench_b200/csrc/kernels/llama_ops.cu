// Elementwise and row-wise kernels of the decoder layer that are not GEMMs: SwiGLU forward / backward and the RMSNorm
// backward. Each is one pass over its tensors with 16-byte accesses (the framework's autograd would run five to eight
// passes over the [tokens, 2 * ffn] activation). Used by the FSDP Llama step.
#include "pkb/api.h"
#include "pkb/fp8_block.cuh"
#include "pkb/host.h"
#include "pkb/ptx.cuh"

namespace pkb {

// gu: [rows, 2F] bf16 (gate | up); a: [rows, F] = silu(gate) * up
__global__ void __launch_bounds__(256)
swiglu_fwd_kernel(const __nv_bfloat16* __restrict__ gu, __nv_bfloat16* __restrict__ a, long long rows, int F) {
  const long long vec_per_row = F / 8;
  const long long total = rows * vec_per_row;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const long long r = i / vec_per_row;
    const long long c = (i - r * vec_per_row) * 8;
    const U4 g4 = ld_global_v4(gu + r * 2 * F + c), u4 = ld_global_v4(gu + r * 2 * F + F + c);
    const uint32_t gw[4] = {g4.x, g4.y, g4.z, g4.w}, uw[4] = {u4.x, u4.y, u4.z, u4.w};
    uint32_t o[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 g = unpack_bf16x2(gw[j]), u = unpack_bf16x2(uw[j]);
      o[j] = pack_bf16x2(silu_f(g.x) * u.x, silu_f(g.y) * u.y);
    }
    st_global_v4(a + r * F + c, U4{o[0], o[1], o[2], o[3]});
  }
}

// dgate = da * up * s * (1 + gate * (1 - s)), dup = da * gate * s, with s = sigmoid(gate)
__global__ void __launch_bounds__(256)
swiglu_bwd_kernel(const __nv_bfloat16* __restrict__ gu, const __nv_bfloat16* __restrict__ da,
                  __nv_bfloat16* __restrict__ dgu, long long rows, int F) {
  const long long vec_per_row = F / 8;
  const long long total = rows * vec_per_row;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const long long r = i / vec_per_row;
    const long long c = (i - r * vec_per_row) * 8;
    const U4 g4 = ld_global_v4(gu + r * 2 * F + c), u4 = ld_global_v4(gu + r * 2 * F + F + c), d4 = ld_global_v4(da + r * F + c);
    const uint32_t gw[4] = {g4.x, g4.y, g4.z, g4.w}, uw[4] = {u4.x, u4.y, u4.z, u4.w}, dw[4] = {d4.x, d4.y, d4.z, d4.w};
    uint32_t og[4], ou[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 g = unpack_bf16x2(gw[j]), u = unpack_bf16x2(uw[j]), d = unpack_bf16x2(dw[j]);
      const float s0 = 1.f / (1.f + __expf(-g.x)), s1 = 1.f / (1.f + __expf(-g.y));
      og[j] = pack_bf16x2(d.x * u.x * s0 * (1.f + g.x * (1.f - s0)), d.y * u.y * s1 * (1.f + g.y * (1.f - s1)));
      ou[j] = pack_bf16x2(d.x * g.x * s0, d.y * g.y * s1);
    }
    st_global_v4(dgu + r * 2 * F + c, U4{og[0], og[1], og[2], og[3]});
    st_global_v4(dgu + r * 2 * F + F + c, U4{ou[0], ou[1], ou[2], ou[3]});
  }
}

// RMSNorm backward. y = x * rstd * gamma:  dxhat = dy * gamma ;  dx = rstd * (dxhat - xhat * mean(dxhat * xhat)) [+ res] ;
// dgamma = sum_rows dy * xhat. A block walks several rows and keeps its dgamma partial sums in registers (each thread owns
// fixed columns); it writes them to its row of the partial buffer, and rmsnorm_dgamma_kernel adds the rows up in block order
// (no atomics: the result does not depend on which block came first).
// Memory bound: x, dy (and res) are read once and dx written once, as 16-byte accesses; the NEXT row's loads are issued before
// the reduction of the current one, so a block always has a row in flight. 4096 x 4096 (100 MB, 15 us at the copy bandwidth):
// 49 us with 2-byte accesses and a global atomic per block and column, 21 us now and 5 us
// for the partial rows.
// ROW_WARPS: warps that share a row; a block of 8 holds 8 / ROW_WARPS rows at a time. With one
// row per block the other threads of a short row had nothing to do: 16384 x 128 55.5 us, 19.2 now (2-byte form 38.8), 65536 x 64 175 / 31.7
// (124), 4096 x 1024 25.6 / 19.5 (21.5), 2048 x 512 19.2 / 15.3 (16.6).
constexpr int kRmsBwdBlocks = 148 * 2;

// Rows a block holds at a time.
static int rmsnorm_bwd_rows_per_block(int H) { return H <= 256 ? 8 : H <= 512 ? 4 : H <= 1024 ? 2 : 1; }

template <int CH, bool RES, int ROW_WARPS>
__global__ void __launch_bounds__(256)
rmsnorm_bwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ gamma, const __nv_bfloat16* __restrict__ dy,
                   const __nv_bfloat16* __restrict__ res, __nv_bfloat16* __restrict__ dx, float* __restrict__ partial, int rows, int H,
                   float eps, float* __restrict__ dg32, __nv_bfloat16* __restrict__ dg16) {
  constexpr int kRows = 8 / ROW_WARPS, kRowThreads = 32 * ROW_WARPS;
  static_assert(CH == 1 || kRows == 1, "rows of more than one chunk have the block to themselves");
  __shared__ float red[2][2][8];
  float dg[CH][8];
  U4 gam[CH], xc[CH], dc[CH];
  const int slot = (int)threadIdx.x / kRowThreads, tx = (int)threadIdx.x & (kRowThreads - 1);
  const int row0 = blockIdx.x * kRows + slot, step = gridDim.x * kRows;
#pragma unroll
  for (int c = 0; c < CH; ++c) {
    const int i = (c * kRowThreads + tx) * 8;
    gam[c] = xc[c] = dc[c] = U4{0u, 0u, 0u, 0u};
    if (i < H) {
      gam[c] = ld_global_nc_v4(gamma + i);
      if (row0 < rows) {
        xc[c] = ld_global_nc_v4(x + (long long)row0 * H + i);
        dc[c] = ld_global_nc_v4(dy + (long long)row0 * H + i);
      }
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) dg[c][j] = 0.f;
  }
  int par = 0;
  for (int row = row0; row - slot < rows; row += step, par ^= 1) {     // all warps of a block take the same number of steps
    const int nrow = row + step;
    U4 xn[CH], dn[CH], rv[RES ? CH : 1];
#pragma unroll
    for (int c = 0; c < CH; ++c) {
      const int i = (c * kRowThreads + tx) * 8;
      xn[c] = dn[c] = U4{0u, 0u, 0u, 0u};
      if (i < H) {
        if (nrow < rows) {
          xn[c] = ld_global_nc_v4(x + (long long)nrow * H + i);
          dn[c] = ld_global_nc_v4(dy + (long long)nrow * H + i);
        }
        if constexpr (RES) rv[c] = row < rows ? ld_global_nc_v4(res + (long long)row * H + i) : U4{0u, 0u, 0u, 0u};
      }
    }
    float ss = 0.f, dot = 0.f;
#pragma unroll
    for (int c = 0; c < CH; ++c) {
      const uint32_t xw[4] = {xc[c].x, xc[c].y, xc[c].z, xc[c].w}, dw[4] = {dc[c].x, dc[c].y, dc[c].z, dc[c].w},
                     gw[4] = {gam[c].x, gam[c].y, gam[c].z, gam[c].w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 xf = unpack_bf16x2(xw[j]), df = unpack_bf16x2(dw[j]), gf = unpack_bf16x2(gw[j]);
        ss += xf.x * xf.x + xf.y * xf.y;
        dot += df.x * gf.x * xf.x + df.y * gf.y * xf.y;
      }
    }
    ss = warp_sum(ss);
    dot = warp_sum(dot);
    float tss = ss, tdot = dot;
    if constexpr (ROW_WARPS > 1) {
      if ((threadIdx.x & 31) == 0) { red[par][0][threadIdx.x >> 5] = ss; red[par][1][threadIdx.x >> 5] = dot; }
      __syncthreads();     // one per row: the next row writes the other half of red
      tss = tdot = 0.f;
#pragma unroll
      for (int w = 0; w < ROW_WARPS; ++w) { tss += red[par][0][slot * ROW_WARPS + w]; tdot += red[par][1][slot * ROW_WARPS + w]; }
    }
    const float rstd = rsqrtf(tss / (float)H + eps);
    const float mean_term = tdot * rstd / (float)H;      // mean(dxhat * xhat), xhat = x * rstd
#pragma unroll
    for (int c = 0; c < CH; ++c) {
      const int i = (c * kRowThreads + tx) * 8;
      const uint32_t xw[4] = {xc[c].x, xc[c].y, xc[c].z, xc[c].w}, dw[4] = {dc[c].x, dc[c].y, dc[c].z, dc[c].w},
                     gw[4] = {gam[c].x, gam[c].y, gam[c].z, gam[c].w};
      uint32_t o[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 xf = unpack_bf16x2(xw[j]), df = unpack_bf16x2(dw[j]), gf = unpack_bf16x2(gw[j]);
        const float h0 = xf.x * rstd, h1 = xf.y * rstd;
        float a0 = rstd * (df.x * gf.x - h0 * mean_term), a1 = rstd * (df.y * gf.y - h1 * mean_term);
        if constexpr (RES) {
          const uint32_t rw[4] = {rv[c].x, rv[c].y, rv[c].z, rv[c].w};
          const float2 rf = unpack_bf16x2(rw[j]);
          a0 += rf.x;
          a1 += rf.y;
        }
        o[j] = pack_bf16x2(a0, a1);
        if (row < rows) {
          dg[c][2 * j] += df.x * h0;
          dg[c][2 * j + 1] += df.y * h1;
        }
      }
      if (i < H && row < rows) st_global_v4(dx + (long long)row * H + i, U4{o[0], o[1], o[2], o[3]});
      xc[c] = xn[c];
      dc[c] = dn[c];
    }
  }
  // a block by itself has the whole sum: no second launch
  auto emit = [&](int i, const float* v) {
    if (gridDim.x > 1) {
      float4* pr = reinterpret_cast<float4*>(partial + (long long)blockIdx.x * H + i);
      pr[0] = make_float4(v[0], v[1], v[2], v[3]);
      pr[1] = make_float4(v[4], v[5], v[6], v[7]);
      return;
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      if (dg32) dg32[i + j] = v[j];
      if (dg16) dg16[i + j] = __float2bfloat16_rn(v[j]);
    }
  };
  if constexpr (kRows == 1) {
#pragma unroll
    for (int c = 0; c < CH; ++c) {
      const int i = (c * kRowThreads + tx) * 8;
      if (i < H) emit(i, dg[c]);
    }
  } else {                 // the rows of the block, in order
    __shared__ float4 sums[kRows - 1][kRowThreads * 2];
    if (slot > 0) {
      sums[slot - 1][tx] = make_float4(dg[0][0], dg[0][1], dg[0][2], dg[0][3]);
      sums[slot - 1][kRowThreads + tx] = make_float4(dg[0][4], dg[0][5], dg[0][6], dg[0][7]);
    }
    __syncthreads();
    if (slot == 0 && tx * 8 < H) {
#pragma unroll
      for (int r = 0; r < kRows - 1; ++r) {
        const float4 a = sums[r][tx], b = sums[r][kRowThreads + tx];
        dg[0][0] += a.x; dg[0][1] += a.y; dg[0][2] += a.z; dg[0][3] += a.w;
        dg[0][4] += b.x; dg[0][5] += b.y; dg[0][6] += b.z; dg[0][7] += b.w;
      }
      emit(tx * 8, dg[0]);
    }
  }
}

// dgamma[c] = sum over the blocks' partial rows, in order: 32 columns per block, eight threads per column take every eighth row.
__global__ void __launch_bounds__(256)
rmsnorm_dgamma_kernel(const float* __restrict__ partial, int nblk, int H, float* __restrict__ dg32, __nv_bfloat16* __restrict__ dg16) {
  __shared__ float s[8][33];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int c = blockIdx.x * 32 + tx;
  float acc = 0.f;
  if (c < H)
    for (int b = ty; b < nblk; b += 8) acc += partial[(long long)b * H + c];
  s[ty][tx] = acc;
  __syncthreads();
  if (ty == 0 && c < H) {
#pragma unroll
    for (int k = 1; k < 8; ++k) acc += s[k][tx];
    if (dg32) dg32[c] = acc;
    if (dg16) dg16[c] = __float2bfloat16_rn(acc);
  }
}

// The form for hidden sizes that are not a multiple of 8 and for tensors off the 16-byte boundary (2-byte accesses, one global atomic
// per block and column).
template <int COLS_PER_THREAD>
__global__ void __launch_bounds__(256)
rmsnorm_bwd_scalar_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ gamma,
                   const __nv_bfloat16* __restrict__ dy, __nv_bfloat16* __restrict__ dx, float* __restrict__ dgamma,
                   int rows, int H, float eps) {
  __shared__ float red[2][8];
  float gam[COLS_PER_THREAD], dg[COLS_PER_THREAD];
#pragma unroll
  for (int j = 0; j < COLS_PER_THREAD; ++j) {
    const int c = threadIdx.x + j * 256;
    gam[j] = c < H ? __bfloat162float(gamma[c]) : 0.f;
    dg[j] = 0.f;
  }
  for (int row = blockIdx.x; row < rows; row += gridDim.x) {
    const __nv_bfloat16* xr = x + (long long)row * H;
    const __nv_bfloat16* dyr = dy + (long long)row * H;
    float xv[COLS_PER_THREAD], dv[COLS_PER_THREAD];
    float ss = 0.f, dot = 0.f;
#pragma unroll
    for (int j = 0; j < COLS_PER_THREAD; ++j) {
      const int c = threadIdx.x + j * 256;
      xv[j] = c < H ? __bfloat162float(xr[c]) : 0.f;
      dv[j] = c < H ? __bfloat162float(dyr[c]) : 0.f;
      ss += xv[j] * xv[j];
      dot += dv[j] * gam[j] * xv[j];
    }
    ss = warp_sum(ss);
    dot = warp_sum(dot);
    if ((threadIdx.x & 31) == 0) { red[0][threadIdx.x >> 5] = ss; red[1][threadIdx.x >> 5] = dot; }
    __syncthreads();
    float tss = 0.f, tdot = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) { tss += red[0][w]; tdot += red[1][w]; }
    __syncthreads();
    const float rstd = rsqrtf(tss / (float)H + eps);
    const float mean_term = tdot * rstd / (float)H;      // mean(dxhat * xhat), xhat = x * rstd
#pragma unroll
    for (int j = 0; j < COLS_PER_THREAD; ++j) {
      const int c = threadIdx.x + j * 256;
      if (c < H) {
        const float xhat = xv[j] * rstd;
        dx[(long long)row * H + c] = __float2bfloat16_rn(rstd * (dv[j] * gam[j] - xhat * mean_term));
        dg[j] += dv[j] * xhat;
      }
    }
  }
#pragma unroll
  for (int j = 0; j < COLS_PER_THREAD; ++j) {
    const int c = threadIdx.x + j * 256;
    if (c < H) atomicAdd(dgamma + c, dg[j]);
  }
}

// d logits of the mean cross-entropy over a vocabulary shard: (exp(logit - lse) - [col == target - vocab_start]) * scale,
// written as bf16 in one pass (lse is the GLOBAL log-sum-exp of the row, natural log).
// A block takes 8192 columns of one row at a time, four 16-byte loads in flight per thread, and the row's constants are read once
// per block instead of once per 16 bytes. 4096 x 128256 (2.1 GB, 321 us at the copy bandwidth): 332 us, 415 us with the form below.
constexpr int kCeBwdCols = 256 * 8 * 4;

// Eight columns; t: the target's column relative to the first of them.
__device__ __forceinline__ U4 ce_bwd8(const U4& v, float l, long long t, float scale) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
  uint32_t o[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 f = unpack_bf16x2(w[j]);
    const float a = (__expf(f.x - l) - (t == 2 * j ? 1.f : 0.f)) * scale;
    const float b = (__expf(f.y - l) - (t == 2 * j + 1 ? 1.f : 0.f)) * scale;
    o[j] = pack_bf16x2(a, b);
  }
  return U4{o[0], o[1], o[2], o[3]};
}

__global__ void __launch_bounds__(256)
ce_bwd_kernel(const __nv_bfloat16* __restrict__ logits, const float* __restrict__ lse, const long long* __restrict__ target,
              __nv_bfloat16* __restrict__ dlog, long long rows, int V, long long vocab_start, float scale,
              const float* __restrict__ upstream) {
  if (upstream != nullptr) scale *= *upstream;     // gradient of the loss itself, kept on the device
  const int c_base = blockIdx.x * kCeBwdCols + (int)threadIdx.x * 8;
  for (long long r = blockIdx.y; r < rows; r += gridDim.y) {
    const float l = lse[r];
    const long long t = target[r] - vocab_start;
    const __nv_bfloat16* src = logits + r * V;
    __nv_bfloat16* dst = dlog + r * V;
    U4 v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (c_base + u * 2048 < V) v[u] = ld_global_nc_v4(src + c_base + u * 2048);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int c = c_base + u * 2048;
      if (c >= V) break;
      st_global_v4(dst + c, ce_bwd8(v[u], l, t - c, scale));
    }
  }
}

// Rows of fewer than 8192 columns, which would leave threads of such a block without a load: 16 bytes per thread across row ends.
// Us, this / the form above: 8192 x 64 6.7 / 22.6, 8192 x 1000 14.2 / 24.7, 4096 x 4096 20.5 / 22.6, 4096 x 8192 34.7 / 28.7.
__global__ void __launch_bounds__(256)
ce_bwd_short_kernel(const __nv_bfloat16* __restrict__ logits, const float* __restrict__ lse, const long long* __restrict__ target,
                    __nv_bfloat16* __restrict__ dlog, long long rows, int V, long long vocab_start, float scale,
                    const float* __restrict__ upstream) {
  if (upstream != nullptr) scale *= *upstream;
  const long long vec_per_row = V / 8;
  const long long total = rows * vec_per_row;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const long long r = i / vec_per_row;
    const int c = (int)(i - r * vec_per_row) * 8;
    st_global_v4(dlog + r * V + c, ce_bwd8(ld_global_nc_v4(logits + r * V + c), lse[r], target[r] - vocab_start - c, scale));
  }
}

// From the statistics of every rank's vocabulary shard ([W, rows, 3]: maximum, sum of exponentials relative to it, target
// logit or 0) the log-sum-exp per row and the mean loss. One block: a few thousand rows of 12 bytes, bound by the latency of
// one launch; it replaces nine elementwise and reduction launches. Rows are added in a fixed order.
__global__ void __launch_bounds__(1024)
ce_loss_kernel(const float* __restrict__ stats, int rows, int world, float* __restrict__ lse, float* __restrict__ loss) {
  __shared__ float red[32];
  float acc = 0.f;
  for (int r = threadIdx.x; r < rows; r += 1024) {
    float gmax = -INFINITY;
    for (int w = 0; w < world; ++w) gmax = fmaxf(gmax, stats[((long long)w * rows + r) * 3]);
    float se = 0.f, tgt = 0.f;
    for (int w = 0; w < world; ++w) {
      const float* st = stats + ((long long)w * rows + r) * 3;
      se += st[1] * expf(st[0] - gmax);
      tgt += st[2];
    }
    const float l = logf(se) + gmax;
    lse[r] = l;
    acc += l - tgt;
  }
  acc = warp_sum(acc);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x < 32) {
    acc = warp_sum(red[threadIdx.x]);
    if (threadIdx.x == 0) *loss = acc / (float)rows;
  }
}

// [S, (hq + 2 hkv) d] (the QKV projection) -> q [S, hq, d] and k [S, hkv, d] with rotate-half RoPE applied, v [S, hkv, d]. A thread
// owns 8 columns of one half of a head and the 8 matching ones of the other half. Memory bound; one pass where the separate
// form took three slice copies and two rotations (6 launches with their backward's negated sine, 10 passes over the projection).
__global__ void __launch_bounds__(256)
qkv_rope_split_kernel(const __nv_bfloat16* __restrict__ qkv, const __nv_bfloat16* __restrict__ cs, const __nv_bfloat16* __restrict__ sn,
                      __nv_bfloat16* __restrict__ q, __nv_bfloat16* __restrict__ k, __nv_bfloat16* __restrict__ v, int tokens, int hq,
                      int hkv, int d) {
  const int per = d >> 4, half = d >> 1, heads = hq + 2 * hkv;
  const unsigned total = (unsigned)tokens * heads * per;
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    const unsigned th = i / per, j = (i - th * per) * 8;
    const unsigned t = th / heads, h = th - t * heads;
    const __nv_bfloat16* src = qkv + (long long)th * d + j;
    U4 lo = ld_global_nc_v4(src), hi = ld_global_nc_v4(src + half);
    __nv_bfloat16* dst;
    if (h < (unsigned)(hq + hkv)) {
      const __nv_bfloat16 *cp = cs + (long long)t * d + j, *sp = sn + (long long)t * d + j;
      const U4 c1 = ld_global_nc_v4(cp), c2 = ld_global_nc_v4(cp + half), s1 = ld_global_nc_v4(sp), s2 = ld_global_nc_v4(sp + half);
      uint32_t a[4] = {lo.x, lo.y, lo.z, lo.w}, b[4] = {hi.x, hi.y, hi.z, hi.w};
      const uint32_t c1w[4] = {c1.x, c1.y, c1.z, c1.w}, c2w[4] = {c2.x, c2.y, c2.z, c2.w}, s1w[4] = {s1.x, s1.y, s1.z, s1.w},
                     s2w[4] = {s2.x, s2.y, s2.z, s2.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 x1 = unpack_bf16x2(a[e]), x2 = unpack_bf16x2(b[e]), C1 = unpack_bf16x2(c1w[e]), C2 = unpack_bf16x2(c2w[e]),
                     S1 = unpack_bf16x2(s1w[e]), S2 = unpack_bf16x2(s2w[e]);
        a[e] = pack_bf16x2(x1.x * C1.x - x2.x * S1.x, x1.y * C1.y - x2.y * S1.y);
        b[e] = pack_bf16x2(x2.x * C2.x + x1.x * S2.x, x2.y * C2.y + x1.y * S2.y);
      }
      lo = U4{a[0], a[1], a[2], a[3]};
      hi = U4{b[0], b[1], b[2], b[3]};
      dst = h < (unsigned)hq ? q + ((long long)t * hq + h) * d + j : k + ((long long)t * hkv + (h - hq)) * d + j;
    } else {
      dst = v + ((long long)t * hkv + (h - hq - hkv)) * d + j;
    }
    st_global_v4(dst, lo);
    st_global_v4(dst + half, hi);
  }
}

__device__ __forceinline__ void load8_f32(const float* p, float (&f)[8]) {
  const U4 a = ld_global_nc_v4(p), b = ld_global_nc_v4(p + 4);
  f[0] = __uint_as_float(a.x); f[1] = __uint_as_float(a.y); f[2] = __uint_as_float(a.z); f[3] = __uint_as_float(a.w);
  f[4] = __uint_as_float(b.x); f[5] = __uint_as_float(b.y); f[6] = __uint_as_float(b.z); f[7] = __uint_as_float(b.w);
}

// The way back: fp32 dq, dk, dv of the attention backward -> the bf16 gradient of the packed projection, the rotation undone
// (sine negated) before the one rounding. One pass instead of three casts, two rotations with negated tables and a concatenation.
__global__ void __launch_bounds__(256)
qkv_rope_merge_kernel(const float* __restrict__ dq, const float* __restrict__ dk, const float* __restrict__ dv,
                      const __nv_bfloat16* __restrict__ cs, const __nv_bfloat16* __restrict__ sn, __nv_bfloat16* __restrict__ dqkv,
                      int tokens, int hq, int hkv, int d) {
  const int per = d >> 4, half = d >> 1, heads = hq + 2 * hkv;
  const unsigned total = (unsigned)tokens * heads * per;
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    const unsigned th = i / per, j = (i - th * per) * 8;
    const unsigned t = th / heads, h = th - t * heads;
    const float* src = h < (unsigned)hq ? dq + ((long long)t * hq + h) * d + j
                       : h < (unsigned)(hq + hkv) ? dk + ((long long)t * hkv + (h - hq)) * d + j
                                                  : dv + ((long long)t * hkv + (h - hq - hkv)) * d + j;
    float a[8], b[8];
    load8_f32(src, a);
    load8_f32(src + half, b);
    if (h < (unsigned)(hq + hkv)) {
      const __nv_bfloat16 *cp = cs + (long long)t * d + j, *sp = sn + (long long)t * d + j;
      const U4 c1 = ld_global_nc_v4(cp), c2 = ld_global_nc_v4(cp + half), s1 = ld_global_nc_v4(sp), s2 = ld_global_nc_v4(sp + half);
      const uint32_t c1w[4] = {c1.x, c1.y, c1.z, c1.w}, c2w[4] = {c2.x, c2.y, c2.z, c2.w}, s1w[4] = {s1.x, s1.y, s1.z, s1.w},
                     s2w[4] = {s2.x, s2.y, s2.z, s2.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 C1 = unpack_bf16x2(c1w[e]), C2 = unpack_bf16x2(c2w[e]), S1 = unpack_bf16x2(s1w[e]), S2 = unpack_bf16x2(s2w[e]);
        const float a0 = a[2 * e], a1 = a[2 * e + 1], b0 = b[2 * e], b1 = b[2 * e + 1];
        a[2 * e] = a0 * C1.x + b0 * S1.x; a[2 * e + 1] = a1 * C1.y + b1 * S1.y;
        b[2 * e] = b0 * C2.x - a0 * S2.x; b[2 * e + 1] = b1 * C2.y - a1 * S2.y;
      }
    }
    __nv_bfloat16* dst = dqkv + (long long)th * d + j;
    st_global_v4(dst, U4{pack_bf16x2(a[0], a[1]), pack_bf16x2(a[2], a[3]), pack_bf16x2(a[4], a[5]), pack_bf16x2(a[6], a[7])});
    st_global_v4(dst + half, U4{pack_bf16x2(b[0], b[1]), pack_bf16x2(b[2], b[3]), pack_bf16x2(b[4], b[5]), pack_bf16x2(b[6], b[7])});
  }
}

// out = a + b over bf16, n a multiple of 8 (residual connections)
__global__ void __launch_bounds__(256)
add_bf16_kernel(const __nv_bfloat16* __restrict__ a, const __nv_bfloat16* __restrict__ b, __nv_bfloat16* __restrict__ out, long long nvec) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < nvec; i += (long long)gridDim.x * blockDim.x) {
    const U4 x = ld_global_nc_v4(a + i * 8), y = ld_global_nc_v4(b + i * 8);
    const uint32_t xw[4] = {x.x, x.y, x.z, x.w}, yw[4] = {y.x, y.y, y.z, y.w};
    uint32_t o[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 f = unpack_bf16x2(xw[j]), g = unpack_bf16x2(yw[j]);
      o[j] = pack_bf16x2(f.x + g.x, f.y + g.y);
    }
    st_global_v4(out + i * 8, U4{o[0], o[1], o[2], o[3]});
  }
}

// Embedding lookup from the wire format: row `tokens[t]` of a [vocab, H] table held as e4m3 bytes with one fp32 scale per 128
// consecutive elements, as bf16. Only the rows that are looked up are converted (the whole table is 1.6 GB of traffic at
// 128256 x 4096, 245 us; 4096 rows of it are 50 MB). A token outside the table gives a zero row and a status word.
constexpr uint32_t kEmbedKernelId = 910;

__global__ void __launch_bounds__(256)
embed_fp8_kernel(const uint8_t* __restrict__ table, const float* __restrict__ scales, const long long* __restrict__ tokens,
                 __nv_bfloat16* __restrict__ out, int n_tokens, int vocab, int H, uint32_t* status) {
  const int per_row = H >> 4;
  const unsigned total = (unsigned)n_tokens * per_row;
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    const unsigned t = i / per_row, c = (i - t * per_row) * 16;
    const long long tok = tokens[t];
    uint32_t o[8] = {0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u};
    if (tok >= 0 && tok < vocab) {
      const long long e = tok * H + c;
      const U4 u = ld_global_nc_v4(table + e);
      const float sc = scales[e >> 7];
      const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        __half2_raw h0 = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)(w[j] & 0xffffu), __NV_E4M3);
        __half2_raw h1 = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)(w[j] >> 16), __NV_E4M3);
        const float2 f0 = __half22float2(*reinterpret_cast<__half2*>(&h0)), f1 = __half22float2(*reinterpret_cast<__half2*>(&h1));
        o[2 * j] = pack_bf16x2(f0.x * sc, f0.y * sc);
        o[2 * j + 1] = pack_bf16x2(f1.x * sc, f1.y * sc);
      }
    } else if (c == 0) {
      record_status(status, kStatusBadArgument, kEmbedKernelId, 0, 0, 1, t);
    }
    st_global_v4(out + (long long)t * H + c, U4{o[0], o[1], o[2], o[3]});
    st_global_v4(out + (long long)t * H + c + 8, U4{o[4], o[5], o[6], o[7]});
  }
}

// Gradient of the lookup, written straight in the wire format of the gradient exchange (e4m3 bytes, one fp32 scale per 128
// elements): one block per position t. The block of a token's FIRST position adds the gradient rows of all positions of that
// token in order (fp32), rounds to bf16 as a dense gradient tensor would hold it, and quantises; the other blocks leave. Rows
// no token touched are the caller's zero bytes with scale 1, which is what quantising a zero row gives. Nothing of the
// size of the table is read, and no dense bf16 gradient exists: it was 1.05 GB filled, copied and quantised per step.
// Finding the positions of a token is one scan of the token list by every block into a bit mask (L2 hits; fine up to
// kEmbedMaxTokens). A token that is there often (padding, a frequent word) is one block's work however often it comes, so its rows
// are loaded eight at a time: the step at 4096 x 4096 with one token for all positions 5.5 + 1.0 ms (one row at a time 15.4).
constexpr int kEmbedMaxTokens = 16384;
constexpr int kEmbedGradThreads = 256;

__global__ void __launch_bounds__(kEmbedGradThreads)
embed_grad_fp8_kernel(const __nv_bfloat16* __restrict__ dx, const long long* __restrict__ tokens, int n_tokens, int vocab, int H,
                      uint8_t* __restrict__ q, float* __restrict__ s, uint32_t* status) {
  extern __shared__ uint32_t hits[];                   // one bit per other position that holds the same token
  __shared__ int s_earlier, s_count;
  constexpr int kWarps = kEmbedGradThreads / 32, kFlight = 8;
  const int t = blockIdx.x;
  const long long tok = tokens[t];
  if (tok < 0 || tok >= vocab) {
    if (threadIdx.x == 0) record_status(status, kStatusBadArgument, kEmbedKernelId, 0, 0, 2, t);
    return;
  }
  if (threadIdx.x == 0) s_earlier = s_count = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int words = (n_tokens + 31) >> 5;
  uint16_t* list = reinterpret_cast<uint16_t*>(hits + words);      // those positions, in order
  for (int w0 = warp * 4; w0 < words; w0 += kWarps * 4) {
    long long v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) v[u] = (w0 + u) * 32 + lane < n_tokens ? tokens[(w0 + u) * 32 + lane] : -1;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int w = w0 + u;
      const unsigned m = __ballot_sync(0xffffffffu, v[u] == tok && w * 32 + lane != t);
      if (lane == 0 && w < words) {
        hits[w] = m;
        if (m) {
          if (w * 32 + __ffs(m) - 1 < t) s_earlier = 1;
          else s_count = 1;
        }
      }
    }
  }
  __syncthreads();
  if (s_earlier) return;
  const bool later = s_count != 0;
  __syncthreads();
  if (later && warp == 0) {
    int base = 0;
    for (int w0 = t >> 5; w0 < words; w0 += 32) {
      unsigned m = w0 + lane < words ? hits[w0 + lane] : 0u;
      int incl = __popc(m);
      const int mine = incl;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int up = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += up;
      }
      for (int at = base + incl - mine; m; m &= m - 1) list[at++] = (uint16_t)((w0 + lane) * 32 + __ffs(m) - 1);
      base += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) s_count = base;
  }
  __syncthreads();
  const int count = later ? s_count : 0;
  for (int c0 = warp * 256; c0 < H; c0 += kWarps * 256) {        // two 128-element groups of the row (H % 128 == 0)
    const int c = c0 + lane * 8;
    const bool in = c < H;
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    auto add = [&](const U4& v) {
      const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 f = unpack_bf16x2(w[j]);
        acc[2 * j] += f.x;
        acc[2 * j + 1] += f.y;
      }
    };
    if (in) add(ld_global_nc_v4(dx + (long long)t * H + c));
    for (int k = 0; k < count; k += kFlight) {
      U4 v[kFlight];
#pragma unroll
      for (int u = 0; u < kFlight; ++u) {
        v[u] = U4{0u, 0u, 0u, 0u};
        if (in && k + u < count) v[u] = ld_global_nc_v4(dx + (long long)list[k + u] * H + c);
      }
#pragma unroll
      for (int u = 0; u < kFlight; ++u)
        if (k + u < count) add(v[u]);
    }
    float amax = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      acc[j] = __bfloat162float(__float2bfloat16_rn(acc[j]));
      amax = fmaxf(amax, fabsf(acc[j]));
    }
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    const float sc = fp8_block_scale(amax, 0);
    uint32_t codes[2];
    fp8_encode8(acc, sc, codes);
    if (in) {
      const long long e = tok * H + c;
      *reinterpret_cast<uint2*>(q + e) = make_uint2(codes[0], codes[1]);
      if ((lane & 15) == 0) s[e >> 7] = sc;
    }
  }
}

}  // namespace pkb

using namespace pkb;

extern "C" int pkb_ce_bwd(const void* logits, const void* lse, const void* target, void* dlog, long long rows, int V,
                          long long vocab_start, float scale, const void* upstream, void* stream) {
  PKB_CHECK_ARG(rows >= 0 && V > 0 && V % 8 == 0, "the vocabulary shard must be a positive multiple of 8");
  if (rows == 0) return kApiOk;
  const __nv_bfloat16* src = static_cast<const __nv_bfloat16*>(logits);
  const float *lp = static_cast<const float*>(lse), *up = static_cast<const float*>(upstream);
  const long long* tp = static_cast<const long long*>(target);
  __nv_bfloat16* dst = static_cast<__nv_bfloat16*>(dlog);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (V < kCeBwdCols) {
    long long blocks = (rows * (V / 8) + 255) / 256;
    if (blocks > 148 * 16) blocks = 148 * 16;
    ce_bwd_short_kernel<<<(int)blocks, 256, 0, s>>>(src, lp, tp, dst, rows, V, vocab_start, scale, up);
  } else {
    dim3 grid((V + kCeBwdCols - 1) / kCeBwdCols, rows < 32768 ? (unsigned)rows : 32768u);
    ce_bwd_kernel<<<grid, 256, 0, s>>>(src, lp, tp, dst, rows, V, vocab_start, scale, up);
  }
  PKB_CHECK_CUDA(cudaGetLastError());
  return kApiOk;
}

extern "C" int pkb_swiglu_fwd(const void* gu, void* a, long long rows, int F, void* stream) {
  PKB_CHECK_ARG(rows >= 0 && F > 0 && F % 8 == 0, "F must be a positive multiple of 8");
  if (rows == 0) return kApiOk;
  long long blocks = (rows * (F / 8) + 255) / 256;
  if (blocks > 148 * 16) blocks = 148 * 16;
  swiglu_fwd_kernel<<<(int)blocks, 256, 0, static_cast<cudaStream_t>(stream)>>>(static_cast<const __nv_bfloat16*>(gu),
                                                                                static_cast<__nv_bfloat16*>(a), rows, F);
  PKB_CHECK_CUDA(cudaGetLastError());
  return kApiOk;
}

extern "C" int pkb_swiglu_bwd(const void* gu, const void* da, void* dgu, long long rows, int F, void* stream) {
  PKB_CHECK_ARG(rows >= 0 && F > 0 && F % 8 == 0, "F must be a positive multiple of 8");
  if (rows == 0) return kApiOk;
  long long blocks = (rows * (F / 8) + 255) / 256;
  if (blocks > 148 * 16) blocks = 148 * 16;
  swiglu_bwd_kernel<<<(int)blocks, 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const __nv_bfloat16*>(gu), static_cast<const __nv_bfloat16*>(da), static_cast<__nv_bfloat16*>(dgu), rows, F);
  PKB_CHECK_CUDA(cudaGetLastError());
  return kApiOk;
}

// Rows of the partial buffer ([rows of it][H] fp32) that pkb_rmsnorm_bwd wants for this many input rows; 0 for hidden sizes
// that take the scalar form.
extern "C" int pkb_rmsnorm_bwd_partials(int rows, int H) {
  if (H % 8 != 0) return 0;
  const int per = rmsnorm_bwd_rows_per_block(H), blocks = (int)(((long long)rows + per - 1) / per);
  if (blocks <= 4) return rows > 0 ? 1 : 0;      // a few steps of one block are shorter than the second launch
  return blocks < kRmsBwdBlocks ? blocks : kRmsBwdBlocks;
}

// dx = gradient of the norm (+ res, bf16 [rows, H], may be null); the gain's gradient goes to dgamma (fp32 [H], may be null) and
// dgamma_bf16 (may be null). partial: scratch of pkb_rmsnorm_bwd_partials(rows, H) x H fp32 values.
// H % 8 != 0, or partial null (tensors off the 16-byte boundary): res and dgamma_bf16 must be null and dgamma is accumulated into
// (zero-filled by the caller).
extern "C" int pkb_rmsnorm_bwd(const void* x, const void* gamma, const void* dy, const void* res, void* dx, void* dgamma,
                               void* dgamma_bf16, void* partial, int rows, int H, float eps, void* stream) {
  PKB_CHECK_ARG(rows >= 0 && H > 0 && H <= 256 * 32, "hidden size must be at most 8192");
  if (rows == 0) return kApiOk;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const __nv_bfloat16 *xp = static_cast<const __nv_bfloat16*>(x), *gp = static_cast<const __nv_bfloat16*>(gamma),
                      *dyp = static_cast<const __nv_bfloat16*>(dy), *rp = static_cast<const __nv_bfloat16*>(res);
  __nv_bfloat16* dxp = static_cast<__nv_bfloat16*>(dx);
  float* dgp = static_cast<float*>(dgamma);
  if (H % 8 == 0 && partial != nullptr) {
    PKB_CHECK_ARG((((uintptr_t)x | (uintptr_t)gamma | (uintptr_t)dy | (uintptr_t)res | (uintptr_t)dx | (uintptr_t)partial) & 15) == 0,
                  "the partial buffer goes with 16-byte aligned tensors");
    const int blocks = pkb_rmsnorm_bwd_partials(rows, H);
    float* pp = static_cast<float*>(partial);
    __nv_bfloat16* dg16 = static_cast<__nv_bfloat16*>(dgamma_bf16);
#define PKB_RMSB(CH, RW)                                                                                                       \
    {                                                                                                                          \
      if (rp) rmsnorm_bwd_kernel<CH, true, RW><<<blocks, 256, 0, s>>>(xp, gp, dyp, rp, dxp, pp, rows, H, eps, dgp, dg16);       \
      else rmsnorm_bwd_kernel<CH, false, RW><<<blocks, 256, 0, s>>>(xp, gp, dyp, rp, dxp, pp, rows, H, eps, dgp, dg16);         \
    }
    switch (rmsnorm_bwd_rows_per_block(H)) {
      case 8: PKB_RMSB(1, 1) break;
      case 4: PKB_RMSB(1, 2) break;
      case 2: PKB_RMSB(1, 4) break;
      default:
        if (H <= 2048) PKB_RMSB(1, 8) else if (H <= 4096) PKB_RMSB(2, 8) else PKB_RMSB(4, 8)
    }
#undef PKB_RMSB
    if (blocks > 1)
      rmsnorm_dgamma_kernel<<<(H + 31) / 32, 256, 0, s>>>(pp, blocks, H, dgp, dg16);
  } else {
    PKB_CHECK_ARG(res == nullptr && dgamma_bf16 == nullptr && dgamma != nullptr, "the scalar form has no residual and writes an fp32 gain gradient");
    const int blocks = rows < 148 * 4 ? rows : 148 * 4;
    if (H <= 256 * 4) rmsnorm_bwd_scalar_kernel<4><<<blocks, 256, 0, s>>>(xp, gp, dyp, dxp, dgp, rows, H, eps);
    else if (H <= 256 * 16) rmsnorm_bwd_scalar_kernel<16><<<blocks, 256, 0, s>>>(xp, gp, dyp, dxp, dgp, rows, H, eps);
    else rmsnorm_bwd_scalar_kernel<32><<<blocks, 256, 0, s>>>(xp, gp, dyp, dxp, dgp, rows, H, eps);
  }
  PKB_CHECK_CUDA(cudaGetLastError());
  return kApiOk;
}

// stats fp32 [W, rows, 3] -> lse fp32 [rows] and the mean loss (fp32 scalar)
extern "C" int pkb_ce_loss(const void* stats, int rows, int world, void* lse, void* loss, void* stream) {
  PKB_CHECK_ARG(rows > 0 && world >= 1, "at least one row");
  ce_loss_kernel<<<1, 1024, 0, static_cast<cudaStream_t>(stream)>>>(static_cast<const float*>(stats), rows, world, static_cast<float*>(lse),
                                                                    static_cast<float*>(loss));
  PKB_CHECK_CUDA(cudaGetLastError());
  return kApiOk;
}

static int qkv_rope_check(const void* a, const void* b, const void* c, const void* e, long long tokens, int hq, int hkv, int d) {
  PKB_CHECK_ARG(tokens >= 0 && hq > 0 && hkv > 0 && d > 0 && d % 16 == 0, "head dimension must be a multiple of 16");
  PKB_CHECK_ARG(tokens * (hq + 2 * hkv) * (d / 16) < (1ll << 31), "too many elements for one call");
  PKB_CHECK_ARG((((uintptr_t)a | (uintptr_t)b | (uintptr_t)c | (uintptr_t)e) & 15) == 0, "tensors must be 16-byte aligned");
  return kApiOk;
}

static int qkv_rope_grid(long long tokens, int hq, int hkv, int d) {
  const long long blocks = (tokens * (hq + 2 * hkv) * (d / 16) + 255) / 256;
  return (int)(blocks > 148 * 8 ? 148 * 8 : blocks);
}

extern "C" int pkb_qkv_rope_split(const void* qkv, const void* cos_t, const void* sin_t, void* q, void* k, void* v, int tokens, int hq,
                                  int hkv, int d, void* stream) {
  if (int rc = qkv_rope_check(qkv, q, k, v, tokens, hq, hkv, d)) return rc;
  if (tokens == 0) return kApiOk;
  qkv_rope_split_kernel<<<qkv_rope_grid(tokens, hq, hkv, d), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const __nv_bfloat16*>(qkv), static_cast<const __nv_bfloat16*>(cos_t), static_cast<const __nv_bfloat16*>(sin_t),
      static_cast<__nv_bfloat16*>(q), static_cast<__nv_bfloat16*>(k), static_cast<__nv_bfloat16*>(v), tokens, hq, hkv, d);
  PKB_CHECK_CUDA(cudaGetLastError());
  return kApiOk;
}

extern "C" int pkb_qkv_rope_merge(const void* dq, const void* dk, const void* dv, const void* cos_t, const void* sin_t, void* dqkv,
                                  int tokens, int hq, int hkv, int d, void* stream) {
  if (int rc = qkv_rope_check(dq, dk, dv, dqkv, tokens, hq, hkv, d)) return rc;
  if (tokens == 0) return kApiOk;
  qkv_rope_merge_kernel<<<qkv_rope_grid(tokens, hq, hkv, d), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const float*>(dq), static_cast<const float*>(dk), static_cast<const float*>(dv), static_cast<const __nv_bfloat16*>(cos_t),
      static_cast<const __nv_bfloat16*>(sin_t), static_cast<__nv_bfloat16*>(dqkv), tokens, hq, hkv, d);
  PKB_CHECK_CUDA(cudaGetLastError());
  return kApiOk;
}

extern "C" int pkb_add_bf16(const void* a, const void* b, void* out, long long n, void* stream) {
  PKB_CHECK_ARG(n >= 0 && n % 8 == 0 && (((uintptr_t)a | (uintptr_t)b | (uintptr_t)out) & 15) == 0, "a multiple of 8 elements, 16-byte aligned");
  if (n == 0) return kApiOk;
  long long blocks = (n / 8 + 255) / 256;
  if (blocks > 148 * 8) blocks = 148 * 8;
  add_bf16_kernel<<<(int)blocks, 256, 0, static_cast<cudaStream_t>(stream)>>>(static_cast<const __nv_bfloat16*>(a),
                                                                              static_cast<const __nv_bfloat16*>(b), static_cast<__nv_bfloat16*>(out), n / 8);
  PKB_CHECK_CUDA(cudaGetLastError());
  return kApiOk;
}

// table [vocab, H] e4m3 bytes, scales fp32 [vocab * H / 128 rounded up], tokens int64 [n]; H % 16 == 0. out bf16 [n, H].
extern "C" int pkb_embed_fp8(const void* table, const void* scales, const void* tokens, void* out, int n, int vocab, int H, void* stream) {
  PKB_CHECK_ARG(n >= 0 && vocab > 0 && H > 0 && H % 16 == 0 && (long long)n * (H / 16) < (1ll << 31), "H must be a multiple of 16");
  PKB_CHECK_ARG((((uintptr_t)table | (uintptr_t)out) & 15) == 0, "table and result must be 16-byte aligned");
  if (n == 0) return kApiOk;
  long long blocks = ((long long)n * (H / 16) + 255) / 256;
  if (blocks > 148 * 8) blocks = 148 * 8;
  embed_fp8_kernel<<<(int)blocks, 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const uint8_t*>(table), static_cast<const float*>(scales), static_cast<const long long*>(tokens),
      static_cast<__nv_bfloat16*>(out), n, vocab, H, status_block_device_ptr());
  PKB_CHECK_CUDA(cudaGetLastError());
  return kApiOk;
}

extern "C" int pkb_embed_grad_max_tokens() { return kEmbedMaxTokens; }

// q (e4m3 bytes, zero-filled by the caller) and s (fp32 per 128 elements, filled with 1): the rows of the n tokens receive the
// quantised sum of their gradient rows dx bf16 [n, H]. H % 128 == 0, n <= pkb_embed_grad_max_tokens().
extern "C" int pkb_embed_grad_fp8(const void* dx, const void* tokens, int n, int vocab, int H, void* q, void* s, void* stream) {
  PKB_CHECK_ARG(n >= 0 && n <= kEmbedMaxTokens && vocab > 0 && H > 0 && H % 128 == 0, "H must be a multiple of 128, at most 16384 tokens");
  PKB_CHECK_ARG((((uintptr_t)dx & 15) | ((uintptr_t)q & 7)) == 0, "misaligned buffers");
  if (n == 0) return kApiOk;
  const int smem = (n + 31) / 32 * 4 + n * 2;          // at most 34 KiB
  embed_grad_fp8_kernel<<<n, kEmbedGradThreads, smem, static_cast<cudaStream_t>(stream)>>>(static_cast<const __nv_bfloat16*>(dx),
                                                                         static_cast<const long long*>(tokens), n, vocab, H,
                                                                         static_cast<uint8_t*>(q), static_cast<float*>(s),
                                                                         status_block_device_ptr());
  PKB_CHECK_CUDA(cudaGetLastError());
  return kApiOk;
}
