// One 128-element block of the 1 x 128 e4m3 format: scale, codes and back.
#pragma once
#include <cuda_fp8.h>

#include "pkb/ptx.cuh"

namespace pkb {

constexpr float kInv448 = 1.0f / 448.0f;

// Scale of a block whose largest magnitude is amax.
__device__ __forceinline__ float fp8_block_scale(float amax, int pow2_scales) {
  float s = amax * kInv448;   // amax / 448 the way PyTorch evaluates a tensor divided by a Python scalar on the GPU: times the rounded reciprocal
  if (pow2_scales && s > 0.f) s = exp2f(ceilf(log2f(s)));  // power-of-two scale (exact to undo)
  return s == 0.f ? 1.0f : s;
}

// Codes of 8 elements of a block with scale s: the correctly rounded quotient x / s, not x * (1 / s): the quotient decides the
// e4m3 code at rounding boundaries, and x / s is what the PyTorch formulation computes. One reciprocal per block, then per
// element a product, its residual and one correction (three FMA-pipe instructions instead of a division each).
__device__ __forceinline__ void fp8_encode8(const float* v, float s, uint32_t* codes) {
  const float inv = __frcp_rn(s);
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const __nv_fp8x2_storage_t lo = __nv_cvt_float2_to_fp8x2(make_float2(div_rn_by(v[4 * j], s, inv), div_rn_by(v[4 * j + 1], s, inv)), __NV_SATFINITE, __NV_E4M3);
    const __nv_fp8x2_storage_t hi = __nv_cvt_float2_to_fp8x2(make_float2(div_rn_by(v[4 * j + 2], s, inv), div_rn_by(v[4 * j + 3], s, inv)), __NV_SATFINITE, __NV_E4M3);
    codes[j] = (uint32_t)lo | ((uint32_t)hi << 16);
  }
}

__device__ __forceinline__ void fp8_decode8(const uint32_t* codes, float s, float* v) {
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    __half2_raw h0 = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)(codes[j] & 0xffffu), __NV_E4M3);
    __half2_raw h1 = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)(codes[j] >> 16), __NV_E4M3);
    const float2 f0 = __half22float2(*reinterpret_cast<__half2*>(&h0));
    const float2 f1 = __half22float2(*reinterpret_cast<__half2*>(&h1));
    v[4 * j] = f0.x * s; v[4 * j + 1] = f0.y * s; v[4 * j + 2] = f1.x * s; v[4 * j + 3] = f1.y * s;
  }
}

}  // namespace pkb
