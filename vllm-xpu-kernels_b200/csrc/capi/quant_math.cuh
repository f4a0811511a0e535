// Scale formulas of the activation quantisations, shared by the stand-alone operators and the
// kernels they are fused into: the same bits come out wherever a row is quantised.  Plain IEEE
// fp32 (no fast-math), so a straightforward fp32 evaluation of the formula agrees.
#pragma once

#include "common.cuh"

namespace b200moe {

__device__ __forceinline__ float round_up_pow2(float s) {
  return exp2f(ceilf(log2f(fmaxf(fabsf(s), 1e-10f))));
}

// Per-token-group FP8 scale of a group with maximum `amax`.
__device__ __forceinline__ float fp8_group_scale(float amax, float eps, float fp8_max, bool ue8m0) {
  const float s = fmaxf(fmaxf(amax, eps) / fp8_max, 1.0f / (fp8_max * 512.0f));
  return ue8m0 ? round_up_pow2(s) : s;
}

// MXFP8: biased exponent of the smallest power of two >= max(amax, 1e-10) / 448 (not below
// 1 / (448 * 512)), found on the bits of the float.
__device__ __forceinline__ uint32_t mxfp8_scale_exponent(float amax) {
  const float s = fmaxf(fmaxf(amax, 1e-10f) * (1.0f / 448.0f), 1.0f / (448.0f * 512.0f));
  const uint32_t bits = __float_as_uint(s);
  return (bits >> 23) + ((bits & 0x7FFFFFu) ? 1u : 0u);
}

// Eight values times `inv`, clamped to +-448, as e4m3.
__device__ __forceinline__ uint2 quantise8_e4m3(const float (&x)[8], float inv) {
  uint32_t w[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    float v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = fmaxf(-448.0f, fminf(x[4 * h + i] * inv, 448.0f));
    const uint32_t lo = __nv_cvt_float2_to_fp8x2(make_float2(v[0], v[1]), __NV_SATFINITE, __NV_E4M3);
    const uint32_t hi = __nv_cvt_float2_to_fp8x2(make_float2(v[2], v[3]), __NV_SATFINITE, __NV_E4M3);
    w[h] = lo | (hi << 16);
  }
  return make_uint2(w[0], w[1]);
}

template <int LANES>
__device__ __forceinline__ float seg_max(float v) {
#pragma unroll
  for (int off = 1; off < LANES; off <<= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, off));
  return v;
}

}  // namespace b200moe
