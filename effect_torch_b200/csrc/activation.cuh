// What the epilogues of several kernels share: the SiLU in the reference's form and the f16 activation hand-off's rounding.
#pragma once

#include <cuda_fp16.h>

#include <cstdint>

namespace etc {

// x * sigmoid(x) with sigmoid(x) = tanh(x / 2) / 2 + 1 / 2 (packages/core/src/Tensor.ts:1240-1245, 1537-1540).
__device__ __forceinline__ float silu_tanh(float x) { return x * (tanhf(x * 0.5f) * 0.5f + 0.5f); }

// Saturates at the f16 range.
__device__ __forceinline__ float sat16(float v) { return fminf(fmaxf(v, -65504.f), 65504.f); }
__device__ __forceinline__ __half half_sat(float v) { return __float2half_rn(sat16(v)); }
__device__ __forceinline__ __half2 half2_sat(float lo, float hi) { return __floats2half2_rn(sat16(lo), sat16(hi)); }
__device__ __forceinline__ uint2 pack4(const float4& v) {
  const __half2 lo = half2_sat(v.x, v.y), hi = half2_sat(v.z, v.w);
  return make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
}

}  // namespace etc
