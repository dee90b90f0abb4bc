// e4m3 conversion shared by the row kernels and the quantisation kernels.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace lmoe {

constexpr float kE4M3Max = 448.0f;

// Eight bf16 values -> eight e4m3 bytes: saturate(x * scale), round to nearest even.
__device__ __forceinline__ uint2 quantize8(const uint4& v, float scale) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
  uint32_t out[2];
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const float2 f0 = __bfloat1622float2(h[2 * k]), f1 = __bfloat1622float2(h[2 * k + 1]);
    const uint32_t lo = __nv_cvt_float2_to_fp8x2(make_float2(f0.x * scale, f0.y * scale), __NV_SATFINITE, __NV_E4M3);
    const uint32_t hi = __nv_cvt_float2_to_fp8x2(make_float2(f1.x * scale, f1.y * scale), __NV_SATFINITE, __NV_E4M3);
    out[k] = lo | (hi << 16);
  }
  return make_uint2(out[0], out[1]);
}

// max |x| over eight bf16 values, as the bit pattern of a non-negative bf16 pair's maximum
__device__ __forceinline__ float absmax8(const uint4& v, float m) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
  __nv_bfloat162 a = __hmax2(__habs2(h[0]), __habs2(h[1])), b = __hmax2(__habs2(h[2]), __habs2(h[3]));
  const float2 f = __bfloat1622float2(__hmax2(a, b));
  return fmaxf(m, fmaxf(f.x, f.y));
}

}  // namespace lmoe
