// One group of the block-scaled fp8 format: 32 values -> e4m3 and the exponent of their power-of-two scale, the smallest
// that brings the largest magnitude inside the e4m3 range (448).  Shared by the quantisation kernel and the GEMM epilogue
// that quantises its result, so that both give the same bytes.
#pragma once
#include <cuda_fp8.h>
#include <cuda_runtime.h>

#include <cstdint>

namespace msccl {
namespace sm100 {

__device__ __forceinline__ int quantize_mx_group(const float (&v)[32], uint32_t (&packed)[8]) {
  float amax = 0.0f;
#pragma unroll
  for (int i = 0; i < 32; ++i) amax = fmaxf(amax, fabsf(v[i]));
  amax = fmaxf(amax, 1.0e-36f);
  // smallest e with amax / 2^e <= 448
  const float ratio = amax / 448.0f;
  int e = ilogbf(ratio);
  if (ldexpf(1.0f, e) < ratio) ++e;
  e = max(-127, min(127, e));
  const float inv = ldexpf(1.0f, -e);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const __nv_fp8x2_storage_t lo = __nv_cvt_float2_to_fp8x2(make_float2(v[4 * i] * inv, v[4 * i + 1] * inv), __NV_SATFINITE, __NV_E4M3);
    const __nv_fp8x2_storage_t hi = __nv_cvt_float2_to_fp8x2(make_float2(v[4 * i + 2] * inv, v[4 * i + 3] * inv), __NV_SATFINITE, __NV_E4M3);
    packed[i] = static_cast<uint32_t>(lo) | (static_cast<uint32_t>(hi) << 16);
  }
  return e;
}

}  // namespace sm100
}  // namespace msccl
