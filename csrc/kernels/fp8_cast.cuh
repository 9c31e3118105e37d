// Block-scaled fp8-e4m3 quantisation shared by the dispatch and cast kernels: per 128 elements
// scale = max(amax, 1e-10) / 448 and q = e4m3(x / scale), the quotient correctly rounded in fp32.
#pragma once
#include <cuda_fp8.h>
#include <stdint.h>

namespace uccl {
namespace fp8 {

__device__ __forceinline__ float block_scale(float amax) { return fmaxf(amax, 1e-10f) / 448.f; }

__device__ __forceinline__ uint32_t pack4(float a, float b, float c, float d) {
  const __nv_fp8x2_storage_t lo = __nv_cvt_float2_to_fp8x2(make_float2(a, b), __NV_SATFINITE, __NV_E4M3);
  const __nv_fp8x2_storage_t hi = __nv_cvt_float2_to_fp8x2(make_float2(c, d), __NV_SATFINITE, __NV_E4M3);
  return static_cast<uint32_t>(lo) | (static_cast<uint32_t>(hi) << 16);
}

// Four elements -> four e4m3 bytes, bit for bit those of the true quotient x / scale, without a
// division per element.  With inv = 1 / scale rounded, r = x * inv lies within 2^-22.9 (two
// roundings) of the exact quotient, whose own rounding adds 2^-24: the rounded quotient is inside
// [r (1 - 2^-21), r (1 + 2^-21)].  Rounding to e4m3 is monotonic, so where both ends give the same
// byte it is the quotient's byte as well.  The ends differ only next to a point halfway between two
// e4m3 values (about one element in 2^18 of ordinary data); those four elements take the division.
__device__ __forceinline__ uint32_t quantise4(float x0, float x1, float x2, float x3, float scale, float inv) {
  constexpr float kUp = 1.0f + 0x1p-21f, kDown = 1.0f - 0x1p-21f;
  const float r0 = x0 * inv, r1 = x1 * inv, r2 = x2 * inv, r3 = x3 * inv;
  const uint32_t up = pack4(r0 * kUp, r1 * kUp, r2 * kUp, r3 * kUp);
  const uint32_t down = pack4(r0 * kDown, r1 * kDown, r2 * kDown, r3 * kDown);
  if (up == down) return up;
  return pack4(__fdiv_rn(x0, scale), __fdiv_rn(x1, scale), __fdiv_rn(x2, scale), __fdiv_rn(x3, scale));
}

}  // namespace fp8
}  // namespace uccl
