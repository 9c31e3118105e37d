// Block-scaled fp8-e4m3 quantisation shared by the kernels of moe.cu and fused_cast.cu (moe_noalloc.cu divides
// for itself, same bytes): per 128 elements
// scale = max(amax, 1e-10) / 448 and q = e4m3(x / scale), the quotient correctly rounded in fp32.
#pragma once
#include <cuda_fp8.h>
#include <stdint.h>

#include "ptx.cuh"

namespace uccl {
namespace fp8 {

__device__ __forceinline__ float block_scale(float amax) { return fmaxf(amax, 1e-10f) / 448.f; }

__device__ __forceinline__ uint32_t pack4(float a, float b, float c, float d) {
  const __nv_fp8x2_storage_t lo = __nv_cvt_float2_to_fp8x2(make_float2(a, b), __NV_SATFINITE, __NV_E4M3);
  const __nv_fp8x2_storage_t hi = __nv_cvt_float2_to_fp8x2(make_float2(c, d), __NV_SATFINITE, __NV_E4M3);
  return static_cast<uint32_t>(lo) | (static_cast<uint32_t>(hi) << 16);
}

using ptx::fma2;
using ptx::mul2;

// Correctly rounded quotients by one divisor, for the many elements that share a scale.  Markstein's
// theorem ("Computation of elementary functions on the IBM RISC System/6000 processor", 1990): with y =
// RN(1 / b) and q within one unit in the last place of a / b, RN(q + RN(a - b q) y) is RN(a / b).
// RN(a y) may be one and a half units off, so a first step makes q faithful and a second one exact.
// It takes and carries -a and -y, which keeps the sign of a zero.  No residual that decides a byte
// can underflow (b >= 1e-10 / 448, and quotients below 2^-10 are zero in e4m3).  An infinite b (an
// infinity in the block) becomes 0 with y = 0: finite elements give zero, infinite ones NaN, as a / b does.
struct Divisor {
  float2 b, ny;
  __device__ __forceinline__ explicit Divisor(float scale) {
    const float d = isinf(scale) ? 0.f : scale, n = -__frcp_rn(scale);
    b = make_float2(d, d);
    ny = make_float2(n, n);
  }
  __device__ __forceinline__ float2 quotient_of_negated(float2 na) const {
    float2 q = mul2(na, ny);
    q = fma2(fma2(q, b, na), ny, q);
    return fma2(fma2(q, b, na), ny, q);
  }
  // e4m3 bytes of four quotients, the elements given with their signs changed
  __device__ __forceinline__ uint32_t quantise4(float2 na, float2 nb) const {
    const float2 p = quotient_of_negated(na), q = quotient_of_negated(nb);
    return pack4(p.x, p.y, q.x, q.y);
  }
};

}  // namespace fp8
}  // namespace uccl
