// Block-scaled fp8-e4m3 quantisation shared by the kernels of moe.cu and fused_cast.cu (moe_noalloc.cu divides
// for itself, same bytes): per 128 elements
// scale = max(amax, 1e-10) / 448 and q = e4m3(x / scale), the bytes of the quotient correctly rounded in fp32.
#pragma once
#include <cuda_fp8.h>
#include <stdint.h>

#include "ptx.cuh"

namespace uccl {
namespace fp8 {

// max(amax, 1e-10) / 448 with the bits of the division, without its slow path: one correction by the residual (Markstein, below)
// of the product with the rounded 1 / 448; all finite amax compared.
__device__ __forceinline__ float block_scale(float amax) {
  constexpr float k448th = 1.f / 448.f;
  const float x = fmaxf(amax, 1e-10f), q = x * k448th;
  return isinf(x) ? x : fmaf(fmaf(q, -448.f, x), k448th, q);
}

__device__ __forceinline__ uint32_t pack4(float a, float b, float c, float d) {
  const __nv_fp8x2_storage_t lo = __nv_cvt_float2_to_fp8x2(make_float2(a, b), __NV_SATFINITE, __NV_E4M3);
  const __nv_fp8x2_storage_t hi = __nv_cvt_float2_to_fp8x2(make_float2(c, d), __NV_SATFINITE, __NV_E4M3);
  return static_cast<uint32_t>(lo) | (static_cast<uint32_t>(hi) << 16);
}

using ptx::fma2;
using ptx::mul2;

// Quotients by one divisor, for the many elements that share a scale.  Markstein's theorem ("Computation of elementary
// functions on the IBM RISC System/6000 processor", 1990): with y = RN(1 / b) and q within one unit in the last place of
// a / b, RN(q + RN(a - b q) y) is RN(a / b).  RN(a y) may be one and a half units off, so the one step taken here can miss
// RN(a / b) by a unit; but it never does where a / b lies within five units of a number between two neighbours of e4m3, nor
// falls on the other side of it, so the byte is that of the division.  All divisors (2^23 significands) are compared at all such
// places; scaling by powers of two changes nothing.  The reciprocal is an approximation and one Newton step, part of what is compared.
// Before, with two steps, and a reciprocal and a division with their slow paths, a cast was bound by its instructions: 64 Mi
// bf16 32.2 us at 1965 MHz and 37.0 at the 1540 MHz that the power cap leaves, now 30.9 and 32.7 (6.2 TB/s).
// It takes and carries -a and -y, which keeps the sign of a zero.  No residual that decides a byte
// can underflow (b >= 1e-10 / 448, and quotients below 2^-10 are zero in e4m3).  An infinite b (an
// infinity in the block) becomes 0 with y = 0: finite elements give zero, infinite ones NaN, as a / b does.
struct Divisor {
  float2 b, ny;
  __device__ __forceinline__ explicit Divisor(float scale) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(scale));
    y = fmaf(fmaf(-scale, y, 1.f), y, y);
    const bool inf = isinf(scale);
    const float d = inf ? 0.f : scale, n = inf ? -0.f : -y;
    b = make_float2(d, d);
    ny = make_float2(n, n);
  }
  __device__ __forceinline__ float2 quotient_of_negated(float2 na) const {
    const float2 q = mul2(na, ny);
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
