// silu(gate) * up for the GEMM epilogues, two elements per instruction and no branch.
#pragma once
#include "ptx.cuh"

namespace uccl {
namespace gemm {

__device__ __forceinline__ float ex2_ftz(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float rcp_ftz(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// -x / (1 + exp(-x)), the quotient rounded to nearest as a division rounds it.  Markstein's method ("Computation of
// elementary functions on the IBM RISC System/6000 processor", 1990): one Newton step makes the reciprocal y of d right to
// the last place but for rare mantissas, and q + (x - d q) y is then the rounded quotient.  Both d and x are taken a
// quarter, so that 1 / d stays a normal number up to where exp(-x) is infinite.  There, for infinite x, for zeros (whose
// sign the residual would lose) and for gates so small that their quarter is rounded, x times a quarter of y is the answer as
// it stands: exp(-x) is 1 for small gates, and the halves of subnormal numbers round once.  What takes the first way is at least
// 2^-122: the smallest quotient of a large negative gate, -88.7 / exp(88.7), is 2^-121.5.
// The results are those of x / (1.f + __expf(-x)) for every x, all 2^32 of them compared.
//
// A division as such has a slow path, and the branch to it ties each element to the one before: 49 cycles per column of a
// warp.  Without a branch the elements of a register block overlap: SwiGLU 4096 x 28672 x 512 220 -> 101 us, 16384 x 4096
// x 128 119 -> 47 us, 1212 x 10192 x 1760 40.3 -> 34.4 us, 64 x 28672 x 4096 (one tile per CTA, whose epilogue nothing
// hides) 45.1 -> 40.3 us.  What the blocks are and what registers they cost stands with swiglu_and_store.
// Signs: the negated reciprocal and quotient are carried, because the packed instructions cannot negate an operand.
__device__ __forceinline__ float2 silu2_negated(float2 x) {
  const float2 p = ptx::mul2(x, make_float2(-1.4426950408889634f, -1.4426950408889634f));
  const float2 t = make_float2(ex2_ftz(p.x), ex2_ftz(p.y));
  const float2 d = ptx::fma2(t, make_float2(0.25f, 0.25f), make_float2(0.25f, 0.25f));
  const float2 nd = ptx::fma2(t, make_float2(-0.25f, -0.25f), make_float2(-0.25f, -0.25f));
  const float2 xq = ptx::mul2(x, make_float2(0.25f, 0.25f));
  float2 ny = make_float2(rcp_ftz(nd.x), rcp_ftz(nd.y));
  const float2 plain = ptx::mul2(x, ptx::mul2(ny, make_float2(0.25f, 0.25f)));
  ny = ptx::fma2(ptx::fma2(d, ny, make_float2(1.f, 1.f)), ny, ny);
  float2 nq = ptx::mul2(xq, ny);
  nq = ptx::fma2(ptx::fma2(d, nq, xq), ny, nq);
  nq.x = fabsf(nq.x) >= 0x1p-122f ? nq.x : plain.x;
  nq.y = fabsf(nq.y) >= 0x1p-122f ? nq.y : plain.y;
  return nq;
}

// bf16 pair of silu(gate) * up
__device__ __forceinline__ uint32_t swiglu2(float2 gate, float2 up) {
  const float2 v = ptx::mul2(silu2_negated(gate), up);
  return ptx::pack_bf16x2(v.x, v.y) ^ 0x80008000u;
}
__device__ __forceinline__ uint32_t swiglu2(const uint32_t* gate, const uint32_t* up) {
  return swiglu2(make_float2(__uint_as_float(gate[0]), __uint_as_float(gate[1])), make_float2(__uint_as_float(up[0]), __uint_as_float(up[1])));
}
__device__ __forceinline__ uint4 swiglu8(const uint32_t* gate, const uint32_t* up) {
  return make_uint4(swiglu2(gate, up), swiglu2(gate + 2, up + 2), swiglu2(gate + 4, up + 4), swiglu2(gate + 6, up + 6));
}

}  // namespace gemm
}  // namespace uccl
