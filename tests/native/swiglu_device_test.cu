// Test-only kernel: the silu of the GEMM epilogues against the division that it stands for, over all fp32 gates.
// Built into tests/native/libuccl_devtest.so and driven through ctypes by tests/test_gemm.py.
#include <cuda_runtime.h>

#include "kernels/swiglu.cuh"

namespace {

__device__ float divided(float x) { return x == 0.f ? x : x / (1.0f + __expf(-x)); }
__device__ bool same(float a, float b) { return __float_as_uint(a) == __float_as_uint(b) || (a != a && b != b); }

// Gate bits [first, first + count); the two places of a pair hold different gates.  out[0]: how many differ, out[1]: bits of one of them.
__global__ void compare_kernel(unsigned first, unsigned count, unsigned* out) {
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) {
    const unsigned bits = first + i, other = bits * 2654435761u + 1u;
    const float x = __uint_as_float(bits), y = __uint_as_float(other);
    const float2 a = uccl::gemm::silu2_negated(make_float2(x, y)), b = uccl::gemm::silu2_negated(make_float2(y, x));
    if (same(-a.x, divided(x)) && same(-b.y, divided(x)) && same(-a.y, divided(y))) continue;
    atomicAdd(out, 1u);
    out[1] = bits;
  }
}

}  // namespace

// `out`: two words of device memory, set to zero by the caller
extern "C" int ucclDevTestSilu(unsigned first, unsigned count, void* out, void* stream) {
  compare_kernel<<<1184, 256, 0, static_cast<cudaStream_t>(stream)>>>(first, count, static_cast<unsigned*>(out));
  return cudaGetLastError() == cudaSuccess ? 0 : 1;
}
