// Test-only kernels: the block-scaled fp8 quantisation against the divisions that it stands for.
// Built into tests/native/libuccl_devtest.so and driven through ctypes by tests/test_gpu_single.py.
#include <cuda_runtime.h>

#include "kernels/fp8_cast.cuh"

namespace {

namespace fp8 = uccl::fp8;

__device__ bool same(float a, float b) { return __float_as_uint(a) == __float_as_uint(b) || (a != a && b != b); }

// Every scale's significand, times 2^exponent, at every place where the byte changes (the numbers half way between two
// neighbours of e4m3) and up to five units around it, both signs.  out[0]: bytes that differ, out[1]: bits of such a scale.
__global__ void divisor_kernel(int exponent, unsigned* out) {
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < 1u << 23; i += gridDim.x * blockDim.x) {
    const float b = ldexpf(__uint_as_float(0x3f800000u | i), exponent);
    const fp8::Divisor div(b);
    for (int k = 0; k < 16; ++k) {
      const float middle = k < 8 ? (17 + 2 * k) / 16.f : (2 * k - 15) * 0x1p-10f;
      for (int d = -5; d <= 5; ++d) {
        const float x = __uint_as_float(__float_as_uint(b * middle) + d);
        const unsigned got = div.quantise4(make_float2(-x, x), make_float2(x, -x));
        const float q = __fdiv_rn(x, b);
        if (got == fp8::pack4(q, -q, -q, q)) continue;
        atomicAdd(out, 1u);
        out[1] = __float_as_uint(b);
      }
    }
  }
}
// Every amax: all 2^31 bit patterns without a sign.
__global__ void scale_kernel(unsigned* out) {
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < 1u << 31; i += gridDim.x * blockDim.x) {
    const float amax = __uint_as_float(i);
    if (same(fp8::block_scale(amax), __fdiv_rn(fmaxf(amax, 1e-10f), 448.f))) continue;
    atomicAdd(out, 1u);
    out[1] = i;
  }
}

}  // namespace

// `out`: two words of device memory, set to zero by the caller
extern "C" int ucclDevTestFp8Divisor(int exponent, void* out, void* stream) {
  divisor_kernel<<<1184, 256, 0, static_cast<cudaStream_t>(stream)>>>(exponent, static_cast<unsigned*>(out));
  return cudaGetLastError() == cudaSuccess ? 0 : 1;
}
extern "C" int ucclDevTestFp8Scale(void* out, void* stream) {
  scale_kernel<<<1184, 256, 0, static_cast<cudaStream_t>(stream)>>>(static_cast<unsigned*>(out));
  return cudaGetLastError() == cudaSuccess ? 0 : 1;
}
