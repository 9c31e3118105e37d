// The collectives of a one-rank communicator: a copy from memory to memory.
#include <algorithm>

#include "collectives.cuh"
#include "gemm_sm100.h"
#include "launch.cuh"
#include "ptx.cuh"

namespace uccl {
namespace dev {

constexpr int kCopyThreads = 256;

// U pieces of W bytes per thread, one CTA width apart, all loads out before the first store.  Bound by memory when large
// and by the launch when small, where cudaMemcpyAsync costs the host 3.0 us and this 2.4.  A reduce-scatter and an
// all-gather in a row: 4096 bf16 elements 6.5 -> 5.1 us, 8 Mi 17.2 -> 12.9 us (5.2 TB/s), 64 Mi fp32 172 -> 159 us (6.75 TB/s).
template <int U, int W>
__global__ void __launch_bounds__(kCopyThreads) local_copy_kernel(const char* src, char* dst, size_t bytes) {
  ptx::launch_dependents();
  ptx::wait_dependencies();
  const size_t pieces = bytes / W, p0 = static_cast<size_t>(blockIdx.x) * (kCopyThreads * U) + threadIdx.x;
  uint32_t v[U][W / 4];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const size_t p = p0 + u * kCopyThreads;
    if (p >= pieces) continue;
    if constexpr (W == 32) {
      ptx::ld_stream_v8(src + p * W, v[u]);
    } else {
      const uint4 x = ptx::ld_stream_v4(src + p * W);
      v[u][0] = x.x, v[u][1] = x.y, v[u][2] = x.z, v[u][3] = x.w;
    }
  }
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const size_t p = p0 + u * kCopyThreads;
    if (p >= pieces) continue;
    if constexpr (W == 32) ptx::st_global_v8(dst + p * W, v[u]);
    else ptx::st_global_v4(dst + p * W, make_uint4(v[u][0], v[u][1], v[u][2], v[u][3]));
  }
  // what is left over is less than a piece
  const size_t rest = pieces * W + threadIdx.x;
  if (blockIdx.x == gridDim.x - 1 && rest < bytes) dst[rest] = src[rest];
}

}  // namespace dev

template <int W>
static cudaError_t launchCopy(const void* src, void* dst, size_t bytes, cudaStream_t s) {
  constexpr size_t T = dev::kCopyThreads;
  const size_t pieces = bytes / W;
  // Four pieces per thread once that still gives every SM the CTAs that it holds of this kernel (44 registers with 32-byte
  // pieces, 28 with 16).  One piece and four, in us: 24 MiB 9.0 and 8.9, 28 MiB 10.1 and 10.0, 32 MiB 11.4 and 11.3.
  constexpr int kResident = W == 32 ? 5 : 8;
  const bool four = pieces >= static_cast<size_t>(deviceSmCount()) * kResident * T * 4;
  const size_t share = four ? 4 * T : T, ctas = std::max<size_t>(1, (pieces + share - 1) / share);
  if (ctas > 0x7fffffffu) return cudaErrorInvalidValue;
  const char* from = static_cast<const char*>(src);
  char* to = static_cast<char*>(dst);
  if (four) return launchOverlapped(dev::local_copy_kernel<4, W>, static_cast<unsigned>(ctas), T, 0, s, from, to, bytes);
  return launchOverlapped(dev::local_copy_kernel<1, W>, static_cast<unsigned>(ctas), T, 0, s, from, to, bytes);
}

cudaError_t launchLocalCopy(const void* src, void* dst, size_t bytes, cudaStream_t s) {
  const uintptr_t both = reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst);
  if ((both & 15) != 0 || bytes == 0) return cudaErrorInvalidValue;
  return (both & 31) == 0 ? launchCopy<32>(src, dst, bytes, s) : launchCopy<16>(src, dst, bytes, s);
}

}  // namespace uccl
