// MoE expert-parallel dispatch and combine as single kernels over NVLink peer memory.
//
// dispatch : a CTA takes one token after the other, sixteen elements per thread.  Quantise: every thread
//            has loaded its 32 bytes of the bf16 row while the CTA dealt with the token before, eight
//            lanes agree on the fp32 scale of their 128 elements (amax / 448), convert to fp8 e4m3 and
//            write one 16-byte piece into one of three row buffers in shared memory.  Scatter: lane k of
//            warp 0 has taken a row slot for the token's k-th expert in the region this rank owns on
//            the expert's rank (one local atomic per token and destination, also a token ahead) and issues
//            bulk copies shared memory -> that rank's receive area for the row and the scales, plus a
//            16-byte descriptor {token, local expert, k, 1}: the SM's copy engine moves the rows
//            while the CTA converts the next tokens.  The last CTA publishes the per-destination row
//            counts and raises an arrival flag on every rank, then waits for everybody else's flag, so
//            the receive area is complete when the kernel ends.
// combine  : a warp takes 256 columns of one token, pulls them from the bf16 expert outputs of its top-k
//            rows on the ranks that computed them (all loads in flight), multiplies by the
//            routing weights, accumulates in fp32 and writes the bf16 result.
// Neither exists in the reference (it has no all-to-all at all, desgin/design-spec.md:1760).
#include <algorithm>

#include "coll_device.cuh"
#include "fp8_cast.cuh"
#include "gemm_sm100.h"
#include "launch.cuh"
#include "moe.h"

namespace uccl {
namespace dev {

constexpr int kMoeMaxTopk = 16;
constexpr int kMoeBufs = 3;

// shared memory of one row buffer: the quantised row, then its scales
__host__ __device__ constexpr int moe_row_smem(int hidden) { return hidden + ((hidden / 128 * 4 + 15) & ~15); }

// Bound by memory (a token is 2 H bytes in and topk (H + H / 32) out), then by latencies when tokens are few.
// A token per CTA instead of one per warp: 4096 tokens x 7168 on 3552 warps were two uneven rounds of long
// serial chains, 91 us, and 96 tokens kept 12 SMs busy for 27 us; now 55 us (5.4 TB/s) and 7 us.
__global__ void __launch_bounds__(512, 2) moe_dispatch_kernel(const __grid_constant__ MoeArgs a) {
  extern __shared__ __align__(16) uint8_t moe_smem[];
  __shared__ int s_row[kMoeBufs][kMoeMaxTopk];  // destination << 24 | slot of a buffer's row, -1: none
  const DevComm& dc = a.dc;
  const int lane = threadIdx.x & 31;
  const int n = dc.nranks, me = dc.rank;
  const int H = a.hidden, nblk = H / 128;
  const int e0 = threadIdx.x * 16;
  const uint32_t scaleBytes = static_cast<uint32_t>(nblk) * 4;
  const bool scalesBulk = (scaleBytes & 15u) == 0;  // a bulk copy moves multiples of 16 bytes
  const bool wide = (reinterpret_cast<uintptr_t>(a.x) & 31) == 0;
  const bool router = threadIdx.x < static_cast<unsigned>(a.topk);  // lanes of warp 0

  uint32_t raw[8];
  auto load = [&](int t) {
#pragma unroll
    for (int j = 0; j < 8; ++j) raw[j] = 0;
    if (t >= a.tokens || e0 >= H) return;
    const char* p = static_cast<const char*>(a.x) + (static_cast<size_t>(t) * H + e0) * 2;
    if (wide) {
      ptx::ld_stream_v8(p, raw);
    } else {
      const uint4 lo = ptx::ld_stream_v4(p), hi = ptx::ld_stream_v4(p + 16);
      raw[0] = lo.x, raw[1] = lo.y, raw[2] = lo.z, raw[3] = lo.w, raw[4] = hi.x, raw[5] = hi.y, raw[6] = hi.z, raw[7] = hi.w;
    }
  };
  // Routing runs ahead, so that no token waits for its latencies: the experts of (t, k) are read two tokens
  // early, the atomics that take row slots are issued one token early (lanes with the same destination
  // share one), and what they returned is looked at when the token's turn comes.
  int next = -1;                    // lane k: expert of the token whose slots are not asked for yet
  int expert = -1, dst = -1, base = 0;
  unsigned same = 0;
  auto read_experts = [&](int t) { next = router && t < a.tokens ? a.topkIdx[static_cast<size_t>(t) * a.topk + lane] : -1; };
  auto take_slots = [&]() {
    expert = next;
    dst = expert >= 0 && expert < a.numExperts ? expert / a.expertsPerRank : -1;
    same = __match_any_sync(0xffffffffu, dst);
    if (dst >= 0 && lane == __ffs(same) - 1) base = static_cast<int>(atomicAdd(a.sendCount + dst, static_cast<uint32_t>(__popc(same))));
  };
  auto place_of = [&]() {  // destination << 24 | slot, or -1
    const int slot = __shfl_sync(0xffffffffu, base, __ffs(same) - 1) + __popc(same & ((1u << lane) - 1));
    if (dst < 0) return -1;
    if (slot < a.rowsPerSource) return (dst << 24) | slot;
    atomicAdd(a.overflow, 1u);
    return -1;
  };

  if (n == 1) ptx::launch_dependents();
  ptx::wait_dependencies();
  int buf = 0;
  load(blockIdx.x);
  if (threadIdx.x < 32) {
    read_experts(blockIdx.x);
    take_slots();
    read_experts(blockIdx.x + gridDim.x);
  }
  for (int t = blockIdx.x; t < a.tokens; t += gridDim.x) {
    uint8_t* rowBuf = moe_smem + buf * moe_row_smem(H);
    float* scaleBuf = reinterpret_cast<float*>(rowBuf + H);
    // ---- quantise (lanes beyond the row take part in the shuffles with zeros)
    __nv_bfloat162 m = __habs2(reinterpret_cast<const __nv_bfloat162&>(raw[0]));
#pragma unroll
    for (int j = 1; j < 8; ++j) m = __hmax2(m, __habs2(reinterpret_cast<const __nv_bfloat162&>(raw[j])));
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) {  // a 128-element block is eight lanes
      const uint32_t other = __shfl_xor_sync(0xffffffffu, reinterpret_cast<const uint32_t&>(m), o);
      m = __hmax2(m, reinterpret_cast<const __nv_bfloat162&>(other));
    }
    const float2 mf = __bfloat1622float2(m);
    const float scale = fp8::block_scale(fmaxf(mf.x, mf.y));
    const fp8::Divisor div(scale);
    uint32_t q[4];
#pragma unroll
    for (int j = 0; j < 4; ++j)  // the divisor takes its elements negated
      q[j] = div.quantise4(ptx::unpack_bf16x2(raw[2 * j] ^ 0x80008000u), ptx::unpack_bf16x2(raw[2 * j + 1] ^ 0x80008000u));
    load(t + gridDim.x);
    if (e0 < H) {
      *reinterpret_cast<uint4*>(rowBuf + e0) = make_uint4(q[0], q[1], q[2], q[3]);
      if ((lane & 7) == 0) scaleBuf[e0 >> 7] = scale;
    }
    int place = -1;
    if (threadIdx.x < 32) {
      place = place_of();
      if (router) s_row[buf][lane] = place;
    }
    // shared-memory writes of every thread become visible to the bulk-copy engine
    ptx::fence_proxy_async_smem();
    __syncthreads();
    // ---- scatter
    if (threadIdx.x < 32) {
      if (router) {
        a.slotOf[static_cast<size_t>(t) * a.topk + lane] = place;
        if (place >= 0) {
          const int dst = place >> 24;
          const size_t r = static_cast<size_t>(me) * a.rowsPerSource + (place & 0xffffff);
          ptx::bulk_store(a.recvX[dst] + r * H, rowBuf, static_cast<uint32_t>(H));
          if (scalesBulk) ptx::bulk_store(a.recvScale[dst] + r * nblk, scaleBuf, scaleBytes);
          *reinterpret_cast<int4*>(a.recvMeta[dst] + r * 4) = make_int4(t, expert - dst * a.expertsPerRank, lane, 1);
        }
        ptx::tma_store_commit();
      }
      take_slots();
      read_experts(t + 2 * gridDim.x);
      // The row of the token before has left its buffer.  Buffer b is written again two barriers after the
      // one that published it, and this warp comes here between them, so nobody writes it too early.
      if (router) ptx::tma_store_wait_read<1>();
    }
    if (!scalesBulk) {
      for (int i = threadIdx.x; i < a.topk * nblk; i += blockDim.x) {
        const int k = i / nblk, b = i - k * nblk, w = s_row[buf][k];
        if (w >= 0) a.recvScale[w >> 24][(static_cast<size_t>(me) * a.rowsPerSource + (w & 0xffffff)) * nblk + b] = scaleBuf[b];
      }
    }
    buf = buf + 1 == kMoeBufs ? 0 : buf + 1;
  }
  // Every bulk copy of this thread has completed (written, not just read) before the CTA reports in, and before a
  // launch that has come up early may read the rows.
  if (router) ptx::tma_store_wait<0>();

  // ---- completion: the last CTA publishes counts and flags, then waits for every source
  __shared__ int s_last;
  __syncthreads();
  if (threadIdx.x == 0) {
    if (n > 1) ptx::fence_sys();
    else __threadfence();  // the slot counter of this CTA's tokens, for the CTA that reads it below
    const uint32_t prev = atomicAdd(a.ctasDone, 1u);
    s_last = prev == gridDim.x - 1;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  if (n == 1) {  // nobody to tell and nobody to wait for
    if (threadIdx.x == 0) {
      const uint32_t rows = *reinterpret_cast<volatile uint32_t*>(a.sendCount);
      a.recvCounts[0][0] = static_cast<int32_t>(min(rows, static_cast<uint32_t>(a.rowsPerSource)));
      *a.sendCount = 0;  // ready for the next call
      *a.ctasDone = 0;
    }
    return;
  }
  const uint32_t e = *a.epoch + 1;
  if (threadIdx.x < static_cast<unsigned>(n)) {
    const int p = threadIdx.x;
    const uint32_t cnt = min(*reinterpret_cast<volatile uint32_t*>(a.sendCount + p), static_cast<uint32_t>(a.rowsPerSource));
    a.recvCounts[p][me] = static_cast<int32_t>(cnt);
    ptx::fence_sys();
    ptx::st_release_sys_u32(a.arrived[p] + me, e);
  }
  __syncthreads();
  if (threadIdx.x < static_cast<unsigned>(n)) {
    a.sendCount[threadIdx.x] = 0;  // ready for the next call
    wait_u32(a.arrived[me] + threadIdx.x, e, dc, DEV_TIMEOUT_MOE, threadIdx.x, e);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    *a.ctasDone = 0;
    *a.epoch = e;
  }
}

// TK = upper bound of top-k the instantiation handles.  Bound by memory: a warp has TK x 512 bytes in flight
// and is done after one pass, so the number of resident warps is what counts.  4096 x 7168 with top-8: 80.5
// us (6.6 TB/s, what a copy reaches) with five CTAs of eight warps per SM, 91 us with four or three, and
// 88 to 110 us with 32-byte loads, whose registers leave three or two; a warp per token, which walks its
// row in serial steps, took 88 us, and 20 us for 96 tokens, which then sit on 12 SMs.
constexpr int kCombineThreads = 256;
template <int TK>
__global__ void __launch_bounds__(kCombineThreads, TK > 8 ? 3 : TK > 4 ? 5 : 6) moe_combine_kernel(const __grid_constant__ MoeArgs a, int chunks) {
  const int lane = threadIdx.x & 31;
  const long item = static_cast<long>(blockIdx.x) * (kCombineThreads / 32) + (threadIdx.x >> 5);
  const int t = static_cast<int>(item / chunks), c = static_cast<int>(item - static_cast<long>(t) * chunks);
  if (t >= a.tokens) return;
  const int H = a.hidden, el = c * 256 + lane * 8;
  if (a.dc.nranks == 1) ptx::launch_dependents();
  ptx::wait_dependencies();
  int slot = -1;
  float weight = 0.f;
  if (lane < a.topk) {
    slot = a.slotOf[static_cast<size_t>(t) * a.topk + lane];
    weight = a.topkWeight[static_cast<size_t>(t) * a.topk + lane];
  }
  uint4 v[TK];
#pragma unroll
  for (int k = 0; k < TK; ++k) {
    const int s = __shfl_sync(0xffffffffu, slot, k);
    if (s >= 0 && el < H)
      v[k] = ptx::ld_stream_v4(a.expertOut[s >> 24] + ((static_cast<size_t>(a.dc.rank) * a.rowsPerSource + (s & 0xffffff)) * H + el) * 2);
  }
  float acc[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) acc[j] = 0.f;
#pragma unroll
  for (int k = 0; k < TK; ++k) {
    const int s = __shfl_sync(0xffffffffu, slot, k);
    const float w = __shfl_sync(0xffffffffu, weight, k);
    if (s >= 0) {
      const uint32_t x[4] = {v[k].x, v[k].y, v[k].z, v[k].w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 p = ptx::unpack_bf16x2(x[j]);
        acc[2 * j] += w * p.x;
        acc[2 * j + 1] += w * p.y;
      }
    }
  }
  if (el >= H) return;
  ptx::st_global_v4(static_cast<char*>(a.out) + (static_cast<size_t>(t) * H + el) * 2, Vec<DT_BF16>::pack(acc));
}

}  // namespace dev

cudaError_t launchMoeDispatch(const MoeArgs& a, cudaStream_t stream) {
  if (a.hidden % 128 != 0 || a.hidden > 8192 || a.topk < 1 || a.topk > dev::kMoeMaxTopk) return cudaErrorInvalidValue;
  const int smem = dev::kMoeBufs * dev::moe_row_smem(a.hidden);  // 25 KiB at most
  const int threads = (a.hidden / 16 + 31) / 32 * 32;
  // as many CTAs as fit at once: 64 registers a thread
  const int perSm = 1024 / threads;
  const int ctas = std::max(1, std::min(a.tokens, deviceSmCount() * perSm));
  // ranks that wait for one another keep to the plain launch
  if (a.dc.nranks == 1) return launchOverlapped(dev::moe_dispatch_kernel, ctas, threads, smem, stream, a);
  dev::moe_dispatch_kernel<<<ctas, threads, smem, stream>>>(a);
  return cudaGetLastError();
}
cudaError_t launchMoeCombine(const MoeArgs& a, cudaStream_t stream) {
  if (a.hidden % 128 != 0 || a.hidden > 8192 || a.topk < 1 || a.topk > dev::kMoeMaxTopk) return cudaErrorInvalidValue;
  if (a.tokens == 0) return cudaSuccess;
  const int chunks = (a.hidden + 255) / 256;
  constexpr int warps = dev::kCombineThreads / 32;
  const unsigned ctas = static_cast<unsigned>((static_cast<long>(a.tokens) * chunks + warps - 1) / warps);
  auto launch = [&](void (*kern)(MoeArgs, int)) {
    if (a.dc.nranks == 1) return launchOverlapped(kern, ctas, dev::kCombineThreads, 0, stream, a, chunks);
    kern<<<ctas, dev::kCombineThreads, 0, stream>>>(a, chunks);
    return cudaGetLastError();
  };
  if (a.topk <= 2) return launch(dev::moe_combine_kernel<2>);
  if (a.topk <= 4) return launch(dev::moe_combine_kernel<4>);
  return a.topk <= 8 ? launch(dev::moe_combine_kernel<8>) : launch(dev::moe_combine_kernel<16>);
}

}  // namespace uccl
