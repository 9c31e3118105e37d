// Reduce-scatter with a fused epilogue: out[i] = cast(scale * sum over ranks of in_r[my chunk][i]).
//
// The sum is carried in fp32 registers from the peer loads to the store, so "sum, scale, change
// the element type" costs no extra pass over memory: bf16 / fp16 / fp32 in, bf16 / fp16 / fp32 or
// fp8-e4m3 out.  With fp8 output every 128 consecutive elements share one fp32 scale
// (amax / 448, the block layout the MoE dispatch uses), written next to the data.
// The reference adds in the 16-bit element type and has no cast or scale
// (src/device/reduce_kernel.hpp:17-20); its design notes list more element types as future work
// (desgin/design-spec.md:1759).
//
// Shape of the kernel (same as the other NVLink collectives): [copy my input into the staging
// area] -> rank barrier -> every CTA pulls its slice of this rank's chunk from all ranks (plain
// peer loads, eight in flight per thread, or multimem.ld_reduce through the switch), scales,
// converts and stores locally -> rank barrier (peers are done reading my memory).
// Work is cut in units of 128 elements so that an fp8 scale block never straddles two CTAs, and
// the 128 elements of a block sit in consecutive lanes of one warp (16 lanes for 16-bit input, 32 for fp32
// input; half as many in the one-rank kernel, whose pieces are twice as long), which makes the block's amax a shuffle reduction.
#include <type_traits>

#include <algorithm>

#include "coll_device.cuh"
#include "collectives.cuh"
#include "fp8_cast.cuh"
#include "gemm_sm100.h"
#include "launch.cuh"

namespace uccl {
namespace dev {

enum : int { OUT_F16 = 0, OUT_BF16 = 1, OUT_F32 = 2, OUT_FP8 = 3 };

template <int OUT, int NE>
__device__ __forceinline__ void store_cast(char* out, size_t elem, const float (&v)[8]) {
  if (OUT == OUT_F32) {
    char* p = out + elem * 4;
    ptx::st_global_v4(p, make_uint4(__float_as_uint(v[0]), __float_as_uint(v[1]), __float_as_uint(v[2]), __float_as_uint(v[3])));
    if (NE == 8)
      ptx::st_global_v4(p + 16, make_uint4(__float_as_uint(v[4]), __float_as_uint(v[5]), __float_as_uint(v[6]), __float_as_uint(v[7])));
  } else if (OUT == OUT_BF16 || OUT == OUT_F16) {
    uint32_t w[4];
#pragma unroll
    for (int j = 0; j < NE / 2; ++j)
      w[j] = OUT == OUT_BF16 ? ptx::pack_bf16x2(v[2 * j], v[2 * j + 1]) : ptx::pack_f16x2(v[2 * j], v[2 * j + 1]);
    char* p = out + elem * 2;
    if (NE == 8) ptx::st_global_v4(p, make_uint4(w[0], w[1], w[2], w[3]));
    else *reinterpret_cast<uint2*>(p) = make_uint2(w[0], w[1]);
  }
}

// quantise with the block's scale: bit-identical to an fp32 restatement of the cast, as in the MoE dispatch
template <int NE>
__device__ __forceinline__ void store_fp8(char* out, size_t elem, const float (&v)[8], float blockScale) {
  const fp8::Divisor div(blockScale);
  uint32_t w[2] = {0, 0};
#pragma unroll
  for (int j = 0; j < NE / 4; ++j)
    w[j] = div.quantise4(make_float2(-v[4 * j], -v[4 * j + 1]), make_float2(-v[4 * j + 2], -v[4 * j + 3]));
  char* p = out + elem;
  if (NE == 8) *reinterpret_cast<uint2*>(p) = make_uint2(w[0], w[1]);
  else *reinterpret_cast<uint32_t*>(p) = w[0];
}

template <int DT, int OUT, bool NVLS>
__global__ void __launch_bounds__(kThreads, 1) reduce_cast_kernel(const __grid_constant__ CastArgs a) {
  using V = Vec<DT>;
  constexpr int NE = V::N;                 // elements per 16-byte input vector: 8 or 4
  constexpr int LANES = 128 / NE;          // lanes that share one 128-element block
  const DevComm& dc = a.dc;
  const int B = gridDim.x, b = blockIdx.x, n = dc.nranks;
  const size_t vecPerChunk = (a.chunkElems + NE - 1) / NE;
  const size_t units = (a.chunkElems + 127) / 128;
  size_t u0, ul;
  split(units, B, b, &u0, &ul);
  const size_t v0 = u0 * LANES, v1 = min(vecPerChunk, (u0 + ul) * LANES);
  if (a.inUser) {
    // my contribution to every rank's chunk goes into the staging area, same slice as I will read
    for (int s = 0; s < n; ++s) {
      const size_t begin = v0 << 4, len = v1 > v0 ? (v1 - v0) << 4 : 0;
      const size_t userBytes = a.chunkElems * V::ES;
      if (begin < userBytes)
        block_copy(const_cast<char*>(a.in[dc.rank]) + s * a.chunkStride + begin, a.inUser + s * a.inStride + begin,
                   min(len, userBytes - begin));
    }
  }
  if (!rank_barrier(dc)) return;
  const size_t mine = static_cast<size_t>(dc.rank) * a.chunkStride;
  // whole warps run every iteration: lanes beyond the slice's last vector still take part in the shuffles
  const size_t vEnd = v1 > v0 ? v0 + ((v1 - v0 + 31) / 32) * 32 : v0;
  for (size_t v = v0 + threadIdx.x; v < vEnd; v += blockDim.x) {
    const bool live = v < v1;
    float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    if (live) {
      const size_t off = mine + (v << 4);
      if (NVLS) {
        V::add(acc, V::mc_reduce(a.inMc + off));
      } else {
        uint4 d[8];
        for (int p0 = 0; p0 < n; p0 += 8) {
          const int m = min(8, n - p0);
#pragma unroll
          for (int j = 0; j < 8; ++j)
            if (j < m) d[j] = ptx::ld_stream_v4(a.in[(dc.rank + p0 + j) % n] + off);
#pragma unroll
          for (int j = 0; j < 8; ++j)
            if (j < m) V::add(acc, d[j]);
        }
      }
#pragma unroll
      for (int e = 0; e < NE; ++e) acc[e] *= a.scale;
    }
    const size_t elem = v * NE;
    if (OUT == OUT_FP8) {
      float amax = 0.f;
#pragma unroll
      for (int e = 0; e < NE; ++e) amax = fmaxf(amax, fabsf(acc[e]));
#pragma unroll
      for (int o = LANES / 2; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
      const float blockScale = fp8::block_scale(amax);
      if (live) {
        store_fp8<NE>(a.out, elem, acc, blockScale);
        if ((v % LANES) == 0) a.outScales[v / LANES] = blockScale;
      }
    } else if (live) {
      store_cast<OUT, NE>(a.out, elem, acc);
    }
  }
  rank_barrier(dc);
}

// One rank: nothing to add and nobody to meet, so the work is a stream from memory to memory.  Every
// thread takes U pieces of 32 input bytes (16 elements of a 16-bit type, 8 of fp32) that lie one CTA
// width apart, with all their loads in flight before the first use: four pieces (fp8 output: two) at four 256-thread
// CTAs per SM are 128 KiB in flight, where the shared kernel above, with one 16-byte load per thread
// on at most kMaxBlocks CTAs, reached a fifth of the memory bandwidth.  A 128-element scale block is
// 8 (or 16) consecutive lanes.
struct CastLocalArgs {
  const char* in;
  char* out;
  float* outScales;
  size_t elems;  // a multiple of 16 input bytes, and of 128 for fp8 output
  float scale;
  int wide;      // both buffers are 32-byte aligned
};

constexpr int kCastThreads = 256;

// Largest magnitude among the input elements of a scale block, which LANES consecutive lanes hold.
// Scaling is monotonic, so it may be applied to the maximum; 16-bit elements are compared two at a time.
template <int DT, int LANES>
__device__ __forceinline__ float piece_amax(const uint32_t (&raw)[8]) {
  if constexpr (DT == DT_F32) {
    float m = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) m = fmaxf(m, fabsf(__uint_as_float(raw[j])));
#pragma unroll
    for (int o = LANES / 2; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    return m;
  } else {
    using T2 = typename std::conditional<DT == DT_BF16, __nv_bfloat162, __half2>::type;
    auto as2 = [](uint32_t w) { return *reinterpret_cast<T2*>(&w); };
    T2 m = __habs2(as2(raw[0]));
#pragma unroll
    for (int j = 1; j < 8; ++j) m = __hmax2(m, __habs2(as2(raw[j])));
#pragma unroll
    for (int o = LANES / 2; o > 0; o >>= 1) m = __hmax2(m, as2(__shfl_xor_sync(0xffffffffu, *reinterpret_cast<uint32_t*>(&m), o)));
    const uint32_t w = *reinterpret_cast<uint32_t*>(&m);
    const float2 f = DT == DT_BF16 ? ptx::unpack_bf16x2(w) : ptx::unpack_f16x2(w);
    return fmaxf(0.f, fmaxf(f.x, f.y));
  }
}

// One CTA's share: U pieces per thread from piece `first` on.
template <int DT, int OUT, int U>
__device__ __forceinline__ void cast_share(const CastLocalArgs& a, size_t first) {
  constexpr int E = 32 / Vec<DT>::ES;  // elements per piece
  constexpr int LANES = 128 / E;    // lanes that share one scale block
  using T2 = typename std::conditional<DT == DT_BF16, __nv_bfloat162, __half2>::type;
  const size_t pieces = (a.elems + E - 1) / E;
  const size_t c0 = first + threadIdx.x;
  uint32_t raw[U][8];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const size_t c = c0 + u * kCastThreads;
    const char* p = a.in + c * 32;
#pragma unroll
    for (int j = 0; j < 8; ++j) raw[u][j] = 0;
    if (c < pieces) {
      if (a.wide && (c + 1) * E <= a.elems) {
        ptx::ld_stream_v8(p, raw[u]);
      } else {
        const uint4 lo = ptx::ld_stream_v4(p);
        raw[u][0] = lo.x, raw[u][1] = lo.y, raw[u][2] = lo.z, raw[u][3] = lo.w;
        if ((c + 1) * E <= a.elems) {  // the last piece may be half a one
          const uint4 hi = ptx::ld_stream_v4(p + 16);
          raw[u][4] = hi.x, raw[u][5] = hi.y, raw[u][6] = hi.z, raw[u][7] = hi.w;
        }
      }
    }
  }
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const size_t c = c0 + u * kCastThreads;
    const bool live = c < pieces, whole = (c + 1) * E <= a.elems;
    // 0 + x, as a sum starts: a zero comes out positive
    float2 v[E / 2];
    const float factor = OUT == OUT_FP8 ? -a.scale : a.scale;  // the divisor takes its elements negated
#pragma unroll
    for (int e = 0; e < E / 2; ++e) {
      float2 x;
      if constexpr (DT == DT_F32) {
        x = ptx::add2(make_float2(0.f, 0.f), make_float2(__uint_as_float(raw[u][2 * e]), __uint_as_float(raw[u][2 * e + 1])));
      } else {  // exact in the 16-bit type, and half the instructions there
        uint32_t z = 0;
        *reinterpret_cast<T2*>(&z) = __hadd2(*reinterpret_cast<T2*>(&z), *reinterpret_cast<T2*>(&raw[u][e]));
        x = DT == DT_BF16 ? ptx::unpack_bf16x2(z) : ptx::unpack_f16x2(z);
      }
      v[e] = ptx::mul2(x, make_float2(factor, factor));
    }
    char* out = a.out + c * E * (OUT == OUT_FP8 ? 1 : OUT == OUT_F32 ? 4 : 2);
    if (OUT == OUT_FP8) {
      const float blockScale = fp8::block_scale(fabsf(piece_amax<DT, LANES>(raw[u]) * a.scale));
      const fp8::Divisor div(blockScale);
      uint32_t w[E / 4];
#pragma unroll
      for (int j = 0; j < E / 4; ++j) w[j] = div.quantise4(v[2 * j], v[2 * j + 1]);
      if (live) {
        if constexpr (E == 16) ptx::st_global_v4(out, make_uint4(w[0], w[1], w[2], w[3]));
        else *reinterpret_cast<uint2*>(out) = make_uint2(w[0], w[1]);
        if (c % LANES == 0) a.outScales[c / LANES] = blockScale;
      }
    } else {
      constexpr int W = OUT == OUT_F32 ? E : E / 2;  // output words of a piece: 16, 8 or 4
      uint32_t w[W];
#pragma unroll
      for (int j = 0; j < W; ++j)
        w[j] = OUT == OUT_F32 ? __float_as_uint((j & 1) ? v[j / 2].y : v[j / 2].x) : OUT == OUT_BF16 ? ptx::pack_bf16x2(v[j].x, v[j].y) : ptx::pack_f16x2(v[j].x, v[j].y);
      if (W == 4) {  // fp32 -> 16 bits: a piece is 16 output bytes, and a half piece is 8
        if (live && whole) ptx::st_global_v4(out, make_uint4(w[0], w[1], w[2], w[3]));
        else if (live) *reinterpret_cast<uint2*>(out) = make_uint2(w[0], w[1]);
      } else {
#pragma unroll
        for (int j = 0; j < W; j += 8) {
          if (!live || (j * 2 >= W && !whole)) continue;
          const uint32_t(&o)[8] = *reinterpret_cast<const uint32_t(*)[8]>(&w[j]);
          if (a.wide && (W == 16 || whole)) {
            ptx::st_global_v8(out + j * 4, o);
          } else {
            ptx::st_global_v4(out + j * 4, make_uint4(o[0], o[1], o[2], o[3]));
            if (W == 16 || whole) ptx::st_global_v4(out + j * 4 + 16, make_uint4(o[4], o[5], o[6], o[7]));
          }
        }
      }
    }
  }
}
// Pieces per thread of a large launch, and CTAs per SM.  A conversion to fp8 takes some eighty instructions a piece, and
// two pieces on six CTAs (40 registers) put more of them beside other CTAs' loads than four pieces on four or two on five: 64 Mi bf16
// 31.1, 31.8 and 32.0 us, 16 Mi 9.2, 10.2 and 9.4, 32 Mi fp32 25.6, 26.4 and 25.6, 20 Mi fp16 10.9, 11.8 and 11.0.  Seven CTAs spill:
// 34.2, 10.2, 25.9, 13.1 (6 Mi fp32 alone is faster, 4.58 and 4.73).  With the other types, bound by loads and stores, it is the same.
template <int OUT>
constexpr int kCastPieces = OUT == OUT_FP8 ? 2 : 4;
template <int DT, int OUT, int U>
__global__ void __launch_bounds__(kCastThreads, U == 2 ? 6 : 4) cast_local_kernel(const __grid_constant__ CastLocalArgs a) {
  ptx::launch_dependents();
  ptx::wait_dependencies();
  cast_share<DT, OUT, U>(a, static_cast<size_t>(blockIdx.x) * (kCastThreads * U));
}
// Fewer CTAs than shares, for a communicator whose CTAs are limited.  A kernel of its own: with this loop around the
// one share of a CTA the launches without a limit took up to 1.3 times as long (4 MiB fp32 -> bf16: 4.4 -> 5.6 us).
template <int DT, int OUT>
__global__ void __launch_bounds__(kCastThreads, 4) cast_limited_kernel(const __grid_constant__ CastLocalArgs a) {
  constexpr size_t kShare = kCastThreads * 4, E = 32 / Vec<DT>::ES;
  for (size_t first = blockIdx.x * kShare; first < (a.elems + E - 1) / E; first += gridDim.x * kShare) cast_share<DT, OUT, 4>(a, first);
}

}  // namespace dev

// `limit`: the most CTAs the launch may have, 0 for none.  A limit is there to keep SMs free for other work, so no launch under
// one comes up beside the launch before, and one that goes in rounds does not let the one behind it come up: that would hold
// room on the SMs for as long as the rounds take.
template <int DT, int OUT>
static cudaError_t launchLocal(const dev::CastLocalArgs& a, int limit, cudaStream_t s) {
  const size_t pieces = (a.elems + 32 / dev::Vec<DT>::ES - 1) / (32 / dev::Vec<DT>::ES);
  // several pieces per thread once four would still give every SM its four CTAs; below that one piece per
  // thread spreads the work over more SMs
  constexpr size_t T = dev::kCastThreads;
  constexpr int U = dev::kCastPieces<OUT>;
  const bool many = pieces >= static_cast<size_t>(deviceSmCount()) * 4 * T * 4;
  const size_t share = many ? U * T : T, ctas = (pieces + share - 1) / share;
  if (limit > 0) {
    void (*kern)(dev::CastLocalArgs) = many ? dev::cast_local_kernel<DT, OUT, U> : dev::cast_local_kernel<DT, OUT, 1>;
    if (ctas > static_cast<size_t>(limit)) kern = dev::cast_limited_kernel<DT, OUT>;
    kern<<<static_cast<unsigned>(std::min<size_t>(ctas, limit)), T, 0, s>>>(a);
    return cudaGetLastError();
  }
  if (many) return launchOverlapped(dev::cast_local_kernel<DT, OUT, U>, static_cast<unsigned>(ctas), T, 0, s, a);
  return launchOverlapped(dev::cast_local_kernel<DT, OUT, 1>, static_cast<unsigned>(ctas), T, 0, s, a);
}

template <int DT>
static cudaError_t launchLocalOut(const dev::CastLocalArgs& a, int outType, int limit, cudaStream_t s) {
  switch (outType) {
    case ucclFloat16: return launchLocal<DT, dev::OUT_F16>(a, limit, s);
    case ucclBfloat16: return launchLocal<DT, dev::OUT_BF16>(a, limit, s);
    case ucclFloat32: return launchLocal<DT, dev::OUT_F32>(a, limit, s);
    case ucclFloat8e4m3: return launchLocal<DT, dev::OUT_FP8>(a, limit, s);
    default: return cudaErrorInvalidValue;
  }
}

template <int DT, bool NVLS>
static cudaError_t launchOut(const CastArgs& a, int blocks, cudaStream_t s) {
  switch (a.outType) {
    case ucclFloat16: dev::reduce_cast_kernel<DT, dev::OUT_F16, NVLS><<<blocks, dev::kThreads, 0, s>>>(a); break;
    case ucclBfloat16: dev::reduce_cast_kernel<DT, dev::OUT_BF16, NVLS><<<blocks, dev::kThreads, 0, s>>>(a); break;
    case ucclFloat32: dev::reduce_cast_kernel<DT, dev::OUT_F32, NVLS><<<blocks, dev::kThreads, 0, s>>>(a); break;
    case ucclFloat8e4m3: dev::reduce_cast_kernel<DT, dev::OUT_FP8, NVLS><<<blocks, dev::kThreads, 0, s>>>(a); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

cudaError_t launchCastKernel(const CastArgs& a, int limit, cudaStream_t s) {
  dev::CastLocalArgs l;
  l.in = a.in[0];
  l.out = a.out;
  l.outScales = a.outScales;
  l.elems = a.chunkElems;
  l.scale = a.scale;
  l.wide = ((reinterpret_cast<uintptr_t>(l.in) | reinterpret_cast<uintptr_t>(l.out)) & 31) == 0;
  switch (a.inType) {
    case ucclFloat16: return launchLocalOut<dev::DT_F16>(l, a.outType, limit, s);
    case ucclBfloat16: return launchLocalOut<dev::DT_BF16>(l, a.outType, limit, s);
    case ucclFloat32: return launchLocalOut<dev::DT_F32>(l, a.outType, limit, s);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t launchReduceCastKernel(const CastArgs& a, int blocks, cudaStream_t s) {
  if (blocks < 1 || blocks > kMaxBlocks) return cudaErrorInvalidValue;
  const bool nvls = a.inMc != nullptr;
  switch (a.inType) {
    case ucclFloat16: return nvls ? launchOut<dev::DT_F16, true>(a, blocks, s) : launchOut<dev::DT_F16, false>(a, blocks, s);
    case ucclBfloat16: return nvls ? launchOut<dev::DT_BF16, true>(a, blocks, s) : launchOut<dev::DT_BF16, false>(a, blocks, s);
    case ucclFloat32: return nvls ? launchOut<dev::DT_F32, true>(a, blocks, s) : launchOut<dev::DT_F32, false>(a, blocks, s);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace uccl
