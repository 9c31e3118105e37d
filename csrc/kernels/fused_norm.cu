// Fused all-reduce + residual add + RMSNorm for tensor-parallel layers (bf16).
//
//   h   = sum over ranks of x_r + residual          (kept as the new residual stream)
//   out = h * rsqrt(mean(h^2) + eps) * gamma
//
// The reference has no fused epilogues.  The library baseline is an all-reduce followed by a
// separate normalisation kernel: the reduced tensor crosses NVLink twice (reduce-scatter and
// all-gather halves) and is then read and written once more from HBM.  Here the token rows are
// sharded over the ranks:
//   phase A  each rank reduces its own rows (multimem.ld_reduce in the switch, or peer loads),
//            adds the residual, rounds to bf16 and stores the new residual row into every rank
//            (multimem.st, or peer stores); it normalises those rows while they are in registers;
//   phase B  after a rank barrier every rank normalises the rows it received, reading each once.
// Only one tensor travels the all-gather direction; the normalised output never crosses NVLink.
// CTA b handles rows b, b+B, ... of every shard in both phases, so the CTA-level rank barrier
// covers exactly the rows it later reads.
#include <algorithm>

#include "coll_device.cuh"
#include "collectives.cuh"
#include "launch.cuh"
#include "gemm_sm100.h"

#ifdef UCCL_EXPERIMENTS
#define UCCL_NORM_DBG(a, bit) (((a).debug & (bit)) != 0)  // leave a phase out to time the rest (benchmarks/fused_layers.py)
#else
#define UCCL_NORM_DBG(a, bit) false
#endif

namespace uccl {
namespace dev {

constexpr int kNormMaxVec = 4;  // 16-byte vectors per thread and row: hidden <= 4 * 512 * 8 = 16384
constexpr int kNormSlots = 8;   // 16-byte vectors a thread keeps in flight: rows per pass x vectors per row
constexpr int kNormMaxRows = 4; // rows a CTA works on per pass

// Sums R per-row partials over the CTA in one pass (two barriers for all rows together).
__device__ __forceinline__ void block_sum_rows(float (&v)[kNormMaxRows]) {
  __shared__ float red[kNormMaxRows][kThreads / 32];
  __shared__ float total[kNormMaxRows];
#pragma unroll
  for (int j = 0; j < kNormMaxRows; ++j)
    for (int o = 16; o > 0; o >>= 1) v[j] += __shfl_xor_sync(0xffffffffu, v[j], o);
  if ((threadIdx.x & 31) == 0) {
#pragma unroll
    for (int j = 0; j < kNormMaxRows; ++j) red[j][threadIdx.x >> 5] = v[j];
  }
  __syncthreads();
  if (threadIdx.x < 32 * kNormMaxRows) {
    const int j = threadIdx.x >> 5, l = threadIdx.x & 31;
    float t = l < kThreads / 32 ? red[j][l] : 0.f;
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (l == 0) total[j] = t;
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < kNormMaxRows; ++j) v[j] = total[j];
  __syncthreads();
}

// One pass = R rows (R * nvecThread <= kNormSlots).  Slot s of a thread is vector s % nvecThread
// of row s / nvecThread of the pass.
struct NormPass {
  int nvecThread;  // vectors per thread and row
  int R;           // rows per pass
  __device__ __forceinline__ bool slot(int s, int rowsHere, int* j, int* v) const {
    *j = s / nvecThread;
    *v = threadIdx.x + (s - *j * nvecThread) * kThreads;
    return *j < rowsHere;
  }
};

// out rows = h * rsqrt(mean(h^2) + eps) * gamma for the rows of one pass held in registers
__device__ __forceinline__ void normalise_rows(const NormPass& np, const uint4 (&h)[kNormSlots], int rowsHere,
                                               const size_t (&rowIdx)[kNormMaxRows], const __nv_bfloat16* gamma, char* out,
                                               size_t rowBytes, float eps, int hidden) {
  const int vecPerRow = hidden >> 3;
  float ss[kNormMaxRows] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int s = 0; s < kNormSlots; ++s) {
    int j, v;
    if (np.slot(s, rowsHere, &j, &v)) {
      const uint32_t w[4] = {h[s].x, h[s].y, h[s].z, h[s].w};
      float t = 0.f;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 f = ptx::unpack_bf16x2(w[e]);
        t += f.x * f.x + f.y * f.y;
      }
#pragma unroll
      for (int jj = 0; jj < kNormMaxRows; ++jj)
        if (jj == j) ss[jj] += t;
    }
  }
  block_sum_rows(ss);
#pragma unroll
  for (int s = 0; s < kNormSlots; ++s) {
    int j, v;
    if (np.slot(s, rowsHere, &j, &v) && v < vecPerRow) {
      float sum = ss[0];
#pragma unroll
      for (int jj = 1; jj < kNormMaxRows; ++jj)
        if (jj == j) sum = ss[jj];
      size_t row = rowIdx[0];
#pragma unroll
      for (int jj = 1; jj < kNormMaxRows; ++jj)
        if (jj == j) row = rowIdx[jj];
      const float rstd = rsqrtf(sum / static_cast<float>(hidden) + eps);
      const uint4 g = *reinterpret_cast<const uint4*>(reinterpret_cast<const char*>(gamma) + (static_cast<size_t>(v) << 4));
      const uint32_t w[4] = {h[s].x, h[s].y, h[s].z, h[s].w};
      const uint32_t gw[4] = {g.x, g.y, g.z, g.w};
      uint32_t o[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 f = ptx::unpack_bf16x2(w[e]);
        const float2 gg = ptx::unpack_bf16x2(gw[e]);
        o[e] = ptx::pack_bf16x2(f.x * rstd * gg.x, f.y * rstd * gg.y);
      }
      ptx::st_global_v4(out + row * rowBytes + (static_cast<size_t>(v) << 4), make_uint4(o[0], o[1], o[2], o[3]));
    }
  }
}

__device__ __forceinline__ uint4 add_bf16x8(uint4 x, uint4 y) {
  float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  Vec<DT_BF16>::add(acc, x);
  Vec<DT_BF16>::add(acc, y);
  return Vec<DT_BF16>::pack(acc);
}

__global__ void __launch_bounds__(kThreads, 1) ar_norm_kernel(const __grid_constant__ ArNormArgs a) {
  const DevComm& dc = a.dc;
  const int B = gridDim.x, b = blockIdx.x, n = dc.nranks, me = dc.rank;
  const int vecPerRow = a.hidden >> 3;
  const size_t rowBytes = static_cast<size_t>(a.hidden) * 2;
  const int perRow = (vecPerRow + kThreads - 1) / kThreads;  // slots per row (same for every thread)
  NormPass np;
  np.nvecThread = perRow;
  np.R = min(kNormMaxRows, kNormSlots / perRow);

  // staged input: CTA b copies the rows it will be asked for by peers (rows b, b+B, ... of every shard)
  if (a.inUser) {
    for (int p = 0; p < n; ++p) {
      size_t ro, rl;
      split(static_cast<size_t>(a.tokens), n, p, &ro, &rl);
      for (size_t r = b; r < rl; r += B)
        block_copy(const_cast<char*>(a.in[me]) + (ro + r) * rowBytes, a.inUser + (ro + r) * rowBytes, rowBytes);
    }
  }
  if (!rank_barrier(dc)) return;

  size_t myOff, myLen;
  split(static_cast<size_t>(a.tokens), n, me, &myOff, &myLen);
  // ---- phase A: my rows (rows b, b+B, ... of my shard).  Through the switch one row per pass is
  // enough to cover the latency (the links, not the loads in flight, are the limit) and lets the
  // stores of one pass travel while the loads of the next are already out; the peer path takes R.
  const NormPass npB = np;
  // Through the switch phase A is a plain all-reduce loop over this rank's rows (reduce in the
  // switch, add the residual, broadcast through the switch), as many rows in flight as the
  // registers hold and no CTA-wide reduction in between; the rows are normalised in phase B with
  // everybody else's, from local memory.  mcRows = 1, 2 or 4 rows per pass, 0 = the older form
  // that normalises its own rows from registers one row per pass.
  const bool splitNorm = a.inMc && a.resOutMc && a.mcRows > 0;
  if (a.inMc) np.R = splitNorm ? max(1, min(np.R, a.mcRows)) : 1;
  for (size_t r0 = b; r0 < (UCCL_NORM_DBG(a, 4) ? 0 : myLen); r0 += static_cast<size_t>(B) * np.R) {
    size_t rowIdx[kNormMaxRows];
    int rowsHere = 0;
#pragma unroll
    for (int j = 0; j < kNormMaxRows; ++j) {
      const size_t r = r0 + static_cast<size_t>(j) * B;
      rowIdx[j] = myOff + (r < myLen ? r : r0);
      if (j < np.R && r < myLen) rowsHere = j + 1;
    }
    uint4 h[kNormSlots], res[kNormSlots];
    // all loads of the pass are issued before the first use
#pragma unroll
    for (int s = 0; s < kNormSlots; ++s) {
      int j, v;
      if (np.slot(s, rowsHere, &j, &v) && v < vecPerRow) {
        size_t row = rowIdx[0];
#pragma unroll
        for (int jj = 1; jj < kNormMaxRows; ++jj)
          if (jj == j) row = rowIdx[jj];
        const size_t off = row * rowBytes + (static_cast<size_t>(v) << 4);
        if (a.inMc) {
          h[s] = ptx::multimem_ld_reduce_bf16x8(a.inMc + off);
        } else {
          float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
          for (int p = 0; p < n; ++p) Vec<DT_BF16>::add(acc, ptx::ld_stream_v4(a.in[(me + p) % n] + off));
          h[s] = Vec<DT_BF16>::pack(acc);
        }
        res[s] = ptx::ld_global_v4(reinterpret_cast<const char*>(a.residual) + off);
      } else {
        h[s] = make_uint4(0, 0, 0, 0);
        res[s] = make_uint4(0, 0, 0, 0);
      }
    }
#pragma unroll
    for (int s = 0; s < kNormSlots; ++s) {
      int j, v;
      if (np.slot(s, rowsHere, &j, &v) && v < vecPerRow) {
        size_t row = rowIdx[0];
#pragma unroll
        for (int jj = 1; jj < kNormMaxRows; ++jj)
          if (jj == j) row = rowIdx[jj];
        const size_t off = row * rowBytes + (static_cast<size_t>(v) << 4);
        h[s] = add_bf16x8(h[s], res[s]);
        if (UCCL_NORM_DBG(a, 2)) {
        } else if (a.resOutMc) {
          ptx::multimem_st_v4(a.resOutMc + off, h[s]);
        } else {
          for (int p = 0; p < n; ++p) ptx::st_global_v4(a.resOut[(me + p) % n] + off, h[s]);
        }
      }
    }
    if (!splitNorm) normalise_rows(np, h, rowsHere, rowIdx, a.gamma, a.outLocal, rowBytes, a.eps, a.hidden);
  }
  if (!rank_barrier(dc)) return;
  // ---- phase B: rows owned by the other ranks, now present in my copy of the residual stream
  for (int q = splitNorm ? 0 : 1; q < (UCCL_NORM_DBG(a, 1) ? 0 : n); ++q) {
    const int p = (me + q) % n;
    size_t ro, rl;
    split(static_cast<size_t>(a.tokens), n, p, &ro, &rl);
    for (size_t r0 = b; r0 < rl; r0 += static_cast<size_t>(B) * npB.R) {
      size_t rowIdx[kNormMaxRows];
      int rowsHere = 0;
#pragma unroll
      for (int j = 0; j < kNormMaxRows; ++j) {
        const size_t r = r0 + static_cast<size_t>(j) * B;
        rowIdx[j] = ro + (r < rl ? r : r0);
        if (j < npB.R && r < rl) rowsHere = j + 1;
      }
      uint4 h[kNormSlots];
#pragma unroll
      for (int s = 0; s < kNormSlots; ++s) {
        int j, v;
        if (npB.slot(s, rowsHere, &j, &v) && v < vecPerRow) {
          size_t row = rowIdx[0];
#pragma unroll
          for (int jj = 1; jj < kNormMaxRows; ++jj)
            if (jj == j) row = rowIdx[jj];
          h[s] = ptx::ld_global_v4(a.resOut[me] + row * rowBytes + (static_cast<size_t>(v) << 4));
        } else {
          h[s] = make_uint4(0, 0, 0, 0);
        }
      }
      normalise_rows(npB, h, rowsHere, rowIdx, a.gamma, a.outLocal, rowBytes, a.eps, a.hidden);
    }
  }
  // staged residual: hand the rows back to the user's buffer
  if (a.resOutUser) {
    for (int p = 0; p < n; ++p) {
      size_t ro, rl;
      split(static_cast<size_t>(a.tokens), n, p, &ro, &rl);
      for (size_t r = b; r < rl; r += B)
        block_copy(a.resOutUser + (ro + r) * rowBytes, a.resOut[me] + (ro + r) * rowBytes, rowBytes);
    }
  }
}

// ------------------------------------------------------------------ one rank
// out = rmsnorm(x + residual) * gamma without any communication: 2 reads and 2 writes per element.
struct NormLocalArgs {
  const char* x;
  const char* residual;
  const char* gamma;
  char* out;
  char* resOut;  // may be `residual`
  int tokens, hidden;
  float eps;
};

// h = bf16(x + residual), and the sum of its squares is added to `ss`
__device__ __forceinline__ uint4 add_square(uint4 x, uint4 res, float& ss) {
  const uint4 h = add_bf16x8(x, res);
  const uint32_t w[4] = {h.x, h.y, h.z, h.w};
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const float2 f = ptx::unpack_bf16x2(w[e]);
    ss += f.x * f.x + f.y * f.y;
  }
  return h;
}
__device__ __forceinline__ uint4 scale_gamma(uint4 h, uint4 g, float rstd) {
  const uint32_t w[4] = {h.x, h.y, h.z, h.w}, gw[4] = {g.x, g.y, g.z, g.w};
  uint32_t o[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const float2 f = ptx::unpack_bf16x2(w[e]), gg = ptx::unpack_bf16x2(gw[e]);
    o[e] = ptx::pack_bf16x2(f.x * rstd * gg.x, f.y * rstd * gg.y);
  }
  return make_uint4(o[0], o[1], o[2], o[3]);
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// W bytes (16 or 32) of a row per piece, NV pieces per thread, `lanes` threads per row and blockDim / lanes
// rows per CTA.  Bound by memory: all loads of a thread are out before the first use, and nothing is
// persistent, so that on every SM some CTAs load while others reduce and store.  8192 x 8192: 82 us =
// 6.5 TB/s, what a copy reaches; one persistent CTA per SM took 109 us (loads into registers, four rows
// per pass) and 100 us (a ring of bulk loads, 190 KiB of them in flight: groups of warps then wait for
// each other's reductions).
template <int NV, int W>
__global__ void __launch_bounds__(NV * W > 32 ? 512 : 1024) add_norm_kernel(const __grid_constant__ NormLocalArgs a, int lanes) {
  __shared__ float part[32];
  constexpr int Q = W / 16;
  const int t = threadIdx.x % lanes, sub = threadIdx.x / lanes;
  const long row = static_cast<long>(blockIdx.x) * (blockDim.x / lanes) + sub;
  const bool live = row < a.tokens;
  const int pieces = live ? (a.hidden * 2) / W : 0;
  const size_t base = static_cast<size_t>(row) * a.hidden * 2;
  uint4 x[NV][Q], r[NV][Q];
  auto load = [](const char* p, uint4 (&v)[Q]) {
    if constexpr (Q == 2) {
      uint32_t w[8];
      ptx::ld_stream_v8(p, w);
      v[0] = make_uint4(w[0], w[1], w[2], w[3]);
      v[1] = make_uint4(w[4], w[5], w[6], w[7]);
    } else {
      v[0] = ptx::ld_stream_v4(p);
    }
  };
  auto store = [](char* p, const uint4 (&v)[Q]) {
    if constexpr (Q == 2) {
      const uint32_t w[8] = {v[0].x, v[0].y, v[0].z, v[0].w, v[1].x, v[1].y, v[1].z, v[1].w};
      ptx::st_global_v8(p, w);
    } else {
      ptx::st_global_v4(p, v[0]);
    }
  };
  ptx::launch_dependents();
  ptx::wait_dependencies();
#pragma unroll
  for (int j = 0; j < NV; ++j) {
    const int v = t + j * lanes;
#pragma unroll
    for (int q = 0; q < Q; ++q) x[j][q] = r[j][q] = make_uint4(0, 0, 0, 0);
    if (v < pieces) {
      load(a.x + base + static_cast<size_t>(v) * W, x[j]);
      load(a.residual + base + static_cast<size_t>(v) * W, r[j]);
    }
  }
  float ss = 0.f;
#pragma unroll
  for (int j = 0; j < NV; ++j) {
    const int v = t + j * lanes;
#pragma unroll
    for (int q = 0; q < Q; ++q) x[j][q] = add_square(x[j][q], r[j][q], ss);
    if (v < pieces) store(a.resOut + base + static_cast<size_t>(v) * W, x[j]);
  }
  ss = warp_sum(ss);
  if (lanes > 32) {
    const int warps = lanes >> 5, l = threadIdx.x & 31;
    if (l == 0) part[threadIdx.x >> 5] = ss;
    __syncthreads();
    ss = warp_sum(l < warps ? part[sub * warps + l] : 0.f);
  }
  const float rstd = rsqrtf(ss / static_cast<float>(a.hidden) + a.eps);
#pragma unroll
  for (int j = 0; j < NV; ++j) {
    const int v = t + j * lanes;
    if (v < pieces) {
#pragma unroll
      for (int q = 0; q < Q; ++q)
        x[j][q] = scale_gamma(x[j][q], ptx::ld_global_v4(a.gamma + static_cast<size_t>(v) * W + q * 16), rstd);
      store(a.out + base + static_cast<size_t>(v) * W, x[j]);
    }
  }
}

}  // namespace dev

template <int W>
static cudaError_t launchNormLocal(const dev::NormLocalArgs& l, cudaStream_t s) {
  const int pieces = l.hidden * 2 / W;
  // two CTAs of rows per SM or fewer (decode): a thread per piece, for the shortest chain.  More rows: up to
  // 64 bytes of either input per thread, so that a barrier and its shuffles pay for more data.
  const int most = l.tokens <= 2 * deviceSmCount() ? (pieces + 1023) / 1024 : (pieces > 32 ? 64 / W : 1);
  const int nv = most <= 1 ? 1 : most <= 2 ? 2 : 4;
  const int lanes = ((pieces + nv - 1) / nv + 31) / 32 * 32;
  const int rows = lanes >= 256 ? 1 : 256 / lanes;
  const unsigned grid = static_cast<unsigned>((static_cast<long>(l.tokens) + rows - 1) / rows);
  if (nv == 1) return launchOverlapped(dev::add_norm_kernel<1, W>, grid, lanes * rows, 0, s, l, lanes);
  if constexpr (W == 16) {  // 32-byte pieces: two at most
    if (nv > 2) return launchOverlapped(dev::add_norm_kernel<4, W>, grid, lanes * rows, 0, s, l, lanes);
  }
  return launchOverlapped(dev::add_norm_kernel<2, W>, grid, lanes * rows, 0, s, l, lanes);
}

cudaError_t launchArNormKernel(const ArNormArgs& a, int blocks, cudaStream_t stream) {
  if (a.hidden % 8 != 0 || a.hidden > dev::kNormMaxVec * dev::kThreads * 8) return cudaErrorInvalidValue;
  if (a.dc.nranks <= 1) {
    dev::NormLocalArgs l;
    l.x = a.inUser;
    l.residual = reinterpret_cast<const char*>(a.residual);
    l.gamma = reinterpret_cast<const char*>(a.gamma);
    l.out = a.outLocal;
    l.resOut = a.resOutUser;
    l.tokens = a.tokens;
    l.hidden = a.hidden;
    l.eps = a.eps;
    const uintptr_t all = reinterpret_cast<uintptr_t>(l.x) | reinterpret_cast<uintptr_t>(l.residual) |
                          reinterpret_cast<uintptr_t>(l.out) | reinterpret_cast<uintptr_t>(l.resOut) | (a.hidden * 2);
    return (all & 31) == 0 ? launchNormLocal<32>(l, stream) : launchNormLocal<16>(l, stream);
  }
  // one cross-rank barrier slot per CTA
  if (blocks < 1 || blocks > kMaxBlocks) return cudaErrorInvalidValue;
  dev::ar_norm_kernel<<<blocks, dev::kThreads, 0, stream>>>(a);
  return cudaGetLastError();
}

}  // namespace uccl
