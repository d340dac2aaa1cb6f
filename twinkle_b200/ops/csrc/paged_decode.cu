// Paged-cache decode attention on the tensor cores: one query token per sequence, bf16 rows of 64 or 128 elements, groups of four query heads
// or more, up to 8 at a time (larger groups take several CTAs).  Score terms and other widths, types and groups go through the vector kernel in
// decode.cu.
//
// What bounds it: the cache, 4·D bytes per token and key head, read once from HBM.  The vector kernel spends 2·G·D fused multiply-adds and 3
// shuffles per head on every token and was bound by them (1.37 TB/s at 16 sequences of 4–8 k tokens, 32 / 8 heads of 128).  Here a warp takes 16 tokens at
// a time with mma.m16n8k16 (the heads are rows 0–7 of A; tcgen05 wants 64 rows at least, of which a group would fill 8), which leaves memory as the
// bound.  32 / 8 heads of 128, us and share of the 6.4 TB/s that a copy reaches, before → now: 256 sequences of 0.6–1.3 k tokens 360 (43 %) → 164
// (95 %), 64 of 0.5–1 k 93 (33 %) → 42 (75 %), 16 of 4–8 k 295 (21 %) → 75 (85 %).
//
// Split: a worker is a warp; tiles of 16 tokens go round robin over all warps of a cluster of S CTAs that share one (sequence, key head).  Each
// warp keeps a ring of STAGES tiles of K and V filled by cp.async, and never waits for another warp before the merge.  The CTA merges
// its warps through shared memory, the cluster its CTAs through distributed shared memory, so there is neither a workspace nor a second launch.
//
// Precision: scores are sums of bf16 products in fp32, scaled afterwards (q is not rounded again).  Probabilities are multiplied as two bf16 parts, whose
// remainder is below 2^-17 of the value, in fp32 sums: rows 0–7 of A carry the leading part, rows 8–15 the rest, at no cost.  The denominator is the sum of the fp32 values.
// The distance from 64 bits is the vector kernel's to five digits (32/8, 32/4 and 16/4 heads, 4 to 64 sequences, contexts of 50 to 8192 tokens: 1.61e-3 to
// 1.69e-3 both, which is the rounding of the result to bf16).  The order of sums follows the number of sequences and the width of the table (cluster_size).
#include <ATen/cuda/CUDAContext.h>
#include <cooperative_groups.h>
#include <torch/types.h>

#include "common.cuh"
#include "host.h"
#include "mma16.cuh"
#include "paged_decode.h"

namespace tk {

using bf16 = __nv_bfloat16;

namespace pd {
constexpr int WARPS = 4, TILE = 16, STAGES = 3, HEADS = 8;
template <int D> constexpr int row_bytes() { return 2 * D; }
template <int D> constexpr int stage_bytes() { return 2 * TILE * row_bytes<D>(); }                // K and V
template <int D> constexpr int smem_bytes() { return WARPS * STAGES * stage_bytes<D>(); }
}  // namespace pd

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool live) {   // zeros when not live
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(live ? 16 : 0) : "memory");
}

// A sum from leading parts and remainders.  An infinite value meets a positive leading part, and a remainder that is zero or negative: the leading sum is the result.
__device__ __forceinline__ float whole(float lead, float rest) { return fabsf(lead) == INFINITY ? lead : lead + rest; }

template <int D>
__global__ void __launch_bounds__(pd::WARPS * 32, 2) paged_decode_mma_kernel(const PagedDecode p) {
  using namespace pd;
  namespace cg = cooperative_groups;
  constexpr int CH = D / 8;                 // 16-byte chunks of a row
  constexpr int RPI = 32 / CH;              // rows that one load instruction of a warp covers
  const cg::cluster_group cluster = cg::this_cluster();
  const int S = gridDim.x, split = blockIdx.x, b = blockIdx.z;
  const int groups = (p.G + HEADS - 1) / HEADS, kvh = blockIdx.y / groups, g0 = blockIdx.y % groups * HEADS, h0 = kvh * p.G + g0, GH = min(HEADS, p.G - g0);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, quad = lane & 3, hrow = lane >> 2;
  const int n = p.seq_lens[b], first = n > 0 ? first_visible(n - 1, p.window, p.chunk) : 0;
  const int base = first & ~(TILE - 1), tiles = n > base ? (n - base + TILE - 1) / TILE : 0, workers = S * WARPS, worker = split * WARPS + warp;
  const int mine = tiles > worker ? (tiles - worker + workers - 1) / workers : 0;

  extern __shared__ __align__(128) uint8_t smem[];
  uint8_t* ring = smem + warp * STAGES * stage_bytes<D>();
  const int* table = p.tables + static_cast<size_t>(b) * p.max_blocks;
  const bf16 *kc = reinterpret_cast<const bf16*>(p.kc), *vc = reinterpret_cast<const bf16*>(p.vc);

  // row of the pools that holds token (lane & 15) of this warp's tile i, or −1; looked up one tile before it is needed
  auto lookup = [&](int i) -> int {
    const int t = base + (worker + i * workers) * TILE + (lane & 15);
    if (i >= mine || t >= n || t < first) return -1;
    return table[t / p.block_size] * p.block_size + t % p.block_size;
  };
  auto fetch = [&](int i, int rows) {
    const uint32_t dst = smem_u32(ring) + (i % STAGES) * stage_bytes<D>();
#pragma unroll
    for (int k = 0; k < TILE / RPI; ++k) {
      const int r = k * RPI + lane / CH, c = lane % CH, row = __shfl_sync(0xffffffffu, rows, r);
      const size_t at = (static_cast<size_t>(max(row, 0)) * p.hkv + kvh) * D + c * 8;
      const uint32_t off = r * row_bytes<D>() + ((c ^ (r & 7)) << 4);      // chunks of a row are exchanged so that ldmatrix meets all banks
      cp_async16(dst + off, kc + at, row >= 0);
      cp_async16(dst + TILE * row_bytes<D>() + off, vc + at, row >= 0);
    }
  };
  int ahead = lookup(0);
#pragma unroll
  for (int i = 0; i < STAGES - 1; ++i) {
    const int rows = ahead;
    ahead = lookup(i + 1);
    if (i < mine) fetch(i, rows);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }

  // the heads' rows of A; rows 8–15 are zero for the scores
  uint32_t qa[D / 16][2];
#pragma unroll
  for (int k = 0; k < D / 16; ++k) {
    qa[k][0] = qa[k][1] = 0u;
    if (hrow < GH) {
      const uint32_t* q = reinterpret_cast<const uint32_t*>(reinterpret_cast<const bf16*>(p.q) + (static_cast<size_t>(b) * p.hq + h0 + hrow) * D + k * 16 + quad * 2);
      qa[k][0] = q[0];
      qa[k][1] = q[4];
    }
  }
  float m = -INFINITY, l = 0.f, acc[D / 8][4];
#pragma unroll
  for (int j = 0; j < D / 8; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;

  for (int i = 0; i < mine; ++i) {
    asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
    __syncwarp();
    {
      const int rows = ahead;
      ahead = lookup(i + STAGES);
      if (i + STAGES - 1 < mine) fetch(i + STAGES - 1, rows);       // the stage that tile i − 1 has left
      asm volatile("cp.async.commit_group;" ::: "memory");
    }
    const uint8_t *ks = ring + (i % STAGES) * stage_bytes<D>(), *vs = ks + TILE * row_bytes<D>();
    float s[2][4] = {};
    {
      const int r = (lane & 7) + ((lane >> 4) << 3), half = (lane >> 3) & 1;      // tokens 0–7 chunks 0, 1; tokens 8–15 chunks 0, 1
#pragma unroll
      for (int k = 0; k < D / 16; ++k) {
        uint32_t bk[4];
        ldsm4(bk, reinterpret_cast<const bf16*>(ks + r * row_bytes<D>() + (((2 * k + half) ^ (r & 7)) << 4)));
        const uint32_t a[4] = {qa[k][0], 0u, qa[k][1], 0u};
        mma(s[0], a, bk[0], bk[1]);
        mma(s[1], a, bk[2], bk[3]);
      }
    }
    const int t0 = base + (worker + i * workers) * TILE + quad * 2;
    float mx = -INFINITY;
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int t = t0 + j * 8 + e;
        s[j][e] = t < n && t >= first ? s[j][e] * p.scale_log2 : -INFINITY;
        mx = fmaxf(mx, s[j][e]);
      }
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
    const float mn = fmaxf(m, mx), sub = mn == -INFINITY ? 0.f : mn;
    if (__any_sync(0xffffffffu, mn != m)) {
      const float corr = fast_exp2(m - sub);       // 2^−∞ = 0 before the first key
      l *= corr;
#pragma unroll
      for (int j = 0; j < D / 8; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[j][e] *= corr;
    }
    m = mn;
    uint32_t a[4];                                  // leading parts in rows 0–7, remainders in rows 8–15
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const float p0 = fast_exp2(s[j][0] - sub), p1 = fast_exp2(s[j][1] - sub);
      l += p0 + p1;
      split2(p0, p1, a[2 * j], a[2 * j + 1]);
    }
    const int r = lane & 15, half = lane >> 4;     // tokens 0–15 of chunk 2j, tokens 0–15 of chunk 2j + 1
#pragma unroll
    for (int j = 0; j < D / 16; ++j) {
      uint32_t bv[4];
      ldsm4t(bv, reinterpret_cast<const bf16*>(vs + r * row_bytes<D>() + (((2 * j + half) ^ (r & 7)) << 4)));
      mma(acc[2 * j], a, bv[0], bv[1]);
      mma(acc[2 * j + 1], a, bv[2], bv[3]);
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  l += __shfl_xor_sync(0xffffffffu, l, 1);
  l += __shfl_xor_sync(0xffffffffu, l, 2);
  __syncthreads();                                  // the rings are free: they take the merge

  float* part = reinterpret_cast<float*>(smem);                       // [WARPS][HEADS][D]
  float* stat = part + WARPS * HEADS * D;                             // [WARPS][HEADS] maximum, sum
  float* sum = stat + 2 * WARPS * HEADS;                              // [HEADS][D] of this CTA, then [HEADS] maximum, [HEADS] sum
  float* top = sum + HEADS * D;
#pragma unroll
  for (int j = 0; j < D / 8; ++j)
    *reinterpret_cast<float2*>(&part[(warp * HEADS + hrow) * D + j * 8 + quad * 2]) = make_float2(whole(acc[j][0], acc[j][2]), whole(acc[j][1], acc[j][3]));
  if (quad == 0) {
    stat[warp * HEADS + hrow] = m;
    stat[(WARPS + warp) * HEADS + hrow] = l;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < HEADS * D; i += WARPS * 32) {
    const int h = i / D;
    float mm = stat[h];
#pragma unroll
    for (int w = 1; w < WARPS; ++w) mm = fmaxf(mm, stat[w * HEADS + h]);
    float o = 0.f, ll = 0.f;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) {
      const float mw = stat[w * HEADS + h], c = mw == -INFINITY ? 0.f : fast_exp2(mw - mm);
      o += part[w * HEADS * D + i] * c;
      ll += stat[(WARPS + w) * HEADS + h] * c;
    }
    sum[i] = o;
    if (i % D == 0) {
      top[h] = mm;
      top[HEADS + h] = ll;
    }
  }
  if (S > 1) cluster.sync(); else __syncthreads();
  // CTA r of the cluster finishes every S-th stretch of 128 results
  for (int i = split * WARPS * 32 + threadIdx.x; i < GH * D; i += S * WARPS * 32) {
    const int h = i / D;
    float mm = -INFINITY, sink = 0.f;
    if (p.sinks != nullptr) mm = sink = __bfloat162float(reinterpret_cast<const bf16*>(p.sinks)[h0 + h]) * 1.4426950408889634f;
    for (int r = 0; r < S; ++r) mm = fmaxf(mm, cluster.map_shared_rank(top, r)[h]);
    float o = 0.f, ll = p.sinks != nullptr ? fast_exp2(sink - mm) : 0.f;
    for (int r = 0; r < S; ++r) {
      const float* t = cluster.map_shared_rank(top, r);
      const float mr = t[h], c = mr == -INFINITY ? 0.f : fast_exp2(mr - mm);
      o += cluster.map_shared_rank(sum, r)[i] * c;
      ll += t[HEADS + h] * c;
    }
    if (p.gate.p != nullptr && (p.gate.e == 0 || i % D < p.gate.e))
      o *= sigmoid_of(__bfloat162float(reinterpret_cast<const bf16*>(p.gate.p)[b * p.gate.ld + (p.gate.e == 0 ? h0 + h : (h0 + h) * p.gate.e + i % D)]));
    reinterpret_cast<bf16*>(p.out)[(static_cast<size_t>(b) * p.hq + h0) * D + i] = __float2bfloat16(ll > 0.f ? o / ll : 0.f);
  }
  if (S > 1) cluster.sync();                        // nobody leaves while its shared memory is read
}

// CTAs of a cluster.  Two CTAs fit an SM, and every CTA costs about 5 us of latency whatever its length, so the split ends where the chip is
// filled once: 16 sequences of 4–8 k tokens on 8 key heads take 106 / 75 / 78 / 84 us with 1 / 2 / 4 / 8 CTAs, 64 of 0.5–1 k 42 / 52 / 69 / 113, one of
// 16 k 130 / 95 / 43 / 25.  A table without room for a tile per warp is not split further.
static int cluster_size(const PagedDecode& p, int B, int groups) {
  const long room = static_cast<long>(p.max_blocks) * p.block_size / (pd::WARPS * pd::TILE), ctas = static_cast<long>(B) * p.hkv * groups;
  int S = 1;
  while (S < 8 && 4 * ctas * S < 7 * num_sms() && 2 * S <= room) S *= 2;
  return S;
}

template <int D>
static void launch(const PagedDecode& p, int B, cudaStream_t stream) {
  static OncePerDevice limit;
  limit(current_device(), [] { TK_CUDA_CHECK(cudaFuncSetAttribute(paged_decode_mma_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, pd::smem_bytes<D>())); });
  const int groups = (p.G + pd::HEADS - 1) / pd::HEADS, S = cluster_size(p, B, groups);
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(S, p.hkv * groups, B);
  cfg.blockDim = dim3(pd::WARPS * 32);
  cfg.dynamicSmemBytes = pd::smem_bytes<D>();
  cfg.stream = stream;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = S;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  TK_CUDA_CHECK(cudaLaunchKernelEx(&cfg, paged_decode_mma_kernel<D>, p));
}

bool paged_decode_mma(const PagedDecode& p, int B, int d, int e, cudaStream_t stream) {
  // cp.async and the query's pairs want the pools on 16-byte and the query on 4-byte boundaries
  const bool aligned = reinterpret_cast<uintptr_t>(p.kc) % 16 == 0 && reinterpret_cast<uintptr_t>(p.vc) % 16 == 0 && reinterpret_cast<uintptr_t>(p.q) % 4 == 0;
  // Groups of one to three heads stay with the vector kernel, which is the slower one there (16/8 heads, one sequence of 1 k tokens: 19.3 us against 6.3): the
  // decoders that have such groups are small and deep, and any other order of these sums moves the logits of a 28-layer stack by 2.7–3.8 %, at the same
  // distance from 64 bits (3.7–4.1 %).  perf/cases.py grants such stacks 3 %, so their steps keep the order that they had.
  if (!aligned || p.G < 4 || d != e || (d != 64 && d != 128) || B > 65535 || p.hkv * ((p.G + pd::HEADS - 1) / pd::HEADS) > 65535) return false;
  if (d == 64) launch<64>(p, B, stream); else launch<128>(p, B, stream);
  return true;
}

}  // namespace tk
