// Flash-attention backward for sm_100a (causal, GQA, packed varlen, D = 128), two tcgen05 kernels:
//
//   flash_bwd_dkdv_kernel : one CTA per (128-row K/V tile, kv head).  Loops over the query heads of the
//       GQA group and over 128-row query blocks:  Sᵀ = K·Qᵀ, dPᵀ = V·dOᵀ (tensor cores → TMEM),
//       Pᵀ = exp2(Sᵀ·c − lse), dSᵀ = Pᵀ∘(dPᵀ − δ) (registers → TMEM), dV += Pᵀ·dO, dK += dSᵀ·Q.
//       dK/dV of the whole group accumulate in TMEM → no atomics, deterministic.
//   flash_bwd_dq_kernel   : one CTA per (128-row query tile, query head).  Loops over 128-row K/V blocks:
//       S = Q·Kᵀ, dP = dO·Vᵀ, dS = P∘(dP − δ), dQ += dS·K.
//   flash_bwd_delta_kernel: δ[h,t] = Σ_d O·dO.
// Recomputing S/dP in both kernels costs 7 instead of 5 GEMMs per tile pair but keeps every
// accumulator on chip without cross-CTA reductions.
//
// What bounds them: the tensor cores, by products of 128x128x16 at 64 cycles.  (Blocks of 64 rows had products that take as long for half the
// work, and two barriers per block on the only path.)  P and dS go back into the TMEM columns of the scores they come from, as the A operand of the
// accumulating products, which leaves shared memory for two stages of 128-row blocks; each WG writes inside the columns that it alone
// reads.  Products that do not wait for the arithmetic in progress run under it: dV and the next Sᵀ while dSᵀ is formed, dK and the next
// dPᵀ while the next Pᵀ is; the next S and dP while dS is.  Products run over K in steps of 16 in the same order as with blocks of 64.
// 32768 tokens in documents of 0.5-8 k, 32/8 heads, us before → now (TFLOP/s of all products): dK/dV 6320 → 3360 (830), dQ 3990 → 2220 (940);
// 8 x 4096, 32/4 heads: 5040 → 2590, 3140 → 1730.
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <cooperative_groups.h>
#include <torch/types.h>

#include "common.cuh"
#include "elect.cuh"
#include "host.h"

namespace tk {

using bf16 = __nv_bfloat16;
CUtensorMap make_head_tmap(const torch::Tensor& t, int rows);

namespace fb {
constexpr int D = 128, BT = 128;              // width, rows of a tile and of a block
constexpr int TILE_BYTES = BT * D * 2;        // 32 KiB (two [128][64] atoms)
constexpr int ATOM = BT * 64 * 2;             // 16 KiB
constexpr int THREADS = 320;  // warps 0-7 compute (two groups of 4, each takes half of a block's columns), 8 producer, 9 MMA
// two tiles that stay (A, B), two streams of blocks in two stages each (X, Y), lse / δ of a block, barriers.  dK/dV: K, V | Q, dO; dQ: Q, dO | K, V
constexpr int SMEM_A = 0, SMEM_B = TILE_BYTES, SMEM_X = 2 * TILE_BYTES, SMEM_Y = SMEM_X + 2 * TILE_BYTES, SMEM_STAT = SMEM_Y + 2 * TILE_BYTES,
              SMEM_BAR = SMEM_STAT + 2 * 2 * BT * 4, SMEM_TOTAL = SMEM_BAR + 256 + 1024;
constexpr int SUM_PITCH = D + 4;              // floats between rows of a partial sum
static_assert(2 * BT * SUM_PITCH * 4 <= SMEM_STAT, "partial sums lie over the tiles");
__device__ __forceinline__ constexpr uint32_t step(int k) { return ((k >> 2) * ATOM + (k & 3) * 32) >> 4; }   // of a K-major operand, 16 along K, in a descriptor
}  // namespace fb

struct BwdParams {
  bf16 *dq, *dk, *dv;    // [T,Hq,D], [T,Hkv,D], [T,Hkv,D]
  const float* lse;      // [Hq,T] natural log
  const float* delta;    // [Hq,T]
  const int* cu;
  int T, hq, hkv;
  float scale, scale_log2;
  int causal;
  const int* cu_k;   // key/value boundaries (== cu for self-attention over the same packing)
  int* err;
};

__global__ void flash_bwd_delta_kernel(const bf16* __restrict__ o, const bf16* __restrict__ dout, float* __restrict__ delta, int T, int hq) {
  // one warp per (token, head); 128 elements → 4 per lane
  const long total = static_cast<long>(T) * hq;
  const int lane = threadIdx.x & 31;
  for (long item = static_cast<long>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5); item < total;
       item += static_cast<long>(gridDim.x) * (blockDim.x >> 5)) {
    const uint2 a = *reinterpret_cast<const uint2*>(o + item * 128 + lane * 4);
    const uint2 b = *reinterpret_cast<const uint2*>(dout + item * 128 + lane * 4);
    float2 a0 = unpack_bf16(a.x), a1 = unpack_bf16(a.y), b0 = unpack_bf16(b.x), b1 = unpack_bf16(b.y);
    float s = warp_sum(a0.x * b0.x + a0.y * b0.y + a1.x * b1.x + a1.y * b1.y);
    if (lane == 0) {
      const int t = static_cast<int>(item / hq), h = static_cast<int>(item % hq);
      delta[static_cast<size_t>(h) * T + t] = s;
    }
  }
}

// ============================================================== dK / dV
// SPLIT: a cluster of gridDim.x / hkv CTAs shares a tile by query heads and adds up through distributed shared memory.
template <bool SPLIT>
__global__ void __launch_bounds__(fb::THREADS, 1)
flash_bwd_dkdv_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                      const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmDO, const BwdParams p) {
  using namespace fb;
  namespace cg = cooperative_groups;
  const int parts = SPLIT ? gridDim.x / p.hkv : 1;
  const int kv_head = blockIdx.x / parts, rank = blockIdx.x % parts, seq = blockIdx.z;
  const int seq_start = p.cu[seq], seq_len = p.cu[seq + 1] - seq_start;          // queries
  const int kv_start = p.cu_k[seq], kv_len = p.cu_k[seq + 1] - kv_start;         // keys / values
  const int q_off = kv_len - seq_len;            // causal: query row r sees keys 0 … r + q_off
  const int n_tiles = (kv_len + BT - 1) / BT;
  if (static_cast<int>(blockIdx.y) >= n_tiles) return;
  const int kv0 = blockIdx.y * BT;               // early tiles have the most query blocks → scheduled first
  const int G = p.hq / p.hkv, heads = G / parts, head0 = kv_head * G + rank * heads;
  const int qb_end = (seq_len + BT - 1) / BT;
  const int qb_begin = p.causal ? min(max(kv0 - q_off, 0) / BT, qb_end) : 0;
  const int per_head = qb_end - qb_begin;
  const int n_iter = per_head * heads;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + SMEM_BAR);
  uint64_t* kv_full = bars;          // 1
  uint64_t* qdo_full = bars + 1;     // 2
  uint64_t* qdo_empty = bars + 3;    // 2
  uint64_t* s_full = bars + 5;
  uint64_t* dp_full = bars + 6;
  uint64_t* p_ready = bars + 7;
  uint64_t* ds_ready = bars + 8;
  uint64_t* acc_done = bars + 9;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 10);
  float* stat = reinterpret_cast<float*>(smem + SMEM_STAT);  // [2 buffers][lse2 | delta][128]

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    mbar_init(kv_full, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&qdo_full[i], 1);
      mbar_init(&qdo_empty[i], 1);
    }
    mbar_init(s_full, 1);
    mbar_init(dp_full, 1);
    mbar_init(p_ready, 256);
    mbar_init(ds_ready, 256);
    mbar_init(acc_done, 1);
    fence_barrier_init();
  }
  if (warp == 9) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(tmem_slot);
  // TMEM columns: Sᵀ [0,128), of which Pᵀ takes [0,32) and [64,96); dPᵀ [128,256), dSᵀ inside it likewise; dV [256,384); dK [384,512)
  const uint32_t t_s = tmem_base, t_dp = tmem_base + 128, t_dv = tmem_base + 256, t_dk = tmem_base + 384;

  if (warp == 8) {
    // producer warp: lane 0 drives TMA; all lanes stage lse (log2 units) and δ of each query block in smem
    if (lane == 0 && n_iter > 0) {     // a tile that no query sees loads nothing: nobody would wait for it
      mbar_expect_tx(kv_full, 2 * TILE_BYTES);
      tma_load_3d(smem + SMEM_A, &tmK, kv_full, 0, kv_head, kv_start + kv0);
      tma_load_3d(smem + SMEM_A + ATOM, &tmK, kv_full, 64, kv_head, kv_start + kv0);
      tma_load_3d(smem + SMEM_B, &tmV, kv_full, 0, kv_head, kv_start + kv0);
      tma_load_3d(smem + SMEM_B + ATOM, &tmV, kv_full, 64, kv_head, kv_start + kv0);
    }
    for (int it = 0; it < n_iter; ++it) {
      const int st = it & 1;
      if (it >= 2) {
        int ok = 1;
        if (lane == 0) ok = mbar_wait(&qdo_empty[st], ((it >> 1) - 1) & 1, p.err, ERR_ATTN_WAIT) ? 1 : 0;
        ok = __shfl_sync(0xffffffffu, ok, 0);
        if (!ok) break;
      }
      const int head = head0 + it / per_head;
      const int qb0 = (qb_begin + it % per_head) * BT;
#pragma unroll
      for (int c = lane; c < BT; c += 32) {
        const int qpos = qb0 + c;
        float l2 = INFINITY, dl = 0.f;   // exp2(s − inf) = 0 for query rows past the end of the sequence
        if (qpos < seq_len) {
          const size_t idx = static_cast<size_t>(head) * p.T + seq_start + qpos;
          l2 = p.lse[idx] * 1.4426950408889634f;
          dl = p.delta[idx];
        }
        stat[st * 2 * BT + c] = -l2;
        stat[st * 2 * BT + BT + c] = -dl;
      }
      __syncwarp();
      if (lane == 0) {
        const int row = seq_start + qb0;
        mbar_expect_tx(&qdo_full[st], 2 * TILE_BYTES);
        tma_load_3d(smem + SMEM_X + st * TILE_BYTES, &tmQ, &qdo_full[st], 0, head, row);
        tma_load_3d(smem + SMEM_X + st * TILE_BYTES + ATOM, &tmQ, &qdo_full[st], 64, head, row);
        tma_load_3d(smem + SMEM_Y + st * TILE_BYTES, &tmDO, &qdo_full[st], 0, head, row);
        tma_load_3d(smem + SMEM_Y + st * TILE_BYTES + ATOM, &tmDO, &qdo_full[st], 64, head, row);
      }
    }
  } else if (warp == 9) {
    // the whole warp walks the loop and one thread issues: descriptors stay in uniform registers
    constexpr uint32_t idesc_s = umma_idesc_bf16(BT, BT, false, false);   // [128 kv] x [128 q], K = d
    constexpr uint32_t idesc_acc = umma_idesc_bf16(BT, D, false, true);   // [128 kv] x [128 d], K = q (B MN-major)
    const uint64_t dK = umma_desc(smem_u32(smem + SMEM_A), 16, 1024), dV = umma_desc(smem_u32(smem + SMEM_B), 16, 1024);
    auto wait = [&](uint64_t* bar, uint32_t parity) { return __all_sync(0xffffffffu, mbar_wait(bar, parity, p.err, ERR_ATTN_WAIT)); };
    auto scores = [&](uint32_t d, uint64_t a, int at, uint64_t* bar) {       // d = a · (tile at `at`)ᵀ
      const uint64_t b = umma_desc(smem_u32(smem + at), 16, 1024);
      if (elect_one()) {
#pragma unroll
        for (int k = 0; k < D / 16; ++k) umma_bf16(d, a + step(k), b + step(k), idesc_s, k ? 1u : 0u);
        umma_commit(bar);
      }
      __syncwarp();
    };
    auto add_up = [&](uint32_t d, uint32_t a, int at, bool first, uint64_t* bar) {      // d += a (tensor memory) · tile
      const uint64_t b = umma_desc(smem_u32(smem + at), ATOM, 1024);
      if (elect_one()) {
        const uint32_t add = !first;
#pragma unroll
        for (int k = 0; k < BT / 16; ++k) umma_bf16_ts(d, a + (k >> 2) * 64 + (k & 3) * 8, b + k * 128, idesc_acc, k > 0 ? 1u : add);
        if (bar != nullptr) umma_commit(bar);
      }
      __syncwarp();
    };
    bool ok = n_iter > 0 && wait(kv_full, 0) && wait(&qdo_full[0], 0);
    if (ok) {
      tc_fence_after();
      scores(t_s, dK, SMEM_X, s_full);
      scores(t_dp, dV, SMEM_Y, dp_full);
    }
    for (int it = 0; ok && it < n_iter; ++it) {
      const int st = it & 1, nx = st ^ 1;
      const bool more = it + 1 < n_iter;
      if (!wait(p_ready, it & 1)) break;
      tc_fence_after();
      add_up(t_dv, t_s, SMEM_Y + st * TILE_BYTES, it == 0, nullptr);            // dV += Pᵀ·dO
      if (more) {
        if (!wait(&qdo_full[nx], ((it + 1) >> 1) & 1)) break;
        tc_fence_after();
        scores(t_s, dK, SMEM_X + nx * TILE_BYTES, s_full);                       // runs after the product that reads Pᵀ
      }
      if (!wait(ds_ready, it & 1)) break;
      tc_fence_after();
      add_up(t_dk, t_dp, SMEM_X + st * TILE_BYTES, it == 0, &qdo_empty[st]);    // dK += dSᵀ·Q
      if (more) scores(t_dp, dV, SMEM_Y + nx * TILE_BYTES, dp_full);
    }
    if (n_iter > 0 && elect_one()) umma_commit(acc_done);
    __syncwarp();
  }
  bool ok = true;
  const int wg = warp >> 2;                       // which half of the 128 queries of a block this thread handles
  const int row = (warp & 3) * 32 + lane;
  const uint32_t lane_off = static_cast<uint32_t>((warp & 3) * 32) << 16;
  const int kv_pos = kv0 + row;
  const bool row_valid = kv_pos < kv_len;
  if (warp < 8) {
    const float2 scale2 = make_float2(p.scale_log2, p.scale_log2);
    for (int it = 0; it < n_iter; ++it) {
      const int qb0 = (qb_begin + it % per_head) * BT + wg * 64;
      const float* lse2 = stat + (it & 1) * 2 * BT + wg * 64;       // negated, as is δ
      const float* dl = lse2 + BT;
      if (!mbar_wait(s_full, it & 1, p.err, ERR_ATTN_WAIT)) { ok = false; break; }
      tc_fence_after();
      // only blocks that touch the causal diagonal need per-element masking; rows past the end of the keys are
      // zeroed wholesale; query rows past the end carry lse = +inf and vanish through exp2
      const bool diag = p.causal && (qb0 + q_off < kv0 + BT - 1);
      float pr[64];
      uint32_t pk[32];
#pragma unroll
      for (int c = 0; c < 64; c += 32) {
        uint32_t s[32];
        tmem_ld32(t_s + wg * 64 + c + lane_off, s);
        tmem_ld_wait();
        const float4* l4 = reinterpret_cast<const float4*>(lse2 + c);
#pragma unroll
        for (int i = 0; i < 32; i += 4) {
          const float4 l = l4[i >> 2];
          const float2 x = fma2(make_float2(__uint_as_float(s[i]), __uint_as_float(s[i + 1])), scale2, make_float2(l.x, l.y));
          const float2 y = fma2(make_float2(__uint_as_float(s[i + 2]), __uint_as_float(s[i + 3])), scale2, make_float2(l.z, l.w));
          pr[c + i] = fast_exp2(x.x);
          pr[c + i + 1] = fast_exp2(x.y);
          pr[c + i + 2] = fast_exp2(y.x);
          pr[c + i + 3] = fast_exp2(y.y);
        }
      }
      if (diag) {
        const int gone = kv_pos - q_off - qb0;      // queries before this one of the half do not see the key
#pragma unroll
        for (int i = 0; i < 64; ++i)
          if (i < gone) pr[i] = 0.f;
      }
      if (!row_valid) {
#pragma unroll
        for (int i = 0; i < 64; ++i) pr[i] = 0.f;
      }
#pragma unroll
      for (int i = 0; i < 32; ++i) pk[i] = pack_bf16(pr[2 * i], pr[2 * i + 1]);
      tmem_st32(t_s + wg * 64 + lane_off, pk);
      tmem_st_wait();
      tc_fence_before();
      mbar_arrive(p_ready);
      if (!mbar_wait(dp_full, it & 1, p.err, ERR_ATTN_WAIT)) { ok = false; break; }
      tc_fence_after();
#pragma unroll
      for (int c = 0; c < 64; c += 32) {
        uint32_t dp[32];
        tmem_ld32(t_dp + wg * 64 + c + lane_off, dp);
        tmem_ld_wait();
        const float4* d4 = reinterpret_cast<const float4*>(dl + c);
#pragma unroll
        for (int i = 0; i < 32; i += 4) {
          const float4 d = d4[i >> 2];
          const float2 x = mul2(make_float2(pr[c + i], pr[c + i + 1]), add2(make_float2(__uint_as_float(dp[i]), __uint_as_float(dp[i + 1])), make_float2(d.x, d.y)));
          const float2 y = mul2(make_float2(pr[c + i + 2], pr[c + i + 3]), add2(make_float2(__uint_as_float(dp[i + 2]), __uint_as_float(dp[i + 3])), make_float2(d.z, d.w)));
          pk[(c + i) >> 1] = pack_bf16(x.x, x.y);
          pk[((c + i) >> 1) + 1] = pack_bf16(y.x, y.y);
        }
      }
      if (!row_valid) {
#pragma unroll
        for (int i = 0; i < 32; ++i) pk[i] = 0u;
      }
      tmem_st32(t_dp + wg * 64 + lane_off, pk);
      tmem_st_wait();
      tc_fence_before();
      mbar_arrive(ds_ready);
    }
    if (n_iter > 0) ok = ok && mbar_wait(acc_done, 0, p.err, ERR_ATTN_WAIT);
    tc_fence_after();
    bf16* dkrow = p.dk + (static_cast<size_t>(kv_start + kv_pos) * p.hkv + kv_head) * D;
    bf16* dvrow = p.dv + (static_cast<size_t>(kv_start + kv_pos) * p.hkv + kv_head) * D;
    if (ok && n_iter > 0) {
#pragma unroll 1
      for (int c = 2 * wg; c < 2 * wg + 2; ++c) {
        uint32_t a[32], b[32];
        tmem_ld32(t_dv + lane_off + c * 32, a);
        tmem_ld32(t_dk + lane_off + c * 32, b);
        tmem_ld_wait();
        if constexpr (SPLIT) {        // the tiles are read for the last time: their place takes the sums, dV then dK
          float* mine = reinterpret_cast<float*>(smem) + row * SUM_PITCH + c * 32;
#pragma unroll
          for (int i = 0; i < 32; i += 4) {
            *reinterpret_cast<uint4*>(mine + i) = make_uint4(a[i], a[i + 1], a[i + 2], a[i + 3]);
            *reinterpret_cast<uint4*>(mine + BT * SUM_PITCH + i) = make_uint4(b[i], b[i + 1], b[i + 2], b[i + 3]);
          }
        } else if (row_valid) {
#pragma unroll
          for (int i = 0; i < 32; i += 8) {
            *reinterpret_cast<uint4*>(dvrow + c * 32 + i) =
                make_uint4(pack_bf16(__uint_as_float(a[i]), __uint_as_float(a[i + 1])), pack_bf16(__uint_as_float(a[i + 2]), __uint_as_float(a[i + 3])),
                           pack_bf16(__uint_as_float(a[i + 4]), __uint_as_float(a[i + 5])), pack_bf16(__uint_as_float(a[i + 6]), __uint_as_float(a[i + 7])));
            *reinterpret_cast<uint4*>(dkrow + c * 32 + i) =
                make_uint4(pack_bf16(__uint_as_float(b[i]) * p.scale, __uint_as_float(b[i + 1]) * p.scale),
                           pack_bf16(__uint_as_float(b[i + 2]) * p.scale, __uint_as_float(b[i + 3]) * p.scale),
                           pack_bf16(__uint_as_float(b[i + 4]) * p.scale, __uint_as_float(b[i + 5]) * p.scale),
                           pack_bf16(__uint_as_float(b[i + 6]) * p.scale, __uint_as_float(b[i + 7]) * p.scale));
          }
        }
      }
    } else if (n_iter == 0 && row_valid && rank == 0) {
      // no query sees this tile (keys of a sequence without queries, or all of them behind every query)
      for (int i = wg * 64; i < wg * 64 + 64; i += 8) {
        *reinterpret_cast<uint4*>(dkrow + i) = make_uint4(0, 0, 0, 0);
        *reinterpret_cast<uint4*>(dvrow + i) = make_uint4(0, 0, 0, 0);
      }
    }
  }
  if constexpr (SPLIT) {
    const cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();
    if (n_iter > 0) {
      const float* sums = reinterpret_cast<const float*>(smem);
      for (int i = rank * THREADS + threadIdx.x; i < 2 * BT * (D / 4); i += parts * THREADS) {
        const int which = i / (BT * (D / 4)), r = i / (D / 4) % BT, c = i % (D / 4) * 4;
        if (kv0 + r >= kv_len) continue;
        float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int k = 0; k < parts; ++k) {
          const float4 v = *reinterpret_cast<const float4*>(cluster.map_shared_rank(sums, k) + (which * BT + r) * SUM_PITCH + c);
          s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
        }
        const float f = which ? p.scale : 1.f;
        *reinterpret_cast<uint2*>((which ? p.dk : p.dv) + (static_cast<size_t>(kv_start + kv0 + r) * p.hkv + kv_head) * D + c) = make_uint2(pack_bf16(s.x * f, s.y * f), pack_bf16(s.z * f, s.w * f));
      }
    }
    cluster.sync();
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 9) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// ==================================================================== dQ
__global__ void __launch_bounds__(fb::THREADS, 1)
flash_bwd_dq_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                    const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmDO, const BwdParams p) {
  using namespace fb;
  const int head = blockIdx.x, seq = blockIdx.z;
  const int seq_start = p.cu[seq], seq_len = p.cu[seq + 1] - seq_start;
  const int n_tiles = (seq_len + BT - 1) / BT;
  if (static_cast<int>(blockIdx.y) >= n_tiles) return;
  const int q0 = (n_tiles - 1 - blockIdx.y) * BT;
  const int kv_head = head / (p.hq / p.hkv);
  const int kv_start = p.cu_k[seq], kv_len = p.cu_k[seq + 1] - kv_start;
  const int q_off = kv_len - seq_len;
  const int kv_end = p.causal ? max(0, min(kv_len, q0 + BT + q_off)) : kv_len;
  const int n_iter = (kv_end + BT - 1) / BT;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + SMEM_BAR);
  uint64_t* qdo_full = bars;         // 1
  uint64_t* kv_full = bars + 1;      // 2
  uint64_t* kv_empty = bars + 3;     // 2
  uint64_t* sd_full = bars + 5;
  uint64_t* dp_empty = bars + 6;
  uint64_t* ds_ready = bars + 7;     // 2
  uint64_t* acc_done = bars + 9;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 10);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    mbar_init(qdo_full, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&kv_full[i], 1);
      mbar_init(&kv_empty[i], 1);
      mbar_init(&ds_ready[i], 256);
    }
    mbar_init(sd_full, 1);
    mbar_init(dp_empty, 256);
    mbar_init(acc_done, 1);
    fence_barrier_init();
  }
  if (warp == 9) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(tmem_slot);
  // TMEM columns: S in two buffers [0,128) [128,256), of which dS takes [0,32) and [64,96); dP [256,384); dQ [384,512)
  const uint32_t t_dp = tmem_base + 256, t_dq = tmem_base + 384;

  if (warp == 8) {
    if (lane == 0 && n_iter > 0) {
      mbar_expect_tx(qdo_full, 2 * TILE_BYTES);
      tma_load_3d(smem + SMEM_A, &tmQ, qdo_full, 0, head, seq_start + q0);
      tma_load_3d(smem + SMEM_A + ATOM, &tmQ, qdo_full, 64, head, seq_start + q0);
      tma_load_3d(smem + SMEM_B, &tmDO, qdo_full, 0, head, seq_start + q0);
      tma_load_3d(smem + SMEM_B + ATOM, &tmDO, qdo_full, 64, head, seq_start + q0);
      for (int it = 0; it < n_iter; ++it) {
        const int st = it & 1;
        if (it >= 2 && !mbar_wait(&kv_empty[st], ((it >> 1) - 1) & 1, p.err, ERR_ATTN_WAIT)) break;
        const int row = kv_start + it * BT;
        mbar_expect_tx(&kv_full[st], 2 * TILE_BYTES);
        tma_load_3d(smem + SMEM_X + st * TILE_BYTES, &tmK, &kv_full[st], 0, kv_head, row);
        tma_load_3d(smem + SMEM_X + st * TILE_BYTES + ATOM, &tmK, &kv_full[st], 64, kv_head, row);
        tma_load_3d(smem + SMEM_Y + st * TILE_BYTES, &tmV, &kv_full[st], 0, kv_head, row);
        tma_load_3d(smem + SMEM_Y + st * TILE_BYTES + ATOM, &tmV, &kv_full[st], 64, kv_head, row);
      }
    }
  } else if (warp == 9) {
    constexpr uint32_t idesc_s = umma_idesc_bf16(BT, BT, false, false);   // [128 q] x [128 kv], K = d
    constexpr uint32_t idesc_acc = umma_idesc_bf16(BT, D, false, true);   // [128 q] x [128 d], K = kv (B MN-major)
    const uint64_t dQ = umma_desc(smem_u32(smem + SMEM_A), 16, 1024), dO = umma_desc(smem_u32(smem + SMEM_B), 16, 1024);
    auto wait = [&](uint64_t* bar, uint32_t parity) { return __all_sync(0xffffffffu, mbar_wait(bar, parity, p.err, ERR_ATTN_WAIT)); };
    auto scores = [&](uint32_t d, uint64_t a, int at, uint64_t* bar) {
      const uint64_t b = umma_desc(smem_u32(smem + at), 16, 1024);
      if (elect_one()) {
#pragma unroll
        for (int k = 0; k < D / 16; ++k) umma_bf16(d, a + step(k), b + step(k), idesc_s, k ? 1u : 0u);
        if (bar != nullptr) umma_commit(bar);
      }
      __syncwarp();
    };
    bool ok = n_iter > 0 && wait(qdo_full, 0) && wait(&kv_full[0], 0);
    if (ok) {
      tc_fence_after();
      scores(tmem_base, dQ, SMEM_X, nullptr);
      scores(t_dp, dO, SMEM_Y, sd_full);
    }
    for (int it = 0; ok && it < n_iter; ++it) {
      if (it + 1 < n_iter) {
        const int nx = (it + 1) & 1;
        if (!wait(&kv_full[nx], ((it + 1) >> 1) & 1)) break;
        tc_fence_after();
        scores(tmem_base + nx * 128, dQ, SMEM_X + nx * TILE_BYTES, nullptr);     // its buffer's dS was read by the product before
        if (!wait(dp_empty, it & 1)) break;
        tc_fence_after();
        scores(t_dp, dO, SMEM_Y + nx * TILE_BYTES, sd_full);
      }
      if (!wait(&ds_ready[it & 1], (it >> 1) & 1)) break;
      tc_fence_after();
      const uint64_t k_ = umma_desc(smem_u32(smem + SMEM_X + (it & 1) * TILE_BYTES), ATOM, 1024);
      if (elect_one()) {
        const uint32_t add = it > 0;
#pragma unroll
        for (int k = 0; k < BT / 16; ++k)   // dQ += dS·K
          umma_bf16_ts(t_dq, tmem_base + (it & 1) * 128 + (k >> 2) * 64 + (k & 3) * 8, k_ + k * 128, idesc_acc, k > 0 ? 1u : add);
        umma_commit(&kv_empty[it & 1]);
      }
      __syncwarp();
    }
    if (n_iter > 0 && elect_one()) umma_commit(acc_done);
    __syncwarp();
  } else {
    const int wg = warp >> 2;
    const int row = (warp & 3) * 32 + lane;
    const uint32_t lane_off = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const int q_pos = q0 + row;
    const bool row_valid = q_pos < seq_len;
    float lse2 = INFINITY, dl = 0.f;
    if (row_valid) {
      const size_t idx = static_cast<size_t>(head) * p.T + seq_start + q_pos;
      lse2 = p.lse[idx] * 1.4426950408889634f;
      dl = p.delta[idx];
    }
    const float2 scale2 = make_float2(p.scale_log2, p.scale_log2), lse_2 = make_float2(-lse2, -lse2), dl_2 = make_float2(-dl, -dl);
    bool ok = true;
    for (int it = 0; it < n_iter; ++it) {
      if (!mbar_wait(sd_full, it & 1, p.err, ERR_ATTN_WAIT)) { ok = false; break; }
      tc_fence_after();
      const int kvb = it * BT + wg * 64;
      const uint32_t t_s = tmem_base + (it & 1) * 128 + wg * 64 + lane_off;
      uint32_t dp[64], pk[32];
      tmem_ld32(t_dp + wg * 64 + lane_off, *reinterpret_cast<uint32_t(*)[32]>(dp));
      tmem_ld32(t_dp + wg * 64 + 32 + lane_off, *reinterpret_cast<uint32_t(*)[32]>(dp + 32));
      tmem_ld_wait();
      tc_fence_before();
      mbar_arrive(dp_empty);             // the next dP may be formed
      // masking is needed only where the block crosses the causal diagonal of this query tile or the end of the keys
      const bool edge = (kvb + 64 > kv_len) || (p.causal && kvb + 63 > q0 + q_off);
      const int last = p.causal ? min(kv_len - 1, q_pos + q_off) - kvb : kv_len - 1 - kvb;      // last visible key of the half
#pragma unroll
      for (int c = 0; c < 64; c += 32) {
        uint32_t s[32];
        tmem_ld32(t_s + c, s);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          const float2 x = fma2(make_float2(__uint_as_float(s[i]), __uint_as_float(s[i + 1])), scale2, lse_2);
          float2 pr = make_float2(fast_exp2(x.x), fast_exp2(x.y));
          if (edge) {
            if (c + i > last) pr.x = 0.f;
            if (c + i + 1 > last) pr.y = 0.f;
          }
          const float2 d = mul2(pr, add2(make_float2(__uint_as_float(dp[c + i]), __uint_as_float(dp[c + i + 1])), dl_2));
          pk[(c + i) >> 1] = pack_bf16(d.x, d.y);
        }
      }
      tmem_st32(t_s, pk);
      tmem_st_wait();
      tc_fence_before();
      mbar_arrive(&ds_ready[it & 1]);
    }
    bf16* dqrow = p.dq + (static_cast<size_t>(seq_start + q_pos) * p.hq + head) * D;
    if (ok && n_iter > 0 && mbar_wait(acc_done, 0, p.err, ERR_ATTN_WAIT)) {
      tc_fence_after();
#pragma unroll 1
      for (int c = 2 * wg; c < 2 * wg + 2; ++c) {
        uint32_t a[32];
        tmem_ld32(t_dq + lane_off + c * 32, a);
        tmem_ld_wait();
        if (row_valid) {
#pragma unroll
          for (int i = 0; i < 32; i += 8)
            *reinterpret_cast<uint4*>(dqrow + c * 32 + i) =
                make_uint4(pack_bf16(__uint_as_float(a[i]) * p.scale, __uint_as_float(a[i + 1]) * p.scale),
                           pack_bf16(__uint_as_float(a[i + 2]) * p.scale, __uint_as_float(a[i + 3]) * p.scale),
                           pack_bf16(__uint_as_float(a[i + 4]) * p.scale, __uint_as_float(a[i + 5]) * p.scale),
                           pack_bf16(__uint_as_float(a[i + 6]) * p.scale, __uint_as_float(a[i + 7]) * p.scale));
        }
      }
    } else if (n_iter == 0 && row_valid) {          // queries before all keys
      for (int i = wg * 64; i < wg * 64 + 64; i += 8) *reinterpret_cast<uint4*>(dqrow + i) = make_uint4(0u, 0u, 0u, 0u);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 9) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

std::vector<torch::Tensor> flash_attn_bwd(const torch::Tensor& dout, const torch::Tensor& q, const torch::Tensor& k, const torch::Tensor& v,
                                          const torch::Tensor& out, const torch::Tensor& lse, const torch::Tensor& cu, int64_t max_seqlen,
                                          bool causal, double scale, const c10::optional<torch::Tensor>& cu_k, int64_t max_seqlen_k) {
  TORCH_CHECK(dout.is_contiguous() && q.is_contiguous() && k.is_contiguous() && v.is_contiguous() && out.is_contiguous(), "contiguous inputs");
  TORCH_CHECK(dout.scalar_type() == torch::kBFloat16 && dout.sizes() == q.sizes(), "dout like q");
  c10::cuda::CUDAGuard guard(q.device());
  const int T = q.size(0), hq = q.size(1), hkv = k.size(1), nseq = cu.numel() - 1;
  auto dq = torch::empty_like(q), dk = torch::empty_like(k), dv = torch::empty_like(v);
  if (T == 0 || nseq <= 0) return {dq, dk, dv};
  auto stream = at::cuda::getCurrentCUDAStream();
  auto delta = torch::empty({hq, T}, q.options().dtype(torch::kFloat32));
  {
    long items = static_cast<long>(T) * hq;
    int blocks = static_cast<int>(std::min<long>((items + 7) / 8, num_sms() * 16L));
    flash_bwd_delta_kernel<<<blocks, 256, 0, stream>>>(reinterpret_cast<const bf16*>(out.data_ptr()), reinterpret_cast<const bf16*>(dout.data_ptr()),
                                                       delta.data_ptr<float>(), T, hq);
  }
  BwdParams p{};
  p.dq = reinterpret_cast<bf16*>(dq.data_ptr()); p.dk = reinterpret_cast<bf16*>(dk.data_ptr()); p.dv = reinterpret_cast<bf16*>(dv.data_ptr());
  p.lse = lse.data_ptr<float>(); p.delta = delta.data_ptr<float>(); p.cu = cu.data_ptr<int>();
  p.T = T; p.hq = hq; p.hkv = hkv; p.scale = static_cast<float>(scale); p.scale_log2 = static_cast<float>(scale * 1.4426950408889634);
  p.causal = causal; p.err = error_word();
  p.cu_k = p.cu;
  if (cu_k.has_value() && cu_k->defined()) {
    TORCH_CHECK(cu_k->is_cuda() && cu_k->scalar_type() == torch::kInt32 && cu_k->is_contiguous() && cu_k->numel() == cu.numel(), "cu_k like cu");
    p.cu_k = cu_k->data_ptr<int>();
  }
  static OncePerDevice limit;
  limit(current_device(), [] {
    TK_CUDA_CHECK(cudaFuncSetAttribute(flash_bwd_dkdv_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, fb::SMEM_TOTAL));
    TK_CUDA_CHECK(cudaFuncSetAttribute(flash_bwd_dkdv_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, fb::SMEM_TOTAL));
    TK_CUDA_CHECK(cudaFuncSetAttribute(flash_bwd_dq_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, fb::SMEM_TOTAL));
  });
  const int tiles = (static_cast<int>(max_seqlen) + fb::BT - 1) / fb::BT;
  const int tiles_k = (static_cast<int>(max_seqlen_k > 0 ? max_seqlen_k : max_seqlen) + fb::BT - 1) / fb::BT;
  CUtensorMap tq = make_head_tmap(q, fb::BT), tdo = make_head_tmap(dout, fb::BT), tk_ = make_head_tmap(k, fb::BT), tv = make_head_tmap(v, fb::BT);
  // Where the tiles leave half of the SMs idle, the query heads of a group are shared out over a cluster, as many parts as fit at once (documents of 700
  // and 324 tokens, 32/8 heads, 72 tiles: 111 us before, 45 with two parts).
  int parts = 1;
  const int G = hq / hkv, rows = (static_cast<int>(k.size(0)) + fb::BT - 1) / fb::BT + nseq - 1;      // tiles of all sequences, at most
  while (parts < 4 && G % (2 * parts) == 0 && 2 * parts * hkv * std::min(rows, tiles_k * nseq) <= num_sms()) parts *= 2;
  if (parts == 1) {
    flash_bwd_dkdv_kernel<false><<<dim3(hkv, tiles_k, nseq), fb::THREADS, fb::SMEM_TOTAL, stream>>>(tq, tk_, tv, tdo, p);
  } else {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(hkv * parts, tiles_k, nseq);
    cfg.blockDim = dim3(fb::THREADS);
    cfg.dynamicSmemBytes = fb::SMEM_TOTAL;
    cfg.stream = stream;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = parts;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    TK_CUDA_CHECK(cudaLaunchKernelEx(&cfg, flash_bwd_dkdv_kernel<true>, tq, tk_, tv, tdo, p));
  }
  flash_bwd_dq_kernel<<<dim3(hq, tiles, nseq), fb::THREADS, fb::SMEM_TOTAL, stream>>>(tq, tk_, tv, tdo, p);
  count_launch(3);
  TK_CUDA_CHECK(cudaGetLastError());
  return {dq, dk, dv};
}

}  // namespace tk
