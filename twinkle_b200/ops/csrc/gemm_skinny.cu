// y = x Wᵀ for few rows (a decode step, a short prompt): the weight is read once and nothing else matters.
//
// The 128x256 tiles of gemm.cu give N / 256 CTAs there: 16 of 148 SMs for a 4096-wide output, 4 for a 1024-wide one, and a 256-row pair tile for 64
// rows.  Here a CTA takes one 128-row tile of x (only its live rows are loaded) and BN weight rows, BN any multiple of 16, and a cluster of S CTAs
// may share a tile by parts of K, added up in rank order through distributed shared memory.  A stage is one TMA load of x and one of W, each KA
// 64-wide swizzle atoms deep (a 3-D map {64, rows, K/64}), the stages fill shared memory, and one tile per CTA leaves nothing to schedule.
// Products run over K in the same steps of 16 as in gemm.cu, so results without a split are the same to the bit; a split in two, which follows the number of rows, halves
// the distance from 64 bits (K = 12288: 1.4e-5 → 6.8e-6).
//
// What bounds it: memory for wide weights (1 x 24576 x 4096: 53 → 36 us at a floor of 31), the issue of products, 35 ns each, for small ones.
// us before → now: 64 rows, N x K 6144 x 4096 30 → 16, 4096 x 4096 29 → 14, 4096 x 12288 76 → 26, 24576 x 4096 53 → 38; 1 row, 1024 x 3072
// 14 → 9.7, 4096 x 12288 76 → 23; 448 rows, 1024 x 2048 16 → 9.
#include <ATen/cuda/CUDAContext.h>
#include <cooperative_groups.h>
#include <torch/types.h>

#include <algorithm>

#include "common.cuh"
#include "elect.cuh"
#include "host.h"
#include "ring.h"

namespace tk {

namespace gs {
constexpr int BM = 128, ATOM = 64, ATOM_ROW = ATOM * 2, MAX_STAGES = 16, THREADS = 192;
constexpr int PAD = 4;                       // floats between rows of a partial sum
}  // namespace gs

struct SkinnyParams {
  void* out;
  int M, N, ldo, out_fp32, accumulate;
  int rows, bn, k_atoms, stages, split;      // live rows of an x tile (multiple of 8), weight rows, atoms of K
  int tmem_cols;
  int* err;
};

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
                 "=r"(r[14]), "=r"(r[15])
               : "r"(taddr)
               : "memory");
}

template <int KA>
__global__ void __launch_bounds__(gs::THREADS) gemm_skinny_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const SkinnyParams p) {
  using namespace gs;
  namespace cg = cooperative_groups;
  const cg::cluster_group cluster = cg::this_cluster();
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem);
  uint64_t* empty = full + MAX_STAGES;
  uint64_t* done = empty + MAX_STAGES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
  uint8_t* ring = smem + 1024;
  const int rank = p.split > 1 ? blockIdx.x % p.split : 0, n0 = (blockIdx.x / p.split) * p.bn, m0 = blockIdx.y * BM;
  const int a_bytes = p.rows * ATOM_ROW * KA, stage_bytes = a_bytes + p.bn * ATOM_ROW * KA;
  const int steps = (p.k_atoms + KA - 1) / KA, s0 = steps * rank / p.split, s1 = steps * (rank + 1) / p.split;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(done, 1);
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, p.tmem_cols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(tmem_slot);
  if (warp == 0) {
    if (lane == 0) {
      int st = 0, ph = 0;
      for (int s = s0; s < s1; ++s) {
        if (!mbar_wait(&empty[st], ph ^ 1, p.err, ERR_PRODUCER_WAIT)) {
          for (int i = ring_first_open(s - s0, p.stages); i < s - s0; ++i) {     // copies in flight land, within the limit, before the CTA exits
            const RingFill f = ring_fill(i, p.stages);
            mbar_wait(&full[f.stage], f.parity, nullptr, 0);
          }
          break;
        }
        mbar_expect_tx(&full[st], stage_bytes);     // atoms past K and rows past the tensors arrive as zeros
        tma_load_3d(ring + st * stage_bytes + a_bytes, &tmB, &full[st], 0, n0, s * KA);
        tma_load_3d(ring + st * stage_bytes, &tmA, &full[st], 0, m0, s * KA);
        if (++st == p.stages) { st = 0; ph ^= 1; }
      }
    }
  } else if (warp == 1) {
    // the whole warp walks the loop and one thread issues, unrolled: descriptors stay in uniform registers (58 → 35 ns per product)
    const uint32_t idesc = umma_idesc_bf16(BM, p.bn, false, false);
    const uint32_t step_a = p.rows * (ATOM_ROW / 16), step_b = p.bn * (ATOM_ROW / 16);       // addresses in a descriptor count 16 bytes
    int st = 0, ph = 0;
    for (int s = s0; s < s1; ++s) {
      if (!__all_sync(0xffffffffu, mbar_wait(&full[st], ph, p.err, ERR_MMA_WAIT_FULL))) break;
      tc_fence_after();
      // rows of x beyond the live ones are whatever lies behind them in the ring: they only reach accumulator rows that nobody stores
      uint64_t da = umma_desc(smem_u32(ring + st * stage_bytes), 16, 1024), db = umma_desc(smem_u32(ring + st * stage_bytes + a_bytes), 16, 1024);
      if (elect_one()) {
#pragma unroll
        for (int a = 0; a < KA; ++a) {
#pragma unroll
          for (int k = 0; k < ATOM / 16; ++k) umma_bf16(tmem, da + 2 * k, db + 2 * k, idesc, a + k == 0 ? s > s0 : 1u);
          da += step_a;
          db += step_b;
        }
        umma_commit(&empty[st]);
      }
      __syncwarp();
      if (++st == p.stages) { st = 0; ph ^= 1; }
    }
    if (elect_one()) umma_commit(done);
  }
  __syncwarp();
  const bool live = warp >= 2 && mbar_wait(done, 0, p.err, ERR_EPI_WAIT);
  const int q = warp & 3, row = q * 32 + lane, m = m0 + row;
  float* part = reinterpret_cast<float*>(ring);
  const int pitch = p.bn + PAD;
  if (live && q * 32 < p.rows) {
    tc_fence_after();
    for (int c = 0; c < p.bn; c += 16) {
      uint32_t r[16];
      tmem_ld16(tmem + c + (static_cast<uint32_t>(q * 32) << 16), r);
      tmem_ld_wait();
      if (p.split > 1) {
        if (row < p.rows) {
#pragma unroll
          for (int j = 0; j < 16; j += 4) *reinterpret_cast<uint4*>(part + row * pitch + c + j) = make_uint4(r[j], r[j + 1], r[j + 2], r[j + 3]);
        }
        continue;
      }
      if (m >= p.M) continue;
#pragma unroll
      for (int j = 0; j < 16; j += 8) {
        const int n = n0 + c + j;
        if (n >= p.N) break;
        float f[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) f[e] = __uint_as_float(r[j + e]);
        if (p.out_fp32) {
          float* o = reinterpret_cast<float*>(p.out) + static_cast<size_t>(m) * p.ldo + n;
          for (int e = 0; e < 8 && n + e < p.N; ++e) o[e] = f[e] + (p.accumulate ? o[e] : 0.f);
        } else {
          __nv_bfloat16* o = reinterpret_cast<__nv_bfloat16*>(p.out) + static_cast<size_t>(m) * p.ldo + n;
          if (n + 8 <= p.N && !p.accumulate) {
            *reinterpret_cast<uint4*>(o) = make_uint4(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]), pack_bf16(f[4], f[5]), pack_bf16(f[6], f[7]));
          } else {
            for (int e = 0; e < 8 && n + e < p.N; ++e) o[e] = __float2bfloat16(f[e] + (p.accumulate ? __bfloat162float(o[e]) : 0.f));
          }
        }
      }
    }
  }
  if (p.split > 1) {
    // the ring is free (the products that read it have retired before anyone writes over it); each CTA of the cluster adds up its share of the tile
    cluster.sync();
    const int rows = min(p.rows, p.M - m0), cols = min(p.bn, p.N - n0), quads = (cols + 3) / 4, items = rows * quads;
    for (int i = rank * THREADS + threadIdx.x; i < items; i += p.split * THREADS) {
      const int r = i / quads, c = i % quads * 4;
      float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
      for (int k = 0; k < p.split; ++k) {
        const float4 v = *reinterpret_cast<const float4*>(cluster.map_shared_rank(part, k) + r * pitch + c);
        s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
      }
      const float f[4] = {s.x, s.y, s.z, s.w};
      const size_t at = static_cast<size_t>(m0 + r) * p.ldo + n0 + c;
      if (p.out_fp32) {
        float* o = reinterpret_cast<float*>(p.out) + at;
        for (int e = 0; e < 4 && c + e < cols; ++e) o[e] = f[e] + (p.accumulate ? o[e] : 0.f);
      } else {
        __nv_bfloat16* o = reinterpret_cast<__nv_bfloat16*>(p.out) + at;
        if (c + 4 <= cols && !p.accumulate) {
          *reinterpret_cast<uint2*>(o) = make_uint2(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]));
        } else {
          for (int e = 0; e < 4 && c + e < cols; ++e) o[e] = __float2bfloat16(f[e] + (p.accumulate ? __bfloat162float(o[e]) : 0.f));
        }
      }
    }
    cluster.sync();
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, p.tmem_cols);
  }
}

// Few rows: up to one tile of them whatever the width (64 x 24576 x 4096: 38 us, 53 in pair tiles), and beyond that where pair tiles would occupy less than the
// chip, or 128x256 tiles less than one wave of it (256 x 4096 x 4096: 16 us, 30 in 128x256 tiles).  At the line both are equal (1024 rows, N x K 4096 x 1024 12.8 us against 13.1, 4096 x
// 4096 31.0 and 31.5, 4096 x 12288 81.0 and 79.1); beyond it wide tiles win (256 x 24576 x 4096: 63 us, 54 in pair tiles).
static bool is_skinny(int M, int N) {
  return M <= 128 || std::min(static_cast<long>((M + 255) / 256) * ((N + 255) / 256), static_cast<long>((M + 127) / 128) * ((N + 255) / 256) / 2) < num_sms() / 2;
}

bool gemm_skinny(const torch::Tensor& a, const torch::Tensor& b, void* out, int M, int N, int K, int ldo, bool out_fp32, bool accumulate, cudaStream_t stream) {
  using namespace gs;
  if (K % ATOM != 0 || !is_skinny(M, N)) return false;
  SkinnyParams p{};
  p.out = out; p.M = M; p.N = N; p.ldo = ldo; p.out_fp32 = out_fp32; p.accumulate = accumulate; p.err = error_word();
  p.rows = std::min(BM, (M + 7) / 8 * 8);
  p.k_atoms = K / ATOM;
  // Tile and split with the least time by what was measured here, in us: an SM takes in 110 KB/us, a product of 16 along K is issued every 35 ns, a
  // tile costs 2 us around that and a split another 3; two CTAs share an SM where there are more than SMs.  A split in two pays from K = 8192 on (64 x
  // 4096 x 12288: 26 us, 37 without); at 4096 it gave nothing over narrow tiles (64 x 4096 x 4096: 13.5 and 13.2), and clusters of 8 CTAs that fill
  // an SM each do not all fit the GPCs at once (28).
  const int mt = (M + BM - 1) / BM, sms = num_sms(), max_split = K >= 8192 ? 2 : 1;
  float best = 1e30f;
  for (int bn = 16; bn <= 256; bn += 16) {
    const long ctas = static_cast<long>((N + bn - 1) / bn) * mt;
    for (int s = 1; s <= max_split; ++s) {
      const float kp = static_cast<float>(K) / s, own = (s > 1 ? 5.f : 2.f), chain = kp * (0.035f / 16.f), load = (p.rows + bn) * kp * (2.f / 110e3f);
      const long n = ctas * s;
      const float cost = n <= sms ? std::max(chain, load) + own : (n + 2 * sms - 1) / (2 * sms) * (std::max(chain, 2.f * load) + own);
      if (cost < best * 0.999f) { best = cost; p.bn = bn; p.split = s; }
    }
  }
  const int tiles = (N + p.bn - 1) / p.bn;
  const bool two = static_cast<long>(tiles) * mt * p.split > sms;           // two CTAs per SM hide each other's start and end
  const int slack = (BM - p.rows) * ATOM_ROW;                               // what products read behind the last live row of the last atom
  const int room = (two ? 112 : 224) * 1024 - 2048 - slack;
  const int per_atom = (p.rows + p.bn) * ATOM_ROW;
  int ka = 4;                                                               // deep stages cost few instructions; at least four of them
  while (ka > 1 && room / (per_atom * ka) < 4) ka /= 2;
  p.stages = std::min({MAX_STAGES, room / (per_atom * ka), std::max(1, (p.k_atoms + ka - 1) / ka)});
  if (p.stages < 1) return false;
  p.tmem_cols = 32;
  while (p.tmem_cols < p.bn) p.tmem_cols *= 2;
  size_t ring = static_cast<size_t>(p.stages) * per_atom * ka + slack;
  if (p.split > 1) ring = std::max(ring, static_cast<size_t>(p.rows) * (p.bn + PAD) * 4);
  CUtensorMap ta = make_tmap_3d(a.data_ptr(), ATOM, M, p.k_atoms, a.stride(0), ATOM, ATOM, p.rows, ka);
  CUtensorMap tb = make_tmap_3d(b.data_ptr(), ATOM, N, p.k_atoms, b.stride(0), ATOM, ATOM, p.bn, ka);
  auto kern = ka == 4 ? gemm_skinny_kernel<4> : ka == 2 ? gemm_skinny_kernel<2> : gemm_skinny_kernel<1>;
  static OncePerDevice limit;
  limit(current_device(), [] {
    for (auto k : {gemm_skinny_kernel<4>, gemm_skinny_kernel<2>, gemm_skinny_kernel<1>}) TK_CUDA_CHECK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, 226 * 1024));
  });
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(tiles * p.split, mt);
  cfg.blockDim = dim3(THREADS);
  cfg.dynamicSmemBytes = ring + 2048;
  cfg.stream = stream;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = p.split;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  TK_CUDA_CHECK(cudaLaunchKernelEx(&cfg, kern, ta, tb, p));
  count_launch();
  return true;
}

}  // namespace tk
