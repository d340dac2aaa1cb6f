// Token sampling: temperature, top-k and top-p by a search for the threshold, Gumbel-max among what is kept, log-prob of the processed
// distribution.
//
// What bounds it: a row of logits is read once (0.6 MB at 152 k tokens) and then searched, a compare and an add per element and threshold.  One CTA
// per row with 15 thresholds for each of both searches in 8 passes over global memory took 1160 us at 64 x 151936 (31 GB/s).  Here a cluster of
// up to 8 CTAs holds a row, each CTA its part as e = exp(x/T − max) in shared memory, and a search is
//   3 passes with 3, 3 and 1 thresholds at powers of two, which end with lo ≤ threshold < 2·lo (or below 2^-31), 2 instructions per threshold,
//   passes with 15 over what lies between, gathered once: a small part of the row, until the bracket is 2^-32 of the largest probability.
// Only the searches that are asked for run.  us before → now: 64 x 151936 top_p 1160 → 116 (now bound by instructions: thresholds and the Gumbel
// hash), top_k 50 1130 → 93, neither 154 → 44, greedy 124 → 14; 256 x 151936 both 2100 → 520; 256 x 32000 top_p 398 → 94; one row of 151936 1127 → 36 (barriers).
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <cooperative_groups.h>
#include <torch/types.h>

#include "common.cuh"
#include "host.h"

namespace tk {

namespace cg = cooperative_groups;

namespace sm {
constexpr int MAX_CTAS = 8, THREADS = 512, WARPS = THREADS / 32, NT = 15;
}

__device__ __forceinline__ uint32_t mix32(uint64_t x) {
  x ^= x >> 33; x *= 0xff51afd7ed558ccdull; x ^= x >> 33; x *= 0xc4ceb9fe1a85ec53ull; x ^= x >> 33;
  return static_cast<uint32_t>(x);
}

struct SampleShared {
  float warp[sm::WARPS][sm::NT + 1];
  float slot[2][sm::MAX_CTAS][sm::NT + 1];   // every CTA's share of a sum or maximum, written by it; two take turns
  float all[sm::NT + 1];
  int idx[sm::WARPS], best_i;
  int overflow;
};

// Sums (or the maximum) of N values over the cluster, the same bits in every thread.
template <int N, bool MAX>
__device__ __forceinline__ void cluster_reduce(const cg::cluster_group& cluster, SampleShared& sh, int& turn, float (&v)[N]) {
  using namespace sm;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if constexpr (N > 4 && !MAX) {
    // 16 sums over 32 lanes in 16 shuffles instead of 80: lanes exchange the halves of their values that the other keeps
    float u[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) u[j] = j < N ? v[j] : 0.f;
#pragma unroll
    for (int h = 8, o = 16; h >= 1; h >>= 1, o >>= 1) {
      const bool upper = lane & o;
#pragma unroll
      for (int j = 0; j < h; ++j) {
        const float give = upper ? u[j] : u[j + h], keep = upper ? u[j + h] : u[j];
        u[j] = keep + __shfl_xor_sync(0xffffffffu, give, o);
      }
    }
    u[0] += __shfl_xor_sync(0xffffffffu, u[0], 1);
    if ((lane & 1) == 0 && lane / 2 < N) sh.warp[warp][lane / 2] = u[0];     // bits 4..1 of the lane chose the halves: value lane / 2
  } else {
#pragma unroll
    for (int j = 0; j < N; ++j) {
      const float w = MAX ? warp_max(v[j]) : warp_sum(v[j]);
      if (lane == 0) sh.warp[warp][j] = w;
    }
  }
  __syncthreads();
  if (threadIdx.x < N) {
    float r = sh.warp[0][threadIdx.x];
#pragma unroll
    for (int w = 1; w < WARPS; ++w) r = MAX ? fmaxf(r, sh.warp[w][threadIdx.x]) : r + sh.warp[w][threadIdx.x];
    const int ctas = cluster.num_blocks();
    for (int c = 0; c < ctas; ++c) cluster.map_shared_rank(&sh, c)->slot[turn][cluster.block_rank()][threadIdx.x] = r;
  }
  cluster.sync();
  if (threadIdx.x < N) {
    float r = sh.slot[turn][0][threadIdx.x];
    const int ctas = cluster.num_blocks();
    for (int c = 1; c < ctas; ++c) r = MAX ? fmaxf(r, sh.slot[turn][c][threadIdx.x]) : r + sh.slot[turn][c][threadIdx.x];
    sh.all[threadIdx.x] = r;
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < N; ++j) v[j] = sh.all[j];
  turn ^= 1;
}

// Bracket of a search: what is kept at `lo` satisfies the demand, what is kept at `hi` does not (or hi is the top, which keeps all that lies above).
struct Bracket {
  float lo, hi, above;   // above: what lies at hi or over it
  bool top;
};

// One CTA's part of a row: e values, in shared memory or (CACHED = false, rows beyond it) formed anew from the logits.
template <bool CACHED>
struct RowPart {
  const float* x;
  float* e;
  float inv_temp, mx;
  int n;
  __device__ __forceinline__ float at(int i) const { return CACHED ? e[i] : __expf(x[i] * inv_temp - mx); }
  // every thread's share in turn, f(e); the cache is filled up to whole vectors with −1, which no threshold keeps
  template <typename F>
  __device__ __forceinline__ void each(F&& f) const {
    if constexpr (CACHED) {
#pragma unroll 2
      for (int i = threadIdx.x; i < (n + 3) / 4; i += sm::THREADS) {
        const float4 v = reinterpret_cast<const float4*>(e)[i];
        f(v.x); f(v.y); f(v.z); f(v.w);
      }
    } else {
      for (int i = threadIdx.x; i < n; i += sm::THREADS) f(at(i));
    }
  }
};

template <int N, bool COUNT>
__device__ __forceinline__ void weigh(float e, const float (&t)[N], float (&acc)[N]) {
#pragma unroll
  for (int j = 0; j < N; ++j) acc[j] += e >= t[j] ? (COUNT ? 1.f : e) : 0.f;
}

// N thresholds (rising) over the whole part; narrows the bracket.
template <int N, bool COUNT, bool CACHED>
__device__ __forceinline__ void coarse(const cg::cluster_group& cluster, SampleShared& sh, int& turn, const RowPart<CACHED>& row, const float (&t)[N], float want, Bracket& b) {
  float acc[N];
#pragma unroll
  for (int j = 0; j < N; ++j) acc[j] = 0.f;
  row.each([&](float e) { weigh<N, COUNT>(e, t, acc); });
  cluster_reduce<N, false>(cluster, sh, turn, acc);
  bool open = true;
#pragma unroll
  for (int j = 0; j < N; ++j) {      // rising thresholds, falling sums
    if (acc[j] >= want) b.lo = t[j];
    else if (open) { b.hi = t[j]; b.above = acc[j]; b.top = false; open = false; }
  }
}

// Highest threshold on e, to 2^-32, that still keeps `want` (tokens, or the mass of e).
template <bool COUNT, bool CACHED>
__device__ float search(const cg::cluster_group& cluster, SampleShared& sh, int& turn, const RowPart<CACHED>& row, float want, float* list, int list_cap) {
  using namespace sm;
  Bracket b{0.f, 1.f, 0.f, true};
  int down = 32;       // lo = 2^-down once it is above 0, and hi = 2·lo
  {
    const float t[3] = {0x1p-24f, 0x1p-16f, 0x1p-8f};
    coarse<3, COUNT>(cluster, sh, turn, row, t, want, b);
    const float s = b.top ? 1.f : b.hi;
    const float u[3] = {s * 0x1p-6f, s * 0x1p-4f, s * 0x1p-2f};
    coarse<3, COUNT>(cluster, sh, turn, row, u, want, b);
    const float h = b.top ? 1.f : b.hi;
    const float v[1] = {h * 0.5f};
    coarse<1, COUNT>(cluster, sh, turn, row, v, want, b);
    down = b.lo > 0.f ? -ilogbf(b.lo) : 32;
  }
  // the bracket is a power of two wide: [2^-down, 2^(1-down)), or [0, 2^-31) of which one half is left to try
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int bits = b.lo > 0.f ? 32 - down : static_cast<int>(32 + ilogbf(b.hi));
  if (bits <= 0) return b.lo;
  // gather what lies inside, warp by warp and in order; a CTA without room goes on with its whole part
  float* mine = list + warp * list_cap;
  int count = 0;
  bool fits = CACHED;
  if constexpr (CACHED) {
    for (int i = threadIdx.x - lane; i < (row.n + 3) / 4; i += THREADS) {
      const float4 v = i + lane < (row.n + 3) / 4 ? reinterpret_cast<const float4*>(row.e)[i + lane] : make_float4(-1.f, -1.f, -1.f, -1.f);
      const float e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const bool in = e[k] >= b.lo && (b.top || e[k] < b.hi);
        const uint32_t who = __ballot_sync(0xffffffffu, in);
        const int at = count + __popc(who & ((1u << lane) - 1u));
        if (in && at < list_cap) mine[at] = e[k];
        count += __popc(who);
      }
    }
    if (threadIdx.x == 0) sh.overflow = 0;
    __syncthreads();
    if (lane == 0 && count > list_cap) sh.overflow = 1;
    __syncthreads();
    fits = sh.overflow == 0;
    __syncwarp();
  }
  const bool top = b.top;
  const float hi = b.hi, base = top ? 0.f : b.above;       // what lies over the bracket counts for every threshold in it
  while (bits > 0) {
    const int step = bits % 4 ? bits % 4 : 4, n = (1 << step) - 1;
    const float d = (b.hi - b.lo) * (1.f / static_cast<float>(1 << step));
    float t[NT], acc[NT];
#pragma unroll
    for (int j = 0; j < NT; ++j) {
      t[j] = j < n ? b.lo + d * static_cast<float>(j + 1) : INFINITY;
      acc[j] = 0.f;
    }
    if (fits) {
      for (int i = lane; i < count; i += 32) weigh<NT, COUNT>(mine[i], t, acc);
    } else {
      row.each([&](float e) {
        if (top || e < hi) weigh<NT, COUNT>(e, t, acc);
      });
    }
    cluster_reduce<NT, false>(cluster, sh, turn, acc);
    float lo = b.lo;
    int last = -1;
#pragma unroll
    for (int j = 0; j < NT; ++j)
      if (j < n && acc[j] + base >= want) { lo = t[j]; last = j; }
    if (last < n - 1) b.hi = lo + d;
    b.lo = lo;
    bits -= step;
  }
  return b.lo;
}

// kept set = {e ≥ τ}: the highest τ that keeps top_k tokens and that keeps the mass top_p, whichever is higher (the smallest such set up to
// ties).  Token = argmax over the kept of (x/T + Gumbel noise), the smaller index among equals.
template <bool CACHED>
__global__ void __launch_bounds__(sm::THREADS, 2)
sample_kernel(const float* __restrict__ logits, const int64_t* __restrict__ seeds, int64_t* __restrict__ tok, float* __restrict__ logprob, int V, int part, float inv_temp, int top_k,
              float top_p, int greedy, int list_cap) {
  using namespace sm;
  extern __shared__ __align__(16) float smem[];
  __shared__ SampleShared sh;
  const cg::cluster_group cluster = cg::this_cluster();
  const int ctas = cluster.num_blocks(), row = blockIdx.x / ctas, rank = blockIdx.x % ctas, begin = min(V, rank * part);
  RowPart<CACHED> p{logits + static_cast<size_t>(row) * V + begin, smem, inv_temp, 0.f, min(V, begin + part) - begin};
  cluster.sync();                     // shares are written into each other's shared memory: everyone is there
  int turn = 0;
  float z = 1.f, kept = 1.f, tau = 0.f;
  if (!greedy) {
    float mx[1] = {-INFINITY};      // of the whole row, in the end
    const bool vec = (reinterpret_cast<uintptr_t>(p.x) & 15) == 0;       // a part starts on 16 bytes where the row does
    if (vec) {
      const int n4 = p.n / 4;
      for (int i = threadIdx.x; i < n4; i += THREADS) {
        float4 v = reinterpret_cast<const float4*>(p.x)[i];
        v.x *= inv_temp; v.y *= inv_temp; v.z *= inv_temp; v.w *= inv_temp;
        mx[0] = fmaxf(mx[0], fmaxf(fmaxf(v.x, v.y), fmaxf(v.z, v.w)));
        if (CACHED) reinterpret_cast<float4*>(smem)[i] = v;
      }
    }
    for (int i = (vec ? p.n / 4 * 4 : 0) + threadIdx.x; i < p.n; i += THREADS) {
      const float v = p.x[i] * inv_temp;
      mx[0] = fmaxf(mx[0], v);
      if (CACHED) smem[i] = v;
    }
    cluster_reduce<1, true>(cluster, sh, turn, mx);      // its barriers also make the cached part visible
    p.mx = mx[0];
    float sum[1] = {0.f};
    if constexpr (CACHED) {
      for (int i = threadIdx.x; i < (p.n + 3) / 4; i += THREADS) {
        float4 v = reinterpret_cast<float4*>(smem)[i];
        v.x = __expf(v.x - p.mx); v.y = __expf(v.y - p.mx); v.z = __expf(v.z - p.mx); v.w = __expf(v.w - p.mx);
        if (4 * i + 3 >= p.n) {
          if (4 * i + 1 >= p.n) v.y = -1.f;
          if (4 * i + 2 >= p.n) v.z = -1.f;
          v.w = -1.f;
        }
        if (4 * i + 3 < p.n) sum[0] += (v.x + v.y) + (v.z + v.w);
        else sum[0] += v.x + (v.y < 0.f ? 0.f : v.y) + (v.z < 0.f ? 0.f : v.z);
        reinterpret_cast<float4*>(smem)[i] = v;
      }
      __syncthreads();
    } else {
      p.each([&](float e) { sum[0] += e; });
    }
    cluster_reduce<1, false>(cluster, sh, turn, sum);
    z = sum[0];
    const bool use_k = top_k > 0 && top_k < V, use_p = top_p < 1.f;
    float* list = smem + (part + 3) / 4 * 4;
    if (use_k) tau = search<true>(cluster, sh, turn, p, static_cast<float>(top_k), list, list_cap);
    if (use_p) {
      __syncthreads();
      tau = fmaxf(tau, search<false>(cluster, sh, turn, p, top_p * z, list, list_cap));
    }
    if (use_k || use_p) {
      float mass[1] = {0.f};
      p.each([&](float e) { mass[0] += e >= tau ? e : 0.f; });
      cluster_reduce<1, false>(cluster, sh, turn, mass);
      kept = mass[0] / z;
    }
  }
  float best = -INFINITY;
  int best_i = 0;
  const uint64_t seed = static_cast<uint64_t>(seeds[row]);
  if (greedy) {
    for (int i = threadIdx.x; i < p.n; i += THREADS) {
      const float score = p.x[i] * inv_temp;
      if (score > best) { best = score; best_i = begin + i; }
    }
  } else {
    // With E = −ln u the score is ln(e / E) + max, and E ≥ 1 − u: an element with e / (1 − u) well below what the warp has already cannot win, and
    // its logarithms are not taken (64 x 151936 without a search: 89 → 71 us, at the occupancy of one CTA per SM).  Near u = 1 the error of __logf is
    // absolute, up to 2^-21.41 by its documentation, so what is compared is (1 − u) − 2^-21; the 0.1 % is for the relative errors of e, of logarithms elsewhere
    // and of scores, whose magnitude is taken to stay below 2^12.  Then nothing that would win is left out, however the row is cut.
    float bar = 0.f;                  // the warp's best e / E, a little less
    for (int i = threadIdx.x; i - static_cast<int>(threadIdx.x & 31) < p.n; i += THREADS) {
      bool open = false;
      float u = 0.f;
      if (i < p.n) {
        const float e = p.at(i);
        u = (static_cast<float>(mix32(seed * 0x9E3779B97F4A7C15ull + static_cast<uint64_t>(begin + i))) + 0.5f) * (1.f / 4294967296.f);
        open = !(e < tau) && !(e < fmaf(-bar, u, bar * (1.f - 0x1p-21f)));
      }
      if (__any_sync(0xffffffffu, open)) {
        if (open) {
          // Hashes from 2^32 − 128 on round to u = 1, where E = 0 would let a token win whatever its logit (one row in 220 at 152 k tokens); they
          // stand for 1 − u = 2^-26 on average.
          const float E = u < 1.f ? -__logf(u) : 0x1p-26f;
          const float score = p.x[i] * inv_temp - __logf(E);
          if (score > best) { best = score; best_i = begin + i; }
        }
        bar = 0.999f * __expf(warp_max(best) - p.mx);
      }
    }
  }
  auto take = [&](float ob, int oi) {
    if (ob > best || (ob == best && oi < best_i)) { best = ob; best_i = oi; }
  };
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float ob = __shfl_xor_sync(0xffffffffu, best, o);
    const int oi = __shfl_xor_sync(0xffffffffu, best_i, o);
    take(ob, oi);
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __syncthreads();
  if (lane == 0) { sh.warp[warp][0] = best; sh.idx[warp] = best_i; }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < WARPS; ++w) take(sh.warp[w][0], sh.idx[w]);
    sh.slot[turn][0][0] = best;
    sh.best_i = best_i;
  }
  cluster.sync();
  if (rank == 0 && threadIdx.x == 0) {
    for (int c = 1; c < ctas; ++c) {
      const SampleShared* o = cluster.map_shared_rank(&sh, c);
      take(o->slot[turn][0][0], o->best_i);
    }
    tok[row] = best_i;
    logprob[row] = greedy ? 0.f : (logits[static_cast<size_t>(row) * V + best_i] * inv_temp - p.mx - __logf(z) - __logf(kept));
  }
  cluster.sync();                     // nobody leaves while its shared memory is read
}

std::vector<torch::Tensor> sample_tokens(const torch::Tensor& logits, double temperature, int64_t top_k, double top_p, const torch::Tensor& seeds) {
  TORCH_CHECK(logits.is_cuda() && logits.scalar_type() == torch::kFloat32 && logits.is_contiguous() && logits.dim() == 2, "logits [B,V] fp32");
  TORCH_CHECK(seeds.is_cuda() && seeds.scalar_type() == torch::kInt64 && seeds.numel() == logits.size(0), "seeds int64 [B]");
  c10::cuda::CUDAGuard guard(logits.device());
  const int B = logits.size(0), V = logits.size(1);
  auto tok = torch::empty({B}, logits.options().dtype(torch::kInt64));
  auto lp = torch::empty({B}, logits.options());
  if (B == 0) return {tok, lp};
  const bool greedy = temperature <= 0.0;
  constexpr int kRoom = 220 * 1024 / 4;                                  // floats of dynamic shared memory
  // CTAs per row: parts of up to 24 k tokens, with which two CTAs fit an SM, and more of them while the rows leave the chip idle and a part has 4 k
  int ctas = 1;
  while (ctas < sm::MAX_CTAS && (V > 24576 * ctas || (B * ctas < 2 * num_sms() && V > 8192 * ctas))) ctas *= 2;
  const int part = ((V + ctas - 1) / ctas + 3) / 4 * 4;
  // a list takes a quarter of the part: the last bracket of the powers of two holds about a sixth of a broad row
  const int list_cap = (part / 4 + sm::WARPS - 1) / sm::WARPS + 8;
  const bool cached = !greedy && part + list_cap * sm::WARPS <= kRoom;   // rows of up to 340 k tokens
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(B * ctas);
  cfg.blockDim = dim3(sm::THREADS);
  cfg.dynamicSmemBytes = cached ? 4 * (part + list_cap * sm::WARPS) : 0;
  cfg.stream = at::cuda::getCurrentCUDAStream();
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = ctas;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  static OncePerDevice limit;
  limit(current_device(), [] { TK_CUDA_CHECK(cudaFuncSetAttribute(sample_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kRoom * 4)); });
  TK_CUDA_CHECK(cudaLaunchKernelEx(&cfg, cached ? sample_kernel<true> : sample_kernel<false>, static_cast<const float*>(logits.data_ptr<float>()),
                                   static_cast<const int64_t*>(seeds.data_ptr<int64_t>()), tok.data_ptr<int64_t>(), lp.data_ptr<float>(), V, part,
                                   greedy ? 1.f : static_cast<float>(1.0 / temperature), static_cast<int>(top_k), static_cast<float>(top_p), greedy ? 1 : 0, list_cap));
  count_launch();
  TK_CUDA_CHECK(cudaGetLastError());
  return {tok, lp};
}

}  // namespace tk
