// Keys and values of a step or of prompts into the paged pools, and the host side of a step's inputs.
//
// Two index_put calls per layer and sequence (prompts: 11 small operations per layer and sequence, 5 us each; a step 2 x 4 us) become one launch of
// 16-byte copies: a row's place is computed once per forward pass, not per layer.
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/extension.h>

#include "common.cuh"
#include "host.h"

namespace tk {

struct CacheWrite {
  const uint4 *k, *v;             // rows of nk and nv vectors, sk and sv vectors apart
  uint4 *kp, *vp;                 // pools, row by row
  const int64_t* rows;            // row of the pools per token
  long total, pool_rows;
  int nk, nv;
  long sk, sv;
  int* err;
};

__global__ void cache_write_kernel(const CacheWrite p) {
  const int n = p.nk + p.nv;
  for (long i = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x; i < p.total; i += static_cast<long>(gridDim.x) * blockDim.x) {
    const long t = i / n;
    const int c = static_cast<int>(i - t * n);
    const int64_t row = p.rows[t];
    if (row < 0 || row >= p.pool_rows) {        // a block list that names no block of the pool: whoever reads the word next raises
      atomicCAS(p.err, 0, ERR_BOUNDS);
      continue;
    }
    if (c < p.nk) p.kp[row * p.nk + c] = p.k[t * p.sk + c];
    else p.vp[row * p.nv + c - p.nk] = p.v[t * p.sv + c - p.nk];
  }
}

// pools [blocks, block_size, heads, ·], rows int64 [T] (block · block_size + offset), k and v [T, heads, ·] with heads side by side.
// A row outside the pools is left out and noted in the error word.
void cache_write(const torch::Tensor& kp, const torch::Tensor& vp, const torch::Tensor& rows, const torch::Tensor& k, const torch::Tensor& v) {
  const int64_t e = k.element_size();
  auto fits = [&](const torch::Tensor& pool, const torch::Tensor& x) {
    TORCH_CHECK(x.is_cuda() && pool.is_cuda() && x.dim() == 3 && pool.dim() == 4 && pool.is_contiguous() && pool.scalar_type() == x.scalar_type() && x.element_size() == e &&
                    pool.size(2) == x.size(1) && pool.size(3) == x.size(2), "pool [blocks, size, heads, width] like the rows [T, heads, width]");
    const int64_t width = x.size(1) * x.size(2);
    TORCH_CHECK(x.stride(2) == 1 && x.stride(1) == x.size(2) && width * e % 16 == 0 && x.stride(0) * e % 16 == 0 && reinterpret_cast<uintptr_t>(x.data_ptr()) % 16 == 0 &&
                    reinterpret_cast<uintptr_t>(pool.data_ptr()) % 16 == 0, "rows of whole 16-byte vectors");
    return static_cast<int>(width * e / 16);
  };
  CacheWrite p{};
  p.nk = fits(kp, k);
  p.nv = fits(vp, v);
  TORCH_CHECK(rows.is_cuda() && rows.scalar_type() == torch::kInt64 && rows.is_contiguous() && rows.numel() == k.size(0) && v.size(0) == k.size(0) &&
                  kp.size(0) * kp.size(1) == vp.size(0) * vp.size(1), "rows int64 [T], pools of the same number of rows");
  c10::cuda::CUDAGuard guard(k.device());
  p.total = k.size(0) * static_cast<long>(p.nk + p.nv);
  if (p.total == 0) return;
  p.k = reinterpret_cast<const uint4*>(k.data_ptr()); p.v = reinterpret_cast<const uint4*>(v.data_ptr());
  p.kp = reinterpret_cast<uint4*>(kp.data_ptr()); p.vp = reinterpret_cast<uint4*>(vp.data_ptr());
  p.rows = rows.data_ptr<int64_t>();
  p.pool_rows = kp.size(0) * kp.size(1);
  p.sk = k.stride(0) * e / 16; p.sv = v.stride(0) * e / 16; p.err = error_word();
  const int blocks = static_cast<int>(std::min<long>((p.total + 255) / 256, num_sms() * 16L));
  cache_write_kernel<<<blocks, 256, 0, at::cuda::getCurrentCUDAStream()>>>(p);
  count_launch();
  TK_CUDA_CHECK(cudaGetLastError());
}

// A step's inputs in one int32 host tensor: block tables [rows, width], lengths [rows], slots [rows]; zeros past the given sequences.
void pack_step(const torch::Tensor& out, int64_t rows, int64_t width, const std::vector<std::vector<int32_t>>& blocks, const std::vector<int32_t>& lens, const std::vector<int32_t>& slots) {
  TORCH_CHECK(!out.is_cuda() && out.scalar_type() == torch::kInt32 && out.is_contiguous() && out.numel() == rows * (width + 2), "out int32 [rows * (width + 2)]");
  TORCH_CHECK(static_cast<int64_t>(blocks.size()) <= rows && lens.size() == blocks.size() && slots.size() == blocks.size(), "one entry per sequence");
  int32_t* p = out.data_ptr<int32_t>();
  std::fill(p, p + out.numel(), 0);
  for (size_t i = 0; i < blocks.size(); ++i) {
    TORCH_CHECK(static_cast<int64_t>(blocks[i].size()) <= width, "block list wider than the table");
    std::copy(blocks[i].begin(), blocks[i].end(), p + i * width);
    p[rows * width + i] = lens[i];
    p[rows * (width + 1) + i] = slots[i];
  }
}

// Rows of the pools for tokens 0 … lens[i] of every sequence, one after the other: int64 [Σ lens] on the host.
torch::Tensor prompt_rows(const std::vector<std::vector<int32_t>>& blocks, const std::vector<int64_t>& lens, int64_t block_size, bool pinned) {
  TORCH_CHECK(blocks.size() == lens.size() && block_size > 0, "one length per sequence");
  int64_t total = 0;
  for (int64_t n : lens) total += n;
  auto out = torch::empty({total}, torch::TensorOptions().dtype(torch::kInt64).pinned_memory(pinned));
  int64_t* p = out.data_ptr<int64_t>();
  for (size_t i = 0; i < lens.size(); ++i) {
    TORCH_CHECK(lens[i] <= static_cast<int64_t>(blocks[i].size()) * block_size, "sequence longer than its blocks");
    for (int64_t t = 0; t < lens[i]; ++t) *p++ = blocks[i][t / block_size] * block_size + t % block_size;
  }
  return out;
}

}  // namespace tk
