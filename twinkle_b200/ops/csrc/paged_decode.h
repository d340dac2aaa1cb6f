// Decode attention against the paged cache on the tensor cores (paged_decode.cu), called by the dispatch in decode.cu.
#pragma once
#include "scores.cuh"

namespace tk {

struct PagedDecode {
  const void *q, *kc, *vc;        // [B, hq, D], [blocks, block_size, hkv, D] bf16
  const int *tables, *seq_lens;   // [B, max_blocks], [B]
  void* out;                      // [B, hq, D]
  const void* sinks;              // [hq] (nullptr: none)
  OutGate gate;
  int hq, hkv, G, block_size, max_blocks, window, chunk;
  float scale_log2;
};

// False when the shape is not one of this kernel's.
bool paged_decode_mma(const PagedDecode& p, int B, int d, int e, cudaStream_t stream);

}  // namespace tk
