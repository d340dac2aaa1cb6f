// Issue of tensor-core products by one thread of a converged warp.
#pragma once
#include <stdint.h>

namespace tk {

// One thread of a converged warp, the same one every time.  A warp that walks its loop together and elects a thread for the issue keeps
// descriptors and addresses in uniform registers; inside `if (lane == 0)` each product first moves them there.
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
  return p != 0;
}

}  // namespace tk
