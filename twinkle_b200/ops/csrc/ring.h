// Which stages of a ring are still being filled, for a producer that gives up: it may not leave while copies into its shared memory are under way.
#pragma once

#ifdef __CUDACC__
#define TK_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define TK_HOST_DEVICE inline
#endif

namespace tk {

// Fill number `fill` (0, 1, …) goes to stage fill % stages, whose barrier completes one phase per fill: this one's has parity (fill / stages) & 1.
// Waiting for any other parity returns at once, or waits for a fill that was never issued.
struct RingFill {
  int stage;
  unsigned parity;
};
TK_HOST_DEVICE RingFill ring_fill(int fill, int stages) { return {fill % stages, static_cast<unsigned>(fill / stages) & 1u}; }
// First of the `issued` fills that may not have landed: a stage is only filled again when its last fill has been used.
TK_HOST_DEVICE int ring_first_open(int issued, int stages) { return issued > stages ? issued - stages : 0; }

}  // namespace tk
