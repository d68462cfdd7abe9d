// Which of an epilogue warp's two staging boxes is written next (plain C++: the order is checked on the CPU).
#pragma once

#ifdef __CUDACC__
#define MSB_HD __host__ __device__ __forceinline__
#else
#define MSB_HD inline
#endif

namespace msb {

// The caller waits for all stores but the newest before it writes the box that take() names, so that must not be the box
// sent last: sent() records it, whatever the order in which the boxes of two outputs were taken and sent.
struct OutTurn {
  int next;
  MSB_HD int take() {
    const int box = next;
    next ^= 1;
    return box;
  }
  MSB_HD void sent(int box) { next = box ^ 1; }
};

}  // namespace msb
