// Barrier of all blocks of a cooperative launch: a counter of arrivals in
// global memory, waited for by one thread of each block, with a limit (2,300
// clocks among 152 blocks).
#pragma once

namespace goal {

constexpr int kSpinLimit = 1 << 22;  // looks at the counter (more than a second)

// By one thread of each block. `count` has to be zero when the kernel begins;
// `target` is the number of arrivals to wait for: the blocks times the barriers
// so far, this one included. False when the wait ran out.
__device__ __forceinline__ bool grid_meet(unsigned* count, unsigned target) {
  asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(count) : "memory");
  unsigned v;
  int spins = 0;
  do {
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(count) : "memory");
  } while (v < target && ++spins < kSpinLimit);
  return v >= target;
}

}  // namespace goal
