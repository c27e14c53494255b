// Barrier of all blocks of a cooperative launch: a counter of arrivals in
// global memory, waited for by one thread of each block, with a limit (2,300
// clocks among 152 blocks).
#pragma once

namespace goal {

constexpr int kWaitLimit = 1 << 22;  // looks at the counter (more than a second)

// The limit of the launches that follow: kWaitLimit, or the one that was set
// (goal_set_wait_limit, so that a test can see a wait run out).
int wait_limit();
void set_wait_limit(int looks);

#ifdef __CUDACC__
// By one thread of each block. `count` has to be zero when the kernel begins;
// `target` is the number of arrivals to wait for: the blocks times the barriers
// so far, this one included. False when the wait ran out, after `limit` looks.
__device__ __forceinline__ bool grid_meet(unsigned* count, unsigned target, int limit) {
  asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(count) : "memory");
  unsigned v;
  int spins = 0;
  do {
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(count) : "memory");
  } while (v < target && ++spins < limit);
  return v >= target;
}
#endif

}  // namespace goal
