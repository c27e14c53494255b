// When and how a solver cycle of N nodes runs as one persistent kernel
// (krylov_coop.cuh), on the host; no device code, so that the rule can be
// checked without a GPU.
#pragma once

#include <algorithm>
#include <cstddef>

namespace goal {

// What of a device the rule needs; launches = cooperative launches are available.
struct CoopDevice {
  int sms = 0, smem = 0;
  bool launches = false;
};
const CoopDevice& coop_device();  // of the current device

// Nodes per CTA and CTAs, one CTA per SM at most.
struct CoopPlan {
  int chunk = 0, grid = 0;
};

// The persistent cycle wins while an Arnoldi step is bound by its launches and
// its few blocks; far enough up, the separate kernels with their more threads in
// flight on the matrix and basis streams are faster, the earlier the more of a
// step the products are. 100 columns in FP64, 3 x 60 inner ones else, ms, kernels ->
// persistent, at nodes below and above each line:
//   one sweep   binary16 301k 18.7 -> 16.8, 358k 22.9 -> 23.0, 405k 24.6 -> 25.3
//               binary32 301k 31.9 -> 22.6, 358k 35.8 -> 33.7, 405k 38.3 -> 36.5
//   two sweeps  binary16 149k 19.1 -> 15.5, 176k 22.0 -> 19.7, 227k 26.0 -> 28.9
//               binary32 149k 26.9 -> 22.2, 176k 35.5 -> 26.8, 227k 40.4 -> 40.8
//   FP64        one 104k 40.3 -> 30.3, 141k 42.6 -> 39.6, 227k 56.1 -> 62.3
//               two 104k 48.3 -> 39.6, 141k 53.1 -> 52.0, 227k 72.5 -> 80.3
//   FP64 inner  one 104k 32.5 -> 25.0, 141k 35.7 -> 32.6, 227k 48.5 -> 51.6
//               two 104k 44.6 -> 40.1, 141k 52.0 -> 52.7, 227k 73.7 -> 80.4
// and at 30k to 69k nodes 1.3 to 2 times faster throughout.
constexpr int kCoopMinNodes = 8;  // of a CTA: a warp of rows
constexpr int kCoopNodesPerSm = 2300, kCoopNodesPerSmSweep2 = 1150, kCoopNodesPerSmFp64 = 900;

inline bool coop_plan(const CoopDevice& d, int N, bool fp64, bool sweep2, CoopPlan& p) {
  if (!d.launches) return false;
  const int per_sm = fp64 ? kCoopNodesPerSmFp64 : sweep2 ? kCoopNodesPerSmSweep2 : kCoopNodesPerSm;
  if (N > per_sm * d.sms) return false;
  p.chunk = std::max(kCoopMinNodes, (N + 8 * d.sms - 1) / (8 * d.sms) * 8);
  p.grid = (N + p.chunk - 1) / p.chunk;
  return true;
}

// Shared memory that a CTA cannot do without, as the kernel lays it out: w, t, h,
// coefficients, scales, rotations, the reduction buffer and row pointers, for
// numbers of `size` bytes and up to m columns.
constexpr int kCoopThreads = 512;            // worker threads of a CTA
constexpr int kCoopWarps = kCoopThreads / 32;
constexpr int kCoopRed = 32 * kCoopWarps;    // entries of the block-level reduction buffer
inline size_t coop_pad(size_t bytes) { return (bytes + 31) / 32 * 32; }
inline size_t coop_fixed_bytes(int chunk, int m, size_t size, bool sweep2) {
  return (sweep2 ? 2 : 1) * coop_pad(size * 4 * chunk) + 11 * coop_pad(size * (m + 2)) + coop_pad(size * kCoopRed) +
         coop_pad(sizeof(int) * (chunk + 1));
}

}  // namespace goal
