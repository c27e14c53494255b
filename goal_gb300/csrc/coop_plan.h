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
// step the products are. Whole solves to 1e-12, ms, kernels -> persistent:
// binary16 inner 5k nodes 28.0 -> 11.3, 36k 58 -> 28, 59k 72.7 -> 44.4, 185k 230
// -> 181, 275k 327 -> 303, 389k 520 -> 512, 531k 710 -> 781; with the second
// sweep 149k 138 -> 109, 185k 182 -> 184, 227k 220 -> 234; binary32 133k 253 ->
// 165, 227k 496 -> 329; FP64 inner 69k 318 -> 212, 133k 544 -> 469; FP64 343
// 26.5 -> 3.9, 36k 1717 -> 828, 69k 5090 -> 3230 (not measured further up).
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
