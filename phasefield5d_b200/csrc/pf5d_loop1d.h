// pf5d_loop1d.h -- the 1D step loops' limits and the split of a solve's points
// over the blocks of its cluster (host code, no CUDA).
#pragma once

#include <cstdint>

namespace pf5d {

constexpr int64_t kLoop1dMax = 16384;        // points of a 1D solve that a cluster advances
constexpr int kLoop1dThreads = 512;          // most threads of a block (128 registers each)
constexpr int kLoop1dBlocks = 16;            // most blocks of a cluster
constexpr int kLoop1dSteps = 2000;           // most steps of a launch
constexpr unsigned long long kLoop1dWaitNs = 2000000000;   // longest wait of a block for the others
constexpr int kLoop1dGroups = (int)(kLoop1dMax / 32);

// Blocks of the cluster, points per block (a multiple of 32) and threads per
// block for n points.  A block evaluates mu/M at its points and one halo
// position on each side: all warps but the last (which sums the misfit
// meanwhile) cover chunk + 2 positions in as few passes as kLoop1dThreads
// allows.
// Every block of the cluster holds points: the messages of a step double as the
// word that its sender has read the step before, and a block without points
// would send no B (203 points on 8 blocks of 32: 7 blocks, no eighth).
struct Loop1dShape {
  int blocks, chunk, threads;
};
inline Loop1dShape loop1d_shape(int64_t n, int max_blocks) {
  Loop1dShape L;
  const int groups = (int)((n + 31) / 32);
  L.blocks = 1;
  while (L.blocks < max_blocks && L.blocks < groups) L.blocks *= 2;
  const int per = (groups + L.blocks - 1) / L.blocks;
  L.chunk = 32 * per;
  L.blocks = (groups + per - 1) / per;
  const int most = kLoop1dThreads - 32;
  const int passes = (L.chunk + 2 + most - 1) / most;
  L.threads = 32 + 32 * (((L.chunk + 2 + passes - 1) / passes + 31) / 32);
  return L;
}

// Whether the loop is the faster form for a call of nsteps steps.  A launch first
// loads and sorts the solve, on 16 SMs; a single step of a long solve costs more
// that way than as separate kernels.  us, kernels -> loop, FP64 and FP32c: 8192
// points 22.5 -> 20.6 and 18.5 -> 17.3, 12000 22.6 -> 23.4 and 18.4 -> 18.4, 16384
// 22.5 -> 28.7 and 18.4 -> 21.4; two steps of 16384 are even.
inline bool loop1d_pays(int64_t n, int64_t nsteps) { return n <= 10240 || nsteps > 1; }

}  // namespace pf5d
