// pf5d_cluster.cuh -- what the 1D step loops share (one thread-block cluster
// advances a whole solve, many steps per launch): the sum behind the closed-form
// elastic term, the messages between the blocks, and the launch.  The split of
// the points over the blocks is in pf5d_loop1d.h.
#pragma once

#include <cstdint>

#include <cooperative_groups.h>

#include "pf5d_host.h"
#include "pf5d_loop1d.h"

namespace pf5d {

// Sum of n values in groups of 32 consecutive ones: a fixed tree within each
// group (group_sum); then each lane adds every 32nd group's sum in order and a
// tree adds the lanes (sum_groups).  The result does not depend on how the
// groups are spread over warps and blocks.  Called by whole warps.
__device__ __forceinline__ double group_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = v + __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ double sum_groups(const double *sums, int n) {
  double v = 0.0;
  for (int g = threadIdx.x & 31; g < n; g += 32) v = v + sums[g];
  return group_sum(v);
}

// group_sum of 16 groups, a lane's value of group j in v[j], with a fifth of the
// shuffles: at each of the first four levels a lane keeps half of its groups and
// hands its values of the other half to the lane that keeps those.  The same
// pairs are added as in group_sum, in either order, so the same bits.  Returns
// the sum of group 8 l4 + 4 l3 + 2 l2 + l1 (the lane's bits).
__device__ __forceinline__ double group_sums16(double v[16]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 16, n = 8; n > 0; o >>= 1, n >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int j = 0; j < n; ++j) {
      const double got = __shfl_xor_sync(0xffffffffu, up ? v[j] : v[j + n], o);
      v[j] = (up ? v[j + n] : v[j]) + got;
    }
  }
  return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);
}

// Sums of all groups of s (n values, s(i) reads one) into sums[], by a block of
// 1024 threads: warp w takes the groups 16 w to 16 w + 15, or every 32nd where
// they are few.
constexpr int kGroupThreads = 1024;
static_assert(kLoop1dGroups == 16 * (kGroupThreads / 32), "16 groups a warp");
template <typename Read>
__device__ __forceinline__ void block_group_sums(double *sums, int64_t n, Read s) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, ng = (int)((n + 31) / 32);
  if (ng > 64) {
    double v[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const int64_t i = 32 * (int64_t)(16 * w + j) + lane;
      v[j] = i < n ? s(i) : 0.0;
    }
    if (16 * w < ng) {
      const double sum = group_sums16(v);
      if ((lane & 1) == 0) sums[16 * w + (lane >> 1)] = sum;
    }
  } else {
    for (int g = w; g < ng; g += kGroupThreads / 32) {
      const int64_t i = 32 * (int64_t)g + lane;
      const double v = group_sum(i < n ? s(i) : 0.0);
      if (lane == 0) sums[g] = v;
    }
  }
  __syncthreads();
}

// Exclusive prefix sum of 256 shared counters by one warp.
__device__ __forceinline__ void scan_bins256(int *bins, int lane) {
  int v[8], sum = 0;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    v[j] = sum;
    sum += bins[8 * lane + j];
  }
  int upto = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, upto, o);
    if (lane >= o) upto += u;
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) bins[8 * lane + j] = upto - sum + v[j];
}

// ------------------------------------------------------------------------
// Messages between the blocks of a cluster: 16 bytes into another block's
// shared memory that also count towards an mbarrier there.  A block waits on
// its own mbarrier for the bytes it expects, so it meets the others without a
// cluster barrier -- whose acquire at cluster scope empties the L1, and with it
// the table nodes that the next step reads again.
// ------------------------------------------------------------------------
__device__ __forceinline__ unsigned shared_addr(const void *p) {
  return (unsigned)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ unsigned rank_addr(unsigned addr, int rank) {
  unsigned r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void send2(unsigned dst, unsigned bar, unsigned long long a,
                                      unsigned long long b) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.b64 [%0], {%1, %2}, [%3];"
               :: "r"(dst), "l"(a), "l"(b), "r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_init(unsigned bar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(bar) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
// One thread per phase: the phase ends when `bytes` have come in.
__device__ __forceinline__ void mbar_expect(unsigned bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" :: "r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ unsigned long long now_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
// Waits of a warp for a phase; false, for all its lanes, when `limit` ns have
// passed (0: one look) or, whatever the clock says, after kMbarTries tries.
constexpr int kMbarTries = 1 << 24;
__device__ __forceinline__ bool mbar_wait(unsigned bar, unsigned parity, unsigned long long limit) {
  unsigned ok;
  asm volatile("{\n.reg .pred p;\n"
               "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n"
               "selp.b32 %0, 1, 0, p;\n}"
               : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
  if (__all_sync(0xffffffffu, ok)) return true;
  if (limit == 0) return false;
  unsigned long long start = 0;
  for (int i = 0; i < kMbarTries; ++i) {
    asm volatile("{\n.reg .pred p;\n"
                 "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
                 "selp.b32 %0, 1, 0, p;\n}"
                 : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    if (__all_sync(0xffffffffu, ok)) return true;
    const unsigned long long now = __shfl_sync(0xffffffffu, now_ns(), 0);
    if (i == 0) start = now;
    else if (now - start > limit) break;
  }
  return false;
}

// The blocks' common verdict after the last step, before any of them stores:
// true where no block gave up.  After a wait that gave up, messages may still be
// on their way to a block that has stopped waiting for them; no block leaves
// before they have come (a few us; kDrainNs, or kMbarTries looks at the clock).
// `failed` in shared memory is 0 since before the first cluster barrier.
constexpr unsigned long long kDrainNs = 1000000;
__device__ __forceinline__ bool cluster_agrees(cooperative_groups::cluster_group &cluster,
                                               unsigned *failed, bool stalled) {
  if (stalled && threadIdx.x < cluster.num_blocks())
    *cluster.map_shared_rank(failed, threadIdx.x) = 1u;
  cluster.sync();
  if (!*reinterpret_cast<volatile unsigned *>(failed)) return true;
  const unsigned long long start = now_ns();
  for (int i = 0; i < kMbarTries && now_ns() - start < kDrainNs; ++i) __nanosleep(1000);
  return false;
}

// Max over the warp of non-negative values, none NaN: their bits are ordered
// as the values are, so two 32-bit reductions replace five rounds of shuffles.
__device__ __forceinline__ double warp_max_nonneg(double v) {
  const unsigned hi = (unsigned)__double2hiint(v), lo = (unsigned)__double2loint(v);
  const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
  const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? lo : 0u);
  return __hiloint2double((int)mh, (int)ml);
}

// One cluster of L.blocks blocks.
template <typename... KArgs, typename... Args>
cudaError_t launch_cluster(void (*kernel)(KArgs...), const Loop1dShape &L, size_t smem,
                           cudaStream_t s, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(L.blocks);
  cfg.blockDim = dim3(L.threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = L.blocks;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}

// Whether this device can hold the cluster (once per solve, at its creation).
template <typename... KArgs>
bool cluster_fits(void (*kernel)(KArgs...), const Loop1dShape &L, size_t smem) {
  // the limit belongs to the kernel, not to the solve: the device's, so that a
  // smaller solve created later leaves a larger one's launches valid
  int dev = 0, most = 0;
  cudaFuncAttributes fa;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess ||
      cudaFuncGetAttributes(&fa, kernel) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  most -= (int)fa.sharedSizeBytes;
  if ((int64_t)smem > most) return false;
  cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
  cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(L.blocks);
  cfg.blockDim = dim3(L.threads);
  cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = L.blocks;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int n = 0;
  const cudaError_t e = cudaOccupancyMaxActiveClusters(&n, kernel, &cfg);
  cudaGetLastError();
  return e == cudaSuccess && n > 0;
}

}  // namespace pf5d
