// pf5d_gather.cuh -- table values (mu, M) of a block of points with the
// gathers of one table cell shared, for the kernels that evaluate every point
// once (the split rate stages): the ordering of a block's points by cell, used
// by both forms, and the FP64 values.
//
// What bounds a one-point-per-thread evaluation is not DRAM (the nodes a
// block touches stay in L1) but the path from L1 into the registers: 16 nodes
// of 80 bytes are 1280 bytes per point, and a warp-wide 16-byte load moves its
// 512 bytes in four cycles even when every lane reads the same address.  So a
// thread takes up to K points of one cell and loads each node once for all of
// them; the weights of its points are formed in registers, and the K * 9
// running sums are independent, which also feeds the FP64 pipe.
//
// A block of NT threads takes NT * PER points:
//   1. gather_add: each point's cell and fractions (interpolation.py:110-121)
//      into shared memory, and its rank among the points of its bin (a hash of
//      the cell; bin 255: outside the linear region; gather_rank).  Lanes of a
//      warp with the same bin take one atomic together, and keep their order;
//   2. gather_sort: prefix sum over the bins, the points in bin order, and
//      each bin's run cut into work items of up to K points;
//   3. gather_values: a thread evaluates an item.  Every point has its own
//      weights ((w0 w1) w2) w3 and the reference's left-to-right 16-term sums,
//      so its values do not depend on which points share the item.  A point
//      whose cell is not the item's (a hash collision) is set aside;
//   4. gather_rest: the points set aside and those outside the linear region,
//      one per thread.
// The values replace the fractions in shared memory at the point's own slot,
// for the caller to read in point order.
#pragma once

#include "pf5d_device.cuh"

namespace pf5d {

constexpr int kGatherBins = 256;
constexpr unsigned kFarCell = ~0u;                              // n^4 cells, n < 256
constexpr int kNoKey = -1;                                      // no point (past the field's edge)

template <int NT_, int PER_, int K_>
struct GatherOrder {
  static constexpr int NT = NT_, PER = PER_, K = K_, N = NT * PER;
  unsigned cell[N];                 // kFarCell: outside the linear region
  int base[kGatherBins + 1];        // points (low half) and items (high half) before each bin
  int wsum[NT / 32 + 1];
  int nleft;
  unsigned items[N / K + kGatherBins];
  unsigned short order[N];
  unsigned short left[N];
};

// FP64: fractions, then values
template <int N>
struct GatherValues {
  double2 v[4][N];                  // t0 t1 | t2 t3, then mu1 mu2 | mu3 mu4 | M_Fe M1 | M2 M3
  double v8[N];                     // M4
};
template <int NT, int PER, int K>
struct GatherSmem : GatherValues<NT * PER>, GatherOrder<NT, PER, K> {};

// Table cell of x exactly as the reference computes it (interpolation.py:103-121).
__device__ __forceinline__ bool cell64(const Table &T, const double x[S], int ii[S], double tt[S]) {
  if (!linear_region(T, x)) return false;
#pragma unroll
  for (int a = 0; a < S; ++a) axis_coord(x[a] * T.inv_step, T.n, ii[a], tt[a]);
  return true;
}

// Before the first gather_add (a barrier must follow).
template <typename G>
__device__ __forceinline__ void gather_begin(G &g, int tid) {
  for (int b = tid; b <= kGatherBins; b += G::NT) g.base[b] = 0;
  if (tid == 0) g.nleft = 0;
}

// Rank of the point in slot q in the bin of its cell (ii, where it lies in the
// linear region); returns bin and rank, key | rank << 16.  Called by the lanes
// `active` of a warp.
template <typename G>
__device__ __forceinline__ int gather_rank(G &g, unsigned active, bool linear, const int ii[S], int n,
                                           int q) {
  const int key = linear ? (int)((unsigned)(41 * ii[0] + 13 * ii[1] + 5 * ii[2] + ii[3]) %
                                 (kGatherBins - 1u))
                         : kGatherBins - 1;
  g.cell[q] = linear ? (((unsigned)ii[0] * n + ii[1]) * n + ii[2]) * n + ii[3] : kFarCell;
  const unsigned same = __match_any_sync(active, key);
  const int lane = threadIdx.x & 31, lead = __ffs(same) - 1;
  int before = 0;
  if (lane == lead) before = atomicAdd(&g.base[key], __popc(same));
  before = __shfl_sync(active, before, lead);
  return key | ((before + __popc(same & ((1u << lane) - 1u))) << 16);
}

// Point x in slot q (valid lanes only hold one); returns gather_rank's answer
// or kNoKey.  Called by whole warps.
template <typename G>
__device__ __forceinline__ int gather_add(G &g, const Table &T, bool valid, const double x[S],
                                          int q) {
  const unsigned active = __ballot_sync(0xffffffffu, valid);
  if (!valid) return kNoKey;
  int ii[S] = {0, 0, 0, 0};
  double tt[S];
  const bool linear = cell64(T, x, ii, tt);
  if (linear) {
    g.v[0][q] = make_double2(tt[0], tt[1]);
    g.v[1][q] = make_double2(tt[2], tt[3]);
  }
  return gather_rank(g, active, linear, ii, T.n, q);
}

// Points in bin order and the work items; kr: gather_add's answers for this
// thread's slots q = j * G::NT + tid.  Returns the item count.
template <typename G>
__device__ __forceinline__ int gather_sort(G &g, const int kr[G::PER], int tid) {
  constexpr int K = G::K;
  __syncthreads();
  for (int b = tid; b < kGatherBins - 1; b += G::NT) {
    const int c = g.base[b];
    g.base[b] = c | (((c + K - 1) / K) << 16);
  }
  __syncthreads();
  const int total = block_exclusive_scan<kGatherBins, G::NT>(g.base, g.wsum, tid);
  if (tid == 0) g.base[kGatherBins] = total;
  __syncthreads();
#pragma unroll
  for (int j = 0; j < G::PER; ++j) {
    if (kr[j] == kNoKey) continue;
    const int b = kr[j] & 0xffff, r = kr[j] >> 16;
    const int at = g.base[b], s = (at & 0xffff) + r;
    g.order[s] = (unsigned short)(j * G::NT + tid);
    if (b != kGatherBins - 1 && r % K == 0) {
      const int run = (g.base[b + 1] & 0xffff) - s;
      g.items[(at >> 16) + r / K] = (unsigned)s | ((unsigned)min(K, run) << 16);
    }
  }
  __syncthreads();
  return total >> 16;
}

template <typename G>
__device__ __forceinline__ void gather_put(G &g, int q, const double v[NP]) {
#pragma unroll
  for (int k = 0; k < 4; ++k) g.v[k][q] = make_double2(v[2 * k], v[2 * k + 1]);
  g.v8[q] = v[8];
}

template <typename G>
__device__ __forceinline__ void gather_get(const G &g, int q, double v[NP]) {
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const double2 a = g.v[k][q];
    v[2 * k] = a.x;
    v[2 * k + 1] = a.y;
  }
  v[8] = g.v8[q];
}

// The points that no item evaluated, one per thread: rest(q).  Barriers before
// and after.
template <typename G, typename Rest>
__device__ __forceinline__ void gather_others(G &g, int tid, Rest rest) {
  __syncthreads();
  const int far0 = g.base[kGatherBins - 1] & 0xffff;
  const int nfar = (g.base[kGatherBins] & 0xffff) - far0, n = nfar + g.nleft;
  for (int l = tid; l < n; l += G::NT) rest(l < nfar ? (int)g.order[far0 + l] : (int)g.left[l - nfar]);
  __syncthreads();
}

// The work items (gather_rest follows).
template <bool VEC, typename G>
__device__ __forceinline__ void gather_values(G &g, const Table &T, int nitems, int tid) {
  constexpr int K = G::K;
  const int64_t s3 = T.stride, s2 = (int64_t)T.n * s3, s1 = (int64_t)T.n * s2,
                s0 = (int64_t)T.n * s1;
  for (int it = tid; it < nitems; it += G::NT) {
    const unsigned e = g.items[it];
    const int s = (int)(e & 0xffffu), m = (int)(e >> 16);
    int q[K];
    double t[K][S], u[K][S];
    const unsigned cell0 = g.cell[g.order[s]];
    unsigned mine = 0;
#pragma unroll
    for (int j = 0; j < K; ++j) {
      q[j] = g.order[s + (j < m ? j : 0)];
      if (j < m) {
        if (g.cell[q[j]] == cell0) mine |= 1u << j;
        else g.left[atomicAdd(&g.nleft, 1)] = (unsigned short)q[j];
      }
      const double2 a = g.v[0][q[j]], b = g.v[1][q[j]];
      t[j][0] = a.x;
      t[j][1] = a.y;
      t[j][2] = b.x;
      t[j][3] = b.y;
#pragma unroll
      for (int d = 0; d < S; ++d) u[j][d] = 1.0 - t[j][d];
    }
    double acc[K][NP];
    const double *base = T.grid + (int64_t)cell0 * s3;
#pragma unroll
    for (int c = 0; c < 16; ++c) {
      const int b0 = (c >> 3) & 1, b1 = (c >> 2) & 1, b2 = (c >> 1) & 1, b3 = c & 1;
      const double *node = base + b0 * s0 + b1 * s1 + b2 * s2 + b3 * s3;
      double v[NP + 1];
      if (VEC) {
        const double2 *n2 = reinterpret_cast<const double2 *>(node);
#pragma unroll
        for (int k = 0; k < (NP + 1) / 2; ++k) {
          const double2 a = __ldg(n2 + k);
          v[2 * k] = a.x;
          v[2 * k + 1] = a.y;
        }
      } else {
#pragma unroll
        for (int p = 0; p < NP; ++p) v[p] = __ldg(node + p);
      }
#pragma unroll
      for (int j = 0; j < K; ++j) {
        const double w = (b0 ? t[j][0] : u[j][0]) * (b1 ? t[j][1] : u[j][1]) *
                         (b2 ? t[j][2] : u[j][2]) * (b3 ? t[j][3] : u[j][3]);
#pragma unroll
        for (int p = 0; p < NP; ++p) {
          const double term = w * v[p];
          acc[j][p] = c == 0 ? term : acc[j][p] + term;
        }
      }
    }
#pragma unroll
    for (int j = 0; j < K; ++j)
      if (mine & (1u << j)) gather_put(g, q[j], acc[j]);
  }
}

// Points set aside and points outside the linear region; point(q, x) gives
// the composition in slot q.  Ends with a barrier.
template <bool VEC, typename G, typename Point>
__device__ __forceinline__ void gather_rest(G &g, const Table &T, int tid, unsigned *flags,
                                            Point point) {
  gather_others(g, tid, [&](int q) {
    double x[S], v[NP];
    point(q, x);
    interp_point<VEC>(T, x, v, flags);
    gather_put(g, q, v);
  });
}

// The four components of a point by loads of W doubles: 4 for a field on a
// 32-byte boundary (one 256-bit load moves half the L1 wavefronts of two
// 16-byte ones, whose lanes each touch half of every line), 2 on 16 bytes.  W is
// known to the kernel: a choice at run time, in the loops, cost the split rate
// stage 5%.  p derives from an after_wait pointer where the kernel waits for
// another.
template <int W>
__device__ __forceinline__ void load_comp4(const double *p, double v[S]) {
  if constexpr (W == 4) {
    asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];"
        : "=d"(v[0]), "=d"(v[1]), "=d"(v[2]), "=d"(v[3])
        : "l"(p));
  } else if constexpr (W == 2) {
    const double2 a = __ldg(reinterpret_cast<const double2 *>(p));
    const double2 b = __ldg(reinterpret_cast<const double2 *>(p) + 1);
    v[0] = a.x;
    v[1] = a.y;
    v[2] = b.x;
    v[3] = b.y;
  } else {
#pragma unroll
    for (int c = 0; c < S; ++c) v[c] = __ldg(p + c);
  }
}
inline bool aligned_to(const void *p, size_t bytes) { return ((uintptr_t)p & (bytes - 1)) == 0; }

}  // namespace pf5d
