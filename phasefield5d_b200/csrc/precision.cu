// precision.cu -- FP32-compensated form of the step loop (the "precision
// form").  Same dataflow and tiling as the FP64 stepper (stepper.cu):
//   cuFFT R2C of the misfit -> B(k)/N multiply -> cuFFT C2R -> fused rate
//   kernel (FP32 interpolation, Laplacian, mu, one flux per face,
//   divergence, a max|dX/dt| slot per block) -> k32_dt (one block: the
//   FP64 dt controller) -> compensated update + clamp + next misfit +
//   out-of-bounds test,
// replayed from CUDA graphs.
//
// Numerics:
//   * the field is D = X - X0 as an FP32 pair (hi, lo); the update adds
//     dt*dX/dt with TwoSum and renormalises, so rounding does not
//     accumulate over thousands of steps;
//   * the table stores mu - mu(X0) (and M) in FP32, so mu gradients are
//     differences of small numbers;
//   * cell fractions come from a host FP64 split of X0/res into integer and
//     fraction plus the FP32 deviation D/res;
//   * FP64: closure X_Fe = 1 - sum X (face flux), linear-region and simplex
//     sums, dt controller, mass/mean reductions.  The k = 0 elastic mode is
//     exactly zero because B(0) = 0.
// Compiled with FMA contraction allowed; the TwoSum update uses explicit
// round-to-nearest intrinsics so it is never contracted.
#include <algorithm>
#include <cstring>
#include <map>
#include <vector>

#include <cufft.h>

#include "pf5d_cluster.cuh"
#include "pf5d_device.cuh"
#include "pf5d_fft.h"
#include "pf5d_fp32c.h"
#include "pf5d_fp32c.cuh"
#include "pf5d_gather.cuh"
#include "pf5d_host.h"
#include "pf5d_split32.cuh"
#include "pf5d_tiles.cuh"
#include "pf5d_window.cuh"

namespace pf5d {

// ------------------------------------------------------------------------
// Rate kernels (same tiling as the FP64 kernels)
// ------------------------------------------------------------------------

template <int TX, int TY, int MINB, bool WIN, int SORT = 0, bool PERPOINT = false>
__global__ void __launch_bounds__(TX * TY, MINB) k32_rate_tile2d(Rate32 P) {
  pdl_wait();
  if (P.st->halt) return;
  extern __shared__ float4 sm4[];
  const int tid = threadIdx.y * TX + threadIdx.x;
  unsigned flags = 0;
  const float vmax = tile2d32_body<TX, TY, WIN, SORT, PERPOINT>(P, blockIdx.x, blockIdx.y, sm4,
                                                               &flags, tid);
  raise_rate_flags(P.st, flags);
  finish_rate32(P, vmax, Tile2dSmem32<TX, TY, SORT>::red(sm4));
}

template <int TX, int TY, int SORT = 0>
constexpr size_t tile2d32_smem() {
  return Tile2dSmem32<TX, TY, SORT>::bytes;
}

template <int TX, int TY, int MINB, bool WIN, int SORT = 0>
__global__ void __launch_bounds__(TX * TY, MINB) k32_rate_march3d(Rate32 P, int zc) {
  using G = PlaneGeom<TX, TY>;
  pdl_wait();
  if (P.st->halt) return;
  extern __shared__ float4 sm4[];
  float4 *win = sm4;
  double *red = reinterpret_cast<double *>(win + kWinNodes32 * 3);
  float *Xs = reinterpret_cast<float *>(red + G::NT / 32);      // [3][S][PX]
  float *Ms = Xs + 3 * S * G::PX;                                // [2][NPM][PM]
  float *Fx = Ms + 2 * NPM * G::PM;
  float *Fy = Fx + S * G::NFX;
  int *wred = reinterpret_cast<int *>(Fy + S * G::NFY);
  int *win_lo = wred + S * (G::NT / 32);
  int *wx = win_lo + S + 1;
  int *wy = wx + G::HX;
  SortScratch32 ss{};
  if constexpr (SORT) ss = SortBytes32<TX, TY>::carve(wy + G::HY);
  const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * TX + tx;
  const int x0 = blockIdx.x * TX, y0 = blockIdx.y * TY;
  const int zb = blockIdx.z * zc;
  const int ze = min(zb + zc, P.nz);
  const int64_t plane = (int64_t)P.ny * P.nx;
  unsigned flags = 0;
  if (tid == 0) win_lo[S] = 0;
  for (int i = tid; i < G::HX + G::HY; i += G::NT) {
    if (i < G::HX) wx[i] = wrap_any(x0 + i - 2, P.nx);
    else wy[i - G::HX] = wrap_any(y0 + (i - G::HX) - 2, P.ny);
  }
  auto xplane = [&](int z) { return Xs + ((z - zb + 3) % 3) * S * G::PX; };
  auto mplane = [&](int z) { return Ms + ((z - zb + 2) & 1) * NPM * G::PM; };
  auto load_x = [&](int z) {
    load_plane32<TX, TY>(P.D, (int64_t)wrap_any(z, P.nz) * plane, wx, wy, P.nx, xplane(z), tid);
  };
  auto compute_mu = [&](int z, bool interior_only) {
    mu_plane32<TX, TY, 3, WIN, SORT>(P, xplane(z - 1), xplane(z), xplane(z + 1), mplane(z),
                                     (int64_t)wrap_any(z, P.nz) * plane, wx, wy, interior_only,
                                     win, wred, win_lo, &flags, tid, ss);
  };
  const int pX = (ty + 2) * G::HX + (tx + 2);
  const int pM = (ty + 1) * G::MX + (tx + 1);
  const bool in_tile = (x0 + tx < P.nx) && (y0 + ty < P.ny);
  __syncthreads();
  load_x(zb - 2);
  load_x(zb - 1);
  load_x(zb);
  __syncthreads();
  compute_mu(zb - 1, true);
  __syncthreads();
  load_x(zb + 1);
  __syncthreads();
  compute_mu(zb, false);
  __syncthreads();
  float Jm[S];
  face32_between<G::PX, G::PM>(P, xplane(zb - 1), mplane(zb - 1), pX, pM, xplane(zb), mplane(zb),
                               pX, pM, Jm);
  float vmax = 0.f;
  for (int z = zb; z < ze; ++z) {
    __syncthreads();
    load_x(z + 2);
    __syncthreads();
    compute_mu(z + 1, false);
    __syncthreads();
    float Jz[S];
    face32_between<G::PX, G::PM>(P, xplane(z), mplane(z), pX, pM, xplane(z + 1), mplane(z + 1),
                                 pX, pM, Jz);
    plane_faces32<TX, TY>(P, xplane(z), mplane(z), Fx, Fy, tid);
    __syncthreads();
    if (in_tile) {
      float out[S];
#pragma unroll
      for (int c = 0; c < S; ++c) {
        const float ay = __fsub_rn(Fy[c * G::NFY + (ty + 1) * TX + tx], Fy[c * G::NFY + ty * TX + tx]);
        const float ax = __fsub_rn(Fx[c * G::NFX + ty * (TX + 1) + tx + 1],
                                   Fx[c * G::NFX + ty * (TX + 1) + tx]);
        out[c] = __fmul_rn(__fadd_rn(__fadd_rn(__fsub_rn(Jz[c], Jm[c]), ay), ax), P.flux_scale);
      }
      store_rate(P.dX, (int64_t)z * plane + (int64_t)(y0 + ty) * P.nx + (x0 + tx), out, vmax);
    }
#pragma unroll
    for (int c = 0; c < S; ++c) Jm[c] = Jz[c];
  }
  raise_rate_flags(P.st, flags);
  finish_rate32(P, vmax, red);
}

template <int TX, int TY, int SORT = 0>
constexpr size_t march3d32_smem() {
  using G = PlaneGeom<TX, TY>;
  return Smem32Tail<TX, TY>::bytes +
         (3 * S * G::PX + 2 * NPM * G::PM + S * G::NFX + S * G::NFY) * sizeof(float) +
         (SORT ? SortBytes32<TX, TY>::bytes : 0);
}

template <int TX>
__global__ void __launch_bounds__(TX) k32_rate_1d(Rate32 P) {
  pdl_wait();
  if (P.st->halt) return;
  constexpr int HX = TX + 4, MX = TX + 2;
  __shared__ float Xs[S][HX];
  __shared__ float Ms[NPM][MX];
  __shared__ float Fx[S][TX + 1];
  __shared__ double red[(TX + 31) / 32];
  const int tx = threadIdx.x;
  const int x0 = blockIdx.x * TX;
  const int n = P.nx;
  unsigned flags = 0;
  for (int pos = tx; pos < HX; pos += TX) {
    const float4 v = __ldg(P.D + wrap_any(x0 + pos - 2, n));
    Xs[0][pos] = v.x;
    Xs[1][pos] = v.y;
    Xs[2][pos] = v.z;
    Xs[3][pos] = v.w;
  }
  __syncthreads();
  for (int pos = tx; pos < MX; pos += TX) {
    const int px = pos + 1;
    float d[S], lap[S];
#pragma unroll
    for (int c = 0; c < S; ++c) {
      d[c] = Xs[c][px];
      const float nb[2] = {Xs[c][px + 1], Xs[c][px - 1]};
      lap[c] = lap32<2>(nb, d[c], P.inv_dx2);
    }
    const float spv = P.sp ? __ldg(P.sp + wrap_any(x0 + pos - 1, n)) : 0.f;
    float v[NPM];
    chem32(P, d, lap, spv, nullptr, nullptr, v, &flags);
#pragma unroll
    for (int r = 0; r < NPM; ++r) Ms[r][pos] = v[r];
  }
  __syncthreads();
  for (int f = tx; f < TX + 1; f += TX) {
    float J[S];
    face32_between<HX, MX>(P, &Xs[0][0], &Ms[0][0], f + 1, f, &Xs[0][0], &Ms[0][0], f + 2, f + 1,
                           J);
#pragma unroll
    for (int c = 0; c < S; ++c) Fx[c][f] = J[c];
  }
  __syncthreads();
  float vmax = 0.f;
  if (x0 + tx < n) {
    float out[S];
#pragma unroll
    for (int c = 0; c < S; ++c) out[c] = (Fx[c][tx + 1] - Fx[c][tx]) * P.flux_scale;
    store_rate(P.dX, x0 + tx, out, vmax);
  }
  raise_rate_flags(P.st, flags);
  finish_rate32(P, vmax, red);
}

// ------------------------------------------------------------------------
// Compensated update, clamp, next misfit, out-of-bounds test
// ------------------------------------------------------------------------
struct Update32 {
  float4 *hi, *lo;
  const float4 *dX;
  int64_t npts;
  StepState32 *st;
  double x0[S];
  double sum_x0;
  float lvec[S];
  float *s;          // next misfit or nullptr
  int oob_interval;
};

// One point's compensated update and clamp: (h, l) += dtf * r, the simplex
// clamp on X = X0 + D in FP64; dd is the new D in FP64.
__device__ __forceinline__ void update_point32(const Update32 &U, float dtf, const float r[S],
                                               float h[S], float l[S], double dd[S]) {
#pragma unroll
  for (int c = 0; c < S; ++c) comp_add(h[c], l[c], __fmul_rn(dtf, r[c]));
  double dsum = 0.0;
#pragma unroll
  for (int c = 0; c < S; ++c) {
    dd[c] = (double)h[c] + (double)l[c];
    dsum = dsum + dd[c];
  }
  const double total = U.sum_x0 + dsum;
  if (total > 1.0) {
    const double inv = 1.0 / total;
#pragma unroll
    for (int c = 0; c < S; ++c) {
      const double dn = (U.x0[c] + dd[c]) * inv - U.x0[c];
      h[c] = (float)dn;
      l[c] = (float)(dn - (double)h[c]);
      dd[c] = (double)h[c] + (double)l[c];
    }
  }
}

__global__ void k32_update(Update32 U) {
  pdl_wait();
  StepState32 *st = U.st;
  if (st->hold) return;
  const float dtf = (float)st->dt;
  const bool check = U.oob_interval > 0 && (st->step % U.oob_interval) == 0;
  unsigned f = 0;
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < U.npts;
       p += (int64_t)gridDim.x * blockDim.x) {
    const float4 H = U.hi[p], L = U.lo[p], R = U.dX[p];
    float h[S] = {H.x, H.y, H.z, H.w}, l[S] = {L.x, L.y, L.z, L.w};
    const float r[S] = {R.x, R.y, R.z, R.w};
    double dd[S];
    update_point32(U, dtf, r, h, l, dd);
    U.hi[p] = make_float4(h[0], h[1], h[2], h[3]);
    U.lo[p] = make_float4(l[0], l[1], l[2], l[3]);
    if (U.s) {
      float acc = 0.f;
#pragma unroll
      for (int c = 0; c < S; ++c) acc = fmaf(h[c] + l[c], U.lvec[c], acc);
      U.s[p] = acc;
    }
    if (check) {
      double x[S];
#pragma unroll
      for (int c = 0; c < S; ++c) x[c] = U.x0[c] + dd[c];
      f |= oob_flags_x(x);
    }
  }
  raise32(st, f);
}

__global__ void k32_split(const double *__restrict__ X, int64_t npts, Update32 U) {
  unsigned f = 0;
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < npts;
       p += (int64_t)gridDim.x * blockDim.x) {
    float h[S], l[S];
    double x[S];
#pragma unroll
    for (int c = 0; c < S; ++c) {
      x[c] = X[4 * p + c];
      const double d = x[c] - U.x0[c];
      h[c] = (float)d;
      l[c] = (float)(d - (double)h[c]);
    }
    U.hi[p] = make_float4(h[0], h[1], h[2], h[3]);
    U.lo[p] = make_float4(l[0], l[1], l[2], l[3]);
    if (U.s) {
      float acc = 0.f;
#pragma unroll
      for (int c = 0; c < S; ++c) acc = fmaf(h[c] + l[c], U.lvec[c], acc);
      U.s[p] = acc;
    }
    if (U.oob_interval > 0) f |= oob_flags_x(x);
  }
  raise32(U.st, f);
}

__global__ void k32_join(const float4 *__restrict__ hi, const float4 *__restrict__ lo,
                         int64_t npts, Update32 U, double *__restrict__ X) {
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < npts;
       p += (int64_t)gridDim.x * blockDim.x) {
    const float4 H = hi[p], L = lo[p];
    const float h[S] = {H.x, H.y, H.z, H.w}, l[S] = {L.x, L.y, L.z, L.w};
#pragma unroll
    for (int c = 0; c < S; ++c) X[4 * p + c] = U.x0[c] + ((double)h[c] + (double)l[c]);
  }
}

constexpr int kMassBlocks = 512;

// FP64 per-component sums of X = X0 + hi + lo; two passes, deterministic.
__global__ void k32_mass_partial(const float4 *__restrict__ hi, const float4 *__restrict__ lo,
                                 int64_t npts, double *partial) {
  __shared__ double red[S][8];
  double acc[S] = {0.0, 0.0, 0.0, 0.0};
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < npts;
       p += (int64_t)gridDim.x * blockDim.x) {
    const float4 H = hi[p], L = lo[p];
    acc[0] += (double)H.x + (double)L.x;
    acc[1] += (double)H.y + (double)L.y;
    acc[2] += (double)H.z + (double)L.z;
    acc[3] += (double)H.w + (double)L.w;
  }
#pragma unroll
  for (int c = 0; c < S; ++c) {
    double v = acc[c];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) red[c][threadIdx.x >> 5] = v;
  }
  __syncthreads();
  if (threadIdx.x < S) {
    double v = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) v += red[threadIdx.x][w];
    partial[blockIdx.x * S + threadIdx.x] = v;
  }
}

__global__ void k32_mass_final(const double *partial, int nparts, double *out) {
  if (threadIdx.x < S) {
    double v = 0.0;
    for (int b = 0; b < nparts; ++b) v += partial[b * S + threadIdx.x];
    out[threadIdx.x] = v;
  }
}

// Split rate evaluation (pf5d_split32.cuh): mu/M of a 1D/2D/3D field, then
// the faces and the divergence of a 2D or 3D one.
// LONGY: as k_chem's.
template <int DIM, int PER, int K, int MINB, bool LONGY = false>
__global__ void __launch_bounds__(kChemNT32, MINB) k32_chem(Rate32 P) {
  using G = ChemTile32<DIM, PER>;
  __shared__ GatherSmem32<kChemNT32, PER, K> g;
  pdl_wait();
  if (P.st->halt) return;
  chem32_body<DIM, PER, K>(P, g, (LONGY ? blockIdx.y : blockIdx.x) * G::BX,
                           (LONGY ? blockIdx.x : blockIdx.y) * G::BY, blockIdx.z * G::BZ);
}

template <int DIM, int PER, int K, int MINB, bool LONGY = false>
void launch_chem32(cudaStream_t s, const Rate32 &P) {
  using G = ChemTile32<DIM, PER>;
  const unsigned gx = (unsigned)((P.nx + G::BX - 1) / G::BX), gy = (unsigned)((P.ny + G::BY - 1) / G::BY);
  const dim3 g(LONGY ? gy : gx, LONGY ? gx : gy, (unsigned)((P.nz + G::BZ - 1) / G::BZ));
  launch_pdl(k32_chem<DIM, PER, K, MINB, LONGY>, g, dim3(kChemNT32), 0, s, P);
}

// A save step's, for any size (the FP64 form's launch_chem_save): 24x24 156 ->
// 148 us, 8192 points 141 -> 138.
template <int DIM>
void launch_chem32_save(cudaStream_t s, const Rate32 &P) {
  if (DIM == 3 && P.ny > 65535 * ChemTile32<3, 4>::BY) launch_chem32<3, 4, 2, 6, true>(s, P);
  else if (P.npts < 65536) launch_chem32<DIM, 1, 2, 6>(s, P);
  else launch_chem32<DIM, 4, 4, 4>(s, P);
}

template <int DIM, int R, int MINB>
__global__ void __launch_bounds__(kFluxThreads32, MINB) k32_flux(Rate32 P, int rows) {
  __shared__ double red[kFluxThreads32 / 32];
  pdl_wait();
  if (P.st->halt) return;
  const float vmax = flux32_body<DIM, R>(P, blockIdx.x, blockIdx.y, blockIdx.z, rows);
  finish_rate32(P, vmax, red);
}

// The dt controller after a rate launch of `nparts` blocks: a block-wide
// max over the slots, then the FP64 rule in thread 0.
constexpr int kDt32Threads = 1024;
__global__ void __launch_bounds__(kDt32Threads) k32_dt(Rate32 P, int nparts) {
  __shared__ double red[kDt32Threads / 32];
  pdl_wait();
  StepState32 *st = P.st;
  if (halted_before_dt(st)) return;
  double m = 0.0;
  for (int i = threadIdx.x; i < nparts; i += kDt32Threads) m = fmax(m, P.partial[i]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < kDt32Threads / 32; ++w) m = fmax(m, red[w]);
    double dt = st->dt;
    if (P.adaptive) dt = adaptive_dt(dt, m, P.ctld, P.t_cfl, P.lower, P.upper, P.factor);
    st->dt = dt;
    st->time = st->time + dt;
    st->xdotmax = m;
    st->step = st->step + 1;
  }
}

// The 1D elastic term in closed form, in place: s -> s' = bn (s - mean s) +
// b0 mean s (bn: B(k) for every k != 0, b0: B(0)), i.e. irfft(B rfft(s))
// exactly (elastic.py:250-263); the mean and the product in FP64, s' rounded
// once to FP32.  One block; the mean is summed in the order of
// pf5d_cluster.cuh, as k32_loop1d sums it.
constexpr int kElastic1dThreads32 = kGroupThreads;
constexpr int64_t kElastic1dMax32 = kLoop1dMax;
__global__ void __launch_bounds__(kElastic1dThreads32)
    k32_elastic1d(float *s, int64_t n, double bn, double b0, const unsigned *halt) {
  __shared__ double sums[kLoop1dGroups];
  pdl_wait();
  if (*halt) return;
  const int t = threadIdx.x, ng = (int)((n + 31) / 32);
  block_group_sums(sums, n, [&](int64_t i) { return (double)s[i]; });
  const double mean = sum_groups(sums, ng) / (double)n;
  for (int64_t i = t; i < n; i += kElastic1dThreads32)
    s[i] = (float)(bn * ((double)s[i] - mean) + b0 * mean);
}

// ------------------------------------------------------------------------
// 1D step loop of the precision form: the FP64 form's k_loop1d (same blocks,
// messages and order of the phases) on the FP32 pair.  A halo entry brings the
// neighbour point's hi part and its misfit.  Values are formed as
// k32_elastic1d, k32_rate_1d, k32_dt and k32_update form them.
//
// Bound by the latency of a step's dependent phases.  Steps of a long run,
// four kernels -> here: 203 points 10.3 -> 2.3 us, 1280 10.7 -> 2.5, 4112 11.4
// -> 3.9, 16384 13.1 -> 9.0.
// ------------------------------------------------------------------------
struct Loop1dSmem32 {
  ulonglong2 sums[kLoop1dGroups];        // B: misfit sum (bits) and flags of every group
  ulonglong2 max[kLoop1dBlocks * (kLoop1dThreads / 32)];   // A: max |dX/dt| (bits), flags
  ulonglong2 halo[4][2];                 // B: positions -2, -1, m, m + 1: hi; misfit
  double own[kLoop1dGroups];             // this block's groups, before they are sent
  unsigned own_flags[kLoop1dGroups];
  double mean;
  unsigned failed, pad;                  // a block gave up
  unsigned long long bar_a, bar_b;
  int bins[256];                         // of the cell sort
};
// then hi [chunk + 4], lo [chunk], per position mu (table), -kappa lap, M_1..4
// and (M_Fe, X_Fe) [chunk + 2], faces [chunk + 1], dX/dt [chunk], the misfit
// [chunk + 2], order [chunk + 2] (16 bit)
inline size_t loop1d_smem32(int chunk) {
  return sizeof(Loop1dSmem32) + sizeof(float4) * (size_t)(3 * chunk + 4 + 3 * (chunk + 2) + chunk + 1) +
         sizeof(float2) * (chunk + 2) + sizeof(float) * (chunk + 2) +
         sizeof(unsigned short) * (chunk + 2);
}
constexpr int kLoop1dResort32 = 128;

template <int MAXT>
__global__ void __launch_bounds__(MAXT, 1)
    k32_loop1d(Rate32 P, Update32 U, double bn, double b0, int chunk, int nsteps,
               unsigned long long limit) {
  cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  extern __shared__ __align__(16) unsigned char lraw[];
  Loop1dSmem32 &sm = *reinterpret_cast<Loop1dSmem32 *>(lraw);
  const int MX = chunk + 2;
  float4 *Hs = reinterpret_cast<float4 *>(lraw + sizeof(Loop1dSmem32));
  float4 *Ls = Hs + chunk + 4, *Vs = Ls + chunk, *Ks = Vs + MX, *Ms = Ks + MX, *Fs = Ms + MX,
         *Ds = Fs + chunk + 1;
  float2 *Es = reinterpret_cast<float2 *>(Ds + chunk);
  float *Qs = reinterpret_cast<float *>(Es + MX);
  unsigned short *order = reinterpret_cast<unsigned short *>(Qs + MX);
  StepState32 *st = P.st;
  if (st->halt) return;
  const int n = P.nx, t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int nw = (int)blockDim.x >> 5, nt = (int)blockDim.x - 32;   // the last warp sums
  const bool worker = t < nt;
  const int rank = (int)cluster.block_rank(), nb = (int)cluster.num_blocks();
  const int i0 = rank * chunk, m = min(chunk, n - i0);     // m > 0 (loop1d_shape)
  const int ng = (n + 31) / 32;
  const unsigned bar_a = shared_addr(&sm.bar_a), bar_b = shared_addr(&sm.bar_b);
  const unsigned bytes_a = 16u * nb * nw, bytes_b = 16u * ng + sizeof(sm.halo);
  double dt = st->dt, time = st->time, xdotmax = st->xdotmax;
  long long step = st->step;
  int to_check = U.oob_interval > 0 ? U.oob_interval - (int)(step % U.oob_interval) : -1;
  unsigned flags = 0;
  bool halt = false, stalled = false, checked = false;

  auto misfit = [&](const float4 &h, const float4 &l) {
    float acc = fmaf(h.x + l.x, U.lvec[0], 0.f);
    acc = fmaf(h.y + l.y, U.lvec[1], acc);
    acc = fmaf(h.z + l.z, U.lvec[2], acc);
    return fmaf(h.w + l.w, U.lvec[3], acc);
  };
  // The halo entry this thread keeps current: entry h of block b holds the
  // point at Hs index hsrc of this block (none: hsrc < 0).  4 * nb <= threads.
  int hsrc = -1;
  unsigned hdst = 0, hbar = 0;
  {
    const int b = t >> 2, h = t & 3;
    if (b < nb) {
      const int bm = min(chunk, n - b * chunk);
      const int src = wrap_any(b * chunk + (h < 2 ? h - 2 : bm + h - 2), n) - i0;
      if (src >= 0 && src < m) {
        hsrc = src + 2;
        hdst = rank_addr(shared_addr(sm.halo[h]), b);
        hbar = rank_addr(bar_b, b);
      }
    }
  }
  auto send_b = [&]() {
    for (int g = warp; 32 * g < m; g += nw)
      if (lane < nb)
        send2(rank_addr(shared_addr(&sm.sums[i0 / 32 + g]), lane), rank_addr(bar_b, lane),
              (unsigned long long)__double_as_longlong(sm.own[g]), sm.own_flags[g]);
    if (hsrc >= 0) {
      const ulonglong2 h = *reinterpret_cast<const ulonglong2 *>(Hs + hsrc);
      send2(hdst, hbar, h.x, h.y);
      send2(hdst + 16, hbar, __float_as_uint(Qs[hsrc - 1]), 0);
    }
  };
  // 32 points from p0 (s: this lane's misfit): their sum and flags
  auto keep_group = [&](float s, int p0, unsigned f) {
    const double v = P.sp ? group_sum(p0 + lane < m ? (double)s : 0.0) : 0.0;
    const unsigned any = __reduce_or_sync(0xffffffffu, f);
    if (lane == 0) {
      sm.own[p0 >> 5] = v;
      sm.own_flags[p0 >> 5] = any;
    }
  };
  // positions in the order of their cells (a counting sort over cell_hash_u)
  auto sort_cells = [&]() {
    for (int b = t; b < 256; b += (int)blockDim.x) sm.bins[b] = 0;
    __syncthreads();
    auto key = [&](int pos) {
      const float4 h = Hs[pos + 1];
      const float d[S] = {h.x, h.y, h.z, h.w};
      float u[S];
#pragma unroll
      for (int c = 0; c < S; ++c) u[c] = fmaf(d[c], P.T.inv_step_f, P.T.fb[c]) + (float)P.T.ib[c];
      return cell_hash_u(u);
    };
    for (int pos = t; pos < m + 2; pos += (int)blockDim.x) atomicAdd(&sm.bins[key(pos)], 1);
    __syncthreads();
    if (warp == 0) scan_bins256(sm.bins, lane);
    __syncthreads();
    for (int pos = t; pos < m + 2; pos += (int)blockDim.x)
      order[atomicAdd(&sm.bins[key(pos)], 1)] = (unsigned short)pos;
    __syncthreads();
  };

  if (t == 0) {
    sm.failed = 0;
    mbar_init(bar_a);
    mbar_init(bar_b);
  }
  for (int p0 = 32 * warp; p0 < m; p0 += 32 * nw) {
    const int p = p0 + lane;
    float s = 0.f;
    if (p < m) {
      const float4 h = U.hi[i0 + p], l = U.lo[i0 + p];
      Hs[p + 2] = h;
      Ls[p] = l;
      s = misfit(h, l);
      Qs[p + 1] = s;
    }
    keep_group(s, p0, 0);
  }
  __syncthreads();
  cluster.sync();                        // every block has started and set up its barriers
  if (t == 0) mbar_expect(bar_b, bytes_b);
  send_b();

  for (int k = 0; k <= nsteps; ++k) {
    // B of the step before (k = 0: the state at the launch)
    if (!stalled && !halt) stalled = !mbar_wait(bar_b, (unsigned)k & 1u, limit);
    if (t < 4) {                         // halo entries into the chunk's rows
      const int p = t < 2 ? t : m + t;
      *reinterpret_cast<ulonglong2 *>(Hs + p) = sm.halo[t][0];
      if (t == 1 || t == 2) Qs[p - 1] = __uint_as_float((unsigned)sm.halo[t][1].x);
    }
    if (checked) {
      unsigned f = 0;
      for (int g = lane; g < ng; g += 32) f |= (unsigned)sm.sums[g].y;
      f = __reduce_or_sync(0xffffffffu, f);
      flags |= f;
      if (f & (PF5D_FLAG_NONFINITE | PF5D_FLAG_OOB_HARD)) halt = true;
    }
    stalled = __syncthreads_or(stalled);
    if (halt || stalled || k == nsteps) break;
    if (k % kLoop1dResort32 == 0) sort_cells();
    unsigned nn = 0;
    if (worker) {
      for (int w = t; w < m + 2; w += nt) {
        const int pos = order[w];
        const float4 h = Hs[pos + 1], hp = Hs[pos + 2], hm = Hs[pos];
        const float d[S] = {h.x, h.y, h.z, h.w};
        const double sd = dsum32(d);
        float v[NP];
        interp32(P, d, sd, nullptr, nullptr, v, &nn);
        const float np[S] = {hp.x, hp.y, hp.z, hp.w}, nm[S] = {hm.x, hm.y, hm.z, hm.w};
        float lk[S];
#pragma unroll
        for (int c = 0; c < S; ++c) {
          const float nb2[2] = {np[c], nm[c]};
          lk[c] = -lap32<2>(nb2, d[c], P.inv_dx2) * P.kappa[c];
        }
        Vs[pos] = make_float4(v[0], v[1], v[2], v[3]);
        Ks[pos] = make_float4(lk[0], lk[1], lk[2], lk[3]);
        Ms[pos] = make_float4(v[5], v[6], v[7], v[8]);
        Es[pos] = make_float2(v[4], (float)(P.c_fe - sd));
      }
    } else {
      if (lane == 0) {
        mbar_expect(bar_a, bytes_a);
        mbar_expect(bar_b, bytes_b);
      }
      if (P.sp) {
        double total = 0.0;
        for (int g = lane; g < ng; g += 32)
          total = total + __longlong_as_double((long long)sm.sums[g].x);
        total = group_sum(total);
        if (lane == 0) sm.mean = total / (double)n;
      }
    }
    __syncthreads();
    // face i lies between mu/M positions i and i+1 (hi positions i+1, i+2)
    const double mean = P.sp ? sm.mean : 0.0;
    auto mu_at = [&](int q) {
      const float spv = P.sp ? (float)(bn * ((double)Qs[q] - mean) + b0 * mean) : 0.f;
      const float4 v = Vs[q], k4 = Ks[q];
      return make_float4(v.x + fmaf(spv, P.lvec[0], k4.x), v.y + fmaf(spv, P.lvec[1], k4.y),
                         v.z + fmaf(spv, P.lvec[2], k4.z), v.w + fmaf(spv, P.lvec[3], k4.w));
    };
    for (int i = t; i < m + 1; i += (int)blockDim.x)
      Fs[i] = face_flux32(P, Hs[i + 1], mu_at(i), Ms[i], Es[i], Hs[i + 2], mu_at(i + 1), Ms[i + 1],
                          Es[i + 1]);
    __syncthreads();
    float vmax32 = 0.f;
    for (int p = t; p < m; p += (int)blockDim.x) {
      const float4 a = Fs[p + 1], b = Fs[p];
      const float4 d = make_float4((a.x - b.x) * P.flux_scale, (a.y - b.y) * P.flux_scale,
                                   (a.z - b.z) * P.flux_scale, (a.w - b.w) * P.flux_scale);
      Ds[p] = d;
      vmax32 = fmaxf(vmax32, fabsf(d.x));
      vmax32 = fmaxf(vmax32, fabsf(d.y));
      vmax32 = fmaxf(vmax32, fabsf(d.z));
      vmax32 = fmaxf(vmax32, fabsf(d.w));
    }
    // non-negative floats are ordered as their bits
    vmax32 = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(vmax32)));
    nn = __reduce_or_sync(0xffffffffu, nn);
    if (lane < nb)
      send2(rank_addr(shared_addr(&sm.max[rank * nw + warp]), lane), rank_addr(bar_a, lane),
            __float_as_uint(vmax32), nn);
    stalled = !mbar_wait(bar_a, (unsigned)k & 1u, limit);           // A
    unsigned gbits = 0;
    nn = 0;
    for (int i = lane; i < nb * nw; i += 32) {
      gbits = max(gbits, (unsigned)sm.max[i].x);
      nn |= (unsigned)sm.max[i].y;
    }
    const double gmax = (double)__uint_as_float(__reduce_max_sync(0xffffffffu, gbits));
    nn = __reduce_or_sync(0xffffffffu, nn);
    flags |= nn;
    // an error of the fallback, the same in every block: stop before the update
    halt = !stalled && (nn & kNNErrorFlags);
    if (!stalled && !halt) {
      if (P.adaptive) dt = adaptive_dt(dt, gmax, P.ctld, P.t_cfl, P.lower, P.upper, P.factor);
      time = time + dt;
      xdotmax = gmax;
      step = step + 1;
      checked = --to_check == 0;
      if (checked) to_check = U.oob_interval;
      const float dtf = (float)dt;
      for (int p0 = 32 * warp; p0 < m; p0 += 32 * nw) {
        const int p = p0 + lane;
        unsigned fo = 0;
        float s = 0.f;
        if (p < m) {
          const float4 H = Hs[p + 2], L = Ls[p], R = Ds[p];
          float h[S] = {H.x, H.y, H.z, H.w}, l[S] = {L.x, L.y, L.z, L.w};
          const float r[S] = {R.x, R.y, R.z, R.w};
          double dd[S];
          update_point32(U, dtf, r, h, l, dd);
          const float4 hn = make_float4(h[0], h[1], h[2], h[3]), ln = make_float4(l[0], l[1], l[2], l[3]);
          Hs[p + 2] = hn;
          Ls[p] = ln;
          s = misfit(hn, ln);
          Qs[p + 1] = s;
          if (checked) {
            double x[S];
#pragma unroll
            for (int c = 0; c < S; ++c) x[c] = U.x0[c] + dd[c];
            fo = oob_flags_x(x);
          }
        }
        keep_group(s, p0, fo);
      }
    }
    __syncthreads();
    // a warp that gave up leaves with its block, after the next barrier
    if (!stalled && !halt) send_b();
  }

  if (cluster_agrees(cluster, &sm.failed, stalled)) {
    for (int p = t; p < m; p += (int)blockDim.x) {
      U.hi[i0 + p] = Hs[p + 2];
      U.lo[i0 + p] = Ls[p];
      P.dX[i0 + p] = Ds[p];
      if (U.s) U.s[i0 + p] = Qs[p + 1];
    }
    if (rank == 0 && t == 0) {
      st->dt = dt;
      st->time = time;
      st->xdotmax = xdotmax;
      st->step = step;
      if (flags) atomicOr(&st->flags, flags);
      if (halt) atomicExch(&st->halt, 1u);
    }
  } else if (rank == 0 && t == 0) {
    atomicOr(&st->flags, PF5D_FLAG_STALLED);
    atomicExch(&st->halt, 1u);
  }
}

__global__ void k32_bmul(cufftComplex *__restrict__ k, const float *__restrict__ bk, int64_t nk,
                         const unsigned *halt) {
  if (halt && *halt) return;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nk;
       i += (int64_t)gridDim.x * blockDim.x) {
    const float b = bk[i];
    cufftComplex v = k[i];
    v.x *= b;
    v.y *= b;
    k[i] = v;
  }
}

// ------------------------------------------------------------------------
// Host side
// ------------------------------------------------------------------------
constexpr int kTX1_32 = 128;
constexpr int kGraphSteps32 = 50;

struct Variant32 {
  int tx, ty, minb;
  int ty2 = 0;                  // rows of a 2D tile, where not ty
  bool split;
  size_t smem2d, smem3d;
  void (*set_attrs)();
  void (*launch2d)(dim3, dim3, size_t, cudaStream_t, const Rate32 &);
  void (*launch3d)(dim3, dim3, size_t, cudaStream_t, const Rate32 &, int);
  std::string (*kernels)(int dim);     // the kernel instances of a 2D/3D rate stage
};

template <int TX, int TY, int MINB, bool WIN = true, int SORT = 0, bool PP = false>
Variant32 make_variant32() {
  Variant32 v;
  v.tx = TX;
  v.ty = TY;
  v.minb = MINB;
  v.split = false;
  v.smem2d = tile2d32_smem<TX, TY, SORT>();
  v.smem3d = march3d32_smem<TX, TY, SORT>();
  v.set_attrs = []() {
    const auto a = cudaFuncAttributeMaxDynamicSharedMemorySize;
    cudaFuncSetAttribute(k32_rate_tile2d<TX, TY, MINB, WIN, SORT, PP>, a,
                         (int)tile2d32_smem<TX, TY, SORT>());
    cudaFuncSetAttribute(k32_rate_march3d<TX, TY, MINB, WIN, SORT>, a,
                         (int)march3d32_smem<TX, TY, SORT>());
  };
  v.launch2d = [](dim3 g, dim3 b, size_t sm, cudaStream_t s, const Rate32 &P) {
    launch_pdl(k32_rate_tile2d<TX, TY, MINB, WIN, SORT, PP>, g, b, sm, s, P);
  };
  v.launch3d = [](dim3 g, dim3 b, size_t sm, cudaStream_t s, const Rate32 &P, int zc) {
    launch_pdl(k32_rate_march3d<TX, TY, MINB, WIN, SORT>, g, b, sm, s, P, zc);
  };
  v.kernels = [](int dim) {
    if (dim == 2) return kname("k32_rate_tile2d", {TX, TY, MINB, WIN, SORT, PP});
    return kname("k32_rate_march3d", {TX, TY, MINB, WIN, SORT});
  };
  return v;
}

// Split variant: k32_chem, then k32_flux; in 2D a warp marches over ROWS rows
// (in 3D grid32_of sets the planes of a chunk).
template <int ROWS, int R, int MINB, int PER, int K, int KMINB>
Variant32 make_split_variant32() {
  Variant32 v;
  v.tx = kFluxCols32;
  v.ty = 4 * R;
  v.ty2 = 4 * ROWS;
  v.minb = MINB;
  v.split = true;
  v.smem2d = v.smem3d = 0;
  v.set_attrs = []() {};
  v.launch2d = [](dim3 g, dim3, size_t, cudaStream_t s, const Rate32 &P) {
    launch_chem32<2, PER, K, KMINB>(s, P);
    launch_pdl(k32_flux<2, 1, MINB>, g, dim3(kFluxThreads32), 0, s, P, ROWS);
  };
  v.launch3d = [](dim3 g, dim3, size_t, cudaStream_t s, const Rate32 &P, int zc) {
    launch_chem32<3, PER, K, KMINB>(s, P);
    launch_pdl(k32_flux<3, R, MINB>, g, dim3(kFluxThreads32), 0, s, P, zc);
  };
  v.kernels = [](int dim) {
    return kname("k32_chem", {dim, PER, K, KMINB, 0}) + " + " +
           kname("k32_flux", {dim, dim == 2 ? 1 : R, MINB});
  };
  return v;
}

const std::vector<Variant32> &variants32() {
  static const std::vector<Variant32> v = {
      make_variant32<32, 8, 2>(), make_variant32<32, 8, 3>(), make_variant32<32, 8, 4>(),
      make_variant32<32, 4, 6>(), make_variant32<64, 4, 3>(), make_variant32<32, 16, 2>(),
      make_variant32<32, 8, 2, false>(), make_variant32<32, 16, 2, false>(),
      make_variant32<32, 8, 2, true, true>(), make_variant32<32, 8, 3, false, true>(),
      make_variant32<32, 16, 2, false, true>(), make_variant32<32, 8, 2, false, true>(),
      make_variant32<32, 8, 3, false, true, true>(), make_variant32<32, 16, 2, false, true, true>(),
      make_variant32<32, 8, 3, false, 2, true>(), make_variant32<32, 16, 2, false, 2, true>(),
      make_variant32<32, 16, 2, false, 2, false>(),
      make_variant32<32, 8, 3, false, false, true>(), make_variant32<32, 16, 2, false, false, true>(),
      make_split_variant32<4, 1, 4, 4, 4, 4>(), make_split_variant32<4, 1, 5, 4, 3, 5>(),
      make_split_variant32<4, 1, 6, 4, 2, 6>(), make_split_variant32<2, 1, 4, 2, 3, 5>(),
      make_split_variant32<2, 1, 4, 1, 2, 6>()};
  return v;
}

struct Stepper32 {
  pf5d_stepper_desc d{};
  bool closed1d = false;         // 1D elastic term in closed form (k32_elastic1d)
  ColPass colp;                // elastic term: batched transforms + one column kernel
  bool use_colpass = false;
  double bn = 0.0, b0 = 0.0;     // its B(k): bn for every k != 0, b0 at k = 0
  bool use_loop1d = false;       // 1D steps by k32_loop1d
  Loop1dShape loop;
  unsigned long long wait_ns = kLoop1dWaitNs;   // its blocks' longest wait
  int64_t shape[3] = {1, 1, 1};
  int64_t npts = 0, nk = 0;
  float4 *hi = nullptr, *lo = nullptr, *dX = nullptr;
  float *s = nullptr, *bk = nullptr;
  cufftComplex *k = nullptr;
  cufftHandle fwd = 0, inv = 0;
  bool plans = false;
  double *mass_ws = nullptr;
  double *partial = nullptr;     // rate kernel block maxima
  float *mm = nullptr;           // split-rate buffers: mu, M, (M_Fe, X_Fe) per point
  StepState32 *st = nullptr;
  Rate32 rp{};
  Update32 up{};
  cudaStream_t cap = nullptr;
  std::map<int64_t, cudaGraphExec_t> graphs;
  dim3 grid, block;
  size_t smem = 0;
  int zc = 1;
  int variant = 0;
  std::string kernels;           // text returned by s32_rate_kernels
};

#define PF5D_CUFFT32(call)                                                         \
  do {                                                                             \
    cufftResult r_ = (call);                                                       \
    if (r_ != CUFFT_SUCCESS) {                                                     \
      set_error("%s:%d %s: cufft error %d", __FILE__, __LINE__, #call, (int)r_);   \
      return PF5D_ERR_CUFFT;                                                       \
    }                                                                              \
  } while (0)

// Grid of the rate kernel of `variant` (and the 3D axis-0 chunk).
static dim3 grid32_of(const Stepper32 *h, int variant, int *zc_out) {
  const Rate32 &P = h->rp;
  *zc_out = 1;
  if (h->d.dim == 1) return dim3((unsigned)((P.nx + kTX1_32 - 1) / kTX1_32));
  const Variant32 &v = variants32()[variant];
  const int ty = h->d.dim == 2 && v.ty2 ? v.ty2 : v.ty;
  const unsigned gx = (unsigned)((P.nx + v.tx - 1) / v.tx), gy = (unsigned)((P.ny + ty - 1) / ty);
  if (h->d.dim == 2) return dim3(gx, gy, 1);
  const int64_t tiles = (int64_t)gx * gy;
  const int64_t target = (int64_t)sm_count() * v.minb * 4;
  int64_t zc = (tiles * P.nz + target - 1) / target;
  zc = std::max<int64_t>(4, std::min<int64_t>(zc, 64));
  zc = std::min<int64_t>(zc, P.nz);
  *zc_out = (int)zc;
  return dim3(gx, gy, (unsigned)((P.nz + zc - 1) / zc));
}

// Block slots needed by the largest rate grid over all variants.
static int64_t max_blocks32(const Stepper32 *h) {
  int64_t m = 1;
  const int nv = h->d.dim == 1 ? 1 : (int)variants32().size();
  for (int v = 0; v < nv; ++v) {
    int zc = 1;
    const dim3 g = grid32_of(h, v, &zc);
    m = std::max<int64_t>(m, (int64_t)g.x * g.y * g.z);
  }
  return m;
}

static pf5d_status configure32(Stepper32 *h, int variant) {
  if (h->d.dim == 1) {
    h->block = dim3(kTX1_32);
    h->grid = grid32_of(h, 0, &h->zc);
    h->smem = 0;
    return PF5D_OK;
  }
  const auto &vars = variants32();
  PF5D_REQUIRE(variant >= 0 && variant < (int)vars.size(), PF5D_ERR_ARG, "bad variant %d",
               variant);
  const Variant32 &v = vars[variant];
  h->variant = variant;
  v.set_attrs();
  PF5D_LAUNCHED();
  h->block = dim3(v.tx, v.ty);
  h->smem = h->d.dim == 2 ? v.smem2d : v.smem3d;
  h->grid = grid32_of(h, variant, &h->zc);
  return PF5D_OK;
}

static pf5d_status launch_rate32(Stepper32 *h, cudaStream_t s) {
  switch (h->d.dim) {
    case 1: launch_pdl(k32_rate_1d<kTX1_32>, h->grid, h->block, 0, s, h->rp); break;
    case 2: variants32()[h->variant].launch2d(h->grid, h->block, h->smem, s, h->rp); break;
    default: variants32()[h->variant].launch3d(h->grid, h->block, h->smem, s, h->rp, h->zc);
  }
  PF5D_LAUNCHED();
  PF5D_CUDA(launch_pdl(k32_dt, dim3(1), dim3(kDt32Threads), 0, s, h->rp,
                       (int)(h->grid.x * h->grid.y * h->grid.z)));
  return PF5D_OK;
}

// The elastic term of a step: s -> s' in place, by cuFFT R2C, the B(k)/N
// multiply and C2R, or in 1D by k32_elastic1d (the closed form).
static pf5d_status elastic32(Stepper32 *h, cudaStream_t s) {
  if (h->closed1d) {
    PF5D_CUDA(launch_pdl(k32_elastic1d, dim3(1), dim3(kElastic1dThreads32), 0, s, h->s, h->npts,
                         h->bn, h->b0, (const unsigned *)&h->st->halt));
    return PF5D_OK;
  }
  if (h->use_colpass) {
    pf5d_status st;
    if ((st = colpass_rows_forward32(&h->colp, h->s, h->k, s)) != PF5D_OK) return st;
    if ((st = colpass_columns32(&h->colp, h->k, h->bk, &h->st->halt, s)) != PF5D_OK) return st;
    return colpass_rows_inverse32(&h->colp, h->k, h->s, s);
  }
    PF5D_CUFFT32(cufftSetStream(h->fwd, s));
    PF5D_CUFFT32(cufftExecR2C(h->fwd, h->s, h->k));
    k32_bmul<<<grid_for(h->nk, 256), 256, 0, s>>>(h->k, h->bk, h->nk, &h->st->halt);
    PF5D_LAUNCHED();
    PF5D_CUFFT32(cufftSetStream(h->inv, s));
    PF5D_CUFFT32(cufftExecC2R(h->inv, h->k, h->s));
  return PF5D_OK;
}

static pf5d_status enqueue32(Stepper32 *h, cudaStream_t s) {
  if (h->d.elastic) {
    const pf5d_status e = elastic32(h, s);
    if (e != PF5D_OK) return e;
  }
  pf5d_status st = launch_rate32(h, s);
  if (st != PF5D_OK) return st;
  PF5D_CUDA(launch_pdl(k32_update, dim3(grid_for(h->npts, 256, 4)), dim3(256), 0, s, h->up));
  PF5D_LAUNCHED();
  return PF5D_OK;
}

static pf5d_status graph32(Stepper32 *h, int64_t n, cudaGraphExec_t *out) {
  auto it = h->graphs.find(n);
  if (it != h->graphs.end()) {
    *out = it->second;
    return PF5D_OK;
  }
  cudaGraph_t g = nullptr;
  PF5D_CUDA(cudaStreamBeginCapture(h->cap, cudaStreamCaptureModeThreadLocal));
  pf5d_status st = PF5D_OK;
  for (int64_t i = 0; i < n && st == PF5D_OK; ++i) st = enqueue32(h, h->cap);
  cudaError_t e = cudaStreamEndCapture(h->cap, &g);
  if (st != PF5D_OK) {
    if (g) cudaGraphDestroy(g);
    return st;
  }
  PF5D_REQUIRE(e == cudaSuccess, PF5D_ERR_CUDA, "graph capture: %s", cudaGetErrorString(e));
  cudaGraphExec_t exec = nullptr;
  e = cudaGraphInstantiate(&exec, g, 0);
  cudaGraphDestroy(g);
  PF5D_REQUIRE(e == cudaSuccess, PF5D_ERR_CUDA, "graph instantiate: %s", cudaGetErrorString(e));
  h->graphs[n] = exec;
  *out = exec;
  return PF5D_OK;
}

// The step loop of a 1D solve (255 registers a thread in small blocks).
using Loop1dKernel32 = void (*)(Rate32, Update32, double, double, int, int, unsigned long long);
static Loop1dKernel32 loop1d_kernel32(const Stepper32 *h) {
  return h->loop.threads <= kLoop1dThreads / 2 ? k32_loop1d<kLoop1dThreads / 2>
                                               : k32_loop1d<kLoop1dThreads>;
}

static void drop_graphs(Stepper32 *h) {
  for (auto &kv : h->graphs) cudaGraphExecDestroy(kv.second);
  h->graphs.clear();
}

pf5d_status s32_create(const pf5d_stepper_desc *desc, const double *X_init, void *stream,
                       Stepper32 **out) {
  PF5D_REQUIRE(desc && X_init && out && desc->grid32, PF5D_ERR_ARG, "null argument");
  PF5D_REQUIRE(desc->node_stride32 == kStride32 && (((uintptr_t)desc->grid32) & 15) == 0,
               PF5D_ERR_ARG, "FP32 table needs %d floats per node, 16-byte aligned", kStride32);
  auto *h = new Stepper32();
  h->d = *desc;
  h->d.bk = nullptr;
  int64_t npts = 1;
  for (int d = 0; d < desc->dim; ++d) {
    h->shape[d] = desc->shape[d];
    npts *= desc->shape[d];
  }
  h->npts = npts;
  auto fail = [&](pf5d_status code) {
    s32_destroy(h);
    return code;
  };
  if (cudaMalloc(&h->hi, npts * sizeof(float4)) != cudaSuccess ||
      cudaMalloc(&h->lo, npts * sizeof(float4)) != cudaSuccess ||
      cudaMalloc(&h->dX, npts * sizeof(float4)) != cudaSuccess ||
      cudaMalloc(&h->st, sizeof(StepState32)) != cudaSuccess ||
      cudaMalloc(&h->mass_ws, (kMassBlocks * S + S) * sizeof(double)) != cudaSuccess ||
      cudaStreamCreateWithFlags(&h->cap, cudaStreamNonBlocking) != cudaSuccess) {
    set_error("device allocation failed");
    return fail(PF5D_ERR_CUDA);
  }
  if (desc->elastic) {
    h->nk = npts / desc->shape[desc->dim - 1] * (desc->shape[desc->dim - 1] / 2 + 1);
    if (desc->dim == 1 && npts <= kElastic1dMax32) {
      // 1D B(k) is one value for every k != 0 (checked exactly): closed form
      bool flat = true;
      for (int64_t i = 2; i < h->nk && flat; ++i) flat = desc->bk[i] == desc->bk[1];
      h->closed1d = flat;
      h->bn = h->nk > 1 ? desc->bk[1] : 0.0;
      h->b0 = desc->bk[0];
    }
    if (desc->dim == 2 && colpass_fits(h->shape[0])) {
      h->use_colpass = colpass_create(desc->dim, h->shape, &h->colp, true) == PF5D_OK;
      if (!h->use_colpass) colpass_destroy(&h->colp);
    }
    if (!h->closed1d && !h->use_colpass) {
      long long n[3];
      for (int d = 0; d < desc->dim; ++d) n[d] = desc->shape[d];
      size_t ws = 0;
      if (cufftCreate(&h->fwd) != CUFFT_SUCCESS || cufftCreate(&h->inv) != CUFFT_SUCCESS ||
          cufftMakePlanMany64(h->fwd, desc->dim, n, nullptr, 1, 0, nullptr, 1, 0, CUFFT_R2C, 1,
                              &ws) != CUFFT_SUCCESS ||
          cufftMakePlanMany64(h->inv, desc->dim, n, nullptr, 1, 0, nullptr, 1, 0, CUFFT_C2R, 1,
                              &ws) != CUFFT_SUCCESS) {
        set_error("cuFFT plan creation failed");
        return fail(PF5D_ERR_CUFFT);
      }
      h->plans = true;
    }
    std::vector<float> b(h->nk);
    const double inv_n = 1.0 / (double)npts;
    for (int64_t i = 0; i < h->nk; ++i) b[i] = (float)(desc->bk[i] * inv_n);
    if (cudaMalloc(&h->s, npts * sizeof(float)) != cudaSuccess ||
        cudaMalloc(&h->k, h->nk * sizeof(cufftComplex)) != cudaSuccess ||
        cudaMalloc(&h->bk, h->nk * sizeof(float)) != cudaSuccess ||
        cudaMemcpy(h->bk, b.data(), h->nk * sizeof(float), cudaMemcpyHostToDevice) != cudaSuccess) {
      set_error("device allocation failed");
      return fail(PF5D_ERR_CUDA);
    }
  }
  Rate32 &P = h->rp;
  if (desc->dim == 1) {
    P.nz = 1; P.ny = 1; P.nx = (int)h->shape[0];
  } else if (desc->dim == 2) {
    P.nz = 1; P.ny = (int)h->shape[0]; P.nx = (int)h->shape[1];
  } else {
    P.nz = (int)h->shape[0]; P.ny = (int)h->shape[1]; P.nx = (int)h->shape[2];
  }
  P.D = h->hi;
  P.sp = desc->elastic ? h->s : nullptr;
  P.dX = h->dX;
  Table32 &T = P.T;
  T.grid = desc->grid32;
  T.coord = desc->node_coord;
  T.n = desc->table_n;
  T.stride = kStride32;
  T.inv_step = 1.0 / desc->resolution;
  T.inv_step_f = (float)T.inv_step;
  T.threshold = 1.0 - 4.0 * desc->resolution - 1e-9;
  T.max_nn_dist = desc->max_nn_dist;
  double sx = 0.0;
  for (int c = 0; c < S; ++c) {
    const double u = desc->x0[c] * T.inv_step;
    const double fl = floor(u);
    T.ib[c] = (int)fl;
    T.fb[c] = (float)(u - fl);
    T.x0[c] = desc->x0[c];
    sx = sx + desc->x0[c];
    P.kappa[c] = (float)desc->kappa[c];
    P.lvec[c] = (float)desc->lvec[c];
    P.x0f[c] = (float)desc->x0[c];
  }
  T.sum_x0 = sx;
  P.c_fe = 1.0 - sx;
  P.flux_scale = (float)(0.5 / (desc->dx * desc->dx));
  P.inv_dx2 = (float)(1.0 / (desc->dx * desc->dx));
  P.ctld = desc->ctld;
  P.t_cfl = desc->t_cfl;
  P.lower = desc->lower_limit;
  P.upper = desc->upper_limit;
  P.factor = desc->max_change_factor;
  P.adaptive = desc->adaptive;
  P.st = h->st;
  if (cudaMalloc(&h->partial, (size_t)max_blocks32(h) * sizeof(double)) != cudaSuccess) {
    set_error("device allocation failed");
    return fail(PF5D_ERR_CUDA);
  }
  P.partial = h->partial;
  P.npts = npts;
  // split buffers: mu (float4), M (float4), (M_Fe, X_Fe) (float2) per point
  if (cudaMalloc(&h->mm, (size_t)npts * (2 * sizeof(float4) + sizeof(float2))) != cudaSuccess) {
    set_error("device allocation failed");
    return fail(PF5D_ERR_CUDA);
  }
  P.mm_mu = reinterpret_cast<float4 *>(h->mm);
  P.mm_m = P.mm_mu + npts;
  P.mm_f = reinterpret_cast<float2 *>(P.mm_m + npts);
  Update32 &U = h->up;
  U.hi = h->hi;
  U.lo = h->lo;
  U.dX = h->dX;
  U.npts = npts;
  U.st = h->st;
  for (int c = 0; c < S; ++c) {
    U.x0[c] = desc->x0[c];
    U.lvec[c] = (float)desc->lvec[c];
  }
  U.sum_x0 = sx;
  U.s = desc->elastic ? h->s : nullptr;
  U.oob_interval = desc->oob_interval;
  pf5d_status st = configure32(h, 0);
  if (st != PF5D_OK) return fail(st);
  if (desc->dim == 1 && npts <= kLoop1dMax && (!desc->elastic || h->closed1d))
    for (int blocks = kLoop1dBlocks; blocks >= 8 && !h->use_loop1d; blocks /= 2) {
      h->loop = loop1d_shape(npts, blocks);
      h->use_loop1d = cluster_fits(loop1d_kernel32(h), h->loop, loop1d_smem32(h->loop.chunk));
    }
  if ((st = s32_reset(h, X_init, desc->dt0, 0.0, stream)) != PF5D_OK) return fail(st);
  *out = h;
  return PF5D_OK;
}

pf5d_status s32_reset(Stepper32 *h, const double *X, double dt, double time, void *stream) {
  cudaStream_t s = as_stream(stream);
  StepState32 init{};
  init.dt = dt;
  init.time = time;
  PF5D_CUDA(cudaMemcpyAsync(h->st, &init, sizeof(init), cudaMemcpyHostToDevice, s));
  if (X) {
    k32_split<<<grid_for(h->npts, 256, 4), 256, 0, s>>>(X, h->npts, h->up);
    PF5D_LAUNCHED();
  }
  PF5D_CUDA(cudaStreamSynchronize(s));
  return PF5D_OK;
}

pf5d_status s32_advance(Stepper32 *h, int64_t nsteps, void *stream) {
  cudaStream_t s = as_stream(stream);
  if (h->use_loop1d && loop1d_pays(h->npts, nsteps)) {
    const size_t sm = loop1d_smem32(h->loop.chunk);
    for (; nsteps > 0; nsteps -= kLoop1dSteps) {
      const int n = (int)std::min<int64_t>(nsteps, kLoop1dSteps);
      PF5D_CUDA(launch_cluster(loop1d_kernel32(h), h->loop, sm, s, h->rp, h->up, h->bn, h->b0,
                               h->loop.chunk, n, h->wait_ns));
    }
    return PF5D_OK;
  }
  while (nsteps > 0) {
    const int64_t n = nsteps < kGraphSteps32 ? nsteps : kGraphSteps32;
    cudaGraphExec_t g = nullptr;
    pf5d_status st = graph32(h, n, &g);
    if (st != PF5D_OK) return st;
    PF5D_CUDA(cudaGraphLaunch(g, s));
    nsteps -= n;
  }
  return PF5D_OK;
}

void s32_set_wait_limit(Stepper32 *h, unsigned long long ns) { h->wait_ns = ns; }

pf5d_status s32_state(Stepper32 *h, pf5d_step_state *out, void *stream) {
  StepState32 hs;
  cudaStream_t s = as_stream(stream);
  PF5D_CUDA(cudaMemcpyAsync(&hs, h->st, sizeof(hs), cudaMemcpyDeviceToHost, s));
  PF5D_CUDA(cudaStreamSynchronize(s));
  out->dt = hs.dt;
  out->time = hs.time;
  out->xdotmax = hs.xdotmax;
  out->step = hs.step;
  out->flags = hs.flags | (hs.halt ? PF5D_FLAG_HALTED : 0u);
  out->halted = hs.halt;
  return PF5D_OK;
}

// FP64 copies for the save-step reductions: dX/dt (4 per point) and mu/M
// (mm_row), from the FP32 buffers.
__global__ void k32_widen(const float *__restrict__ src, int64_t n, double *__restrict__ dst) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    dst[i] = (double)src[i];
}

// FP64 mu/M rows (mm_row: mu_1..4, M_Fe, M_1..4) from the split buffers.
__global__ void k32_widen_mm(Rate32 P, double *__restrict__ dst) {
  const int64_t n = P.npts;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const float4 mu = P.mm_mu[i], m = P.mm_m[i];
    const float2 f = P.mm_f[i];
    const float v[NP] = {mu.x, mu.y, mu.z, mu.w, f.x, m.x, m.y, m.z, m.w};
#pragma unroll
    for (int r = 0; r < NP; ++r) dst[mm_index(n, r, i)] = (double)v[r];
  }
}

pf5d_status s32_step_save_inputs(Stepper32 *h, double *X_out, double *dX_out, double *mm_out,
                                 void *stream) {
  cudaStream_t s = as_stream(stream);
  if (h->d.elastic) {
    const pf5d_status e = elastic32(h, s);
    if (e != PF5D_OK) return e;
  }
  pf5d_status st = launch_rate32(h, s);
  if (st != PF5D_OK) return st;
  switch (h->d.dim) {
    case 1: launch_chem32_save<1>(s, h->rp); break;
    case 2: launch_chem32_save<2>(s, h->rp); break;
    default: launch_chem32_save<3>(s, h->rp);
  }
  PF5D_LAUNCHED();
  k32_join<<<grid_for(h->npts, 256, 4), 256, 0, s>>>(h->hi, h->lo, h->npts, h->up, X_out);
  PF5D_LAUNCHED();
  k32_widen<<<grid_for(4 * h->npts, 256, 4), 256, 0, s>>>(reinterpret_cast<const float *>(h->dX),
                                                          4 * h->npts, dX_out);
  PF5D_LAUNCHED();
  k32_widen_mm<<<grid_for(h->npts, 256, 4), 256, 0, s>>>(h->rp, mm_out);
  PF5D_LAUNCHED();
  return PF5D_OK;
}

pf5d_status s32_step_update(Stepper32 *h, void *stream) {
  cudaStream_t s = as_stream(stream);
  k32_update<<<grid_for(h->npts, 256, 4), 256, 0, s>>>(h->up);
  PF5D_LAUNCHED();
  return PF5D_OK;
}

pf5d_status s32_field(Stepper32 *h, double *X_out, void *stream) {
  cudaStream_t s = as_stream(stream);
  k32_join<<<grid_for(h->npts, 256, 4), 256, 0, s>>>(h->hi, h->lo, h->npts, h->up, X_out);
  PF5D_LAUNCHED();
  return PF5D_OK;
}

pf5d_status s32_mass(Stepper32 *h, double *mean_out, void *stream) {
  cudaStream_t s = as_stream(stream);
  const unsigned nb = std::min<unsigned>(kMassBlocks, grid_for(h->npts, 256, 4));
  k32_mass_partial<<<nb, 256, 0, s>>>(h->hi, h->lo, h->npts, h->mass_ws);
  PF5D_LAUNCHED();
  k32_mass_final<<<1, 32, 0, s>>>(h->mass_ws, (int)nb, h->mass_ws + kMassBlocks * S);
  PF5D_LAUNCHED();
  double sums[S];
  PF5D_CUDA(cudaMemcpyAsync(sums, h->mass_ws + kMassBlocks * S, sizeof(sums),
                            cudaMemcpyDeviceToHost, s));
  PF5D_CUDA(cudaStreamSynchronize(s));
  for (int c = 0; c < S; ++c) mean_out[c] = h->d.x0[c] + sums[c] / (double)h->npts;
  return PF5D_OK;
}

int32_t s32_variant_count() { return (int32_t)variants32().size(); }

const char *s32_rate_kernels(Stepper32 *h) {
  if (h->d.dim == 1) h->kernels = kname("k32_rate_1d", {kTX1_32});
  else h->kernels = variants32()[h->variant].kernels(h->d.dim);
  h->kernels += " + k32_dt";
  return h->kernels.c_str();
}

int32_t s32_launches_per_step(const Stepper32 *h) {
  if (h->use_loop1d) return 1;
  const bool split = h->d.dim >= 2 && variants32()[h->variant].split;
  return (split ? 4 : 3) + (h->d.elastic ? 1 : 0);   // rate (+chem), dt, update (+ B(k))
}

pf5d_status s32_set_variant(Stepper32 *h, int32_t variant) {
  pf5d_status st = configure32(h, variant);
  if (st == PF5D_OK) drop_graphs(h);
  return st;
}

pf5d_status s32_autotune(Stepper32 *h, int32_t *variant, float *best_ms, void *stream) {
  cudaStream_t s = as_stream(stream);
  if (h->d.dim == 1) {
    if (variant) *variant = 0;
    if (best_ms) *best_ms = 0.f;
    return PF5D_OK;
  }
  StepState32 saved;
  PF5D_CUDA(cudaMemcpyAsync(&saved, h->st, sizeof(saved), cudaMemcpyDeviceToHost, s));
  PF5D_CUDA(cudaStreamSynchronize(s));
  cudaEvent_t e0, e1;
  PF5D_CUDA(cudaEventCreate(&e0));
  PF5D_CUDA(cudaEventCreate(&e1));
  int best = h->variant;
  float best_t = 1e30f;
  for (int v = 0; v < (int)variants32().size(); ++v) {
    if (configure32(h, v) != PF5D_OK) continue;
    if (launch_rate32(h, s) != PF5D_OK) {
      cudaGetLastError();
      continue;
    }
    PF5D_CUDA(cudaEventRecord(e0, s));
    pf5d_status st = PF5D_OK;
    for (int r = 0; r < 5 && st == PF5D_OK; ++r) st = launch_rate32(h, s);
    PF5D_CUDA(cudaEventRecord(e1, s));
    PF5D_CUDA(cudaEventSynchronize(e1));
    float ms = 0.f;
    PF5D_CUDA(cudaEventElapsedTime(&ms, e0, e1));
    if (st == PF5D_OK && ms / 5 < best_t) {
      best_t = ms / 5;
      best = v;
    }
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  pf5d_status st = configure32(h, best);
  if (st != PF5D_OK) return st;
  drop_graphs(h);
  PF5D_CUDA(cudaMemcpyAsync(h->st, &saved, sizeof(saved), cudaMemcpyHostToDevice, s));
  PF5D_CUDA(cudaStreamSynchronize(s));
  if (variant) *variant = best;
  if (best_ms) *best_ms = best_t;
  return PF5D_OK;
}

pf5d_status s32_launch_stage(Stepper32 *h, int32_t stage, void *stream) {
  cudaStream_t s = as_stream(stream);
  switch (stage) {
    case PF5D_STAGE_RATE:
      return launch_rate32(h, s);
    case PF5D_STAGE_UPDATE:
      k32_update<<<grid_for(h->npts, 256, 4), 256, 0, s>>>(h->up);
      PF5D_LAUNCHED();
      return PF5D_OK;
    // 1D closed form: the whole elastic term is the FFT_FWD stage
    case PF5D_STAGE_FFT_FWD:
      PF5D_REQUIRE(h->d.elastic, PF5D_ERR_ARG, "elasticity is off");
      if (h->closed1d) return elastic32(h, s);
      if (h->use_colpass) return colpass_rows_forward32(&h->colp, h->s, h->k, s);
      PF5D_CUFFT32(cufftSetStream(h->fwd, s));
      PF5D_CUFFT32(cufftExecR2C(h->fwd, h->s, h->k));
      return PF5D_OK;
    case PF5D_STAGE_BMUL:
      PF5D_REQUIRE(h->d.elastic, PF5D_ERR_ARG, "elasticity is off");
      if (h->closed1d) return PF5D_OK;
      if (h->use_colpass) return colpass_columns32(&h->colp, h->k, h->bk, &h->st->halt, s);
      k32_bmul<<<grid_for(h->nk, 256), 256, 0, s>>>(h->k, h->bk, h->nk, &h->st->halt);
      PF5D_LAUNCHED();
      return PF5D_OK;
    case PF5D_STAGE_FFT_INV:
      PF5D_REQUIRE(h->d.elastic, PF5D_ERR_ARG, "elasticity is off");
      if (h->closed1d) return PF5D_OK;
      if (h->use_colpass) return colpass_rows_inverse32(&h->colp, h->k, h->s, s);
      PF5D_CUFFT32(cufftSetStream(h->inv, s));
      PF5D_CUFFT32(cufftExecC2R(h->inv, h->k, h->s));
      return PF5D_OK;
    default:
      set_error("unknown stage %d", stage);
      return PF5D_ERR_ARG;
  }
}

float *s32_rate(Stepper32 *h) { return reinterpret_cast<float *>(h->dX); }

void s32_destroy(Stepper32 *h) {
  if (!h) return;
  drop_graphs(h);
  if (h->plans) {
    cufftDestroy(h->fwd);
    cufftDestroy(h->inv);
  }
  cudaFree(h->hi);
  cudaFree(h->lo);
  cudaFree(h->dX);
  cudaFree(h->s);
  cudaFree(h->bk);
  colpass_destroy(&h->colp);
  cudaFree(h->k);
  cudaFree(h->st);
  cudaFree(h->mass_ws);
  cudaFree(h->partial);
  cudaFree(h->mm);
  if (h->cap) cudaStreamDestroy(h->cap);
  delete h;
}

}  // namespace pf5d
