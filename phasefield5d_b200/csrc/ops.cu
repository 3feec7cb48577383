// ops.cu -- one device kernel per reference hot-path function, behind the
// C ABI of include/pf5d.h.  These are the drop-in forms of the reference's
// separate passes (interpolator_nb, calculate_laplacian, the fused divergence,
// abs_max, clamp_simplex, the update, out_of_bounds); the fused step loop in
// stepper.cu reuses the same device routines.
//
// Compiled with -fmad=false: FP64 results equal the reference's Numba kernels
// bit for bit.
#include <cmath>
#include <cstring>
#include <mutex>
#include <vector>

#include "pf5d_device.cuh"
#include "pf5d_gather.cuh"
#include "pf5d_host.h"

namespace pf5d {

static thread_local std::string g_last_error;

void set_error(const char *fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof(buf), fmt, ap);
  va_end(ap);
  g_last_error = buf;
}

int sm_count() {
  static int cached[64] = {0};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) dev = 0;
  if (cached[dev] == 0) {
    int n = 0;
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    cached[dev] = n > 0 ? n : 148;
  }
  return cached[dev];
}

// ------------------------------------------------------------------ interp
__global__ void k_interp4d(const double *__restrict__ comp, int64_t npts, Table T,
                           double *__restrict__ out, int64_t out_stride, uint8_t *mask,
                           unsigned *flags) {
  unsigned f = 0;
  for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < npts;
       r += (int64_t)gridDim.x * blockDim.x) {
    double x[S];
    const double2 a = reinterpret_cast<const double2 *>(comp + 4 * r)[0];
    const double2 b = reinterpret_cast<const double2 *>(comp + 4 * r)[1];
    x[0] = a.x; x[1] = a.y; x[2] = b.x; x[3] = b.y;
    double v[NP];
    const bool lin = interp_point(T, x, v, &f);
    if (mask) mask[r] = lin ? 1 : 0;
    double *o = out + r * out_stride;
#pragma unroll
    for (int p = 0; p < NP; ++p) o[p] = v[p];
  }
  if (flags && f) atomicOr(flags, f);
}

// --------------------------------------------------------------- laplacian
// operators.py:32-76; neighbour order +axis0, -axis0, +axis1, -axis1, +axis2, -axis2.
__global__ void k_laplacian(int dim, int64_t n0, int64_t n1, int64_t n2, int nc,
                            const double *__restrict__ c, double inv_dx2,
                            double *__restrict__ out) {
  const int64_t npts = n0 * n1 * n2;
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < npts;
       p += (int64_t)gridDim.x * blockDim.x) {
    const int64_t k = p % n2, j = (p / n2) % n1, i = p / (n2 * n1);
    if (dim == 1) {
      const int64_t ip = wrap_p(i, n0), im = wrap_m(i, n0);
      for (int s = 0; s < nc; ++s)
        out[p * nc + s] = (c[ip * nc + s] + c[im * nc + s] - 2.0 * c[p * nc + s]) * inv_dx2;
    } else if (dim == 2) {
      const int64_t ip = wrap_p(i, n0) * n1 + j, im = wrap_m(i, n0) * n1 + j;
      const int64_t jp = i * n1 + wrap_p(j, n1), jm = i * n1 + wrap_m(j, n1);
      for (int s = 0; s < nc; ++s)
        out[p * nc + s] = (c[ip * nc + s] + c[im * nc + s] + c[jp * nc + s] + c[jm * nc + s] -
                           4.0 * c[p * nc + s]) * inv_dx2;
    } else {
      const int64_t ip = (wrap_p(i, n0) * n1 + j) * n2 + k, im = (wrap_m(i, n0) * n1 + j) * n2 + k;
      const int64_t jp = (i * n1 + wrap_p(j, n1)) * n2 + k, jm = (i * n1 + wrap_m(j, n1)) * n2 + k;
      const int64_t kp = (i * n1 + j) * n2 + wrap_p(k, n2), km = (i * n1 + j) * n2 + wrap_m(k, n2);
      for (int s = 0; s < nc; ++s)
        out[p * nc + s] = (c[ip * nc + s] + c[im * nc + s] + c[jp * nc + s] + c[jm * nc + s] +
                           c[kp * nc + s] + c[km * nc + s] - 6.0 * c[p * nc + s]) * inv_dx2;
    }
  }
}

// Four components in 16-byte aligned rows, one point per thread: a block is 32
// columns by 8 rows of a plane, so a point's in-plane neighbours are its own
// lines.  Bound by the reads: 128^3 72 us with 64-bit index arithmetic and scalar
// loads -> 35.
template <int DIM, int W>
__global__ void __launch_bounds__(256) k_laplacian4(int n0, int n1, int n2,
                                                    const double *__restrict__ c, double inv_dx2,
                                                    double *__restrict__ out) {
  // (z, y, x) of the point: axes from the back, the missing ones of length 1
  const int x = blockIdx.x * 32 + threadIdx.x, y = blockIdx.y * 8 + threadIdx.y, z = blockIdx.z;
  const int nx = DIM == 1 ? n0 : (DIM == 2 ? n1 : n2), ny = DIM == 1 ? 1 : (DIM == 2 ? n0 : n1);
  const int nz = DIM == 3 ? n0 : 1;
  if (x >= nx || y >= ny) return;
  auto at = [&](int zz, int yy, int xx) { return 4 * (((int64_t)zz * ny + yy) * nx + xx); };
  double v[S], lap[S], a[S], b[S];
  load_comp4<W>(c + at(z, y, x), v);
  if (DIM == 3) {
    load_comp4<W>(c + at(z + 1 == nz ? 0 : z + 1, y, x), a);
    load_comp4<W>(c + at(z == 0 ? nz - 1 : z - 1, y, x), b);
#pragma unroll
    for (int s = 0; s < S; ++s) lap[s] = a[s] + b[s];
  }
  if (DIM >= 2) {
    load_comp4<W>(c + at(z, y + 1 == ny ? 0 : y + 1, x), a);
    load_comp4<W>(c + at(z, y == 0 ? ny - 1 : y - 1, x), b);
#pragma unroll
    for (int s = 0; s < S; ++s) lap[s] = DIM == 3 ? (lap[s] + a[s]) + b[s] : a[s] + b[s];
  }
  load_comp4<W>(c + at(z, y, x + 1 == nx ? 0 : x + 1), a);
  load_comp4<W>(c + at(z, y, x == 0 ? nx - 1 : x - 1), b);
#pragma unroll
  for (int s = 0; s < S; ++s) {
    const double sum = DIM == 1 ? a[s] + b[s] : (lap[s] + a[s]) + b[s];
    lap[s] = (sum - 2.0 * DIM * v[s]) * inv_dx2;
  }
  double2 *o = reinterpret_cast<double2 *>(out + at(z, y, x));
  o[0] = make_double2(lap[0], lap[1]);
  o[1] = make_double2(lap[2], lap[3]);
}

// Whether k_laplacian4's 32x8 tiles are full enough: a quarter of the lanes
// along the last axis and 20 points a block.  us, k_laplacian -> k_laplacian4:
// 512x512x2 (2 lanes of 32) 21 -> 62, 5000x50x8 (8 lanes) 69 -> 62, 25000x1x8
// (8 points a block) 11 -> 17, 12500x2x8 (16) 10.5 -> 10.5.  1D tiles are one
// row of 32 points: 22 -> 19 at 10^6.
static bool laplacian4_pays(int dim, int64_t nx, int64_t ny, int64_t nz) {
  const int64_t tx = (nx + 31) / 32, ty = (ny + 7) / 8;
  return dim == 1 || (nx >= 8 * tx && nx * ny * nz >= 20 * tx * ty * nz);
}

struct Kappa {
  double k[8];
};

__global__ void k_kappa_subtract(double *mu, int64_t mu_stride, double *lap, Kappa kap,
                                 int64_t npts, int nc) {
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < npts;
       p += (int64_t)gridDim.x * blockDim.x)
    for (int s = 0; s < nc; ++s) {
      const double l = lap[p * nc + s] * kap.k[s];
      lap[p * nc + s] = l;
      mu[p * mu_stride + s] = mu[p * mu_stride + s] - l;
    }
}

// ------------------------------------------------------------- divergence
// fluxes.py:296-395: per point, both faces per axis (gradients inline), then
// (f0p - f0m + f1p - f1m + f2p - f2m) * inv_dx left to right.
__device__ __forceinline__ void load4(const double *p, double v[S]) {
#pragma unroll
  for (int s = 0; s < S; ++s) v[s] = p[s];
}
__device__ __forceinline__ void load5(const double *p, double v[NM]) {
#pragma unroll
  for (int s = 0; s < NM; ++s) v[s] = p[s];
}

// One point per thread, both faces of every axis: any shape.
__global__ void k_divergence_points(int dim, int64_t n0, int64_t n1, int64_t n2,
                                    const double *__restrict__ X, const double *__restrict__ M,
                                    int64_t ms, const double *__restrict__ mu, int64_t mus,
                                    double inv_dx, double *__restrict__ out) {
  const int64_t npts = n0 * n1 * n2;
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < npts;
       p += (int64_t)gridDim.x * blockDim.x) {
    const int64_t k = p % n2, j = (p / n2) % n1, i = p / (n2 * n1);
    int64_t nb[6];
    nb[0] = (wrap_p(i, n0) * n1 + j) * n2 + k;
    nb[1] = (wrap_m(i, n0) * n1 + j) * n2 + k;
    nb[2] = (i * n1 + wrap_p(j, n1)) * n2 + k;
    nb[3] = (i * n1 + wrap_m(j, n1)) * n2 + k;
    nb[4] = (i * n1 + j) * n2 + wrap_p(k, n2);
    nb[5] = (i * n1 + j) * n2 + wrap_m(k, n2);
    double Xc[S], Mc[NM], muc[S];
    load4(X + p * S, Xc);
    load5(M + p * ms, Mc);
    load4(mu + p * mus, muc);
    double acc[S];
    for (int f = 0; f < 2 * dim; ++f) {
      const int64_t q = nb[f];
      double Xn[S], Mn[NM], mun[S], g[S], J[S];
      load4(X + q * S, Xn);
      load5(M + q * ms, Mn);
      load4(mu + q * mus, mun);
#pragma unroll
      for (int s = 0; s < S; ++s) g[s] = (f & 1) ? (muc[s] - mun[s]) * inv_dx : (mun[s] - muc[s]) * inv_dx;
      face_flux(Xc, Mc, Xn, Mn, g, J);
#pragma unroll
      for (int s = 0; s < S; ++s) {
        if (f == 0) acc[s] = J[s];
        else if (f & 1) acc[s] = acc[s] - J[s];
        else acc[s] = acc[s] + J[s];
      }
    }
#pragma unroll
    for (int s = 0; s < S; ++s) out[p * S + s] = acc[s] * inv_dx;
  }
}

// A warp takes 32 neighbouring columns of the last axis and marches along the
// first, as the split rate stage's k_flux: the face along the march is carried,
// the face between columns handed on by shuffles (30 columns are finished), and
// in 3D the rows above and below are read where the block's other warps read
// them.  1D: no march; the faces between columns are all there is.
// ROWS9: mu and M are the two parts of rows of nine values (interp[..., :4] and
// interp[..., 4:]); a warp then reads its 32 rows, one run of 2304 bytes, in
// memory order and turns them in shared memory, where loads of a column of the
// rows would touch 18 lines each.
// Bound by the latency of the loads.  128^3, rows of nine: 212 us with
// k_divergence_points -> 162.
constexpr int kDivThreads = 128, kDivCols = 30;

struct DivView {
  const double *X, *mu, *M;
  int64_t mus, ms;
};

struct DivPoint {
  double x[S], mu[S], m[NM];
};

template <int DIM, bool ROWS9, int W>
__global__ void __launch_bounds__(kDivThreads, 4)
    k_divergence(int n0, int n1, int n2, DivView V, double inv_dx, double *__restrict__ out, int rows) {
  __shared__ double turn[kDivThreads / 32][ROWS9 ? 32 * NP : 1];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int nx = DIM == 1 ? n0 : (DIM == 2 ? n1 : n2), ny = DIM == 3 ? n1 : 1;
  const int nm = DIM == 1 ? 1 : n0;                    // length of the march
  // block: column tile, then (2D) four chunks of the march or (3D) four rows,
  // then (3D) a chunk
  const int tiles = (nx + kDivCols - 1) / kDivCols, ny4 = (ny + 3) / 4;
  const int rest = blockIdx.x / tiles;
  const int tile = DIM == 1 ? blockIdx.x * 4 + w : blockIdx.x % tiles;
  const int y = DIM == 3 ? rest % ny4 * 4 + w : 0;
  const int64_t first64 = DIM == 1 ? 0 : (int64_t)(DIM == 3 ? rest / ny4 : rest * 4 + w) * rows;
  if (first64 >= nm || y >= ny || tile >= tiles) return;       // whole warps
  const int first = (int)first64, last = min(first + rows, nm);
  const int col0 = tile * kDivCols - 1, col = col0 + lane, x = wrap_any(col, nx);
  int off[NP];                                         // this lane's elements of a row of rows
  if (ROWS9) {
#pragma unroll
    for (int k = 0; k < NP; ++k) {
      const int e = lane + 32 * k;
      off[k] = wrap_any(col0 + e / NP, nx) * NP + e % NP;
    }
  }
  auto load = [&](int i, int yy, DivPoint &q) {
    const int64_t line = ((int64_t)i * ny + yy) * nx, p = line + x;
    load_comp4<W>(V.X + 4 * p, q.x);
    if (ROWS9) {
      double *buf = turn[w];
      double v[NP];
#pragma unroll
      for (int k = 0; k < NP; ++k) v[k] = __ldg(V.mu + line * NP + off[k]);
      __syncwarp();
#pragma unroll
      for (int k = 0; k < NP; ++k) buf[lane + 32 * k] = v[k];
      __syncwarp();
#pragma unroll
      for (int s = 0; s < S; ++s) q.mu[s] = buf[lane * NP + s];
#pragma unroll
      for (int s = 0; s < NM; ++s) q.m[s] = buf[lane * NP + S + s];
    } else {
#pragma unroll
      for (int s = 0; s < S; ++s) q.mu[s] = __ldg(V.mu + p * V.mus + s);
#pragma unroll
      for (int s = 0; s < NM; ++s) q.m[s] = __ldg(V.M + p * V.ms + s);
    }
  };
  auto face = [&](const DivPoint &lo, const DivPoint &hi, double J8[S]) {
    double g[S];
#pragma unroll
    for (int s = 0; s < S; ++s) g[s] = (hi.mu[s] - lo.mu[s]) * inv_dx;
    face_flux8(lo.x, lo.m, hi.x, hi.m, g, J8);
  };
  const double inv_dx8 = 0.125 * inv_dx;
  const bool out2 = ((uintptr_t)out & 15) == 0;
  const int yp = y + 1 == ny ? 0 : y + 1, ym = y == 0 ? ny - 1 : y - 1;
  DivPoint cur;
  double Jm[S];
  load(first, y, cur);
  if (DIM > 1) {
    DivPoint below;
    load(first == 0 ? nm - 1 : first - 1, y, below);
    face(below, cur, Jm);
  }
  for (int i = first; i < last; ++i) {
    DivPoint up, nb;
    double jx[S], jl[S], jyp[S], jym[S], jz[S];
    if (DIM > 1) load(i + 1 == nm ? 0 : i + 1, y, up);
#pragma unroll
    for (int s = 0; s < S; ++s) {
      nb.x[s] = __shfl_down_sync(0xffffffffu, cur.x[s], 1);
      nb.mu[s] = __shfl_down_sync(0xffffffffu, cur.mu[s], 1);
    }
#pragma unroll
    for (int s = 0; s < NM; ++s) nb.m[s] = __shfl_down_sync(0xffffffffu, cur.m[s], 1);
    face(cur, nb, jx);
#pragma unroll
    for (int s = 0; s < S; ++s) jl[s] = __shfl_up_sync(0xffffffffu, jx[s], 1);
    if (DIM == 3) {
      load(i, yp, nb);
      face(cur, nb, jyp);
      load(i, ym, nb);
      face(nb, cur, jym);
    }
    if (DIM > 1) face(cur, up, jz);
    if (lane > 0 && lane <= kDivCols && col < nx) {
      double *o = out + 4 * (((int64_t)i * ny + y) * nx + x);
      double v[S];
#pragma unroll
      for (int s = 0; s < S; ++s) {
        if (DIM == 1) {
          v[s] = jx[s] - jl[s];
        } else {
          v[s] = jz[s] - Jm[s];
          if (DIM == 3) v[s] = (v[s] + jyp[s]) - jym[s];
          v[s] = (v[s] + jx[s]) - jl[s];
        }
        v[s] = v[s] * inv_dx8;
      }
      if (out2) {
        reinterpret_cast<double2 *>(o)[0] = make_double2(v[0], v[1]);
        reinterpret_cast<double2 *>(o)[1] = make_double2(v[2], v[3]);
      } else {
#pragma unroll
        for (int s = 0; s < S; ++s) o[s] = v[s];
      }
    }
    if (DIM > 1) {
#pragma unroll
      for (int s = 0; s < S; ++s) Jm[s] = jz[s];
      cur = up;
    }
  }
}

// Whether the march is the faster form: it spends a warp on 30 columns and, in
// 3D, a block on four rows, full or not; reading rows of nine through shared
// memory costs it more.  Measured from 16,000 to 3,000,000 points; us, a point
// per thread -> march:
//   2D, rows of nine: 12 columns of 32 lanes 4.7 -> 6.2 (16,000 points), 14
//     columns 8.1 -> 8.1; apart: 8 columns 16.5 -> 18.7, 9 columns 74 -> 61;
//   3D, rows of nine: 24 columns (0.75) 170 -> 165, 20 (0.62) 12.4 -> 14.4;
//     2 or 3 rows of 4 still 258 -> 178, 6 rows of 8 12.4 -> 14.4, 1 row of 4
//     18.7 -> 25; few blocks do not hide its longer steps: 16,000 points 6.3 ->
//     8.3, 40,000 8.3 -> 8.3, 160,000 18.5 -> 14.5; apart: 31 columns in two
//     warps (0.48) 22.8 -> 22.8, 12 (0.37) 20.8 -> 22.8; with rows to spare from
//     0.68 on.
static bool march_pays(int dim, int64_t npts, int64_t n1, int64_t nx, bool rows9) {
  const int64_t lanes = 32 * ((nx + kDivCols - 1) / kDivCols);
  if (dim == 1) return true;
  if (dim == 2) return 100 * nx >= (rows9 ? 43 : 27) * lanes;
  const bool full = 8 * n1 >= 28 * ((n1 + 3) / 4);                 // 7 of 8 rows
  if (rows9)
    return 100 * nx >= 68 * lanes && ((full && npts >= 32768) || n1 == 2 || n1 == 3);
  return 100 * nx >= (full ? 45 : 68) * lanes && n1 >= 2;
}

static bool rows_of_nine(const DivView &V, int64_t nx) {
  return V.M == V.mu + S && V.mus == NP && V.ms == NP &&
         nx < (1 << 27);                               // 32-bit offsets in a row of rows
}

template <int DIM>
static void launch_divergence(int n0, int n1, int n2, const DivView &V, double inv_dx, double *out,
                              cudaStream_t s) {
  const int nx = DIM == 1 ? n0 : (DIM == 2 ? n1 : n2), nm = DIM == 1 ? 1 : n0;
  const int tiles = (nx + kDivCols - 1) / kDivCols;
  // rows of a march: 16 (one face more per 16 rows), fewer where that leaves
  // less than 12 warps per SM
  const int64_t lines = (int64_t)tiles * (DIM == 3 ? (n1 + 3) / 4 * 4 : 1) * nm;
  const int64_t fill = lines / ((int64_t)sm_count() * 12);
  const int rows = (int)(fill < 2 ? 2 : (fill > 16 ? 16 : fill));
  const int64_t chunks = (nm + rows - 1) / rows;
  const int64_t blocks = DIM == 1   ? (tiles + 3) / 4
                         : DIM == 2 ? tiles * ((chunks + 3) / 4)
                                    : tiles * chunks * ((n1 + 3) / 4);
  const dim3 grid((unsigned)blocks);
  const bool wide = aligned_to(V.X, 32);
  const bool rows9 = rows_of_nine(V, nx);
  auto kernel = rows9 ? (wide ? k_divergence<DIM, true, 4> : k_divergence<DIM, true, 1>)
                      : (wide ? k_divergence<DIM, false, 4> : k_divergence<DIM, false, 1>);
  kernel<<<grid, kDivThreads, 0, s>>>(n0, n1, n2, V, inv_dx, out, rows);
}

// ---------------------------------------------- save-step gradients/fluxes
__global__ void k_gradients_pm(int dim, int64_t n0, int64_t n1, int64_t n2, int nc,
                               const double *__restrict__ c, int64_t cs, double inv_dx,
                               double *__restrict__ gp, double *__restrict__ gm) {
  const int64_t npts = n0 * n1 * n2;
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < npts;
       p += (int64_t)gridDim.x * blockDim.x) {
    const int64_t k = p % n2, j = (p / n2) % n1, i = p / (n2 * n1);
    int64_t pp[3], pm[3];
    pp[0] = (wrap_p(i, n0) * n1 + j) * n2 + k;
    pm[0] = (wrap_m(i, n0) * n1 + j) * n2 + k;
    pp[1] = (i * n1 + wrap_p(j, n1)) * n2 + k;
    pm[1] = (i * n1 + wrap_m(j, n1)) * n2 + k;
    pp[2] = (i * n1 + j) * n2 + wrap_p(k, n2);
    pm[2] = (i * n1 + j) * n2 + wrap_m(k, n2);
    for (int d = 0; d < dim; ++d)
      for (int s = 0; s < nc; ++s) {
        const double center = c[p * cs + s];
        gp[(d * npts + p) * nc + s] = (c[pp[d] * cs + s] - center) * inv_dx;
        gm[(d * npts + p) * nc + s] = (center - c[pm[d] * cs + s]) * inv_dx;
      }
  }
}

__global__ void k_fluxes_pm(int dim, int64_t n0, int64_t n1, int64_t n2,
                            const double *__restrict__ X, const double *__restrict__ M, int64_t ms,
                            const double *__restrict__ gp, const double *__restrict__ gm,
                            double *__restrict__ fp, double *__restrict__ fm) {
  const int64_t npts = n0 * n1 * n2;
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < npts;
       p += (int64_t)gridDim.x * blockDim.x) {
    const int64_t k = p % n2, j = (p / n2) % n1, i = p / (n2 * n1);
    int64_t pp[3], pm[3];
    pp[0] = (wrap_p(i, n0) * n1 + j) * n2 + k;
    pm[0] = (wrap_m(i, n0) * n1 + j) * n2 + k;
    pp[1] = (i * n1 + wrap_p(j, n1)) * n2 + k;
    pm[1] = (i * n1 + wrap_m(j, n1)) * n2 + k;
    pp[2] = (i * n1 + j) * n2 + wrap_p(k, n2);
    pm[2] = (i * n1 + j) * n2 + wrap_m(k, n2);
    double Xc[S], Mc[NM];
    load4(X + p * S, Xc);
    load5(M + p * ms, Mc);
    for (int d = 0; d < dim; ++d) {
      const int64_t o = (d * npts + p) * S;
      double Xn[S], Mn[NM], g[S], J[S];
      load4(X + pp[d] * S, Xn);
      load5(M + pp[d] * ms, Mn);
      load4(gp + o, g);
      face_flux(Xc, Mc, Xn, Mn, g, J);
#pragma unroll
      for (int s = 0; s < S; ++s) fp[o + s] = J[s];
      load4(X + pm[d] * S, Xn);
      load5(M + pm[d] * ms, Mn);
      load4(gm + o, g);
      face_flux(Xc, Mc, Xn, Mn, g, J);
#pragma unroll
      for (int s = 0; s < S; ++s) fm[o + s] = J[s];
    }
  }
}

// ------------------------------------------------------------- reductions
constexpr int kAbsMaxBlocks = 1024;
constexpr int kAbsMaxThreads = 256;

// Pass 1: per-block max |a| (NaN ignored, like `if v > m: m = v`).
__global__ void k_absmax_partial(const double *__restrict__ a, int64_t n,
                                 double *__restrict__ partial) {
  __shared__ double red[kAbsMaxThreads / 32];
  double m = 0.0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const double v = fabs(a[i]);
    if (v > m) m = v;
  }
  m = block_max<kAbsMaxThreads>(m, red);
  if (threadIdx.x == 0) partial[blockIdx.x] = m;
}

// Pass 2: one block folds the partials into *result.
__global__ void k_absmax_final(const double *__restrict__ partial, int nparts, double *result) {
  __shared__ double red[kAbsMaxThreads / 32];
  double m = 0.0;
  for (int i = threadIdx.x; i < nparts; i += blockDim.x) m = fmax(m, partial[i]);
  m = block_max<kAbsMaxThreads>(m, red);
  if (threadIdx.x == 0) *result = m;
}

// Per-device workspace for the block partials of abs_max (allocated once).
static std::mutex g_ws_mutex;
static double *g_absmax_ws[64] = {nullptr};

static pf5d_status absmax_workspace(double **out) {
  int dev = 0;
  PF5D_CUDA(cudaGetDevice(&dev));
  PF5D_REQUIRE(dev >= 0 && dev < 64, PF5D_ERR_ARG, "device ordinal %d out of range", dev);
  std::lock_guard<std::mutex> lock(g_ws_mutex);
  if (!g_absmax_ws[dev]) PF5D_CUDA(cudaMalloc(&g_absmax_ws[dev], kAbsMaxBlocks * sizeof(double)));
  *out = g_absmax_ws[dev];
  return PF5D_OK;
}

// Scratch of pf5d_oob_stats (five words).  A call takes one and gives it back
// once its stream has been synchronised, so whoever takes it next, on any stream
// or thread, finds it unused; at most kOobScratch are kept per device.  An
// allocation per call had the driver map and unmap memory at every
// synchronisation.  A call on 200x160 / 128^3 points, median (99th percentile):
// 594 us (59 ms) / 1276 us (5.9 ms) -> 36 (47) / 48 (58).
constexpr size_t kOobScratch = 8;
constexpr int kOobDevices = 64;
static std::vector<unsigned long long *> g_oob_free[kOobDevices];

static pf5d_status oob_scratch_take(int dev, unsigned long long **out, cudaStream_t s) {
  if (dev < kOobDevices) {
    std::lock_guard<std::mutex> lock(g_ws_mutex);
    if (!g_oob_free[dev].empty()) {
      *out = g_oob_free[dev].back();
      g_oob_free[dev].pop_back();
      return PF5D_OK;
    }
  }
  PF5D_CUDA(cudaMallocAsync(out, 5 * sizeof(unsigned long long), s));
  return PF5D_OK;
}

static void oob_scratch_give(int dev, unsigned long long *d, cudaStream_t s) {
  if (dev < kOobDevices) {
    std::lock_guard<std::mutex> lock(g_ws_mutex);
    if (g_oob_free[dev].size() < kOobScratch) {
      g_oob_free[dev].push_back(d);
      return;
    }
  }
  cudaFreeAsync(d, s);
}

__global__ void k_clamp(double *X, int64_t npts, int nc) {
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < npts;
       p += (int64_t)gridDim.x * blockDim.x) {
    double total = 0.0;
    for (int s = 0; s < nc; ++s) total = total + X[p * nc + s];
    if (total > 1.0) {
      const double inv = 1.0 / total;
      for (int s = 0; s < nc; ++s) X[p * nc + s] = X[p * nc + s] * inv;
    }
  }
}

__global__ void k_update(double *X, double *dX, int64_t n, double dt) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const double d = dX[i] * dt;
    dX[i] = d;
    X[i] = X[i] + d;
  }
}

// Order-preserving map of doubles to unsigned keys (for atomic min/max).
__device__ __forceinline__ unsigned long long dkey(double v) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(v);
  return (b >> 63) ? ~b : (b | 0x8000000000000000ULL);
}
__host__ __device__ inline double dkey_inv(unsigned long long k) {
  const unsigned long long b = (k >> 63) ? (k & 0x7fffffffffffffffULL) : ~k;
  double v;
  memcpy(&v, &b, sizeof(v));
  return v;
}

// stats: [0] non-finite count, [1] max row sum key, [2] min row sum key,
// [3] max component key, [4] min component key.  Row sums left to right
// (numpy's sum over a length-4 axis).
//
// Bound by the one read of X.  A thread folds its points, a warp its lanes and
// a block its warps, so a block touches each of the five words once: with one
// atomic per thread the same-address atomics took 783 us at 128^3 points,
// 16 us now.
constexpr int kOobThreads = 256, kOobStats = 5;

__device__ __forceinline__ unsigned long long oob_fold(int i, unsigned long long a,
                                                       unsigned long long b) {
  return i == 0 ? a + b : (i & 1) ? max(a, b) : min(a, b);
}

// VEC4: four components per point in 16-byte aligned rows (two double2 loads).
template <bool VEC4>
__global__ void __launch_bounds__(kOobThreads)
    k_oob_stats(const double *__restrict__ X, int64_t npts, int nc, unsigned long long *stats) {
  __shared__ unsigned long long red[kOobThreads / 32][kOobStats];
  unsigned long long k[kOobStats] = {0, 0, ~0ULL, 0, ~0ULL};
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < npts;
       p += (int64_t)gridDim.x * blockDim.x) {
    double sum = 0.0;
    bool finite = true;
    auto take = [&](double v) {
      if (!isfinite(v)) {
        finite = false;
        ++k[0];
      } else {
        k[3] = max(k[3], dkey(v));
        k[4] = min(k[4], dkey(v));
      }
      sum = sum + v;
    };
    if (VEC4) {
      const double2 a = __ldg(reinterpret_cast<const double2 *>(X) + 2 * p);
      const double2 b = __ldg(reinterpret_cast<const double2 *>(X) + 2 * p + 1);
      take(a.x);
      take(a.y);
      take(b.x);
      take(b.y);
    } else {
      for (int s = 0; s < nc; ++s) take(X[p * nc + s]);
    }
    if (finite) {
      k[1] = max(k[1], dkey(sum));
      k[2] = min(k[2], dkey(sum));
    }
  }
#pragma unroll
  for (int i = 0; i < kOobStats; ++i) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) k[i] = oob_fold(i, k[i], __shfl_xor_sync(0xffffffffu, k[i], o));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5][i] = k[i];
  }
  __syncthreads();
  if (threadIdx.x < kOobStats) {
    const int i = threadIdx.x;
    unsigned long long v = red[0][i];
    for (int w = 1; w < kOobThreads / 32; ++w) v = oob_fold(i, v, red[w][i]);
    if (i == 0) {
      if (v) atomicAdd(&stats[0], v);
    } else if (i & 1) {
      atomicMax(&stats[i], v);
    } else {
      atomicMin(&stats[i], v);
    }
  }
}

static bool dims_ok(int32_t dim, const int64_t *shape, int64_t &n0, int64_t &n1, int64_t &n2) {
  if (dim < 1 || dim > 3 || !shape) return false;
  n0 = shape[0];
  n1 = dim > 1 ? shape[1] : 1;
  n2 = dim > 2 ? shape[2] : 1;
  return n0 > 0 && n1 > 0 && n2 > 0;
}

}  // namespace pf5d

using namespace pf5d;

extern "C" {

const char *pf5d_last_error(void) { return g_last_error.c_str(); }
int32_t pf5d_version(void) { return 100; }

pf5d_status pf5d_interp4d(const double *comp, int64_t npts, const double *grid, int32_t n,
                          int32_t nprops, int32_t node_stride, double resolution,
                          const double *node_coord, double max_nn_dist, double *out,
                          int64_t out_stride, uint8_t *mask, uint32_t *flags, void *stream) {
  PF5D_REQUIRE(npts >= 0, PF5D_ERR_ARG, "npts < 0");
  if (npts == 0) return PF5D_OK;
  PF5D_REQUIRE(comp && grid && node_coord && out, PF5D_ERR_ARG, "null pointer");
  PF5D_REQUIRE(nprops == NP, PF5D_ERR_ARG, "nprops must be %d (got %d)", NP, nprops);
  PF5D_REQUIRE(node_stride >= nprops && n >= 2, PF5D_ERR_ARG, "bad table geometry");
  PF5D_REQUIRE(out_stride >= nprops, PF5D_ERR_ARG, "out_stride < nprops");
  PF5D_REQUIRE(((uintptr_t)comp & 15) == 0, PF5D_ERR_ARG, "comp must be 16-byte aligned");
  Table T;
  T.grid = grid;
  T.coord = node_coord;
  T.n = n;
  T.stride = node_stride;
  T.inv_step = 1.0 / resolution;
  T.threshold = 1.0 - 4.0 * resolution - 1e-9;
  T.max_nn_dist = max_nn_dist;
  k_interp4d<<<grid_for(npts, 128), 128, 0, as_stream(stream)>>>(comp, npts, T, out, out_stride,
                                                                  mask, flags);
  PF5D_LAUNCHED();
  return PF5D_OK;
}

pf5d_status pf5d_laplacian(int32_t dim, const int64_t *shape, int32_t ncomp, const double *c,
                           double dx, double *out, void *stream) {
  int64_t n0, n1, n2;
  PF5D_REQUIRE(dims_ok(dim, shape, n0, n1, n2), PF5D_ERR_DIM,
               "Laplacian not implemented for spatial_dims=%d", dim);
  PF5D_REQUIRE(c && out && ncomp > 0, PF5D_ERR_ARG, "bad arguments");
  const double inv_dx2 = 1.0 / (dx * dx);
  const int64_t npts = n0 * n1 * n2;
  const int64_t ny = dim == 1 ? 1 : shape[dim - 2], nx = shape[dim - 1], nz = dim == 3 ? n0 : 1;
  if (ncomp == S && (((uintptr_t)c | (uintptr_t)out) & 15) == 0 && nx < (1 << 30) &&
      ny <= 8 * 65535 && nz <= 65535 && laplacian4_pays(dim, nx, ny, nz)) {
    const dim3 grid((unsigned)((nx + 31) / 32), (unsigned)((ny + 7) / 8), (unsigned)nz), block(32, 8);
    const bool wide = aligned_to(c, 32);
    auto kernel = dim == 1   ? (wide ? k_laplacian4<1, 4> : k_laplacian4<1, 2>)
                  : dim == 2 ? (wide ? k_laplacian4<2, 4> : k_laplacian4<2, 2>)
                             : (wide ? k_laplacian4<3, 4> : k_laplacian4<3, 2>);
    kernel<<<grid, block, 0, as_stream(stream)>>>((int)n0, (int)n1, (int)n2, c, inv_dx2, out);
  } else {
    k_laplacian<<<grid_for(npts, 256), 256, 0, as_stream(stream)>>>(dim, n0, n1, n2, ncomp, c,
                                                                     inv_dx2, out);
  }
  PF5D_LAUNCHED();
  return PF5D_OK;
}

pf5d_status pf5d_kappa_subtract(double *mu, int64_t mu_stride, double *lap, const double *kappa,
                                int64_t npts, int32_t ncomp, void *stream) {
  PF5D_REQUIRE(mu && lap && kappa && ncomp > 0 && ncomp <= 8 && mu_stride >= ncomp,
               PF5D_ERR_ARG, "bad arguments");
  if (npts <= 0) return PF5D_OK;
  Kappa k{};
  for (int s = 0; s < ncomp; ++s) k.k[s] = kappa[s];
  k_kappa_subtract<<<grid_for(npts, 256), 256, 0, as_stream(stream)>>>(mu, mu_stride, lap, k,
                                                                        npts, ncomp);
  PF5D_LAUNCHED();
  return PF5D_OK;
}

pf5d_status pf5d_divergence_from_mu(int32_t dim, const int64_t *shape, int32_t ncomp,
                                    const double *X, const double *M, int64_t m_stride,
                                    const double *mu, int64_t mu_stride, double inv_dx,
                                    double *out, void *stream) {
  int64_t n0, n1, n2;
  PF5D_REQUIRE(dims_ok(dim, shape, n0, n1, n2), PF5D_ERR_DIM,
               "Unsupported system_dim=%d. Choose 1, 2, or 3.", dim);
  PF5D_REQUIRE(ncomp == S, PF5D_ERR_ARG, "ncomp must be %d", S);
  PF5D_REQUIRE(X && M && mu && out && m_stride >= NM && mu_stride >= S, PF5D_ERR_ARG,
               "bad arguments");
  const DivView V{X, mu, M, mu_stride, m_stride};
  const int a = (int)n0, b = (int)n1, c = (int)n2;
  cudaStream_t s = as_stream(stream);
  const int64_t nx = dim == 1 ? n0 : (dim == 2 ? n1 : n2), npts = n0 * n1 * n2;
  if (!march_pays(dim, npts, n1, nx, rows_of_nine(V, nx)))
    k_divergence_points<<<grid_for(npts, 128), 128, 0, s>>>(dim, n0, n1, n2, X, M, m_stride, mu,
                                                            mu_stride, inv_dx, out);
  else if (dim == 1) launch_divergence<1>(a, b, c, V, inv_dx, out, s);
  else if (dim == 2) launch_divergence<2>(a, b, c, V, inv_dx, out, s);
  else launch_divergence<3>(a, b, c, V, inv_dx, out, s);
  PF5D_LAUNCHED();
  return PF5D_OK;
}

pf5d_status pf5d_gradients_pm(int32_t dim, const int64_t *shape, int32_t ncomp, const double *c,
                              int64_t c_stride, double dx, double *gp, double *gm, void *stream) {
  int64_t n0, n1, n2;
  PF5D_REQUIRE(dims_ok(dim, shape, n0, n1, n2), PF5D_ERR_DIM,
               "Gradients not implemented for spatial_dims=%d", dim);
  PF5D_REQUIRE(c && gp && gm && ncomp > 0 && c_stride >= ncomp, PF5D_ERR_ARG, "bad arguments");
  const int64_t npts = n0 * n1 * n2;
  k_gradients_pm<<<grid_for(npts, 256), 256, 0, as_stream(stream)>>>(dim, n0, n1, n2, ncomp, c,
                                                                      c_stride, 1.0 / dx, gp, gm);
  PF5D_LAUNCHED();
  return PF5D_OK;
}

pf5d_status pf5d_fluxes_pm(int32_t dim, const int64_t *shape, int32_t ncomp, const double *X,
                           const double *M, int64_t m_stride, const double *gp, const double *gm,
                           double *fp, double *fm, void *stream) {
  int64_t n0, n1, n2;
  PF5D_REQUIRE(dims_ok(dim, shape, n0, n1, n2), PF5D_ERR_DIM,
               "Unsupported system_dim=%d. Choose 1, 2, or 3.", dim);
  PF5D_REQUIRE(ncomp == S && X && M && gp && gm && fp && fm && m_stride >= NM, PF5D_ERR_ARG,
               "bad arguments");
  const int64_t npts = n0 * n1 * n2;
  k_fluxes_pm<<<grid_for(npts, 128), 128, 0, as_stream(stream)>>>(dim, n0, n1, n2, X, M,
                                                                  m_stride, gp, gm, fp, fm);
  PF5D_LAUNCHED();
  return PF5D_OK;
}

pf5d_status pf5d_abs_max(const double *a, int64_t n, double *result, void *stream) {
  PF5D_REQUIRE(result && (a || n == 0) && n >= 0, PF5D_ERR_ARG, "bad arguments");
  double *ws = nullptr;
  pf5d_status st = absmax_workspace(&ws);
  if (st != PF5D_OK) return st;
  const unsigned blocks = n > 0 ? grid_for(n, kAbsMaxThreads) : 1;
  const unsigned nb = blocks < kAbsMaxBlocks ? blocks : kAbsMaxBlocks;
  k_absmax_partial<<<nb, kAbsMaxThreads, 0, as_stream(stream)>>>(a, n, ws);
  PF5D_LAUNCHED();
  k_absmax_final<<<1, kAbsMaxThreads, 0, as_stream(stream)>>>(ws, (int)nb, result);
  PF5D_LAUNCHED();
  return PF5D_OK;
}

pf5d_status pf5d_clamp_simplex(double *X, int64_t npts, int32_t ncomp, void *stream) {
  PF5D_REQUIRE(X && ncomp > 0 && npts >= 0, PF5D_ERR_ARG, "bad arguments");
  if (npts == 0) return PF5D_OK;
  k_clamp<<<grid_for(npts, 256), 256, 0, as_stream(stream)>>>(X, npts, ncomp);
  PF5D_LAUNCHED();
  return PF5D_OK;
}

pf5d_status pf5d_update(double *X, double *dXdt, int64_t n, double dt, void *stream) {
  PF5D_REQUIRE(X && dXdt && n >= 0, PF5D_ERR_ARG, "bad arguments");
  if (n == 0) return PF5D_OK;
  k_update<<<grid_for(n, 256), 256, 0, as_stream(stream)>>>(X, dXdt, n, dt);
  PF5D_LAUNCHED();
  return PF5D_OK;
}

pf5d_status pf5d_oob_stats(const double *X, int64_t npts, int32_t ncomp, double *stats,
                           void *stream) {
  PF5D_REQUIRE(X && stats && ncomp > 0 && npts > 0, PF5D_ERR_ARG, "bad arguments");
  cudaStream_t s = as_stream(stream);
  cudaStreamCaptureStatus capturing;
  PF5D_CUDA(cudaStreamIsCapturing(s, &capturing));
  PF5D_REQUIRE(capturing == cudaStreamCaptureStatusNone, PF5D_ERR_CUDA,
               "out_of_bounds reads its result back: not under capture");
  unsigned long long init[5] = {0ULL, 0ULL, ~0ULL, 0ULL, ~0ULL};
  unsigned long long *d = nullptr, h[5];
  int dev = 0;
  PF5D_CUDA(cudaGetDevice(&dev));
  pf5d_status st = oob_scratch_take(dev, &d, s);
  if (st != PF5D_OK) return st;
  PF5D_CUDA(cudaMemcpyAsync(d, init, sizeof(init), cudaMemcpyHostToDevice, s));
  if (ncomp == 4 && ((uintptr_t)X & 15) == 0)
    k_oob_stats<true><<<grid_for(npts, kOobThreads), kOobThreads, 0, s>>>(X, npts, ncomp, d);
  else
    k_oob_stats<false><<<grid_for(npts, kOobThreads), kOobThreads, 0, s>>>(X, npts, ncomp, d);
  PF5D_LAUNCHED();
  PF5D_CUDA(cudaMemcpyAsync(h, d, sizeof(h), cudaMemcpyDeviceToHost, s));
  PF5D_CUDA(cudaStreamSynchronize(s));
  oob_scratch_give(dev, d, s);
  stats[0] = (double)h[0];
  stats[1] = dkey_inv(h[1]);
  stats[2] = dkey_inv(h[2]);
  stats[3] = dkey_inv(h[3]);
  stats[4] = dkey_inv(h[4]);
  return PF5D_OK;
}

double pf5d_adaptive_dt(double dt_current, double xdotmax, double ctld, double t_cfl,
                        double lower_limit, double upper_limit, double max_change_factor) {
  return adaptive_dt(dt_current, xdotmax, ctld, t_cfl, lower_limit, upper_limit,
                     max_change_factor);
}

}  // extern "C"
