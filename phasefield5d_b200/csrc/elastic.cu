// elastic.cu -- rank-1 Khachaturyan elastic term around one cuFFT pair
// (phasefield5d/solver/elastic.py:147-263, scipy path 242-263):
//   s(x)  = sum_s (X[x,s] - X0[s]) * l[s]            (k_misfit, elastic.py:21-29)
//   S(k)  = rfftn(s) * B(k)                          (cuFFT D2Z + k_bmul)
//   s'(x) = irfftn(S)                                (cuFFT Z2D; 1/N folded into B)
//   mu   += s'(x) * l                                (k_expand_add)
// Compiled with -fmad=false.
#include <cmath>
#include <vector>

#include "pf5d_device.cuh"
#include "pf5d_fft.h"
#include "pf5d_colfft.cuh"

namespace pf5d {

#define PF5D_CUFFT(call)                                                           \
  do {                                                                             \
    cufftResult r_ = (call);                                                       \
    if (r_ != CUFFT_SUCCESS) {                                                     \
      set_error("%s:%d %s: cufft error %d", __FILE__, __LINE__, #call, (int)r_);   \
      return PF5D_ERR_CUFFT;                                                       \
    }                                                                              \
  } while (0)

pf5d_status fft_create(int dim, const int64_t *shape, FFTPair *p, bool plans) {
  PF5D_REQUIRE(dim >= 1 && dim <= 3, PF5D_ERR_DIM,
               "make_elastic_updater not implemented for spatial_dim=%d", dim);
  long long n[3];
  int64_t npts = 1;
  for (int d = 0; d < dim; ++d) {
    PF5D_REQUIRE(shape[d] > 0, PF5D_ERR_ARG, "bad shape");
    n[d] = shape[d];
    npts *= shape[d];
  }
  const int64_t nk = npts / shape[dim - 1] * (shape[dim - 1] / 2 + 1);
  p->npts = npts;
  p->nk = nk;
  if (!plans) return PF5D_OK;
  size_t ws = 0;
  PF5D_CUFFT(cufftCreate(&p->fwd));
  PF5D_CUFFT(cufftMakePlanMany64(p->fwd, dim, n, nullptr, 1, 0, nullptr, 1, 0, CUFFT_D2Z, 1, &ws));
  PF5D_CUFFT(cufftCreate(&p->inv));
  PF5D_CUFFT(cufftMakePlanMany64(p->inv, dim, n, nullptr, 1, 0, nullptr, 1, 0, CUFFT_Z2D, 1, &ws));
  p->ready = true;
  return PF5D_OK;
}

void fft_destroy(FFTPair *p) {
  if (p->ready) {
    cufftDestroy(p->fwd);
    cufftDestroy(p->inv);
  }
  p->ready = false;
}

pf5d_status fft_forward(FFTPair *p, double *s, cufftDoubleComplex *k, cudaStream_t stream) {
  PF5D_CUFFT(cufftSetStream(p->fwd, stream));
  PF5D_CUFFT(cufftExecD2Z(p->fwd, s, k));
  return PF5D_OK;
}

pf5d_status fft_inverse(FFTPair *p, cufftDoubleComplex *k, double *s, cudaStream_t stream) {
  PF5D_CUFFT(cufftSetStream(p->inv, stream));
  PF5D_CUFFT(cufftExecZ2D(p->inv, k, s));
  return PF5D_OK;
}

// ------------------------------------------------------------------------
// Column pass: along axis 0 of the spectrum, the length-N transform, the
// B(k)/N multiply and the inverse transform, COLS neighbouring columns per
// block (N / 8 threads each, pf5d_colfft.cuh); the spectrum is read and written
// once.  The twiddles and B(k) do not depend on the kernel before, so they are
// loaded ahead of the wait for it.
//
// Bound by latency in 2D (one round of blocks): 512^2 8.4 us as one 256-thread
// block per column with every stage in shared memory, 4.4 here, the whole term
// 14.5 -> 10.0 (FP32c 12.5 -> 8.1), with the same bits.  By HBM in 3D: 256^3
// 84 us for 0.68 GB (8.1 TB/s of which L2 serves a part), the whole term
// 364 us with cuFFT's 3D plans and a separate multiply -> 312; 64x100x90
// 26 -> 19.5.  The precision form keeps the 3D plans: its elastic term is FP32,
// and another order of roundings there shows in late fields (4e-10 of X).
// ------------------------------------------------------------------------
template <typename C, int N, int COLS>
__global__ void __launch_bounds__(N / 8 * COLS)
    k_colpass(C *__restrict__ k, const typename CT<C>::R *__restrict__ bk, int64_t ncol,
              const C *__restrict__ table, const unsigned *halt) {
  using F = ColFFT<C, N, COLS>;
  extern __shared__ __align__(16) unsigned char craw[];
  C *buf = reinterpret_cast<C *>(craw);
  const int cc = threadIdx.x % COLS, t = threadIdx.x / COLS;
  const int64_t c = (int64_t)blockIdx.x * COLS + cc;
  const bool valid = c < ncol;
  F fft;
  fft.load_twiddles(table, t);
  typename CT<C>::R m[8];
#pragma unroll
  for (int r = 0; r < 8; ++r) m[r] = valid ? __ldg(bk + (int64_t)(t + F::T * r) * ncol + c) : 0;
  pdl_wait();
  if (halt && *halt) return;
  C v[8];
#pragma unroll
  for (int r = 0; r < 8; ++r) v[r] = valid ? k[(int64_t)(t + F::T * r) * ncol + c] : cmk<C>(0, 0);
  fft.template run<false>(v, buf, t, cc);
#pragma unroll
  for (int r = 0; r < 8; ++r) v[r] = cmk<C>(v[r].x * m[r], v[r].y * m[r]);
  fft.template run<true>(v, buf, t, cc);
  if (!valid) return;
#pragma unroll
  for (int r = 0; r < 8; ++r) k[(int64_t)(t + F::T * r) * ncol + c] = v[r];
}

template <typename C>
static pf5d_status colpass_dispatch(const ColPass *c, C *k, const typename CT<C>::R *bk,
                                    const C *tw, const unsigned *halt, cudaStream_t stream);

pf5d_status colpass_create(int dim, const int64_t *shape, ColPass *c, bool fp32) {
  const int64_t n0 = shape[0], last = shape[dim - 1];
  PF5D_REQUIRE((dim == 2 || dim == 3) && colpass_fits(n0) && last >= 2, PF5D_ERR_ARG,
               "column pass needs a power-of-two axis 0 in [8, 1024]");
  c->n0 = (int)n0;
  c->ncol = (dim == 3 ? shape[1] : 1) * (last / 2 + 1);
  c->fp32 = fp32;
  long long n[2] = {(long long)shape[1], (long long)last};
  size_t ws = 0;
  PF5D_CUFFT(cufftCreate(&c->rfwd));
  PF5D_CUFFT(cufftMakePlanMany64(c->rfwd, dim - 1, n, nullptr, 1, 0, nullptr, 1, 0,
                                 fp32 ? CUFFT_R2C : CUFFT_D2Z, n0, &ws));
  PF5D_CUFFT(cufftCreate(&c->rinv));
  PF5D_CUFFT(cufftMakePlanMany64(c->rinv, dim - 1, n, nullptr, 1, 0, nullptr, 1, 0,
                                 fp32 ? CUFFT_C2R : CUFFT_Z2D, n0, &ws));
  c->ready = true;
  // exp(-2 pi i m / n0) in FP64, rounded once for the FP32 form
  std::vector<double2> tw(n0);
  std::vector<float2> tw32(n0);
  const double pi = 3.14159265358979323846;
  for (int64_t m = 0; m < n0; ++m) {
    const double ang = 2.0 * pi * (double)m / (double)n0;
    tw[m] = make_double2(std::cos(ang), -std::sin(ang));
    tw32[m] = make_float2((float)tw[m].x, (float)tw[m].y);
  }
  if (fp32) {
    PF5D_CUDA(cudaMalloc(&c->tw32, tw32.size() * sizeof(float2)));
    PF5D_CUDA(cudaMemcpy(c->tw32, tw32.data(), tw32.size() * sizeof(float2), cudaMemcpyHostToDevice));
    return colpass_dispatch<float2>(c, nullptr, nullptr, nullptr, nullptr, nullptr);
  }
  PF5D_CUDA(cudaMalloc(&c->tw, tw.size() * sizeof(double2)));
  PF5D_CUDA(cudaMemcpy(c->tw, tw.data(), tw.size() * sizeof(double2), cudaMemcpyHostToDevice));
  return colpass_dispatch<double2>(c, nullptr, nullptr, nullptr, nullptr, nullptr);
}

void colpass_destroy(ColPass *c) {
  if (c->ready) {
    cufftDestroy(c->rfwd);
    cufftDestroy(c->rinv);
  }
  cudaFree(c->tw);
  cudaFree(c->tw32);
  c->tw = nullptr;
  c->tw32 = nullptr;
  c->ready = false;
}

pf5d_status colpass_rows_forward(ColPass *c, double *s, cufftDoubleComplex *k,
                                 cudaStream_t stream) {
  PF5D_CUFFT(cufftSetStream(c->rfwd, stream));
  PF5D_CUFFT(cufftExecD2Z(c->rfwd, s, k));
  return PF5D_OK;
}

pf5d_status colpass_rows_inverse(ColPass *c, cufftDoubleComplex *k, double *s,
                                 cudaStream_t stream) {
  PF5D_CUFFT(cufftSetStream(c->rinv, stream));
  PF5D_CUFFT(cufftExecZ2D(c->rinv, k, s));
  return PF5D_OK;
}

template <typename C, int N, int COLS>
static pf5d_status launch_colpass(const ColPass *c, C *k, const typename CT<C>::R *bk,
                                  const C *tw, const unsigned *halt, cudaStream_t stream) {
  const int smem = N * COLS * (int)sizeof(C);
  if (!k) {                          // set-up call from colpass_create
    PF5D_CUDA(cudaFuncSetAttribute(k_colpass<C, N, COLS>,
                                   cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    return PF5D_OK;
  }
  PF5D_CUDA(launch_pdl(k_colpass<C, N, COLS>, dim3((unsigned)((c->ncol + COLS - 1) / COLS)),
                       dim3(N / 8 * COLS), smem, stream, k, bk, c->ncol, tw, halt));
  return PF5D_OK;
}

// Columns per block: 8 fill whole lines, but a 2D spectrum has too few columns
// for that many per SM; 2 there.
template <typename C, int N>
static pf5d_status launch_columns(const ColPass *c, C *k, const typename CT<C>::R *bk,
                                  const C *tw, const unsigned *halt, cudaStream_t stream) {
  constexpr int MANY = N <= 512 ? 8 : 4;
  if (c->ncol >= (int64_t)sm_count() * 2 * MANY)
    return launch_colpass<C, N, MANY>(c, k, bk, tw, halt, stream);
  return launch_colpass<C, N, 2>(c, k, bk, tw, halt, stream);
}

template <typename C>
static pf5d_status colpass_dispatch(const ColPass *c, C *k, const typename CT<C>::R *bk,
                                    const C *tw, const unsigned *halt, cudaStream_t stream) {
  switch (c->n0) {
    case 8: return launch_columns<C, 8>(c, k, bk, tw, halt, stream);
    case 16: return launch_columns<C, 16>(c, k, bk, tw, halt, stream);
    case 32: return launch_columns<C, 32>(c, k, bk, tw, halt, stream);
    case 64: return launch_columns<C, 64>(c, k, bk, tw, halt, stream);
    case 128: return launch_columns<C, 128>(c, k, bk, tw, halt, stream);
    case 256: return launch_columns<C, 256>(c, k, bk, tw, halt, stream);
    case 512: return launch_columns<C, 512>(c, k, bk, tw, halt, stream);
    case 1024: return launch_columns<C, 1024>(c, k, bk, tw, halt, stream);
    default: set_error("column pass: unsupported n0 %d", c->n0); return PF5D_ERR_ARG;
  }
}

pf5d_status colpass_columns(ColPass *c, cufftDoubleComplex *k, const double *bk,
                            const unsigned *halt, cudaStream_t stream) {
  return colpass_dispatch<double2>(c, reinterpret_cast<double2 *>(k), bk, c->tw, halt, stream);
}

pf5d_status colpass_columns32(ColPass *c, cufftComplex *k, const float *bk,
                              const unsigned *halt, cudaStream_t stream) {
  return colpass_dispatch<float2>(c, reinterpret_cast<float2 *>(k), bk, c->tw32, halt, stream);
}

pf5d_status colpass_rows_forward32(ColPass *c, float *s, cufftComplex *k, cudaStream_t stream) {
  PF5D_CUFFT(cufftSetStream(c->rfwd, stream));
  PF5D_CUFFT(cufftExecR2C(c->rfwd, s, k));
  return PF5D_OK;
}

pf5d_status colpass_rows_inverse32(ColPass *c, cufftComplex *k, float *s, cudaStream_t stream) {
  PF5D_CUFFT(cufftSetStream(c->rinv, stream));
  PF5D_CUFFT(cufftExecC2R(c->rinv, k, s));
  return PF5D_OK;
}

__global__ void k_misfit(const double *__restrict__ X, int64_t npts, Vec4 x0, Vec4 l,
                         double *__restrict__ s, const unsigned *halt) {
  if (halt && *halt) return;
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < npts;
       p += (int64_t)gridDim.x * blockDim.x) {
    const double2 a = reinterpret_cast<const double2 *>(X + 4 * p)[0];
    const double2 b = reinterpret_cast<const double2 *>(X + 4 * p)[1];
    double acc = 0.0;
    acc = acc + (a.x - x0.v[0]) * l.v[0];
    acc = acc + (a.y - x0.v[1]) * l.v[1];
    acc = acc + (b.x - x0.v[2]) * l.v[2];
    acc = acc + (b.y - x0.v[3]) * l.v[3];
    s[p] = acc;
  }
}

// numpy's complex *= real multiplies both parts by the real factor.
__global__ void k_bmul(cufftDoubleComplex *__restrict__ k, const double *__restrict__ bk,
                       int64_t nk, const unsigned *halt) {
  if (halt && *halt) return;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nk;
       i += (int64_t)gridDim.x * blockDim.x) {
    const double b = bk[i];
    cufftDoubleComplex v = k[i];
    v.x = v.x * b;
    v.y = v.y * b;
    k[i] = v;
  }
}

// One component of one point per thread: four lanes cover the 32 bytes of a
// point, so a warp touches a quarter of the lines that one point per lane would
// (rows of nine values at 128^3: 56 -> 44 us).
__global__ void k_expand_add(double *mu, int64_t mus, const double *__restrict__ s, Vec4 l,
                             int64_t npts) {
  const int c = threadIdx.x & 3;                     // the grid's stride keeps it
  const double lc = c == 0 ? l.v[0] : (c == 1 ? l.v[1] : (c == 2 ? l.v[2] : l.v[3]));
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < 4 * npts;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t p = i >> 2;
    mu[p * mus + c] = mu[p * mus + c] + s[p] * lc;
  }
}

pf5d_status launch_misfit(const double *X, int64_t npts, Vec4 x0, Vec4 l, double *s,
                          const unsigned *halt, cudaStream_t stream) {
  k_misfit<<<grid_for(npts, 256), 256, 0, stream>>>(X, npts, x0, l, s, halt);
  PF5D_LAUNCHED();
  return PF5D_OK;
}

pf5d_status launch_bmul(cufftDoubleComplex *k, const double *bk, int64_t nk, const unsigned *halt,
                        cudaStream_t stream) {
  k_bmul<<<grid_for(nk, 256), 256, 0, stream>>>(k, bk, nk, halt);
  PF5D_LAUNCHED();
  return PF5D_OK;
}

pf5d_status launch_expand_add(double *mu, int64_t mu_stride, const double *s, Vec4 l,
                              int64_t npts, cudaStream_t stream) {
  k_expand_add<<<grid_for(4 * npts, 256), 256, 0, stream>>>(mu, mu_stride, s, l, npts);
  PF5D_LAUNCHED();
  return PF5D_OK;
}

pf5d_status upload_bk_scaled(const double *bk_host, int64_t nk, int64_t npts, double **bk_dev) {
  std::vector<double> h(nk);
  const double inv_n = 1.0 / (double)npts;
  for (int64_t i = 0; i < nk; ++i) h[i] = bk_host[i] * inv_n;
  PF5D_CUDA(cudaMalloc(bk_dev, nk * sizeof(double)));
  PF5D_CUDA(cudaMemcpy(*bk_dev, h.data(), nk * sizeof(double), cudaMemcpyHostToDevice));
  return PF5D_OK;
}

}  // namespace pf5d

using namespace pf5d;

struct pf5d_elastic {
  int dim = 0;
  Vec4 x0{}, l{};
  FFTPair fft;
  ColPass colp;                      // in place of fft where axis 0 allows it
  bool use_colpass = false;
  double *bk = nullptr;
  double *s = nullptr;
  cufftDoubleComplex *k = nullptr;
};

extern "C" {

pf5d_status pf5d_elastic_create(int32_t dim, const int64_t *shape, const double *x0,
                                const double *lvec, const double *bk, pf5d_elastic **out) {
  PF5D_REQUIRE(out && shape && x0 && lvec && bk, PF5D_ERR_ARG, "null argument");
  auto *h = new pf5d_elastic();
  h->dim = dim;
  for (int c = 0; c < 4; ++c) {
    h->x0.v[c] = x0[c];
    h->l.v[c] = lvec[c];
  }
  if ((dim == 2 || dim == 3) && colpass_fits(shape[0])) {
    h->use_colpass = colpass_create(dim, shape, &h->colp, false) == PF5D_OK;
    if (!h->use_colpass) colpass_destroy(&h->colp);
  }
  pf5d_status st = fft_create(dim, shape, &h->fft, !h->use_colpass);
  if (st == PF5D_OK) st = upload_bk_scaled(bk, h->fft.nk, h->fft.npts, &h->bk);
  if (st == PF5D_OK && cudaMalloc(&h->s, h->fft.npts * sizeof(double)) != cudaSuccess)
    st = PF5D_ERR_CUDA;
  if (st == PF5D_OK && cudaMalloc(&h->k, h->fft.nk * sizeof(cufftDoubleComplex)) != cudaSuccess)
    st = PF5D_ERR_CUDA;
  if (st != PF5D_OK) {
    pf5d_elastic_destroy(h);
    return st;
  }
  *out = h;
  return PF5D_OK;
}

pf5d_status pf5d_elastic_apply(pf5d_elastic *h, double *mu, int64_t mu_stride, const double *X,
                               void *stream) {
  PF5D_REQUIRE(h && mu && X && mu_stride >= 4, PF5D_ERR_ARG, "bad arguments");
  PF5D_REQUIRE(((uintptr_t)X & 15) == 0, PF5D_ERR_ARG, "X must be 16-byte aligned");
  cudaStream_t s = as_stream(stream);
  pf5d_status st;
  if ((st = launch_misfit(X, h->fft.npts, h->x0, h->l, h->s, nullptr, s)) != PF5D_OK) return st;
  if (h->use_colpass) {
    if ((st = colpass_rows_forward(&h->colp, h->s, h->k, s)) != PF5D_OK) return st;
    if ((st = colpass_columns(&h->colp, h->k, h->bk, nullptr, s)) != PF5D_OK) return st;
    if ((st = colpass_rows_inverse(&h->colp, h->k, h->s, s)) != PF5D_OK) return st;
  } else {
    if ((st = fft_forward(&h->fft, h->s, h->k, s)) != PF5D_OK) return st;
    if ((st = launch_bmul(h->k, h->bk, h->fft.nk, nullptr, s)) != PF5D_OK) return st;
    if ((st = fft_inverse(&h->fft, h->k, h->s, s)) != PF5D_OK) return st;
  }
  return launch_expand_add(mu, mu_stride, h->s, h->l, h->fft.npts, s);
}

pf5d_status pf5d_elastic_destroy(pf5d_elastic *h) {
  if (!h) return PF5D_OK;
  fft_destroy(&h->fft);
  colpass_destroy(&h->colp);
  cudaFree(h->bk);
  cudaFree(h->s);
  cudaFree(h->k);
  delete h;
  return PF5D_OK;
}

}  // extern "C"
