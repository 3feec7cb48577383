// pf5d_colfft.cuh -- complex FFTs of a power-of-two length along a column, for
// the elastic term's column pass: a thread holds 8 elements in registers, the
// N / 8 threads of a column exchange them through shared memory between the
// stages.  Forward exp(-2 pi i jk/N), inverse exp(+2 pi i jk/N), both
// unnormalised.
//
// A mixed-radix Stockham autosort (decimation in time): radix-8 stages of span
// 1, 8, 64, then one radix-4 or radix-2 stage for what is left, each in natural
// order.  Thread t holds the elements t + (N/8) k, which are what every stage
// reads and what the last one leaves, so a transform exchanges only between its
// stages, and the inverse can follow the forward one in the same registers.
#pragma once

#include <cuda_runtime.h>

namespace pf5d {

// complex type traits of the column pass (FP64 double2, FP32c float2)
template <typename C> struct CT;
template <> struct CT<double2> { using R = double; };
template <> struct CT<float2> { using R = float; };
template <typename C>
__device__ __forceinline__ C cmk(typename CT<C>::R a, typename CT<C>::R b) {
  C c;
  c.x = a;
  c.y = b;
  return c;
}

template <typename C>
__device__ __forceinline__ C cmul(C a, C b) {
  return cmk<C>(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
template <typename C>
__device__ __forceinline__ C cadd(C a, C b) { return cmk<C>(a.x + b.x, a.y + b.y); }
template <typename C>
__device__ __forceinline__ C csub(C a, C b) { return cmk<C>(a.x - b.x, a.y - b.y); }
// times -i (forward) or +i (inverse)
template <typename C, bool INV>
__device__ __forceinline__ C crot(C a) {
  return INV ? cmk<C>(-a.y, a.x) : cmk<C>(a.y, -a.x);
}

template <typename C, bool INV>
__device__ __forceinline__ void dft4(C *u) {
  const C c0 = cadd(u[0], u[2]), c1 = cadd(u[1], u[3]);
  const C d0 = csub(u[0], u[2]), d1 = crot<C, INV>(csub(u[1], u[3]));
  u[0] = cadd(c0, c1);
  u[1] = cadd(d0, d1);
  u[2] = csub(c0, c1);
  u[3] = csub(d0, d1);
}

// Radix-8 by decimation in frequency: two length-4 transforms of the sums
// and of the twiddled differences (W8^n, n < 4).
template <typename C, bool INV>
__device__ __forceinline__ void dft8(C *v) {
  constexpr typename CT<C>::R h = (typename CT<C>::R)0.70710678118654752440;
  C a[4], b[4];
#pragma unroll
  for (int n = 0; n < 4; ++n) {
    a[n] = cadd(v[n], v[n + 4]);
    b[n] = csub(v[n], v[n + 4]);
  }
  b[1] = cmul(b[1], cmk<C>(h, INV ? h : -h));
  b[2] = crot<C, INV>(b[2]);
  b[3] = cmul(b[3], cmk<C>(-h, INV ? h : -h));
  dft4<C, INV>(a);
  dft4<C, INV>(b);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    v[2 * k] = a[k];
    v[2 * k + 1] = b[k];
  }
}

template <typename C, int R, bool INV>
__device__ __forceinline__ void dftr(C *v) {
  if constexpr (R == 8) {
    dft8<C, INV>(v);
  } else if constexpr (R == 4) {
    dft4<C, INV>(v);
  } else {
    const C a = v[0];
    v[0] = cadd(a, v[1]);
    v[1] = csub(a, v[1]);
  }
}

// The transform of one column by T = N / 8 threads.  A block's columns are
// neighbours in memory: element e of column cc of COLS columns sits at
// e * COLS + cc in shared memory.
template <typename C, int N, int COLS>
struct ColFFT {
  static constexpr int T = N / 8;
  static constexpr int kRadix8 = N >= 512 ? 3 : (N >= 64 ? 2 : 1);       // radix-8 stages
  static constexpr int L = N >> (3 * kRadix8);                           // radix of the last: 1 (none), 2, 4
  static constexpr int kStages = kRadix8 + (L > 1 ? 1 : 0);

  C tw[kStages][7];                 // twiddles of the registers 1..7, stages 1..

  // Stage s has span 8^s; its butterfly j = t (radix 8) or t, t + T, .. (last)
  // takes element j + (N / R) r with exp(-2 pi i r (j mod span) / (R span)).
  // table[m] = exp(-2 pi i m / N).
  __device__ __forceinline__ void load_twiddles(const C *__restrict__ table, int t) {
#pragma unroll
    for (int s = 1; s < kStages; ++s)
#pragma unroll
      for (int k = 1; k < 8; ++k) tw[s][k - 1] = table[twiddle(s, t, k)];
  }

  // v: x[t + T k] in register k, before and after
  template <bool INV>
  __device__ __forceinline__ void run(C v[8], C *buf, int t, int cc) const {
#pragma unroll
    for (int s = 0; s < kStages; ++s) {
      const bool tail = s == kRadix8;
      if (s > 0) {
#pragma unroll
        for (int k = 1; k < 8; ++k) {
          if (tail && k < 8 / L) continue;             // r = 0
          const C w = tw[s][k - 1];
          v[k] = cmul(v[k], INV ? cmk<C>(w.x, -w.y) : w);
        }
      }
      if (!tail) {
        dft8<C, INV>(v);
      } else if constexpr (L > 1) {
        // butterfly b of this thread: registers b + (8 / L) r
#pragma unroll
        for (int b = 0; b < 8 / L; ++b) {
          C u[L];
#pragma unroll
          for (int r = 0; r < L; ++r) u[r] = v[b + (8 / L) * r];
          dftr<C, L, INV>(u);
#pragma unroll
          for (int r = 0; r < L; ++r) v[b + (8 / L) * r] = u[r];
        }
      }
      if (s + 1 < kStages) {                           // to the next stage's elements
        const int span = 1 << (3 * s), m = t & (span - 1), d = (t - m) * 8 + m;
        __syncthreads();
#pragma unroll
        for (int r = 0; r < 8; ++r) buf[(d + r * span) * COLS + cc] = v[r];
        __syncthreads();
#pragma unroll
        for (int r = 0; r < 8; ++r) v[r] = buf[(t + T * r) * COLS + cc];
      }
    }
  }

 private:
  static __device__ __forceinline__ int twiddle(int s, int t, int k) {
    const int span = 1 << (3 * s);
    if (s < kRadix8) return k * (t & (span - 1)) * (N / (8 * span));
    const int b = k % (8 / L), r = k / (8 / L);        // last stage: span N / L
    return r * (t + T * b);
  }
};

}  // namespace pf5d
