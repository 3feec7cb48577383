// pf5d_split32.cuh -- the two halves of the FP32c form's split rate
// evaluation, for one solve's kernels (precision.cu) and the batched ones
// (batch.cu).
#pragma once

#include "pf5d_fp32c.cuh"
#include "pf5d_gather.cuh"

namespace pf5d {

// ------------------------------------------------------------------------
// First half: mu/M and the closure X_Fe at every point of a 1D/2D/3D field
// into the split buffers (mm_mu, mm_m, mm_f).  The table values come first, up to K points of a cell per node load
// (pf5d_gather.cuh); then each thread takes its own points in order:
// Laplacian (neighbour order +axis0, -axis0, ...), mu offset, closure.  A
// thread's points are consecutive along y (2D) or z (3D), so it loads each
// point of that axis once.  Every value is formed by the same routines, in the
// same order, as in the fused kernels (weights32 / corner_acc32, mu_offset32,
// dsum32).
//
// Bound by the L1 data path, like the FP64 form's k_chem.  Rate stage (both
// kernels, ms), earlier kernels -> here: 256^3 0.927 -> 0.830, with two phases
// 1.21 -> 0.99; 512^2 0.0318 (fused) -> 0.0187.  512 points per block (PER = 4)
// keep a cell's run longer than K; below about 400^2 they leave SMs idle, and
// PER = 1 or 2 takes 0.0131 instead of 0.0161 at 389x250.  In 3D K = 2 with 24
// warps per SM beats K = 4 with 16 (0.95); in 2D, where few blocks run at a
// time anyway, K = 4 wins by a little.
// ------------------------------------------------------------------------
template <int NT, int PER, int K>
struct GatherSmem32 : GatherOrder<NT, PER, K> {
  float4 v[2][NT * PER];            // fractions, then mu 1..4 | M_Fe, M_1..3
  float v8[NT * PER];               // M_4
};

constexpr int kChemNT32 = 128;

template <int DIM, int PER>
struct ChemTile32 {
  static constexpr int NT = kChemNT32;
  static constexpr int BX = DIM == 1 ? NT * PER : 32;
  static constexpr int BY = DIM == 1 ? 1 : (DIM == 2 ? NT / 32 * PER : NT / 32);
  static constexpr int BZ = DIM == 3 ? PER : 1;
};

// The block's points: those from (bz, by, bx) on.
template <int DIM, int PER, int K>
__device__ __forceinline__ void chem32_body(const Rate32 &P, GatherSmem32<kChemNT32, PER, K> &g,
                                            int bx, int by, int bz) {
  constexpr int NT = kChemNT32;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const Table32 &T = P.T;
  const int64_t plane = (int64_t)P.ny * P.nx;
  // the point in slot q = j * NT + w * 32 + lane
  auto px = [&](int j, int l, int v) { return DIM == 1 ? bx + j * NT + v * 32 + l : bx + l; };
  auto py = [&](int j, int v) { return DIM == 1 ? 0 : (DIM == 2 ? by + PER * v + j : by + v); };
  auto pz = [&](int j) { return DIM == 3 ? bz + j : 0; };
  auto at = [&](int z, int y, int x) { return z * plane + (int64_t)y * P.nx + x; };
  gather_begin(g, tid);
  __syncthreads();
  int kr[PER];
#pragma unroll
  for (int j = 0; j < PER; ++j) {
    const int x = px(j, lane, w), y = py(j, w), z = pz(j);
    const bool valid = x < P.nx && y < P.ny && z < P.nz;
    const unsigned active = __ballot_sync(0xffffffffu, valid);
    kr[j] = kNoKey;
    if (valid) {
      const float4 d4 = __ldg(P.D + at(z, y, x));
      const float d[S] = {d4.x, d4.y, d4.z, d4.w};
      int ii[S] = {0, 0, 0, 0};
      float tt[S];
      const bool linear = cell32(T, d, dsum32(d), ii, tt);
      const int q = j * NT + tid;
      if (linear) g.v[0][q] = make_float4(tt[0], tt[1], tt[2], tt[3]);
      kr[j] = gather_rank(g, active, linear, ii, T.n, q);
    }
  }
  const int nitems = gather_sort(g, kr, tid);
  const float4 *g4 = reinterpret_cast<const float4 *>(T.grid);
  const int64_t s3 = 3, s2 = 3 * (int64_t)T.n, s1 = s2 * T.n, s0 = s1 * T.n;
  for (int it = tid; it < nitems; it += NT) {
    const unsigned e = g.items[it];
    const int s = (int)(e & 0xffffu), m = (int)(e >> 16);
    int q[K];
    Weights32 W[K];
    const unsigned cell0 = g.cell[g.order[s]];
    unsigned mine = 0;
#pragma unroll
    for (int j = 0; j < K; ++j) {
      q[j] = g.order[s + (j < m ? j : 0)];
      if (j < m) {
        if (g.cell[q[j]] == cell0) mine |= 1u << j;
        else g.left[atomicAdd(&g.nleft, 1)] = (unsigned short)q[j];
      }
      const float4 t4 = g.v[0][q[j]];
      const float tt[S] = {t4.x, t4.y, t4.z, t4.w};
      W[j] = weights32(tt);
    }
    float acc[K][NP];
    const float4 *base = g4 + (int64_t)cell0 * 3;
#pragma unroll
    for (int c = 0; c < 16; ++c) {
      const int b0 = (c >> 3) & 1, b1 = (c >> 2) & 1, b2 = (c >> 1) & 1, b3 = c & 1;
      const float4 *node = base + b0 * s0 + b1 * s1 + b2 * s2 + b3 * s3;
      const float4 a = __ldg(node), b = __ldg(node + 1), f = __ldg(node + 2);
#pragma unroll
      for (int j = 0; j < K; ++j) corner_acc32(c, W[j].wa[c >> 2] * W[j].wb[c & 3], a, b, f, acc[j]);
    }
#pragma unroll
    for (int j = 0; j < K; ++j)
      if (mine & (1u << j)) {
        g.v[0][q[j]] = make_float4(acc[j][0], acc[j][1], acc[j][2], acc[j][3]);
        g.v[1][q[j]] = make_float4(acc[j][4], acc[j][5], acc[j][6], acc[j][7]);
        g.v8[q[j]] = acc[j][8];
      }
  }
  unsigned flags = 0;
  gather_others(g, tid, [&](int q) {
    const int j = q / NT, v = (q / 32) % (NT / 32);
    const float4 d4 = __ldg(P.D + at(pz(j), py(j, v), px(j, q & 31, v)));
    const float d[S] = {d4.x, d4.y, d4.z, d4.w};
    float o[NP];
    interp32(P, d, dsum32(d), nullptr, nullptr, o, &flags);
    g.v[0][q] = make_float4(o[0], o[1], o[2], o[3]);
    g.v[1][q] = make_float4(o[4], o[5], o[6], o[7]);
    g.v8[q] = o[8];
  });
  raise_rate_flags(P.st, flags);
  if (kr[0] == kNoKey) return;                  // none of this thread's points is in the field
  const int x0 = px(0, lane, w), y0 = py(0, w), z0 = pz(0);
  float4 below, dc = __ldg(P.D + at(z0, y0, x0)), above;   // along the marching axis
  if (DIM == 2) below = __ldg(P.D + at(0, y0 == 0 ? P.ny - 1 : y0 - 1, x0));
  if (DIM == 3) below = __ldg(P.D + at(z0 == 0 ? P.nz - 1 : z0 - 1, y0, x0));
#pragma unroll
  for (int j = 0; j < PER; ++j) {
    if (kr[j] == kNoKey) break;
    const int x = px(j, lane, w), y = py(j, w), z = pz(j), q = j * NT + tid;
    constexpr int NB = 2 * DIM;
    float4 n4[NB];
    int k = 0;
    if (DIM == 1) {
      if (j > 0) dc = __ldg(P.D + at(0, 0, x));
    } else {
      above = __ldg(P.D + (DIM == 2 ? at(0, y + 1 == P.ny ? 0 : y + 1, x)
                                    : at(z + 1 == P.nz ? 0 : z + 1, y, x)));
      n4[k++] = above;
      n4[k++] = below;
    }
    if (DIM == 3) {
      n4[k++] = __ldg(P.D + at(z, y + 1 == P.ny ? 0 : y + 1, x));
      n4[k++] = __ldg(P.D + at(z, y == 0 ? P.ny - 1 : y - 1, x));
    }
    n4[k++] = __ldg(P.D + at(z, y, x + 1 == P.nx ? 0 : x + 1));
    n4[k] = __ldg(P.D + at(z, y, x == 0 ? P.nx - 1 : x - 1));
    const int64_t gi = at(z, y, x);
    const float d[S] = {dc.x, dc.y, dc.z, dc.w};
    float lap[S], off[S];
    {
      float n[S][NB];
#pragma unroll
      for (int i = 0; i < NB; ++i) {
        n[0][i] = n4[i].x;
        n[1][i] = n4[i].y;
        n[2][i] = n4[i].z;
        n[3][i] = n4[i].w;
      }
#pragma unroll
      for (int c = 0; c < S; ++c) lap[c] = lap32<NB>(n[c], d[c], P.inv_dx2);
    }
    mu_offset32(P, lap, P.sp ? __ldg(P.sp + gi) : 0.f, off);
    const float4 a = g.v[0][q], b = g.v[1][q];
    P.mm_mu[gi] = make_float4(a.x + off[0], a.y + off[1], a.z + off[2], a.w + off[3]);
    P.mm_m[gi] = make_float4(b.y, b.z, b.w, g.v8[q]);
    P.mm_f[gi] = make_float2(b.x, (float)(P.c_fe - dsum32(d)));
    if (DIM != 1) {
      below = dc;
      dc = above;
    }
  }
}

// ------------------------------------------------------------------------
// Second half: faces and divergence from D and the
// split buffers, without shared memory or barriers, as the FP64 form's k_flux:
// a warp of 32 columns (30 of them finished) marches along axis 0, carries the
// face along the march, and hands on the face between columns by shuffles.
// Same face routine and divergence order as the fused kernels.
//
// Bound by the latency of its loads and by issue.  256^3: 0.337 ms as a 32x8
// tile with a shared cp.async ring and five faces per point.
// ------------------------------------------------------------------------
constexpr int kFluxThreads32 = 128, kFluxCols32 = 30;

struct Pt32 {
  float4 d, mu, m;
  float2 f;
};

__device__ __forceinline__ Pt32 load_pt32(const Rate32 &P, int64_t g) {
  return Pt32{__ldg(P.D + g), __ldg(P.mm_mu + g), __ldg(P.mm_m + g), __ldg(P.mm_f + g)};
}

__device__ __forceinline__ float4 face_pts32(const Rate32 &P, const Pt32 &lo, const Pt32 &hi) {
  return face_flux32(P, lo.d, lo.mu, lo.m, lo.f, hi.d, hi.mu, hi.m, hi.f);
}

__device__ __forceinline__ float4 shfl_down4(const float4 &v) {
  return make_float4(__shfl_down_sync(0xffffffffu, v.x, 1), __shfl_down_sync(0xffffffffu, v.y, 1),
                     __shfl_down_sync(0xffffffffu, v.z, 1), __shfl_down_sync(0xffffffffu, v.w, 1));
}

// The block's part: strip bx of 30 columns, part by of axis 1 (3D) and bz of
// the march (2D: by).  Returns this thread's max |dX/dt|.
template <int DIM, int R>
__device__ __forceinline__ float flux32_body(const Rate32 &P, int bx, int by, int bz, int rows) {
  static_assert(DIM == 3 || R == 1, "rows per thread are of axis 1");
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int col = bx * kFluxCols32 + lane - 1, x = wrap_any(col, P.nx);
  // axis 0: the march, over [first, last); 3D: axis 1 is this warp's R rows
  const int n0 = DIM == 3 ? P.nz : P.ny;
  const int y = (by * 4 + w) * R;              // 3D
  const int first = (DIM == 3 ? bz : by * 4 + w) * rows;
  const int last = min(first + rows, n0);
  const bool out_lane = lane > 0 && lane <= kFluxCols32 && col < P.nx;
  float vmax = 0.f;
  if (first < n0 && (DIM == 2 || y < P.ny)) {          // whole warps
    auto at = [&](int i, int yy) {
      return DIM == 3 ? ((int64_t)i * P.ny + yy) * P.nx + x : (int64_t)i * P.nx + x;
    };
    // a thread's rows past the field's last one repeat it and write nothing
    auto row = [&](int r) { return DIM == 3 ? min(y + r, P.ny - 1) : 0; };
    const int ym = y == 0 ? P.ny - 1 : y - 1, yp = y + R >= P.ny ? 0 : y + R;
    Pt32 cur[R];
    float4 jm[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const Pt32 below = load_pt32(P, at(first == 0 ? n0 - 1 : first - 1, row(r)));
      cur[r] = load_pt32(P, at(first, row(r)));
      jm[r] = face_pts32(P, below, cur[r]);
    }
    for (int i = first; i < last; ++i) {
      const int ip = i + 1 == n0 ? 0 : i + 1;
      Pt32 up[R];
#pragma unroll
      for (int r = 0; r < R; ++r) up[r] = load_pt32(P, at(ip, row(r)));
      float4 jym = make_float4(0.f, 0.f, 0.f, 0.f);
      if (DIM == 3) jym = face_pts32(P, load_pt32(P, at(i, ym)), cur[0]);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        Pt32 nb{shfl_down4(cur[r].d), shfl_down4(cur[r].mu), shfl_down4(cur[r].m),
                make_float2(__shfl_down_sync(0xffffffffu, cur[r].f.x, 1),
                            __shfl_down_sync(0xffffffffu, cur[r].f.y, 1))};
        const float4 jx = face_pts32(P, cur[r], nb);
        const float4 jl = make_float4(
            __shfl_up_sync(0xffffffffu, jx.x, 1), __shfl_up_sync(0xffffffffu, jx.y, 1),
            __shfl_up_sync(0xffffffffu, jx.z, 1), __shfl_up_sync(0xffffffffu, jx.w, 1));
        float4 jyp = jym;
        if (DIM == 3) {
          // the last row's upper neighbour (for a row that repeats: unused)
          if (r == R - 1 || y + r + 1 >= P.ny) nb = load_pt32(P, at(i, yp));
          else nb = cur[r + 1 < R ? r + 1 : r];
          jyp = face_pts32(P, cur[r], nb);
        }
        const float4 jz = face_pts32(P, cur[r], up[r]);
        float out[S];
        const float az[S] = {jz.x - jm[r].x, jz.y - jm[r].y, jz.z - jm[r].z, jz.w - jm[r].w};
        const float ay[S] = {jyp.x - jym.x, jyp.y - jym.y, jyp.z - jym.z, jyp.w - jym.w};
        const float ax[S] = {jx.x - jl.x, jx.y - jl.y, jx.z - jl.z, jx.w - jl.w};
#pragma unroll
        for (int c = 0; c < S; ++c)
          out[c] = (DIM == 3 ? (az[c] + ay[c]) + ax[c] : az[c] + ax[c]) * P.flux_scale;
        if (out_lane && (DIM == 2 || y + r < P.ny)) store_rate(P.dX, at(i, row(r)), out, vmax);
        jm[r] = jz;
        jym = jyp;
        cur[r] = up[r];
      }
    }
  }
  return vmax;
}

}  // namespace pf5d
