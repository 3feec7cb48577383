// The shared table gathers of the mu/M kernels (pf5d_gather.cuh) run on the
// host, for the sanitizers: see test_gather_host.py.
#include "cuda_runtime.h"

#include "pf5d_gather.cuh"

using namespace pf5d;

// One block of k_chem's table values: the ordering, the shared gathers, the rest.
template <int PER, int K>
static bool block(const Table &T, const std::vector<double> &pts, int nvalid, const char *what) {
  constexpr int NT = 128, N = NT * PER;
  using G = GatherSmem<NT, PER, K>;
  std::vector<G> store(1);
  G &g = store[0];
  std::memset(static_cast<void *>(&g), 0xff, sizeof(G));
  std::vector<double> out(N * NP, 0.0);
  std::vector<unsigned> flags(NT, 0u);
  run_block(NT, [&](int tid) {
    gather_begin(g, tid);
    __syncthreads();
    int kr[PER];
    for (int j = 0; j < PER; ++j) {
      const int q = j * NT + tid;
      double x[S] = {0.0, 0.0, 0.0, 0.0};
      if (q < nvalid) for (int c = 0; c < S; ++c) x[c] = pts[4 * q + c];
      kr[j] = gather_add(g, T, q < nvalid, x, q);
    }
    const int items = gather_sort(g, kr, tid);
    gather_values<true>(g, T, items, tid);
    gather_rest<true>(g, T, tid, &flags[tid], [&](int q, double x[S]) {
      if (q >= nvalid) std::abort();
      for (int c = 0; c < S; ++c) x[c] = pts[4 * q + c];
    });
    for (int j = 0; j < PER; ++j)
      if (kr[j] != kNoKey) gather_get(g, j * NT + tid, &out[(j * NT + tid) * NP]);
  });
  unsigned any = 0, want_any = 0;
  for (unsigned f : flags) any |= f;
  for (int q = 0; q < nvalid; ++q) {
    double v[NP];
    interp_point<true>(T, &pts[4 * q], v, &want_any);
    if (std::memcmp(v, &out[q * NP], sizeof(v)) != 0 &&
        !(std::isnan(v[0]) && std::isnan(out[q * NP]))) {
      std::printf("%s, PER %d, K %d, %d points: slot %d\n", what, PER, K, nvalid, q);
      return false;
    }
  }
  if (any != want_any) std::printf("%s: flags %x, not %x\n", what, any, want_any);
  return any == want_any;
}

int main() {
  const int n = 11;
  const double h = 0.1;
  std::vector<double> coord(n), grid((size_t)n * n * n * n * 10);
  for (int i = 0; i < n; ++i) coord[i] = i / 10.0;
  std::mt19937_64 rng(5);
  std::uniform_real_distribution<double> u01(0.0, 1.0);
  size_t at = 0;
  for (int a = 0; a < n; ++a)
    for (int b = 0; b < n; ++b)
      for (int c = 0; c < n; ++c)
        for (int d = 0; d < n; ++d)
          for (int p = 0; p < 10; ++p)
            grid[at++] = a + b + c + d <= n - 1 ? u01(rng) : std::numeric_limits<double>::quiet_NaN();
  const Table T{grid.data(), coord.data(), n, 10, 1.0 / h, 1.0 - 4.0 * h - 1e-9, 0.0};
  const double inf = std::numeric_limits<double>::infinity();
  const char *kinds[] = {"one cell", "linear region", "mixed", "outside", "far off", "not finite",
                         "two cells of a bin"};
  for (int kind = 0; kind < 7; ++kind) {
    std::vector<double> pts(4 * 512);
    for (int q = 0; q < 512; ++q) {
      double *x = &pts[4 * q];
      for (int c = 0; c < S; ++c) {
        const double r = u01(rng);
        if (kind == 0) x[c] = 0.1 * r;
        if (kind == 1) x[c] = 0.15 * r;
        if (kind == 2) x[c] = 0.4 * r;
        if (kind == 3) x[c] = 1.3 * r - 0.1;
        if (kind == 4) x[c] = 1e3 * (r - 0.5);
        if (kind == 5) x[c] = r < 0.1 ? inf : r < 0.2 ? -inf : r < 0.3 ? std::nan("") : 0.2 * r;
        // cells (0, 1, 0, 0) and (0, 0, 2, 3) share a bin: 13 = 2 * 5 + 3
        const double one[S] = {0.01, 0.15, 0.05, 0.05}, other[S] = {0.01, 0.05, 0.25, 0.35};
        if (kind == 6) x[c] = q & 1 ? one[c] : other[c];
      }
    }
    for (int nv : {1, 31, 88, 128, 300, 511, 512}) {
      const char *what = kinds[kind];
      if (nv <= 128 && !block<1, 2>(T, pts, nv, what)) return 1;
      if (nv <= 256 && !(block<2, 2>(T, pts, nv, what) && block<2, 3>(T, pts, nv, what))) return 1;
      if (!(block<4, 2>(T, pts, nv, what) && block<4, 3>(T, pts, nv, what) &&
            block<4, 4>(T, pts, nv, what)))
        return 1;
    }
  }
  return 0;
}
