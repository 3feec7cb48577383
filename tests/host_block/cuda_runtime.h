// Host stand-ins for the CUDA names that the headers under test use: a block's
// threads are threads, its barriers are barriers, and the lanes of a warp's
// collective meet under a lock.
#pragma once

#include <atomic>
#include <cmath>
#include <condition_variable>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <limits>
#include <map>
#include <mutex>
#include <random>
#include <thread>
#include <vector>

#include <pthread.h>

#define __host__
#define __device__
#define __forceinline__ inline
#define __noinline__
struct double2 { double x, y; };
inline double2 make_double2(double x, double y) { return {x, y}; }
struct Index { unsigned x, y, z; };
inline thread_local Index threadIdx;
inline Index blockDim;
inline pthread_barrier_t block_barrier;

struct Meeting {                     // of the lanes of a mask
  int count = 0;
  unsigned turn = 0;
  uint64_t in[32], out[32];
};
struct Warp {
  std::mutex m;
  std::condition_variable cv;
  std::map<unsigned, Meeting> of;
};
inline Warp warps[32];
inline const uint64_t *meet(unsigned mask, uint64_t v) {
  const int lane = threadIdx.x & 31;
  if (!(mask >> lane & 1)) std::abort();
  Warp &w = warps[threadIdx.x >> 5];
  std::unique_lock<std::mutex> lock(w.m);
  Meeting &a = w.of[mask];
  a.in[lane] = v;
  if (++a.count == __builtin_popcount(mask)) {
    std::memcpy(a.out, a.in, sizeof(a.in));
    a.count = 0;
    ++a.turn;
    w.cv.notify_all();
  } else {
    const unsigned turn = a.turn;
    w.cv.wait(lock, [&] { return a.turn != turn; });
  }
  thread_local uint64_t mine[32];
  std::memcpy(mine, a.out, sizeof(mine));
  return mine;
}
template <typename T> uint64_t bits(T v) { uint64_t b = 0; std::memcpy(&b, &v, sizeof(v)); return b; }
template <typename T> T unbits(uint64_t b) { T v; std::memcpy(&v, &b, sizeof(v)); return v; }
inline void __syncthreads() { pthread_barrier_wait(&block_barrier); }
inline unsigned __ballot_sync(unsigned mask, bool p) {
  const uint64_t *o = meet(mask, p);
  unsigned r = 0;
  for (int l = 0; l < 32; ++l) if (mask >> l & 1 && o[l]) r |= 1u << l;
  return r;
}
inline unsigned __match_any_sync(unsigned mask, int v) {
  const uint64_t *o = meet(mask, bits(v));
  unsigned r = 0;
  for (int l = 0; l < 32; ++l) if (mask >> l & 1 && o[l] == bits(v)) r |= 1u << l;
  return r;
}
template <typename T> T __shfl_sync(unsigned mask, T v, int lane) {
  const uint64_t *o = meet(mask, bits(v));
  if (!(mask >> lane & 1)) std::abort();
  return unbits<T>(o[lane]);
}
template <typename T> T __shfl_up_sync(unsigned mask, T v, int d) {
  const uint64_t *o = meet(mask, bits(v));
  const int l = (int)(threadIdx.x & 31) - d;
  return l < 0 ? v : unbits<T>(o[l]);
}
template <typename T> T __shfl_xor_sync(unsigned mask, T v, int d) {
  return unbits<T>(meet(mask, bits(v))[(threadIdx.x & 31) ^ d]);
}
inline int atomicAdd(int *p, int v) { return __atomic_fetch_add(p, v, __ATOMIC_RELAXED); }
inline unsigned atomicOr(unsigned *p, unsigned v) { return __atomic_fetch_or(p, v, __ATOMIC_RELAXED); }
inline unsigned atomicExch(unsigned *p, unsigned v) { return __atomic_exchange_n(p, v, __ATOMIC_RELAXED); }
template <typename T> T __ldg(const T *p) { return *p; }
inline int __popc(unsigned v) { return __builtin_popcount(v); }
inline int __ffs(int v) { return __builtin_ffs(v); }
inline double __longlong_as_double(long long v) { return unbits<double>((uint64_t)v); }
inline int __double2int_rn(double v) { return (int)std::nearbyint(v); }
using std::fabs; using std::isfinite; using std::fmin; using std::fmax; using std::floor; using std::sqrt;
inline int min(int a, int b) { return a < b ? a : b; }
inline int max(int a, int b) { return a > b ? a : b; }

template <typename F> void run_block(int nt, F thread) {
  pthread_barrier_init(&block_barrier, nullptr, nt);
  blockDim = {(unsigned)nt, 1, 1};
  for (Warp &w : warps) w.of.clear();
  std::vector<std::thread> ts;
  for (int t = 0; t < nt; ++t)
    ts.emplace_back([=] { threadIdx = {(unsigned)t, 0, 0}; thread(t); });
  for (auto &t : ts) t.join();
  pthread_barrier_destroy(&block_barrier);
}
