// Runs device code of prender_gb300/csrc on the host: one thread per lane of a
// warp, warp intrinsics as exchanges between the lanes' threads.  As CUDA
// defines them, shuffles and votes carry values but order no memory (relaxed
// atomics here, so a thread sanitizer sees a missing fence), and __syncwarp
// orders the memory of all lanes.  All lanes take part in every intrinsic.
#pragma once
#include <cuda_runtime.h>
#include <math.h>
#include <sched.h>
#include <stdint.h>
#include <string.h>

#include <atomic>
#include <thread>
#include <vector>

namespace host {
struct Index {
  unsigned int x, y, z;
};
constexpr int kMaxLanes = 32;
inline int lanes = 1;  // lanes of the warp that runs
inline thread_local int lane = 0;
inline thread_local uint32_t epoch = 0;
// a lane writes slot e % 2 again only after it has seen every lane's e + 1,
// which each writes after it has read all of e
inline std::atomic<uint64_t> slots[2][kMaxLanes];
inline std::atomic<uint32_t> arrived{0}, sense{0};

inline void exchange(uint32_t v, uint32_t out[kMaxLanes]) {
  if (lanes == 1) {
    out[0] = v;
    return;
  }
  const uint32_t e = ++epoch;
  slots[e & 1][lane].store((uint64_t)e << 32 | v, std::memory_order_relaxed);
  for (int l = 0; l < lanes; l++) {
    uint64_t got;
    while ((uint32_t)((got = slots[e & 1][l].load(std::memory_order_relaxed)) >> 32) != e) sched_yield();
    out[l] = (uint32_t)got;
  }
}
template <class F>
void run_warp(int n, F f) {
  lanes = n;
  for (auto& s : slots)
    for (auto& q : s) q.store(0);
  arrived.store(0);
  sense.store(0);
  std::vector<std::thread> t;
  for (int l = 0; l < n; l++)
    t.emplace_back([l, &f] {
      lane = l;
      epoch = 0;
      f(l);
    });
  for (auto& x : t) x.join();
  lanes = 1;
}
}  // namespace host

struct HostThreadIdx {
  struct X {
    operator unsigned int() const { return (unsigned int)host::lane; }
  } x;
};
inline HostThreadIdx threadIdx;
inline constexpr host::Index blockIdx{0, 0, 0}, blockDim{32, 1, 1}, gridDim{1, 1, 1};
#define __launch_bounds__(...)
#define __global__ static

inline unsigned int __ballot_sync(unsigned int, int p) {
  uint32_t v[host::kMaxLanes];
  host::exchange(p ? 1u : 0u, v);
  unsigned int m = 0;
  for (int l = 0; l < host::lanes; l++) m |= v[l] << l;
  return m;
}
inline int __any_sync(unsigned int m, int p) { return __ballot_sync(m, p) != 0; }
inline unsigned int __activemask() { return host::lanes == 32 ? 0xffffffffu : (1u << host::lanes) - 1u; }
template <class T>
T __shfl_sync(unsigned int, T x, int src) {
  uint32_t b[sizeof(T) / 4], v[host::kMaxLanes];
  memcpy(b, &x, sizeof(T));
  for (uint32_t& w : b) {
    host::exchange(w, v);
    w = v[src & 31];
  }
  memcpy(&x, b, sizeof(T));
  return x;
}
template <class T>
T __shfl_up_sync(unsigned int m, T x, int d) {
  return __shfl_sync(m, x, host::lane >= d ? host::lane - d : host::lane);
}
template <class T>
T __shfl_down_sync(unsigned int m, T x, int d) {
  return __shfl_sync(m, x, host::lane + d < host::lanes ? host::lane + d : host::lane);
}
inline void __syncwarp() {
  if (host::lanes == 1) return;
  const uint32_t s = host::sense.load(std::memory_order_relaxed);
  if (host::arrived.fetch_add(1, std::memory_order_acq_rel) + 1 == (uint32_t)host::lanes) {
    host::arrived.store(0, std::memory_order_relaxed);
    host::sense.store(s + 1, std::memory_order_release);
  } else {
    while (host::sense.load(std::memory_order_acquire) == s) sched_yield();
  }
}

inline int __ffs(int v) { return ffs(v); }
inline int __ffsll(long long v) { return ffsll(v); }
inline int __popc(unsigned int v) { return __builtin_popcount(v); }
inline uint32_t __umulhi(uint32_t a, uint32_t b) { return (uint32_t)(((uint64_t)a * b) >> 32); }
inline uint32_t __byte_perm(uint32_t a, uint32_t b, uint32_t s) {
  const uint64_t w = (uint64_t)b << 32 | a;
  uint32_t r = 0;
  for (int k = 0; k < 4; k++) r |= (uint32_t)((w >> (8 * ((s >> (4 * k)) & 7))) & 0xFF) << (8 * k);
  return r;
}
inline float __int_as_float(int v) { float f; memcpy(&f, &v, 4); return f; }
inline float __uint_as_float(uint32_t v) { float f; memcpy(&f, &v, 4); return f; }
inline int __float_as_int(float f) { int v; memcpy(&v, &f, 4); return v; }
inline uint32_t __float_as_uint(float f) { uint32_t v; memcpy(&v, &f, 4); return v; }
inline int __double2hiint(double d) { uint64_t v; memcpy(&v, &d, 8); return (int)(v >> 32); }
inline int __double2loint(double d) { uint64_t v; memcpy(&v, &d, 8); return (int)(uint32_t)v; }
inline float __fmul_rn(float a, float b) { return a * b; }
inline float __fadd_rn(float a, float b) { return a + b; }
inline float __fsub_rn(float a, float b) { return a - b; }
inline float __fdividef(float a, float b) { return a / b; }
inline double __dmul_rn(double a, double b) { return a * b; }
inline double __dadd_rn(double a, double b) { return a + b; }
inline double __dsub_rn(double a, double b) { return a - b; }
inline double __ddiv_rn(double a, double b) { return a / b; }
inline double __dsqrt_rn(double a) { return sqrt(a); }
inline float __double2float_rn(double d) { return (float)d; }
inline float __double2float_ru(double d) {
  const float f = (float)d;
  return (double)f < d ? nextafterf(f, INFINITY) : f;
}
inline float rsqrtf(float x) { return 1.0f / sqrtf(x); }
template <class T>
T __ldg(const T* p) { return *p; }
inline unsigned int atomicOr(unsigned int* p, unsigned int v) { return __atomic_fetch_or(p, v, __ATOMIC_RELAXED); }
inline unsigned int atomicAdd(unsigned int* p, unsigned int v) { return __atomic_fetch_add(p, v, __ATOMIC_RELAXED); }
inline unsigned long long atomicAdd(unsigned long long* p, unsigned long long v) {
  return __atomic_fetch_add(p, v, __ATOMIC_RELAXED);
}
inline int min(int a, int b) { return a < b ? a : b; }
inline int max(int a, int b) { return a > b ? a : b; }
inline unsigned int min(unsigned int a, unsigned int b) { return a < b ? a : b; }
