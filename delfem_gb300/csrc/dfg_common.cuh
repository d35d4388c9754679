// dfg_common.cuh -- shared device helpers for libdfg (sm_103a only).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#ifndef __CUDACC__
#error "dfg_common.cuh is device code"
#endif

namespace dfg {

// Sentinels marking "not yet written" in sweep output buffers.  They are
// negative quiet NaNs with a payload that GPU arithmetic never produces
// (arithmetic NaNs are canonical), so a consumer that reads anything else
// has read the producer's final value.
constexpr uint64_t kSentinel64 = 0xFFF4BADBADBADBADull;
constexpr uint32_t kSentinel32 = 0xFFB4BADBu;

__device__ __forceinline__ bool is_sentinel(double v) {
  return (uint64_t)__double_as_longlong(v) == kSentinel64;
}
__device__ __forceinline__ bool is_sentinel(float v) {
  return __float_as_uint(v) == kSentinel32;
}
template <typename T> __device__ __forceinline__ T sentinel_value();
template <> __device__ __forceinline__ double sentinel_value<double>() {
  return __longlong_as_double((long long)kSentinel64);
}
template <> __device__ __forceinline__ float sentinel_value<float>() {
  return __uint_as_float(kSentinel32);
}

// gpu-scope relaxed accesses (morally strong: a poll sees the producer's store)
__device__ __forceinline__ double ld_relaxed(const double* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return __longlong_as_double((long long)v);
}
__device__ __forceinline__ float ld_relaxed(const float* p) {
  unsigned v;
  asm volatile("ld.relaxed.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return __uint_as_float(v);
}
__device__ __forceinline__ void st_relaxed(double* p, double v) {
  asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"((unsigned long long)__double_as_longlong(v)) : "memory");
}
__device__ __forceinline__ void st_relaxed(float* p, float v) {
  asm volatile("st.relaxed.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(__float_as_uint(v)) : "memory");
}
__device__ __forceinline__ int ld_relaxed_int(const int* p) {
  int v;
  asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Ampere-style asynchronous global->shared copies
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async8(void* smem, const void* gmem) {
  unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async4(void* smem, const void* gmem) {
  unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// What a sweep takes off a row's right-hand side: component p of t[p] - sum over e, q
// of block(e)(p, q) x(e)(q), entry after entry, as the strip and the one-CTA kernel
// evaluate a row.
//
// FOUR (single solves, FP32, 3x3 blocks: 21 products per component in a tetrahedral
// mesh): four sums, entry e in sum e % 4, apart from the right-hand side.  One chain
// from the right-hand side on has 1.9 times the error of the level-scheduled kernel's
// sums over lanes, where these solves would otherwise sweep (elasticity on 56^3 cells,
// sweep against FP64: 1.02e-7, levels 5.4e-8, four sums 5.4e-8).  It costs 1 % on 24^3
// cells (84.2 -> 85.3 us per iteration) and less on 56^3 (130.7 -> 131.0 ms).  Four sums
// of which one starts at the right-hand side are 1.15 times as inexact as the levels,
// two sums 1.07 times, and either half of that cost.  The server's kernels give the
// same bits in one chain.
constexpr bool sweep_four(bool fp32, int b) { return fp32 && b == 3; }
template <typename T, int B, int P, bool FOUR>
struct RowSum {
  static constexpr int N = FOUR ? 4 : 1;
  T s[N][P];
  __device__ __forceinline__ void start(const T (&t)[P]) {
#pragma unroll
    for (int k = 0; k < N; ++k)
#pragma unroll
      for (int p = 0; p < P; ++p) s[k][p] = N == 1 ? t[p] : T(0);
  }
  __device__ __forceinline__ void add(int e, int p, T a, T x) {
    if (N == 1) s[0][p] -= a * x;
    else s[e % N][p] += a * x;
  }
  __device__ __forceinline__ T row(int p, T t) const {
    if constexpr (N == 1) return s[0][p];
    else return t - ((s[0][p] + s[1][p]) + (s[2][p] + s[3][p]));
  }
};

// Programmatic dependent launch (kernels launched with
// cudaLaunchAttributeProgrammaticStreamSerialization): wait until the
// previous kernel in the stream has finished and its writes are visible,
// then let the next kernel launch so that its start overlaps this one.  In a
// kernel launched in plain stream order both are no-ops.
__device__ __forceinline__ void pdl_enter() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// error word shared by all kernels of a context (0 = ok)
enum : int { kErrNone = 0, kErrTimeout = 1, kErrBadIndex = 2 };

// Device-side wait budget: a wait gives up after this many SM clock cycles
// (about two seconds at 2 GHz), records kErrTimeout with where it happened,
// and every other waiter of the launch leaves as soon as it sees the record.
constexpr long long kWaitCycles = 4000000000ll;
// Bound on waiting for a copy already in flight before a failing CTA leaves.
constexpr long long kDrainCycles = 2000000ll;
// wait sites recorded with a timeout (error word [1])
enum : int { kSiteEmpty = 1, kSiteRecLoad = 2, kSitePoll = 3, kSiteRecCompute = 4, kSiteFull = 5, kSiteRange = 6 };

}  // namespace dfg
