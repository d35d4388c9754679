// k_feed.cuh -- what a kernel that writes a residual does for the sweeps that
// follow it (SweepFeed, device helpers).
#pragma once
#include "dfg_common.cuh"
#include "k_solve.h"

namespace dfg {

// element k of a residual into the forward sweep's input (Z: the sweeps' type)
template <typename Z, typename R>
__device__ __forceinline__ void feed_put(const SweepFeed& f, long long k, R r) {
  if (f.in) reinterpret_cast<Z*>(f.in)[f.pos ? f.pos[k] : k] = (Z)r;
}
// the exchange buffers to the sentinel, by all threads of the grid
template <typename Z>
__device__ __forceinline__ void feed_fill(const SweepFeed& f) {
  const long long first = blockIdx.x * (long long)blockDim.x + threadIdx.x, step = (long long)gridDim.x * blockDim.x;
#pragma unroll
  for (int i = 0; i < 2; ++i)
    for (long long k = first; k < f.nfill[i]; k += step) reinterpret_cast<Z*>(f.fill[i])[k] = sentinel_value<Z>();
}

}  // namespace dfg
