// k_iter.cu -- what a PCG iteration does between two preconditioner
// applications, in one launch: r.z and beta, the direction update, A p with
// p.Ap and alpha, the r/x update with r.r and the stop test
// (LsSol::Solve_PCG, src/ls/solver_ls_iter.cpp:100-172).
//
// As four launches this took about 30 us per iteration on a small system, most
// of it launch latency, reductions and the last block's tail: a warp-wide FP64
// addition takes its scheduler 64 cycles on GB300, so a 256-thread block sum
// alone costs over 1,000.  Here one cooperative grid stays resident and meets
// at barriers (of the grid 1.1 us each).  A reduction leaves its partials in memory,
// and after the barrier every block adds them itself, in the same order, so no
// block waits for another to publish a total.
//
// p.Ap of blocks of 256 threads comes from the product's own warps: a slice's
// share is one warp's tree, a virtual block's the tree over its 16 slices, which
// every block takes after the barrier (a barrier and a pass less: 2D elasticity on
// 200x100 cells 242.9 -> 240.2 us per iteration, 24^3 208 -> 205.6).
//
// The sums are those of the separate launches (k_reduce.cuh), bit for bit:
// kRedGrid virtual blocks of kRedTpb elements, or of kSpmvTpb rows for p.Ap,
// each summed by warps (xor tree) and then over its warps, and the partials in
// index order.  An FP32-factor solve of 1,000 iterations stops at a solution
// whose tenth digit depends on such roundings.  The product itself is spread
// over the SMs where a virtual block's 512 rows would crowd a few of them: rows
// go to warps slice by slice, one warp per scheduler on as many SMs as there
// are (a row of 3x3 blocks of a tetrahedral mesh is 135 FP64 FMAs; on 31 SMs the
// product of 15,625 rows took 22 us, spread 7.5); with blocks of 1024 threads p.Ap
// is summed after another barrier.
//
// Measured on GB300, a whole PCG iteration (four launches -> one): Poisson
// 24x24 54.7 -> 51.1 us, 128x128 148 -> 137, 301x257 FP32 everything 122 -> 114,
// cantilever 200x100 262 -> 251, 401x199 FP32 factor 153 -> 142, elasticity 24^3
// 234 -> 216, 56^3 FP32 factor 327 -> 300 (some 3 % of it the sweeps'); now, with
// what is said here and shorter sweeps, 39, 127, 107, 212, 132, 154 and 275.
//
// Waits are bounded; one that gives up records kErrTimeout.
#include <algorithm>
#include <cmath>

#include "dfg_common.cuh"
#include "k_feed.cuh"
#include "k_mbar.cuh"
#include "k_rowmv.cuh"
#include "k_solve.h"

namespace dfg {

namespace {

// xor tree over the warp; n: lanes from n on hold zeros, so that the levels that
// would only add them are left out
__device__ __forceinline__ double warp_total(double v, int n = 32) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    if (o < n) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Sums over virtual blocks of NW warps by the warps of this block, NW of them at
// a time: v is the thread's value of virtual block vb (of nvb; nothing where
// there is none).  The total goes to part[vb].
template <int NW>
__device__ __forceinline__ void block_part(double v, int vb, int nvb, double* ws, double* part) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __syncthreads();  // ws of the sum before has been read
  v = warp_total(v);
  if (lane == 0) ws[warp] = v;
  __syncthreads();
  if (warp % NW == 0 && vb < nvb) {
    double t = lane < NW ? ws[warp + lane] : 0.0;
#pragma unroll
    for (int o = NW / 2; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (lane == 0) part[vb] = t;
  }
}

// The sum of all virtual blocks' partials as NT threads take it (thread i adds
// i and i + NT, then a block of NT/32 warps as above), and what f makes of it, in
// every thread: f is one thread's (a division by 32 warps takes the schedulers
// 4 us).  At least NT/2 threads take part; those of NT = 512 hold two values.
template <int NT, typename P, typename F>
__device__ __forceinline__ double2 with_total(int nvb, double* ws, P&& part, F&& f) {
  __shared__ double2 both;
  constexpr int NW = NT / 32;
  static_assert(kRedGrid <= 512 && kRedGrid > 256, "one value per thread of 512, up to two of 256");
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, per = blockDim.x < NT ? 2 : 1;
  auto value = [&](int i) {
    double t = i < nvb ? part(i) : 0.0;
    if (NT == 256 && i + NT < nvb) t += part(i + NT);
    return t;
  };
  __syncthreads();
  for (int h = 0; h < per; ++h) {
    const int w = warp + h * (NT / 2 / 32);
    if (threadIdx.x < NT / per && w * 32 < nvb) {  // (whole warps; the others' sums are zero)
      const double t = warp_total(value(w * 32 + lane), nvb);
      if (lane == 0) ws[w] = t;
    } else if (threadIdx.x < NT / per && lane == 0) {
      ws[w] = 0.0;
    }
  }
  __syncthreads();
  if (warp == 0) {
    double t = lane < NW ? ws[lane] : 0.0;
#pragma unroll
    for (int o = NW / 2; o > 0; o >>= 1)
      if (o * 32 < nvb) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (lane == 0) both = make_double2(t, f(t));
  }
  __syncthreads();
  return both;
}

__device__ __forceinline__ auto in_memory(const double* part) {
  return [part](int i) { return ld_relaxed(part + i); };
}

__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// The blocks' barrier: of one cluster, or of the whole cooperative grid.
template <bool CLUSTER>
struct GridWalk {
  unsigned* bar;   // arrivals; back to zero when the launch ends
  int* err;
  unsigned target = 0;
  bool ok = true;

  // Every thread of every block; false once a wait has given up.
  __device__ bool sync() {
    if constexpr (CLUSTER) {
      cluster_sync();
      return true;
    }
    __shared__ int s_ok;
    target += gridDim.x;
    __syncthreads();
    if (threadIdx.x == 0) {
      __threadfence();
      atomicAdd(bar, 1u);
      int good = 1;
      const long long t0 = clock64();
      for (unsigned n = 1;; ++n) {
        unsigned v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(bar) : "memory");
        if (v >= target) break;
        if ((n & 63) == 0) {
          if (ld_relaxed_int(err) != 0) { good = 0; break; }
          if (clock64() - t0 > kWaitCycles) {
            record_fail(err, kErrTimeout, kSiteRange, -1, (int)target);
            good = 0;
            break;
          }
        }
      }
      s_ok = good;
    }
    __syncthreads();
    ok = s_ok != 0;
    return ok;
  }
  // The launch's last meeting, without a wait: true in the block that comes
  // last, which also sets the counter back (in a cluster: in block 0).
  __device__ bool last() {
    if constexpr (CLUSTER) {
      cluster_sync();
      return blockIdx.x == 0;
    }
    __shared__ int s_last;
    target += gridDim.x;
    __syncthreads();
    if (threadIdx.x == 0) {
      __threadfence();
      s_last = atomicAdd(bar, 1u) + 1u == target;
      if (s_last) {
        *bar = 0u;
        __threadfence();
      }
    }
    __syncthreads();
    return s_last != 0;
  }
};

// Elements of the vectors: virtual block vb holds the elements vb*kRedTpb + t +
// j*kRedGrid*kRedTpb.  Calls f(k) for the thread's elements, which returns what
// they add to its sum; the sums go to part[0 .. nvb).  TPB / kRedTpb virtual
// blocks at a time (of 1024 threads, 512 then rest).
template <int TPB, typename F>
__device__ __forceinline__ void vector_pass(long long m, int nvb, double* ws, double* part, F&& f) {
  constexpr int V = TPB / kRedTpb >= 2 ? 2 : 1, NW = kRedTpb / 32;
  const int half = threadIdx.x / kRedTpb, t = threadIdx.x % kRedTpb;
  for (int v0 = blockIdx.x; v0 < nvb; v0 += gridDim.x * V) {
    const int vb = half < V ? v0 + half * (int)gridDim.x : nvb;
    double sum = 0.0;
    if (vb < nvb)
      for (long long k = (long long)vb * kRedTpb + t; k < m; k += (long long)kRedGrid * kRedTpb) f(k, sum);
    block_part<NW>(sum, vb, nvb, ws, part);
  }
}

// p.q over virtual blocks of kSpmvTpb rows, two at a time (1024 threads)
template <typename T, int B>
__device__ __forceinline__ void rows_pass(int n, const T* p, const T* q, int nvb, double* ws, double* part) {
  constexpr int kAll = kRedGrid * kSpmvTpb, NW = kSpmvTpb / 32;
  auto rows = [&](int i, double& sum) {
    for (; i < n; i += kAll)
#pragma unroll
      for (int d = 0; d < B; ++d) sum += (double)p[(size_t)i * B + d] * (double)q[(size_t)i * B + d];
  };
  const int half = threadIdx.x / kSpmvTpb, t = threadIdx.x % kSpmvTpb;
  for (int v0 = blockIdx.x; v0 < nvb; v0 += gridDim.x * 2) {
    const int vb = v0 + half * (int)gridDim.x;
    double sum = 0.0;
    if (vb < nvb) rows(vb * kSpmvTpb + t, sum);
    block_part<NW>(sum, vb, nvb, ws, part);
  }
}

// q = A p, slices of 32 rows over the warps of all blocks; part != nullptr: the
// warps' shares of p.q, one per slice
template <typename T, int B>
__device__ __forceinline__ void spread_product(const MatView& A, const T* p, T* q, double* part) {
  const T* sval = reinterpret_cast<const T*>(A.sval);
  const int lane = threadIdx.x & 31, nw = blockDim.x >> 5, nsl = (A.n + 31) >> 5;
  for (int s = blockIdx.x + gridDim.x * (threadIdx.x >> 5); s < nsl; s += gridDim.x * nw) {
    const int i = s * 32 + lane;
    double sum = 0.0;
    if (i < A.n) {
      T y[B];
      sell_row_mv<T, B>(i, A.sptr, A.swidth, A.scol, sval, p, y);
#pragma unroll
      for (int d = 0; d < B; ++d) {
        q[(size_t)i * B + d] = y[d];
        sum += (double)p[(size_t)i * B + d] * (double)y[d];
      }
    }
    if (part) {
      sum = warp_total(sum);
      if (lane == 0) part[s] = sum;
    }
  }
}

// p.q from the slices' shares, and what f makes of it: a virtual block of
// kSpmvTpb rows is 16 slices, its sum their xor tree.  For blocks of 256 threads.
template <typename F>
__device__ __forceinline__ double2 with_slices(int n, int nvr, double* ws, const double* part, F&& f) {
  constexpr int kMaxVb = kIterSlices / 16;
  __shared__ double vbs[kMaxVb];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nsl = (n + 31) >> 5;
  double t[(kMaxVb + 15) / 16];
#pragma unroll
  for (int k = 0; k < (kMaxVb + 15) / 16; ++k) {
    const int sl = k * 256 + (int)threadIdx.x;
    t[k] = sl < nsl ? ld_relaxed(part + sl) : 0.0;
  }
#pragma unroll
  for (int k = 0; k < (kMaxVb + 15) / 16; ++k) {
    const int vb = k * 16 + warp * 2 + (lane >> 4);
    if (k * 16 + warp * 2 < nvr) {
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) t[k] += __shfl_xor_sync(0xffffffffu, t[k], o);
      if (lane % 16 == 0 && vb < kMaxVb) vbs[vb] = t[k];
    }
  }
  return with_total<kSpmvTpb>(nvr, ws, [&](int i) { return vbs[i]; }, f);
}

__device__ __forceinline__ int virtual_blocks(long long n, int per) {
  return (int)min((n + per - 1) / per, (long long)kRedGrid);
}

}  // namespace

// FP64 vectors; Z: the preconditioned residual's type.  first: the direction
// and r.z are set (the first iteration).
template <typename Z, int B, int TPB, bool CLUSTER>
__global__ void __launch_bounds__(TPB, 1) k_pcg_iter(MatView A, PcgVecs v, PcgState* st, IterRed red, int* tickets,
                                                  int first) {
  __shared__ double ws[32];
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    if (!v.feed.early) tickets[0] = 0;
    tickets[1] = 0;
  }
  const int failed = ld_relaxed_int(red.err);
  if (st->done) return;
  if (failed) {
    if (blockIdx.x == 0 && threadIdx.x == 0) st->done = kDoneError;
    return;
  }
  GridWalk<CLUSTER> g{red.bar, red.err};
  double *part_rz = red.part, *part_pq = red.part + kRedGrid, *part_rr = red.part + 2 * kRedGrid;
  const int nvb = virtual_blocks(v.m, kRedTpb), nvr = virtual_blocks(A.n, kSpmvTpb);
  const Z* z = reinterpret_cast<const Z*>(v.z);
  double rz = st->rz;
  if (!first) {
    vector_pass<TPB>(v.m, nvb, ws, part_rz, [&](long long k, double& s) { s += v.r[k] * (double)z[k]; });
    if (!g.sync()) return;
    const double2 tb = with_total<kRedTpb>(nvb, ws, in_memory(part_rz), [&](double t) { return t / rz; });
    const double beta = tb.y;
    rz = tb.x;
    // p := beta p; p := p + 1.0 z (SCAL + AXPY)
    const long long step = (long long)gridDim.x * TPB;
    for (long long k = blockIdx.x * (long long)TPB + threadIdx.x; k < v.m; k += step)
      v.p[k] = __dadd_rn(__dmul_rn(v.p[k], beta), (double)z[k]);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      st->beta = beta;
      st->rz = rz;
      st->it += 1;
    }
    if (!g.sync()) return;
  }
  double2 pa;  // p.q, alpha
  if constexpr (TPB == 256) {
    spread_product<double, B>(A, v.p, v.q, red.slices);
    if (!g.sync()) return;
    pa = with_slices(A.n, nvr, ws, red.slices, [&](double t) { return rz / t; });
  } else {
    spread_product<double, B>(A, v.p, v.q, nullptr);
    if (!g.sync()) return;
    rows_pass<double, B>(A.n, v.p, v.q, nvr, ws, part_pq);
    if (!g.sync()) return;
    pa = with_total<kSpmvTpb>(nvr, ws, in_memory(part_pq), [&](double t) { return rz / t; });
  }
  const double alpha = pa.y;
  // r := r - alpha q; x := x + alpha p (AXPY, no-op for alpha == 0)
  vector_pass<TPB>(v.m, nvb, ws, part_rr, [&](long long k, double& s) {
    double r = v.r[k];
    if (alpha != 0.0) {
      r = __dadd_rn(r, __dmul_rn(-alpha, v.q[k]));
      v.r[k] = r;
      v.x[k] = __dadd_rn(v.x[k], __dmul_rn(alpha, v.p[k]));
    }
    s += r * r;
    feed_put<Z>(v.feed, k, r);
  });
  feed_fill<Z>(v.feed);
  if (!g.last()) return;
  const double rr = with_total<kRedTpb>(nvb, ws, in_memory(part_rr), [](double t) { return t; }).x;
  if (threadIdx.x == 0) {
    st->pap = pa.x;
    st->alpha = alpha;
    st->rr = rr;
    const double ratio = rr * st->inv_rr0;
    if (ratio < st->tol2) {
      st->done = 1;
      st->conv = sqrt(ratio);
      st->iter_out = st->it;
    } else if (st->it + 1 >= st->maxit) {
      st->done = 2;
      st->conv = sqrt(ratio);
      st->iter_out = st->maxit;
    } else if (!(ratio == ratio)) {
      st->done = 3;  // NaN
      st->conv = ratio;
      st->iter_out = st->it;
    }
  }
}

// the FP32-everything form: FP32 vectors and products, FP64 sums and correction
template <int B, int TPB, bool CLUSTER>
__global__ void __launch_bounds__(TPB, 1) k_mix_iter(MatView A, MixVecs v, PcgState* st, IterRed red, int* tickets,
                                                  int first) {
  __shared__ double ws[32];
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    if (!v.feed.early) tickets[0] = 0;
    tickets[1] = 0;
  }
  const int failed = ld_relaxed_int(red.err);
  if (st->done) return;
  if (failed) {
    if (blockIdx.x == 0 && threadIdx.x == 0) st->done = kDoneError;
    return;
  }
  GridWalk<CLUSTER> g{red.bar, red.err};
  double *part_rz = red.part, *part_pq = red.part + kRedGrid, *part_rr = red.part + 2 * kRedGrid;
  const int nvb = virtual_blocks(v.m, kRedTpb), nvr = virtual_blocks(A.n, kSpmvTpb);
  double rz = st->rz;
  if (!first) {
    vector_pass<TPB>(v.m, nvb, ws, part_rz, [&](long long k, double& s) { s += (double)v.r[k] * (double)v.z[k]; });
    if (!g.sync()) return;
    const double2 tb = with_total<kRedTpb>(nvb, ws, in_memory(part_rz), [&](double t) { return t / rz; });
    rz = tb.x;
    const float beta = (float)tb.y;
    const long long step = (long long)gridDim.x * TPB;
    for (long long k = blockIdx.x * (long long)TPB + threadIdx.x; k < v.m; k += step) v.p[k] = v.z[k] + beta * v.p[k];
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      st->beta = tb.y;
      st->rz = rz;
      st->it += 1;
    }
    if (!g.sync()) return;
  }
  double2 pa;  // p.q, alpha
  if constexpr (TPB == 256) {
    spread_product<float, B>(A, v.p, v.q, red.slices);
    if (!g.sync()) return;
    pa = with_slices(A.n, nvr, ws, red.slices, [&](double t) { return rz / t; });
  } else {
    spread_product<float, B>(A, v.p, v.q, nullptr);
    if (!g.sync()) return;
    rows_pass<float, B>(A.n, v.p, v.q, nvr, ws, part_pq);
    if (!g.sync()) return;
    pa = with_total<kSpmvTpb>(nvr, ws, in_memory(part_pq), [&](double t) { return rz / t; });
  }
  const double alpha = pa.y;
  const float alpha32 = (float)alpha;
  vector_pass<TPB>(v.m, nvb, ws, part_rr, [&](long long k, double& s) {
    float r = v.r[k];
    if (alpha != 0.0) {
      r = r - alpha32 * v.q[k];
      v.r[k] = r;
      v.d[k] = v.d[k] + alpha * (double)v.p[k];
    }
    s += (double)r * (double)r;
    feed_put<float>(v.feed, k, r);
  });
  feed_fill<float>(v.feed);
  if (!g.last()) return;
  const double rr = with_total<kRedTpb>(nvb, ws, in_memory(part_rr), [](double t) { return t; }).x;
  if (threadIdx.x == 0) {
    st->pap = pa.x;
    st->alpha = alpha;
    st->rr = rr;
    if (!(rr == rr)) {
      st->done = 3;
    } else if (rr < st->tolb2) {
      st->done = 5;
    } else if (rr < st->delta2 * st->rr_ref) {
      st->done = 4;
    } else if (st->it + 1 >= st->maxit) {
      st->done = 2;
    }
    st->iter_out = st->it + 1;
  }
}

// ------------------------------------------------------------------ launchers

// One block per SM: 1024 threads where every warp of 256 would have more than a
// slice, else 256, on as many SMs as four slices (one per scheduler) each give
// work to.  Small systems run in one cluster of 16 blocks: its barrier takes
// 0.2 us instead of 1.1, which outweighs the SMs not used up to some 6,000
// unknowns (whole iterations, grid / cluster: Poisson on 24x24 cells 42.9 / 40.9
// us, 63x63 69.7 / 66.9, 88x88 90.9 / 93.7; elasticity on 11^3 cells 107 / 105, 14^3
// 130 / 132; clusters of 8: 63x63 71.5).
struct IterShape {
  int grid, tpb;
  bool cluster;
};
constexpr int kIterCluster = 16, kIterClusterUnknowns = 6144;
static IterShape iter_shape(int n, int b, int nsm) {
  if (n > std::min(nsm * kSpmvTpb / 2, kIterSlices * 32)) return {nsm, 1024, false};
  const int g = std::max(1, std::min((n + 127) / 128, nsm));
  if (n * b <= kIterClusterUnknowns) return {std::min(g, kIterCluster), 256, true};
  return {g, 256, false};
}

template <typename... KArgs>
static cudaError_t launch_iter(void (*k)(KArgs...), const IterShape& sh, cudaStream_t s, KArgs... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(sh.grid);
  cfg.blockDim = dim3(sh.tpb);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  if (sh.cluster) {
    // more than 8 blocks in a cluster
    const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return e;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = sh.grid;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  } else {
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
  }
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k, args...);
}

cudaError_t pcg_iter(const MatView& A, const PcgVecs& v, PcgState* st, IterRed red, int* tickets, bool fp32z,
                     bool first, int nsm, cudaStream_t s) {
  const IterShape sh = iter_shape(A.n, A.b, nsm);
#define DFG_ITER(Z, B)                                                                                     \
  return sh.cluster      ? launch_iter(k_pcg_iter<Z, B, 256, true>, sh, s, A, v, st, red, tickets, (int)first)  \
         : sh.tpb == 256 ? launch_iter(k_pcg_iter<Z, B, 256, false>, sh, s, A, v, st, red, tickets, (int)first) \
                         : launch_iter(k_pcg_iter<Z, B, 1024, false>, sh, s, A, v, st, red, tickets, (int)first)
  switch (A.b) {
    case 1: if (fp32z) { DFG_ITER(float, 1); } else { DFG_ITER(double, 1); }
    case 2: if (fp32z) { DFG_ITER(float, 2); } else { DFG_ITER(double, 2); }
    case 3: if (fp32z) { DFG_ITER(float, 3); } else { DFG_ITER(double, 3); }
    default: return cudaErrorInvalidValue;
  }
#undef DFG_ITER
}

cudaError_t mix_iter(const MatView& A, const MixVecs& v, PcgState* st, IterRed red, int* tickets, bool first, int nsm,
                     cudaStream_t s) {
  const IterShape sh = iter_shape(A.n, A.b, nsm);
#define DFG_ITER(B)                                                                                     \
  return sh.cluster      ? launch_iter(k_mix_iter<B, 256, true>, sh, s, A, v, st, red, tickets, (int)first)  \
         : sh.tpb == 256 ? launch_iter(k_mix_iter<B, 256, false>, sh, s, A, v, st, red, tickets, (int)first) \
                         : launch_iter(k_mix_iter<B, 1024, false>, sh, s, A, v, st, red, tickets, (int)first)
  switch (A.b) {
    case 1: DFG_ITER(1);
    case 2: DFG_ITER(2);
    case 3: DFG_ITER(3);
    default: return cudaErrorInvalidValue;
  }
#undef DFG_ITER
}

}  // namespace dfg
