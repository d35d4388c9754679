// k_ilu.cu -- numeric block ILU factorisation, level-scheduled.
//
// Restates CMatDiaFrac_BlkCrs::DoILUDecomp (src/matvec/matdiafrac_blkcrs.cpp:
// 774-1107) for 1x1, 2x2 and 3x3 blocks, on the factor's own pattern (A's
// for ILU(0), with fill-in for ILU(k)).  Row i only reads rows k < i that
// are finished (they sit in earlier levels of the forward dependency DAG)
// and only writes its own row, so all rows of one level run in parallel, one
// thread each.  This file is compiled with -fmad=false and every expression
// keeps the reference's operand order, so the factor is bit-identical to the
// reference's (the division 1.0/det is IEEE-rounded on both sides).
#include <algorithm>

#include "dfg_common.cuh"
#include "k_ilu.h"
#include "k_mbar.cuh"

namespace dfg {

// position of column j inside row i (CRS slot) or -1; the reference uses a
// scatter array row2crs_f for the same lookup
__device__ __forceinline__ int find_slot(const int* colind, int c0, int c1, int j) {
  int lo = c0, hi = c1;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (colind[mid] < j) lo = mid + 1; else hi = mid;
  }
  return (lo < c1 && colind[lo] == j) ? lo : -1;
}

template <int B>
__global__ void k_ilu_level(const int* __restrict__ rows, int cnt, const int* __restrict__ rowptr,
                            const int* __restrict__ colind, const int* __restrict__ diaind,
                            double* fdiag, double* foffd, int* nsing) {
  constexpr int BS = B * B;
  pdl_enter();  // the previous level (a programmatic dependency) is complete
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= cnt) return;
  const int i = rows[t];
  const int r0 = rowptr[i], r1 = rowptr[i + 1], di = diaind[i];
  double* pii = fdiag + (size_t)i * BS;
  for (int ik = r0; ik < di; ++ik) {
    const int k = colind[ik];
    const double* pik = foffd + (size_t)ik * BS;
    double lik[BS];
#pragma unroll
    for (int m = 0; m < BS; ++m) lik[m] = pik[m];  // A_ik already holds the updates of all k' < k
    for (int kj = diaind[k]; kj < rowptr[k + 1]; ++kj) {
      const int j = colind[kj];
      const double* pkj = foffd + (size_t)kj * BS;
      double* pij;
      if (j != i) {
        const int ij = find_slot(colind, r0, r1, j);
        if (ij < 0) continue;
        pij = foffd + (size_t)ij * BS;
      } else {
        pij = pii;
      }
      if constexpr (B == 1) {
        pij[0] -= lik[0] * pkj[0];
      } else if constexpr (B == 2) {
        pij[0] -= lik[0] * pkj[0] + lik[1] * pkj[2];
        pij[1] -= lik[0] * pkj[1] + lik[1] * pkj[3];
        pij[2] -= lik[2] * pkj[0] + lik[3] * pkj[2];
        pij[3] -= lik[2] * pkj[1] + lik[3] * pkj[3];
      } else {
#pragma unroll
        for (int r = 0; r < 3; ++r) {
          pij[r * 3 + 0] -= lik[r * 3 + 0] * pkj[0] + lik[r * 3 + 1] * pkj[3] + lik[r * 3 + 2] * pkj[6];
          pij[r * 3 + 1] -= lik[r * 3 + 0] * pkj[1] + lik[r * 3 + 1] * pkj[4] + lik[r * 3 + 2] * pkj[7];
          pij[r * 3 + 2] -= lik[r * 3 + 0] * pkj[2] + lik[r * 3 + 1] * pkj[5] + lik[r * 3 + 2] * pkj[8];
        }
      }
    }
  }
  // pivot inverse (matdiafrac_blkcrs.cpp:885-895 / 933-951 / 998-1013)
  bool sing = false;
  if constexpr (B == 1) {
    const double v = pii[0];
    if (fabs(v) > 1.0e-30) pii[0] = 1.0 / v; else sing = true;
  } else if constexpr (B == 2) {
    const double det = pii[0] * pii[3] - pii[1] * pii[2];
    if (fabs(det) > 1.0e-30) {
      const double inv_det = 1.0 / det;
      const double t0 = pii[0];
      pii[0] = inv_det * pii[3];
      pii[1] = -inv_det * pii[1];
      pii[2] = -inv_det * pii[2];
      pii[3] = inv_det * t0;
    } else {
      sing = true;
    }
  } else {
    const double* a = pii;
    const double det = a[0] * a[4] * a[8] + a[3] * a[7] * a[2] + a[6] * a[1] * a[5]
                     - a[0] * a[7] * a[5] - a[6] * a[4] * a[2] - a[3] * a[1] * a[8];
    if (fabs(det) > 1.0e-30) {
      const double inv_det = 1.0 / det;
      double t[9];
#pragma unroll
      for (int m = 0; m < 9; ++m) t[m] = pii[m];
      pii[0] = inv_det * (t[4] * t[8] - t[5] * t[7]);
      pii[1] = inv_det * (t[2] * t[7] - t[1] * t[8]);
      pii[2] = inv_det * (t[1] * t[5] - t[2] * t[4]);
      pii[3] = inv_det * (t[5] * t[6] - t[3] * t[8]);
      pii[4] = inv_det * (t[0] * t[8] - t[2] * t[6]);
      pii[5] = inv_det * (t[2] * t[3] - t[0] * t[5]);
      pii[6] = inv_det * (t[3] * t[7] - t[4] * t[6]);
      pii[7] = inv_det * (t[1] * t[6] - t[0] * t[7]);
      pii[8] = inv_det * (t[0] * t[4] - t[1] * t[3]);
    } else {
      sing = true;
    }
  }
  if (sing) atomicAdd(nsing, 1);
  // U'_ij = D_i^-1 A_ij, j > i
  double d[BS];
#pragma unroll
  for (int m = 0; m < BS; ++m) d[m] = pii[m];
  for (int ij = di; ij < r1; ++ij) {
    double* p = foffd + (size_t)ij * BS;
    if constexpr (B == 1) {
      p[0] = p[0] * d[0];
    } else if constexpr (B == 2) {
      const double t0 = p[0], t1 = p[1], t2 = p[2], t3 = p[3];
      p[0] = d[0] * t0 + d[1] * t2;
      p[1] = d[0] * t1 + d[1] * t3;
      p[2] = d[2] * t0 + d[3] * t2;
      p[3] = d[2] * t1 + d[3] * t3;
    } else {
      double t[9];
#pragma unroll
      for (int m = 0; m < 9; ++m) t[m] = p[m];
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        p[r * 3 + 0] = d[r * 3 + 0] * t[0] + d[r * 3 + 1] * t[3] + d[r * 3 + 2] * t[6];
        p[r * 3 + 1] = d[r * 3 + 0] * t[1] + d[r * 3 + 1] * t[4] + d[r * 3 + 2] * t[7];
        p[r * 3 + 2] = d[r * 3 + 0] * t[2] + d[r * 3 + 1] * t[5] + d[r * 3 + 2] * t[8];
      }
    }
  }
}

// ----------------------------------------------------------- one launch, warps
//
// The same factorisation with the rows' arithmetic spread over a warp and one
// launch for all levels.  A thread per row (above) is bound by its chain of
// FP64 operations, 64 cycles each on GB300 for a warp whatever its active
// lanes: about 1,700 for a 3x3 row of a tetrahedral mesh, 130 us per level.
// Here G lanes work on a row: lane (j, c) holds component c of the block that
// one upper entry j of row k updates, so the updates by a row k take one
// round of 2b operations instead of one per block and component, the pivot's
// products are taken by one lane each, and every operand is in shared memory.
// Each component is computed by the reference's operations in its order.
//
// Units of 32/G rows of one level are claimed in level order through a ticket.
// A warp loads what earlier rows do not change (its rows' columns, A's values,
// the places that each update goes to) first, then polls the upper blocks of
// its lower rows: the factor's off-diagonal storage was filled with the sweeps'
// NaN sentinel, each value is written once, so whatever else is read is final
// and no fence or counter stands between two levels.  A unit only waits for
// units claimed earlier, by warps that are running, so nothing depends on how
// many CTAs are resident; every wait is bounded.
//
// Measured on GB300, SetValue as a whole, a thread per row and a launch per
// level -> this kernel: 1x1 blocks 128x128 cells 1.92 -> 0.48 ms, 300x300 4.65 ->
// 1.08; 2x2 200x100 4.77 -> 0.71, 401x199 9.46 -> 1.42, ILU(1) 161x83 7.88 ->
// 0.83; 3x3 24^3 9.7 -> 0.70, 56^3 25.6 -> 2.7 ms.  (Counters of finished units
// with release and acquire instead of the sentinel: 1.27, 3.36, 1.56, 3.34,
// 1.48, 1.09 and 8.3 ms.)  What bounds it now: the FP64 chain of a row per
// level in narrow levels (1.9 us per level, 1x1), the FP64 pipes in wide ones.
template <int B>
struct IluLanes;
template <> struct IluLanes<1> { static constexpr int G = 8, J = 8; };
template <> struct IluLanes<2> { static constexpr int G = 16, J = 4; };
template <> struct IluLanes<3> { static constexpr int G = 32, J = 3; };

static size_t ilu_group_bytes(int b, int maxrow, int maxlow, int maxu) {
  const size_t bs = (size_t)b * b;
  return ((size_t)(maxrow + 1 + maxu) * bs * 8 + (size_t)(maxrow + 2 * maxu + 2 * (maxlow + 1)) * 4 + 15) / 16 * 16;
}
constexpr int kIluWarps = 4;  // per CTA, one per scheduler

template <int B>
__global__ void __launch_bounds__(kIluWarps * 32, 2) k_ilu(IluArgs a, size_t group_bytes) {
  constexpr int BS = B * B, G = IluLanes<B>::G, J = IluLanes<B>::J;
  extern __shared__ __align__(16) unsigned char smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane / G, sub = lane - g * G;
  const int jl = sub / BS, comp = sub - jl * BS, r = comp / B, c = comp - r * B;
  unsigned char* base = smem + (size_t)(warp * (32 / G) + g) * group_bytes;
  double* rowv = reinterpret_cast<double*>(base);   // off-diagonal slots, then the diagonal at slot maxrow
  double* uv = rowv + (a.maxrow + 1) * BS;          // upper entries of the lower rows
  int* col = reinterpret_cast<int*>(uv + a.maxu * BS);
  int* usrc = col + a.maxrow;                       // their CRS slots
  int* utgt = usrc + a.maxu;                        // the slots they update in this row, -1: none
  int* ubeg = utgt + a.maxu;                        // first upper entry of each lower row
  int* ud = ubeg + a.maxlow + 1;                    // its CRS slot
  int* ticket = a.sync;
  int* err = a.sync + 4;
  int u = 0;
  if (lane == 0) u = atomicAdd(ticket, 1);
  for (;;) {
    u = __shfl_sync(0xffffffffu, u, 0);
    if (u >= a.nunits) break;
    const int2 un = a.units[u];
    int next = 0;
    if (lane == 0) next = atomicAdd(ticket, 1);  // (claims are worked off in order)
    const bool on = g < un.y;
    const int i = on ? a.rows[un.x + g] : 0;
    const int r0 = on ? a.rowptr[i] : 0, nrow = on ? a.rowptr[i + 1] - r0 : 0, nlow = on ? a.diaind[i] - r0 : 0;
    // what earlier rows do not change
    for (int q = sub; q < nrow; q += G) col[q] = a.colind[r0 + q];
    for (int q = sub; q < nrow * BS; q += G) rowv[q] = a.aoffd[(size_t)r0 * BS + q];
    if (on)
      for (int q = sub; q < BS; q += G) rowv[a.maxrow * BS + q] = a.adiag[(size_t)i * BS + q];
    __syncwarp();
    for (int q = sub; q < nlow; q += G) {
      const int k = col[q], d0 = a.diaind[k];
      ud[q] = d0;
      ubeg[q + 1] = a.rowptr[k + 1] - d0;
    }
    if (sub == 0) ubeg[0] = 0;
    __syncwarp();
    if (sub == 0)
      for (int q = 0; q < nlow; ++q) ubeg[q + 1] += ubeg[q];
    __syncwarp();
    const int nu = on ? ubeg[nlow] : 0;
    for (int e = sub; e < nu; e += G) {
      int kk = 0;
      while (ubeg[kk + 1] <= e) ++kk;
      const int src = ud[kk] + e - ubeg[kk], j = a.colind[src];
      usrc[e] = src;
      int lo = 0, hi = nrow;
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (col[mid] < j) lo = mid + 1; else hi = mid;
      }
      utgt[e] = j == i ? a.maxrow : (lo < nrow && col[lo] == j) ? lo : -1;
    }
    __syncwarp();
    // the lower rows' upper blocks, as they are finished
    bool ok = true;
    {
      constexpr int U = 4;
      const int tot = nu * BS;
      long long t0 = 0;
      for (int q = sub; q < tot && ok; q += U * G) {
        double v[U];
        const double* p[U];
#pragma unroll
        for (int t = 0; t < U; ++t) {
          const int at = min(q + t * G, tot - 1), e = at / BS;
          p[t] = &a.foffd[(size_t)usrc[e] * BS + (at - e * BS)];
          v[t] = ld_relaxed(p[t]);
        }
        for (unsigned n = 1;; ++n) {
          bool wait = false;
#pragma unroll
          for (int t = 0; t < U; ++t) wait |= is_sentinel(v[t]);
          if (!wait) break;
#pragma unroll
          for (int t = 0; t < U; ++t)
            if (is_sentinel(v[t])) v[t] = ld_relaxed(p[t]);
          if ((n & 255) == 0) {
            if (t0 == 0) t0 = clock64();
            if (clock64() - t0 > kWaitCycles) record_fail(err, kErrTimeout, kSitePoll, -1, i);
            if (ld_relaxed_int(err) != 0) {
              ok = false;
              break;
            }
          }
        }
#pragma unroll
        for (int t = 0; t < U; ++t)
          if (q + t * G < tot) uv[q + t * G] = v[t];
      }
    }
    if (!__all_sync(0xffffffffu, ok)) break;
    int most = nlow;
#pragma unroll
    for (int o = 16; o >= G; o >>= 1) most = max(most, __shfl_xor_sync(0xffffffffu, most, o));
    for (int kk = 0; kk < most; ++kk) {
      if (kk < nlow && jl < J) {
        double l[B];  // A_ik holds the updates of all k' < k
#pragma unroll
        for (int q = 0; q < B; ++q) l[q] = rowv[kk * BS + r * B + q];
        for (int e = ubeg[kk] + jl; e < ubeg[kk + 1]; e += J) {
          const int t = utgt[e];
          if (t < 0) continue;
          const double* pk = uv + e * BS;
          double* p = rowv + t * BS + comp;
          if constexpr (B == 1) *p -= l[0] * pk[0];
          else if constexpr (B == 2) *p -= l[0] * pk[c] + l[1] * pk[2 + c];
          else *p -= l[0] * pk[c] + l[1] * pk[3 + c] + l[2] * pk[6 + c];
        }
      }
      __syncwarp();
    }
    // pivot inverse (matdiafrac_blkcrs.cpp:885-895 / 933-951 / 998-1013)
    const double* t = rowv + a.maxrow * BS;
    bool sing = false;
    double dv = 0.0;  // component `comp` of D^-1 (lanes jl == 0)
    if constexpr (B == 1) {
      const double v = t[0];
      sing = !(fabs(v) > 1.0e-30);
      dv = sing ? v : 1.0 / v;
    } else if constexpr (B == 2) {
      const double det = t[0] * t[3] - t[1] * t[2];
      sing = !(fabs(det) > 1.0e-30);
      if (sing) {
        dv = t[comp];
      } else {
        const double inv_det = 1.0 / det;
        dv = (r == c ? inv_det : -inv_det) * t[r == c ? 3 - comp : comp];
      }
    } else {
      // the six products of the determinant, one per lane: nibble m of the
      // constants holds an index of product m
      const int m = 4 * (sub < 6 ? sub : 0);
      const double pr = t[0x360630 >> m & 15] * t[0x147174 >> m & 15] * t[0x825528 >> m & 15];
      const double det = __shfl_sync(0xffffffffu, pr, 0) + __shfl_sync(0xffffffffu, pr, 1) +
                         __shfl_sync(0xffffffffu, pr, 2) - __shfl_sync(0xffffffffu, pr, 3) -
                         __shfl_sync(0xffffffffu, pr, 4) - __shfl_sync(0xffffffffu, pr, 5);
      sing = !(fabs(det) > 1.0e-30);
      if (sing) {
        dv = t[comp];
      } else {  // component (t[p] t[q] - t[u] t[v]) / det, the indices likewise
        const int n = 4 * comp;
        const double inv_det = 1.0 / det;
        dv = inv_det * (t[0x013205124ull >> n & 15] * t[0x467386578ull >> n & 15] -
                        t[0x104023215ull >> n & 15] * t[0x376568487ull >> n & 15]);
      }
    }
    __syncwarp();
    if (sub < BS) rowv[a.maxrow * BS + comp] = dv;
    if (on && sub == 0 && sing) atomicAdd(a.sync + 1, 1);
    __syncwarp();
    // out: L as it is, U'_ij = D_i^-1 A_ij (j > i), D^-1
    if (jl < J) {
      double d[B];
#pragma unroll
      for (int q = 0; q < B; ++q) d[q] = t[r * B + q];
      for (int s = jl; s < nrow; s += J) {
        const double* p = rowv + s * BS;
        double v = p[comp];
        if (s >= nlow) {
          if constexpr (B == 1) v = p[0] * d[0];
          else if constexpr (B == 2) v = d[0] * p[c] + d[1] * p[2 + c];
          else v = d[0] * p[c] + d[1] * p[3 + c] + d[2] * p[6 + c];
        }
        st_relaxed(&a.foffd[(size_t)(r0 + s) * BS + comp], v);
      }
      if (on && jl == 0) a.fdiag[(size_t)i * BS + comp] = dv;
    }
    __syncwarp();
    u = next;
  }
}

IluPlan ilu_plan(int b, const std::vector<int>& lev_ptr, const std::vector<int>& lev_rows, const int* rowptr,
                 const int* colind, const int* diaind) {
  IluPlan P;
  const int G = b == 1 ? 8 : b == 2 ? 16 : 32, per = 32 / G;
  for (size_t l = 0; l + 1 < lev_ptr.size(); ++l) {
    int k = 0;
    for (int p = lev_ptr[l]; p < lev_ptr[l + 1]; p += per, ++k)
      P.units.push_back(make_int2(p, std::min(per, lev_ptr[l + 1] - p)));
    P.max_level_units = std::max(P.max_level_units, k);
  }
  for (int row : lev_rows) {
    int nu = 0;
    for (int q = rowptr[row]; q < diaind[row]; ++q) nu += rowptr[colind[q] + 1] - diaind[colind[q]];
    P.maxrow = std::max(P.maxrow, rowptr[row + 1] - rowptr[row]);
    P.maxlow = std::max(P.maxlow, diaind[row] - rowptr[row]);
    P.maxu = std::max(P.maxu, nu);
  }
  P.warp_bytes = per * ilu_group_bytes(b, P.maxrow, P.maxlow, P.maxu);
  if (P.warp_bytes * kIluWarps > 96 * 1024) P.warp_bytes = 0;
  return P;
}

template <int B>
static cudaError_t launch_ilu_b(const IluPlan& P, const IluArgs& a, int nsm, cudaStream_t st) {
  const size_t smem = P.warp_bytes * kIluWarps;
  cudaError_t e = cudaFuncSetAttribute(k_ilu<B>, cudaFuncAttributeMaxDynamicSharedMemorySize, 96 * 1024);
  if (e != cudaSuccess) return e;
  // enough warps for three levels' units (those of the next levels load while
  // they wait), at most per_sm CTAs, one warp per scheduler each: with more the
  // units of a wide level pile up on some of the schedulers
  // (3x3, 56^3: 8.3 ms with ten CTAs per SM, 2.7 with two and the sentinel)
  constexpr int per_sm = 2;
  const int grid = std::max(1, std::min((3 * P.max_level_units + kIluWarps - 1) / kIluWarps, nsm * per_sm));
  k_ilu<B><<<grid, kIluWarps * 32, smem, st>>>(a, P.warp_bytes / (32 / IluLanes<B>::G));
  return cudaGetLastError();
}

cudaError_t launch_ilu(int b, const IluPlan& P, const IluArgs& a, int nsm, cudaStream_t st) {
  if (a.nunits <= 0) return cudaSuccess;
  switch (b) {
    case 1: return launch_ilu_b<1>(P, a, nsm, st);
    case 2: return launch_ilu_b<2>(P, a, nsm, st);
    case 3: return launch_ilu_b<3>(P, a, nsm, st);
    default: return cudaErrorInvalidValue;
  }
}

// SetValue_Initialize for a factor with fill-in (matvec/matdiafrac_blkcrs.h:
// 90-96): the factor storage was zeroed; every block of A goes to the slot of
// the same column in the factor pattern.  One thread per value.
__global__ void k_factor_init(long long nval, int bs, const int* __restrict__ a2f, const double* __restrict__ offd,
                              double* __restrict__ foffd) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nval) return;
  const long long c = t / bs;
  foffd[(size_t)a2f[c] * bs + (t - c * bs)] = offd[t];
}

cudaError_t launch_factor_init(int B, long long nnz_a, const int* a2f, const double* offd, double* foffd,
                               cudaStream_t st) {
  const long long nval = nnz_a * B * B;
  if (nval <= 0) return cudaSuccess;
  const int tpb = 256;
  k_factor_init<<<(unsigned)((nval + tpb - 1) / tpb), tpb, 0, st>>>(nval, B * B, a2f, offd, foffd);
  return cudaGetLastError();
}

cudaError_t launch_ilu_level(int B, const int* rows, int cnt, const int* rowptr, const int* colind,
                             const int* diaind, double* fdiag, double* foffd, int* nsing, cudaStream_t st,
                             bool dependent) {
  if (cnt <= 0) return cudaSuccess;
  const int tpb = 64;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((cnt + tpb - 1) / tpb);
  cfg.blockDim = dim3(tpb);
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = dependent ? 1 : 0;
  switch (B) {
    case 1: return cudaLaunchKernelEx(&cfg, k_ilu_level<1>, rows, cnt, rowptr, colind, diaind, fdiag, foffd, nsing);
    case 2: return cudaLaunchKernelEx(&cfg, k_ilu_level<2>, rows, cnt, rowptr, colind, diaind, fdiag, foffd, nsing);
    case 3: return cudaLaunchKernelEx(&cfg, k_ilu_level<3>, rows, cnt, rowptr, colind, diaind, fdiag, foffd, nsing);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace dfg
