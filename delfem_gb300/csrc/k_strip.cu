// k_strip.cu -- forward / backward substitution of the block ILU factor
// (CMatDiaFrac_BlkCrs::ForwardSubstitution / BackwardSubstitution,
// src/matvec/matdiafrac_blkcrs.cpp:332-669) in the reference's natural order,
// one warp per strip of rows (3x3 FP64: four).
//
// What bounds a sweep is its chain of dependency levels, so the kernel is
// built around the time from one level to the next.  A strip (strip.cpp) holds
// up to RW grid lines; its warp takes one level of the strip per step, the
// rows' dependencies inside the strip coming from a shared-memory ring of the
// warp's own results: store, __syncwarp, load -- 33 cycles on GB300 -- and no
// barrier between warps.  Everything else a step needs is brought to shared
// memory ahead of it:
//   * the step records (dependency codes, factor blocks, output positions) and
//     the right-hand sides, both contiguous in step order, by two TMA bulk
//     copies per chunk of steps, NS chunks ahead, from a loader warp (issuing
//     them takes 230 cycles, which the compute warp paid per chunk before);
//   * the values of other strips by a receiver warp beside each compute warp.
//     A row that another strip needs is also written to an exchange buffer in
//     global memory that was filled with a NaN sentinel; the receiver's lanes
//     poll the strip's items, listed in the order of first use, a few each in
//     flight, and put them into the warp's mailbox (a ring of slots) as they
//     arrive.  `delivered` counts the arrived prefix; a step says how many
//     items it needs, one compare when they are there.
// Measured on GB300, FP32, per sweep (forward / backward): the 1000x500
// cantilever 0.13 / 0.12 ms (ranged kernel 1.09 / 1.10), Poisson on 301x257
// cells 45 / 45 us (one CTA per sweep 200 / 196), elasticity on 56^3 cells 81 /
// 77 us (a launch per level 345 / 306).  FP64: the cantilever 0.57 / 0.40 ms
// (2.36 / 2.08), Poisson on 128x128 cells 64 / 54 us (133 / 123).  Inside one
// strip a level costs 103 (1x1 blocks) to 490 (3x3, 7 entries) cycles in FP32
// and 380 to 1,280 in FP64, where each warp-wide FMA takes its scheduler 64; a
// hand-off between strips costs 1,500 to 3,000, of which the L2 takes 600-900.
//
// Strips are claimed in order, W per CTA, through a ticket, so a strip only
// waits on strips already running, whatever the number of resident CTAs.
// Every wait is bounded; one that gives up records kErrTimeout, and the launch
// drains its copies and returns.
//
// A row is evaluated by the operations of the one-CTA kernel in its order (RowSum,
// then D^-1), and of the ranged kernel in batched launches, so these give the same
// bits; with split, column by column.
//
// Chunk layout: [need: CH ints, kStripHdr bytes][steps: step_bytes each]; a
// step is pieces of 16 bytes per lane, piece j of lane l at (j*32 + l)*16:
// MC pieces of metadata (16-bit codes, output position, exchange slot), then
// VC pieces of values (the lane's factor rows entry by entry, then its D^-1
// row(s) in the forward sweep).
#include "dfg_common.cuh"
#include "k_mbar.cuh"
#include "k_strip.h"

namespace dfg {

__device__ __forceinline__ int ld_acquire_s(const int* p) {
  int v;
  asm volatile("ld.acquire.cta.shared::cta.s32 %0, [%1];" : "=r"(v) : "r"(smem_u32(p)) : "memory");
  return v;
}
__device__ __forceinline__ void st_release_s(int* p, int v) {
  asm volatile("st.release.cta.shared::cta.s32 [%0], %1;" ::"r"(smem_u32(p)), "r"(v) : "memory");
}

// a row's value as the ring, mailbox and exchange buffer hold it
template <typename T, int N>
struct alignas(N * sizeof(T) > 16 ? 16 : N * sizeof(T)) Vec {
  T v[N];
};

// Relaxed gpu-scope load of a row's value under a predicate (no branch); v is
// left as it is otherwise.  Each element is compared with the sentinel by
// itself, so no atomicity beyond an element is needed.
__device__ __forceinline__ void xload(bool on, const float* p, Vec<float, 1>& v) {
  asm volatile("{\n .reg .pred q;\n setp.ne.s32 q, %1, 0;\n @q ld.relaxed.gpu.global.f32 %0, [%2];\n}"
               : "+f"(v.v[0]) : "r"((int)on), "l"(p));
}
__device__ __forceinline__ void xload(bool on, const double* p, Vec<double, 1>& v) {
  asm volatile("{\n .reg .pred q;\n setp.ne.s32 q, %1, 0;\n @q ld.relaxed.gpu.global.f64 %0, [%2];\n}"
               : "+d"(v.v[0]) : "r"((int)on), "l"(p));
}
__device__ __forceinline__ void xload(bool on, const float* p, Vec<float, 2>& v) {
  asm volatile("{\n .reg .pred q;\n setp.ne.s32 q, %2, 0;\n @q ld.relaxed.gpu.global.v2.f32 {%0, %1}, [%3];\n}"
               : "+f"(v.v[0]), "+f"(v.v[1]) : "r"((int)on), "l"(p));
}
__device__ __forceinline__ void xload(bool on, const double* p, Vec<double, 2>& v) {
  asm volatile("{\n .reg .pred q;\n setp.ne.s32 q, %2, 0;\n @q ld.relaxed.gpu.global.v2.f64 {%0, %1}, [%3];\n}"
               : "+d"(v.v[0]), "+d"(v.v[1]) : "r"((int)on), "l"(p));
}
__device__ __forceinline__ void xload(bool on, const float* p, Vec<float, 4>& v) {
  asm volatile("{\n .reg .pred q;\n setp.ne.s32 q, %4, 0;\n @q ld.relaxed.gpu.global.v4.f32 {%0, %1, %2, %3}, [%5];\n}"
               : "+f"(v.v[0]), "+f"(v.v[1]), "+f"(v.v[2]), "+f"(v.v[3]) : "r"((int)on), "l"(p));
}
__device__ __forceinline__ void xload(bool on, const double* p, Vec<double, 4>& v) {
  asm volatile("{\n .reg .pred q;\n setp.ne.s32 q, %3, 0;\n @q ld.relaxed.gpu.global.v2.f64 {%0, %1}, [%4];\n"
               " @q ld.relaxed.gpu.global.f64 %2, [%4+16];\n}"
               : "+d"(v.v[0]), "+d"(v.v[1]), "+d"(v.v[2]) : "r"((int)on), "l"(p));
}
// Stores under a predicate (no branch): a row's value at p when on >= 0.  The
// exchange stores are gpu-scope relaxed.
__device__ __forceinline__ void xstore(int on, float* p, const Vec<float, 1>& y) {
  asm volatile("{\n .reg .pred q;\n setp.ge.s32 q, %0, 0;\n @q st.relaxed.gpu.global.f32 [%1], %2;\n}" ::"r"(on), "l"(p),
               "f"(y.v[0]));
}
__device__ __forceinline__ void xstore(int on, double* p, const Vec<double, 1>& y) {
  asm volatile("{\n .reg .pred q;\n setp.ge.s32 q, %0, 0;\n @q st.relaxed.gpu.global.f64 [%1], %2;\n}" ::"r"(on), "l"(p),
               "d"(y.v[0]));
}
__device__ __forceinline__ void xstore(int on, float* p, const Vec<float, 2>& y) {
  asm volatile("{\n .reg .pred q;\n setp.ge.s32 q, %0, 0;\n @q st.relaxed.gpu.global.v2.f32 [%1], {%2, %3};\n}" ::"r"(on),
               "l"(p), "f"(y.v[0]), "f"(y.v[1]));
}
__device__ __forceinline__ void xstore(int on, float* p, const Vec<float, 4>& y) {
  asm volatile("{\n .reg .pred q;\n setp.ge.s32 q, %0, 0;\n @q st.relaxed.gpu.global.v4.f32 [%1], {%2, %3, %4, %5};\n}" ::"r"(on),
               "l"(p), "f"(y.v[0]), "f"(y.v[1]), "f"(y.v[2]), "f"(y.v[3]));
}
__device__ __forceinline__ void ostore(int on, float* p, const Vec<float, 4>& y) {  // three elements
  asm volatile(
      "{\n .reg .pred q;\n setp.ge.s32 q, %0, 0;\n @q st.global.f32 [%1], %2;\n @q st.global.f32 [%1+4], %3;\n"
      " @q st.global.f32 [%1+8], %4;\n}" ::"r"(on),
      "l"(p), "f"(y.v[0]), "f"(y.v[1]), "f"(y.v[2]));
}
__device__ __forceinline__ void ostore(int on, float* p, const Vec<float, 1>& y) {
  asm volatile("{\n .reg .pred q;\n setp.ge.s32 q, %0, 0;\n @q st.global.f32 [%1], %2;\n}" ::"r"(on), "l"(p), "f"(y.v[0]));
}
__device__ __forceinline__ void ostore(int on, double* p, const Vec<double, 1>& y) {
  asm volatile("{\n .reg .pred q;\n setp.ge.s32 q, %0, 0;\n @q st.global.f64 [%1], %2;\n}" ::"r"(on), "l"(p), "d"(y.v[0]));
}
__device__ __forceinline__ void ostore(int on, float* p, const Vec<float, 2>& y) {
  asm volatile("{\n .reg .pred q;\n setp.ge.s32 q, %0, 0;\n @q st.global.v2.f32 [%1], {%2, %3};\n}" ::"r"(on), "l"(p),
               "f"(y.v[0]), "f"(y.v[1]));
}

// The receiver of one strip: polls its items in the exchange buffer and
// delivers them to the mailbox in order.  Two sets of H batches of 32 items are
// in flight; a set that is through makes room for the next one.  More in flight
// slow everyone's polls down (3D elasticity, 56^3 FP64: 251 us per sweep with
// H = 1, 265 with 2, 309 with 4), fewer starve short steps (3D Poisson, 44^3
// FP32: 47, 41 and 45 us).
template <typename T, int B, int H>
__device__ __forceinline__ void receive(const StripSlot& S, int r, unsigned char* mail, int* delivered,
                                        const int* consumed, int* err, int lane) {
  constexpr int BP = B == 3 ? 4 : B;
  constexpr int VS = BP * (int)sizeof(T);
  constexpr int M = strip_mailbox(VS);
  constexpr int U = 2 * H;
  const int i0 = S.item_ptr[r], cnt = S.item_ptr[r + 1] - i0;
  const int2* __restrict__ items = S.items + i0;
  const T* xch = reinterpret_cast<const T*>(S.xch);
  auto item = [&](int q) { return q < cnt ? items[q] : make_int2(0, 0); };
  int2 it[U], nxt[H];
  unsigned got = 0;  // bit u: this lane's item of batch u has been delivered
#pragma unroll
  for (int u = 0; u < U; ++u) it[u] = item(u * 32 + lane);
#pragma unroll
  for (int u = 0; u < H; ++u) nxt[u] = item((U + u) * 32 + lane);
  int base = 0;
  bool started = false;  // until the first item is there it is polled alone: a strip far from the front leaves the L2 to the others
  long long t0 = clock64();
  for (unsigned n = 1; base < cnt; ++n) {
    if ((n & 63) == 0) {
      if (ld_relaxed_int(err) != 0) return;
      if (clock64() - t0 > kWaitCycles) {
        if (lane == 0) record_fail(err, kErrTimeout, kSitePoll, -1, r);
        return;
      }
    }
    const int done_steps = cnt > M ? ld_acquire_s(consumed) : 0;
    Vec<T, BP> v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
#pragma unroll
      for (int d = 0; d < BP; ++d) v[u].v[d] = sentinel_value<T>();
      xload(!(got >> u & 1) && base + u * 32 + lane < cnt && it[u].y <= done_steps && (started || (u == 0 && lane == 0)), xch + (size_t)it[u].x * BP, v[u]);
    }
    const unsigned had = got;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      bool ok = true;
#pragma unroll
      for (int d = 0; d < B; ++d) ok &= !is_sentinel(v[u].v[d]);
      if (ok) *reinterpret_cast<Vec<T, BP>*>(mail + (size_t)((base + u * 32 + lane) % M) * VS) = v[u];
      got |= (unsigned)ok << u;
    }
    if (!__any_sync(0xffffffffu, got != had)) continue;
    t0 = clock64();
    started = true;
    // the delivered prefix over the batches in flight
    int pre = base;
    bool whole = true;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const unsigned b = __ballot_sync(0xffffffffu, got >> u & 1);
      pre += whole ? __popc(b & ~(b + 1u)) : 0;
      whole = whole && b == 0xffffffffu;
    }
    __syncwarp();
    if (lane == 0) st_release_s(delivered, pre);
    if (pre >= cnt) break;
    if (pre - base >= 32 * H) {
#pragma unroll
      for (int u = 0; u < H; ++u) {
        it[u] = it[H + u];
        it[H + u] = nxt[u];
      }
      got >>= H;
      base += 32 * H;
#pragma unroll
      for (int u = 0; u < H; ++u) nxt[u] = item(base + (U + u) * 32 + lane);
    }
  }
}

// (one CTA per SM in the bounds: without it ptxas aims at several and keeps
// steps to 64 registers and fewer, 2 to 10 % slower)
template <typename T, int B, bool FWD, int NE, bool SPLIT, bool FOUR>
__global__ void __launch_bounds__((2 * kStripMaxWarps + 1) * 32, 1) k_strip(StripArgs a) {
  constexpr int SZ = (int)sizeof(T);
  constexpr StripDims D = strip_dims(B, SZ, FWD, NE, SPLIT);
  constexpr int LPR = D.LPR, Q = D.Q, RW = D.RW, MC = D.MC, VC = D.VC, CH = D.CH, VS = D.VS;
  constexpr int BP = B == 3 ? 4 : B;          // elements of a row's value, padded
  constexpr int PER16 = 16 / SZ;
  constexpr int EV = B * B / LPR;             // values per entry and lane
  constexpr int RHS_CHUNK = CH * D.rhs_bytes;
  // values are loaded a step ahead where two sets of them fit the registers
  constexpr int VB = VC <= 8 ? 2 : 1;
  constexpr int HB = B == 3 ? 1 : 2;
  // A step's stores to global memory are issued in the next step, while that
  // step's dependency loads are under way, instead of between its result and
  // them (one strip of 2000 lines, cycles per level: 1x1 FP32 113 -> 103, FP64 403
  // -> 379; 2x2 FP32 147 -> 135, FP64 709 -> 699).  3x3 steps are long: there the
  // exchange store goes at once, since waiting costs the next strip more (FP64
  // 24^3 cells 100.4 us per sweep held back, 98.0 at once).
  constexpr bool XNOW = B == 3;
  constexpr int G = D.G;
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ int s_group, s_slot, s_stop;
  const int W = a.W, NS = a.NS;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool compute = warp < W * Q, load_warp = warp == W * Q + W;
  const int w = compute ? warp / Q : load_warp ? min(lane, W - 1) : warp - W * Q;  // (the loader's lane w serves strip w)
  uint64_t* full = reinterpret_cast<uint64_t*>(smem) + w * NS;
  int* delivered = reinterpret_cast<int*>(smem + (size_t)W * NS * 8) + w * 4;
  int* consumed = delivered + 1;
  unsigned char* rstage = smem + strip_stage_offset(D, W, NS, w);  // NS chunks of records
  unsigned char* vstage = rstage + (size_t)NS * D.chunk_bytes;     // NS chunks of right-hand sides
  unsigned char* region = smem + strip_region_offset(D, W, NS, w);
  if (compute && lane < kStripZero / 4) reinterpret_cast<unsigned*>(region)[lane] = 0u;
  if (threadIdx.x == 0) {
    for (int s = 0; s < W * NS; ++s) mbar_init(reinterpret_cast<uint64_t*>(smem) + s, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // One solve's sweep claims its first strips and asks for their first records
  // before it waits for the kernel ahead of it: the factor does not change
  // within a solve, and the ticket is reset by another kernel than that one
  // (a PCG iteration, Poisson on 24x24 cells 50 -> 47 us, on 128x128 134 -> 131, on
  // 301x257, FP32 everything, 111 -> 109).
  bool fresh = a.batch == nullptr;
  if (!fresh) pdl_enter();
  int st = 0, ph = 0;  // stage and phase of the strip's next chunk (compute warps and loader alike)
  for (;;) {
    int issued = 0;  // loader: chunks of the strip issued
    if (compute && lane == 0) {
      *delivered = 0;
      *consumed = 0;
    }
    if (threadIdx.x == 0) {
      int t = atomicAdd(a.ticket, 1), j = 0;
      if (const StripBatch* bt = a.batch) {
        const int n = bt->nslots;
        if (n == 0 || t >= bt->group_start[n]) {
          t = -1;
        } else {
          int lo = 0, hi = n - 1;  // last j with group_start[j] <= t
          while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (bt->group_start[mid] <= t) lo = mid; else hi = mid - 1;
          }
          j = lo;
          t = ld_relaxed_int(bt->slot[j].done) != 0 ? -2 : t - bt->group_start[j];
        }
      } else if (t * W >= a.one.nstrips) {
        t = -1;
      }
      s_group = t;
      s_slot = j;
    }
    __syncthreads();
    const int group = s_group;
    const StripSlot S = a.batch ? a.batch->slot[s_slot] : a.one;
    if (fresh) {
      fresh = false;
      const int r0 = group * W + w;
      const bool mine = load_warp && lane < W && group >= 0 && r0 < S.nstrips;
      const int c0 = mine ? S.strip_chunk[r0] : 0, first = mine ? min(S.strip_chunk[r0 + 1] - c0, NS) : 0;
      for (; issued < first; ++issued) {
        mbar_expect_tx(&full[issued], D.chunk_bytes + RHS_CHUNK);
        tma_load_1d(rstage + (size_t)issued * D.chunk_bytes, S.rec + (size_t)(c0 + issued) * D.chunk_bytes,
                    D.chunk_bytes, &full[issued]);
      }
      pdl_enter();
      for (int k = 0; k < first; ++k)
        tma_load_1d(vstage + (size_t)k * RHS_CHUNK,
                    reinterpret_cast<const unsigned char*>(S.in) + (size_t)(c0 + k) * RHS_CHUNK, RHS_CHUNK, &full[k]);
      if (a.other_ticket && blockIdx.x == 0 && threadIdx.x == 0) *a.other_ticket = 0;
      if (S.done && *S.done) {
        for (int k = 0; k < first; ++k) mbar_drain(&full[k], 0);
        return;
      }
    }
    if (group == -1) break;
    if (group == -2) {  // a finished solve
      __syncthreads();
      continue;
    }
    const int r = group * W + w;
    if (load_warp) {
      // -------------------------------------------------------------- loader
      // lane w keeps warp w's stages filled: a chunk's records and its
      // right-hand sides, NS chunks ahead of the chunks the warp has finished
      const bool on = lane < W && r < S.nstrips;
      const int c0 = on ? S.strip_chunk[r] : 0, nch = on ? S.strip_chunk[r + 1] - c0 : 0;
      const unsigned char* rec = S.rec + (size_t)(c0 + issued) * D.chunk_bytes;
      const unsigned char* in = reinterpret_cast<const unsigned char*>(S.in) + (size_t)(c0 + issued) * RHS_CHUNK;
      bool failing = false;
      for (unsigned n = 1; __any_sync(0xffffffffu, issued < nch && !failing); ++n) {
        if (issued < nch && !failing) {
          const int done = ld_acquire_s(consumed) / CH;
          for (; issued < strip_issue_end(done, NS, nch); ++issued) {
            const int s = (st + issued) % NS;
            mbar_expect_tx(&full[s], D.chunk_bytes + RHS_CHUNK);
            tma_load_1d(rstage + (size_t)s * D.chunk_bytes, rec, D.chunk_bytes, &full[s]);
            tma_load_1d(vstage + (size_t)s * RHS_CHUNK, in, RHS_CHUNK, &full[s]);
            rec += D.chunk_bytes;
            in += RHS_CHUNK;
          }
          if ((n & 63) == 0) failing = ld_relaxed_int(a.err) != 0;
        }
        __nanosleep(64);
      }
    } else if (r < S.nstrips) {
      if (!compute) {
        receive<T, B, HB>(S, r, region + kStripZero + kStripRing * RW * VS, delivered, consumed, a.err, lane);
      } else {
        // ------------------------------------------------------------- compute
        const int c0 = S.strip_chunk[r], nch = S.strip_chunk[r + 1] - c0;
        const int tid = warp % Q * 32 + lane;                             // lane of the strip
        const int lr = strip_row(D, tid), el = lane - lane / LPR * LPR;  // row of the step, part of it (LPR > 1)
        // the strip's warps meet after every step
        auto step_sync = [&] {
          if constexpr (Q == 1) __syncwarp();
          else asm volatile("bar.sync %0, %1;" ::"r"(1 + w), "n"(32 * Q) : "memory");
        };
        const int p = SPLIT ? el / B : el, col = SPLIT ? el % B : 0;  // component, column of the block
        T* out = reinterpret_cast<T*>(S.out) + p;
        T* xch = reinterpret_cast<T*>(S.xch) + p;
        // one step's data, loaded a step ahead of its use; the addresses taken
        // from its metadata are worked out a step ahead too (the empty asm
        // statements keep them there), so that after the __syncwarp only the
        // loads themselves are left on the chain
        int4 meta[MC];
        Vec<T, PER16> val[VB][VC];
        T t[2][LPR == 1 ? B : 1];
        unsigned cd[2][NE];
        int o[2], xs[2];
        T *op[2], *xp[2];
        auto load = [&](int k, const unsigned char* sp, const unsigned char* vp) {
#pragma unroll
          for (int j = 0; j < MC; ++j) meta[j] = *reinterpret_cast<const int4*>(sp + j * 512 * Q);
#pragma unroll
          for (int j = 0; j < VC; ++j)
            if (VB == 2) val[k % VB][j] = *reinterpret_cast<const Vec<T, PER16>*>(sp + (MC + j) * 512 * Q);
          const T* rh = reinterpret_cast<const T*>(vp);
          if constexpr (LPR == 1) {
#pragma unroll
            for (int d = 0; d < B; ++d) t[k][d] = rh[lane * B + d];
          } else if constexpr (SPLIT) {
            t[k][0] = col == 0 && lr < RW ? rh[lr * B + p] : T(0);
          } else {
            t[k][0] = rh[lane];
          }
        };
        auto decode = [&](int k) {
          auto mint = [&](int i) -> int {
            return (i & 3) == 0 ? meta[i / 4].x : (i & 3) == 1 ? meta[i / 4].y : (i & 3) == 2 ? meta[i / 4].z : meta[i / 4].w;
          };
#pragma unroll
          for (int e = 0; e < NE; ++e) {
            cd[k][e] = (e & 1) ? (unsigned)mint(e / 2) >> 16 : (unsigned)mint(e / 2) & 0xffffu;
            asm volatile("" : "+r"(cd[k][e]));
          }
          o[k] = mint((NE + 1) / 2);
          xs[k] = mint((NE + 1) / 2 + 1);
          if (SPLIT && col != 0) o[k] = xs[k] = -1;
          op[k] = out + (long long)o[k] * B;
          xp[k] = xch + (long long)xs[k] * BP;
          asm volatile("" : "+l"(op[k]), "+l"(xp[k]));
        };
        T* const ring0 = reinterpret_cast<T*>(region + kStripZero) + lr * BP;
        // the sum over the columns of a row's component (SPLIT)
        auto columns = [&](T v) -> T {
          if constexpr (B == 2) {
            return v + __shfl_xor_sync(0xffffffffu, v, 1);
          } else {
            const int l0 = lane - el + p * B;
            const T sum = __shfl_sync(0xffffffffu, v, l0) + __shfl_sync(0xffffffffu, v, l0 + 1);
            return sum + __shfl_sync(0xffffffffu, v, l0 + 2);
          }
        };
        bool abort = false;
        Vec<T, LPR == 1 ? BP : 1> yl;  // the last step's result
#pragma unroll
        for (int d = 0; d < (LPR == 1 ? BP : 1); ++d) yl.v[d] = 0;
        o[1] = xs[1] = -1;
        op[1] = out;
        xp[1] = xch;
        // waits until the progress word reaches `want`; its last value
        auto wait_for = [&](const int* word, int want, int site) -> int {
          int v;
          long long t0 = 0;
          for (unsigned n = 1; !__all_sync(0xffffffffu, (v = ld_acquire_s(word)) >= want); ++n) {
            if ((n & 255) == 0) {
              if (n == 256) t0 = clock64();
              const bool late = clock64() - t0 > kWaitCycles;
              if (late && lane == 0) record_fail(a.err, kErrTimeout, site, -1, r);
              if (__any_sync(0xffffffffu, late || ld_relaxed_int(a.err) != 0)) {
                abort = true;
                break;
              }
            }
          }
          return __shfl_sync(0xffffffffu, v, 0);
        };
        abort = !__all_sync(0xffffffffu, mbar_wait(&full[st], (unsigned)ph, a.err, kSiteFull, -1, r));
        int have = 0;
        const unsigned char *const sp0 = rstage + kStripHdr + tid * 16, *const vp0 = vstage;
        const unsigned char *sp = sp0 + (size_t)st * D.chunk_bytes, *vp = vp0 + (size_t)st * RHS_CHUNK;
        int need[CH];  // (one in G is used)
        auto load_need = [&](const unsigned char* s) {
#pragma unroll
          for (int j = G - 1; j < CH; j += G) need[j] = reinterpret_cast<const int*>(s - kStripHdr - tid * 16)[j];
        };
        if (!abort) {
          load(0, sp, vp);
          decode(0);
          load_need(sp);
        }
        T* rg = ring0;
        // (a strip of several warps meets in every step, also after one has given up)
        for (int c = 0; c < nch && (Q > 1 || !abort); ++c) {
          if (++st == NS) { st = 0; ph ^= 1; }
          // the test for the next chunk takes about 100 cycles: asked for here,
          // looked at in the last step
          const bool landed = c + 1 < nch && mbar_test_wait(&full[st], (unsigned)ph);
          const unsigned char* sp1 = st == 0 ? sp0 : sp + D.chunk_bytes;
          const unsigned char* vp1 = st == 0 ? vp0 : vp + RHS_CHUNK;
#pragma unroll
          for (int j = 0; j < CH; ++j) {
            if (Q > 1 && abort) {
              step_sync();
              continue;
            }
            if (j % G == 0 && need[j + G - 1] > have) {
              // only padding is left of the strip (the last step's stores are in set 1)
              static_assert(!D.ends || G % 2 == 0, "the end is seen in an even step");
              if (D.ends && need[j + G - 1] == kStripEnd) break;
              have = wait_for(delivered, need[j + G - 1], kSitePoll);
              if (abort) {
                if (Q == 1) break;
                step_sync();
                continue;
              }
            }
            constexpr int K2 = 2;
            const int k = j % K2;
            if (VB == 1) {
#pragma unroll
              for (int v = 0; v < VC; ++v)
                val[0][v] = *reinterpret_cast<const Vec<T, PER16>*>(sp + j * D.step_bytes + (MC + v) * 512 * Q);
            }
            auto A = [&](int i) -> T { return val[k % VB][i / PER16].v[i % PER16]; };
            // dependency values
            Vec<T, SPLIT ? 1 : BP> x[NE];
#pragma unroll
            for (int e = 0; e < NE; ++e) {
              const float* at = reinterpret_cast<const float*>(smem) + cd[k][e];
              x[e] = reinterpret_cast<const Vec<T, SPLIT ? 1 : BP>*>(at)[col];
            }
            // the last step's result leaves
            if (!XNOW) xstore(xs[k ^ 1], xp[k ^ 1], yl);
            ostore(o[k ^ 1], op[k ^ 1], yl);
            // the next step's data
            const bool more = j + 1 < CH || c + 1 < nch;
            if (j + 1 < CH) {
              load((j + 1) % K2, sp + (j + 1) * D.step_bytes, vp + (j + 1) * D.rhs_bytes);
            } else if (c + 1 < nch) {
              if (!__all_sync(0xffffffffu, landed) &&
                  !__all_sync(0xffffffffu, mbar_wait(&full[st], (unsigned)ph, a.err, kSiteFull, -1, r))) {
                abort = true;
                if (Q == 1) break;
                step_sync();
                continue;
              }
              load(0, sp1, vp1);
              load_need(sp1);
            }
            if (SZ == 8 && more) decode((j + 1) % K2);
            // the rows
            if constexpr (LPR == 1) {
              RowSum<T, B, B, FOUR> sum;
              sum.start(t[k]);
#pragma unroll
              for (int e = 0; e < NE; ++e)
#pragma unroll
                for (int d = 0; d < B; ++d)
#pragma unroll
                  for (int q = 0; q < B; ++q) sum.add(e, d, A(e * EV + d * B + q), x[e].v[q]);
              T acc[B];
#pragma unroll
              for (int d = 0; d < B; ++d) acc[d] = sum.row(d, t[k][d]);
              Vec<T, BP> y;
              y.v[BP - 1] = 0;
#pragma unroll
              for (int d = 0; d < B; ++d) {
                if constexpr (FWD) {
                  T u = A(NE * EV + d * B) * acc[0];
#pragma unroll
                  for (int q = 1; q < B; ++q) u += A(NE * EV + d * B + q) * acc[q];
                  y.v[d] = u;
                } else {
                  y.v[d] = acc[d];
                }
              }
              *reinterpret_cast<Vec<T, BP>*>(rg + j * RW * BP) = y;
              yl = y;
              if (XNOW) xstore(xs[k], xp[k], yl);
              if (SZ == 4 && more) decode((j + 1) % K2);
            } else if constexpr (SPLIT) {
              T acc = t[k][0];
#pragma unroll
              for (int e = 0; e < NE; ++e) acc -= A(e) * x[e].v[0];
              acc = columns(acc);
              if constexpr (FWD) acc = columns(A(NE) * __shfl_sync(0xffffffffu, acc, lane - el + col * B));
              if (lr < RW) rg[j * RW * BP + p] = acc;
              yl.v[0] = acc;
              if (XNOW) xstore(xs[k], xp[k], yl);
            } else {
              RowSum<T, B, 1, FOUR> sum;
              sum.start(t[k]);
#pragma unroll
              for (int e = 0; e < NE; ++e)
#pragma unroll
                for (int q = 0; q < B; ++q) sum.add(e, 0, A(e * EV + q), x[e].v[q]);
              T acc = sum.row(0, t[k][0]);
              if constexpr (FWD) {
                const int l0 = lane - p;
                T y = A(NE * EV) * __shfl_sync(0xffffffffu, acc, l0);
#pragma unroll
                for (int q = 1; q < B; ++q) {
                  const T tq = __shfl_sync(0xffffffffu, acc, l0 + q);
                  y += A(NE * EV + q) * tq;
                }
                acc = y;
              }
              if (lr < RW) rg[j * RW * BP + p] = acc;
              yl.v[0] = acc;
              if (XNOW) xstore(xs[k], xp[k], yl);
              if (SZ == 4 && more) decode((j + 1) % K2);
            }
            step_sync();
          }
          if (Q == 1 && abort) break;
          // the chunk's stage is free (warp 0 waited for its copies, unless it gave up)
          if (strip_publishes(Q > 1 && abort) && tid == 0) st_release_s(consumed, (c + 1) * CH);
          sp = sp1;
          vp = vp1;
          rg = (c + 1) * CH % kStripRing == 0 ? ring0 : rg + CH * RW * BP;
        }
        if (abort) {
          if (lane == 0) record_fail(a.err, kErrTimeout, kSiteRange, -1, r);
        } else {
          if (!XNOW) xstore(xs[1], xp[1], yl);
          ostore(o[1], op[1], yl);
        }
      }
    }
    __syncthreads();
    if (threadIdx.x == 0) s_stop = ld_relaxed_int(a.err) != 0;
    __syncthreads();
    if (s_stop) {  // copies in flight land before the CTA leaves (bounded)
      for (int k = strip_drain_begin(ld_acquire_s(consumed), CH); k < issued; ++k)
        mbar_drain(&full[(st + k) % NS], (unsigned)(ph ^ ((st + k) / NS & 1)));
      break;
    }
    if (load_warp && r < S.nstrips) {
      const int nch = S.strip_chunk[r + 1] - S.strip_chunk[r];
      ph ^= (st + nch) / NS & 1;
      st = (st + nch) % NS;
    }
  }
}

// ------------------------------------------------------------------ records

__global__ void k_strip_meta(int CH, int lane_pieces, int step_bytes, int chunk_bytes, const int* __restrict__ meta,
                             const int* __restrict__ need, unsigned char* rec) {
  unsigned char* ck = rec + (size_t)blockIdx.x * chunk_bytes;
  if (threadIdx.x < kStripHdr / 4)
    reinterpret_cast<int*>(ck)[threadIdx.x] = (int)threadIdx.x < CH ? need[(size_t)blockIdx.x * CH + threadIdx.x] : 0;
  const int per = lane_pieces;  // pieces per step
  const int4* m = reinterpret_cast<const int4*>(meta) + (size_t)blockIdx.x * CH * per;
  for (int i = threadIdx.x; i < CH * per; i += blockDim.x)
    reinterpret_cast<int4*>(ck + kStripHdr + (size_t)(i / per) * step_bytes)[i % per] = m[i];
}

// one block per step: value k of lane l in piece k / (16 / sizeof(T))
template <typename T, int B, bool FWD>
__global__ void k_strip_pack(StripPackArgs a) {
  constexpr int SZ = (int)sizeof(T), PER16 = 16 / SZ, BS = B * B;
  const int LPR = a.d.LPR, EV = BS / LPR, lanes = 32 * a.d.Q;
  const long long s = blockIdx.x;
  const int RW = a.d.RW, ne = a.ne;
  T* v = reinterpret_cast<T*>(a.rec + (size_t)(s / a.d.CH) * a.d.chunk_bytes + kStripHdr +
                              (size_t)(s % a.d.CH) * a.d.step_bytes + (size_t)a.d.MC * lanes * 16);
  for (int i = threadIdx.x; i < a.d.VC * lanes * PER16; i += blockDim.x) {
    const int lane = i / PER16 % lanes, k = (i / PER16 / lanes) * PER16 + i % PER16;
    const int l = strip_row(a.d, lane), p = lane % 32 % LPR, e = k / EV, q = k - e * EV;
    double x = 0.0;
    if (l < RW) {
      const int m = p * EV + q;
      if (e < ne) {
        const int c = a.ent_slot[((size_t)s * RW + l) * ne + e];
        if (c >= 0) x = a.foffd[(size_t)c * BS + m];
      } else if (FWD && e == ne) {
        const int row = a.step_rows[(size_t)s * RW + l];
        if (row >= 0) x = a.fdiag[(size_t)row * BS + m];
      }
    }
    v[i] = (T)x;
  }
}

// ------------------------------------------------------------------ launchers

cudaError_t launch_strip_meta(const StripDims& d, int nchunks, const int* meta, const int* need, unsigned char* rec,
                              cudaStream_t st) {
  if (nchunks <= 0) return cudaSuccess;
  k_strip_meta<<<nchunks, 128, 0, st>>>(d.CH, d.MC * 32 * d.Q, d.step_bytes, d.chunk_bytes, meta, need, rec);
  return cudaGetLastError();
}

template <typename T, bool FWD>
static cudaError_t pack_t(const StripPackArgs& a, cudaStream_t st) {
  if (a.nsteps <= 0) return cudaSuccess;
  switch (a.b) {
    case 1: k_strip_pack<T, 1, FWD><<<(unsigned)a.nsteps, 128, 0, st>>>(a); break;
    case 2: k_strip_pack<T, 2, FWD><<<(unsigned)a.nsteps, 128, 0, st>>>(a); break;
    case 3: k_strip_pack<T, 3, FWD><<<(unsigned)a.nsteps, 128, 0, st>>>(a); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

cudaError_t launch_strip_pack(bool forward, bool fp32, const StripPackArgs& a, cudaStream_t st) {
  if (fp32) return forward ? pack_t<float, true>(a, st) : pack_t<float, false>(a, st);
  return forward ? pack_t<double, true>(a, st) : pack_t<double, false>(a, st);
}

// calls f(kernel) for the instance of (fp32, b, forward, ne, split, four)
template <typename T, int B, bool FWD, bool SPLIT, bool FOUR = false, typename F>
static cudaError_t with_class(int ne, F&& f) {
  switch (ne) {
    case 3: return f(k_strip<T, B, FWD, 3, SPLIT, FOUR>);
    case 4: return f(k_strip<T, B, FWD, 4, SPLIT, FOUR>);
    case 7: return f(k_strip<T, B, FWD, 7, SPLIT, FOUR>);
    case 16: return f(k_strip<T, B, FWD, 16, SPLIT, FOUR>);
    default: return cudaErrorInvalidValue;
  }
}
template <typename T, typename F>
static cudaError_t with_block(int b, bool forward, int ne, F&& f) {
  switch (b) {
    case 1: return forward ? with_class<T, 1, true, false>(ne, f) : with_class<T, 1, false, false>(ne, f);
    case 2: return forward ? with_class<T, 2, true, false>(ne, f) : with_class<T, 2, false, false>(ne, f);
    case 3: return forward ? with_class<T, 3, true, false>(ne, f) : with_class<T, 3, false, false>(ne, f);
    default: return cudaErrorInvalidValue;
  }
}
template <typename F>
static cudaError_t with_kernel(bool fp32, int b, bool forward, int ne, bool split, bool four, F&& f) {
  if (four)
    return forward ? with_class<float, 3, true, false, true>(ne, f) : with_class<float, 3, false, false, true>(ne, f);
  if (split && b == 2) return forward ? with_class<double, 2, true, true>(ne, f) : with_class<double, 2, false, true>(ne, f);
  if (split && b == 3) return forward ? with_class<double, 3, true, true>(ne, f) : with_class<double, 3, false, true>(ne, f);
  return fp32 ? with_block<float>(b, forward, ne, f) : with_block<double>(b, forward, ne, f);
}

cudaError_t launch_strip(bool forward, bool fp32, int b, const StripArgs& a, int grid, size_t smem, cudaStream_t st,
                         bool dep) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  const int Q = a.split && b == 3 ? 4 : 1;  // warps per strip
  cfg.blockDim = dim3(32 * (a.W * (Q + 1) + 1));
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = dep ? 1 : 0;
  return with_kernel(fp32, b, forward, a.ne, a.split, !a.batch && sweep_four(fp32, b), [&](auto k) { return cudaLaunchKernelEx(&cfg, k, a); });
}

cudaError_t strip_set_smem_limits(size_t max_smem) {
  auto set = [&](auto k) { return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)max_smem); };
  for (int fwd = 0; fwd < 2; ++fwd)
    for (int ne : {3, 4, 7, 16})
      for (int b = 1; b <= 3; ++b)
        for (int fp32 = 0; fp32 < 2; ++fp32)
          for (int form = 0; form <= (strip_can_split(b, fp32 ? 4 : 8) || sweep_four(fp32, b) ? 1 : 0); ++form) {
            const cudaError_t e = with_kernel(fp32, b, fwd, ne, form && !fp32, form && fp32, set);
            if (e != cudaSuccess) return e;
          }
  return cudaSuccess;
}

}  // namespace dfg
