// k_strip.h -- plan and launch interface of the strip sweeps (k_strip.cu,
// plans in strip.cpp).
#pragma once
#include <cuda_runtime.h>

#include <cstddef>
#include <vector>

namespace dfg {

// A strip is a set of rows that, grouped by their dependency level inside the
// strip, number at most RW per level, and whose other dependencies lie in
// earlier strips: up to RW consecutive grid lines of a structured 2D mesh, a
// tile of neighbouring lines of neighbouring planes of a 3D one.  One warp
// sweeps a strip, one level ("step") at a time.
//
// Shapes that follow from the block size, the element size, the direction and
// the entry class (entries per row: 3, 4, 7 or 16).
struct StripDims {
  bool split;  // a lane per element of a row's blocks
  int LPR;     // lanes per row: 1, b (lane = one component of a row) or b*b
  int Q;       // warps per strip
  int RW;      // rows per step
  int MC;      // 16-byte pieces of metadata per lane and step
  int VC;      // 16-byte pieces of factor values per lane and step
  int CH;      // steps per chunk (the unit copied into shared memory)
  int G;       // steps per test of the mailbox
  bool ends;   // the test also sees the strip's end (else the padding of its last chunk is swept)
  int VS;      // bytes of one row's value in the ring, the mailbox and the exchange buffer
  int step_bytes, rhs_bytes, chunk_bytes;
};
constexpr int kStripHdr = 32;    // bytes before a chunk's steps: CH counts of mailbox items needed
constexpr int kStripRing = 32;   // ring depth in steps
constexpr int kStripZero = 32;   // zero bytes at the start of a warp's value region (padding entries)
constexpr int kStripMaxWarps = 4;
constexpr int kStripEnd = 0x7fffffff;  // item count of steps after a strip's last: the strip is done

// Lanes per row.  An FP64 step costs 64 cycles of its scheduler per
// warp-wide FMA whatever the number of active lanes: there each component of a
// row takes its own lane, which divides the step's chain by b.  FP32 rows stay in
// one lane: more lanes per row would make steps shorter (3x3, 7 entries: 330
// cycles a level against 490) but strips smaller and hand-offs between them more, and
// those weigh more (elasticity on 56^3 cells 102 us per sweep with three lanes
// per row, 81 with one; on 24^3 37 and 34).  3x3 rows of more than 7 entries do
// not fit one lane's registers.
//
// split (2x2 and 3x3 FP64): each element of the blocks takes a lane, a row's sum being
// that of its columns' sums.  2x2 with 3 entries: 6 dependent operations a level
// instead of 8 (backward 4 instead of 6), for strips of 8 lines instead of 16: 2D
// elasticity on 200x100 cells 129 / 100 -> 116 / 83 us per sweep (forward /
// backward), 1000x500 594 / 479 -> 567 / 404, ILU(1) on 161x83 162 / 130 -> 135 /
// 100.  3x3 FP64 with 7 entries: 12 operations instead of 24 (9 instead of 21), by
// four warps, one per scheduler, that meet at a barrier after every step; 12 lines
// per strip instead of 10 (24^3 cells 98 / 90 -> 73 / 62 us).  The sums round differently from those of the other sweep kernels (their
// error against a wider type is no larger); the server, whose kernels give the
// same bits, does not split.
__host__ __device__ constexpr int strip_lpr(int b, int elem, int ne, bool split) {
  return split ? b * b : elem == 8 || (b == 3 && ne > 7) ? b : 1;
}
constexpr bool strip_can_split(int b, int elem) { return b >= 2 && elem == 8; }
// row of a step that lane t of the strip's 32 Q works on (RW: none)
__host__ __device__ constexpr int strip_row(const StripDims& d, int t) {
  const int per = 32 / d.LPR, l = t % 32 / d.LPR;
  return l < per ? t / 32 * per + l : d.RW;
}
__host__ __device__ constexpr StripDims strip_dims(int b, int elem, bool forward, int ne, bool split) {
  StripDims d{};
  d.split = split;
  d.LPR = strip_lpr(b, elem, ne, split);
  d.Q = split && b == 3 ? 4 : 1;
  d.RW = 32 / d.LPR * d.Q;
  d.MC = ((ne + 1) / 2 + 2 + 3) / 4;
  const int per_lane = (ne + (forward ? 1 : 0)) * (b * b / d.LPR);
  d.VC = (per_lane * elem + 15) / 16;
  d.VS = (b == 3 ? 4 : b) * elem;
  d.step_bytes = 512 * d.Q * (d.MC + d.VC);
  d.rhs_bytes = d.RW * b * elem;
  d.CH = d.step_bytes <= 2560 ? 8 : d.step_bytes <= 6144 ? 4 : 2;
  // short steps share a test (it is a branch, about 10 cycles, and waiting for
  // the last of four steps' items costs a hand-off three steps: 2x2 FP64, 200x100
  // cells, 133 us per sweep with four, 125 with one; 1x1 FP64, 128x128, 67 and 69)
  d.G = (elem == 4 || b == 1) && ne <= 4 && d.CH >= 4 ? 4 : 1;
  // the padding is up to 7 steps of 380 cycles in 1x1 FP64 (Poisson on 128x128 cells
  // 134 us per PCG iteration with it, 131 without); the other kinds' steps are
  // shorter, or fewer to a chunk, and the test costs them 1 to 3 % in every step
  d.ends = elem == 8 && d.G > 1;
  d.chunk_bytes = kStripHdr + d.CH * d.step_bytes;
  return d;
}
// entry class of rows with at most `maxe` entries; 0 = too many
inline int strip_class(int maxe) { return maxe <= 3 ? 3 : maxe <= 4 ? 4 : maxe <= 7 ? 7 : maxe <= 16 ? 16 : 0; }
// mailbox slots per warp: enough for the items of several chunks, 8-16 KB
__host__ __device__ constexpr int strip_mailbox(int VS) { return VS <= 8 ? 1024 : 512; }

// Steps are numbered with every strip padded to whole chunks: step s lies in
// chunk s / CH.  pos[row] = s * RW + row's place in the step is the row's
// place in the sweep's "step order", the order of its input.
struct StripPlan {
  bool forward = true;
  int n = 0, b = 1, elem = 8, ne = 0, nstrips = 0, nchunks = 0, nexport = 0;
  StripDims d{};
  std::vector<int> strip_chunk;  // nstrips + 1: first chunk
  std::vector<int> strip_steps;  // nstrips: steps that hold rows
  std::vector<int> item_ptr;     // nstrips + 1
  std::vector<int> items;        // per item {exchange slot, step at which its mailbox slot is free}
  std::vector<int> pos;          // n
  std::vector<int> need;         // nchunks * CH: mailbox items a step needs delivered, or kStripEnd
  std::vector<int> step_rows;    // nchunks * CH * RW, -1 = empty
  std::vector<int> ent_slot;     // nchunks * CH * RW * ne: CRS slot of the block, -1 = padding
  std::vector<int> codes;        // same shape: byte offset into the warp's value region
  std::vector<int> exports;      // nchunks * CH * RW: exchange slot of the row, -1 = none
  int levels = 0;                // dependency levels of the sweep
  long long chain = 0;           // its longest chain in steps, a hand-off between strips counted kStripHop
  long long steps() const { return (long long)nchunks * d.CH; }
};
__host__ __device__ constexpr size_t strip_up128(size_t v) { return (v + 127) / 128 * 128; }
// A warp's value region: zero bytes, ring, mailbox.
__host__ __device__ constexpr size_t strip_region_bytes(const StripDims& d) {
  return strip_up128(kStripZero + (size_t)kStripRing * d.RW * d.VS + (size_t)strip_mailbox(d.VS) * d.VS);
}
__host__ __device__ constexpr size_t strip_stage_bytes(const StripDims& d, int NS) {
  return strip_up128((size_t)NS * (d.chunk_bytes + d.CH * d.rhs_bytes) + 16);
}
// Shared memory: the chunk barriers and two progress words of every warp, then
// per warp its stages and its region.
__host__ __device__ constexpr size_t strip_stage_offset(const StripDims& d, int W, int NS, int w) {
  return strip_up128((size_t)W * NS * 8 + (size_t)W * 16) + w * (strip_stage_bytes(d, NS) + strip_region_bytes(d));
}
__host__ __device__ constexpr size_t strip_region_offset(const StripDims& d, int W, int NS, int w) {
  return strip_stage_offset(d, W, NS, w) + strip_stage_bytes(d, NS);
}
inline size_t strip_smem_bytes(const StripDims& d, int W, int NS) { return strip_stage_offset(d, W, NS, W); }
// Places for rows in the steps, per row.
inline double strip_fill(const StripPlan& P) { return (double)P.steps() * P.d.RW / P.n; }
// Whether the strips are those of a grid's numbering: few, or long and full ones
// (rows for two and a half steps or more in a strip, a row or more in every sixth
// place) whose chain is at most 10 times the levels'.  Grids row by row have chains
// of 1.0 to 2.7 times in 2D and up to 5.3 in 3D, with the boundary first or last up
// to 9.3 in 3D.  Where rows that follow one another lie far apart (numbered by
// distance from a point, by coordinate, at random, as an unstructured mesher does)
// strips hold a row or two per step or end after a few steps, and every step
// waits for other strips.
constexpr int kStripHop = 15;  // a hand-off between strips in steps (FP32, 1x1)
constexpr long long kStripChain = 10;
inline bool strip_like_grid(const StripPlan& P) {
  return P.nstrips <= 16 || (P.chain <= kStripChain * P.levels && 2LL * P.n >= 5LL * P.nstrips * P.d.RW &&
                             strip_fill(P) <= 6.0);
}
// Whether a plan is worth building at all.  Beside a grid's: records of up to 8 MB,
// or chains of up to 10 times the levels' with up to 16 places per row.  Beyond,
// records are tens of times the factor's bytes (an x-sorted Delaunay mesh of 100,000
// nodes: 76,000 strips, 1.3 GB of FP32 1x1 records for 1.2 MB of factor) and the
// sweeps slower than the older kinds (3,172 us per iteration, 1,135 with one CTA per
// sweep).
inline bool strip_suits(const StripPlan& P) {
  return strip_like_grid(P) || (size_t)P.nchunks * P.d.chunk_bytes <= (8u << 20) ||
         (P.chain <= kStripChain * P.levels && strip_fill(P) <= 16.0);
}
// Whether a plan that suits also serves a solve among many.  A strip keeps its CTA
// from its claim to its end, so a solve of many strips that wait for one another
// keeps the other solves out, whatever its own time.  Measured on GB300, 12 equal
// requests at once, FP32 factor, the older kinds -> strips: 20,000-node Delaunay
// meshes of jittered grid points 2D 1x1 (382 strips, rows for 1.6 steps each, fill
// 27) 87 -> 182 ms, 3D 1x1 (818, 0.8, 20) 154 -> 161; 2D sorted by coordinate
// (13,000, 0.05, 167) 127 -> 1,965; by reverse Cuthill-McKee (2,808, 0.2, 37) 109 ->
// 649; but 3D grids with the boundary first (48, 12.8, 2.9) 41 -> 33, and by reverse
// Cuthill-McKee at 4,000 nodes (143, 0.9, 16) 67 -> 13.
inline bool strip_serves(const StripPlan& P) {
  return strip_like_grid(P) || (P.chain <= kStripChain * P.levels &&
                                (P.nstrips <= 64 || (P.nstrips <= 160 && strip_fill(P) <= 16.0)));
}
// False when the rows do not fit the sweep: more than 16 entries in a row, more
// dependencies on other strips within a chunk than the mailbox holds, or (suited)
// a plan that does not suit.
// split: only where strip_can_split.  min_ne: an entry class that is not gone
// below (0, or one of strip_class's).
bool strip_plan(int n, int b, int elem, const int* rowptr, const int* colind, const int* diaind, bool forward,
                bool split, StripPlan& P, int min_ne = 0, bool suited = false);
// Both directions ([0] forward) in one entry class, that of the widest row of
// either.  By itself a direction takes the class of its own widest row, and in
// meshes whose numbering is not a grid's the two differ (a triangle grid with its
// boundary nodes numbered first: 7 lower entries, 3 upper ones).
bool strip_plan_both(int n, int b, int elem, const int* rowptr, const int* colind, const int* diaind, bool split,
                     StripPlan (&P)[2], bool suited = false);
// Metadata of every step and lane as the records hold it ([step][piece][lane]
// of 4 ints): ne 16-bit codes (offset / 4 from the start of the CTA's dynamic
// shared memory, for W warps of NS stages each), then the output position (-1:
// empty lane) and the exchange slot (-1: none).  out_pos[row]: where the row's
// result goes.
std::vector<int> strip_meta(const StripPlan& P, const int* out_pos, int W, int NS);

// A strip's chunk stages.  `consumed` counts the steps of the chunks that its
// warps are through with; the loader keeps the NS chunks from there on issued.
// Chunk c of the strip lies in stage c % NS, so a stage is issued again only
// when its copies have landed and been read.  A strip that has given up
// publishes nothing more: the chunks from `consumed` on that were issued are then
// those whose copies may be in flight, and the launch waits for them.
// (Conditions without a value to test: one more test per chunk on the compute warp's
// way cost 0.9 % of elasticity on 401x199 cells.)
__host__ __device__ constexpr bool strip_publishes(bool gave_up) { return !gave_up; }  // (chunk + 1) * CH steps
__host__ __device__ constexpr int strip_issue_end(int chunks_done, int NS, int nchunks) {
  return nchunks < chunks_done + NS ? nchunks : chunks_done + NS;
}
__host__ __device__ constexpr int strip_drain_begin(int consumed, int CH) { return consumed / CH; }

// One solve's sweep.
struct StripSlot {
  const unsigned char* rec;  // chunks
  const int* strip_chunk;
  const int* item_ptr;
  const int2* items;
  const void* in;            // right-hand sides in step order
  void* out;
  void* xch;                 // exchange buffer, sentinel-filled before the sweep
  const int* done;           // optional: nonzero = skip
  int nstrips;
};
// Several independent sweeps in one launch (the serving path): a ticket t
// names group t - group_start[j] (of W strips) of the slot j with
// group_start[j] <= t < group_start[j + 1]; finished solves' groups are
// skipped.
constexpr int kStripMaxSlots = 256;
struct StripBatch {
  int nslots;
  int group_start[kStripMaxSlots + 1];
  StripSlot slot[kStripMaxSlots];
};
struct StripArgs {
  StripSlot one;
  const StripBatch* batch;  // non-null: batched launch (`one` unused)
  // 0 when the launch can begin.  A launch that may begin before the kernel
  // ahead of it has ended (programmatic dependence) has it reset by an earlier
  // kernel: the backward sweep resets the forward one's (other_ticket), the
  // kernel after the backward sweep the backward one's.
  int* ticket;
  int* other_ticket;  // optional: set to 0
  int* err;      // device error word
  int ne;        // entry class
  bool split;    // StripDims
  int W;         // strips (compute warps) per CTA
  int NS;        // chunk stages per warp
};
cudaError_t launch_strip(bool forward, bool fp32, int b, const StripArgs& a, int grid, size_t smem, cudaStream_t st,
                         bool dep);
cudaError_t strip_set_smem_limits(size_t max_smem);
// places the metadata and the item counts into the records (once per plan)
cudaError_t launch_strip_meta(const StripDims& d, int nchunks, const int* meta, const int* need, unsigned char* rec,
                              cudaStream_t st);
// fills the records' values from the factor
struct StripPackArgs {
  StripDims d;
  int ne, b;
  long long nsteps;
  unsigned char* rec;
  const int* ent_slot;
  const int* step_rows;
  const double* fdiag;
  const double* foffd;
};
cudaError_t launch_strip_pack(bool forward, bool fp32, const StripPackArgs& a, cudaStream_t st);

}  // namespace dfg
