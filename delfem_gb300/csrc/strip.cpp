// strip.cpp -- host-side plans of the strip sweeps (k_strip.cu): rows into
// strips and steps, dependencies into ring and mailbox references.
#include <algorithm>
#include <cstdlib>

#include "k_strip.h"

namespace dfg {

namespace {

// The rows of a sweep: position p of the sweep order is row p forward, row
// n-1-p backward; a row's entries point to earlier positions.
struct Rows {
  int n;
  bool forward;
  const int *rowptr, *colind, *diaind;
  const int* glev;  // dependency level in the whole sweep
  int row(int p) const { return forward ? p : n - 1 - p; }
  int pos(int row) const { return forward ? row : n - 1 - row; }
  int first(int row) const { return forward ? rowptr[row] : diaind[row]; }
  int end(int row) const { return forward ? diaind[row] : rowptr[row + 1]; }
};

// Rows share a step by their level inside the strip.  A row whose level in the
// whole sweep says that it could run this much earlier, or only this much
// later, than the rows it would share a step with does not join them.
constexpr int kDrift = 4;

// Strips of consecutive rows: the row that would be the RW+1st of a level
// starts the next strip (in a structured mesh the first row of grid line
// RW+1), and so does a row that has drifted.
void run_strips(const Rows& R, int RW, std::vector<int>& strip, std::vector<int>& lev, std::vector<int>& lane,
                std::vector<int>& steps) {
  steps.clear();
  std::vector<int> cnt;
  for (int p = 0; p < R.n;) {
    const int p0 = p, g0 = R.glev[R.row(p0)];
    cnt.clear();
    for (; p < R.n; ++p) {
      const int row = R.row(p);
      int lv = 0;
      for (int c = R.first(row); c < R.end(row); ++c)
        if (R.pos(R.colind[c]) >= p0) lv = std::max(lv, lev[R.colind[c]] + 1);
      const int drift = R.glev[row] - lv - g0;
      if (drift > kDrift || drift < -kDrift) break;
      if (lv < (int)cnt.size() && cnt[lv] == RW) break;
      if (lv >= (int)cnt.size()) cnt.resize(lv + 1, 0);
      lev[row] = lv;
      lane[row] = cnt[lv]++;
      strip[row] = (int)steps.size();
    }
    steps.push_back((int)cnt.size());
  }
}

// Strips that are tiles of grid lines: by neighbouring lines of bz
// neighbouring planes, by * bz <= RW.  A plane of a 3D mesh handed on plane by
// plane costs a hand-off per plane; with tiles a dependency chain changes
// strips once per bz planes and once per by lines.  Lines and planes are read
// off the dependencies: a row that does not depend on the row before it starts
// a line, a line none of whose rows depends on the line before it starts a
// plane.  False when there are no planes, when tiles would not cut the
// hand-offs, or when some dependency does not respect the tiles' order.
bool tile_strips(const Rows& R, int RW, std::vector<int>& strip, std::vector<int>& lev, std::vector<int>& lane,
                 std::vector<int>& steps) {
  const int n = R.n;
  std::vector<int> line(n), plane, y;  // line of a position; plane and place in it of a line
  int nl = 0;
  bool linked = false;  // the current line depends on the line before it
  auto close_line = [&] {
    if (plane.empty() || !linked) {
      plane.push_back(plane.empty() ? 0 : plane.back() + 1);
      y.push_back(0);
    } else {
      plane.push_back(plane.back());
      y.push_back(y.back() + 1);
    }
    linked = false;
  };
  for (int p = 0; p < n; ++p) {
    const int row = R.row(p);
    bool next = p > 0;
    for (int c = R.first(row); c < R.end(row); ++c) next &= R.pos(R.colind[c]) != p - 1;
    if (next) {
      close_line();
      ++nl;
    }
    line[p] = nl;
    for (int c = R.first(row); c < R.end(row); ++c) linked |= line[R.pos(R.colind[c])] == nl - 1;
  }
  close_line();
  ++nl;
  const int nz = plane.back() + 1;
  int ny = 0;
  for (int l = 0; l < nl; ++l) ny = std::max(ny, y[l] + 1);
  if (nz < 2 || ny < 2) return false;
  int by = 1, bz = 1, hops = ny + nz;
  for (int a = 1; a <= std::min(RW, ny); ++a) {
    const int c = std::min(RW / a, nz), h = (ny + a - 1) / a + (nz + c - 1) / c;
    if (h < hops || (h == hops && std::abs(a - c) < std::abs(by - bz))) { by = a; bz = c; hops = h; }
  }
  if (hops >= nz + (ny + RW - 1) / RW) return false;
  const int ty = (ny + by - 1) / by, nt = ty * ((nz + bz - 1) / bz);
  std::vector<std::vector<int>> cnt(nt);
  std::vector<int> g0(nt, -1);
  for (int p = 0; p < n; ++p) {
    const int row = R.row(p), t = plane[line[p]] / bz * ty + y[line[p]] / by;
    int lv = 0;
    for (int c = R.first(row); c < R.end(row); ++c) {
      const int k = R.colind[c];
      if (strip[k] > t) return false;
      if (strip[k] == t) lv = std::max(lv, lev[k] + 1);
    }
    if (g0[t] < 0) g0[t] = R.glev[row];
    const int drift = R.glev[row] - lv - g0[t];
    if (drift > kDrift || drift < -kDrift) return false;
    if (lv >= (int)cnt[t].size()) cnt[t].resize(lv + 1, 0);
    if (cnt[t][lv] == RW) return false;
    lev[row] = lv;
    lane[row] = cnt[t][lv]++;
    strip[row] = t;
  }
  // tiles without rows (the last planes may be short) are dropped
  std::vector<int> id(nt, -1);
  steps.clear();
  for (int t = 0; t < nt; ++t)
    if (!cnt[t].empty()) {
      id[t] = (int)steps.size();
      steps.push_back((int)cnt[t].size());
    }
  for (int i = 0; i < n; ++i) strip[i] = id[strip[i]];
  return true;
}

// The longest chain of steps: a step follows the one before it in its strip and,
// a hand-off later, those of other strips that its rows depend on.
long long longest_chain(const Rows& R, const std::vector<int>& strip, const std::vector<int>& lev,
                        const std::vector<int>& steps) {
  const int nstrips = (int)steps.size();
  if (nstrips == 1) return steps[0];
  std::vector<int> first(nstrips + 1, 0);  // a strip's first step
  for (int r = 0; r < nstrips; ++r) first[r + 1] = first[r] + steps[r];
  std::vector<int> ptr(first[nstrips] + 1, 0), rows(R.n);  // rows by step
  for (int i = 0; i < R.n; ++i) ++ptr[first[strip[i]] + lev[i]];
  for (int s = 0; s < first[nstrips]; ++s) ptr[s + 1] += ptr[s];
  for (int i = R.n - 1; i >= 0; --i) rows[--ptr[first[strip[i]] + lev[i]]] = i;
  std::vector<long long> t(first[nstrips]);
  long long most = 0;
  for (int r = 0; r < nstrips; ++r)
    for (int s = first[r]; s < first[r + 1]; ++s) {
      long long v = s > first[r] ? t[s - 1] : 0;
      for (int p = ptr[s]; p < ptr[s + 1]; ++p)
        for (int c = R.first(rows[p]); c < R.end(rows[p]); ++c) {
          const int k = R.colind[c];
          if (strip[k] != r) v = std::max(v, t[first[strip[k]] + lev[k]] + kStripHop);
        }
      t[s] = v + 1;
      most = std::max(most, t[s]);
    }
  return most;
}

}  // namespace

bool strip_plan(int n, int b, int elem, const int* rowptr, const int* colind, const int* diaind, bool forward, bool split,
                StripPlan& P, int min_ne, bool suited) {
  P = StripPlan{};
  P.forward = forward;
  P.n = n;
  P.b = b;
  P.elem = elem;
  auto row_of = [&](int p) { return forward ? p : n - 1 - p; };
  auto first_entry = [&](int row) { return forward ? rowptr[row] : diaind[row]; };
  auto end = [&](int row) { return forward ? diaind[row] : rowptr[row + 1]; };
  int maxe = 0;
  for (int i = 0; i < n; ++i) maxe = std::max(maxe, end(i) - first_entry(i));
  P.ne = strip_class(maxe);
  if (n == 0 || P.ne == 0) return false;
  P.ne = std::max(P.ne, min_ne);
  P.d = strip_dims(b, elem, forward, P.ne, split);
  const int RW = P.d.RW, CH = P.d.CH, ne = P.ne;

  // level of every row in the whole sweep
  std::vector<int> glev(n), lev(n), lane(n), strip(n);
  for (int p = 0; p < n; ++p) {
    const int row = row_of(p);
    int lv = 0;
    for (int c = first_entry(row); c < end(row); ++c) lv = std::max(lv, glev[colind[c]] + 1);
    glev[row] = lv;
  }
  const Rows R{n, forward, rowptr, colind, diaind, glev.data()};
  std::vector<int> steps;
  if (!tile_strips(R, RW, strip, lev, lane, steps)) run_strips(R, RW, strip, lev, lane, steps);
  P.nstrips = (int)steps.size();
  P.strip_steps = steps;
  P.strip_chunk.push_back(0);
  for (int r = 0; r < P.nstrips; ++r) P.strip_chunk.push_back(P.strip_chunk.back() + (steps[r] + CH - 1) / CH);
  P.nchunks = P.strip_chunk.back();
  const size_t nsteps = (size_t)P.steps();
  if ((double)nsteps * RW * b > 2147483647.0) return false;  // places are int
  P.levels = *std::max_element(glev.begin(), glev.end()) + 1;
  P.chain = longest_chain(R, strip, lev, steps);
  if (suited && !strip_suits(P)) return false;
  P.pos.resize(n);
  P.step_rows.assign(nsteps * RW, -1);
  for (int row = 0; row < n; ++row) {
    P.pos[row] = (P.strip_chunk[strip[row]] * CH + lev[row]) * RW + lane[row];
    P.step_rows[P.pos[row]] = row;
  }
  // references: a dependency finished by the same strip within the last
  // kStripRing steps is read from the ring; any other one is an item of the
  // strip's mailbox, listed in the order of first use.  Item k occupies slot
  // k mod M; an item whose slot was taken over since is listed again.  The
  // receiver may fill slot k mod M once the warp has finished the chunk of
  // the last step that uses item k - M.
  const int M = strip_mailbox(P.d.VS);
  P.need.assign(nsteps, 0);
  P.ent_slot.assign(nsteps * RW * ne, -1);
  P.codes.assign(nsteps * RW * ne, 0);
  P.exports.assign(nsteps * RW, -1);
  P.item_ptr.assign(1, 0);
  std::vector<int> xslot(n, -1), item_of(n, -1), item_strip(n, -1), last_use;
  const int ring0 = kStripZero, mail0 = kStripZero + kStripRing * RW * P.d.VS;
  for (int r = 0; r < P.nstrips; ++r) {
    const int s0 = P.strip_chunk[r] * CH;
    last_use.clear();
    for (int s = 0; s < P.strip_steps[r]; ++s) {
      for (int l = 0; l < RW; ++l) {
        const size_t at = (size_t)(s0 + s) * RW + l;
        const int row = P.step_rows[at];
        if (row < 0) continue;
        for (int c = first_entry(row); c < end(row); ++c) {
          const int k = colind[c];
          const size_t e = at * ne + (c - first_entry(row));
          P.ent_slot[e] = c;
          if (strip[k] == r && s - lev[k] < kStripRing) {
            P.codes[e] = ring0 + ((lev[k] % kStripRing) * RW + lane[k]) * P.d.VS;
            continue;
          }
          int it = item_strip[k] == r ? item_of[k] : -1;
          if (it < 0 || (int)last_use.size() > it + M) {  // not listed, or item it + M has its slot
            it = (int)last_use.size();
            const int free_at = it >= M ? last_use[it - M] + 1 : 0;
            if (free_at > s / CH * CH) return false;
            item_of[k] = it;
            item_strip[k] = r;
            last_use.push_back(s);
            if (xslot[k] < 0) xslot[k] = P.nexport++;
            P.items.push_back(xslot[k]);
            P.items.push_back(free_at);
          }
          last_use[it] = s;
          const int c0 = s0 + s / CH * CH;  // a step's count covers the steps of its chunk before it
          for (int q = s0 + s; q < c0 + CH; ++q) P.need[q] = std::max(P.need[q], it + 1);
          P.codes[e] = mail0 + (it % M) * P.d.VS;
        }
      }
    }
    P.item_ptr.push_back((int)(P.items.size() / 2));
    // (steps of a test's group that has rows keep their counts)
    for (int q = s0 + (P.strip_steps[r] + P.d.G - 1) / P.d.G * P.d.G; P.d.ends && q < P.strip_chunk[r + 1] * CH; ++q)
      P.need[q] = kStripEnd;
  }
  for (int row = 0; row < n; ++row)
    if (xslot[row] >= 0) P.exports[P.pos[row]] = xslot[row];
  return true;
}

bool strip_plan_both(int n, int b, int elem, const int* rowptr, const int* colind, const int* diaind, bool split,
                     StripPlan (&P)[2], bool suited) {
  int maxe = 0;
  for (int i = 0; i < n; ++i) maxe = std::max({maxe, diaind[i] - rowptr[i], rowptr[i + 1] - diaind[i]});
  const int ne = strip_class(maxe);
  if (ne == 0) return false;
  for (int dir = 0; dir < 2; ++dir)
    if (!strip_plan(n, b, elem, rowptr, colind, diaind, dir == 0, split, P[dir], ne, suited)) return false;
  return true;
}

std::vector<int> strip_meta(const StripPlan& P, const int* out_pos, int W, int NS) {
  const int RW = P.d.RW, MC = P.d.MC, ne = P.ne, lanes = 32 * P.d.Q;
  const size_t nsteps = (size_t)P.steps();
  std::vector<int> m(nsteps * MC * lanes * 4, 0);
  const int iout = (ne + 1) / 2;
  int strip = 0;
  for (size_t s = 0; s < nsteps; ++s) {
    while ((long long)P.strip_chunk[strip + 1] * P.d.CH <= (long long)s) ++strip;
    const unsigned region = (unsigned)strip_region_offset(P.d, W, NS, strip % W);
    for (int lane = 0; lane < lanes; ++lane) {
      auto put = [&](int i) -> int& { return m[((s * MC + i / 4) * lanes + lane) * 4 + (i & 3)]; };
      const int l = strip_row(P.d, lane);
      const size_t at = s * RW + l;
      const int row = l < RW ? P.step_rows[at] : -1;
      put(iout) = row >= 0 ? out_pos[row] : -1;
      put(iout + 1) = row >= 0 ? P.exports[at] : -1;
      for (int e = 0; e < ne; ++e)
        put(e / 2) |= (int)((region + (row >= 0 ? (unsigned)P.codes[at * ne + e] : 0u)) / 4 << (16 * (e & 1)));
    }
  }
  return m;
}

}  // namespace dfg
