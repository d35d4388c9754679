// strip.cpp -- host-side plans of the strip sweeps (k_strip.cu): rows into
// strips and steps, dependencies into ring and mailbox references.
#include <algorithm>
#include <cstring>

#include "k_strip.h"

namespace dfg {

bool strip_plan(int n, int b, int elem, const int* rowptr, const int* colind, const int* diaind, bool forward,
                StripPlan& P) {
  P = StripPlan{};
  P.forward = forward;
  P.n = n;
  P.b = b;
  P.elem = elem;
  auto row_of = [&](int p) { return forward ? p : n - 1 - p; };
  auto first = [&](int row) { return forward ? rowptr[row] : diaind[row]; };
  auto end = [&](int row) { return forward ? diaind[row] : rowptr[row + 1]; };
  int maxe = 0;
  for (int i = 0; i < n; ++i) maxe = std::max(maxe, end(i) - first(i));
  P.ne = strip_class(maxe);
  if (n == 0 || P.ne == 0) return false;
  P.d = strip_dims(b, elem, forward, P.ne);
  const int RW = P.d.RW, CH = P.d.CH, ne = P.ne;

  // strips: rows in order, each at its dependency level inside the strip.  The
  // row that would be the RW+1st of a level starts the next strip (in a
  // structured mesh the first row of grid line RW+1), and so does a row whose
  // level in the whole sweep says that it could run much earlier or only much
  // later than the rows it would share a step with: the first row of the next
  // plane of a 3D mesh, which would otherwise wait for the last lines of this
  // one, plane after plane.
  constexpr int kDrift = 4;
  std::vector<int> lev(n), lane(n), strip(n), cnt, glev(n);
  for (int p = 0; p < n; ++p) {
    const int row = row_of(p);
    int lv = 0;
    for (int c = first(row); c < end(row); ++c) lv = std::max(lv, glev[colind[c]] + 1);
    glev[row] = lv;
  }
  P.strip_chunk.push_back(0);
  for (int p = 0; p < n;) {
    const int p0 = p;
    cnt.clear();
    for (; p < n; ++p) {
      const int row = row_of(p);
      int lv = 0;
      for (int c = first(row); c < end(row); ++c) {
        const int k = colind[c];
        if ((forward ? k : n - 1 - k) >= p0) lv = std::max(lv, lev[k] + 1);
      }
      const int drift = glev[row] - lv - glev[row_of(p0)];
      if (drift > kDrift || drift < -kDrift) break;
      if (lv >= (int)cnt.size()) cnt.resize(lv + 1, 0);
      if (cnt[lv] == RW) break;
      lev[row] = lv;
      lane[row] = cnt[lv]++;
      strip[row] = P.nstrips;
    }
    // a level opened by the row that broke the strip is empty: drop it
    while (!cnt.empty() && cnt.back() == 0) cnt.pop_back();
    P.strip_steps.push_back((int)cnt.size());
    P.strip_chunk.push_back(P.strip_chunk.back() + ((int)cnt.size() + CH - 1) / CH);
    ++P.nstrips;
  }
  P.nchunks = P.strip_chunk.back();
  const size_t nsteps = (size_t)P.steps();
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
        for (int c = first(row); c < end(row); ++c) {
          const int k = colind[c];
          const size_t e = at * ne + (c - first(row));
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
  }
  for (int row = 0; row < n; ++row)
    if (xslot[row] >= 0) P.exports[P.pos[row]] = xslot[row];
  return true;
}

std::vector<int> strip_meta(const StripPlan& P, const int* out_pos, int W, int NS) {
  const int RW = P.d.RW, LPR = P.d.LPR, MC = P.d.MC, ne = P.ne;
  const size_t nsteps = (size_t)P.steps();
  std::vector<int> m(nsteps * MC * 128, 0);
  const int iout = (ne + 1) / 2;
  int strip = 0;
  for (size_t s = 0; s < nsteps; ++s) {
    while ((long long)P.strip_chunk[strip + 1] * P.d.CH <= (long long)s) ++strip;
    const unsigned region = (unsigned)strip_region_offset(P.d, W, NS, strip % W);
    for (int lane = 0; lane < 32; ++lane) {
      auto put = [&](int i) -> int& { return m[((s * MC + i / 4) * 32 + lane) * 4 + (i & 3)]; };
      const int l = lane / LPR;
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
