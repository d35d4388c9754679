// Entry classes of a matrix's two strip plans: made each by itself, and for
// both directions together (strip_plan_both), whose padded plan is checked
// against the rows.
#include <algorithm>
#include <vector>

#include "../../delfem_gb300/csrc/k_strip.h"

using namespace dfg;

// ne: forward and backward alone, then together; returns 0, -1 (refused) or
// the number of the check that failed
extern "C" int emul_strip_pair(int n, int b, int elem, const int* rowptr, const int* colind, int split, int* ne) {
  std::vector<int> diaind(n);
  for (int i = 0; i < n; ++i) diaind[i] = (int)(std::lower_bound(colind + rowptr[i], colind + rowptr[i + 1], i) - colind);
  for (int dir = 0; dir < 2; ++dir) {
    StripPlan P;
    if (!strip_plan(n, b, elem, rowptr, colind, diaind.data(), dir == 0, split != 0, P)) return -1;
    ne[dir] = P.ne;
  }
  StripPlan P[2];
  if (!strip_plan_both(n, b, elem, rowptr, colind, diaind.data(), split != 0, P)) return -1;
  for (int dir = 0; dir < 2; ++dir) {
    const StripPlan& Q = P[dir];
    ne[2 + dir] = Q.ne;
    if (Q.forward != (dir == 0)) return 1;
    const StripDims d = strip_dims(b, elem, dir == 0, Q.ne, split != 0);
    if (d.RW != Q.d.RW || d.CH != Q.d.CH || d.step_bytes != Q.d.step_bytes) return 2;
    for (int i = 0; i < n; ++i) {
      const int c0 = dir == 0 ? rowptr[i] : diaind[i], c1 = dir == 0 ? diaind[i] : rowptr[i + 1];
      for (int e = 0; e < Q.ne; ++e) {
        const size_t at = (size_t)Q.pos[i] * Q.ne + e;
        if (Q.ent_slot[at] != (c0 + e < c1 ? c0 + e : -1)) return 3;
        if ((Q.codes[at] == 0) != (c0 + e >= c1)) return 4;  // padding reads the zero bytes
      }
    }
  }
  return 0;
}
