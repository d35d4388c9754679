// What the rules of k_strip.h say of a matrix's strip plans.
#include <algorithm>
#include <vector>

#include "../../delfem_gb300/csrc/k_strip.h"

using namespace dfg;

// Bits: 1 a grid's strips (strip_like_grid), 2 they suit (strip_suits) and serve
// (strip_serves); refused: -1 before the tables, -2 by the mailbox's limit
extern "C" int emul_strip_choice(int n, int b, int elem, const int* rowptr, const int* colind, int forward,
                                 int split, int suited, long long* chain) {
  std::vector<int> diaind(n);
  for (int i = 0; i < n; ++i) diaind[i] = (int)(std::lower_bound(colind + rowptr[i], colind + rowptr[i + 1], i) - colind);
  StripPlan P;
  if (!strip_plan(n, b, elem, rowptr, colind, diaind.data(), forward != 0, split != 0, P, 0, suited != 0))
    return P.pos.empty() ? -1 : -2;
  // the chain again, strip after strip, from the plan's places
  std::vector<long long> end((size_t)P.steps(), 0);
  chain[0] = P.chain;
  chain[1] = 0;
  for (int r = 0; r < P.nstrips; ++r) {
    long long before = 0;
    for (int s = P.strip_chunk[r] * P.d.CH, k = 0; k < P.strip_steps[r]; ++k, ++s) {
      long long t = before;
      for (int l = 0; l < P.d.RW; ++l) {
        const int row = P.step_rows[(size_t)s * P.d.RW + l];
        if (row < 0) continue;
        for (int c = forward ? rowptr[row] : diaind[row]; c < (forward ? diaind[row] : rowptr[row + 1]); ++c) {
          const int of = P.pos[colind[c]] / P.d.RW;
          if (of < P.strip_chunk[r] * P.d.CH) t = std::max(t, end[of] + kStripHop);
        }
      }
      before = end[s] = t + 1;
      chain[1] = std::max(chain[1], before);
    }
  }
  return (strip_like_grid(P) ? 1 : 0) | (strip_suits(P) && strip_serves(P) ? 2 : 0);
}
