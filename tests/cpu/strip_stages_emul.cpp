// A strip's chunk stages when the strip gives up: the loader, the strip's first
// warp and the copies as k_strip.cu runs them, in an order drawn from `seed`.
#include <algorithm>
#include <random>
#include <vector>

#include "../../delfem_gb300/csrc/k_strip.h"

using namespace dfg;

// The first warp gives up before chunk `fail` (nch: never): it then walks the
// remaining chunks without waiting for their copies.  Returns 0, or 1: a stage
// was issued again with its copy in flight, 2: the launch ended with a copy in
// flight, 3: a strip that did not give up was not swept to its end.
extern "C" int emul_strip_stages(int nch, int CH, int NS, int fail, int slow, unsigned seed) {
  std::mt19937 rng(seed);
  std::vector<char> issued_at(NS, 0);  // copy in flight per stage
  std::vector<int> stage_chunk(NS, -1);
  int issued = 0, consumed = 0, c = 0;
  bool done = false;
  while (!done) {
    const unsigned what = rng() % (slow ? 8 : 3);
    if (what == 0) {  // loader
      for (const int done_chunks = consumed / CH; issued < strip_issue_end(done_chunks, NS, nch); ++issued) {
        if (issued_at[issued % NS]) return 1;
        issued_at[issued % NS] = 1;
        stage_chunk[issued % NS] = issued;
      }
    } else if (what == 1) {  // a copy lands
      issued_at[rng() % NS] = 0;
    } else if (what == 2 || c >= fail) {  // first warp: a chunk
      if (c < nch && (c >= fail || (stage_chunk[c % NS] == c && !issued_at[c % NS]))) {
        if (strip_publishes(c >= fail)) consumed = (c + 1) * CH;
        ++c;
      }
      done = c == nch;
    }
  }
  if (fail >= nch) return consumed == nch * CH ? 0 : 3;
  for (int k = strip_drain_begin(consumed, CH); k < issued; ++k) issued_at[k % NS] = 0;
  return std::count(issued_at.begin(), issued_at.end(), 1) ? 2 : 0;
}
