// Executes a strip sweep's plan (strip_plan, strip_meta) as k_strip.cu reads
// it, with row numbers in place of values: every reference of every step must
// find the row of its dependency, whether the receiver delivers items as late
// or as early as the kernel allows.
#include <vector>

#include "../../delfem_gb300/csrc/k_strip.h"

using namespace dfg;

// info: strips, steps, exchange slots, items; returns 0, or the number of the
// check that failed (-1: the rows do not fit the sweep)
extern "C" int emul_strip(int n, int b, int elem, const int* rowptr, const int* colind, int forward, int eager,
                          int split, long long* info) {
  std::vector<int> diaind(n);
  for (int i = 0; i < n; ++i) {
    int d = rowptr[i];
    while (d < rowptr[i + 1] && colind[d] < i) ++d;
    diaind[i] = d;
  }
  StripPlan P;
  if (!strip_plan(n, b, elem, rowptr, colind, diaind.data(), forward != 0, split != 0, P)) return -1;
  const StripDims& d = P.d;
  const int W = d.Q > 1 ? 1 : 3, NS = 2, lanes = 32 * d.Q;
  const int M = strip_mailbox(d.VS), ne = P.ne, iout = (ne + 1) / 2;
  if (d.CH * 4 > kStripHdr || strip_smem_bytes(d, W, NS) / 4 > 65536) return 1;
  if (d.chunk_bytes % 16 || d.CH * d.rhs_bytes % 16) return 2;
  std::vector<int> ident(n);
  for (int i = 0; i < n; ++i) ident[i] = i;
  const std::vector<int> meta = strip_meta(P, ident.data(), W, NS);
  std::vector<int> xch(P.nexport, -1), seen(n, 0);
  info[0] = P.nstrips; info[1] = 0; info[2] = P.nexport; info[3] = (long long)P.items.size() / 2;
  std::vector<int> region(strip_region_bytes(d) / 4);
  for (int r = 0; r < P.nstrips; ++r) {
    std::fill(region.begin(), region.end(), -2);
    for (int k = 0; k < kStripZero / 4; ++k) region[k] = -1;
    const int i0 = P.item_ptr[r], cnt = P.item_ptr[r + 1] - i0, s0 = P.strip_chunk[r] * d.CH;
    int delivered = 0, consumed = 0;
    auto deliver = [&](int upto) {  // as far as the exchange buffer and the flow control allow
      while (delivered < upto && delivered < cnt) {
        const int x = P.items[2 * (i0 + delivered)], free_at = P.items[2 * (i0 + delivered) + 1];
        if (free_at > consumed || xch[x] < 0) return;
        region[(kStripZero + kStripRing * d.RW * d.VS + (delivered % M) * d.VS) / 4] = xch[x];
        ++delivered;
      }
    };
    info[1] += P.strip_steps[r];
    for (int s = 0; s < P.strip_steps[r]; ++s) {
      deliver(eager ? cnt : P.need[s0 + s]);
      if (P.need[s0 + s] > delivered) return 3;  // would wait for ever
      std::vector<int> done_rows(d.RW, -1);
      for (int lane = 0; lane < lanes; ++lane) {
        auto get = [&](int i) { return meta[(((size_t)(s0 + s) * d.MC + i / 4) * lanes + lane) * 4 + (i & 3)]; };
        const int row = get(iout), l = strip_row(d, lane);
        if (row < 0) continue;
        if (l >= d.RW || P.pos[row] != (s0 + s) * d.RW + l) return 4;
        if (lane % 32 % d.LPR == 0 && seen[row]++) return 5;
        const int c0 = forward ? rowptr[row] : diaind[row], c1 = forward ? diaind[row] : rowptr[row + 1];
        for (int e = 0; e < ne; ++e) {
          const int cd = (int)((unsigned)get(e / 2) >> (16 * (e & 1)) & 0xffffu);
          const int at = cd - (int)strip_region_offset(d, W, NS, r % W) / 4;
          if (at < 0 || at >= (int)region.size() || region[at] != (c0 + e < c1 ? colind[c0 + e] : -1)) return 6;
          if (P.ent_slot[((size_t)(s0 + s) * d.RW + l) * ne + e] != (c0 + e < c1 ? c0 + e : -1)) return 7;
        }
        done_rows[l] = row;
        if (get(iout + 1) >= 0) xch[get(iout + 1)] = row;
      }
      for (int l = 0; l < d.RW; ++l) region[(kStripZero + ((s % kStripRing) * d.RW + l) * d.VS) / 4] = done_rows[l];
      if ((s + 1) % d.CH == 0) consumed = s + 1;
    }
    for (int q = s0; q < P.strip_chunk[r + 1] * d.CH; ++q)  // the end mark: after the last group of steps with rows
      if ((P.need[q] == kStripEnd) != (d.ends && (q - s0) / d.G * d.G >= P.strip_steps[r])) return 9;
  }
  for (int i = 0; i < n; ++i)
    if (seen[i] != 1) return 8;
  return 0;
}
