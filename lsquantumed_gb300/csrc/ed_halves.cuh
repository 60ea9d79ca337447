// The basis as runs of rows: a state splits into its high half c1 and its low
// half c0 (the two-table rank), and the states of one c1 are one run of rows
// starting at T1[c1], in the order of the low halves of popcount nup -
// popc(c1).  Kernels that take a run per warp, or a column of the low halves
// per thread, share this geometry.
#pragma once
#include "ed_internal.h"
#include <cstring>

constexpr int CR_MAXW0 = 14;
constexpr int CR_CLASSES = CR_MAXW0 + 1;

// Low halves of one popcount and the high halves that go with them.
struct CorrGeom {
  int w0, w1, N;
  int nlow[CR_CLASSES], low_off[CR_CLASSES];    // low halves of popcount k: lows[low_off[k] ..]
  int nhigh[CR_CLASSES], high_off[CR_CLASSES];  // high halves of popcount nup - k
  int chunks[CR_CLASSES];                       // pieces of the low halves
  int prefix[CR_CLASSES + 1];                   // work items of the classes below k
};

// Classes of low halves with popcount k and the high halves of popcount
// nup - k; items of class k = chunks * per(k).
template <typename F>
static CorrGeom corr_geom(const ed_basis* b, int nup, int chunk, F per) {
  CorrGeom g;
  memset(&g, 0, sizeof(g));
  g.w0 = b->lin_w0;
  g.w1 = b->nspins - b->lin_w0;
  g.N = b->nspins;
  int lo = 0, n = 0;
  for (int k = 0; k < CR_CLASSES; ++k) {
    g.prefix[k] = n;
    if (k > g.w0) continue;
    g.nlow[k] = (int)ed_binom(g.w0, k);
    g.low_off[k] = lo;
    lo += g.nlow[k];
    const int h = nup - k;
    if (h >= 0 && h <= g.w1) {
      g.nhigh[k] = (int)ed_binom(g.w1, h);
      int ho = 0;
      for (int q = 0; q < h; ++q) ho += (int)ed_binom(g.w1, q);
      g.high_off[k] = ho;
      g.chunks[k] = (g.nlow[k] + chunk - 1) / chunk;
      n += g.chunks[k] * per(g.nhigh[k]);
    }
  }
  g.prefix[CR_CLASSES] = n;
  return g;
}
