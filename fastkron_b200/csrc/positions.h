// The positions (m, a, b) of a pass as one index, for the kernels that take arbitrary strides.
#pragma once

#include "fk_common.h"

namespace fkb {

// J = (i2*n1 + i1)*n0 + i0.  Element g of position J: input at sum i*xs + g*xsG, output likewise.
struct PosDim { uint64_t n; int64_t xs, zs; };

// Orders the three indices so that neighbouring positions are neighbours in memory on the side whose lanes
// run along the positions: the output unless its group index is contiguous, else the input.  Indices that are
// one dense index on both sides are merged; extents of 1 come last.
inline void orderPositions(const Pass& ps, PosDim (&d)[3]) {
  d[0] = {ps.B, ps.xsB, ps.zsB};
  d[1] = {ps.A, ps.xsA, ps.zsA};
  d[2] = {ps.M, ps.xsM, ps.zsM};
  for (int i = 1; i < 3; i++) {
    const bool lead = d[i].n > 1 && (ps.zsG != 1 ? d[i].zs == 1 : ps.xsG != 1 && d[i].xs == 1);
    if (lead) { const PosDim t = d[i]; for (int k = i; k > 0; k--) d[k] = d[k - 1]; d[0] = t; }
  }
  auto onesLast = [&] {
    for (int i = 0; i < 2; i++)
      for (int k = 0; k < 2; k++) if (d[k].n == 1) { const PosDim t = d[k]; d[k] = d[k + 1]; d[k + 1] = t; }
  };
  onesLast();
  // neighbours that are one dense index on both sides become one
  for (int i = 0; i < 2; i++)
    for (int k = 0; k < 2; k++)
      if (d[k + 1].n > 1 && d[k + 1].xs == (int64_t)d[k].n * d[k].xs && d[k + 1].zs == (int64_t)d[k].n * d[k].zs) {
        d[k].n *= d[k + 1].n;
        d[k + 1].n = 1;
        onesLast();
      }
}

// True when groups of `vec` neighbouring positions are contiguous (stride 1, never straddling an index) on the
// input (in) or output side and every other stride keeps a 16-byte aligned base aligned.
inline bool positionsVectorise(const PosDim (&d)[3], bool in, int64_t sG, int64_t vec) {
  auto s = [&](int i) { return in ? d[i].xs : d[i].zs; };
  return s(0) == 1 && d[0].n % vec == 0 && (d[1].n == 1 || s(1) % vec == 0) && (d[2].n == 1 || s(2) % vec == 0) && sG % vec == 0;
}

}  // namespace fkb
