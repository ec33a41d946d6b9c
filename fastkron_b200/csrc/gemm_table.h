// Which large-factor (GEMM-style) kernels exist; shared by the planner and the
// launcher.  One entry per (element type, P, Q); TJ is the tile width along the
// trailing index.
#pragma once

#include <stdint.h>
#include "fk_common.h"

namespace fkb {

inline int gemmTileJ(DType) { return 128; }

inline bool gemmShapeInTable(DType dt, uint32_t P, uint32_t Q) {
  if (dt == DType::F32) return (P == 64 && Q == 64) || (P == 128 && Q == 128);
  return P == 64 && Q == 64;
}

// B is the trailing extent of the dense row-major view [chunks][P][B].
inline bool gemmEligible(DType dt, uint32_t P, uint32_t Q, uint64_t B) {
  if (!gemmShapeInTable(dt, P, Q)) return false;
  const uint64_t vec = 16 / dtypeSize(dt), TJ = (uint64_t)gemmTileJ(dt);
  if (B == 1) return true;
  if (B % vec != 0) return false;
  return (B % TJ == 0) || (TJ % B == 0);
}

// The any-shape large-factor kernel (kernel_gemm_any.cu) takes every single-factor pass whose
// factor has at least 64 elements, and smaller factors from 5x5 on (measured on B200 against the
// one-thread-per-output kernel: 6x6 and 7x7 passes 1.8-1.9 times faster, 5x5 1.2 times, 3x3
// slower); what is left stays with the tile kernels or, for the few shapes those do not cover,
// with the one-thread-per-output kernel.  The measurement hook fkbSetAnyMinElems replaces the
// rule by "P*Q >= n" (process-wide; 0 restores the rule).
inline int gAnyMinElems = 0;
inline bool gemmAnyEligible(uint32_t P, uint32_t Q) {
  if (gAnyMinElems > 0) return (uint64_t)P * Q >= (uint64_t)gAnyMinElems;
  return (uint64_t)P * Q >= 64 || (P >= 5 && Q >= 5);
}

// The split tensor-core kernel (kernel_gemm_split.cu), fp32: factors up to 128 on either side; `total` is the
// number of positions (rows of the contraction).  Measured on B200, FMA kernels -> this one, 25 million elements, pass
// with p contiguous / with j contiguous: 36x36 182/158 -> 83/68 us, 64x64 85/84 -> 59/48, 100x100 229/207 -> 67/62; 48 -> 24 columns 51/27
// -> 48/25, about even, and 64 -> 17 loses (55/21 -> 67/17: the fixed work per tile is spread over few outputs).  Below 24x24 the FMA
// kernels are bound by memory themselves (24x24 three times, 256 rows: 58 us, 78 us here).  At 1024 positions (eight tiles) a
// launch takes 12.4 us on the FMA kernel and 13.7 here (64x64); fewer have never been faster here.  (These times are the
// six-product form's; the present one takes 1.05 to 1.3 times as long.  Between 24x24 and 36x36 the line is not measured.)
inline bool gemmSplitEligible(uint32_t P, uint32_t Q, uint64_t total) {
  return P >= 17 && Q >= 20 && P <= 128 && Q <= 128 && P * Q >= 1024 && total >= 1024 && total < (1ull << 31);
}

}  // namespace fkb
