// Sizes of a chain pass (kernel_chain.cu: several consecutive factors of any shape contracted in shared
// memory in one launch), shared by the planner, which may only form groups that fit, and the launcher.
#pragma once

#include <stddef.h>
#include "fk_common.h"

namespace fkb {

constexpr int kChainThreads = 256;
constexpr unsigned kChainMaxQB = 8;                 // outputs of one column a thread accumulates at a time
constexpr size_t kChainSmem3 = 74 * 1024;           // three CTAs per SM
constexpr size_t kChainSmem2 = 112 * 1024;          // two
constexpr size_t kChainSmemMax = kChainSmem2;
// Resident CTAs of a tile of `smem` bytes: an SM has 228 KB, of which each takes 1 KB besides its own.
inline unsigned chainCtasPerSm(size_t smem) { const size_t n = 228 * 1024 / (smem + 1024); return n > 3 ? 3 : (unsigned)n; }

struct ChainShape {
  unsigned G, H;                                    // products of the P's and of the Q's
  unsigned W;                                       // columns (positions) per tile, a power of two times the vector
  unsigned pitch;                                   // elements between the rows of a tile
  unsigned qb[kMaxGroup], nb[kMaxGroup], fb[kMaxGroup];   // outputs per thread, blocks of them, padded row piece
  size_t offB, offF, offT, smem;                    // bytes: second buffer, factors, column tables, total
};

// False when the kernel does not take the group: its tile does not fit shared memory or the positions need more than 31
// bits.  The planner forms no other groups, and the launcher declines no other (a group has no kernel to fall back to).  `contig`: the group index is contiguous on the input or
// the output side (columns are then written and read across the tile's rows, which wants an odd pitch).
inline bool chainShape(DType dt, int nf, const uint32_t* P, const uint32_t* Q, bool contig, uint64_t total, int smCount, ChainShape* s) {
  if (total >= (1ull << 31)) return false;
  const size_t es = dtypeSize(dt);
  const unsigned vec = (unsigned)(16 / es);
  uint64_t cur = 1, most[2], h = 1;
  for (int k = 0; k < nf; k++) { cur *= P[k]; h *= Q[k]; if (cur > 65536 || h > 65536) return false; }
  s->G = (unsigned)cur; s->H = (unsigned)h;
  most[0] = cur; most[1] = 0;
  size_t f = 0;
  for (int k = nf - 1; k >= 0; k--) {
    cur = cur / P[k] * Q[k];
    if (cur > 65536) return false;
    uint64_t& m = most[(nf - k) & 1];
    if (cur > m) m = cur;
    s->nb[k] = (Q[k] + kChainMaxQB - 1) / kChainMaxQB;
    s->qb[k] = (Q[k] + s->nb[k] - 1) / s->nb[k];
    s->fb[k] = (s->qb[k] + vec - 1) / vec * vec;
    f += (size_t)P[k] * s->nb[k] * s->fb[k] * es;
  }
  auto size = [&](unsigned W) {
    s->W = W;
    s->pitch = contig && (W / vec) % 2 == 0 ? W + vec : W;
    s->offB = (size_t)most[0] * s->pitch * es;
    s->offF = s->offB + (size_t)most[1] * s->pitch * es;
    s->offT = (s->offF + f + 15) / 16 * 16;
    s->smem = s->offT + 2 * (size_t)W * sizeof(long long);
    return s->smem;
  };
  // the widest tile that leaves room for three CTAs per SM, else for two
  unsigned W = 0;
  for (unsigned w = 16 * vec; w >= vec && !W; w /= 2) if (size(w) <= kChainSmem3) W = w;
  for (unsigned w = 16 * vec; w >= vec && !W; w /= 2) if (size(w) <= kChainSmem2) W = w;
  if (!W) return false;
  // narrower while the grid would leave SMs idle
  while (W > vec && (total + W - 1) / W < 2 * (uint64_t)smCount) W /= 2;
  size(W);
  return true;
}

}  // namespace fkb
