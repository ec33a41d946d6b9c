// Large-factor pass of fp32 operands on the tensor cores with fp32 results.  Every operand is split into three bf16
// numbers, v = h + m + l with 6, 8 and the remaining bits, which hold all 24 of a float, and the eight products of pieces
// down to m*l and l*m are accumulated by tcgen05.mma (l*l, below 2^-30 of the product, is left out).
//
// The tensor cores cut every addend off two bits below the accumulator and every sum at 24 bits, both toward zero, so a sum
// of one sign loses on average half a unit in the last place per step, always in the same direction and adding up over the
// factors of a call.  Three things keep that out of the results:
//   h has 6 bits only: products of two have 12, and a few of them add up without anything to cut off;
//   h*h is summed in accumulators of 32 products each, which the epilogue adds with rounding to nearest;
//   the other seven products, at most 2^-5 of the whole together, have an accumulator of their own, added last.
// Error against 64-bit arithmetic (relative 2-norm, B200) of the FMA kernels and here: 64x64 twice 2.0e-7 and 4.2e-8 on values
// in [-1, 1), 1.15e-7 and 3.1e-8 on [0, 1); 127x127 twice 2.9e-7 and 5.1e-8, 1.6e-7 and 3.7e-8.  It is larger than theirs only where
// products of one sign spread over many magnitudes (lognormal values with sigma 2 and more, 1.0 to 3.7 times): the bits of
// the small ones beside the large are still cut.
//
// One pass is  Z[j][q] = sum_p X[j][p] * F[p][q]  over the J = M*A*B positions (m, a, b) of the pass,
// any strides, any P and Q up to 128, any alignment.  A tile is 128 positions times all of Q, in blocks of 64 columns:
//   D[128 x 64] (TMEM, fp32) += A[128 x P] (TMEM, bf16) * B[P x 64] (shared memory, bf16),  tcgen05.mma.kind::f16.
// Why A sits in TMEM: the positions come with j contiguous (B > 1) or p contiguous (B == 1), at any
// alignment.  A converter thread owns one position: it reads its P values from shared memory, splits them in
// registers and writes them to its TMEM lane with tcgen05.st.  The transposition that the j-contiguous
// operand needs happens on that way for nothing, and the tensor cores read X without touching shared
// memory (with the three copies there, operand reads alone would take as long as the HBM transfer).
//
// Warp roles (672 threads, one CTA per SM, persistent):
//   0-7   epilogue: tcgen05.ld of the accumulators (a lane quarter each, alternate groups of 32 columns), their sum,
//         alpha / beta*Y, stores
//   8-19  converters.  Three warps share 32 positions and take the chunks of 16 p, tile after tile, in turns; each loads its
//         chunks with cp.async into a private ring of stages, so between load and conversion there is no barrier, only a
//         __syncwarp
//   20    MMA issue and the TMEM allocation.  The whole warp walks the loop (its values then stay in uniform
//         registers, where the instruction wants them) and one elected lane issues
// A is handed over chunk by chunk: the MMAs of a chunk, all eight products, follow its conversion, and its place in
// TMEM is free again when they are done.  Accumulators are two rings, h*h and the rest.
// Every wait on a barrier is bounded; one that gives up raises the abort flag that ends all roles.  21 warps leave 80 registers a
// thread, the fewest with which nothing is spilled (25 warps: 72, and with all of the SM's memory taken as shared memory
// a spilled register comes back from L2: 64x64 four times, 64 rows, 9.3 ms against 8.5).
//
// Bound by issue slots (60 % busy) and by the hand-overs between the roles.  The contraction length is a template parameter
// because the MMAs are issued by one lane: with run-time descriptors a 128x64x16 MMA took 126-152 clocks.
//
// Operands a bf16 split cannot hold are found while splitting: elements with a remainder after the third piece
// (infinities, NaN, and numbers below about 2^-110 whose last bits lie under the smallest bf16 denormal 2^-133; the
// tensor cores take and give denormals in full), and magnitudes from 2^127 or whose sums could overflow.  A row with such
// an element, or every row when the factor has one, takes the FMA chain over p instead, the numbers of the FMA kernels: the
// epilogue leaves it out and marks the tile, and after the last tile the whole CTA contracts the marked ones from shared memory.
#include <stdlib.h>

#include <cuda_bf16.h>

#include "kernels.h"
#include "gemm_table.h"
#include "positions.h"
#include "tcgen05.cuh"

namespace fkb {
namespace tc {

constexpr int kSplitEpiWarps = 8, kSplitConvWarps = 12, kSplitSubs = kSplitConvWarps / 4;
constexpr int kSplitMmaWarp = kSplitEpiWarps + kSplitConvWarps;
constexpr int kSplitThreads = 32 * (kSplitMmaWarp + 1);
constexpr int kSplitRows = 128;
constexpr int kSplitChunk = 16;                    // p per stage: a stage is 32 positions x 16 p of one converter warp
constexpr int kSplitStageElems = 32 * kSplitChunk;
constexpr int kSplitMaxStages = 8;
constexpr int kSplitSmem = (227 - 3) * 1024;         // dynamic shared memory; the static part is below 3 KB
constexpr int kXposePitch = 36;                    // 32 columns and an odd number of 16-byte units per row
constexpr size_t kXposeBytes = kSplitEpiWarps * 32 * kXposePitch * sizeof(float);
constexpr unsigned kBlockN = 64;                   // columns of an accumulator: wider results go in blocks of 64
constexpr unsigned kTileBits = 2048;               // marks of tiles with rows for the FMA chain; tiles that share one are looked at
constexpr unsigned kFmaChunk = 16, kFmaPitch = kSplitRows + 4;   // p per stage of the FMA chain, elements between them
constexpr unsigned kOutPitch = kBlockN + 4;        // elements between the rows of its result
constexpr unsigned kFmaThreads = 512, kLoadX = kFmaChunk * kSplitRows / kFmaThreads, kLoadF = kFmaChunk * kBlockN / kFmaThreads;
static_assert(kFmaChunk * (kFmaPitch + kBlockN) <= kSplitRows * kOutPitch && kFmaThreads <= kSplitThreads, "the result takes the place of a stage");
// Steps of 16 products of h*h that share an accumulator.  With four, smooth one-signed factors (exp(-|i-j|/3)) err more than in
// the FMA chain (3.7e-7 against 1.7e-7, 64x64 twice); with one the epilogue reads twice as many (64x64: 10.0 ms against 8.9).
constexpr unsigned kHhSteps = 2;
// A buffers: from P = 81 on the accumulators leave room for one.
__host__ __device__ constexpr unsigned aBuffers(unsigned ks) { return ks > 5 ? 1 : 2; }
constexpr unsigned kMaxSlots = 8;                  // accumulators
constexpr unsigned kHuge = 254u << 23;             // 2^127 as float bits

// n / d for n < 2^31:  n * ceil(2^(31+l) / d) >> (31 + l), l = ceil(log2 d); the factor fits 32 bits (m == 0: d is 1).
struct PosDiv { unsigned d, m, s; };
static PosDiv posDiv(unsigned d) {
  unsigned l = 0;
  while ((1ull << l) < d) l++;
  if (l == 0) return PosDiv{1, 0, 0};
  return PosDiv{d, (unsigned)(((1ull << (31 + l)) + d - 1) / d), l - 1};
}
__device__ __forceinline__ unsigned quot(unsigned n, const PosDiv& f) { return f.m == 0 ? n : __umulhi(n, f.m) >> f.s; }

struct SplitArgs {
  const float* X; float* Z; const float* Y; const float* F;
  long long fsP, fsQ;
  unsigned P, Q;
  unsigned N;                                      // Q rounded up to 16
  unsigned stages;                                 // per converter warp, 1 .. kSplitMaxStages
  unsigned slotCols, sSlots, slots;                // TMEM columns of an accumulator; 0 .. sSlots-1 take small terms, sSlots .. slots-1 h*h, each a ring
  // position J = (i2*n1 + i1)*n0 + i0; element (J, p) of X at sum i*xs + p*xsP, (J, q) of Z and Y at sum i*zs + q*zsQ
  PosDiv n0, n1;
  unsigned xs0, xs1, xs2, zs0, zs1, zs2;           // elements
  long long xsP, zsQ;
  unsigned total, numTiles;
  float alpha, beta;
  int epilogue;
  int vecX;                                        // 16-byte loads allowed
  int outT, vecZ;                                  // the output is contiguous along q; 16-byte stores along it
};

// Shared memory by its 32-bit address: two registers fewer per pointer, and none may be spilled here (with
// all of the SM's memory taken as shared memory, a spilled register comes back from L2).
// valid == false: nothing is read, the destination is zero-filled.
template <int BYTES>
__device__ __forceinline__ void cpAsyncFill(unsigned dst, const float* src, bool valid) {
  const int n = valid ? BYTES : 0;
  if (BYTES == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(n) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(dst), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ float ldShared(unsigned a) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];\n" : "=f"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ float4 ldShared4(unsigned a) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];\n" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
  return v;
}
// all but the newest `n` groups of this thread are complete
__device__ __forceinline__ void cpAsyncWaitUpTo(unsigned n) {
  switch (n) {
    case 0: asm volatile("cp.async.wait_group 0;\n" ::: "memory"); break;
    case 1: asm volatile("cp.async.wait_group 1;\n" ::: "memory"); break;
    case 2: asm volatile("cp.async.wait_group 2;\n" ::: "memory"); break;
    case 3: asm volatile("cp.async.wait_group 3;\n" ::: "memory"); break;
    case 4: asm volatile("cp.async.wait_group 4;\n" ::: "memory"); break;
    case 5: asm volatile("cp.async.wait_group 5;\n" ::: "memory"); break;
    case 6: asm volatile("cp.async.wait_group 6;\n" ::: "memory"); break;
    default: asm volatile("cp.async.wait_group 7;\n" ::: "memory"); break;
  }
}

// A, B bf16, D fp32, both K-major, M = 128
__device__ __forceinline__ unsigned splitInstrDesc(unsigned n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((n >> 3) << 17) | ((unsigned)(kSplitRows >> 4) << 24);
}
__device__ __forceinline__ unsigned electOne() {
  unsigned e;
  asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(e));
  return e;
}
// executed by the whole warp, issued by the lane with `elected` != 0
__device__ __forceinline__ void mmaBf16TmemA(unsigned elected, unsigned d, unsigned a, unsigned long long b, unsigned idesc, unsigned accumulate) {
  asm volatile(
      "{\n .reg .pred p, e;\n setp.ne.b32 p, %4, 0;\n setp.ne.b32 e, %5, 0;\n"
      " @e tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}\n"
      ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(accumulate), "r"(elected) : "memory");
}

// Two neighbouring values of the contraction index as packed bf16 pairs (x0 in the low half): h to 6 bits and m to 8, each
// rounded to nearest, and what is left, l.  h + m + l is x (6 + 1 + 8 + 1 + 8 bits: a remainder rounded to nearest has one
// bit less) unless l has bits below a bf16's, which the caller finds in the low half of `left`, as with values that are
// not finite.
__device__ __forceinline__ void split2(float x0, float x1, unsigned& h, unsigned& m, unsigned& l, unsigned& left) {
  const unsigned h0 = (__float_as_uint(x0) + 0x20000u) & 0xFFFC0000u, h1 = (__float_as_uint(x1) + 0x20000u) & 0xFFFC0000u;
  const float r0 = x0 - __uint_as_float(h0), r1 = x1 - __uint_as_float(h1);   // exact
  const __nv_bfloat162 mp = __floats2bfloat162_rn(r0, r1);
  const unsigned l0 = __float_as_uint(r0 - __low2float(mp)), l1 = __float_as_uint(r1 - __high2float(mp));   // exact
  h = __byte_perm(h0, h1, 0x7632);
  m = *reinterpret_cast<const unsigned*>(&mp);
  l = __byte_perm(l0, l1, 0x7632);
  left |= l0 | l1;
}

// Offset of position J by the strides s0, s1, s2 of its three indices.
__device__ __forceinline__ long long positionOf(const SplitArgs& a, unsigned J, unsigned s0, unsigned s1, unsigned s2) {
  const unsigned r0 = quot(J, a.n0), i0 = J - r0 * a.n0.d, i2 = quot(r0, a.n1), i1 = r0 - i2 * a.n1.d;
  return (long long)((unsigned long long)i0 * s0 + (unsigned long long)i1 * s1 + (unsigned long long)i2 * s2);
}

// Columns c0 .. c0+31 of this lane's position J, whose results start at zoff, with alpha and beta*Y; executed by a whole
// warp with scratch sc (32 rows of kXposePitch).
__device__ __forceinline__ void storeBlock(const SplitArgs& a, float* sc, float (&r)[32], unsigned c0, unsigned J, long long zoff, bool store) {
  const int lane = threadIdx.x & 31;
  const bool epi = a.epilogue != 0;
  const bool useY = epi && a.beta != 0.f && a.Y != nullptr;
  const bool linear = a.n0.d == a.total;
  if (!a.outT) {
    float* z = a.Z + zoff + (long long)c0 * a.zsQ;
    if (!epi) {
      if (store && c0 + 32 <= a.Q) {
#pragma unroll
        for (unsigned i = 0; i < 32; i++, z += a.zsQ) *z = r[i];
      } else if (store) {
#pragma unroll
        for (unsigned i = 0; i < 32; i++, z += a.zsQ)
          if (c0 + i < a.Q) *z = r[i];
      }
    } else if (store) {
      const float* y = a.Y + zoff + (long long)c0 * a.zsQ;
#pragma unroll
      for (unsigned g = 0; g < 32; g += 4) {            // Y may be Z: read a batch ahead of its stores
        float yv[4];
#pragma unroll
        for (unsigned i = 0; i < 4; i++) yv[i] = useY && c0 + g + i < a.Q ? y[(long long)(g + i) * a.zsQ] : 0.f;
#pragma unroll
        for (unsigned i = 0; i < 4; i++, z += a.zsQ) {
          float v = a.alpha * r[g + i];
          if (useY) v = fmaf(a.beta, yv[i], v);
          if (c0 + g + i < a.Q) *z = v;
        }
      }
    }
  } else {
    // Lanes hold positions, the output wants lanes along q: through the warp's scratch, 32 columns (a whole
    // 128-byte line of every row) at a time.
    const unsigned stores = __ballot_sync(0xffffffffu, store);
#pragma unroll
    for (unsigned i = 0; i < 32; i += 4)
      *reinterpret_cast<float4*>(sc + lane * kXposePitch + i) = make_float4(r[i], r[i + 1], r[i + 2], r[i + 3]);
    __syncwarp();
    // offset of row rr of this warp's 32, also on lanes whose own position lies beyond the last
    auto rowOff = [&](unsigned rr) -> long long {
      if (linear) return (long long)((unsigned long long)(J - (unsigned)lane + rr) * a.zs0);
      return __shfl_sync(0xffffffffu, zoff, (int)rr);
    };
    // (reads of a batch of rows ahead of their stores: a store may alias the scratch as far as the compiler knows)
    if (a.vecZ) {
      const unsigned q = c0 + 4 * ((unsigned)lane & 7u);           // Q % 4 == 0: whole vectors
#pragma unroll 1
      for (unsigned b = 0; b < 32; b += 8) {
        float4 v[2];
        long long o[2];
#pragma unroll
        for (unsigned i = 0; i < 2; i++) {
          const unsigned rr = b + 4 * i + ((unsigned)lane >> 3);
          v[i] = *reinterpret_cast<const float4*>(sc + rr * kXposePitch + 4 * (lane & 7));
          o[i] = rowOff(rr) + q;
        }
#pragma unroll
        for (unsigned i = 0; i < 2; i++) {
          const unsigned rr = b + 4 * i + ((unsigned)lane >> 3);
          if (q >= a.Q || !(stores >> rr & 1u)) continue;
          if (epi) {
            v[i].x = a.alpha * v[i].x; v[i].y = a.alpha * v[i].y; v[i].z = a.alpha * v[i].z; v[i].w = a.alpha * v[i].w;
            if (useY) {
              const float4 y = *reinterpret_cast<const float4*>(a.Y + o[i]);
              v[i].x = fmaf(a.beta, y.x, v[i].x); v[i].y = fmaf(a.beta, y.y, v[i].y);
              v[i].z = fmaf(a.beta, y.z, v[i].z); v[i].w = fmaf(a.beta, y.w, v[i].w);
            }
          }
          *reinterpret_cast<float4*>(a.Z + o[i]) = v[i];
        }
      }
    } else {
      const unsigned q = c0 + (unsigned)lane;
#pragma unroll 2
      for (unsigned b = 0; b < 32; b += 4) {
        float v[4];
#pragma unroll
        for (unsigned i = 0; i < 4; i++) v[i] = sc[(b + i) * kXposePitch + lane];
#pragma unroll
        for (unsigned i = 0; i < 4; i++) {
          const long long o = rowOff(b + i) + q;
          if (q < a.Q && (stores >> (b + i) & 1u)) {
            if (epi) { v[i] = a.alpha * v[i]; if (useY) v[i] = fmaf(a.beta, a.Y[o], v[i]); }
            a.Z[o] = v[i];
          }
        }
      }
    }
    __syncwarp();
  }
}

// Rows whose operands a split does not hold, after the tiles on the tensor cores: the FMA chain over p, by the whole CTA.  Stages
// of kFmaChunk p go through registers into shared memory (past the L1, of which next to nothing is left) while 16 warps
// contract the one before, 4 positions x 4 columns a thread.  A function of its own, so that it takes no registers from the
// roles; what its loops need of the arguments is read once (through a reference each reading goes to memory).
// marks == nullptr: every row.  268 MB in and out, a factor that cannot be split: 64x64 733 us (FMA kernel 190), 128x128 with 134 MB 1085
// (338), 36x36 997 (680); a row in a thousand 264 / 429 / 374.  Bound by the latency of its stages: it is the route for rare operands.
template <bool XT>
__device__ __noinline__ void fmaTiles(const SplitArgs& args, float* xpose, float* ring, const unsigned* marks, unsigned rowHuge) {
  const unsigned tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const unsigned first = blockIdx.x, step = gridDim.x;
  const unsigned P = args.P, Q = args.Q, N = args.N, total = args.total;
  const unsigned tiles = first < args.numTiles ? (args.numTiles - first + step - 1) / step : 0;
  const float* const X = args.X;
  const float* const F = args.F;
  const long long xsP = args.xsP;
  const bool fRows = args.fsQ == 1;                              // factor stored as [p][q], else [q][p]
  // shared memory: [kFmaChunk][kFmaPitch] of X, [kFmaChunk][kBlockN] of the factor; the result takes their place
  const unsigned xs = smemAddr(ring), fs = xs + kFmaChunk * kFmaPitch * 4u;
  long long* const xo = reinterpret_cast<long long*>(ring + kSplitRows * kOutPitch);   // [kSplitRows], -1 beyond the last position
  for (unsigned it = 0; it < tiles; it++) {
    if (marks != nullptr && (marks[it % kTileBits / 32] >> (it & 31u) & 1u) == 0) continue;
    const unsigned J0 = (first + it * step) * (unsigned)kSplitRows;
    __syncthreads();
    if (tid < kSplitRows) xo[tid] = J0 + tid < total ? positionOf(args, J0 + tid, args.xs0, args.xs1, args.xs2) : -1;
    __syncthreads();
    float vx[kLoadX], vf[kLoadF];
    auto fetch = [&](unsigned p0, unsigned cb) {
#pragma unroll
      for (unsigned i = 0; i < kLoadX; i++) {
        const unsigned e = i * kFmaThreads + tid, p = p0 + (XT ? e % kFmaChunk : e / kSplitRows);
        const long long o = xo[XT ? e / kFmaChunk : e % kSplitRows];
        vx[i] = o >= 0 && p < P ? __ldcg(X + o + p * xsP) : 0.f;
      }
#pragma unroll
      for (unsigned i = 0; i < kLoadF; i++) {
        const unsigned e = i * kFmaThreads + tid, p = p0 + (fRows ? e / kBlockN : e % kFmaChunk), q = cb + (fRows ? e % kBlockN : e / kFmaChunk);
        vf[i] = p < P && q < Q ? __ldcg(F + (fRows ? p * Q + q : q * P + p)) : 0.f;
      }
    };
    for (unsigned cb = 0; cb < N; cb += kBlockN) {
      float r[16], mx = 0.f;
      unsigned left = 0;
#pragma unroll
      for (unsigned i = 0; i < 16; i++) r[i] = 0.f;
      if (tid < kFmaThreads) fetch(0, cb);
#pragma unroll 1
      for (unsigned p0 = 0; p0 < P; p0 += kFmaChunk) {
        if (tid < kFmaThreads) {
#pragma unroll
          for (unsigned i = 0; i < kLoadX; i++) {
            const unsigned e = i * kFmaThreads + tid;
            ring[(XT ? e % kFmaChunk : e / kSplitRows) * kFmaPitch + (XT ? e / kFmaChunk : e % kSplitRows)] = vx[i];
          }
#pragma unroll
          for (unsigned i = 0; i < kLoadF; i++) {
            const unsigned e = i * kFmaThreads + tid;
            ring[kFmaChunk * kFmaPitch + (fRows ? e : e % kFmaChunk * kBlockN + e / kFmaChunk)] = vf[i];
          }
        }
        __syncthreads();
        if (tid < kFmaThreads) {
          if (p0 + kFmaChunk < P) fetch(p0 + kFmaChunk, cb);
          unsigned x = xs + 16 * lane, f = fs + 16 * warp;
          const unsigned n = min(P - p0, kFmaChunk);
#pragma unroll 4
          for (unsigned p = 0; p < n; p++, x += kFmaPitch * 4, f += kBlockN * 4) {
            const float4 xv = ldShared4(x), fv = ldShared4(f);
            const float xa[4] = {xv.x, xv.y, xv.z, xv.w};
#pragma unroll
            for (unsigned i = 0; i < 4; i++) {
              r[4 * i] = fmaf(xa[i], fv.x, r[4 * i]);
              r[4 * i + 1] = fmaf(xa[i], fv.y, r[4 * i + 1]);
              r[4 * i + 2] = fmaf(xa[i], fv.z, r[4 * i + 2]);
              r[4 * i + 3] = fmaf(xa[i], fv.w, r[4 * i + 3]);
            }
          }
        }
        if (marks != nullptr && warp < kSplitEpiWarps) {        // the converters' verdict on this thread's row
#pragma unroll 2
          for (unsigned p = 0; p < kFmaChunk; p += 2) {
            const unsigned y = xs + (p * kFmaPitch + (warp & 3u) * 32u + lane) * 4u;
            const float x0 = ldShared(y), x1 = ldShared(y + kFmaPitch * 4);
            unsigned h, m, l;
            split2(x0, x1, h, m, l, left);
            mx = fmaxf(mx, fmaxf(fabsf(x0), fabsf(x1)));
          }
        }
        __syncthreads();
      }
      // one position and 32 columns a thread, as the stores want them
      if (tid < kFmaThreads) {
#pragma unroll
        for (unsigned i = 0; i < 4; i++)
          *reinterpret_cast<float4*>(ring + (4 * lane + i) * kOutPitch + 4 * warp) = make_float4(r[4 * i], r[4 * i + 1], r[4 * i + 2], r[4 * i + 3]);
      }
      __syncthreads();
      if (warp < kSplitEpiWarps) {
        const unsigned row = (warp & 3u) * 32u + lane, c0 = (warp >> 2) * 32u, J = J0 + row;
        float z[32];
#pragma unroll
        for (unsigned i = 0; i < 32; i += 4) {
          const float4 v = ldShared4(xs + (row * kOutPitch + c0 + i) * 4u);
          z[i] = v.x; z[i + 1] = v.y; z[i + 2] = v.z; z[i + 3] = v.w;
        }
        const bool mine = marks == nullptr || (left & 0xFFFFu) != 0 || __float_as_uint(mx) >= rowHuge;
        storeBlock(args, xpose + warp * 32 * kXposePitch, z, cb + c0, J, positionOf(args, J, args.zs0, args.zs1, args.zs2), J < total && mine);
      }
      __syncthreads();
    }
  }
}

// XT: the contracted index is contiguous in X (lanes load along p); otherwise lanes load along j.
// KS: steps of 16 along the contraction.
template <bool XT, int KS>
__global__ void __launch_bounds__(kSplitThreads, 1) gemmSplitKernel(const __grid_constant__ SplitArgs a) {
  constexpr unsigned K = 16 * KS, ks = KS, half = K / 2;     // half: TMEM columns of one piece of A
  constexpr unsigned slabs = (K + 63) / 64;
  constexpr unsigned hSlots = (KS + kHhSteps - 1) / kHhSteps;  // accumulators of h*h per block of columns
  extern __shared__ unsigned char smemRaw[];
  unsigned char* base = reinterpret_cast<unsigned char*>(((uintptr_t)smemRaw + 1023) & ~(uintptr_t)1023);
  const unsigned pieceBytes = slabs * a.N * 128u;            // one bf16 copy of the factor: [K/64][N rows q][64 k], 128-byte swizzle
  unsigned char* Fs = base;
  float* xpose = reinterpret_cast<float*>(base + 3 * pieceBytes);                             // outT only
  float* ring = xpose + (a.outT ? kXposeBytes / sizeof(float) : 0);
  __shared__ __align__(8) unsigned long long aFull[2][8], aEmpty[2][8], dFull[kMaxSlots], dEmpty[kMaxSlots], drained;
  __shared__ unsigned tmemBaseSlot;
  __shared__ int abortFlag, factorSpecial;
  __shared__ unsigned rowHuge;
  __shared__ unsigned tileMarks[kTileBits / 32], anyMark;
  __shared__ unsigned factorMax;                             // float bits of the largest magnitude
  __shared__ unsigned short rowState[8][kSplitRows];  // tile it, position: (it >> 3) + 1 if its row cannot be split

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  constexpr unsigned nA = aBuffers(KS);
  constexpr unsigned aCols = 3 * half;                     // TMEM columns of one A buffer: [h][m][l]

  if (tid == 0) {
    for (int i = 0; i < 16; i++) { mbarInit(&aFull[i >> 3][i & 7], 4); mbarInit(&aEmpty[i >> 3][i & 7], 1); }
    // dFull: the commit of the MMAs, and an ordinary arrival that carries what the converters wrote (rowState)
    for (unsigned i = 0; i < kMaxSlots; i++) { mbarInit(&dFull[i], 2); mbarInit(&dEmpty[i], kSplitEpiWarps); }
    mbarInit(&drained, 1);
    abortFlag = 0; factorSpecial = 0; anyMark = 0;
    factorMax = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == kSplitMmaWarp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smemAddr(&tmemBaseSlot)), "r"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  __syncthreads();
  for (unsigned i = tid; i < kTileBits / 32; i += kSplitThreads) tileMarks[i] = 0;
  for (unsigned i = tid; i < 8 * kSplitRows; i += kSplitThreads) (&rowState[0][0])[i] = 0;
  // factor -> three bf16 copies, row q, k contiguous: 16-byte unit (k % 64) / 8 XOR (q % 8)
  unsigned fMax = 0, fLeft = 0;
  auto putFactor = [&](unsigned kp, unsigned q) {
    const unsigned k = 2 * kp;
    const bool okQ = q < a.Q;
    const float* f = a.F + (long long)k * a.fsP + (long long)q * a.fsQ;
    const float v0 = okQ && k < a.P ? f[0] : 0.f, v1 = okQ && k + 1 < a.P ? f[a.fsP] : 0.f;
    unsigned h, m, l;
    split2(v0, v1, h, m, l, fLeft);
    fMax = max(fMax, max(__float_as_uint(v0) & 0x7FFFFFFFu, __float_as_uint(v1) & 0x7FFFFFFFu));
    unsigned char* d = Fs + (k >> 6) * (a.N * 128u) + q * 128u + ((((k & 63) >> 3) ^ (q & 7)) << 4) + (k & 7) * 2u;
    *reinterpret_cast<unsigned*>(d) = h;
    *reinterpret_cast<unsigned*>(d + pieceBytes) = m;
    *reinterpret_cast<unsigned*>(d + 2 * pieceBytes) = l;
  };
  if (a.fsP != 1 || a.fsQ == 1) {
    for (unsigned kp = warp; kp < K / 2; kp += kSplitThreads / 32)
      for (unsigned q = lane; q < a.N; q += 32) putFactor(kp, q);
  } else {
    for (unsigned q = warp; q < a.N; q += kSplitThreads / 32)
      for (unsigned kp = lane; kp < K / 2; kp += 32) putFactor(kp, q);
  }
  fMax = __reduce_max_sync(0xffffffffu, fMax);
  if (lane == 0) atomicMax(&factorMax, fMax);
  if ((fLeft & 0xFFFFu) != 0 || fMax >= kHuge) factorSpecial = 1;
  asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");      // generic-proxy writes -> tensor-core reads
  fenceBeforeSync();
  __syncthreads();
  fenceAfterSync();
  // the row magnitude at which a sum of 128 products may pass 2^126 (terms of a split could become infinities of
  // opposite signs)
  if (tid == 0) rowHuge = min(kHuge, __float_as_uint(0x1p119f / __uint_as_float(factorMax)));
  __syncthreads();
  const unsigned tmemBase = *(volatile unsigned*)&tmemBaseSlot;
  volatile int* abortP = &abortFlag;
  const unsigned dCol = tmemBase + nA * aCols;

  const unsigned first = blockIdx.x, step = gridDim.x;
  const unsigned myTiles = first < a.numTiles && factorSpecial == 0 ? (a.numTiles - first + step - 1) / step : 0;

  if (warp < kSplitEpiWarps) {
    // ---- epilogue ----------------------------------------------------------------------------
    const unsigned quarter = (unsigned)warp & 3u, part = (unsigned)warp >> 2;
    float* const sc = xpose + warp * 32 * kXposePitch;
    // take(): the MMAs into accumulator `sl` are complete; give(): this warp has read it.  Each set has full-barriers of
    // its own (a wait for a later phase than the next is none); bit `sl` of phases: parity of the next one of `sl`.
    unsigned sSlot = 0, slot = a.sSlots, phases = 0;
    auto take = [&](unsigned sl) {
      const bool all = __all_sync(0xffffffffu, waitBounded(&dFull[sl], phases >> sl & 1u, abortP));
      phases ^= 1u << sl;
      fenceAfterSync();
      return all;
    };
    auto give = [&](unsigned sl) {
      fenceBeforeSync();
      __syncwarp();
      if (lane == 0) mbarArrive(&dEmpty[sl]);
    };
    bool alive = true;
    for (unsigned it = 0; alive && it < myTiles; it++) {
      const unsigned J = (first + it * step) * (unsigned)kSplitRows + quarter * 32u + (unsigned)lane;
      const bool live = J < a.total;
      const long long zoff = positionOf(a, J, a.zs0, a.zs1, a.zs2);
      bool special = false, store = false;
#pragma unroll 1
      for (unsigned cb = 0; cb < a.N; cb += kBlockN) {
        const unsigned c0 = cb + part * 32u;
        const unsigned tcol = dCol + part * 32u + ((quarter * 32u) << 16);
        float r[32];
        // h*h first, then the small terms: one rounding to nearest per accumulator
        auto addFrom = [&](unsigned sl) {
#pragma unroll
          for (unsigned g = 0; g < 32; g += 16) {
            unsigned t[16];
            tmemLoad16(tcol + sl * a.slotCols + g, t);
            tmemLoadWait();
#pragma unroll
            for (unsigned i = 0; i < 16; i++) r[g + i] += __uint_as_float(t[i]);
          }
        };
#pragma unroll 1
        for (unsigned h = 0; h < hSlots; h++) {
          if (!take(slot)) { alive = false; break; }
          if (c0 < a.N) {
            if (h == 0) { tmemLoad32(tcol + slot * a.slotCols, reinterpret_cast<unsigned(&)[32]>(r)); tmemLoadWait(); }
            else addFrom(slot);
          }
          give(slot);
          if (++slot == a.slots) slot = a.sSlots;
        }
        if (!alive || !take(sSlot)) { alive = false; break; }
        if (cb == 0) {
          special = live && rowState[it & 7][quarter * 32 + lane] == (unsigned short)((it >> 3) + 1u);
          store = live && !special;
        }
        if (c0 < a.N) addFrom(sSlot);
        give(sSlot);
        if (++sSlot == a.sSlots) sSlot = 0;
        storeBlock(a, sc, r, c0, J, zoff, store);
      }
      if (part == 0 && __any_sync(0xffffffffu, special) && lane == 0) {
        atomicOr(&tileMarks[it % kTileBits / 32], 1u << (it & 31u));
        anyMark = 1;
      }
    }
  } else if (warp < kSplitMmaWarp) {
    // ---- converters ----------------------------------------------------------------------------
    const unsigned cw = (unsigned)(warp - kSplitEpiWarps);
    const unsigned sub = cw >> 2, quarter = cw & 3u;
    constexpr unsigned stageBytes = kSplitStageElems * 4;
    const unsigned myRing = smemAddr(ring) + cw * a.stages * stageBytes;
    // The chunks of this CTA's tiles, one after the other, go round the three warps of a quarter.  The loads run ahead of
    // the conversion by the depth of the ring: chunk ldN.
    const unsigned chunks = myTiles * ks;
    unsigned ldN = sub, ldTile = ~0u, ldMask = 0;
    // Input offsets of what this lane fetches, once per tile: ldOff of the position along j (the first of four with
    // 16-byte loads), or, with lanes along p, of position `lane`; ldRow, 16-byte loads along p: of the rows
    // lane / 4 + 8 i, in units of 16 bytes.  ldMask: which of them exist.
    long long ldOff = 0;
    unsigned ldRow[XT ? 4 : 1];
    auto offsetOf = [&](unsigned J) { return positionOf(a, J, a.xs0, a.xs1, a.xs2); };
    auto load = [&](unsigned st) {
      if (ldN < chunks) {
        const unsigned tile = ldN / ks;
        if (tile != ldTile) {
          ldTile = tile;
          const unsigned J0 = (first + tile * step) * (unsigned)kSplitRows + quarter * 32u;
          const unsigned rows = a.total > J0 ? min(a.total - J0, 32u) : 0u;
          if constexpr (!XT) {
            const unsigned j = a.vecX ? (unsigned)(lane & 7) * 4u : (unsigned)lane;   // n0 % 4 == 0 with 16-byte loads: whole vectors
            ldMask = j < rows ? 1u : 0u;
            ldOff = offsetOf(J0 + j);
          } else if (a.vecX) {
            const long long off = offsetOf(J0 + (unsigned)lane);
            ldMask = 0;
#pragma unroll
            for (int i = 0; i < 4; i++) {
              const unsigned row = ((unsigned)lane >> 2) + 8u * i;
              ldRow[i] = __shfl_sync(0xffffffffu, (unsigned)(off >> 2), (int)row) + ((unsigned)lane & 3u);
              if (row < rows) ldMask |= 1u << i;
            }
          } else {
            ldOff = offsetOf(J0 + (unsigned)lane);
            ldMask = rows;
          }
        }
        const unsigned p0 = (ldN - tile * ks) * kSplitChunk;
        const bool whole = p0 + kSplitChunk <= a.P;     // else p beyond P: zeros
        if constexpr (!XT) {
          if (a.vecX) {
            if (ldMask) {
              const float* x = a.X + ldOff + (long long)(p0 + ((unsigned)lane >> 3)) * a.xsP;
              const unsigned d = st + 16u * (unsigned)lane;
              if (whole) {
#pragma unroll
                for (int i = 0; i < 4; i++, x += 4 * a.xsP) cpAsyncFill<16>(d + i * 512, x, true);
              } else {
#pragma unroll
                for (unsigned i = 0; i < 4; i++, x += 4 * a.xsP) {
                  const bool ok = p0 + ((unsigned)lane >> 3) + 4 * i < a.P;
                  cpAsyncFill<16>(d + i * 512, ok ? x : a.X, ok);
                }
              }
            }
          } else if (ldMask) {
            const float* x = a.X + ldOff + (long long)p0 * a.xsP;
            const unsigned d = st + 4u * (unsigned)lane;
            if (whole) {
#pragma unroll
              for (int i = 0; i < kSplitChunk; i++, x += a.xsP) cpAsyncFill<4>(d + i * 128, x, true);
            } else {
#pragma unroll
              for (unsigned i = 0; i < kSplitChunk; i++, x += a.xsP) cpAsyncFill<4>(d + i * 128, p0 + i < a.P ? x : a.X, p0 + i < a.P);
            }
          }
        } else if (a.vecX) {
          const bool okP = p0 + 4 * ((unsigned)lane & 3u) < a.P;          // P % 4 == 0: whole vectors
#pragma unroll
          for (int i = 0; i < 4; i++) {
            const unsigned row = ((unsigned)lane >> 2) + 8u * i;
            if (ldMask >> i & 1u)
              cpAsyncFill<16>(st + row * 64 + ((((unsigned)lane & 3u) ^ (row >> 1 & 3u)) << 4), okP ? a.X + (4ll * ldRow[i] + p0) : a.X, okP);
          }
        } else {
          const unsigned pl = (unsigned)lane & 15u, p = p0 + pl;
          const bool okP = p < a.P;
          const float* xp = a.X + p;
#pragma unroll 8
          for (unsigned i = 0; i < 16; i++) {
            const unsigned row = ((unsigned)lane >> 4) + 2 * i;
            const long long ro = __shfl_sync(0xffffffffu, ldOff, (int)row);
            if (row < ldMask) cpAsyncFill<4>(st + row * 64 + ((((pl >> 2) ^ (row >> 1 & 3u)) << 4) | ((pl & 3u) << 2)), okP ? xp + ro : a.X, okP);
          }
        }
        ldN += kSplitSubs;
      }
      asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    for (unsigned s = 0; s < a.stages; s++) load(myRing + s * stageBytes);
    unsigned s = 0;
#pragma unroll 1
    for (unsigned n = sub; n < chunks; n += kSplitSubs) {
      const unsigned it = n / ks, c = n - it * ks, g = it % nA;
      cpAsyncWaitUpTo(a.stages - 1);
      __syncwarp();
      const unsigned st = myRing + s * stageBytes;
      float x[16];
      if constexpr (!XT) {
#pragma unroll
        for (int i = 0; i < 16; i++) x[i] = ldShared(st + i * 128 + 4 * lane);
      } else {
#pragma unroll
        for (int i = 0; i < 4; i++) {
          const float4 v = ldShared4(st + lane * 64 + ((i ^ (lane >> 1 & 3)) << 4));
          x[4 * i] = v.x; x[4 * i + 1] = v.y; x[4 * i + 2] = v.z; x[4 * i + 3] = v.w;
        }
      }
      __syncwarp();                                         // the stage has been read by every lane
      load(st);
      if (++s == a.stages) s = 0;
      unsigned h[8], m[8], l[8], left = 0;
      float mx = 0.f;
#pragma unroll
      for (int i = 0; i < 8; i++) {
        split2(x[2 * i], x[2 * i + 1], h[i], m[i], l[i], left);
        mx = fmaxf(mx, fmaxf(fabsf(x[2 * i]), fabsf(x[2 * i + 1])));
      }
      // (the use before the last one of this chunk has been consumed: 3 chunks are fewer than the buffers hold)
      if (!__all_sync(0xffffffffu, waitBounded(&aEmpty[g][c], (it / nA & 1u) ^ 1u, abortP))) break;
      fenceAfterSync();
      const unsigned col = tmemBase + g * aCols + c * 8u + ((quarter * 32u) << 16);
      tmemStore8(col, h);
      tmemStore8(col + half, m);
      tmemStore8(col + 2 * half, l);
      if ((left & 0xFFFFu) != 0 || __float_as_uint(mx) >= rowHuge) rowState[it & 7][quarter * 32 + lane] = (unsigned short)((it >> 3) + 1u);
      tmemStoreWait();
      fenceBeforeSync();
      __syncwarp();
      if (lane == 0) mbarArrive(&aFull[g][c]);
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  } else {
    // ---- MMA issue -------------------------------------------------------------------------------
    const unsigned elected = electOne();
    const unsigned long long bDesc = smemDesc(smemAddr(Fs), 16u, 1024u, kSwz128);
    const unsigned pieceUnits = pieceBytes >> 4, slabUnits = a.N * 8u;   // descriptor addresses are in 16-byte units
    unsigned sSlot = 0, sPhase = 1, slot = a.sSlots, phase = 1;
    bool alive = true;
    auto waitFor = [&](unsigned long long* bar, unsigned ph) {
      if (alive) alive = __all_sync(0xffffffffu, waitBounded(bar, ph, abortP));
    };
    auto give = [&](unsigned sl) {
      if (elected) {
        mmaCommit(&dFull[sl]);
        mbarArrive(&dFull[sl]);
      }
      __syncwarp();
    };
    for (unsigned it = 0; alive && it < myTiles; it++) {
      const unsigned g = it % nA, aPhase = it / nA & 1u;
      const unsigned tA = g * aCols;                           // the allocation is all of TMEM, it starts at 0
#pragma unroll 1
      for (unsigned cb = 0; alive && cb < a.N; cb += kBlockN) {
        const unsigned idesc = splitInstrDesc(min(a.N - cb, kBlockN));
        const unsigned long long bBlock = bDesc + cb * 8u;     // rows of 128 bytes
        const bool lastBlock = cb + kBlockN >= a.N;
        const unsigned tS = nA * aCols + sSlot * a.slotCols;
        waitFor(&dEmpty[sSlot], sPhase);
        unsigned tH = 0;
#pragma unroll
        for (unsigned k = 0; k < ks; k++) {
          if (cb == 0) waitFor(&aFull[g][k], aPhase);
          if (k % kHhSteps == 0) {
            waitFor(&dEmpty[slot], phase);
            tH = nA * aCols + slot * a.slotCols;
          }
          if (!alive) break;
          fenceAfterSync();
          const unsigned long long bK = bBlock + (k >> 2) * slabUnits + (k & 3u) * 2u;
          // piece pa of X times piece pb of the factor: h*h, and everything but it and l*l into the tile's small terms
          mmaBf16TmemA(elected, tH, tA + k * 8u, bK, idesc, k % kHhSteps != 0 ? 1u : 0u);
          if (k % kHhSteps == kHhSteps - 1 || k == ks - 1) {
            give(slot);
            if (++slot == a.slots) { slot = a.sSlots; phase ^= 1u; }
          }
#pragma unroll
          for (int t = 0; t < 7; t++) {
            constexpr unsigned pa[7] = {1, 2, 2, 0, 1, 1, 0}, pb[7] = {2, 1, 0, 2, 1, 0, 1};
            mmaBf16TmemA(elected, tS, tA + pa[t] * half + k * 8u, bK + pb[t] * pieceUnits, idesc, t > 0 || k > 0 ? 1u : 0u);
          }
          if (lastBlock && elected) mmaCommit(&aEmpty[g][k]);
          __syncwarp();
        }
        if (alive) give(sSlot);
        if (++sSlot == a.sSlots) { sSlot = 0; sPhase ^= 1u; }
      }
    }
    // No MMA may be in flight when the tensor memory goes back, also after a wait that gave up; about two seconds at most.
    if (elected) mmaCommit(&drained);
    __syncwarp();
    const long long t0 = clock64();
    while (!mbarTryWait(&drained, 0u) && clock64() - t0 < 4000000000ll) {}
  }

  // ---- teardown: every role gets here (all waits are bounded); release TMEM ----------------------
  fenceBeforeSync();
  __syncthreads();
  if (warp == kSplitMmaWarp) {
    __syncwarp();
    fenceAfterSync();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmemBase), "r"(512) : "memory");
  }
  if (abortFlag == 0 && (factorSpecial != 0 || anyMark != 0)) fmaTiles<XT>(a, xpose, ring, factorSpecial != 0 ? nullptr : tileMarks, rowHuge);
}

static unsigned long long gSplitLaunches = 0;
static int gSplitOff = 0;                          // measurement hook fkbSetSplitOff

template <bool XT, int KS>
static fastKronError launchSplitOne(const SplitArgs& a, const LaunchCtx& cx) {
  auto kern = gemmSplitKernel<XT, KS>;
  static bool attrDev[kMaxDevices] = {false};
  bool& attr = attrDev[currentDeviceSlot()];
  if (!attr) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSplitSmem) != cudaSuccess) {
      cudaGetLastError();
      return fastKronKernelNotFound;
    }
    attr = true;
  }
  unsigned grid = (unsigned)cx.smCount;
  if (grid > a.numTiles) grid = a.numTiles;
  // the whole shared memory, so that no second CTA lands on the SM and waits for the tensor memory of the first
  kern<<<grid, kSplitThreads, kSplitSmem, cx.stream>>>(a);
  gSplitLaunches++;
  return cudaToFk(cudaGetLastError());
}

template <bool XT>
static fastKronError launchSplitK(const SplitArgs& a, const LaunchCtx& cx) {
  switch ((a.P + 15) / 16) {
    case 2: return launchSplitOne<XT, 2>(a, cx);
    case 3: return launchSplitOne<XT, 3>(a, cx);
    case 4: return launchSplitOne<XT, 4>(a, cx);
    case 5: return launchSplitOne<XT, 5>(a, cx);
    case 6: return launchSplitOne<XT, 6>(a, cx);
    case 7: return launchSplitOne<XT, 7>(a, cx);
    case 8: return launchSplitOne<XT, 8>(a, cx);
    default: return fastKronKernelNotFound;
  }
}

}  // namespace tc

// Passes this kernel takes; anything else returns fastKronKernelNotFound and runs on the FMA kernels.
fastKronError launchGemmSplit(const Pass& ps, const LaunchCtx& cx) {
  using namespace tc;
  if (gSplitOff || cx.dt != DType::F32 || ps.nf != 1 || cx.batch > 1 || cx.scatter.parts > 0 || cx.pSplit != 0) return fastKronKernelNotFound;
  const uint64_t total = ps.M * ps.A * ps.B;
  if (!gemmSplitEligible(ps.P[0], ps.Q[0], total)) return fastKronKernelNotFound;

  SplitArgs a;
  a.X = (const float*)cx.src; a.Z = (float*)cx.dst; a.Y = (const float*)cx.Y; a.F = (const float*)cx.F[0];
  a.fsP = cx.fsP; a.fsQ = cx.fsQ;
  a.P = ps.P[0]; a.Q = ps.Q[0];
  a.N = (a.Q + 15) / 16 * 16;
  a.xsP = ps.xsG; a.zsQ = ps.zsG;
  a.alpha = (float)cx.alpha; a.beta = (float)cx.beta; a.epilogue = ps.epilogue ? 1 : 0;
  const bool xt = ps.xsG == 1;
  a.outT = ps.zsG == 1 ? 1 : 0;
  PosDim d[3];
  orderPositions(ps, d);
  a.n0 = posDiv((unsigned)d[0].n); a.n1 = posDiv((unsigned)d[1].n);
  unsigned* const strides[3][2] = {{&a.xs0, &a.zs0}, {&a.xs1, &a.zs1}, {&a.xs2, &a.zs2}};
  for (int i = 0; i < 3; i++) {
    if (d[i].n == 1) d[i].xs = d[i].zs = 0;                    // never multiplied
    if (d[i].xs < 0 || d[i].zs < 0 || d[i].xs >> 32 != 0 || d[i].zs >> 32 != 0) return fastKronKernelNotFound;
    *strides[i][0] = (unsigned)d[i].xs;
    *strides[i][1] = (unsigned)d[i].zs;
  }
  a.total = (unsigned)total;
  a.numTiles = (unsigned)((total + kSplitRows - 1) / kSplitRows);
  const bool al = ((uintptr_t)a.X & 15) == 0;
  auto m4 = [](int64_t v) { return v % 4 == 0; };
  // (16-byte units of the input offset are 32-bit there)
  const bool fits = d[0].n * (uint64_t)llabs(d[0].xs) + d[1].n * (uint64_t)llabs(d[1].xs) + d[2].n * (uint64_t)llabs(d[2].xs) < (1ull << 34);
  if (xt) a.vecX = al && fits && a.P % 4 == 0 && (d[0].n == 1 || m4(a.xs0)) && (d[1].n == 1 || m4(a.xs1)) && (d[2].n == 1 || m4(a.xs2));
  else a.vecX = al && positionsVectorise(d, true, a.xsP, 4);

  a.vecZ = a.outT && a.Q % 4 == 0 && ((uintptr_t)a.Z & 15) == 0 && ((uintptr_t)a.Y & 15) == 0 && (d[0].n == 1 || m4(a.zs0)) &&
           (d[1].n == 1 || m4(a.zs1)) && (d[2].n == 1 || m4(a.zs2));
  a.slotCols = a.N > 32 ? kBlockN : 32;
  // A second accumulator for the small terms where there is room for at least four of h*h.
  const unsigned ks = (a.P + 15) / 16, fit = (512 - aBuffers(ks) * 24 * ks) / a.slotCols;
  a.slots = fit < kMaxSlots ? fit : kMaxSlots;
  a.sSlots = a.slots >= 6 ? 2 : 1;
  const size_t factor = 3 * (size_t)((a.P + 63) / 64) * a.N * 128;
  const size_t stage = kSplitConvWarps * (size_t)kSplitStageElems * sizeof(float);    // one stage of every converter warp
  const size_t n = (kSplitSmem - 1024 - factor - (a.outT ? kXposeBytes : 0)) / stage;
  a.stages = (unsigned)(n > kSplitMaxStages ? kSplitMaxStages : n);
  return xt ? launchSplitK<true>(a, cx) : launchSplitK<false>(a, cx);
}

int gemmSplitTimeouts() {
  int v = 0;
  if (cudaMemcpyFromSymbol(&v, tc::gTcTimeouts, sizeof(int)) != cudaSuccess) { cudaGetLastError(); return -1; }
  return v;
}

}  // namespace fkb

// Non-zero if a bounded barrier wait of the split kernel ever gave up in this process (tests).
extern "C" int fkbGemmSplitTimeouts() { return fkb::gemmSplitTimeouts(); }
// Launches of the split kernel by this process so far (tests).
extern "C" unsigned long long fkbGemmSplitLaunches() { return fkb::tc::gSplitLaunches; }
// Measurement and cross-check hook: 1 = the passes of the split kernel run on the FMA kernels instead.
extern "C" void fkbSetSplitOff(int off) { fkb::tc::gSplitOff = off; }
