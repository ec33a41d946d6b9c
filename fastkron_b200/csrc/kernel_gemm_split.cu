// Large-factor pass of fp32 operands on the tensor cores with fp32 results: every operand is split
// EXACTLY into three bf16 numbers, v = h + m + l (8 + 8 + 8 significant bits hold the 24 of a float),
// and a product is formed as  h*h + (h*m + m*h) + (m*m + h*l + l*h)  with fp32 accumulation.  The three
// terms left out (m*l, l*m, l*l) are below 2^-26 of the product; the six kept ones are exact in the
// multiplier, so what remains is the rounding of the accumulator, once per 16 products instead of once per
// product as in an FMA chain.  The small terms are accumulated first, so that only the P/16 steps of h*h
// round at the magnitude of the result.
//
// One pass is  Z[j][q] = sum_p X[j][p] * F[p][q]  over the J = M*A*B positions (m, a, b) of the pass,
// any strides, any P and Q up to 128, any alignment.  A tile is 128 positions times all of Q:
//   D[128 x Q] (TMEM, fp32) += A[128 x P] (TMEM, bf16) * B[P x Q] (shared memory, bf16),  tcgen05.mma.kind::f16.
// Why A sits in TMEM: the positions come with j contiguous (B > 1) or p contiguous (B == 1), at any
// alignment.  A converter thread owns one position: it reads its P values from shared memory, splits them in
// registers and writes them to its TMEM lane with tcgen05.st.  The transposition that the j-contiguous
// operand needs happens on that way for nothing, and the tensor cores read X without touching shared
// memory (with the three copies there, operand reads alone would take as long as the HBM transfer).
//
// Warp roles (800 threads, one CTA per SM, persistent):
//   0-7   epilogue: tcgen05.ld of the accumulator (a lane quarter each, alternate groups of 32 columns),
//         alpha / beta*Y, stores
//   8-23  converters, two groups of eight warps that take alternate tiles.  Two warps share 32 positions and
//         take alternate chunks of 16 p; each loads its chunks with cp.async into a private ring of stages, so
//         between load and conversion there is no barrier, only a __syncwarp
//   24    MMA issue and the TMEM allocation.  The whole warp walks the loop (its values then stay in uniform
//         registers, where the instruction wants them) and one elected lane issues
// Every wait on a barrier is bounded; one that gives up raises the abort flag that ends all roles.
//
// Bound by HBM traffic and, where P is small, by the fixed work of a tile.  Measured on B200, 268 MB in and out (81 us at the copy
// rate), 64x64: 97 us a pass with j contiguous (FMA kernel 187), 127 us with p contiguous (cold X; 59 against 85 us at
// 100 MB); 128x128 and 134 MB (40 us): 64 / 74 us (FMA 320).  The contraction length is a template parameter because the MMAs are issued by
// one lane: with run-time descriptors a 128x64x16 MMA took 126-152 clocks, with immediate ones the passes no longer
// notice twice the MMAs.
//
// Operands a bf16 split cannot hold are found while splitting: elements with a remainder after the third piece
// (infinities, NaN, and numbers below about 2^-110 whose last bits lie under the smallest bf16 denormal 2^-133; the
// tensor cores take and give denormals in full), and magnitudes from 2^127 or whose sums could overflow.  A row with such
// an element, or every row when the factor has one, is recomputed by its epilogue thread as the plain FMA chain over p.
#include <stdlib.h>

#include <cuda_bf16.h>

#include "kernels.h"
#include "gemm_table.h"
#include "positions.h"
#include "tcgen05.cuh"

namespace fkb {
namespace tc {

constexpr int kSplitEpiWarps = 8, kSplitConvWarps = 16;
constexpr int kSplitMmaWarp = kSplitEpiWarps + kSplitConvWarps;
constexpr int kSplitThreads = 32 * (kSplitMmaWarp + 1);
constexpr int kSplitRows = 128;
constexpr int kSplitChunk = 16;                    // p per stage: a stage is 32 positions x 16 p of one converter warp
constexpr int kSplitStageElems = 32 * kSplitChunk;
constexpr int kSplitMaxStages = 5;
constexpr int kSplitSmem = (227 - 3) * 1024;         // dynamic shared memory; the static part is below 3 KB
constexpr int kXposePitch = 36;                    // 32 columns and an odd number of 16-byte units per row
constexpr size_t kXposeBytes = kSplitEpiWarps * 32 * kXposePitch * sizeof(float);
constexpr unsigned kHuge = 254u << 23;             // 2^127 as float bits

struct SplitArgs {
  const float* X; float* Z; const float* Y; const float* F;
  long long fsP, fsQ;
  unsigned P, Q;
  unsigned N;                                      // Q rounded up to 16
  unsigned stages;                                 // per converter warp, 1 .. kSplitMaxStages
  // position J = (i2*n1 + i1)*n0 + i0; element (J, p) of X at sum i*xs + p*xsP, (J, q) of Z and Y at sum i*zs + q*zsQ
  unsigned n0, n1;
  long long xs0, xs1, xs2, xsP;
  long long zs0, zs1, zs2, zsQ;
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
    default: asm volatile("cp.async.wait_group 4;\n" ::: "memory"); break;
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

// Two neighbouring values of the contraction index as packed bf16 pairs (x0 in the low half).  Returns 0 when h + m + l
// is x for both, something else when a remainder is left or a value is not finite.
__device__ __forceinline__ unsigned split2(float x0, float x1, unsigned& h, unsigned& m, unsigned& l) {
  const __nv_bfloat162 hp = __floats2bfloat162_rn(x0, x1);
  const float r0 = x0 - __low2float(hp), r1 = x1 - __high2float(hp);          // exact
  const __nv_bfloat162 mp = __floats2bfloat162_rn(r0, r1);
  const float s0 = r0 - __low2float(mp), s1 = r1 - __high2float(mp);          // exact
  const __nv_bfloat162 lp = __floats2bfloat162_rn(s0, s1);
  h = *reinterpret_cast<const unsigned*>(&hp);
  m = *reinterpret_cast<const unsigned*>(&mp);
  l = *reinterpret_cast<const unsigned*>(&lp);
  return __float_as_uint(s0 - __low2float(lp)) | __float_as_uint(s1 - __high2float(lp));
}

// XT: the contracted index is contiguous in X (lanes load along p); otherwise lanes load along j.
// KS: steps of 16 along the contraction.
template <bool XT, int KS>
__global__ void __launch_bounds__(kSplitThreads, 1) gemmSplitKernel(const SplitArgs a) {
  constexpr unsigned K = 16 * KS, ks = KS, half = K / 2;     // half: TMEM columns of one piece of A
  constexpr unsigned slabs = (K + 63) / 64;
  extern __shared__ unsigned char smemRaw[];
  unsigned char* base = reinterpret_cast<unsigned char*>(((uintptr_t)smemRaw + 1023) & ~(uintptr_t)1023);
  const unsigned pieceBytes = slabs * a.N * 128u;            // one bf16 copy of the factor: [K/64][N rows q][64 k], 128-byte swizzle
  unsigned char* Fs = base;
  float* xpose = reinterpret_cast<float*>(base + 3 * pieceBytes);                             // outT only
  float* ring = xpose + (a.outT ? kXposeBytes / sizeof(float) : 0);
  __shared__ __align__(8) unsigned long long aFull[2], aEmpty[2], dFull[2], dEmpty[2];
  __shared__ unsigned tmemBaseSlot;
  __shared__ int abortFlag, factorSpecial;
  __shared__ unsigned rowHuge;
  __shared__ unsigned factorMax;                             // float bits of the largest magnitude
  __shared__ unsigned char rowState[4][2][kSplitRows];       // 1: the position's row cannot be split; from its two converter warps

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  constexpr unsigned aCols = 3 * half;                     // TMEM columns of one A buffer: [h][m][l]
  const unsigned dCols = (a.N + 31) & ~31u;                  // one accumulator (read back 32 columns at a time)
  const unsigned nD = 2 * aCols + 2 * dCols <= 512 ? 2 : 1;  // accumulators; P, Q <= 128 leave room for one

  if (tid == 0) {
    for (int i = 0; i < 2; i++) { mbarInit(&aFull[i], kSplitConvWarps / 2); mbarInit(&aEmpty[i], 1); mbarInit(&dFull[i], 1); mbarInit(&dEmpty[i], kSplitEpiWarps); }
    abortFlag = 0; factorSpecial = 0;
    factorMax = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == kSplitMmaWarp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smemAddr(&tmemBaseSlot)), "r"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  __syncthreads();
  // factor -> three bf16 copies, row q, k contiguous: 16-byte unit (k % 64) / 8 XOR (q % 8)
  unsigned fMax = 0, fLeft = 0;
  auto putFactor = [&](unsigned kp, unsigned q) {
    const unsigned k = 2 * kp;
    const bool okQ = q < a.Q;
    const float* f = a.F + (long long)k * a.fsP + (long long)q * a.fsQ;
    const float v0 = okQ && k < a.P ? f[0] : 0.f, v1 = okQ && k + 1 < a.P ? f[a.fsP] : 0.f;
    unsigned h, m, l;
    fLeft |= split2(v0, v1, h, m, l);
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
  if (fLeft != 0 || fMax >= kHuge) factorSpecial = 1;
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
  const unsigned dCol = tmemBase + 2 * aCols;

  const unsigned first = blockIdx.x, step = gridDim.x;
  const unsigned myTiles = first < a.numTiles ? (a.numTiles - first + step - 1) / step : 0;

  if (warp < kSplitEpiWarps) {
    // ---- epilogue ----------------------------------------------------------------------------
    const unsigned quarter = (unsigned)warp & 3u, part = (unsigned)warp >> 2;
    const bool epi = a.epilogue != 0;
    const bool useY = epi && a.beta != 0.f && a.Y != nullptr;
    const bool allSpecial = factorSpecial != 0;
    const bool linear = a.n0 == a.total;
    float* sc = xpose + warp * 32 * kXposePitch;
    for (unsigned it = 0; it < myTiles; it++) {
      const unsigned d = nD == 2 ? (it & 1u) : 0u, use = nD == 2 ? (it >> 1) : it;
      const unsigned J = (first + it * step) * (unsigned)kSplitRows + quarter * 32u + (unsigned)lane;
      const bool live = J < a.total;
      const unsigned r0 = J / a.n0, i0 = J - r0 * a.n0, i2 = r0 / a.n1, i1 = r0 - i2 * a.n1;
      const long long zoff = (long long)i0 * a.zs0 + (long long)i1 * a.zs1 + (long long)i2 * a.zs2;
      bool ok = !*abortP && waitBounded(&dFull[d], use & 1u, abortP);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      fenceAfterSync();
      const bool special = live && (allSpecial || (rowState[it & 3][0][quarter * 32 + lane] | rowState[it & 3][1][quarter * 32 + lane]) != 0);
      const bool store = live && !special;
      const unsigned tcol = dCol + d * dCols + ((quarter * 32u) << 16);
#pragma unroll 1
      for (unsigned c0 = part * 32u; c0 < a.N || c0 < 64u; c0 += 64) {
        unsigned r[32];
        if (c0 < a.N) {
          tmemLoad32(tcol + c0, r);
          tmemLoadWait();
        }
        if (c0 + 64 >= a.N) {                                 // accumulator fully read: hand it back
          fenceBeforeSync();
          __syncwarp();
          if (lane == 0) mbarArrive(&dEmpty[d]);
        }
        if (!a.outT) {
          float* z = a.Z + zoff + (long long)c0 * a.zsQ;
          if (!epi) {
            if (store && c0 + 32 <= a.Q) {
#pragma unroll
              for (unsigned i = 0; i < 32; i++, z += a.zsQ) *z = __uint_as_float(r[i]);
            } else if (store) {
#pragma unroll
              for (unsigned i = 0; i < 32; i++, z += a.zsQ)
                if (c0 + i < a.Q) *z = __uint_as_float(r[i]);
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
                float v = a.alpha * __uint_as_float(r[g + i]);
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
            *reinterpret_cast<uint4*>(sc + lane * kXposePitch + i) = make_uint4(r[i], r[i + 1], r[i + 2], r[i + 3]);
          __syncwarp();
          // offset of row rr of this warp's 32, also on lanes whose own position lies beyond the last
          auto rowOff = [&](unsigned rr) -> long long {
            if (linear) return (long long)(J - (unsigned)lane + rr) * a.zs0;
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
      if (special && part == 0) {
        const float* x = a.X + (long long)i0 * a.xs0 + (long long)i1 * a.xs1 + (long long)i2 * a.xs2;
        for (unsigned q = 0; q < a.Q; q++) {
          float acc = 0.f;
          for (unsigned p = 0; p < a.P; p++) acc = fmaf(x[(long long)p * a.xsP], a.F[(long long)p * a.fsP + (long long)q * a.fsQ], acc);
          const long long o = zoff + (long long)q * a.zsQ;
          if (epi) { acc = a.alpha * acc; if (useY) acc = fmaf(a.beta, a.Y[o], acc); }
          a.Z[o] = acc;
        }
      }
    }
  } else if (warp < kSplitMmaWarp) {
    // ---- converters ----------------------------------------------------------------------------
    const unsigned cw = (unsigned)(warp - kSplitEpiWarps);
    const unsigned group = cw >> 3, sub = (cw >> 2) & 1u, quarter = cw & 3u;
    constexpr unsigned stageBytes = kSplitStageElems * 4;
    const unsigned myRing = smemAddr(ring) + cw * a.stages * stageBytes;
    // this warp takes the chunks sub, sub + 2, ... of the ks
    const unsigned myGroupTiles = ks > sub && myTiles > group ? (myTiles - group + 1) / 2 : 0;
    // the loads run ahead of the conversion by the depth of the ring: tile ldTile (of this group), chunk ldC
    unsigned ldTile = 0, ldC = sub, ldMask = 0;
    // Input offsets of what this lane fetches, once per tile: ldOff of the position along j (the first of four with
    // 16-byte loads), or, with lanes along p, of position `lane`; ldRow, 16-byte loads along p: of the rows
    // lane / 4 + 8 i, in units of 16 bytes.  ldMask: which of them exist.
    long long ldOff = 0;
    unsigned ldRow[XT ? 4 : 1];
    auto offsetOf = [&](unsigned J) {
      const unsigned r0 = J / a.n0, i0 = J - r0 * a.n0, i2 = r0 / a.n1, i1 = r0 - i2 * a.n1;
      return (long long)i0 * a.xs0 + (long long)i1 * a.xs1 + (long long)i2 * a.xs2;
    };
    auto load = [&](unsigned st) {
      if (ldTile < myGroupTiles) {
        if (ldC == sub) {
          const unsigned J0 = (first + (2 * ldTile + group) * step) * (unsigned)kSplitRows + quarter * 32u;
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
        const unsigned p0 = ldC * kSplitChunk;
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
        ldC += 2;
        if (ldC >= ks) { ldC = sub; ldTile++; }
      }
      asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    for (unsigned s = 0; s < a.stages; s++) load(myRing + s * stageBytes);
    unsigned s = 0;
    const unsigned aBase = tmemBase + group * aCols + ((quarter * 32u) << 16);
    for (unsigned li = 0; li < myGroupTiles; li++) {
      bool ok = !*abortP && waitBounded(&aEmpty[group], (li & 1u) ^ 1u, abortP);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      fenceAfterSync();
      __nv_bfloat162 mx = __floats2bfloat162_rn(0.f, 0.f);
      unsigned left = 0;
#pragma unroll 1
      for (unsigned c = sub; c < ks; c += 2) {
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
        unsigned h[8], m[8], l[8];
#pragma unroll
        for (int i = 0; i < 8; i++) {
          left |= split2(x[2 * i], x[2 * i + 1], h[i], m[i], l[i]);
          mx = __hmax2(mx, __habs2(*reinterpret_cast<const __nv_bfloat162*>(&h[i])));
        }
        const unsigned col = aBase + c * 8u;
        tmemStore8(col, h);
        tmemStore8(col + half, m);
        tmemStore8(col + 2 * half, l);
      }
      const unsigned bits = __float_as_uint(__bfloat162float(__hmax(__low2bfloat16(mx), __high2bfloat16(mx))));
      rowState[(2 * li + group) & 3][sub][quarter * 32 + lane] = left != 0 || bits >= rowHuge ? 1 : 0;
      tmemStoreWait();
      fenceBeforeSync();
      __syncwarp();
      if (lane == 0) mbarArrive(&aFull[group]);
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  } else {
    // ---- MMA issue -------------------------------------------------------------------------------
    const unsigned elected = electOne();
    const unsigned idesc = splitInstrDesc(a.N);
    const unsigned long long bDesc = smemDesc(smemAddr(Fs), 16u, 1024u, kSwz128);
    const unsigned pieceUnits = pieceBytes >> 4, slabUnits = a.N * 8u;   // descriptor addresses are in 16-byte units
    for (unsigned it = 0; it < myTiles; it++) {
      const unsigned g = it & 1u, aUse = it >> 1;
      const unsigned d = nD == 2 ? g : 0u, dUse = nD == 2 ? aUse : it;
      bool ok = !*abortP && waitBounded(&aFull[g], aUse & 1u, abortP) && waitBounded(&dEmpty[d], (dUse & 1u) ^ 1u, abortP);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      fenceAfterSync();
      const unsigned tA = g * aCols, tD = 2 * aCols + d * dCols;         // the allocation is all of TMEM, it starts at 0
      // six sweeps over the contraction index, the small terms first: piece pa of X times piece pb of the factor
#pragma unroll
      for (int t = 0; t < 6; t++) {
        constexpr unsigned pa[6] = {2, 0, 1, 1, 0, 0}, pb[6] = {0, 2, 1, 0, 1, 0};
#pragma unroll
        for (unsigned k = 0; k < ks; k++)
          mmaBf16TmemA(elected, tD, tA + pa[t] * half + k * 8u, bDesc + pb[t] * pieceUnits + (k >> 2) * slabUnits + (k & 3u) * 2u, idesc,
                       t > 0 || k > 0 ? 1u : 0u);
      }
      if (elected) {
        mmaCommit(&aEmpty[g]);
        mmaCommit(&dFull[d]);
      }
      __syncwarp();
    }
  }

  // ---- teardown: every role gets here (all waits are bounded); release TMEM ----------------------
  fenceBeforeSync();
  __syncthreads();
  if (warp == kSplitMmaWarp) {
    __syncwarp();
    fenceAfterSync();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmemBase), "r"(512) : "memory");
  }
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
  a.n0 = (unsigned)d[0].n; a.n1 = (unsigned)d[1].n;
  a.xs0 = d[0].xs; a.xs1 = d[1].xs; a.xs2 = d[2].xs;
  a.zs0 = d[0].zs; a.zs1 = d[1].zs; a.zs2 = d[2].zs;
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
