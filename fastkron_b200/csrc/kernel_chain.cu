// Several consecutive factors of any shape (square or not, any size, any strides, any alignment) contracted in
// shared memory in one launch:  Z[j][h] = sum_g X[j][g] * (F_0 (x) F_1 (x) ... )[g][h]  for every position j,
// one factor after the other, last first, products of an output accumulated over p ascending as everywhere else.
//
// What bounds the passes it replaces is one read and one write of the whole matrix per factor (and, for a few
// rows, one launch per factor); a group of nf factors reads and writes it once.
//
// A tile is W positions ("columns") times the group index, [g][W] with the columns contiguous, in two
// buffers that the steps alternate between (a factor that is not square changes the size).  A thread takes
// one 16-byte vector of columns and up to eight outputs q of it: per p one vector of the tile and eight
// factor values (broadcast) from shared memory feed 8 x 4 (fp32) or 8 x 2 (fp64) multiply-adds, the ratio at which
// the shared-memory and FMA pipes take about the same time; more outputs per thread would leave small tiles
// without enough threads.  Where the group index is the contiguous one in memory, lanes run along it and each
// thread gathers the vector of columns from its VEC rows, so global accesses stay coalesced and the shared
// tile needs no second layout (the row pitch is then an odd number of vectors: no bank conflicts).
#include <cuda_runtime.h>

#include "kernels.h"
#include "chain_table.h"
#include "positions.h"
#include "kernel_tile.cuh"   // Vec16, cpAsync16

namespace fkb {

// n / d for n * d < 2^32: high word of n * ceil(2^32 / d)
struct FastDiv { unsigned d, m; };
static FastDiv fastDiv(unsigned d) { return FastDiv{d, d > 1 ? (unsigned)(((1ull << 32) + d - 1) / d) : 0u}; }
__device__ __forceinline__ unsigned quot(unsigned n, const FastDiv& f) { return f.d == 1 ? n : __umulhi(n, f.m); }

template <typename T>
struct ChainArgs {
  const T* X; T* Z; const T* Y;
  const T* F[kMaxGroup];
  long long fsP[kMaxGroup], fsQ[kMaxGroup];
  unsigned P[kMaxGroup], Q[kMaxGroup], qb[kMaxGroup], fb[kMaxGroup];
  FastDiv nb[kMaxGroup], inner[kMaxGroup];          // blocks of outputs; product of the later Q's
  unsigned outer[kMaxGroup];                        // product of the earlier P's
  int nf;
  FastDiv G, H;
  unsigned W, logW, pitch, offB, offF, offT;
  unsigned n0, n1;
  long long xs0, xs1, xs2, xsG, zs0, zs1, zs2, zsG;
  unsigned total, numTiles;
  int vecX, vecZ, epilogue;
  T alpha, beta;
};

// acc[q][c] += f[q] * x[c]; fp32 with the packed FMA (two independent IEEE FMAs per instruction)
template <typename T, int QB>
struct ChainAcc {
  static constexpr int VEC = Vec16<T>::N;
  T v[QB][VEC];
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int q = 0; q < QB; q++)
#pragma unroll
      for (int c = 0; c < VEC; c++) v[q][c] = T(0);
  }
  __device__ __forceinline__ void add(int q, T f, const Vec16<T>& x) {
#pragma unroll
    for (int c = 0; c < VEC; c++) v[q][c] = fma(x.v[c], f, v[q][c]);
  }
  __device__ __forceinline__ Vec16<T> get(int q) const {
    Vec16<T> o;
#pragma unroll
    for (int c = 0; c < VEC; c++) o.v[c] = v[q][c];
    return o;
  }
};
template <int QB>
struct ChainAcc<float, QB> {
  float2 v[QB][2];
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int q = 0; q < QB; q++) v[q][0] = v[q][1] = make_float2(0.f, 0.f);
  }
  __device__ __forceinline__ void add(int q, float f, const Vec16<float>& x) {
    const float2 ff = make_float2(f, f);
    v[q][0] = __ffma2_rn(make_float2(x.v[0], x.v[1]), ff, v[q][0]);
    v[q][1] = __ffma2_rn(make_float2(x.v[2], x.v[3]), ff, v[q][1]);
  }
  __device__ __forceinline__ Vec16<float> get(int q) const {
    Vec16<float> o;
    o.v[0] = v[q][0].x; o.v[1] = v[q][0].y; o.v[2] = v[q][1].x; o.v[3] = v[q][1].y;
    return o;
  }
};

// One factor over the tile: [outer][P][inner][W] -> [outer][Q][inner][W].
template <typename T, int QB>
__device__ __forceinline__ void chainStep(const ChainArgs<T>& a, int k, const T* __restrict__ in, T* __restrict__ out,
                                          const T* __restrict__ Fs) {
  using V = Vec16<T>;
  constexpr int VEC = V::N, FB = (QB + VEC - 1) / VEC * VEC;
  const unsigned P = a.P[k], Q = a.Q[k], inner = a.inner[k].d, nb = a.nb[k].d;
  const unsigned logC = a.logW - (VEC == 4 ? 2 : 1);
  const unsigned items = (a.outer[k] * inner * nb) << logC;
  const unsigned step = inner * a.pitch, frow = nb * FB;
  for (unsigned it = threadIdx.x; it < items; it += kChainThreads) {
    const unsigned c = it & ((1u << logC) - 1), r = it >> logC;
    const unsigned r2 = quot(r, a.inner[k]), i = r - r2 * inner;
    const unsigned o = quot(r2, a.nb[k]), b = r2 - o * nb;
    const T* x = in + (o * P * inner + i) * a.pitch + c * VEC;
    const T* f = Fs + b * FB;
    ChainAcc<T, QB> acc;
    acc.clear();
#pragma unroll 4
    for (unsigned p = 0; p < P; p++) {
      const V xv = *reinterpret_cast<const V*>(x);
      V fv[FB / VEC];
#pragma unroll
      for (int g = 0; g < FB / VEC; g++) fv[g] = *reinterpret_cast<const V*>(f + g * VEC);
#pragma unroll
      for (int q = 0; q < QB; q++) acc.add(q, fv[q / VEC].v[q % VEC], xv);
      x += step; f += frow;
    }
    const unsigned q0 = b * QB;
    T* z = out + ((o * Q + q0) * inner + i) * a.pitch + c * VEC;
#pragma unroll
    for (int q = 0; q < QB; q++)
      if (q0 + q < Q) *reinterpret_cast<V*>(z + q * step) = acc.get(q);
  }
}

template <typename T>
__global__ void __launch_bounds__(kChainThreads, 3) chainKernel(const __grid_constant__ ChainArgs<T> a) {
  using V = Vec16<T>;
  constexpr int VEC = V::N;
  extern __shared__ __align__(1024) unsigned char smemRaw[];
  T* const bufA = reinterpret_cast<T*>(smemRaw);
  T* const bufB = reinterpret_cast<T*>(smemRaw + a.offB);
  T* const Fs = reinterpret_cast<T*>(smemRaw + a.offF);
  long long* const xo = reinterpret_cast<long long*>(smemRaw + a.offT);   // column offsets, -1 beyond the last position
  long long* const zo = xo + a.W;
  const unsigned tid = threadIdx.x;
  const unsigned logC = a.logW - (VEC == 4 ? 2 : 1);

  // factor k as [p][block][fb], blocks of qb outputs padded to whole vectors
  {
    T* d = Fs;
    for (int k = 0; k < a.nf; k++) {
      const unsigned row = a.nb[k].d * a.fb[k];
      const T* F = a.F[k];
      for (unsigned i = tid; i < a.P[k] * a.Q[k]; i += kChainThreads) {
        unsigned p, q;
        if (a.fsQ[k] == 1) { p = i / a.Q[k]; q = i - p * a.Q[k]; } else { q = i / a.P[k]; p = i - q * a.P[k]; }   // the stored order
        const unsigned b = q / a.qb[k];
        d[p * row + b * a.fb[k] + (q - b * a.qb[k])] = F[(long long)p * a.fsP[k] + (long long)q * a.fsQ[k]];
      }
      d += a.P[k] * row;
    }
  }

  for (unsigned tile = blockIdx.x; tile < a.numTiles; tile += gridDim.x) {
    __syncthreads();                                 // the previous tile has been stored
    if (tid < a.W) {
      const unsigned J = tile * a.W + tid;
      const unsigned r0 = J / a.n0, i0 = J - r0 * a.n0, i2 = r0 / a.n1, i1 = r0 - i2 * a.n1;
      const bool live = J < a.total;
      xo[tid] = live ? (long long)i0 * a.xs0 + (long long)i1 * a.xs1 + (long long)i2 * a.xs2 : -1;
      zo[tid] = live ? (long long)i0 * a.zs0 + (long long)i1 * a.zs1 + (long long)i2 * a.zs2 : -1;
    }
    __syncthreads();

    // ---- load --------------------------------------------------------------------------------
    const T* X = a.X;
    if (a.xsG == 1) {
      const unsigned units = a.G.d << logC;
#pragma unroll 4
      for (unsigned u = tid; u < units; u += kChainThreads) {
        const unsigned c = quot(u, a.G), g = u - c * a.G.d;
        V v;
#pragma unroll
        for (int e = 0; e < VEC; e++) {
          const long long off = xo[c * VEC + e];
          v.v[e] = off >= 0 ? X[off + g] : T(0);
        }
        *reinterpret_cast<V*>(bufA + g * a.pitch + c * VEC) = v;
      }
    } else if (a.vecX) {
      const unsigned units = a.G.d << logC;
      for (unsigned u = tid; u < units; u += kChainThreads) {
        const unsigned c = u & ((1u << logC) - 1), g = u >> logC;
        const long long off = xo[c * VEC];
        if (off >= 0) cpAsync16(bufA + g * a.pitch + c * VEC, X + off + (long long)g * a.xsG);
      }
    } else {
      const unsigned units = a.G.d << a.logW;
      for (unsigned u = tid; u < units; u += kChainThreads) {
        const unsigned c = u & (a.W - 1), g = u >> a.logW;
        const long long off = xo[c];
        if (off >= 0) {
          const unsigned s = (unsigned)__cvta_generic_to_shared(bufA + g * a.pitch + c);
          asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(s), "l"(X + off + (long long)g * a.xsG), "n"((int)sizeof(T)) : "memory");
        }
      }
    }
    cpAsyncWaitAll();
    __syncthreads();

    // ---- factors, last first --------------------------------------------------------------------
    const T* in = bufA;
    T* out = bufB;
    unsigned foff = 0;
    for (int k = 0; k < a.nf; k++) foff += a.P[k] * a.nb[k].d * a.fb[k];
    for (int k = a.nf - 1; k >= 0; k--) {
      foff -= a.P[k] * a.nb[k].d * a.fb[k];
      const T* f = Fs + foff;
      switch (a.qb[k]) {
        case 1: chainStep<T, 1>(a, k, in, out, f); break;
        case 2: chainStep<T, 2>(a, k, in, out, f); break;
        case 3: chainStep<T, 3>(a, k, in, out, f); break;
        case 4: chainStep<T, 4>(a, k, in, out, f); break;
        case 5: chainStep<T, 5>(a, k, in, out, f); break;
        case 6: chainStep<T, 6>(a, k, in, out, f); break;
        case 7: chainStep<T, 7>(a, k, in, out, f); break;
        default: chainStep<T, 8>(a, k, in, out, f); break;
      }
      __syncthreads();
      const T* done = out;
      out = const_cast<T*>(in);
      in = done;
    }

    // ---- store (alpha / beta*Y on the epilogue pass) -----------------------------------------------
    T* Z = a.Z;
    const bool epi = a.epilogue != 0;
    const bool useY = epi && a.beta != T(0) && a.Y != nullptr;
    const T* Y = a.Y;
    if (a.zsG == 1) {
      const unsigned units = a.H.d << logC;
      for (unsigned u = tid; u < units; u += kChainThreads) {
        const unsigned c = quot(u, a.H), h = u - c * a.H.d;
        V v = *reinterpret_cast<const V*>(in + h * a.pitch + c * VEC);
        T y[VEC];
#pragma unroll
        for (int e = 0; e < VEC; e++) {
          const long long off = zo[c * VEC + e];
          y[e] = useY && off >= 0 ? Y[off + h] : T(0);
        }
#pragma unroll
        for (int e = 0; e < VEC; e++) {
          const long long off = zo[c * VEC + e];
          if (epi) v.v[e] = a.alpha * v.v[e];
          if (useY) v.v[e] = fma(a.beta, y[e], v.v[e]);
          if (off >= 0) Z[off + h] = v.v[e];
        }
      }
    } else if (a.vecZ) {
      const unsigned units = a.H.d << logC;
#pragma unroll 2
      for (unsigned u = tid; u < units; u += kChainThreads) {
        const unsigned c = u & ((1u << logC) - 1), h = u >> logC;
        const long long off = zo[c * VEC];
        if (off < 0) continue;
        V v = *reinterpret_cast<const V*>(in + h * a.pitch + c * VEC);
        if (epi) {
#pragma unroll
          for (int e = 0; e < VEC; e++) v.v[e] = a.alpha * v.v[e];
          if (useY) {
            const V y = *reinterpret_cast<const V*>(Y + off + (long long)h * a.zsG);
#pragma unroll
            for (int e = 0; e < VEC; e++) v.v[e] = fma(a.beta, y.v[e], v.v[e]);
          }
        }
        *reinterpret_cast<V*>(Z + off + (long long)h * a.zsG) = v;
      }
    } else {
      const unsigned units = a.H.d << a.logW;
#pragma unroll 2
      for (unsigned u = tid; u < units; u += kChainThreads) {
        const unsigned c = u & (a.W - 1), h = u >> a.logW;
        const long long off = zo[c];
        if (off < 0) continue;
        T v = in[h * a.pitch + c];
        if (epi) v = a.alpha * v;
        if (useY) v = fma(a.beta, Y[off + (long long)h * a.zsG], v);
        Z[off + (long long)h * a.zsG] = v;
      }
    }
  }
}

template <typename T>
static fastKronError launchChainT(const Pass& ps, const LaunchCtx& cx) {
  constexpr int VEC = Vec16<T>::N;
  const uint64_t total = ps.M * ps.A * ps.B;
  ChainShape s;
  if (total == 0) return fastKronSuccess;
  if (cx.batch > 1 || cx.scatter.parts > 0 || cx.pSplit != 0 ||
      !chainShape(cx.dt, ps.nf, ps.P, ps.Q, ps.xsG == 1 || ps.zsG == 1, total, cx.smCount, &s))
    return fastKronKernelNotFound;
  ChainArgs<T> a;
  a.X = (const T*)cx.src; a.Z = (T*)cx.dst; a.Y = (const T*)cx.Y;
  a.nf = ps.nf;
  unsigned outer = 1, inner = 1;
  for (int k = 0; k < ps.nf; k++) {
    a.F[k] = (const T*)cx.F[k];
    a.P[k] = ps.P[k]; a.Q[k] = ps.Q[k]; a.qb[k] = s.qb[k]; a.fb[k] = s.fb[k]; a.nb[k] = fastDiv(s.nb[k]);
    // (p, q) of every factor lies as factor 0's stride pair says: one of the two is 1
    if (cx.fPMajor) { a.fsP[k] = ps.Q[k]; a.fsQ[k] = 1; } else { a.fsP[k] = 1; a.fsQ[k] = ps.P[k]; }
    a.outer[k] = outer;
    outer *= ps.P[k];
  }
  for (int k = ps.nf - 1; k >= 0; k--) { a.inner[k] = fastDiv(inner); inner *= ps.Q[k]; }
  a.G = fastDiv(s.G); a.H = fastDiv(s.H);
  a.W = s.W; a.pitch = s.pitch; a.offB = (unsigned)s.offB; a.offF = (unsigned)s.offF; a.offT = (unsigned)s.offT;
  a.logW = 0;
  while ((1u << a.logW) < a.W) a.logW++;
  PosDim d[3];
  orderPositions(ps, d);
  a.n0 = (unsigned)d[0].n; a.n1 = (unsigned)d[1].n;
  a.xs0 = d[0].xs; a.xs1 = d[1].xs; a.xs2 = d[2].xs; a.xsG = ps.xsG;
  a.zs0 = d[0].zs; a.zs1 = d[1].zs; a.zs2 = d[2].zs; a.zsG = ps.zsG;
  auto al16 = [](const void* p) { return ((uintptr_t)p & 15) == 0; };
  a.vecX = al16(a.X) && positionsVectorise(d, true, a.xsG, VEC);
  a.vecZ = al16(a.Z) && (a.Y == nullptr || al16(a.Y)) && positionsVectorise(d, false, a.zsG, VEC);
  a.alpha = (T)cx.alpha; a.beta = (T)cx.beta; a.epilogue = ps.epilogue ? 1 : 0;
  a.total = (unsigned)total;
  a.numTiles = (a.total + a.W - 1) / a.W;

  auto kern = chainKernel<T>;
  static bool attrDev[kMaxDevices] = {false};
  bool& attr = attrDev[currentDeviceSlot()];
  if (!attr) {
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kChainSmemMax);
    if (e != cudaSuccess) return cudaToFk(e);
    attr = true;
  }
  unsigned grid = (unsigned)cx.smCount * chainCtasPerSm(s.smem);
  if (grid > a.numTiles) grid = a.numTiles;
  kern<<<grid, kChainThreads, s.smem, cx.stream>>>(a);
  return cudaToFk(cudaGetLastError());
}

fastKronError launchChain(const Pass& ps, const LaunchCtx& cx) {
  return cx.dt == DType::F32 ? launchChainT<float>(ps, cx) : launchChainT<double>(ps, cx);
}

}  // namespace fkb
