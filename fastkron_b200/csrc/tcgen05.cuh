// Primitives shared by the tensor-core kernels (kernel_gemm_tc.cu, kernel_gemm_split.cu):
// mbarriers with bounded waits, shared-memory matrix descriptors, tcgen05 loads, stores, fences
// and commits.  One CTA, no cluster launch, no multicast.
#pragma once

#include <cuda_runtime.h>

namespace fkb {
namespace tc {

// Set when a bounded wait on a barrier gave up.  One copy per translation unit.
static __device__ int gTcTimeouts = 0;

__device__ __forceinline__ unsigned smemAddr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbarInit(unsigned long long* bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smemAddr(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbarExpectTx(unsigned long long* bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smemAddr(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbarArrive(unsigned long long* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(smemAddr(bar)) : "memory");
}
__device__ __forceinline__ bool mbarTryWait(unsigned long long* bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok) : "r"(smemAddr(bar)), "r"(parity) : "memory");
  return ok != 0;
}
// About two seconds at most; also gives up as soon as another role has raised the abort flag.
__device__ __forceinline__ bool waitBounded(unsigned long long* bar, unsigned parity, volatile int* abortFlag) {
  if (mbarTryWait(bar, parity)) return true;
  const long long t0 = clock64();
  while (!mbarTryWait(bar, parity)) {
    if (*abortFlag) return false;
    if (clock64() - t0 > 4000000000ll) { *abortFlag = 1; atomicExch(&gTcTimeouts, 1); return false; }
  }
  return true;
}

// Shared-memory matrix descriptor of tcgen05.mma: start address, leading and stride byte
// offsets (all in 16-byte units), descriptor version 1, swizzle mode.
//   kSwz128: rows of 128 bytes, 16-byte units XOR (row % 8); used for K-major operands
//            (8 rows per atom; SBO = distance between 8-row groups).
//   kSwz128Atom32: rows of 128 bytes, 32-byte units XOR (row % 4); the only swizzle TF32
//            operands may have when their M / N index is the contiguous one.  A row is one k,
//            an atom is 4 rows: SBO = distance between atoms along k (512 bytes for packed
//            rows), LBO = distance between atoms of 32 elements along M / N.
constexpr unsigned long long kSwz128 = 2, kSwz128Atom32 = 1;
__device__ __forceinline__ unsigned long long smemDesc(unsigned addr, unsigned lboBytes, unsigned sboBytes,
                                                       unsigned long long swizzle) {
  return (unsigned long long)((addr & 0x3FFFFu) >> 4) | ((unsigned long long)(lboBytes >> 4) << 16) |
         ((unsigned long long)(sboBytes >> 4) << 32) | (1ull << 46) | (swizzle << 61);
}
__device__ __forceinline__ void mmaCommit(unsigned long long* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(smemAddr(bar)) : "memory");
}
__device__ __forceinline__ void tmemLoad32(unsigned taddr, unsigned (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmemLoad16(unsigned taddr, unsigned (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmemLoadWait() { asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory"); }
__device__ __forceinline__ void tmemStore8(unsigned taddr, const unsigned (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};\n" ::"r"(taddr), "r"(r[0]), "r"(r[1]),
               "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}
__device__ __forceinline__ void tmemStoreWait() { asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory"); }
__device__ __forceinline__ void fenceBeforeSync() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void fenceAfterSync() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }

}  // namespace tc
}  // namespace fkb
