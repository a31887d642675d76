// What the kernels share that expand weights into tensor memory (gemm_tmem.cu, decode_tmem.cu): waits of whole warps, the one- and two-SM
// forms of the tensor-memory instructions, flags of partial tiles, tensor maps.
#pragma once
#include <cuda.h>

#include <cstdlib>

#include "common.cuh"
#include "umma.cuh"

namespace lb {
namespace {

using namespace umma;

constexpr int MAX_GRID = 160;
constexpr int SMEM_MAX = 227 * 1024 - 1024;   // dynamic; 1 KB is left for a kernel's static part, and one with more takes it off

// Which parts of the partial tiles are written: a flag per part (the kernels say which) holds the tag of the launch that wrote the
// part last.  A launch's tag is the epoch it finds, plus one; the last of its CTAs to have read the epoch raises it.  So no flag of an
// earlier launch ever matches, one that gave up and left flags without a reader included, and nothing is cleared between launches.
struct Sync {
  unsigned epoch, readers;
  unsigned flags[MAX_GRID * 64];
};

// ------------------------------------------------------------------------------------ PTX forms
__device__ __forceinline__ uint32_t mapa(uint32_t addr, uint32_t rank) { return map_to_rank(addr, rank); }
__device__ __forceinline__ void mbar_arrive_remote(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];\n" ::"r"(cluster_addr) : "memory");
}
// A value that all lanes of the warp hold alike, told to the compiler: what follows from such values, branches on them included, stays in the warp's uniform
// registers, where the operands of tcgen05.mma, its commits and TMA copies have to be.  From vector registers (a warp number as threadIdx.x >> 5, a
// quotient or an address read from shared memory is enough) every MMA took 48 to 58 clocks to issue and a commit 100, whatever their size; so an MMA
// takes 9 clocks with 16 columns, 16 with 32, 64 with 128: the tensor pipe's own.
__device__ __forceinline__ int same(int v) { return __shfl_sync(0xffffffffu, v, 0); }
__device__ __forceinline__ uint32_t same(uint32_t v) { return __shfl_sync(0xffffffffu, v, 0); }
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}\n" : "=r"(p));
  return p != 0;
}
// Looks for up to a hardware-set time (the thread sleeps meanwhile): a waiting warp takes no issue slots from the expanders.
// (Spinning, the four epilogue warps and the MMA warp issued a third of all instructions.)
__device__ __forceinline__ bool mbar_sleep_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// A whole warp waits, together: every lane looks and all branches are on votes, so the warp never diverges here (what
// follows are .aligned instructions and values the compiler keeps in the warp's uniform registers).
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity, volatile int *abort) {
  if (__all_sync(0xffffffffu, mbar_sleep_wait(bar, parity))) return true;
  const unsigned long long t0 = global_ns();
  while (!__all_sync(0xffffffffu, mbar_sleep_wait(bar, parity))) {
    if (__any_sync(0xffffffffu, *abort != 0)) return false;
    if (__any_sync(0xffffffffu, global_ns() - t0 > 1000000000ull)) {
      *abort = 1;
      return false;
    }
  }
  return true;
}
template <int CG>
__device__ __forceinline__ void alloc512(uint32_t smem_dst) {
  if constexpr (CG == 1) {
    tmem_alloc(smem_dst, 512);
    tmem_relinquish();
  } else {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;\n" ::"r"(smem_dst) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;\n" ::: "memory");
  }
}
template <int CG>
__device__ __forceinline__ void dealloc512(uint32_t taddr) {
  if constexpr (CG == 1) tmem_dealloc(taddr, 512);
  else asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;\n" ::"r"(taddr) : "memory");
}
// D[tmem] (+)= A[tmem] x B[smem]; with CG = 2 each CTA of the pair holds half of the rows of A and D and half of the
// columns (tokens) of B at the same addresses, and the first CTA issues for both
template <int CG>
__device__ __forceinline__ void mma_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  if constexpr (CG == 1)
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}\n" ::"r"(d_tmem),
        "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
  else
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}\n" ::"r"(d_tmem),
        "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
template <int CG>
__device__ __forceinline__ void commit(uint32_t bar) {  // CG = 2: on this barrier of both CTAs
  if constexpr (CG == 1) mma_commit(bar);
  else
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n" ::"r"(bar), "h"((uint16_t)3)
                 : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};\n" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]),
      "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory"); }

__device__ __forceinline__ bool wait_flag(const unsigned *flag, unsigned tag, bool mine, volatile int *abort) {  // whole warp, a flag to each lane that has one
  const unsigned long long t0 = global_ns();
  for (uint32_t i = 1;; i++) {
    unsigned v = tag;
    if (mine) asm volatile("ld.acquire.gpu.global.u32 %0, [%1];\n" : "=r"(v) : "l"(flag) : "memory");
    if (__all_sync(0xffffffffu, v == tag)) return true;
    if ((i & 15u) == 0) {
      if (__any_sync(0xffffffffu, *abort != 0)) return false;
      if (__any_sync(0xffffffffu, global_ns() - t0 > 1000000000ull)) break;
    }
  }
  *abort = 1;
  return false;
}

// ------------------------------------------------------------------------------------ host
typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                                  const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn encode_fn() {
  static const EncodeTiledFn fn = [] {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    const cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q);
    return e == cudaSuccess && q == cudaDriverEntryPointSuccess ? (EncodeTiledFn)p : (EncodeTiledFn) nullptr;
  }();
  return fn;
}
int knob(const char *name, int otherwise) {
  const char *e = getenv(name);
  return e ? atoi(e) : otherwise;
}

}  // namespace
}  // namespace lb
