// tcgen05 / TMA helpers of the tensor-core kernels: mbarriers (every wait bounded), tensor copies, shared-memory matrix
// descriptors, MMA issue and TMEM reads.
#pragma once
#include <cuda.h>

#include "kernels.cuh"

namespace tsb {

constexpr unsigned kTcSpin = 1u << 22;

__device__ __forceinline__ uint32_t s_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void tc_mbar_init(uint64_t* bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(s_u32(bar)), "r"(count));
}
__device__ __forceinline__ void tc_mbar_expect_tx(uint64_t* bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(s_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool tc_mbar_wait(uint64_t* bar, unsigned parity) {
  const uint32_t a = s_u32(bar);
  for (unsigned i = 0; i < kTcSpin; ++i) {
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(a), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  return false;
}
// Shared-memory matrix descriptor (sm_100 format): start address, leading / stride byte offsets in 16-byte units,
// version 1, 128-byte swizzle.
__device__ __forceinline__ uint64_t make_desc(uint32_t smem_addr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_addr >> 4) & 0x3FFF);
  d |= (uint64_t)((lbo_bytes >> 4) & 0x3FFF) << 16;
  d |= (uint64_t)((sbo_bytes >> 4) & 0x3FFF) << 32;
  d |= (uint64_t)1 << 46;  // descriptor version (Blackwell)
  d |= (uint64_t)2 << 61;  // SWIZZLE_128B
  return d;
}
__device__ __forceinline__ void umma_f16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(s_u32(bar)) : "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t* r) {
  __syncwarp();
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
        "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
        "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
        "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// ---- the same for a whole warp -------------------------------------------------------------------------------------------
// One elected lane issues; the loop around it is the warp's.  In a branch of one lane every operand of these instructions, which live in
// uniform registers, is moved there one by one, and rebuilding 64-bit descriptors for each product made a step of four products 630 cycles
// of one thread's dependent instructions whatever their width (256 x 256: 512 of tensor time, 256 x 128: 256).  Descriptors are therefore a
// constant upper word and a lower word that only ever has offsets added (the address field cannot carry: shared memory ends below 2^18).
__device__ __forceinline__ bool elect_one() {
  uint32_t e;
  asm volatile("{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\tselp.u32 %0, 1, 0, q;\n\t}" : "=r"(e));
  return e != 0;
}
__device__ __forceinline__ uint32_t desc_lo(uint32_t smem_addr, uint32_t lbo_bytes) { return ((smem_addr >> 4) & 0x3FFF) | ((lbo_bytes >> 4) << 16); }
__device__ __forceinline__ uint32_t desc_hi(uint32_t sbo_bytes) { return (sbo_bytes >> 4) | (1u << 14) | (2u << 29); }
#define TSB_ELECTED_MMA(NAME, GROUP)                                                                                                        \
  __device__ __forceinline__ void NAME(uint32_t tmem_d, uint32_t a_lo, uint32_t a_hi, uint32_t b_lo, uint32_t b_hi, uint32_t idesc,       \
                                       uint32_t accumulate) {                                                                               \
    asm volatile(                                                                                                                           \
        "{\n\t.reg .pred p, q;\n\t.reg .b64 da, db;\n\t"                                                                                    \
        "elect.sync _|q, 0xffffffff;\n\t"                                                                                                  \
        "setp.ne.b32 p, %6, 0;\n\t"                                                                                                        \
        "mov.b64 da, {%1, %2};\n\tmov.b64 db, {%3, %4};\n\t"                                                                              \
        "@q tcgen05.mma.cta_group::" GROUP ".kind::f16 [%0], da, db, %5, p;\n\t}" ::"r"(tmem_d),                                           \
        "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate)                                                             \
        : "memory");                                                                                                                        \
  }
TSB_ELECTED_MMA(umma_el, "1")
TSB_ELECTED_MMA(umma_pair_el, "2")
#undef TSB_ELECTED_MMA
__device__ __forceinline__ void umma_commit_el(uint32_t bar) {
  asm volatile(
      "{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\t"
      "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(bar)
      : "memory");
}
// arrives at this barrier of both CTAs of a pair when the products issued so far are done
__device__ __forceinline__ void umma_commit_pair_el(uint32_t bar) {
  asm volatile(
      "{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\t"
      "@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n\t}" ::"r"(bar), "h"((uint16_t)3)
      : "memory");
}
__device__ __forceinline__ void tc_mbar_expect_el(uint32_t bar, unsigned bytes) {
  asm volatile("{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\t@q mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n\t}" ::"r"(bar), "r"(bytes) : "memory");
}
// takes `bytes` off what a phase waits for, as a copy that lands does
__device__ __forceinline__ void tc_mbar_complete_el(uint32_t bar, unsigned bytes) {
  asm volatile("{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\t@q mbarrier.complete_tx.relaxed.cta.shared::cta.b64 [%0], %1;\n\t}" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void tma_load_2d_el(uint32_t dst, const CUtensorMap* map, int c0, int c1, uint32_t bar) {
  asm volatile(
      "{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\t"
      "@q cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];\n\t}" ::"r"(dst),
      "l"(map), "r"(bar), "r"(c0), "r"(c1)
      : "memory");
}
__device__ __forceinline__ void tc_bulk_g2s_el(uint32_t dst, const void* src, unsigned bytes, uint32_t bar) {
  asm volatile(
      "{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\t"
      "@q cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n\t}" ::"r"(dst), "l"(src), "r"(bytes), "r"(bar)
      : "memory");
}
__device__ __forceinline__ bool tc_try_wait(uint32_t bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded; gives up early when another wait of the CTA has (*err), raises *err when it runs out itself.  For whole warps: their lanes poll for
// themselves and may see a phase end, or the error, at different polls, so the warp votes on each, and one answer sends all of it on or out of
// its loop (the elected issue behind it needs all lanes).
__device__ __forceinline__ bool tc_wait_or(uint32_t bar, unsigned parity, volatile int* err, unsigned limit = kTcSpin) {
  if (__all_sync(0xffffffffu, tc_try_wait(bar, parity))) return true;
#pragma unroll 1
  for (unsigned i = 1; i < limit; ++i) {
    if (__all_sync(0xffffffffu, tc_try_wait(bar, parity))) return true;
    if ((i & 63) == 63 && __any_sync(0xffffffffu, *err != 0)) return false;
  }
  *err = 1;
  return false;
}
__device__ __forceinline__ bool tc_wait_short(uint32_t bar, unsigned parity) {   // bounded, raises nothing
#pragma unroll 1
  for (unsigned i = 0; i < kTcSpin; ++i)
    if (tc_try_wait(bar, parity)) return true;
  return false;
}
// How a CTA may end, whichever of its waits has run out: its copies have landed (the copying warp sees to the last `asked` of a ring) and its
// products are done (the issuing warp waits for a commit behind them) before its shared memory and TMEM go to another CTA.  Both are waited
// for in every case and not upon an error flag, which another warp may raise after it was looked at; those warps have nothing else to do.
__device__ __forceinline__ void tc_land(uint32_t full, int stages, int asked) {
#pragma unroll 1
  for (int j = max(0, asked - stages); j < asked; ++j) tc_wait_short(full + (j % stages) * 8, (unsigned)((j / stages) & 1));
}
// what a warp's index is to the compiler: the same in all lanes
__device__ __forceinline__ int warp_index() { return __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0); }

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn get_encode();       // cuTensorMapEncodeTiled, or null where the driver has none

}  // namespace tsb
