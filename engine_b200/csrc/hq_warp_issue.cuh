// Copies, arrivals, commits and waits issued by a whole warp: the instruction is predicated on the lane elect.sync picks,
// the warp does not branch.  From a branch for one lane a tcgen05.mma costs about 75 cycles and a commit 125, whatever the
// width; a round {wait, arrive, copy} of an issuing warp stays a chain of about five hundred cycles, so what a round copies
// should be large, or several warps take the rounds in turn.
#pragma once
#include <cuda.h>

#include "hq_common.cuh"
#include "hq_ring.h"

namespace hq {

constexpr uint32_t kWaitSuspendNs = 20000;

__device__ __forceinline__ bool warp_test(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      "selp.u32 %0, 1, 0, p;\n"
      "}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait whose polls suspend the warp for long: twenty-odd warps that poll at the default rate keep the barrier unit
// busy enough to slow down the arrivals and copy instructions of the others.  A plain test goes first: on a phase that is
// complete already, the usual case in a ring that runs ahead, it takes 66 cycles, a try_wait with a time limit 100 to 127
// (65,536 x 4,096 at 16 rows on the dequantizing GEMM: Q4_K 69.9 -> 67.2 us, FP8 55.1 -> 52.8).
__device__ __forceinline__ bool warp_wait(uint64_t* bar, uint32_t parity, uint32_t spin_limit) {
  if (warp_test(bar, parity)) return true;
  for (uint32_t i = 0; i < spin_limit; ++i) {
    uint32_t ok;
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n"
        "selp.u32 %0, 1, 0, p;\n"
        "}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity), "r"(kWaitSuspendNs)
        : "memory");
    if (ok) return true;
  }
  return false;
}
// The same for the loops whose instruction count matters: no branch the compiler has to treat as divergent (its convergence
// barriers are instructions too), the outcome as a value.  Whole converged warps only.
__device__ __forceinline__ uint32_t warp_wait_uni(uint32_t bar, uint32_t parity, uint32_t spin_limit) {
  uint32_t ok;
  asm volatile(
      "{\n"
      ".reg .pred p, q;\n"
      ".reg .u32 n;\n"
      "mov.u32 %0, 1;\n"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      "vote.sync.all.pred p, p, 0xffffffff;\n"
      "@p bra.uni DONE;\n"
      "mov.u32 n, %3;\n"
      "POLL:\n"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %4;\n"
      "vote.sync.all.pred p, p, 0xffffffff;\n"
      "@p bra.uni DONE;\n"
      "setp.gt.u32 q, n, 1;\n"
      "sub.u32 n, n, 1;\n"
      "@q bra.uni POLL;\n"
      "mov.u32 %0, 0;\n"
      "DONE:\n"
      "}\n"
      : "=&r"(ok)
      : "r"(bar), "r"(parity), "r"(spin_limit), "r"(kWaitSuspendNs)
      : "memory");
  return ok;
}
// Remembers a wait that ran out (`spin` 0) in a word of shared memory, without a branch.
//
// An MMA-issuing warp must not branch on its waits' outcome: where the compiler has to take control flow for divergent, the
// operands of tcgen05.mma move from vector to uniform registers for every instruction, 120 to 140 cycles an MMA instead of 40
// to 70.  Such a warp keeps issuing after a time-out, on whatever its stages hold, and leaves this word for the warps that
// would store the products.
__device__ __forceinline__ void warp_mark_late(uint32_t word, uint32_t spin) {
  asm volatile(
      "{\n"
      ".reg .pred q;\n"
      "setp.eq.u32 q, %1, 0;\n"
      "@q st.shared.u32 [%0], 1;\n"
      "}\n" ::"r"(word),
      "r"(spin)
      : "memory");
}
// No copy may still be writing a CTA's shared memory when it exits: bounded wait of a copying warp for the stages ring_drain
// names (bar[slot] completes with a stage's copies).  On the normal path whoever reads the stages waits for the same.
__device__ __forceinline__ bool warp_drain(uint64_t* bar, int next, int slots, int slot, int parity, int warps, int me,
                                           uint32_t spin_limit) {
  return ring_drain(next, slots, slot, parity, warps, me, [&](int s, int ph) { return warp_wait(&bar[s], ph, spin_limit); });
}
// mbarrier arrivals by the elected lane of a whole warp, as a predicated instruction: a branch for one lane costs the
// other roles' warps instruction fetches (and this one several hundred cycles when it misses)
__device__ __forceinline__ void warp_arrive_at(uint32_t bar) {
  asm volatile(
      "{\n"
      ".reg .pred e;\n"
      "elect.sync _|e, 0xffffffff;\n"
      "@e mbarrier.arrive.shared::cta.b64 _, [%0];\n"
      "}\n" ::"r"(bar)
      : "memory");
}
__device__ __forceinline__ void warp_arrive(uint64_t* bar) { warp_arrive_at(smem_u32(bar)); }
// The same by a warp that keeps its waits' outcome in `spin` (warp_wait_uni): once one has run out it arrives no more, so whoever
// would take what it hands on runs out too, and stores nothing.  (A word of shared memory that the storing warps looked at per
// item cost the 64-token Q4_K layer 1 %.)
__device__ __forceinline__ void warp_arrive_live(uint64_t* bar, uint32_t spin) {
  asm volatile(
      "{\n"
      ".reg .pred e, q;\n"
      "elect.sync _|e, 0xffffffff;\n"
      "setp.ne.and.u32 q, %1, 0, e;\n"
      "@q mbarrier.arrive.shared::cta.b64 _, [%0];\n"
      "}\n" ::"r"(smem_u32(bar)), "r"(spin)
      : "memory");
}
__device__ __forceinline__ void warp_arrive_expect(uint64_t* bar, uint32_t bytes) {
  asm volatile(
      "{\n"
      ".reg .pred e;\n"
      "elect.sync _|e, 0xffffffff;\n"
      "@e mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n"
      "}\n" ::"r"(smem_u32(bar)),
      "r"(bytes)
      : "memory");
}

// box copies by the elected lane of a whole warp
__device__ __forceinline__ void warp_tma_3d(uint32_t dst, const CUtensorMap* map, int x, int y, int z, uint64_t* bar) {
  asm volatile(
      "{\n"
      ".reg .pred e;\n"
      "elect.sync _|e, 0xffffffff;\n"
      "@e cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];\n"
      "}\n" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
      : "memory");
}
__device__ __forceinline__ void warp_tma_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
  asm volatile(
      "{\n"
      ".reg .pred e;\n"
      "elect.sync _|e, 0xffffffff;\n"
      "@e cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];\n"
      "}\n" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(smem_u32(bar))
      : "memory");
}

// K-major operand tile of 128-byte rows, 128-byte swizzle, 8-row groups 1024 bytes apart, descriptor version 1
__device__ __forceinline__ uint64_t mx_smem_desc(uint32_t smem_addr) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_addr >> 4) & 0x3FFFu);
  d |= (uint64_t)1 << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}
// block-scaled products, kind::mxf8f6f4: one MMA of K = 32
__device__ __forceinline__ void warp_mx_mma(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t sfa,
                                            uint32_t sfb, uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p, e;\n"
      "elect.sync _|e, 0xffffffff;\n"
      "setp.ne.b32 p, %6, 0;\n"
      "@e tcgen05.mma.cta_group::1.kind::mxf8f6f4.block_scale.scale_vec::1X [%0], %1, %2, %3, [%4], [%5], p;\n"
      "}\n" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(sfa), "r"(sfb), "r"(accumulate)
      : "memory");
}
// 128 k of block-scaled products, kind::mxf8f6f4: four MMAs of K = 32, 32 bytes along the swizzled rows of both operands and one
// scale byte (instruction descriptor bits [4,6) of B, [29,31) of A) apart.  One election for the four: with one each, and their
// operands made one by one, an MMA took 101 to 140 cycles to issue where the tensor core needs 44 (48 columns) to 96 (192).
__device__ __forceinline__ void warp_mx_mma128(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t sfa, uint32_t sfb,
                                               uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p, e;\n"
      ".reg .b64 a1, b1;\n"
      ".reg .b32 i1;\n"
      "elect.sync _|e, 0xffffffff;\n"
      "setp.ne.b32 p, %6, 0;\n"
      "@e tcgen05.mma.cta_group::1.kind::mxf8f6f4.block_scale.scale_vec::1X [%0], %1, %2, %3, [%4], [%5], p;\n"
      "add.s64 a1, %1, 2;\n"
      "add.s64 b1, %2, 2;\n"
      "add.u32 i1, %3, 0x20000010;\n"
      "@e tcgen05.mma.cta_group::1.kind::mxf8f6f4.block_scale.scale_vec::1X [%0], a1, b1, i1, [%4], [%5], 1;\n"
      "add.s64 a1, %1, 4;\n"
      "add.s64 b1, %2, 4;\n"
      "add.u32 i1, %3, 0x40000020;\n"
      "@e tcgen05.mma.cta_group::1.kind::mxf8f6f4.block_scale.scale_vec::1X [%0], a1, b1, i1, [%4], [%5], 1;\n"
      "add.s64 a1, %1, 6;\n"
      "add.s64 b1, %2, 6;\n"
      "add.u32 i1, %3, 0x60000030;\n"
      "@e tcgen05.mma.cta_group::1.kind::mxf8f6f4.block_scale.scale_vec::1X [%0], a1, b1, i1, [%4], [%5], 1;\n"
      "}\n" ::"r"(d),
      "l"(a), "l"(b), "r"(idesc), "r"(sfa), "r"(sfb), "r"(accumulate)
      : "memory");
}

// tcgen05.commit by the elected lane
__device__ __forceinline__ void warp_commit(uint64_t* bar) {
  asm volatile(
      "{\n"
      ".reg .pred e;\n"
      "elect.sync _|e, 0xffffffff;\n"
      "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n"
      "}\n" ::"r"(smem_u32(bar))
      : "memory");
}

}  // namespace hq
