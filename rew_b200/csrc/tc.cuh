// tcgen05 (5th-generation tensor core) inline-PTX wrappers shared by the kernels that keep an operand or
// the accumulator in tensor memory.
#pragma once
#include <stdint.h>

#include "ptx.cuh"

namespace rewb {
namespace tc {

// One lane of a converged warp, the same one every time, for roles of a single thread.  Measured against a branch on the lane's number, and
// together with issuing the four products of a 64-deep stage in one block of code (below): 148 CTAs, M = 128, cycles a product of 16 k,
// N = 16 to 128 lane test 90 (144 with descriptors built at run time), elected 49 to 64, elected and in fours 40 to 64; N = 256 128 in
// every form, which is the tensor core's own rate (N = 128: 64).  Likely cause: elect.sync tells the compiler that one lane is left, as a
// test of the lane's number does not, and these instructions take operands that are the same for a whole warp.
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
  return p != 0;
}

// Shared-memory operands as the two words of a descriptor.  The high word is the same for every operand of a kernel with one
// stride-byte-offset, the low word is (address >> 4) | (leading byte offset >> 4) << 16, so stepping an operand by `bytes` (a
// multiple of 16, inside the 256 KB window) is one 32-bit add of bytes >> 4.
__device__ __forceinline__ uint32_t desc_lo(uint32_t saddr, uint32_t lbo_bytes) {
  return ((saddr & 0x3FFFFu) >> 4) | ((lbo_bytes >> 4) << 16);
}
__device__ __forceinline__ constexpr uint32_t desc_hi(uint32_t sbo_bytes) { return (sbo_bytes >> 4) | (1u << 14) | (2u << 29); }

// Descriptor steps from one product of 16 k to the next inside a 128-byte swizzled tile, in units of 16 bytes
constexpr int K_MAJOR = 32 >> 4;      // k runs along the 128-byte rows
constexpr int MN_MAJOR = 2048 >> 4;   // k runs across them: two atoms of eight rows

// Four products in a row: D[tmem] (+)= A[smem] * B[smem] over 64 k; `accumulate` is about the first.  GROUP = 2: a pair of CTAs.
template <int A_STEP, int B_STEP, int GROUP = 1>
__device__ __forceinline__ void umma4_bf16_ss(uint32_t d_tmem, uint32_t alo, uint32_t blo, uint32_t hi, uint32_t idesc, uint32_t accumulate) {
#define REWB_UMMA4_SS(INSTR, MASK)                                                                                         \
  asm volatile(                                                                                                            \
      "{\n\t.reg .pred p, q;\n\t.reg .b32 u, v;\n\t.reg .b64 a0, a1, a2, a3, b0, b1, b2, b3;\n\t"                            \
      "setp.ne.b32 p, %5, 0;\n\tsetp.eq.b32 q, 0, 0;\n\t"                                                                 \
      "mov.b64 a0, {%1, %3};\n\tmov.b64 b0, {%2, %3};\n\t"                                                                \
      "add.u32 u, %1, %6;\n\tadd.u32 v, %2, %7;\n\tmov.b64 a1, {u, %3};\n\tmov.b64 b1, {v, %3};\n\t"                      \
      "add.u32 u, %1, 2 * %6;\n\tadd.u32 v, %2, 2 * %7;\n\tmov.b64 a2, {u, %3};\n\tmov.b64 b2, {v, %3};\n\t"              \
      "add.u32 u, %1, 3 * %6;\n\tadd.u32 v, %2, 3 * %7;\n\tmov.b64 a3, {u, %3};\n\tmov.b64 b3, {v, %3};\n\t" INSTR        \
      " [%0], a0, b0, %4, " MASK "p;\n\t" INSTR " [%0], a1, b1, %4, " MASK "q;\n\t" INSTR " [%0], a2, b2, %4, " MASK       \
      "q;\n\t" INSTR " [%0], a3, b3, %4, " MASK "q;\n\t}" ::"r"(d_tmem),                                                   \
      "r"(alo), "r"(blo), "r"(hi), "r"(idesc), "r"(accumulate), "n"(A_STEP), "n"(B_STEP), "r"(0u)                           \
      : "memory")
  if constexpr (GROUP == 1)
    REWB_UMMA4_SS("tcgen05.mma.cta_group::1.kind::f16", "");
  else
    REWB_UMMA4_SS("tcgen05.mma.cta_group::2.kind::f16", "{%8, %8, %8, %8, %8, %8, %8, %8}, ");
#undef REWB_UMMA4_SS
}
// The same with A in tensor memory (8 columns for 16 k)
template <int B_STEP>
__device__ __forceinline__ void umma4_bf16_ts(uint32_t d_tmem, uint32_t a_tmem, uint32_t blo, uint32_t hi, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t.reg .b32 v, a1, a2, a3;\n\t.reg .b64 b0, b1, b2, b3;\n\t"
      "setp.ne.b32 p, %5, 0;\n\tsetp.eq.b32 q, 0, 0;\n\t"
      "mov.b64 b0, {%2, %3};\n\t"
      "add.u32 v, %2, %6;\n\tmov.b64 b1, {v, %3};\n\tadd.u32 a1, %1, 8;\n\t"
      "add.u32 v, %2, 2 * %6;\n\tmov.b64 b2, {v, %3};\n\tadd.u32 a2, %1, 16;\n\t"
      "add.u32 v, %2, 3 * %6;\n\tmov.b64 b3, {v, %3};\n\tadd.u32 a3, %1, 24;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], b0, %4, p;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [a1], b1, %4, q;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [a2], b2, %4, q;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [a3], b3, %4, q;\n\t}" ::"r"(d_tmem),
      "r"(a_tmem), "r"(blo), "r"(hi), "r"(idesc), "r"(accumulate), "n"(B_STEP)
      : "memory");
}
__device__ __forceinline__ void commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// Takes `cols` columns of tensor memory for the CTA (GROUP = 2: for a pair of CTAs), by one whole warp, and then lets the stream's
// next launch start.  Always in this order, which is why no kernel that takes tensor memory calls pdl_launch_dependents itself:
// tcgen05.alloc waits without limit for columns that other CTAs of the SM hold.  Were a CTA to let later launches start first, one
// of them could take the columns it still needs and hold them while it waits for this launch to end: neither would.  In this order
// a launch starts only when every CTA of the launch ahead has its columns or has left, so whoever holds columns waits for launches
// that need no more of them, and they end.
template <int GROUP = 1>
__device__ __forceinline__ void alloc_then_launch_dependents(uint32_t* slot_in_smem, uint32_t cols) {
  if constexpr (GROUP == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot_in_smem)), "r"(cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  } else {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot_in_smem)), "r"(cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  pdl_launch_dependents();
}
__device__ __forceinline__ void dealloc(uint32_t base, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(base), "r"(cols) : "memory");
}
// 32 consecutive 32-bit columns of this thread's lane: tensor memory -> registers
__device__ __forceinline__ void ld32(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
// 16 of them
__device__ __forceinline__ void ld16(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
// registers -> 32 consecutive 32-bit columns of this thread's lane
__device__ __forceinline__ void st32(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
        "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]),
        "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]),
        "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

// The same without the wait: issue several, then wait_ld() / wait_st() once.
__device__ __forceinline__ void ld32_issue(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void st32_issue(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
        "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]),
        "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]),
        "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// registers -> 16 consecutive 32-bit columns of this thread's lane
__device__ __forceinline__ void st16(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
        "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

}  // namespace tc
}  // namespace rewb
