// tcgen05 / mbarrier / bulk-copy building blocks shared by the tensor-core kernels (w4_tc5.cu,
// dense_gemm.cu).  Every wait is bounded.
#pragma once

#include <cstdint>

namespace tb {
namespace tc5 {

constexpr long long kWaitCycles = 4000000000ll;  // ~2 s

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void bulk_g2s(void* dst_smem, const void* src_gmem, uint32_t bytes, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst_smem)),
      "l"(src_gmem), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}
// Bounded wait: false (with the abort word and *fault raised) when the limit ran out here or elsewhere in the CTA.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile int* s_abort, int* fault) {
  const uint32_t addr = smem_u32(bar);
  long long t0 = 0;
  for (uint32_t i = 0;; ++i) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(addr), "r"(parity)
        : "memory");
    if (ok) return true;
    if ((i & 127) == 127) {
      if (*s_abort) return false;
      if (t0 == 0) t0 = clock64();
      else if (clock64() - t0 > kWaitCycles) {
        *s_abort = 1;
        atomicExch(fault, 1);
        return false;
      }
    }
  }
}
// Ready already (the usual case for the issuing thread)?  One instruction, no loop.
__device__ __forceinline__ bool mbar_ready(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// One lane of a converged warp.  MMAs and commits are issued inside `if (elect_one())`: the compiler knows that one thread
// runs there and takes their operands from uniform registers.  Behind `if (lane == 0)` it cannot know that and moves
// every operand with a loop over the active lanes: an MMA then costs its thread 123 cycles whatever its size, against 12.5
// (N = 16), 19 (N = 32), 34 (N = 64) and 126 (N = 256, the tensor pipe's own time), measured with M = 128, K = 16.
__device__ __forceinline__ bool elect_one() {
  uint32_t e;
  asm volatile("{\n\t.reg .pred e;\n\telect.sync _|e, 0xffffffff;\n\tselp.u32 %0, 1, 0, e;\n\t}" : "=r"(e));
  return e != 0;
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// Upper word of the shared-memory matrix descriptor of a K-major tile of 128-byte rows with the 128-byte
// swizzle: 1024 bytes between groups of 8 rows (bits 32-45, in 16-byte units), descriptor version 1 (bits
// 46-47), layout type 2 = SWIZZLE_128B (bits 61-63).  The lower word is the start address in 16-byte units
// (bits 0-13) and leading offset 1 (bits 16-29, unused with a swizzle).
constexpr uint32_t kDescHi = (uint32_t)(1024 >> 4) | (1u << 14) | (2u << 29);

// Arrives on `bar` once every MMA issued so far by this thread has finished.
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// 8 consecutive 32-bit columns of this thread's lane of tensor memory (no wait).
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}
// D (tensor memory, fp32) (+)= A (shared memory, bf16) * B (shared memory, bf16)^T; lower descriptor words.
__device__ __forceinline__ void mma_bf16_ss(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      ".reg .b64 ad, bd;\n\t"
      "setp.ne.b32 p, %5, 0;\n\t"
      "mov.b64 ad, {%1, %3};\n\t"
      "mov.b64 bd, {%2, %3};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], ad, bd, %4, p;\n\t"
      "}\n" ::"r"(d_tmem),
      "r"(a_lo), "r"(b_lo), "r"(kDescHi), "r"(idesc), "r"(acc)
      : "memory");
}

}  // namespace tc5
}  // namespace tb
