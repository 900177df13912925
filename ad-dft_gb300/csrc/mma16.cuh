// What the tcgen05 kernels share: mbarriers, bulk copies and tensor memory, then tcgen05.mma kind::f16 on no-swizzle
// K-major operands and digits, for the digit-slice kernels.
//
// The issuing warp runs its loop as a whole (uniform values stay in uniform registers) and one elected
// lane issues; an operand descriptor is a constant upper word and a lower word that offsets are added
// to.  Building 64-bit descriptors in one divergent lane cost 100 to 160 cycles per MMA beside
// busy warps; the MMAs themselves take 40 (N = 32) to 128 (N = 256) cycles.
#pragma once
#include "common.cuh"

namespace addft {

__device__ __forceinline__ uint32_t smem_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void bar_init(uint64_t *bar, int count = 1) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count));
}
__device__ __forceinline__ void bar_arrive(uint64_t *bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}
__device__ __forceinline__ void bar_expect(uint64_t *bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
}
// Bounded wait for the completion of the mbarrier phase with this parity; false when LIMIT looks did not see it.
template <int LIMIT>
__device__ __forceinline__ bool bar_wait(uint64_t *bar, uint32_t parity) {
  for (int it = 0; it < LIMIT; ++it) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.b32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}
// the barrier completes when the MMAs issued so far have
__device__ __forceinline__ void mma_commit(uint64_t *bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_addr(bar))
               : "memory");
}
__device__ __forceinline__ void bulk_copy(uint32_t dst, const void *src, uint32_t bytes, uint64_t *bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src),
      "r"(bytes), "r"(smem_addr(bar))
      : "memory");
}

__device__ __forceinline__ void tmem_alloc(uint32_t *slot, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(slot)), "r"(ncols));
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
}
__device__ __forceinline__ void tmem_free(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols));
}
#define TMEM_LD8(taddr, r)                                                                        \
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"           \
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), \
                 "=r"(r[7])                                                                      \
               : "r"(taddr))

// x 2^n as products with factors in range
__device__ __forceinline__ double scale2(double x, int n) {
  const int a = n / 2, b = n - a;
  auto p2 = [](int t) { return __hiloint2double((max(min(t, 1023), -1022) + 1023) << 20, 0); };
  return x * p2(a) * p2(b);
}

// Digit s of two numbers of S digits as FP16, in the halves of a word.  The numbers hold 128 more in every byte but the
// top one: 0x6400 + n is the FP16 number 1024 + n, and minus 1152 leaves the balanced digit, exactly.
template <int S>
__device__ __forceinline__ uint32_t digit_pair(uint64_t q0, uint64_t q1, int s) {
  uint32_t w, h;
  if (s == 0) {   // top digit: signed, -128 .. 128
    const int a = (int)((int64_t)q0 >> (8 * (S - 1))) + 128, b = (int)((int64_t)q1 >> (8 * (S - 1))) + 128;
    w = ((uint32_t)a | ((uint32_t)b << 16)) + 0x64006400u;
  } else {        // byte S - 1 - s of both numbers into the low bytes of the halves
    const int k = S - 1 - s, y = k & 3;
    const uint32_t a = (uint32_t)(q0 >> (k >= 4 ? 32 : 0)), b = (uint32_t)(q1 >> (k >= 4 ? 32 : 0));
    w = __byte_perm(__byte_perm(a, b, y | ((y + 4) << 4)), 0x64646464u, 0x4140);
  }
  asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(h) : "r"(w), "r"(0x64806480u));
  return h;
}

// lower descriptor word: start address and 128 B between the two core matrices of 16 k
__device__ __forceinline__ uint32_t desc_lo(uint32_t smem_addr) { return (smem_addr >> 4) | ((128u >> 4) << 16); }
// upper word: 256 B between 8-row groups, fixed 0b001, no swizzle
constexpr uint32_t kDescHi = (256u >> 4) | (1u << 14);

// instruction descriptor: FP16 operands, FP32 accumulator, M = 128
__host__ __device__ constexpr uint32_t idesc_f16(int N, bool neg_a) {
  return (1u << 4) | (neg_a ? 1u << 13 : 0u) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}

__device__ __forceinline__ void mma_f16(uint32_t d, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\tmov.b64 da, {%1, %4};\n\tmov.b64 db, {%2, %4};\n\t"
      "setp.ne.b32 p, %5, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %3, p;\n\t}" ::"r"(d),
      "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(kDescHi), "r"(acc)
      : "memory");
}

// true in one lane of the (converged) warp
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.b32 %0, 1, 0, p;\n\t}" : "=r"(p));
  return p != 0;
}

}  // namespace addft
