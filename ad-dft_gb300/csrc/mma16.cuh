// tcgen05.mma kind::f16 on no-swizzle K-major operands, for the digit-slice kernels.
//
// The issuing warp runs its loop as a whole (uniform values stay in uniform registers) and one elected
// lane issues; an operand descriptor is a constant upper word and a lower word that offsets are added
// to.  Building 64-bit descriptors in one divergent lane cost 100 to 160 cycles per MMA beside
// busy warps; the MMAs themselves take 40 (N = 32) to 128 (N = 256) cycles.
#pragma once
#include "common.cuh"

namespace addft {

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
