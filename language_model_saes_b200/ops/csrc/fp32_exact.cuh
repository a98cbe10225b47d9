// fp32 arithmetic as IEEE 754 has it (subnormals included), and the error bound of the estimated products (fp32_gemm.cu).
#pragma once
#include "common.cuh"

namespace lmsae {

// (the intrinsics flush subnormals under this build's flags)
#define LMSAE_F32_OP(name, op)                                             \
  __device__ __forceinline__ float name(float a, float b) {                \
    float r;                                                               \
    asm(op " %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));                     \
    return r;                                                              \
  }
LMSAE_F32_OP(add_rn, "add.rn.f32")
LMSAE_F32_OP(mul_rn, "mul.rn.f32")
LMSAE_F32_OP(mul_up, "mul.rp.f32")
LMSAE_F32_OP(div_rn, "div.rn.f32")
#undef LMSAE_F32_OP
__device__ __forceinline__ float fma_rn(float a, float b, float c) {
  float r;
  asm("fma.rn.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

// Bound on the error of an estimated sum of K terms, relative to the product of the two rows' 2-norms (which bounds the sum of the
// magnitudes of its terms), in units of 2^-24 (what the parts add up to):
//   K          roundings of the sum in order that it stands for, one per term
//   17 K / 16  accumulations of the product of the high parts, sixteen terms an instruction: what is there and the sixteen products may each
//              lose a unit to the alignment; the two products of 2^-8 and less that come before it: 2 * 17 K / 16 / 128 at most
//   192        what the two parts leave of an operand (2^-18 of it, twice) and the product of the two low parts (2^-18)
//   128        the rounding of the ends themselves (a sum is at most about the product of the norms) and margin for what the hardware
//              does not document (measured: 2 units in all)
// The norms are rounded up where they are made, by 5 % (split_bf16_kernel) or 0.1 % (half_rows_kernel), which covers their own rounding (K / 64
// and less of these units). What is of second order is in the 2.1 K, of which the terms above take 2.08 K: parts may exceed their operands by 2^-9 each, 0.0042 K
// of the accumulations, and K 2^-24 times the K roundings in order is less than 0.0005 K.
__host__ __device__ __forceinline__ float estimate_rel(int K) { return ((float)K * 2.1f + 320.0f) * 5.9604645e-8f; }

// The same for one fp16 part an operand, its row scaled so that the largest magnitude is in [2^14, 2^15) (half_rows_kernel): 2.1 K and 128 as
// above (the accumulations are those of one product), 8 for the product of what the two operands lost (2^-11 of each at most), and
// to that what they lost itself, as it was measured: `lost` of the row and the largest of all columns.
__host__ __device__ __forceinline__ float estimate_rel_half(int K) { return ((float)K * 2.1f + 136.0f) * 5.9604645e-8f; }
__device__ __forceinline__ float half_rel(float rel, float lost, const uint32_t* most_lost) {
  return 1.000001f * (rel + lost + __uint_as_float(*most_lost));
}

}  // namespace lmsae
