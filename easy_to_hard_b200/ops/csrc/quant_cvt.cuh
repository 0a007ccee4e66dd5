// Exact expansion of int8 and packed int4 weights to bf16 pairs, shared by the kernels that read
// quantised weights.
#pragma once
#include <cuda_bf16.h>
#include <stdint.h>

namespace e2h {

// These few instructions are what the kernels of quantised weights wait for: bitwise and permute
// instructions take two cycles of a scheduler's ALU each. Counted in a loop of conversions, four warps per
// scheduler, cycles per word: int8 15.9 -> 11.5 with the bits split before the permutes and not after, int4
// 30.3 -> 25.3 with `and` and `or` as the one instruction that the compiler does not make of them where
// both operands are constants.
__device__ __forceinline__ uint32_t and_or(uint32_t x, uint32_t mask, uint32_t bits) {
  uint32_t d;
  asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(d) : "r"(x), "r"(mask), "r"(bits));
  return d;
}

// four signed bytes (one 32-bit word) -> two packed bf16x2 words, exactly.
// For a byte s = low7 - 128 * sign: bf16 bits 0x4300 | low7 are the number 128 + low7; subtracting
// 0x4300 | sign bit, which is bf16(128) (sign clear) or bf16(256) (sign set), leaves s. All three values
// are exact in bf16, so is the result.
__device__ __forceinline__ void cvt4_s8_bf16(uint32_t w, uint32_t& lo, uint32_t& hi) {
  const uint32_t low7 = w & 0x7F7F7F7Fu, sign = w & 0x80808080u;
  const uint32_t x01 = __byte_perm(low7, 0x43434343u, 0x5140);   // [0x43:low7 of s1 | 0x43:low7 of s0]
  const uint32_t c01 = __byte_perm(sign, 0x43434343u, 0x5140);
  const uint32_t x23 = __byte_perm(low7, 0x43434343u, 0x5342);
  const uint32_t c23 = __byte_perm(sign, 0x43434343u, 0x5342);
  const __nv_bfloat162 r01 = __hsub2(*reinterpret_cast<const __nv_bfloat162*>(&x01),
                                     *reinterpret_cast<const __nv_bfloat162*>(&c01));
  const __nv_bfloat162 r23 = __hsub2(*reinterpret_cast<const __nv_bfloat162*>(&x23),
                                     *reinterpret_cast<const __nv_bfloat162*>(&c23));
  lo = *reinterpret_cast<const uint32_t*>(&r01);
  hi = *reinterpret_cast<const uint32_t*>(&r23);
}

// four unsigned nibbles -> exact bf16 (q - 8) * scale + zero with a rounding after every step,
// the arithmetic of the reference's int4 linear ((q - 8) * scales + zeros in bf16,
// models/quantize.py:108-116). The packed word holds 8 consecutive k as
// sum_j q[2j] << 4j | q[2j+1] << (16 + 4j), so (w >> 4j) & 0x000F000F is the pair (2j, 2j+1)
// already in bf16x2 position: OR-ing 0x4300 makes each half the bf16 number 128 + q.
__device__ __forceinline__ uint32_t cvt2_u4_bf16(uint32_t w, int j, __nv_bfloat162 scale,
                                                 __nv_bfloat162 zero) {
  const uint32_t t = and_or(w >> (4 * j), 0x000F000Fu, 0x43004300u);
  const uint32_t c136 = 0x43084308u;                       // bf16(136) = 128 + 8, twice
  __nv_bfloat162 v = __hsub2(*reinterpret_cast<const __nv_bfloat162*>(&t),
                             *reinterpret_cast<const __nv_bfloat162*>(&c136));
  v = __hadd2_rn(__hmul2_rn(v, scale), zero);   // _rn: never contracted into one fused op
  return *reinterpret_cast<const uint32_t*>(&v);
}

}  // namespace e2h
