// Exact expansion of int8 and packed int4 weights to bf16 pairs, shared by the kernels that read
// quantised weights.
#pragma once
#include <cuda_bf16.h>
#include <stdint.h>

namespace e2h {

// four signed bytes (one 32-bit word) -> two packed bf16x2 words, exactly.
// For a byte s = low7 - 128 * sign: bf16 bits 0x4300 | low7 are the number 128 + low7; subtracting
// bf16(128) = 0x4300 (sign clear) or bf16(256) = 0x4380 (sign set) leaves s. All three values
// are exact in bf16, so is the result.
__device__ __forceinline__ void cvt4_s8_bf16(uint32_t w, uint32_t& lo, uint32_t& hi) {
  const uint32_t t01 = __byte_perm(w, 0x43434343u, 0x5140);   // [0x43:s1 | 0x43:s0]
  const uint32_t t23 = __byte_perm(w, 0x43434343u, 0x5342);   // [0x43:s3 | 0x43:s2]
  const uint32_t x01 = t01 & 0x437F437Fu, c01 = (t01 & 0x00800080u) | 0x43004300u;
  const uint32_t x23 = t23 & 0x437F437Fu, c23 = (t23 & 0x00800080u) | 0x43004300u;
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
  const uint32_t t = ((w >> (4 * j)) & 0x000F000Fu) | 0x43004300u;
  const uint32_t c136 = 0x43084308u;                       // bf16(136) = 128 + 8, twice
  __nv_bfloat162 v = __hsub2(*reinterpret_cast<const __nv_bfloat162*>(&t),
                             *reinterpret_cast<const __nv_bfloat162*>(&c136));
  v = __hadd2_rn(__hmul2_rn(v, scale), zero);   // _rn: never contracted into one fused op
  return *reinterpret_cast<const uint32_t*>(&v);
}

}  // namespace e2h
