// bf16 image of a quantised weight matrix, for products of many tokens (one expansion pass, then the
// bf16 GEMM).
//
// Bound by memory: the codes are read once and 2 bytes per weight written. Every thread turns 8
// codes into one 16-byte store, so that both sides of a warp are contiguous, with kExpandVec such
// pieces in flight. Before, int8 went through a converting copy (22016 x 4096 codes: 119 us) and int4
// through nine element-wise passes over 32-bit codes (about 850 us for the same matrix).
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "quant_cvt.cuh"

namespace e2h {

constexpr int kExpandVec = 4;
constexpr int kExpandThreads = 256;

// QB = 8: src int8 [F, K], row pitch ld bytes. QB = 4: src packed nibbles (gemm_w8.cu), sz
// [K / g][F][2]. dst bf16 [F, K] dense, K % 8 == 0 (and g % 8 == 0).
template <int QB>
__global__ void __launch_bounds__(kExpandThreads)
expand_weight_kernel(const uint8_t* __restrict__ src, long long ld, const __nv_bfloat162* __restrict__ sz,
                     int groupsize, __nv_bfloat16* __restrict__ dst, int F, int K) {
  const int per_row = K >> 3;                       // pieces of 8 codes
  const long long total = (long long)F * per_row;
  const long long first = (long long)blockIdx.x * (kExpandThreads * kExpandVec) + threadIdx.x;
  uint2 raw[kExpandVec];
  __nv_bfloat162 pair[kExpandVec];
#pragma unroll
  for (int v = 0; v < kExpandVec; ++v) {
    const long long i = first + v * kExpandThreads;
    raw[v] = make_uint2(0u, 0u);
    if (i >= total) continue;
    const int f = (int)(i / per_row), w = (int)(i - (long long)f * per_row);
    const uint8_t* s = src + (long long)f * ld;
    if constexpr (QB == 8) {
      raw[v] = *reinterpret_cast<const uint2*>(s + (long long)w * 8);
    } else {
      raw[v].x = *reinterpret_cast<const uint32_t*>(s + (long long)w * 4);
      pair[v] = sz[(long long)((w * 8) / groupsize) * F + f];
    }
  }
#pragma unroll
  for (int v = 0; v < kExpandVec; ++v) {
    const long long i = first + v * kExpandThreads;
    if (i >= total) continue;
    uint32_t o[4];
    if constexpr (QB == 8) {
      cvt4_s8_bf16(raw[v].x, o[0], o[1]);
      cvt4_s8_bf16(raw[v].y, o[2], o[3]);
    } else {
      const __nv_bfloat162 sc = __bfloat162bfloat162(pair[v].x);
      const __nv_bfloat162 zr = __bfloat162bfloat162(pair[v].y);
#pragma unroll
      for (int j = 0; j < 4; ++j) o[j] = cvt2_u4_bf16(raw[v].x, j, sc, zr);
    }
    reinterpret_cast<uint4*>(dst)[i] = make_uint4(o[0], o[1], o[2], o[3]);
  }
}

}  // namespace e2h

// bits 8: src int8 [F, K] with row pitch ld (bytes, a multiple of 8), src 8-byte aligned. bits 4: src
// packed nibbles [F, K / 2] with row pitch ld (a multiple of 4), sz bf16 [K / groupsize][F][2],
// groupsize a multiple of 8. dst bf16 [F, K], 16-byte aligned, K % 8 == 0.
extern "C" int e2h_expand_weight(const void* src, long long ld, int bits, const void* sz,
                                 int groupsize, void* dst, int F, int K, void* stream_v) {
  using namespace e2h;
  if (F <= 0 || K <= 0 || (K % 8) || ((uintptr_t)dst & 15)) return -1;
  const long long total = (long long)F * (K / 8);
  const long long blocks = (total + kExpandThreads * kExpandVec - 1) / (kExpandThreads * kExpandVec);
  if (blocks > 0x7fffffffLL) return -2;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_v);
  if (bits == 8) {
    if (((uintptr_t)src & 7) || (ld % 8)) return -3;
    expand_weight_kernel<8><<<(unsigned)blocks, kExpandThreads, 0, stream>>>(
        static_cast<const uint8_t*>(src), ld, nullptr, 8, static_cast<__nv_bfloat16*>(dst), F, K);
  } else if (bits == 4) {
    if (((uintptr_t)src & 3) || (ld % 4) || sz == nullptr || groupsize <= 0 || (groupsize % 8) ||
        (K % groupsize) || ((uintptr_t)sz & 3))
      return -3;
    expand_weight_kernel<4><<<(unsigned)blocks, kExpandThreads, 0, stream>>>(
        static_cast<const uint8_t*>(src), ld, static_cast<const __nv_bfloat162*>(sz), groupsize,
        static_cast<__nv_bfloat16*>(dst), F, K);
  } else {
    return -4;
  }
  return (int)cudaGetLastError();
}
