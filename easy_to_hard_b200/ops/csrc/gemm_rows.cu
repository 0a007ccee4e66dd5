// Products of a few rows (T <= 16) with bf16, int8 or int4 weights: a weight stream.
//
// What bounds it is HBM, so the layout is chosen for bytes in flight and for little fixed cost, not
// for tensor throughput (a decode step of one row needs a hundredth of the tensor peak):
//   * a warp owns MT x 16 weight rows and a slice of K; the warps of a CTA split K, their partial
//     sums meet in shared memory, and one warp runs the epilogue (gemm_epilogue.cuh: a lane owns a
//     feature). No tensor memory, TMA descriptors, barriers or clusters to set up: the tcgen05 kernel
//     (gemm_umma.cu) spends about 7 us per launch on those and one CTA of it fills an SM, so that
//     the next kernel's loads begin when it exits; CTAs of this kernel come and go one by one;
//   * weights go straight from global memory into the A fragments of mma.m16n8k16. The sum over k
//     may be taken in any order, so lane (g, t) takes 16 consecutive bytes of rows g and g + 8 and
//     the same k of activation row g as its B fragment: every load is 16 bytes wide and nothing is
//     exchanged between lanes. int8 and int4 codes are expanded in registers, exactly as in the
//     converting kernel (gemm_w8.cu), whose round trip through tensor memory held 8 rows of int4
//     to an eighth of the bandwidth;
//   * every lane copies its vectors to shared memory with cp.async and reads back what it copied
//     itself: bytes in flight are bound by shared memory instead of registers (a double buffer in
//     registers held 22016 x 4096 int8 weights to 25 us where this takes 21), and no barrier is
//     needed. The first ring is filled before the wait for the preceding kernel (weights are never
//     written by a predecessor of a PDL chain);
//   * activations come through L1 and L2 the same way, T rows of them for every tile: from 9 rows on
//     they are what long sums wait for (rows_pays in ops/gemm.py).
//
// Time per launch in a chain of launches with distinct weights (L2 cold), tcgen05 kernel -> this one:
//                                     bf16, 1 row     bf16, 16 rows   int8, 8 rows    int4, 8 rows
//   12288 x 4096                      33.8 -> 21.3    26.2 -> 22.4    30.0 -> 15.6    29.7 -> 14.6 us
//   4096 x 4096 + residual            12.6 ->  7.4    12.7 -> 10.3    13.5 ->  7.8    13.6 ->  7.5
//   2 x 11008 x 4096, gated           47.4 -> 30.4    42.7 -> 35.7    50.6 -> 22.4    49.9 -> 20.7
//   4096 x 11008 + residual           21.9 -> 16.4    (not taken)     22.9 -> 13.7    22.5 -> 14.6
//   256 x 256                          6.0 ->  1.8
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include "gemm_epilogue.cuh"
#include "gemm_umma.cuh"
#include "launch.cuh"
#include "ptx.cuh"
#include "quant_cvt.cuh"

namespace e2h {

constexpr int kRowsMaxWarps = 8;

// 16 (or 4) bytes from global to shared memory, zeros where `in` is false; nothing is read then.
__device__ __forceinline__ void cp_async16_once(uint32_t dst, const void* src, bool in, uint64_t policy) {
  asm volatile("cp.async.cg.shared.global.L2::cache_hint.L2::256B [%0], [%1], 16, %2, %3;" ::"r"(dst),
               "l"(src), "r"(in ? 16 : 0), "l"(policy)
               : "memory");
}
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool in) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(in ? 16 : 0)
               : "memory");
}
__device__ __forceinline__ void cp_async4(uint32_t dst, const void* src, bool in) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(in ? 4 : 0)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

__device__ __forceinline__ void mma_bf16(float* c, uint32_t a0, uint32_t a1, uint32_t a2,
                                         uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, "
      "{%8, %9}, {%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// One unit: 16 bytes of each of the warp's rows per lane, KU = 64 / bits * 8 consecutive k of 4 lanes.
template <int QB>
struct RowsUnit {
  static constexpr int k_lane = 128 / QB;      // k per lane: 8, 16, 32
  static constexpr int k = 4 * k_lane;         // 32, 64, 128
  static constexpr int b_vec = k_lane / 8;     // 16-byte activation vectors per lane: 1, 2, 4
};

// Shared memory of one warp: a ring of S stages of UN units, a unit being the lane-major vectors
// [MT][2] of A, [NT][b_vec] of B and, for int4, [MT][2] (scale, zero) pairs. RB bytes of it at most: 12 KB,
// with which 16 warps share an SM, or 8 KB for 24.
template <int QB, int MT, int NT, int RB>
struct RowsRing {
  using U = RowsUnit<QB>;
  static constexpr int a_bytes = MT * 2 * 512, b_bytes = NT * U::b_vec * 512;
  static constexpr int unit_bytes = a_bytes + b_bytes + (QB == 4 ? MT * 2 * 128 : 0);
  static constexpr int UN = QB == 16 && MT == 1 && RB > 8192 ? 2 : 1;
  static constexpr int stage_bytes = UN * unit_bytes;
  static constexpr int want = RB / stage_bytes;
  static constexpr int S = want < 2 ? 2 : want > 8 ? 8 : want;
  static constexpr int bytes = S * stage_bytes;
};

// QB: bits per weight. MT: 16-row tiles of a warp (a gated product: tile 0 of A above tile 0 of A2).
// NT: groups of 8 rows of B. SHARE: CTAs take equal shares instead of whole tiles.
template <int QB, int MT, int NT, bool DUAL, int RB, bool SHARE>
__global__ void __launch_bounds__(kRowsMaxWarps * 32, 2) gemm_rows_kernel(const E2hGemmParams p) {
  using U = RowsUnit<QB>;
  using R = RowsRing<QB, MT, NT, RB>;
  static_assert(!DUAL || MT == 2, "a gated product pairs two tiles");
  constexpr int FT = DUAL ? 16 : 16 * MT;      // output features of a CTA
  constexpr int PITCH = 8 * NT + 4;            // floats per feature in the exchange buffer
  static_assert(MT * 16 * PITCH * 4 <= R::bytes, "the exchange buffer reuses the ring");
  extern __shared__ __align__(128) uint8_t rows_smem[];

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const int g = lane >> 2, t4 = lane & 3;
  // this CTA's features: a tile, or an equal share of at most as many, in pairs (the rotation turns pairs)
  int f0 = blockIdx.x * FT, f1 = f0 + FT;
  if constexpr (SHARE) {
    const long long pairs = (p.F + 1) / 2;
    f0 = 2 * (int)(blockIdx.x * pairs / gridDim.x);
    f1 = min(2 * (int)((blockIdx.x + 1) * pairs / gridDim.x), p.F);
  }
  pdl_launch_dependents();

  // this lane's rows (one past the share is not loaded, and masked at the end)
  const uint8_t* arow[MT][2];
  int frow[MT][2];
  bool own[MT][2];
#pragma unroll
  for (int m = 0; m < MT; ++m) {
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const int at = f0 + (DUAL ? 0 : 16 * m) + g + 8 * r, f = min(at, p.F - 1);
      own[m][r] = !SHARE || at < f1;
      const void* base = (DUAL && m == 1) ? p.a2 : p.a;
      const long long ld = (DUAL && m == 1) ? p.lda2 : p.lda;   // bf16: elements, else bytes
      frow[m][r] = f;
      arow[m][r] = static_cast<const uint8_t*>(base) + (long long)f * ld * (QB == 16 ? 2 : 1) +
                   t4 * 16;
    }
  }
  const __nv_bfloat16* brow[NT];
#pragma unroll
  for (int n = 0; n < NT; ++n)
    brow[n] = static_cast<const __nv_bfloat16*>(p.b) + (long long)min(8 * n + g, p.T - 1) * p.ldb +
              t4 * U::k_lane;
  const int units = (p.K + U::k - 1) / U::k;
  const int u0 = (int)((long long)warp * units / nw), u1 = (int)((long long)(warp + 1) * units / nw);
  const int gshift = QB == 4 ? __ffs(p.groupsize) - 1 : 0;

  const uint64_t once = policy_evict_first();
  uint8_t* ring = rows_smem + warp * R::bytes;
  const uint32_t ring_a = smem_u32(ring) + lane * 16, ring_z = smem_u32(ring) + lane * 4;
  // stage s of the ring <- units u .. u + UN - 1
  auto load_a = [&](int s, int u) {
#pragma unroll
    for (int i = 0; i < R::UN; ++i) {
      const bool in = u + i < u1 && (u + i) * U::k + t4 * U::k_lane < p.K;
      const uint32_t dst = s * R::stage_bytes + i * R::unit_bytes;
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const bool mine = in && own[m][r];
          cp_async16_once(ring_a + dst + (m * 2 + r) * 512,
                          mine ? arow[m][r] + (long long)(u + i) * 64 : arow[m][r], mine, once);
          if constexpr (QB == 4) {
            const __nv_bfloat162* z =
                static_cast<const __nv_bfloat162*>((DUAL && m == 1) ? p.qsz2 : p.qsz);
            const long long grp = in ? ((u + i) * U::k + t4 * U::k_lane) >> gshift : 0;
            cp_async4(ring_z + dst + R::a_bytes + R::b_bytes + (m * 2 + r) * 128,
                      z + grp * p.F + frow[m][r], in);
          }
        }
    }
  };
  auto load_b = [&](int s, int u) {
#pragma unroll
    for (int i = 0; i < R::UN; ++i) {
      const bool in = u + i < u1 && (u + i) * U::k + t4 * U::k_lane < p.K;
      const uint32_t dst = ring_a + s * R::stage_bytes + i * R::unit_bytes + R::a_bytes;
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int v = 0; v < U::b_vec; ++v)
          cp_async16(dst + (n * U::b_vec + v) * 512, in ? brow[n] + (u + i) * U::k + 8 * v : brow[n],
                     in && 8 * n + g < p.T);
    }
  };

  float acc[MT][NT][4];
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[m][n][j] = 0.f;

  // weights are never written by a predecessor of a PDL chain: they stream before the wait
#pragma unroll
  for (int s = 0; s < R::S; ++s) load_a(s, u0 + s * R::UN);
  pdl_wait_prior();
#pragma unroll
  for (int s = 0; s < R::S; ++s) {
    load_b(s, u0 + s * R::UN);
    cp_async_commit();
  }
  int s = 0;
  for (int u = u0; u < u1; u += R::UN) {
    cp_async_wait<R::S - 1>();          // every lane reads back what it copied itself
    const uint8_t* st = ring + s * R::stage_bytes + lane * 16;
#pragma unroll
    for (int i = 0; i < R::UN; ++i, st += R::unit_bytes) {
      uint32_t b[NT][U::b_vec * 4];
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int v = 0; v < U::b_vec; ++v)
          *reinterpret_cast<uint4*>(&b[n][4 * v]) =
              *reinterpret_cast<const uint4*>(st + R::a_bytes + (n * U::b_vec + v) * 512);
#pragma unroll
      for (int m = 0; m < MT; ++m) {
        uint32_t lo[4], hi[4];
        *reinterpret_cast<uint4*>(lo) = *reinterpret_cast<const uint4*>(st + m * 1024);
        *reinterpret_cast<uint4*>(hi) = *reinterpret_cast<const uint4*>(st + m * 1024 + 512);
        if constexpr (QB == 16) {
#pragma unroll
          for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int n = 0; n < NT; ++n)
              mma_bf16(acc[m][n], lo[2 * h], hi[2 * h], lo[2 * h + 1], hi[2 * h + 1], b[n][2 * h],
                       b[n][2 * h + 1]);
        } else if constexpr (QB == 8) {
#pragma unroll
          for (int w = 0; w < 4; ++w) {
            uint32_t l0, l1, h0, h1;
            cvt4_s8_bf16(lo[w], l0, l1);
            cvt4_s8_bf16(hi[w], h0, h1);
#pragma unroll
            for (int n = 0; n < NT; ++n)
              mma_bf16(acc[m][n], l0, h0, l1, h1, b[n][2 * w], b[n][2 * w + 1]);
          }
        } else {
          const uint8_t* zp = st - lane * 12 + R::a_bytes + R::b_bytes + m * 256;
          const __nv_bfloat162 pl = *reinterpret_cast<const __nv_bfloat162*>(zp);
          const __nv_bfloat162 ph = *reinterpret_cast<const __nv_bfloat162*>(zp + 128);
          const __nv_bfloat162 sl = __bfloat162bfloat162(pl.x), zl = __bfloat162bfloat162(pl.y);
          const __nv_bfloat162 sh = __bfloat162bfloat162(ph.x), zh = __bfloat162bfloat162(ph.y);
#pragma unroll
          for (int w = 0; w < 4; ++w)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const uint32_t l0 = cvt2_u4_bf16(lo[w], 2 * h, sl, zl);
              const uint32_t l1 = cvt2_u4_bf16(lo[w], 2 * h + 1, sl, zl);
              const uint32_t h0 = cvt2_u4_bf16(hi[w], 2 * h, sh, zh);
              const uint32_t h1 = cvt2_u4_bf16(hi[w], 2 * h + 1, sh, zh);
#pragma unroll
              for (int n = 0; n < NT; ++n)
                mma_bf16(acc[m][n], l0, h0, l1, h1, b[n][4 * w + 2 * h], b[n][4 * w + 2 * h + 1]);
            }
        }
      }
    }
    // the stage has been read into registers that the products above consumed
    load_a(s, u + R::S * R::UN);
    load_b(s, u + R::S * R::UN);
    cp_async_commit();
    if (++s == R::S) s = 0;
  }
  cp_async_wait<0>();
  __syncwarp();
  float* red = reinterpret_cast<float*>(ring);   // this warp's partial sums, over its own ring

  // partial sums [feature][token]; accumulator rows g and g + 8, columns 2 t4 and 2 t4 + 1
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int r = 0; r < 2; ++r)
        *reinterpret_cast<float2*>(
            &red[(m * 16 + g + 8 * r) * PITCH + 8 * n + 2 * t4]) =
            make_float2(acc[m][n][2 * r], acc[m][n][2 * r + 1]);
  __syncthreads();
  if (warp >= NT || 8 * warp >= p.T) return;

  // epilogue: warp n finishes tokens 8 n .. 8 n + 7, a lane owns a feature
  const bool lane_ok = lane < f1 - f0;
  const int row = lane_ok ? lane : 0;
  float v[8], v2[DUAL ? 8 : 1];
#pragma unroll
  for (int j = 0; j < 8; ++j) v[j] = 0.f;
  if constexpr (DUAL) {
#pragma unroll
    for (int j = 0; j < 8; ++j) v2[j] = 0.f;
  }
  for (int w = 0; w < nw; ++w) {
    const float* src = reinterpret_cast<const float*>(rows_smem + w * R::bytes) + row * PITCH + 8 * warp;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const float4 q = *reinterpret_cast<const float4*>(src + 4 * h);
      v[4 * h] += q.x; v[4 * h + 1] += q.y; v[4 * h + 2] += q.z; v[4 * h + 3] += q.w;
      if constexpr (DUAL) {
        const float4 q2 = *reinterpret_cast<const float4*>(src + 16 * PITCH + 4 * h);
        v2[4 * h] += q2.x; v2[4 * h + 1] += q2.y; v2[4 * h + 2] += q2.z; v2[4 * h + 3] += q2.w;
      }
    }
  }
  epilogue8<DUAL>(p, lane_ok ? f0 + lane : p.F, 8 * warp, v, v2, p.T);
}

template <int QB, int MT, int NT, bool DUAL, int RB, bool SHARE>
static int rows_launch(const E2hGemmParams& p, int ctas, int warps, cudaStream_t stream) {
  auto kern = gemm_rows_kernel<QB, MT, NT, DUAL, RB, SHARE>;
  constexpr int warp_bytes = RowsRing<QB, MT, NT, RB>::bytes;
  static SmemAsk ask;
  const cudaError_t e = ask(kern, kRowsMaxWarps * warp_bytes);
  if (e != cudaSuccess) return (int)e;
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3(ctas, 1, 1);
  cfg.blockDim = dim3(32 * warps, 1, 1);
  cfg.dynamicSmemBytes = (size_t)warps * warp_bytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  if (p.pdl || g_pdl) {
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.numAttrs = 1;
  }
  cfg.attrs = attr;
  return (int)cudaLaunchKernelEx(&cfg, kern, p);
}

template <int QB, int NT>
static int rows_dispatch(const E2hGemmParams& p, int mt, int ctas, int warps, bool share,
                         bool short_ring, cudaStream_t stream) {
  if (p.dual) return rows_launch<QB, 2, NT, true, 12288, false>(p, ctas, warps, stream);
  if constexpr (QB == 16 && NT == 1) {
    if (short_ring && mt == 2) return rows_launch<QB, 2, NT, false, 8192, true>(p, ctas, warps, stream);
    if (short_ring) return rows_launch<QB, 1, NT, false, 8192, true>(p, ctas, warps, stream);
  }
  if constexpr (QB == 8 || (QB == 16 && NT == 1)) {
    if (share && mt == 2) return rows_launch<QB, 2, NT, false, 12288, true>(p, ctas, warps, stream);
  }
  if constexpr (QB != 4 && NT == 1) {
    if (share) return rows_launch<QB, 1, NT, false, 12288, true>(p, ctas, warps, stream);
  }
  if (mt == 2) return rows_launch<QB, 2, NT, false, 12288, false>(p, ctas, warps, stream);
  return rows_launch<QB, 1, NT, false, 12288, false>(p, ctas, warps, stream);
}

}  // namespace e2h

// The parameter block of e2h_gemm_umma (K-major operands, no groups, batches, signals or row-major
// outputs), T <= 16. bits: 16 bf16 weights (lda in elements), 8 int8 (p.scale set), 4 packed int4
// (p.qsz, p.groupsize) with lda in bytes as for e2h_gemm_w8 / _w4. Rows of the weights and of B start
// on 16-byte boundaries; K is a multiple of 128 / bits (whole 16-byte pieces), of 128 for int4.
extern "C" int e2h_gemm_rows(const E2hGemmParams* pp, int bits, void* stream_v) {
  using namespace e2h;
  const E2hGemmParams& p = *pp;
  if (p.F <= 0 || p.T <= 0 || p.K <= 0 || p.T > 16) return -1;
  if (bits != 16 && bits != 8 && bits != 4) return -2;
  if (p.a_mn_major || p.b_mn_major || p.a_tiled || p.n_groups || p.n_batch || p.n_signal) return -5;
  if (p.epi == E2H_EPI_ROWMAJOR_F32_ACC || p.epi == E2H_EPI_ROWMAJOR_BF16 || p.epi == E2H_EPI_GATE)
    return -5;
  if ((p.bias || p.act || p.tail_from) && p.epi != E2H_EPI_STORE_BF16 && p.epi != E2H_EPI_STORE_F32)
    return -5;
  if ((p.out_scale != 0.f || p.softcap != 0.f) && p.epi != E2H_EPI_STORE_F32) return -5;
  if (p.epi == E2H_EPI_RESIDUAL_F32 && p.aux != p.out) return -5;
  if (p.tail_from && (p.epi != E2H_EPI_STORE_BF16 || p.tail == nullptr)) return -5;
  const bool gated = p.epi == E2H_EPI_SWIGLU || p.epi == E2H_EPI_DUAL_STORE;
  if (gated != (p.dual != 0) || (p.dual && p.a2 == nullptr)) return -5;
  const int ae = bits == 16 ? 8 : 16;       // elements (bytes) of lda per 16 bytes
  if ((p.lda % ae) || (p.ldb % 8) || (p.dual && (p.lda2 % ae))) return -6;
  if (((uintptr_t)p.a & 15) || ((uintptr_t)p.b & 15) || (p.dual && ((uintptr_t)p.a2 & 15))) return -7;
  if (p.K % (bits == 4 ? 128 : 128 / bits)) return -8;
  if (bits == 8 && p.scale == nullptr) return -9;
  if (bits == 4 && (p.qsz == nullptr || (p.dual && p.qsz2 == nullptr) || p.groupsize < 32 ||
                    (p.groupsize & (p.groupsize - 1)) || (p.K % p.groupsize)))
    return -9;
  const int units = (p.K * (bits / 4) + 127) / 128;      // of 64 bytes of a row
  // Two tiles per warp halve the reads of B; with few features the tiles themselves are what fills
  // the SMs (4096 features, one row: 7.4 us with one tile, 9.0 with two). From 9 rows on those reads
  // weigh more than the weights, and one round of tiles of 32 features is enough (8192 x 8192, 16 rows,
  // one -> two: int4 40.9 -> 22.9 us, int8 25.7 -> 21.6, bf16 29.0 -> 27.0), but for short sums (512:
  // int8 4.6 -> 5.3). Eight warps split K where the tiles alone would leave an SM with less than 16
  // warps; from 9 rows on the reads of B leave room for fewer (12288 features, 16 rows: 24.2 us with
  // eight warps, 21.9 with four).
  const bool wide = p.T > 8 && p.K >= 2048;
  const int mt = p.F >= 32 * 148 * (wide ? 1 : 2) ? 2 : 1;     // (rows_pays in ops/gemm.py knows this)
  const int ft = p.dual ? 16 : 16 * mt;
  const int tiles = (p.F + ft - 1) / ft;
  // Three or four tiles a SM: as many CTAs there, with equal shares of the features. With whole tiles some SMs
  // had one more than others, and with more CTAs than fit at once a last round ran half empty (12288
  // features are 384 tiles on 296 places). bf16, up to 8 rows: three a SM fit at once with a ring of 8 KB, four
  // make two rounds with 12 KB. us with whole tiles -> shares, one row (eight rows gain alike):
  //     bf16 5120 x 5120 (3 of 16) 13.9 -> 11.7   12288 x 4096 (3 of 32) 21.6 -> 18.1   13824 x 16384 66.6 -> 69.8
  //          8192 x 4096 (4 of 16) 14.9 -> 13.3   15360 x 5120 (4 of 32) 28.3 -> 26.9   8192 x 11008 32.0 -> 30.4
  //     int8 12288 x 4096 0.90 of the time, 5120 x 4096 0.93, 15360 x 4096 0.88, 16 rows 12288 x 4096 0.85
  // Eight warps for four tiles a SM from where their longer sums pay: tiles of 32 features from K = 4096 on
  // (15360 x 4096 four warps 1.02, eight 0.97 of the time with whole tiles; x 2048 0.89 and 1.00), tiles of 16
  // from 12288 on (9216 x 8192 0.95 and 1.04, x 16384 1.08 and 1.02). Where shares gain nothing:
  //   - five and six tiles a SM: bf16 0.97 to 1.07, int8 0.96 to 1.08; one or two, and seven and more, lost 3 to 5 %
  //   - int8 tiles of 16 with K above 8192 (5120 x 8192 0.97, x 11008 1.02, x 16384 1.04); tiles of 32 gain up
  //     to 16384 (0.95 to 0.99)
  //   - int8 from 9 rows on, but for three tiles of 32 (0.82 to 0.85 from K = 4096 on; four 1.00 to 1.04); bf16 there
  //   - int4, whose time goes with the tiles' arithmetic, used rows or not (5120 x 13824, 8 rows 25.7 -> 38.8 us),
  //     and gated products
  const int per_sm = (tiles + 147) / 148;
  const bool share = !p.dual && (per_sm == 3 || per_sm == 4) &&
                     (bits == 16  ? p.T <= 8
                      : bits == 8 ? (p.T <= 8 ? mt == 2 || p.K <= 8192 : mt == 2 && per_sm == 3)
                                  : false);
  const int ctas = share ? 148 * per_sm : tiles;
  const bool short_ring = share && bits == 16 && per_sm == 3;
  int warps = tiles >= 148 * (p.T > 8 || share ? 2 : 4) ? 4 : 8;
  if (short_ring || (share && bits == 16 && p.K >= (mt == 2 ? 4096 : 12288))) warps = 8;
  while (warps > 2 && units < 2 * warps) warps >>= 1;    // (the epilogue of 16 rows takes two)
  cudaStream_t stream = static_cast<cudaStream_t>(stream_v);
#define E2H_ROWS(QB_)                                                                           \
  return p.T <= 8 ? rows_dispatch<QB_, 1>(p, mt, ctas, warps, share, short_ring, stream)        \
                  : rows_dispatch<QB_, 2>(p, mt, ctas, warps, share, short_ring, stream)
  if (bits == 16) E2H_ROWS(16);
  if (bits == 8) E2H_ROWS(8);
  E2H_ROWS(4);
#undef E2H_ROWS
}
