// 16-byte-vectorised forms of the row-wise and element-wise kernels for the large-token
// (training / prefill / scoring) shapes, where these ops are pure HBM streams: every thread
// moves 8 bf16 per load / store and a row of up to 8192 features lives in registers between
// the reduction and the write, so each byte is touched once.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "ptx.cuh"

namespace e2h {

struct alignas(16) BF8 {
  __nv_bfloat162 v[4];
};

__device__ __forceinline__ void unpack8(const BF8& b, float* f) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    f[2 * i] = __bfloat162float(b.v[i].x);
    f[2 * i + 1] = __bfloat162float(b.v[i].y);
  }
}
__device__ __forceinline__ BF8 pack8(const float* f) {
  BF8 b;
#pragma unroll
  for (int i = 0; i < 4; ++i) b.v[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
  return b;
}

// sum over the block of two values at once; red must hold 64 floats
__device__ __forceinline__ float2 block_sum2(float a, float b, float* red) {
  a = warp_sum(a);
  b = warp_sum(b);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  if (lane == 0) {
    red[warp] = a;
    red[32 + warp] = b;
  }
  __syncthreads();
  a = lane < nw ? red[lane] : 0.f;
  b = lane < nw ? red[32 + lane] : 0.f;
  a = warp_sum(a);
  b = warp_sum(b);
  return make_float2(a, b);
}

// How many blocks of a row-wise kernel run at once: its rows are dealt out over them.
template <typename Kernel>
inline int resident_blocks(Kernel* kernel, int threads, int rows) {
  int dev = 0, sms = 148, per = 0;
  if (cudaGetDevice(&dev) == cudaSuccess)
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, threads, 0) != cudaSuccess || per < 1)
    per = 1;
  return rows < sms * per ? rows : sms * per;
}

// Row-wise RMSNorm kernels of many rows. They are HBM streams, and with one block per row they were not
// bound by it: a row's load, the sum over the block and the store wait for one another, and a block that
// ends makes room for the next one's load only then (49152 x 4096: 2.9 TB/s). Here a block stays, takes
// every gridDim.x-th row, and its loads of the next row are under way while it sums and stores this
// one. A thread owns the same vectors of every row, NV of 16 bytes, so that the weight is loaded once,
// and the sums have the order they had with one block per row. One block per row -> blocks that stay (floor
// at the copy rate): 49152 x 4096 forward 258 -> 148 us (123), backward 496 -> 270 (246), embedding and norm
// 500 -> 194 (184); 12288 x 4096 73 -> 44 (31), 133 -> 75 (61), 133 -> 55 (46); 22432 x 8192 240 -> 140
// (112), 545 -> 302 (224), 381 -> 204 (168).

// Where the row of a token starts in the embedding table. An id outside the table is reported and never
// dereferenced (nullptr: the row counts as zeros).
__device__ __forceinline__ const __nv_bfloat16* emb_row(const int* tokens, int t,
                                                        const __nv_bfloat16* emb, int emb_rows,
                                                        int dim, int* status) {
  const int id = tokens[t];
  if (id >= 0 && id < emb_rows) return emb + (long long)id * dim;
  if (threadIdx.x == 0 && status) atomicCAS(status, 0, kStatusBadArgs);
  return nullptr;
}

// x_out[t] = bf16(bf16(x[t] * rstd) * w). EMB: x is the embedding table and row t of the input is that of
// token t, which also goes to h_out.
template <int NV, bool EMB>
__global__ void __launch_bounds__(256) rmsnorm_rows_kernel(
    const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ weight,
    __nv_bfloat16* __restrict__ out, float* __restrict__ rstd_out, int rows, int dim, float eps,
    const int* __restrict__ tokens, int emb_rows, __nv_bfloat16* __restrict__ h_out, int* status) {
  __shared__ float red[2][64];
  const int nvec = dim >> 3;
  BF8 raw[NV], w[NV];
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    const int i = threadIdx.x + k * blockDim.x;
    if (i < nvec) w[k] = *reinterpret_cast<const BF8*>(weight + 8 * i);
  }
  auto load = [&](int row) {
    const __nv_bfloat16* src =
        EMB ? emb_row(tokens, row, x, emb_rows, dim, status) : x + (long long)row * dim;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      const int i = threadIdx.x + k * blockDim.x;
      if (i < nvec) raw[k] = EMB && src == nullptr ? BF8{} : *reinterpret_cast<const BF8*>(src + 8 * i);
    }
  };
  load(blockIdx.x);
  int turn = 0;
  for (int row = blockIdx.x; row < rows; row += gridDim.x, turn ^= 1) {
    BF8 cur[NV];
    float ss = 0.f;
#pragma unroll
    for (int k = 0; k < NV; ++k) cur[k] = raw[k];
    if (row + gridDim.x < rows) load(row + gridDim.x);
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      const int i = threadIdx.x + k * blockDim.x;
      if (i < nvec) {
        float v[8];
        unpack8(cur[k], v);
#pragma unroll
        for (int e = 0; e < 8; ++e) ss += v[e] * v[e];
      }
    }
    // (two buffers: a warp writes one again only after all have passed the barrier of the other)
    ss = block_sum2(ss, 0.f, red[turn]).x;
    const float rstd = rsqrtf(ss / dim + eps);
    if (rstd_out && threadIdx.x == 0) rstd_out[row] = rstd;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      const int i = threadIdx.x + k * blockDim.x;
      if (i < nvec) {
        float v[8], f[8], o[8];
        unpack8(cur[k], v);
        unpack8(w[k], f);
#pragma unroll
        for (int e = 0; e < 8; ++e) o[e] = bf16_round(v[e] * rstd) * f[e];
        *reinterpret_cast<BF8*>(out + (long long)row * dim + 8 * i) = pack8(o);
        if (EMB) *reinterpret_cast<BF8*>(h_out + (long long)row * dim + 8 * i) = cur[k];
      }
    }
  }
}

// dx = rstd * (dy*w) - x * rstd^3 / dim * sum(dy*w*x) (+ dres)
template <int NV>
__global__ void __launch_bounds__(256) rmsnorm_bwd_rows_kernel(
    const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ dy,
    const __nv_bfloat16* __restrict__ weight, const __nv_bfloat16* __restrict__ dres,
    __nv_bfloat16* __restrict__ dx, int rows, int dim, float eps) {
  __shared__ float red[2][64];
  const int nvec = dim >> 3;
  BF8 xn[NV], gn[NV], rn[NV], w[NV];
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    const int i = threadIdx.x + k * blockDim.x;
    if (i < nvec) w[k] = *reinterpret_cast<const BF8*>(weight + 8 * i);
  }
  auto load = [&](int row) {
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      const int i = threadIdx.x + k * blockDim.x;
      if (i < nvec) {
        const long long at = (long long)row * dim + 8 * i;
        xn[k] = *reinterpret_cast<const BF8*>(x + at);
        gn[k] = *reinterpret_cast<const BF8*>(dy + at);
        if (dres) rn[k] = *reinterpret_cast<const BF8*>(dres + at);
      }
    }
  };
  load(blockIdx.x);
  int turn = 0;
  for (int row = blockIdx.x; row < rows; row += gridDim.x, turn ^= 1) {
    BF8 xc[NV], gc[NV], rc[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      xc[k] = xn[k];
      gc[k] = gn[k];
      rc[k] = rn[k];
    }
    if (row + gridDim.x < rows) load(row + gridDim.x);
    float ss = 0.f, dot = 0.f;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      const int i = threadIdx.x + k * blockDim.x;
      if (i < nvec) {
        float xv[8], g[8], f[8];
        unpack8(xc[k], xv);
        unpack8(gc[k], g);
        unpack8(w[k], f);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          g[e] *= f[e];
          ss += xv[e] * xv[e];
          dot += xv[e] * g[e];
        }
      }
    }
    const float2 s = block_sum2(ss, dot, red[turn]);
    const float rstd = rsqrtf(s.x / dim + eps);
    const float coef = s.y * rstd * rstd * rstd / dim;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      const int i = threadIdx.x + k * blockDim.x;
      if (i < nvec) {
        float xv[8], g[8], f[8], o[8];
        unpack8(xc[k], xv);
        unpack8(gc[k], g);
        unpack8(w[k], f);
#pragma unroll
        for (int e = 0; e < 8; ++e) o[e] = g[e] * f[e] * rstd - xv[e] * coef;
        if (dres) {
          float r[8];
          unpack8(rc[k], r);
#pragma unroll
          for (int e = 0; e < 8; ++e) o[e] += r[e];
        }
        *reinterpret_cast<BF8*>(dx + (long long)row * dim + 8 * i) = pack8(o);
      }
    }
  }
}

__global__ void swiglu_fwd_vec_kernel(const __nv_bfloat16* __restrict__ g,
                                      const __nv_bfloat16* __restrict__ u,
                                      __nv_bfloat16* __restrict__ out, long long nvec) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nvec;
       i += (long long)gridDim.x * blockDim.x) {
    float a[8], b[8], o[8];
    unpack8(reinterpret_cast<const BF8*>(g)[i], a);
    unpack8(reinterpret_cast<const BF8*>(u)[i], b);
#pragma unroll
    for (int e = 0; e < 8; ++e) o[e] = bf16_round(silu(a[e])) * b[e];
    reinterpret_cast<BF8*>(out)[i] = pack8(o);
  }
}

__global__ void swiglu_bwd_vec_kernel(const __nv_bfloat16* __restrict__ g,
                                      const __nv_bfloat16* __restrict__ u,
                                      const __nv_bfloat16* __restrict__ dact,
                                      __nv_bfloat16* __restrict__ dg,
                                      __nv_bfloat16* __restrict__ du, long long nvec) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nvec;
       i += (long long)gridDim.x * blockDim.x) {
    float a[8], b[8], d[8], og[8], ou[8];
    unpack8(reinterpret_cast<const BF8*>(g)[i], a);
    unpack8(reinterpret_cast<const BF8*>(u)[i], b);
    unpack8(reinterpret_cast<const BF8*>(dact)[i], d);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const float sig = 1.f / (1.f + __expf(-a[e]));
      og[e] = d[e] * b[e] * (sig * (1.f + a[e] * (1.f - sig)));
      ou[e] = d[e] * (a[e] * sig);
    }
    reinterpret_cast<BF8*>(dg)[i] = pack8(og);
    reinterpret_cast<BF8*>(du)[i] = pack8(ou);
  }
}

// Interleaved-pair RoPE, 4 pairs per thread. x rows are `ld` elements apart; only the first
// n_heads * head_dim elements of a row are rotated.
__global__ void rope_vec_kernel(const __nv_bfloat16* __restrict__ x, __nv_bfloat16* __restrict__ out,
                                const __nv_bfloat16* __restrict__ freqs,
                                const int* __restrict__ pos, int n_heads, int head_dim,
                                long long ld, int inverse) {
  const int t = blockIdx.x;
  const int vec_per_head = head_dim >> 3;
  const int p = pos[t];
  const __nv_bfloat16* fr = freqs + (long long)p * head_dim;     // [head_dim/2][2]
  for (int i = threadIdx.x; i < n_heads * vec_per_head; i += blockDim.x) {
    const int h = i / vec_per_head, j = i - h * vec_per_head;
    const long long o = (long long)t * ld + (long long)h * head_dim + 8 * j;
    float v[8], cs[8], r[8];
    unpack8(*reinterpret_cast<const BF8*>(x + o), v);
    unpack8(*reinterpret_cast<const BF8*>(fr + 8 * j), cs);      // (cos, sin) x 4 pairs
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float c = cs[2 * e], s = inverse ? -cs[2 * e + 1] : cs[2 * e + 1];
      r[2 * e] = v[2 * e] * c - v[2 * e + 1] * s;
      r[2 * e + 1] = v[2 * e + 1] * c + v[2 * e] * s;
    }
    *reinterpret_cast<BF8*>(out + o) = pack8(r);
  }
}

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

}  // namespace e2h
