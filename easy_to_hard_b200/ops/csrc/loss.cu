// Fused log-softmax / cross-entropy / log-prob gather / entropy over fp32 logits, forward and
// backward, with a vocabulary-parallel form: each rank runs the kernels on its logits shard and
// only four numbers per token (max, sum-exp, target logit, sum of p*x) cross ranks.
//
// Reference semantics: token cross-entropy in fp32 with ignore_index (train_sft.py:98-115),
// per-token log-probs and entropies of temperature-scaled logits (models/rl_model.py:134-160),
// the three-reduction vocab-parallel cross-entropy (models/tp.py:888-969).
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <float.h>
#include <stdint.h>

#include "launch.cuh"
#include "ptx.cuh"

namespace e2h {

constexpr int kCeThreads = 512;

__device__ __forceinline__ float block_reduce(float v, float* red, bool is_max) {
  v = is_max ? warp_max(v) : warp_sum(v);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __syncthreads();
  if (lane == 0) red[warp] = v;
  __syncthreads();
  float t = lane < (blockDim.x >> 5) ? red[lane] : (is_max ? -FLT_MAX : 0.f);
  t = is_max ? warp_max(t) : warp_sum(t);
  return t;
}

// A sum moved to a higher maximum. Where the factor is 0 the sum is left out: entries at the lowest finite
// value (a mask) make u infinite, and 0 * -inf would be NaN. A NaN stays.
__device__ __forceinline__ float ce_rescale(float v, float r) {
  return r == 0.f && !isnan(v) ? 0.f : v * r;
}

// Running (max, sum of exp, sum of exp * z) of N more values.
template <int N>
__device__ __forceinline__ void ce_step(const float* z, float& m, float& s, float& u) {
  float mn = m;
#pragma unroll
  for (int k = 0; k < N; ++k) mn = fmaxf(mn, z[k]);
  if (mn > m) {
    const float r = __expf(m - mn);
    s = ce_rescale(s, r);
    u = ce_rescale(u, r);
    m = mn;
  }
#pragma unroll
  for (int k = 0; k < N; ++k) {
    const float e = __expf(z[k] - m);
    s += e;
    u += e * z[k];
  }
}

// stats[row] = (m, s, tgt, u):  m = max_i z_i, s = sum exp(z_i - m), u = sum exp(z_i - m) z_i,
// tgt = z_target if the target lies in this shard else 0,  with z = logits * inv_temp.
// Bound by memory: one pass with a running maximum per thread, 64 bytes of the row in flight per thread
// (4096 x 32016: 334 us in two passes of 4-byte loads, 105 now, 5.0 TB/s). VEC: rows start on 16-byte
// boundaries.
template <bool VEC>
__global__ void __launch_bounds__(kCeThreads)
ce_stats_kernel(const float* __restrict__ logits, long long ld, int vocab,
                const long long* __restrict__ targets, int vocab_start, float inv_temp,
                float4* __restrict__ stats) {
  __shared__ float red[32];
  pdl_wait_prior();  // launched through the PDL-capable helper: wait before any global access
  const int row = blockIdx.x;
  const float* x = logits + (long long)row * ld;
  float m = -FLT_MAX, s = 0.f, u = 0.f;
  int done = 0;
  if constexpr (VEC) {
    constexpr int N = 4;
    const float4* x4 = reinterpret_cast<const float4*>(x);
    const int n_vec = vocab >> 2;
    int i = threadIdx.x;
    for (; i + (N - 1) * kCeThreads < n_vec; i += N * kCeThreads) {
      float4 q[N];
#pragma unroll
      for (int k = 0; k < N; ++k) q[k] = x4[i + k * kCeThreads];
      float z[4 * N];
#pragma unroll
      for (int k = 0; k < N; ++k) {
        z[4 * k] = q[k].x * inv_temp;
        z[4 * k + 1] = q[k].y * inv_temp;
        z[4 * k + 2] = q[k].z * inv_temp;
        z[4 * k + 3] = q[k].w * inv_temp;
      }
      ce_step<4 * N>(z, m, s, u);
    }
    for (; i < n_vec; i += kCeThreads) {
      const float4 q = x4[i];
      const float z[4] = {q.x * inv_temp, q.y * inv_temp, q.z * inv_temp, q.w * inv_temp};
      ce_step<4>(z, m, s, u);
    }
    done = n_vec << 2;
  }
  for (int i = done + threadIdx.x; i < vocab; i += kCeThreads) {
    const float z = x[i] * inv_temp;
    ce_step<1>(&z, m, s, u);
  }
  const float gm = block_reduce(m, red, true);
  const float r = __expf(m - gm);       // (a thread without values: s = u = 0)
  s = block_reduce(ce_rescale(s, r), red, false);
  u = block_reduce(ce_rescale(u, r), red, false);
  if (threadIdx.x == 0) {
    const long long t = targets[row] - vocab_start;
    const float tgt = (t >= 0 && t < vocab) ? x[t] * inv_temp : 0.f;
    stats[row] = make_float4(gm, s, tgt, u);
  }
}

// dlogits[row, i] = inv_temp * ( g_lp * ((i == target) - p_i) - g_ent * p_i * (z_i - lse + H) )
// with p_i = exp(z_i - lse); lse / H are the full-vocabulary values of the row.
// VEC: rows of both start on 16-byte boundaries; a thread turns 8 logits into one 16-byte store
// (4096 x 32016: 285 -> 136 us).
template <bool VEC>
__global__ void __launch_bounds__(kCeThreads)
ce_grad_kernel(const float* __restrict__ logits, long long ld, int vocab,
               const long long* __restrict__ targets, int vocab_start, float inv_temp,
               const float* __restrict__ lse, const float* __restrict__ ent,
               const float* __restrict__ g_lp, const float* __restrict__ g_ent,
               __nv_bfloat16* __restrict__ dlogits, long long ldd) {
  pdl_wait_prior();  // launched through the PDL-capable helper: wait before any global access
  const int row = blockIdx.x;
  const float* x = logits + (long long)row * ld;
  __nv_bfloat16* d = dlogits + (long long)row * ldd;
  const float L = lse[row];
  const float glp = g_lp ? g_lp[row] : 0.f;
  const float gen = g_ent ? g_ent[row] : 0.f;
  const float H = (g_ent && ent) ? ent[row] : 0.f;
  const long long t = targets[row] - vocab_start;
  auto grad = [&](float xv, int i) {
    const float z = xv * inv_temp;
    const float p = __expf(z - L);
    float g = glp * ((i == t ? 1.f : 0.f) - p);
    if (gen != 0.f) g -= gen * p * (z - L + H);
    return g * inv_temp;
  };
  int done = 0;
  if constexpr (VEC) {
    const float4* x4 = reinterpret_cast<const float4*>(x);
    const int n_vec = vocab >> 3;
#pragma unroll 2
    for (int i = threadIdx.x; i < n_vec; i += kCeThreads) {
      const float4 a = x4[2 * i], b = x4[2 * i + 1];
      const float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
      uint4 o;
      __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
      for (int k = 0; k < 4; ++k)
        h[k] = __floats2bfloat162_rn(grad(v[2 * k], 8 * i + 2 * k),
                                     grad(v[2 * k + 1], 8 * i + 2 * k + 1));
      reinterpret_cast<uint4*>(d)[i] = o;
    }
    done = n_vec << 3;
  }
  for (int i = done + threadIdx.x; i < vocab; i += kCeThreads)
    d[i] = __float2bfloat16_rn(grad(x[i], i));
}

}  // namespace e2h

extern "C" int e2h_ce_stats(const float* logits, long long ld, int rows, int vocab,
                            const long long* targets, int vocab_start, float inv_temp,
                            float* stats, void* stream) {
  using namespace e2h;
  const bool vec = ((uintptr_t)logits & 15) == 0 && ld % 4 == 0;
  return (int)launch(vec ? ce_stats_kernel<true> : ce_stats_kernel<false>, dim3(rows),
                     dim3(kCeThreads), 0, (cudaStream_t)stream, logits, ld, vocab, targets,
                     vocab_start, inv_temp, reinterpret_cast<float4*>(stats));
}

extern "C" int e2h_ce_grad(const float* logits, long long ld, int rows, int vocab,
                           const long long* targets, int vocab_start, float inv_temp,
                           const float* lse, const float* ent, const float* g_lp,
                           const float* g_ent, void* dlogits, long long ldd, void* stream) {
  using namespace e2h;
  const bool vec = (((uintptr_t)logits | (uintptr_t)dlogits) & 15) == 0 && ld % 4 == 0 && ldd % 8 == 0;
  return (int)launch(vec ? ce_grad_kernel<true> : ce_grad_kernel<false>, dim3(rows),
                     dim3(kCeThreads), 0, (cudaStream_t)stream, logits, ld, vocab, targets,
                     vocab_start, inv_temp, lse, ent, g_lp, g_ent,
                     static_cast<__nv_bfloat16*>(dlogits), ldd);
}
