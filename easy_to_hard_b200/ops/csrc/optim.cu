// Fused AdamW update (one pass over parameter, gradient and both moments) plus the helpers
// of the two-phase global gradient clip: a squared-norm partial reduction and a kernel that
// turns the reduced norm into a clip coefficient on the device, so that the optimizer step
// needs no host synchronisation.
//
// Update rule = the reference's memory-efficient AdamW
// (training_utils/memory_efficient_adam.py:61-104):
//   p *= 1 - lr*wd;  m = b1*m + (1-b1)*g;  v = b2*v + (1-b2)*g*g   (in the state dtype)
//   denom = sqrt(v)/sqrt(bc2) + eps;  p -= (lr/bc1) * m / denom     (in the parameter dtype)
// Parameter, gradient and state may each be fp32 or bf16.
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <stdint.h>

#include "ptx.cuh"

namespace e2h {

template <typename T> __device__ __forceinline__ float ldf(const T* p, long long i);
template <> __device__ __forceinline__ float ldf<float>(const float* p, long long i) { return p[i]; }
template <> __device__ __forceinline__ float ldf<__nv_bfloat16>(const __nv_bfloat16* p, long long i) {
  return __bfloat162float(p[i]);
}
template <typename T> __device__ __forceinline__ void stf(T* p, long long i, float v);
template <> __device__ __forceinline__ void stf<float>(float* p, long long i, float v) { p[i] = v; }
template <> __device__ __forceinline__ void stf<__nv_bfloat16>(__nv_bfloat16* p, long long i, float v) {
  p[i] = __float2bfloat16_rn(v);
}
template <typename T> __device__ __forceinline__ float rnd(float v);
template <> __device__ __forceinline__ float rnd<float>(float v) { return v; }
template <> __device__ __forceinline__ float rnd<__nv_bfloat16>(float v) { return bf16_round(v); }

struct AdamCoef {
  float coef, decay, b1, b2, eps, step, inv_sqrt_bc2;
};
// One element; pv, mv, vv are updated.
template <typename P, typename S>
__device__ __forceinline__ void adam_one(const AdamCoef& c, float& pv, float g, float& mv, float& vv) {
  if (c.decay != 1.f) pv = rnd<P>(pv * c.decay);
  const float gv = rnd<S>(g * c.coef);
  mv = rnd<S>(rnd<S>(c.b1 * mv) + (1.f - c.b1) * gv);
  vv = rnd<S>(rnd<S>(c.b2 * vv) + (1.f - c.b2) * gv * gv);
  const float denom = rnd<S>(rnd<S>(sqrtf(vv) * c.inv_sqrt_bc2) + c.eps);
  pv = pv - c.step * rnd<P>(mv) / rnd<P>(denom);
}

// four elements as one access
__device__ __forceinline__ void ld4(const float* p, long long i, float* v) {
  *reinterpret_cast<float4*>(v) = __ldcs(reinterpret_cast<const float4*>(p) + i);
}
__device__ __forceinline__ void ld4(const __nv_bfloat16* p, long long i, float* v) {
  const uint2 q = __ldcs(reinterpret_cast<const uint2*>(p) + i);
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&q);
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    v[2 * k] = __bfloat162float(h[k].x);
    v[2 * k + 1] = __bfloat162float(h[k].y);
  }
}
__device__ __forceinline__ void st4(float* p, long long i, const float* v) {
  __stcs(reinterpret_cast<float4*>(p) + i, *reinterpret_cast<const float4*>(v));
}
__device__ __forceinline__ void st4(__nv_bfloat16* p, long long i, const float* v) {
  uint2 q;
  __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&q);
  h[0] = __floats2bfloat162_rn(v[0], v[1]);
  h[1] = __floats2bfloat162_rn(v[2], v[3]);
  __stcs(reinterpret_cast<uint2*>(p) + i, q);
}

// Bound by memory: 30 bytes an element in fp32 (four streams in, three and the bf16 copy out). VEC = 4:
// a thread moves four elements per access (202M elements with the copy: 1257 -> 972 us, 6.2 TB/s); VEC = 1
// for buffers that do not start on a 16-byte boundary.
template <typename P, typename G, typename S, int VEC>
__global__ void adamw_kernel(P* __restrict__ p, const G* __restrict__ g, S* __restrict__ m,
                             S* __restrict__ v, long long n, float lr, float b1, float b2, float eps,
                             float wd, float bc1, float bc2, const float* __restrict__ clip_coef,
                             __nv_bfloat16* __restrict__ p_bf16_copy) {
  AdamCoef c;
  c.coef = clip_coef ? *clip_coef : 1.f;
  c.decay = wd != 0.f ? 1.f - lr * wd : 1.f;
  c.b1 = b1;
  c.b2 = b2;
  c.eps = eps;
  c.step = lr / bc1;
  c.inv_sqrt_bc2 = rsqrtf(bc2);
  const long long first = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const long long stride = (long long)gridDim.x * blockDim.x;
  const long long n_vec = VEC == 4 ? n / 4 : 0;
  if constexpr (VEC == 4) {
    for (long long i = first; i < n_vec; i += stride) {
      float pv[4], gv[4], mv[4], vv[4];
      ld4(p, i, pv);
      ld4(g, i, gv);
      ld4(m, i, mv);
      ld4(v, i, vv);
#pragma unroll
      for (int k = 0; k < 4; ++k) adam_one<P, S>(c, pv[k], gv[k], mv[k], vv[k]);
      st4(p, i, pv);
      st4(m, i, mv);
      st4(v, i, vv);
      if (p_bf16_copy) st4(p_bf16_copy, i, pv);
    }
  }
  for (long long i = n_vec * 4 + first; i < n; i += stride) {
    float pv = ldf<P>(p, i), mv = ldf<S>(m, i), vv = ldf<S>(v, i);
    adam_one<P, S>(c, pv, ldf<G>(g, i), mv, vv);
    stf<P>(p, i, pv);
    stf<S>(m, i, mv);
    stf<S>(v, i, vv);
    if (p_bf16_copy) p_bf16_copy[i] = __float2bfloat16_rn(pv);
  }
}

// dst (fp32) = src (bf16): 8 bytes read and 16 written per thread and step (202M elements: 254 us, 4.8
// TB/s).
__global__ void widen_kernel(const __nv_bfloat16* __restrict__ src, float* __restrict__ dst,
                             long long n) {
  const long long first = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = first; i < n / 4; i += stride) {
    float v[4];
    ld4(src, i, v);
    reinterpret_cast<float4*>(dst)[i] = *reinterpret_cast<const float4*>(v);
  }
  for (long long i = n / 4 * 4 + first; i < n; i += stride) dst[i] = __bfloat162float(src[i]);
}

// out[0] += sum(x^2) (fp32 atomics; one atomic per CTA)
template <typename T>
__global__ void sqnorm_kernel(const T* __restrict__ x, long long n, float* __restrict__ out) {
  __shared__ float red[32];
  float s = 0.f;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const float v = ldf<T>(x, i);
    s += v * v;
  }
  s = warp_sum(s);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    float t = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.f;
    t = warp_sum(t);
    if (threadIdx.x == 0) atomicAdd(out, t);
  }
}

// coef = min(1, max_norm / (sqrt(sqnorm) + 1e-6)); norm_out = sqrt(sqnorm)
__global__ void clip_coef_kernel(const float* sqnorm, float max_norm, float* coef,
                                 float* norm_out) {
  const float nrm = sqrtf(*sqnorm);
  *norm_out = nrm;
  *coef = fminf(1.f, max_norm / (nrm + 1e-6f));
}

template <typename P, typename G, typename S>
static int launch_adamw(void* p, const void* g, void* m, void* v, long long n, float lr, float b1,
                        float b2, float eps, float wd, float bc1, float bc2, const float* clip,
                        void* p_bf16, cudaStream_t st) {
  // four elements per access where every buffer allows it
  const uintptr_t bits = (uintptr_t)p | (uintptr_t)g | (uintptr_t)m | (uintptr_t)v | (uintptr_t)p_bf16;
  const bool vec = (bits & 15) == 0 && n >= 4;
  long long blocks = ((vec ? n / 4 : n) + 255) / 256;
  if (blocks > 148 * 8) blocks = 148 * 8;
  if (blocks < 1) blocks = 1;
  if (vec)
    adamw_kernel<P, G, S, 4><<<(unsigned)blocks, 256, 0, st>>>(
        (P*)p, (const G*)g, (S*)m, (S*)v, n, lr, b1, b2, eps, wd, bc1, bc2, clip,
        (__nv_bfloat16*)p_bf16);
  else
    adamw_kernel<P, G, S, 1><<<(unsigned)blocks, 256, 0, st>>>(
        (P*)p, (const G*)g, (S*)m, (S*)v, n, lr, b1, b2, eps, wd, bc1, bc2, clip,
        (__nv_bfloat16*)p_bf16);
  return (int)cudaGetLastError();
}

}  // namespace e2h

using namespace e2h;

// dtype codes: 0 = fp32, 1 = bf16.  p_bf16_copy (optional) receives the updated parameter in
// bf16 -- the compute copy that the next forward pass gathers.
extern "C" int e2h_adamw(void* p, const void* g, void* m, void* v, long long n, int p_dt, int g_dt,
                         int s_dt, float lr, float b1, float b2, float eps, float wd, float bc1,
                         float bc2, const float* clip_coef, void* p_bf16_copy, void* stream) {
  cudaStream_t st = (cudaStream_t)stream;
  typedef __nv_bfloat16 bf;
#define GO(P, G, S) \
  return launch_adamw<P, G, S>(p, g, m, v, n, lr, b1, b2, eps, wd, bc1, bc2, clip_coef, p_bf16_copy, st)
  const int code = p_dt * 4 + g_dt * 2 + s_dt;
  switch (code) {
    case 0: GO(float, float, float);
    case 1: GO(float, float, bf);
    case 2: GO(float, bf, float);
    case 3: GO(float, bf, bf);
    case 4: GO(bf, float, float);
    case 5: GO(bf, float, bf);
    case 6: GO(bf, bf, float);
    case 7: GO(bf, bf, bf);
  }
#undef GO
  return -1;
}

extern "C" int e2h_sqnorm(const void* x, long long n, int dt, float* out, void* stream) {
  long long blocks = (n + 1023) / 1024;
  if (blocks > 148 * 8) blocks = 148 * 8;
  if (blocks < 1) blocks = 1;
  if (dt == 0)
    sqnorm_kernel<float><<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>((const float*)x, n, out);
  else
    sqnorm_kernel<__nv_bfloat16><<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>(
        (const __nv_bfloat16*)x, n, out);
  return (int)cudaGetLastError();
}

extern "C" int e2h_clip_coef(const float* sqnorm, float max_norm, float* coef, float* norm_out,
                             void* stream) {
  clip_coef_kernel<<<1, 1, 0, (cudaStream_t)stream>>>(sqnorm, max_norm, coef, norm_out);
  return (int)cudaGetLastError();
}

// src bf16 (8-byte aligned), dst fp32 (16-byte aligned)
extern "C" int e2h_widen(const void* src, void* dst, long long n, void* stream) {
  if (n <= 0) return n == 0 ? 0 : -1;
  if (((uintptr_t)src & 7) || ((uintptr_t)dst & 15)) return -2;
  long long blocks = (n / 4 + 255) / 256;
  if (blocks > 148 * 16) blocks = 148 * 16;
  if (blocks < 1) blocks = 1;
  widen_kernel<<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>((const __nv_bfloat16*)src,
                                                                  (float*)dst, n);
  return (int)cudaGetLastError();
}
