// Small kernels of the RL loop.
//
//   decode_qkv_rope_cache: what lies between the fused qkv projection and attention in a decode
//       step, in one launch: split q / k / v, rotate q and k, write k and v into the cache slot.
//   adamw_step: fused AdamW update over a flat parameter group: bf16 parameter, fp32 master
//       copy, fp32 moments, fp32 or bf16 gradient, bias correction and decoupled weight decay.
//
// Neither exists in the reference (its executor comments defer generation to a future vLLM
// integration, rl_engine/executors/rollout.py:33).
#include <cstdint>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

namespace ka {
namespace {

constexpr int kD = 128;
// qkv: [B, (hq + 2 hkv) * 128] bf16 (row stride qkv_stride), the output of the fused projection.
// pos [B]: position of the new token; slot [1]: cache row to write (both on the device, so a
// CUDA graph can replay the launch). q_out [B, hq, 128] rotated; cache_k / cache_v
// [B, max_len, hkv, 128]: row [b, slot] receives the rotated key and the value.
// The rotation is rope_kernel's arithmetic (elementwise.cu), so the bits are the same.
__global__ void __launch_bounds__(64)
decode_qkv_rope_cache_kernel(const __nv_bfloat16* __restrict__ qkv, long long qkv_stride,
                             const long long* __restrict__ pos, const long long* __restrict__ slot,
                             const float* __restrict__ cos_t, const float* __restrict__ sin_t,
                             __nv_bfloat16* __restrict__ q_out, __nv_bfloat16* __restrict__ cache_k,
                             __nv_bfloat16* __restrict__ cache_v, int hq, int hkv, int max_len) {
  constexpr int half = kD / 2;
  const int b = blockIdx.y, head = blockIdx.x, j = threadIdx.x;  // head in [0, hq + 2 hkv)
  const __nv_bfloat16* src = qkv + b * qkv_stride + static_cast<long long>(head) * kD;
  const long long s = slot[0];
  if (head < hq + hkv) {
    const long long p = pos[b];
    const float c = cos_t[p * half + j], sn = sin_t[p * half + j];
    const float a = __bfloat162float(src[j]), bb = __bfloat162float(src[j + half]);
    const __nv_bfloat16 lo = __float2bfloat16_rn(__fsub_rn(__fmul_rn(a, c), __fmul_rn(bb, sn)));
    const __nv_bfloat16 hi = __float2bfloat16_rn(__fadd_rn(__fmul_rn(bb, c), __fmul_rn(a, sn)));
    __nv_bfloat16* dst = head < hq ? q_out + (static_cast<long long>(b) * hq + head) * kD
                                   : cache_k + ((static_cast<long long>(b) * max_len + s) * hkv + (head - hq)) * kD;
    dst[j] = lo;
    dst[j + half] = hi;
  } else {
    __nv_bfloat16* dst = cache_v + ((static_cast<long long>(b) * max_len + s) * hkv + (head - hq - hkv)) * kD;
    dst[j] = src[j];
    dst[j + half] = src[j + half];
  }
}

// One element of the update (shared by the scalar and the 4-wide kernel: same bits).
__device__ __forceinline__ float adamw_one(float g, float& m, float& v, float& w, float lr, float beta1, float beta2,
                                           float eps, float weight_decay, float bc1, float bc2, float grad_scale) {
  g = __fmul_rn(g, grad_scale);
  m = __fmaf_rn(beta1, m, __fmul_rn(1.f - beta1, g));
  v = __fmaf_rn(beta2, v, __fmul_rn(1.f - beta2, __fmul_rn(g, g)));
  const float mh = __fdiv_rn(m, bc1);
  const float vh = __fdiv_rn(v, bc2);
  w = __fsub_rn(w, __fmul_rn(lr, __fmul_rn(weight_decay, w)));
  w = __fsub_rn(w, __fmul_rn(lr, __fdiv_rn(mh, __fadd_rn(__fsqrt_rn(vh), eps))));
  return w;
}

// Four elements per thread with 16-byte (fp32) / 8-byte (bf16) accesses; elements past the last
// multiple of four are handled one by one by the first threads.
template <typename G>
__global__ void __launch_bounds__(256)
adamw_kernel(__nv_bfloat16* __restrict__ param, float* __restrict__ master, const G* __restrict__ grad,
             float* __restrict__ m, float* __restrict__ v, long long n, float lr, float beta1, float beta2, float eps,
             float weight_decay, float bc1, float bc2, float grad_scale) {
  const long long n4 = n / 4;
  const long long tid = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
  const long long stride = static_cast<long long>(gridDim.x) * blockDim.x;
  for (long long i = tid; i < n4; i += stride) {
    float g[4];
    if constexpr (sizeof(G) == 2) {
      const uint2 raw = reinterpret_cast<const uint2*>(grad)[i];
      const __nv_bfloat162 a = *reinterpret_cast<const __nv_bfloat162*>(&raw.x);
      const __nv_bfloat162 b = *reinterpret_cast<const __nv_bfloat162*>(&raw.y);
      g[0] = __bfloat162float(a.x); g[1] = __bfloat162float(a.y); g[2] = __bfloat162float(b.x); g[3] = __bfloat162float(b.y);
    } else {
      const float4 t = reinterpret_cast<const float4*>(grad)[i];
      g[0] = t.x; g[1] = t.y; g[2] = t.z; g[3] = t.w;
    }
    float4 m4 = reinterpret_cast<float4*>(m)[i], v4 = reinterpret_cast<float4*>(v)[i];
    float4 w4 = reinterpret_cast<float4*>(master)[i];
    adamw_one(g[0], m4.x, v4.x, w4.x, lr, beta1, beta2, eps, weight_decay, bc1, bc2, grad_scale);
    adamw_one(g[1], m4.y, v4.y, w4.y, lr, beta1, beta2, eps, weight_decay, bc1, bc2, grad_scale);
    adamw_one(g[2], m4.z, v4.z, w4.z, lr, beta1, beta2, eps, weight_decay, bc1, bc2, grad_scale);
    adamw_one(g[3], m4.w, v4.w, w4.w, lr, beta1, beta2, eps, weight_decay, bc1, bc2, grad_scale);
    reinterpret_cast<float4*>(m)[i] = m4;
    reinterpret_cast<float4*>(v)[i] = v4;
    reinterpret_cast<float4*>(master)[i] = w4;
    const __nv_bfloat162 o0 = __floats2bfloat162_rn(w4.x, w4.y), o1 = __floats2bfloat162_rn(w4.z, w4.w);
    uint2 o;
    o.x = *reinterpret_cast<const uint32_t*>(&o0);
    o.y = *reinterpret_cast<const uint32_t*>(&o1);
    reinterpret_cast<uint2*>(param)[i] = o;
  }
  for (long long i = n4 * 4 + tid; i < n; i += stride) {
    float g;
    if constexpr (sizeof(G) == 2) g = __bfloat162float(grad[i]); else g = grad[i];
    float mi = m[i], vi = v[i], w = master[i];
    adamw_one(g, mi, vi, w, lr, beta1, beta2, eps, weight_decay, bc1, bc2, grad_scale);
    m[i] = mi;
    v[i] = vi;
    master[i] = w;
    param[i] = __float2bfloat16_rn(w);
  }
}

}  // namespace
}  // namespace ka

extern "C" {

// See decode_qkv_rope_cache_kernel. head_dim is 128.
int ka_decode_qkv_rope_cache(const void* qkv, long long qkv_stride, const long long* pos, const long long* slot,
                             const float* cos_t, const float* sin_t, void* q_out, void* cache_k, void* cache_v,
                             int batch, int hq, int hkv, int max_len, void* stream) {
  using namespace ka;
  if (batch <= 0) return 0;
  dim3 grid(static_cast<unsigned>(hq + 2 * hkv), static_cast<unsigned>(batch));
  decode_qkv_rope_cache_kernel<<<grid, 64, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const __nv_bfloat16*>(qkv), qkv_stride, pos, slot, cos_t, sin_t, static_cast<__nv_bfloat16*>(q_out),
      static_cast<__nv_bfloat16*>(cache_k), static_cast<__nv_bfloat16*>(cache_v), hq, hkv, max_len);
  return cudaGetLastError() == cudaSuccess ? 0 : -11;
}

// step >= 1; grad_is_bf16 selects the gradient type; grad_scale multiplies the gradient first.
int ka_adamw_step(void* param, float* master, const void* grad, int grad_is_bf16, float* m, float* v, long long n,
                  float lr, float beta1, float beta2, float eps, float weight_decay, int step, float grad_scale,
                  int num_sms, void* stream) {
  using namespace ka;
  if (n <= 0) return 0;
  const float bc1 = 1.f - powf(beta1, static_cast<float>(step));
  const float bc2 = 1.f - powf(beta2, static_cast<float>(step));
  long long blocks = (n / 4 + 255) / 256;
  if (blocks < 1) blocks = 1;
  if (blocks > static_cast<long long>(num_sms) * 16) blocks = static_cast<long long>(num_sms) * 16;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (grad_is_bf16)
    adamw_kernel<__nv_bfloat16><<<static_cast<int>(blocks), 256, 0, st>>>(
        static_cast<__nv_bfloat16*>(param), master, static_cast<const __nv_bfloat16*>(grad), m, v, n, lr, beta1, beta2,
        eps, weight_decay, bc1, bc2, grad_scale);
  else
    adamw_kernel<float><<<static_cast<int>(blocks), 256, 0, st>>>(static_cast<__nv_bfloat16*>(param), master,
                                                                 static_cast<const float*>(grad), m, v, n, lr, beta1,
                                                                 beta2, eps, weight_decay, bc1, bc2, grad_scale);
  return cudaGetLastError() == cudaSuccess ? 0 : -11;
}

}  // extern "C"
