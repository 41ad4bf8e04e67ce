// Per-token log-probability from materialised logits, one pass, no temporaries.
//
//   logp[r] = scale * logits[r, ids[r]] - logsumexp_v(scale * logits[r, v])
//
// This is the operation the reference implements as chunked `log_softmax(...).gather(...)`
// (rl_engine/kernels/sampling.py:91-112), which writes and re-reads a [chunk, V] temporary.
// Here one CTA streams a row once with 16-byte loads and keeps an online (max, sum-exp) per
// thread; the per-thread states are merged in a fixed butterfly order, so a row's result
// does not depend on how many rows are in the call.
#include <cstdint>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <math_constants.h>

#include "common/ptx.cuh"
#include "sampling.h"

namespace ka {
namespace {

constexpr int kThreads = 512;
constexpr int kWarps = kThreads / 32;
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLn2 = 0.6931471805599453f;

template <typename T>
struct Cvt;
template <>
struct Cvt<float> {
  static constexpr int kVec = 4;
  __device__ static float f(float v) { return v; }
};
template <>
struct Cvt<__nv_bfloat16> {
  static constexpr int kVec = 8;
  __device__ static float f(__nv_bfloat16 v) { return __bfloat162float(v); }
};
template <>
struct Cvt<__half> {
  static constexpr int kVec = 8;
  __device__ static float f(__half v) { return __half2float(v); }
};

// state: sum_j 2^(x_j*s2 - R) with R = round(m*s2)
__device__ __forceinline__ void fold_vec(const float* x, int n, float s2, float& m, float& l) {
  float mx = x[0];
#pragma unroll
  for (int j = 1; j < 8; ++j)
    if (j < n) mx = fmaxf(mx, x[j]);
  const float mn = fmaxf(m, mx);
  const float neg_old = __fmul_rn(-m, s2);
  const float neg = __fmul_rn(-mn, s2);
  float acc = 0.f;
#pragma unroll
  for (int j = 0; j < 8; ++j)
    if (j < n) acc = __fadd_rn(acc, ex2_approx(__fmaf_rn(x[j], s2, neg)));
  l = __fmaf_rn(l, ex2_approx(__fsub_rn(neg, neg_old)), acc);
  m = mn;
}

__device__ __forceinline__ void merge_state(float& m, float& l, float m2, float l2, float s2) {
  const float mn = fmaxf(m, m2);
  const float a = (m == -CUDART_INF_F) ? 0.f : ex2_approx(__fsub_rn(__fmul_rn(-mn, s2), __fmul_rn(-m, s2)));
  const float b = (m2 == -CUDART_INF_F) ? 0.f : ex2_approx(__fsub_rn(__fmul_rn(-mn, s2), __fmul_rn(-m2, s2)));
  l = __fadd_rn(__fmul_rn(l, a), __fmul_rn(l2, b));
  m = mn;
}

// The 16 bytes that start `off` bytes into a and run on into b; off: 2 .. 14 in steps of an element.
template <typename T>
__device__ __forceinline__ uint4 bytes_from(const uint4& a, const uint4& b, int off) {
  if constexpr (sizeof(T) == 4) {
    const bool one = off == 4, two = off == 8;
    return make_uint4(one ? a.y : two ? a.z : a.w, one ? a.z : two ? a.w : b.x, one ? a.w : two ? b.x : b.y,
                      one ? b.x : two ? b.y : b.z);
  }
  uint32_t w0 = a.x, w1 = a.y, w2 = a.z, w3 = a.w, w4 = b.x, w5 = b.y, w6 = b.z;
  if (off & 8) {
    w0 = w2;
    w1 = w3;
    w2 = w4;
    w3 = w5;
    w4 = w6;
    w5 = b.w;
  }
  if (off & 4) {
    w0 = w1;
    w1 = w2;
    w2 = w3;
    w3 = w4;
    w4 = w5;
  }
  const int bits = (off & 2) * 8;
  return make_uint4(__funnelshift_r(w0, w1, bits), __funnelshift_r(w1, w2, bits), __funnelshift_r(w2, w3, bits),
                    __funnelshift_r(w3, w4, bits));
}

// Thread t takes the vectors t, t + 512, ... of 16 bytes of a row, counted from the row's first element,
// wherever that lies: a row off a 16-byte boundary is read as aligned pairs of vectors and put together
// by shifts (its first and last vector element by element, so that nothing outside of the row is touched).
// A row's result therefore does not depend on where it starts. (Odd vocabularies put seven rows of eight off a
// boundary. bf16, 50257 columns, us: element by element 22.5 for 8 rows, 30.8 for 592 and 88 for 2048; so
// 13.3, 25.6 and 68.2; fp32 36.9 and 102.4 for 592 and 2048 rows, now 35.7 and 100.6. The second vector of a pair
// from the next lane instead of from L1: 75.8 for 2048 rows of bf16.)
template <typename T, bool kAligned, int kBatch, int kCtas>
__global__ void __launch_bounds__(kThreads, kCtas)
logits_logp_kernel(const T* __restrict__ logits, long long row_stride, int v, const long long* __restrict__ ids,
                   float scale, float* __restrict__ logp, float* __restrict__ lse, int rows) {
  __shared__ float s_m[kWarps], s_l[kWarps];
  constexpr int kVec = Cvt<T>::kVec;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const float s2 = scale * kLog2e;
  const int nvec = v / kVec;
  for (int row = blockIdx.x; row < rows; row += gridDim.x) {
    const T* rp = logits + static_cast<long long>(row) * row_stride;
    const int off = kAligned ? 0 : static_cast<int>(reinterpret_cast<uintptr_t>(rp) & 15u);
    float m = -CUDART_INF_F, l = 0.f;
    float x[8];
    auto take = [&](const uint4& raw) {
      const T* e = reinterpret_cast<const T*>(&raw);
#pragma unroll
      for (int j = 0; j < kVec; ++j) x[j] = Cvt<T>::f(e[j]);
      fold_vec(x, kVec, s2, m, l);
    };
    if (kAligned || off == 0) {
      const uint4* p = reinterpret_cast<const uint4*>(rp);
      for (int i = tid; i < nvec; i += kThreads * kBatch) {
        uint4 raw[kBatch];
#pragma unroll
        for (int u = 0; u < kBatch; ++u)
          if (i + u * kThreads < nvec) raw[u] = __ldcs(p + i + u * kThreads);
#pragma unroll
        for (int u = 0; u < kBatch; ++u)
          if (i + u * kThreads < nvec) take(raw[u]);
      }
    } else {
      const uint4* p = reinterpret_cast<const uint4*>(reinterpret_cast<const unsigned char*>(rp) - off);
      // aligned vectors 1 .. last are inside the row, and so are the row's vectors 1 .. last - 1 in pairs of them
      const long long bytes = static_cast<long long>(v) * static_cast<int>(sizeof(T));
      const int last = static_cast<int>((bytes + off) / 16) - 1;
      for (int i = tid; i < nvec; i += kThreads * kBatch) {
        uint4 a[kBatch], b[kBatch];
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
          const int j = i + u * kThreads;
          if (j > 0 && j < last) {
            a[u] = __ldg(p + j);
            b[u] = __ldg(p + j + 1);
          }
        }
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
          const int j = i + u * kThreads;
          if (j > 0 && j < last) {
            take(bytes_from<T>(a[u], b[u], off));
          } else if (j < nvec) {
#pragma unroll
            for (int e = 0; e < kVec; ++e) x[e] = Cvt<T>::f(rp[j * kVec + e]);
            fold_vec(x, kVec, s2, m, l);
          }
        }
      }
    }
    for (int i = nvec * kVec + tid; i < v; i += kThreads) {
      x[0] = Cvt<T>::f(rp[i]);
      fold_vec(x, 1, s2, m, l);
    }
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float m2 = __shfl_xor_sync(0xffffffffu, m, o);
      const float l2 = __shfl_xor_sync(0xffffffffu, l, o);
      // both partners must compute the same value: order the pair by lane
      float ma = (lane & o) ? m2 : m, la = (lane & o) ? l2 : l;
      const float mb = (lane & o) ? m : m2, lb = (lane & o) ? l : l2;
      merge_state(ma, la, mb, lb, s2);
      m = ma;
      l = la;
    }
    if (lane == 0) {
      s_m[warp] = m;
      s_l[warp] = l;
    }
    __syncthreads();
    if (tid == 0) {
      float mm = s_m[0], ll = s_l[0];
      for (int w = 1; w < kWarps; ++w) merge_state(mm, ll, s_m[w], s_l[w], s2);
      const float out_lse = __fmaf_rn(lg2_approx(ll), kLn2, __fmul_rn(mm, scale));
      if (lse) lse[row] = out_lse;
      const long long id = ids[row];
      float r = 0.f;
      if (id >= 0 && id < v) r = __fsub_rn(__fmul_rn(Cvt<T>::f(rp[id]), scale), out_lse);
      logp[row] = r;
    }
    __syncthreads();
  }
}

template <typename T>
int launch(const void* logits, long long row_stride, int rows, int v, const long long* ids, float scale, float* logp,
           float* lse, int num_sms, cudaStream_t st) {
  const bool aligned = (reinterpret_cast<uintptr_t>(logits) & 15u) == 0 && (row_stride * sizeof(T)) % 16 == 0;
  // Up to two rows per SM a row's time is the latency of its own loads: eight of them in flight per thread
  // (bf16, 128256 columns, us: 20.5 -> 15.4 for 8 rows, 22.5 -> 17.4 for 148, 24.6 -> 21.5 for 200). With more rows
  // four CTAs per SM overlap one another's loads and ends of rows; two CTAs with eight loads are slower there.
  const bool few = rows <= num_sms * 2;
  auto* kernel = few ? (aligned ? logits_logp_kernel<T, true, 8, 2> : logits_logp_kernel<T, false, 2, 2>)
                     : (aligned ? logits_logp_kernel<T, true, 1, 4> : logits_logp_kernel<T, false, 1, 4>);
  const int slots = num_sms * (few ? 2 : 4), grid = rows < slots ? rows : slots;
  kernel<<<grid, kThreads, 0, st>>>(static_cast<const T*>(logits), row_stride, v, ids, scale, logp, lse, rows);
  return cudaGetLastError() == cudaSuccess ? 0 : -11;
}

}  // namespace
}  // namespace ka

// logits: [rows, vocab] with `row_stride` elements between rows; ids: [rows] int64 (ids
// outside [0, vocab) give 0); logp / lse: [rows] fp32 (lse may be null). scale > 0.
extern "C" int ka_logits_logp(const void* logits, int dtype, long long row_stride, int rows, int vocab,
                              const long long* ids, float scale, float* logp, float* lse, int num_sms,
                              void* stream) {
  using namespace ka;
  if (rows <= 0) return 0;
  if (vocab <= 0 || !(scale > 0.f)) return -1;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  switch (dtype) {
    case KA_DTYPE_F32:
      return launch<float>(logits, row_stride, rows, vocab, ids, scale, logp, lse, num_sms, st);
    case KA_DTYPE_BF16:
      return launch<__nv_bfloat16>(logits, row_stride, rows, vocab, ids, scale, logp, lse, num_sms, st);
    case KA_DTYPE_F16:
      return launch<__half>(logits, row_stride, rows, vocab, ids, scale, logp, lse, num_sms, st);
    default:
      return -2;
  }
}
