// Memory-bound layer ops of the decoder, each a single pass with 16-byte accesses and fp32
// math: RMSNorm (with optional fused residual add), rotary embedding, SwiGLU.
// Every reduction runs in a fixed order inside one CTA, so a row's output depends on that row
// only (batch invariance). None of these exists in the reference, which only names them
// (rl_engine/platforms/constants.py:75-80, README feature list).
#include <cstdint>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "common/ptx.cuh"

namespace ka {
namespace {

constexpr float kLog2e = 1.4426950408889634f;

struct alignas(16) Bf16x8 {
  __nv_bfloat16 v[8];
};

__device__ __forceinline__ float block_sum_fixed(float v, float* s_warp, int n_warps) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, o));
  if (lane == 0) s_warp[warp] = v;
  __syncthreads();
  float t = 0.f;
  for (int w = 0; w < n_warps; ++w) t = __fadd_rn(t, s_warp[w]);  // same order in every thread
  __syncthreads();
  return t;
}

// y = (x [+ residual]) * rsqrt(mean(x^2) + eps) * w ; if residual_out: residual_out = x + residual
// One CTA per row, D % 8 == 0; for many rows, and for rows longer than rmsnorm_reg_kernel holds.
__global__ void __launch_bounds__(256)
rmsnorm_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ residual,
               const __nv_bfloat16* __restrict__ w, __nv_bfloat16* __restrict__ y,
               __nv_bfloat16* __restrict__ residual_out, int rows, int d, float eps) {
  __shared__ float s_warp[8];
  const int nvec = d / 8;
  for (int row = blockIdx.x; row < rows; row += gridDim.x) {
    const Bf16x8* xp = reinterpret_cast<const Bf16x8*>(x + static_cast<size_t>(row) * d);
    const Bf16x8* rp = residual ? reinterpret_cast<const Bf16x8*>(residual + static_cast<size_t>(row) * d) : nullptr;
    Bf16x8* ro = residual_out ? reinterpret_cast<Bf16x8*>(residual_out + static_cast<size_t>(row) * d) : nullptr;
    float ss = 0.f;
    for (int i = threadIdx.x; i < nvec; i += blockDim.x) {
      Bf16x8 a = xp[i];
      if (rp) {
        const Bf16x8 b = rp[i];
#pragma unroll
        for (int j = 0; j < 8; ++j)
          a.v[j] = __float2bfloat16_rn(__fadd_rn(__bfloat162float(a.v[j]), __bfloat162float(b.v[j])));
        if (ro) ro[i] = a;
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float f = __bfloat162float(a.v[j]);
        ss = __fmaf_rn(f, f, ss);
      }
    }
    const float total = block_sum_fixed(ss, s_warp, blockDim.x >> 5);
    const float inv = __fdiv_rn(1.f, __fsqrt_rn(__fadd_rn(__fdiv_rn(total, static_cast<float>(d)), eps)));
    const Bf16x8* wp = reinterpret_cast<const Bf16x8*>(w);
    Bf16x8* yp = reinterpret_cast<Bf16x8*>(y + static_cast<size_t>(row) * d);
    const Bf16x8* src = (rp && ro) ? reinterpret_cast<const Bf16x8*>(ro) : xp;
    for (int i = threadIdx.x; i < nvec; i += blockDim.x) {
      Bf16x8 a = src[i];
      if (rp && !ro) {
        const Bf16x8 b = rp[i];
#pragma unroll
        for (int j = 0; j < 8; ++j)
          a.v[j] = __float2bfloat16_rn(__fadd_rn(__bfloat162float(a.v[j]), __bfloat162float(b.v[j])));
      }
      const Bf16x8 ww = wp[i];
      Bf16x8 o;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float n = __fmul_rn(__bfloat162float(a.v[j]), inv);
        // round the normalised value to bf16 before the weight, as the usual bf16 module does
        o.v[j] = __float2bfloat16_rn(__fmul_rn(__bfloat162float(__float2bfloat16_rn(n)), __bfloat162float(ww.v[j])));
      }
      yp[i] = o;
    }
  }
}

// The same row in registers (d <= 2048 * VPT): x, residual and weight are requested together, the
// row is touched once, and what is left is one memory latency, one block reduction and the
// stores. Sums run in rmsnorm_kernel's order, so the bits are the same. What it gives is beside the
// rule that picks it, in ka_rmsnorm.
template <int VPT>
__global__ void __launch_bounds__(256, VPT == 4 ? 2 : 4)
rmsnorm_reg_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ residual,
                   const __nv_bfloat16* __restrict__ w, __nv_bfloat16* __restrict__ y,
                   __nv_bfloat16* __restrict__ residual_out, int rows, int d, float eps) {
  __shared__ float s_warp[2][8];
  const int nvec = d / 8, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int flip = 0;
  for (int row = blockIdx.x; row < rows; row += gridDim.x, flip ^= 1) {
    const size_t off = static_cast<size_t>(row) * d;
    Bf16x8 a[VPT], b[VPT], ww[VPT];
#pragma unroll
    for (int k = 0; k < VPT; ++k) {
      const int i = threadIdx.x + k * 256;
      if (i >= nvec) continue;
      a[k] = reinterpret_cast<const Bf16x8*>(x + off)[i];
      if (residual) b[k] = reinterpret_cast<const Bf16x8*>(residual + off)[i];
      ww[k] = reinterpret_cast<const Bf16x8*>(w)[i];
    }
    float ss = 0.f;
#pragma unroll
    for (int k = 0; k < VPT; ++k) {
      const int i = threadIdx.x + k * 256;
      if (i >= nvec) continue;
      if (residual) {
#pragma unroll
        for (int j = 0; j < 8; ++j)
          a[k].v[j] = __float2bfloat16_rn(__fadd_rn(__bfloat162float(a[k].v[j]), __bfloat162float(b[k].v[j])));
        if (residual_out) reinterpret_cast<Bf16x8*>(residual_out + off)[i] = a[k];
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float f = __bfloat162float(a[k].v[j]);
        ss = __fmaf_rn(f, f, ss);
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss = __fadd_rn(ss, __shfl_xor_sync(0xffffffffu, ss, o));
    if (lane == 0) s_warp[flip][warp] = ss;
    __syncthreads();     // the other half of s_warp serves the next row, so one barrier per row is enough
    float total = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) total = __fadd_rn(total, s_warp[flip][k]);
    const float inv = __fdiv_rn(1.f, __fsqrt_rn(__fadd_rn(__fdiv_rn(total, static_cast<float>(d)), eps)));
#pragma unroll
    for (int k = 0; k < VPT; ++k) {
      const int i = threadIdx.x + k * 256;
      if (i >= nvec) continue;
      Bf16x8 o;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float n = __fmul_rn(__bfloat162float(a[k].v[j]), inv);
        o.v[j] = __float2bfloat16_rn(__fmul_rn(__bfloat162float(__float2bfloat16_rn(n)), __bfloat162float(ww[k].v[j])));
      }
      reinterpret_cast<Bf16x8*>(y + off)[i] = o;
    }
  }
}

// Rotary embedding, "rotate half" convention: for i < hd/2
//   out[i]        = x[i] * cos[pos, i] - x[i + hd/2] * sin[pos, i]
//   out[i + hd/2] = x[i + hd/2] * cos[pos, i] + x[i] * sin[pos, i]
// x: [tokens, heads, hd] (token stride given), cos/sin: [max_pos, hd/2] fp32, in place.
__global__ void __launch_bounds__(256)
rope_kernel(__nv_bfloat16* __restrict__ x, long long token_stride, const long long* __restrict__ positions,
            const float* __restrict__ cos_t, const float* __restrict__ sin_t, int tokens, int heads, int hd) {
  const int half = hd / 2;
  const long long total = static_cast<long long>(tokens) * heads * half;
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int j = static_cast<int>(i % half);
    const long long th = i / half;
    const int h = static_cast<int>(th % heads);
    const long long t = th / heads;
    const long long pos = positions[t];
    const float c = cos_t[pos * half + j], s = sin_t[pos * half + j];
    __nv_bfloat16* p = x + t * token_stride + static_cast<long long>(h) * hd;
    const float a = __bfloat162float(p[j]), b = __bfloat162float(p[j + half]);
    p[j] = __float2bfloat16_rn(__fsub_rn(__fmul_rn(a, c), __fmul_rn(b, s)));
    p[j + half] = __float2bfloat16_rn(__fadd_rn(__fmul_rn(b, c), __fmul_rn(a, s)));
  }
}

// The same rotation with 16-byte accesses: a thread takes eight consecutive pairs (j .. j + 7 and
// their partners in the second half). hd / 2 must be a multiple of 8, rows 16-byte aligned.
__global__ void __launch_bounds__(256)
rope_vec8_kernel(__nv_bfloat16* __restrict__ x, long long token_stride, const long long* __restrict__ positions,
                 const float* __restrict__ cos_t, const float* __restrict__ sin_t, int tokens, int heads, int hd) {
  const int half = hd / 2, groups = half / 8;
  const long long total = static_cast<long long>(tokens) * heads * groups;
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int j = static_cast<int>(i % groups) * 8;
    const long long th = i / groups;
    const int h = static_cast<int>(th % heads);
    const long long t = th / heads;
    const long long pos = positions[t];
    const float4* cp = reinterpret_cast<const float4*>(cos_t + pos * half + j);
    const float4* sp = reinterpret_cast<const float4*>(sin_t + pos * half + j);
    const float4 c0 = cp[0], c1 = cp[1], s0 = sp[0], s1 = sp[1];
    const float c[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
    const float sn[8] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w};
    __nv_bfloat16* p = x + t * token_stride + static_cast<long long>(h) * hd;
    Bf16x8 lo = *reinterpret_cast<const Bf16x8*>(p + j), hi = *reinterpret_cast<const Bf16x8*>(p + j + half);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const float a = __bfloat162float(lo.v[e]), b = __bfloat162float(hi.v[e]);
      lo.v[e] = __float2bfloat16_rn(__fsub_rn(__fmul_rn(a, c[e]), __fmul_rn(b, sn[e])));
      hi.v[e] = __float2bfloat16_rn(__fadd_rn(__fmul_rn(b, c[e]), __fmul_rn(a, sn[e])));
    }
    *reinterpret_cast<Bf16x8*>(p + j) = lo;
    *reinterpret_cast<Bf16x8*>(p + j + half) = hi;
  }
}

// The fused qkv projection cut into its parts with q and k rotated, and the way back:
//   kBackward = false: qkv [rows, (hq + 2 hkv) * 128] -> q, k (rotated), v, each [tokens, heads, 128]
//   kBackward = true:  dq, dk (rotated by the opposite angle), dv -> dqkv; rows past `tokens` are zeroed
// Bound by the bytes: every element is read once and written once, 16 bytes per access. A thread
// takes eight pairs of one head (rope_vec8_kernel's arithmetic, the same bits) for two tokens;
// a block is 32 heads x 8 groups of pairs, so no index is divided.
// 4096 tokens, 32 + 8 + 8 heads: slices, copies, rotation and their autograd took about 300 us of
// a layer's forward and backward, this takes two launches.
constexpr int kQkvTokens = 2;

template <bool kBackward>
__global__ void __launch_bounds__(256)
qkv_rope_kernel(__nv_bfloat16* __restrict__ qkv, long long qkv_stride, const long long* __restrict__ positions,
                const float* __restrict__ cos_t, const float* __restrict__ sin_t, __nv_bfloat16* __restrict__ q,
                __nv_bfloat16* __restrict__ k, __nv_bfloat16* __restrict__ v, int rows, int tokens, int hq, int hkv) {
  constexpr int kHd = 128, kHalf = 64;
  const int head = blockIdx.y * 32 + (threadIdx.x >> 3), j = (threadIdx.x & 7) * 8;
  if (head >= hq + 2 * hkv) return;
  __nv_bfloat16* part = head < hq ? q : (head < hq + hkv ? k : v);
  const int heads = head < hq ? hq : hkv, h = head < hq ? head : (head < hq + hkv ? head - hq : head - hq - hkv);
  const bool rotate = head < hq + hkv;
#pragma unroll
  for (int n = 0; n < kQkvTokens; ++n) {
    const long long t = static_cast<long long>(blockIdx.x) * kQkvTokens + n;
    if (t >= rows) return;
    __nv_bfloat16* joint = qkv + t * qkv_stride + static_cast<long long>(head) * kHd + j;
    __nv_bfloat16* own = part + (t * heads + h) * kHd + j;
    Bf16x8 lo, hi;
    if (t < tokens) {
      const __nv_bfloat16* src = kBackward ? own : joint;
      lo = *reinterpret_cast<const Bf16x8*>(src);
      hi = *reinterpret_cast<const Bf16x8*>(src + kHalf);
      if (rotate) {
        const long long pos = positions[t];
        const float4* cp = reinterpret_cast<const float4*>(cos_t + pos * kHalf + j);
        const float4* sp = reinterpret_cast<const float4*>(sin_t + pos * kHalf + j);
        const float4 c0 = cp[0], c1 = cp[1], s0 = sp[0], s1 = sp[1];
        const float c[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
        const float sn[8] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w};
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const float a = __bfloat162float(lo.v[e]), b = __bfloat162float(hi.v[e]);
          const float se = kBackward ? -sn[e] : sn[e];
          lo.v[e] = __float2bfloat16_rn(__fsub_rn(__fmul_rn(a, c[e]), __fmul_rn(b, se)));
          hi.v[e] = __float2bfloat16_rn(__fadd_rn(__fmul_rn(b, c[e]), __fmul_rn(a, se)));
        }
      }
    } else if constexpr (kBackward) {
#pragma unroll
      for (int e = 0; e < 8; ++e) lo.v[e] = hi.v[e] = __float2bfloat16_rn(0.f);
    } else {
      return;
    }
    __nv_bfloat16* dst = kBackward ? joint : own;
    *reinterpret_cast<Bf16x8*>(dst) = lo;
    *reinterpret_cast<Bf16x8*>(dst + kHalf) = hi;
  }
}

__device__ __forceinline__ float tanh_approx(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ float silu_f(float g) {
  // g * sigmoid(g) = g * (0.5 + 0.5 * tanh(g / 2)): one special-function op per element
  // (the result is rounded to bf16, tanh.approx is accurate to about 2^-11)
  return __fmul_rn(g, __fmaf_rn(0.5f, tanh_approx(__fmul_rn(0.5f, g)), 0.5f));
}

// out[r, j] = silu(gate[r, j]) * up[r, j]; gate/up are column halves of one [rows, 2f] tensor
// when up == gate + f (row stride 2f), or separate tensors.
__global__ void __launch_bounds__(256)
swiglu_kernel(const __nv_bfloat16* __restrict__ gate, const __nv_bfloat16* __restrict__ up, long long in_stride,
              __nv_bfloat16* __restrict__ out, int rows, int f) {
  const int nvec = f / 8;
  const long long total = static_cast<long long>(rows) * nvec;
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const long long r = i / nvec;
    const int c = static_cast<int>(i % nvec);
    const Bf16x8 g = reinterpret_cast<const Bf16x8*>(gate + r * in_stride)[c];
    const Bf16x8 u = reinterpret_cast<const Bf16x8*>(up + r * in_stride)[c];
    Bf16x8 o;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float a = __bfloat162float(__float2bfloat16_rn(silu_f(__bfloat162float(g.v[j]))));
      o.v[j] = __float2bfloat16_rn(__fmul_rn(a, __bfloat162float(u.v[j])));
    }
    reinterpret_cast<Bf16x8*>(out + r * static_cast<long long>(f))[c] = o;
  }
}

// Backward of SwiGLU: d_gate = d_out * up * (sig + g*sig*(1-sig)), d_up = d_out * silu(g).
__global__ void __launch_bounds__(256)
swiglu_bwd_kernel(const __nv_bfloat16* __restrict__ gate, const __nv_bfloat16* __restrict__ up, long long in_stride,
                  const __nv_bfloat16* __restrict__ d_out, __nv_bfloat16* __restrict__ d_gate,
                  __nv_bfloat16* __restrict__ d_up, long long dgrad_stride, int rows, int f) {
  const int nvec = f / 8;
  const long long total = static_cast<long long>(rows) * nvec;
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const long long r = i / nvec;
    const int c = static_cast<int>(i % nvec);
    const Bf16x8 g = reinterpret_cast<const Bf16x8*>(gate + r * in_stride)[c];
    const Bf16x8 u = reinterpret_cast<const Bf16x8*>(up + r * in_stride)[c];
    const Bf16x8 d = reinterpret_cast<const Bf16x8*>(d_out + r * static_cast<long long>(f))[c];
    Bf16x8 dg, du;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float gf = __bfloat162float(g.v[j]), uf = __bfloat162float(u.v[j]), df = __bfloat162float(d.v[j]);
      const float sig = __fdiv_rn(1.f, __fadd_rn(1.f, ex2_approx(__fmul_rn(-gf, kLog2e))));
      const float dsilu = __fmaf_rn(__fmul_rn(gf, sig), __fsub_rn(1.f, sig), sig);
      dg.v[j] = __float2bfloat16_rn(__fmul_rn(__fmul_rn(df, uf), dsilu));
      du.v[j] = __float2bfloat16_rn(__fmul_rn(df, __fmul_rn(gf, sig)));
    }
    reinterpret_cast<Bf16x8*>(d_gate + r * dgrad_stride)[c] = dg;
    reinterpret_cast<Bf16x8*>(d_up + r * dgrad_stride)[c] = du;
  }
}

// Backward of y = bf16(bf16(x * inv) * w).
//   dx = inv * (dy*w - n * mean(dy*w*n)),  n = x * inv;   dw_partial[chunk] = sum_rows dy * n
// One CTA per chunk of kRmsChunk rows (fixed, so the order in which rows enter d_w does not
// depend on the grid); 16 rows give 4096 tokens 256 CTAs, one wave of two per SM (64 rows left
// more than half of the SMs idle: 92 us). With `d_res` the gradient that reaches x past the norm
// (the residual stream) is added to the rounded dx, which saves a pass. Threads own columns. kRows
// rows are worked on at once (two up to d = 2048, else one): their x and dy vectors are loaded once into
// registers and serve both steps (the two sums, then dx / dw), and the sums of all of them share one
// block reduction with a single barrier.
constexpr int kRmsChunk = 16;

// Fixed-order sums of R values per thread over the CTA (8 warps): lanes by xor-shuffle, then the
// eight warp sums left to right, the same in every thread. One barrier: the caller alternates
// between two halves of shared memory.
template <int R>
__device__ __forceinline__ void block_sum_fixed_multi(float (&v)[R], float (*s_warp)[8]) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int r = 0; r < R; ++r) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v[r] = __fadd_rn(v[r], __shfl_xor_sync(0xffffffffu, v[r], o));
    if (lane == 0) s_warp[r][warp] = v[r];
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < R; ++r) {
    float t = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) t = __fadd_rn(t, s_warp[r][w]);
    v[r] = t;
  }
}

__device__ __forceinline__ void unpack2(uint32_t w, float& lo, float& hi) {
  lo = __uint_as_float(w << 16);
  hi = __uint_as_float(w & 0xFFFF0000u);
}

// VPT: 16-byte vectors per thread and row (d <= 2048 * VPT); kRows: rows in flight. Both sums of a
// row, x^2 and (dy*w)*x, are taken in one pass (the mean of dy*w*n is the second times inv / d), and
// the next rows are loaded before the reduction where the registers allow it (VPT <= 2): with a
// reduction each and the loads behind them, 4096 rows of 4096 took 51 us, 38 us this way.
template <int VPT, int kRows>
__global__ void __launch_bounds__(256, 2)
rmsnorm_bwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w,
                   const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ d_res,
                   __nv_bfloat16* __restrict__ dx, float* __restrict__ dw_part, int rows, int d, float eps) {
  constexpr bool kAhead = VPT <= 2;
  __shared__ float s_warp[2][2 * kRows][8];
  const int chunk = blockIdx.x;
  const int r0 = chunk * kRmsChunk, r1 = min(rows, r0 + kRmsChunk);
  const int nvec = d / 8;
  const float inv_d = __fdiv_rn(1.f, static_cast<float>(d));
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  float dw_acc[VPT][8];
  uint4 wv[VPT];
#pragma unroll
  for (int a = 0; a < VPT; ++a) {
    const int i = threadIdx.x + a * 256;
    if (kAhead) wv[a] = i < nvec ? reinterpret_cast<const uint4*>(w)[i] : zero;
#pragma unroll
    for (int j = 0; j < 8; ++j) dw_acc[a][j] = 0.f;
  }
  auto weight = [&](int a) {                  // kept, or re-read (it stays in L1)
    const int i = threadIdx.x + a * 256;
    if constexpr (kAhead) return wv[a];
    return i < nvec ? reinterpret_cast<const uint4*>(w)[i] : zero;
  };
  uint4 xv[kRows][VPT], gv[kRows][VPT];
  auto load = [&](int row0, uint4 (&xs)[kRows][VPT], uint4 (&gs)[kRows][VPT]) {
#pragma unroll
    for (int r = 0; r < kRows; ++r)
#pragma unroll
      for (int a = 0; a < VPT; ++a) {
        const int i = threadIdx.x + a * 256;
        const bool in = row0 + r < r1 && i < nvec;
        xs[r][a] = in ? reinterpret_cast<const uint4*>(x + static_cast<size_t>(row0 + r) * d)[i] : zero;
        gs[r][a] = in ? reinterpret_cast<const uint4*>(dy + static_cast<size_t>(row0 + r) * d)[i] : zero;
      }
  };
  int flip = 0;
  if (kAhead) load(r0, xv, gv);
#pragma unroll 1
  for (int row0 = r0; row0 < r1; row0 += kRows, flip ^= 1) {
    uint4 nx[kAhead ? kRows : 1][VPT], ng[kAhead ? kRows : 1][VPT];
    if constexpr (kAhead)
      load(row0 + kRows, nx, ng);
    else
      load(row0, xv, gv);
    float red[2 * kRows];
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
      float ss = 0.f, dot = 0.f;
#pragma unroll
      for (int a = 0; a < VPT; ++a) {
        const uint4 wa = weight(a);
        const uint32_t* xw = reinterpret_cast<const uint32_t*>(&xv[r][a]);
        const uint32_t* gw = reinterpret_cast<const uint32_t*>(&gv[r][a]);
        const uint32_t* ww = reinterpret_cast<const uint32_t*>(&wa);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          float x0, x1, g0, g1, w0, w1;
          unpack2(xw[j], x0, x1);
          unpack2(gw[j], g0, g1);
          unpack2(ww[j], w0, w1);
          ss = __fmaf_rn(x0, x0, ss);
          ss = __fmaf_rn(x1, x1, ss);
          dot = __fmaf_rn(__fmul_rn(g0, w0), x0, dot);
          dot = __fmaf_rn(__fmul_rn(g1, w1), x1, dot);
        }
      }
      red[2 * r] = ss;
      red[2 * r + 1] = dot;
    }
    block_sum_fixed_multi<2 * kRows>(red, s_warp[flip]);
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
      const int row = row0 + r;
      if (row >= r1) break;  // uniform over the CTA
      const float inv = __fdiv_rn(1.f, __fsqrt_rn(__fadd_rn(__fdiv_rn(red[2 * r], static_cast<float>(d)), eps)));
      const float mean_dot = __fmul_rn(__fmul_rn(red[2 * r + 1], inv), inv_d);
#pragma unroll
      for (int a = 0; a < VPT; ++a) {
        const int i = threadIdx.x + a * 256;
        if (i >= nvec) continue;
        const uint32_t* xw = reinterpret_cast<const uint32_t*>(&xv[r][a]);
        const uint32_t* gw = reinterpret_cast<const uint32_t*>(&gv[r][a]);
        const uint4 wa = weight(a);
        const uint32_t* ww = reinterpret_cast<const uint32_t*>(&wa);
        uint4 rr = zero;
        if (d_res) rr = reinterpret_cast<const uint4*>(d_res + static_cast<size_t>(row) * d)[i];
        const uint32_t* rw = reinterpret_cast<const uint32_t*>(&rr);
        uint4 o;
        uint32_t* ow = reinterpret_cast<uint32_t*>(&o);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          float xf[2], gf[2], wf[2], rf[2];
          unpack2(xw[j], xf[0], xf[1]);
          unpack2(gw[j], gf[0], gf[1]);
          unpack2(ww[j], wf[0], wf[1]);
          unpack2(rw[j], rf[0], rf[1]);
          __nv_bfloat16 ob[2];
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const float n = __fmul_rn(xf[e], inv);
            ob[e] = __float2bfloat16_rn(__fmul_rn(inv, __fmaf_rn(-n, mean_dot, __fmul_rn(gf[e], wf[e]))));
            dw_acc[a][2 * j + e] = __fmaf_rn(gf[e], n, dw_acc[a][2 * j + e]);  // rows enter in increasing order
            if (d_res) ob[e] = __float2bfloat16_rn(__fadd_rn(__bfloat162float(ob[e]), rf[e]));
          }
          ow[j] = static_cast<uint32_t>(__bfloat16_as_ushort(ob[0])) |
                  (static_cast<uint32_t>(__bfloat16_as_ushort(ob[1])) << 16);
        }
        reinterpret_cast<uint4*>(dx + static_cast<size_t>(row) * d)[i] = o;
      }
    }
    if constexpr (kAhead) {
#pragma unroll
      for (int r = 0; r < kRows; ++r)
#pragma unroll
        for (int a = 0; a < VPT; ++a) {
          xv[r][a] = nx[r][a];
          gv[r][a] = ng[r][a];
        }
    }
  }
#pragma unroll
  for (int a = 0; a < VPT; ++a) {
    const int i = threadIdx.x + a * 256;
    if (i >= nvec) continue;
    float4* dst = reinterpret_cast<float4*>(dw_part + static_cast<size_t>(chunk) * d + i * 8);
    dst[0] = make_float4(dw_acc[a][0], dw_acc[a][1], dw_acc[a][2], dw_acc[a][3]);
    dst[1] = make_float4(dw_acc[a][4], dw_acc[a][5], dw_acc[a][6], dw_acc[a][7]);
  }
}

// d_w[c] = sum over chunks of dw_part[chunk][c]: eight interleaved sets of chunks (each in index
// order), then the sets in order. A block is 32 columns x 8 sets, so that 256 chunks are 32
// dependent adds and not 256.
__global__ void __launch_bounds__(256)
rmsnorm_dw_kernel(const float* __restrict__ dw_part, __nv_bfloat16* __restrict__ dw, int chunks, int d) {
  __shared__ float s_part[8][32];
  const int col = threadIdx.x & 31, set = threadIdx.x >> 5, c = blockIdx.x * 32 + col;
  float acc = 0.f;
  if (c < d) {
#pragma unroll 4
    for (int k = set; k < chunks; k += 8) acc = __fadd_rn(acc, dw_part[static_cast<size_t>(k) * d + c]);
  }
  s_part[set][col] = acc;
  __syncthreads();
  if (set == 0 && c < d) {
#pragma unroll
    for (int w = 1; w < 8; ++w) acc = __fadd_rn(acc, s_part[w][col]);
    dw[c] = __float2bfloat16_rn(acc);
  }
}

int grid_for(long long work_items, int threads, int num_sms) {
  long long g = (work_items + threads - 1) / threads;
  const long long cap = static_cast<long long>(num_sms) * 8;
  if (g > cap) g = cap;
  return g < 1 ? 1 : static_cast<int>(g);
}

// Whether every pointer is 16-byte aligned (null is).
template <typename... P>
bool aligned16(P... p) {
  return ((reinterpret_cast<uintptr_t>(p) | ...) & 15u) == 0;
}

}  // namespace
}  // namespace ka

extern "C" {

int ka_rmsnorm(const void* x, const void* residual, const void* w, void* y, void* residual_out, int rows, int d,
               float eps, int num_sms, void* stream) {
  using namespace ka;
  if (rows <= 0) return 0;
  if (d % 8 != 0) return -1;
  const int grid = rows < num_sms * 8 ? rows : num_sms * 8;
  // Rows that are all resident at once take the register kernel: what counts there is one row's latency.
  // With the residual add, loop / register kernel in us: d = 4096: 2.9 / 2.1 (8 rows), 4.4 / 3.6 (296), 4.8 / 4.4 (592);
  // d = 8192: 4.5 / 3.1 (8), 6.7 / 5.2 (296). With more rows the loop's eight CTAs per SM hide more of it
  // (d = 4096: 6.9 / 6.9 for 1024 rows, 92 / 96 for 16384; d = 8192: 8.7 / 8.8 for 512, 175 / 246 for 16384). Both give
  // the same bits.
  auto* kernel = rmsnorm_kernel;
  if (d <= 8192 && rows <= num_sms * (d <= 4096 ? 4 : 2))
    kernel = d <= 2048 ? rmsnorm_reg_kernel<1> : (d <= 4096 ? rmsnorm_reg_kernel<2> : rmsnorm_reg_kernel<4>);
  kernel<<<grid, 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const __nv_bfloat16*>(x), static_cast<const __nv_bfloat16*>(residual),
      static_cast<const __nv_bfloat16*>(w), static_cast<__nv_bfloat16*>(y), static_cast<__nv_bfloat16*>(residual_out),
      rows, d, eps);
  return cudaGetLastError() == cudaSuccess ? 0 : -11;
}

int ka_rope(void* x, long long token_stride, const long long* positions, const float* cos_t, const float* sin_t,
            int tokens, int heads, int hd, int num_sms, void* stream) {
  using namespace ka;
  if (tokens <= 0) return 0;
  if (hd % 2 != 0) return -1;
  if ((hd / 2) % 8 == 0 && token_stride % 8 == 0 && aligned16(x, cos_t, sin_t)) {
    const long long groups = static_cast<long long>(tokens) * heads * (hd / 16);
    rope_vec8_kernel<<<grid_for(groups, 256, num_sms), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<__nv_bfloat16*>(x), token_stride, positions, cos_t, sin_t, tokens, heads, hd);
    return cudaGetLastError() == cudaSuccess ? 0 : -11;
  }
  const long long total = static_cast<long long>(tokens) * heads * (hd / 2);
  rope_kernel<<<grid_for(total, 256, num_sms), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<__nv_bfloat16*>(x), token_stride, positions, cos_t, sin_t, tokens, heads, hd);
  return cudaGetLastError() == cudaSuccess ? 0 : -11;
}

// See qkv_rope_kernel. head_dim is 128, qkv [rows, width] with width = (hq + 2 hkv) * 128, positions [tokens] on
// the device; everything but the positions 16-byte aligned.
int ka_qkv_rope(void* qkv, long long qkv_stride, int width, const long long* positions, const float* cos_t,
                const float* sin_t, void* q, void* k, void* v, int rows, int tokens, int hq, int hkv, int backward,
                void* stream) {
  using namespace ka;
  if (rows <= 0) return 0;
  if (hq < 0 || hkv < 0 || width != (hq + 2 * hkv) * 128 || qkv_stride < width || qkv_stride % 8 != 0 || tokens > rows)
    return -1;
  if (!aligned16(qkv, cos_t, sin_t, q, k, v)) return -2;
  const dim3 grid(static_cast<unsigned>((rows + kQkvTokens - 1) / kQkvTokens),
                  static_cast<unsigned>((hq + 2 * hkv + 31) / 32));
  auto* kernel = backward ? qkv_rope_kernel<true> : qkv_rope_kernel<false>;
  kernel<<<grid, 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<__nv_bfloat16*>(qkv), qkv_stride, positions, cos_t, sin_t, static_cast<__nv_bfloat16*>(q),
      static_cast<__nv_bfloat16*>(k), static_cast<__nv_bfloat16*>(v), rows, tokens, hq, hkv);
  return cudaGetLastError() == cudaSuccess ? 0 : -11;
}

int ka_swiglu(const void* gate, const void* up, long long in_stride, void* out, int rows, int f, int num_sms,
              void* stream) {
  using namespace ka;
  if (rows <= 0) return 0;
  if (f % 8 != 0 || in_stride % 8 != 0) return -1;
  const long long total = static_cast<long long>(rows) * (f / 8);
  swiglu_kernel<<<grid_for(total, 256, num_sms), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const __nv_bfloat16*>(gate), static_cast<const __nv_bfloat16*>(up), in_stride,
      static_cast<__nv_bfloat16*>(out), rows, f);
  return cudaGetLastError() == cudaSuccess ? 0 : -11;
}

int ka_swiglu_bwd(const void* gate, const void* up, long long in_stride, const void* d_out, void* d_gate, void* d_up,
                  long long dgrad_stride, int rows, int f, int num_sms, void* stream) {
  using namespace ka;
  if (rows <= 0) return 0;
  if (f % 8 != 0 || in_stride % 8 != 0 || dgrad_stride % 8 != 0) return -1;
  const long long total = static_cast<long long>(rows) * (f / 8);
  swiglu_bwd_kernel<<<grid_for(total, 256, num_sms), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const __nv_bfloat16*>(gate), static_cast<const __nv_bfloat16*>(up), in_stride,
      static_cast<const __nv_bfloat16*>(d_out), static_cast<__nv_bfloat16*>(d_gate), static_cast<__nv_bfloat16*>(d_up),
      dgrad_stride, rows, f);
  return cudaGetLastError() == cudaSuccess ? 0 : -11;
}

// Rows per partial sum of the weight gradient (the size of dw_part follows from it).
int ka_rmsnorm_bwd_chunk() { return ka::kRmsChunk; }

// x, dy: [rows, d] bf16; d_res: null or [rows, d], added to dx; dx: [rows, d] bf16; dw: [d] bf16; dw_part: scratch of
// ceil(rows / ka_rmsnorm_bwd_chunk()) * d floats. d % 8 == 0 and d <= 8192; all but dw 16-byte aligned.
int ka_rmsnorm_bwd(const void* x, const void* w, const void* dy, const void* d_res, void* dx, void* dw, float* dw_part,
                   int rows, int d, float eps, void* stream) {
  using namespace ka;
  if (rows <= 0) return 0;
  if (d % 8 != 0 || d > 8192) return -1;
  if (!aligned16(x, w, dy, d_res, dx, dw_part)) return -2;
  const int chunks = (rows + kRmsChunk - 1) / kRmsChunk;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const __nv_bfloat16* xb = static_cast<const __nv_bfloat16*>(x);
  const __nv_bfloat16* wb = static_cast<const __nv_bfloat16*>(w);
  const __nv_bfloat16* gb = static_cast<const __nv_bfloat16*>(dy);
  const __nv_bfloat16* rb = static_cast<const __nv_bfloat16*>(d_res);
  __nv_bfloat16* ob = static_cast<__nv_bfloat16*>(dx);
  const int vpt = (d / 8 + 255) / 256;
  if (vpt <= 1)
    rmsnorm_bwd_kernel<1, 2><<<chunks, 256, 0, st>>>(xb, wb, gb, rb, ob, dw_part, rows, d, eps);
  else if (vpt == 2)
    rmsnorm_bwd_kernel<2, 1><<<chunks, 256, 0, st>>>(xb, wb, gb, rb, ob, dw_part, rows, d, eps);
  else
    rmsnorm_bwd_kernel<4, 1><<<chunks, 256, 0, st>>>(xb, wb, gb, rb, ob, dw_part, rows, d, eps);
  rmsnorm_dw_kernel<<<(d + 31) / 32, 256, 0, st>>>(dw_part, static_cast<__nv_bfloat16*>(dw), chunks, d);
  return cudaGetLastError() == cudaSuccess ? 0 : -11;
}

}  // extern "C"
