// Single-token attention against a KV cache (rollout phase), grouped KV heads, head_dim 128.
//
// What bounds it is the read of the cache, so the keys of a sequence are spread over enough
// CTAs that their loads fill the memory pipe, and every K and V row is loaded once, 16 bytes
// per lane, for all query heads of its GQA group.
//
//   * Keys are cut into blocks of 8 * KPB. Block i belongs to stripe i % 8, and inside a block
//     half-warp w of the CTA's eight takes keys [w * KPB, (w + 1) * KPB). A half-warp covers a
//     row with 16 lanes x 8 dimensions and keeps its own running (max, sum, acc): the loop over
//     blocks has no CTA-wide barrier, and the loads of the next block are in flight while the
//     current one is computed.
//   * The eight half-warp states of a stripe are merged in half-warp order, the eight stripes in
//     stripe order. This decomposition depends on the number of keys alone, so a row's bits do
//     not depend on its batch. How many CTAs work on a (sequence, KV head) does: a cluster of
//     S = 1, 2, 4 or 8 CTAs takes 8 / S stripes each, the smallest S that gives about four CTAs
//     per SM, and the merge reads the other CTAs' stripes through distributed shared memory.
//   * Scores: fp32, summed over the 16 lanes by exchanging halves of the vector of (head, key)
//     partial sums, so 32 sums cost 30 shuffles instead of 128 and each lane ends up with the
//     scores whose exponentials it takes. Probabilities and accumulators stay in fp32.
//
// The reference has no decode attention (its executor comments defer generation to a future
// vLLM integration, rl_engine/executors/rollout.py:33).
#include <cstdint>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math_constants.h>

#include "common/ptx.cuh"

namespace ka {
namespace {

constexpr int kD = 128;
constexpr int kDecThreads = 128;
constexpr float kLog2e = 1.4426950408889634f;

// General form, any head grouping and any alignment of the cache: one CTA per query head.
// q: [B, Hq, D]; cache_k / cache_v: [B, max_len, Hkv, D]; lens[b]: valid keys (incl. the new
// token); out: [B, Hq, D].
__global__ void __launch_bounds__(kDecThreads)
attention_decode_kernel(const __nv_bfloat16* __restrict__ q, const __nv_bfloat16* __restrict__ cache_k,
                        const __nv_bfloat16* __restrict__ cache_v, const int* __restrict__ lens,
                        __nv_bfloat16* __restrict__ out, int hq, int hkv, int max_len, float scale) {
  extern __shared__ float s_scores[];  // [max_len]
  __shared__ float s_q[kD];
  __shared__ float s_red[kDecThreads / 32];
  const int b = blockIdx.x / hq, h = blockIdx.x % hq;
  const int hk = h / (hq / hkv);
  const int n = lens[b];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  s_q[tid] = __bfloat162float(q[(static_cast<size_t>(b) * hq + h) * kD + tid]);
  __syncthreads();
  const float c = scale * kLog2e;
  // scores: one warp per key, lanes split the head dimension
  float wmax = -CUDART_INF_F;
  for (int j = warp; j < n; j += kDecThreads / 32) {
    const __nv_bfloat16* kp = cache_k + ((static_cast<size_t>(b) * max_len + j) * hkv + hk) * kD;
    float acc = 0.f;
#pragma unroll
    for (int t = 0; t < kD / 32; ++t) acc = __fmaf_rn(s_q[lane + 32 * t], __bfloat162float(kp[lane + 32 * t]), acc);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc = __fadd_rn(acc, __shfl_xor_sync(0xffffffffu, acc, o));
    if (lane == 0) s_scores[j] = acc;
    wmax = fmaxf(wmax, acc);
  }
  if (lane == 0) s_red[warp] = wmax;
  __syncthreads();
  float m = s_red[0];
  for (int w = 1; w < kDecThreads / 32; ++w) m = fmaxf(m, s_red[w]);
  // probabilities; the normaliser is summed by one thread in key order
  for (int j = tid; j < n; j += kDecThreads) s_scores[j] = ex2_approx(__fmul_rn(__fsub_rn(s_scores[j], m), c));
  __syncthreads();
  // output: thread d owns one element of the head dimension, keys in order
  float acc = 0.f, l = 0.f;
  for (int j = 0; j < n; ++j) {
    const float p = s_scores[j];
    l = __fadd_rn(l, p);
    acc = __fmaf_rn(p, __bfloat162float(cache_v[((static_cast<size_t>(b) * max_len + j) * hkv + hk) * kD + tid]), acc);
  }
  out[(static_cast<size_t>(b) * hq + h) * kD + tid] = __float2bfloat16_rn(__fdiv_rn(acc, l));
}

constexpr int kStripes = 8;

template <int GQ>
struct Split {
  static constexpr int kKpb = GQ == 1 ? 16 : (GQ == 8 ? 4 : 8);   // keys per half-warp and block
  static constexpr int kScores = GQ * kKpb;                       // per half-warp and block: 16 or 32
  static constexpr int kOwn = kScores / 16;                       // scores a lane ends up with
  static constexpr int kLanesPerHead = 16 / GQ;
  static constexpr int kBlockKeys = 8 * kKpb;
};

// Shared memory: half-warp exchange of probabilities and states, then one state per stripe.
template <int GQ>
struct SplitSmem {
  float p[8][Split<GQ>::kKpb][GQ];
  float alpha[8][GQ];
  float hw_ml[8][GQ][2];
  float hw_acc[8][GQ][kD];
  float st_ml[kStripes][GQ][2];      // only the first 8 / S stripes are used
  // followed by float st_acc[8 / S][GQ][kD]
};

__device__ __forceinline__ void unpack8(const uint4& r, float (&f)[8]) {
  const uint32_t w[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    f[2 * i] = __uint_as_float(w[i] << 16);
    f[2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u);
  }
}

// (d0, d1) = (a0, a1) * (b0, b1) + (d0, d1), each lane rounded like fma.rn
__device__ __forceinline__ void fma2(float& d0, float& d1, float a0, float a1, float b0, float b1) {
  asm("{\n\t.reg .b64 ra, rb, rc;\n\tmov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\tmov.b64 rc, {%0, %1};\n\t"
      "fma.rn.f32x2 rc, ra, rb, rc;\n\tmov.b64 {%0, %1}, rc;\n\t}"
      : "+f"(d0), "+f"(d1)
      : "f"(a0), "f"(a1), "f"(b0), "f"(b1));
}

__device__ __forceinline__ float ld_cluster_f32(uint32_t addr) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
  return v;
}

// Weight of a partial state with maximum m against the merged maximum M; an empty state
// (m = -inf) weighs nothing, also when M is -inf.
__device__ __forceinline__ float state_weight(float m, float M, float c) {
  return m == -CUDART_INF_F ? 0.f : ex2_approx(__fmul_rn(__fsub_rn(m, M), c));
}

template <int GQ>
__global__ void __launch_bounds__(kDecThreads, GQ == 8 ? 2 : 3)
attention_decode_split_kernel(const __nv_bfloat16* __restrict__ q, const __nv_bfloat16* __restrict__ cache_k,
                              const __nv_bfloat16* __restrict__ cache_v, const int* __restrict__ lens,
                              __nv_bfloat16* __restrict__ out, int hq, int hkv, int max_len, float scale, int splits) {
  using T = Split<GQ>;
  constexpr int KPB = T::kKpb;
  extern __shared__ __align__(16) uint8_t smem_raw[];
  SplitSmem<GQ>& sm = *reinterpret_cast<SplitSmem<GQ>*>(smem_raw);
  float* st_acc = reinterpret_cast<float*>(smem_raw + sizeof(SplitSmem<GQ>));   // [8 / S][GQ][kD]

  const int rank = splits == 1 ? 0 : static_cast<int>(cluster_ctarank());
  const int bh = blockIdx.x / splits;
  const int b = bh / hkv, hk = bh % hkv;
  const int n = lens[b];
  const int per_cta = kStripes / splits;
  const int tid = threadIdx.x, hw = tid >> 4, ln = tid & 15;
  const float c = scale * kLog2e;
  const size_t kv_row = static_cast<size_t>(hkv) * kD;
  const __nv_bfloat16* kbase = cache_k + (static_cast<size_t>(b) * max_len * hkv + hk) * kD + ln * 8;
  const __nv_bfloat16* vbase = cache_v + (static_cast<size_t>(b) * max_len * hkv + hk) * kD + ln * 8;

  float qr[GQ][8];
#pragma unroll
  for (int g = 0; g < GQ; ++g)
#pragma unroll
    for (int e = 0; e < 8; ++e)
      qr[g][e] = __bfloat162float(q[(static_cast<size_t>(b) * hq + hk * GQ + g) * kD + ln * 8 + e]);

  // The blocks of this CTA: stripes [rank * per_cta, (rank + 1) * per_cta), each stripe's blocks
  // in increasing order. (stripe, block) walks that list.
  const int n_blocks = (n + T::kBlockKeys - 1) / T::kBlockKeys;
  const int stripe_end = (rank + 1) * per_cta;
  uint4 kr[KPB], vr[KPB];
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  auto load = [&](const __nv_bfloat16* base, int blk, uint4 (&r)[KPB]) {
    const int key0 = blk * T::kBlockKeys + hw * KPB;
#pragma unroll
    for (int i = 0; i < KPB; ++i)
      r[i] = key0 + i < n ? *reinterpret_cast<const uint4*>(base + (key0 + i) * kv_row) : zero;
  };

  int stripe = rank * per_cta;
  int blk = stripe;
  if (blk < n_blocks) {
    load(kbase, blk, kr);
    load(vbase, blk, vr);
  }
  for (; stripe < stripe_end; ++stripe) {
    float acc[GQ][8];
#pragma unroll
    for (int g = 0; g < GQ; ++g)
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[g][e] = 0.f;
    float m_run = -CUDART_INF_F, l_run = 0.f;      // of the head whose scores this lane owns
    for (blk = stripe; blk < n_blocks; blk += kStripes) {
      // the block after this one, in this stripe or at the start of the next
      int nblk = blk + kStripes;
      if (nblk >= n_blocks) nblk = stripe + 1 < stripe_end ? stripe + 1 : n_blocks;
      float s[T::kScores];                          // index = head * KPB + key
#pragma unroll
      for (int i = 0; i < KPB; ++i) {
        float kf[8];
        unpack8(kr[i], kf);
#pragma unroll
        for (int g = 0; g < GQ; ++g) {
          float a0 = 0.f, a1 = 0.f;
#pragma unroll
          for (int e = 0; e < 8; e += 2) fma2(a0, a1, qr[g][e], qr[g][e + 1], kf[e], kf[e + 1]);
          s[g * KPB + i] = __fadd_rn(a0, a1);
        }
      }
      if (nblk < n_blocks) load(kbase, nblk, kr);
      // sum over the 16 lanes: each step halves the vector, lane l keeps the part its bit names
#pragma unroll
      for (int step = 0; step < 4; ++step) {
        const int mask = 8 >> step, half = T::kScores >> (step + 1);
        const bool upper = (ln & mask) != 0;
#pragma unroll
        for (int i = 0; i < half; ++i) {
          const float keep = upper ? s[half + i] : s[i], give = upper ? s[i] : s[half + i];
          s[i] = __fadd_rn(keep, __shfl_xor_sync(0xffffffffu, give, mask));
        }
      }
      // lane ln owns scores ln * kOwn .. : head ln / kLanesPerHead
      const int own_head = ln / T::kLanesPerHead;
      const int own_key = (ln % T::kLanesPerHead) * T::kOwn;
      const int key0 = blk * T::kBlockKeys + hw * KPB + own_key;
      float mb = -CUDART_INF_F;
#pragma unroll
      for (int i = 0; i < T::kOwn; ++i) {
        if (key0 + i >= n) s[i] = -CUDART_INF_F;
        mb = fmaxf(mb, s[i]);
      }
#pragma unroll
      for (int o = T::kLanesPerHead >> 1; o > 0; o >>= 1) mb = fmaxf(mb, __shfl_xor_sync(0xffffffffu, mb, o));
      const float m_new = fmaxf(m_run, mb);
      const float m_ref = m_new == -CUDART_INF_F ? 0.f : m_new;   // nothing but -inf so far: every weight is 0
      const float al = m_run == -CUDART_INF_F ? 0.f : ex2_approx(__fmul_rn(__fsub_rn(m_run, m_ref), c));
      m_run = m_new;
      l_run = __fmul_rn(l_run, al);
#pragma unroll
      for (int i = 0; i < T::kOwn; ++i) {
        const float pr = ex2_approx(__fmul_rn(__fsub_rn(s[i], m_ref), c));
        l_run = __fadd_rn(l_run, pr);
        sm.p[hw][own_key + i][own_head] = pr;
      }
      if (ln % T::kLanesPerHead == 0) sm.alpha[hw][own_head] = al;
      __syncwarp();
      float ag[GQ];
#pragma unroll
      for (int g = 0; g < GQ; ++g) ag[g] = sm.alpha[hw][g];
#pragma unroll
      for (int g = 0; g < GQ; ++g)
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[g][e] = __fmul_rn(acc[g][e], ag[g]);
#pragma unroll
      for (int i = 0; i < KPB; ++i) {
        float vf[8], pg[GQ];
        unpack8(vr[i], vf);
#pragma unroll
        for (int g = 0; g < GQ; ++g) pg[g] = sm.p[hw][i][g];
#pragma unroll
        for (int g = 0; g < GQ; ++g)
#pragma unroll
          for (int e = 0; e < 8; e += 2) fma2(acc[g][e], acc[g][e + 1], pg[g], pg[g], vf[e], vf[e + 1]);
      }
      if (nblk < n_blocks) load(vbase, nblk, vr);
      __syncwarp();                                 // p and alpha are rewritten by the next block
    }
    // ---- merge the eight half-warps of this stripe (in order) into its state
#pragma unroll
    for (int o = T::kLanesPerHead >> 1; o > 0; o >>= 1) l_run = __fadd_rn(l_run, __shfl_xor_sync(0xffffffffu, l_run, o));
    if (ln % T::kLanesPerHead == 0) {
      sm.hw_ml[hw][ln / T::kLanesPerHead][0] = m_run;
      sm.hw_ml[hw][ln / T::kLanesPerHead][1] = l_run;
    }
#pragma unroll
    for (int g = 0; g < GQ; ++g)
#pragma unroll
      for (int e = 0; e < 8; e += 4)
        *reinterpret_cast<float4*>(&sm.hw_acc[hw][g][ln * 8 + e]) =
            make_float4(acc[g][e], acc[g][e + 1], acc[g][e + 2], acc[g][e + 3]);
    __syncthreads();
    const int ls = stripe - rank * per_cta;
#pragma unroll
    for (int g = 0; g < GQ; ++g) {
      float M = sm.hw_ml[0][g][0];
#pragma unroll
      for (int w = 1; w < 8; ++w) M = fmaxf(M, sm.hw_ml[w][g][0]);
      float a = 0.f, l = 0.f;
#pragma unroll
      for (int w = 0; w < 8; ++w) {
        const float wt = state_weight(sm.hw_ml[w][g][0], M, c);
        l = __fmaf_rn(wt, sm.hw_ml[w][g][1], l);
        a = __fmaf_rn(wt, sm.hw_acc[w][g][tid], a);
      }
      st_acc[(ls * GQ + g) * kD + tid] = a;
      if (tid == 0) {
        sm.st_ml[ls][g][0] = M;
        sm.st_ml[ls][g][1] = l;
      }
    }
    __syncthreads();
  }

  // ---- merge the stripes in order; CTA r of the cluster writes its share of the outputs
  if (splits > 1) {
    cluster_arrive();
    cluster_wait();
  }
  const int share = GQ * kD / splits;
  const uint32_t ml_base = smem_u32(&sm.st_ml[0][0][0]), acc_base = smem_u32(st_acc);
  for (int i = tid; i < share; i += kDecThreads) {
    const int o = rank * share + i, g = o / kD, d = o % kD;
    float ms[kStripes], lsum[kStripes], as[kStripes];
#pragma unroll
    for (int s = 0; s < kStripes; ++s) {
      const int owner = s / per_cta, ls = s - owner * per_cta;
      const uint32_t ml = ml_base + (ls * GQ + g) * 8, ac = acc_base + ((ls * GQ + g) * kD + d) * 4;
      if (splits > 1) {
        const uint32_t mlr = mapa_u32(ml, owner);
        ms[s] = ld_cluster_f32(mlr);
        lsum[s] = ld_cluster_f32(mlr + 4);
        as[s] = ld_cluster_f32(mapa_u32(ac, owner));
      } else {
        ms[s] = sm.st_ml[ls][g][0];
        lsum[s] = sm.st_ml[ls][g][1];
        as[s] = st_acc[(ls * GQ + g) * kD + d];
      }
    }
    float M = ms[0];
#pragma unroll
    for (int s = 1; s < kStripes; ++s) M = fmaxf(M, ms[s]);
    float a = 0.f, l = 0.f;
#pragma unroll
    for (int s = 0; s < kStripes; ++s) {
      const float wt = state_weight(ms[s], M, c);
      l = __fmaf_rn(wt, lsum[s], l);
      a = __fmaf_rn(wt, as[s], a);
    }
    out[(static_cast<size_t>(b) * hq + hk * GQ + g) * kD + d] = __float2bfloat16_rn(__fdiv_rn(a, l));
  }
  if (splits > 1) {      // nobody leaves while its shared memory may still be read
    cluster_arrive();
    cluster_wait();
  }
}

template <int GQ>
int launch_split(const __nv_bfloat16* q, const __nv_bfloat16* k, const __nv_bfloat16* v, const int* lens,
                 __nv_bfloat16* out, int batch, int hq, int hkv, int max_len, float scale, cudaStream_t st) {
  // About four CTAs per SM of a 148-SM device keep enough loads in flight; more CTAs than that
  // only add merges. (The result does not depend on this choice.)
  constexpr long long kWanted = 4 * 148;
  int splits = 1;
  while (splits < kStripes && static_cast<long long>(batch) * hkv * splits < kWanted) splits *= 2;
  const int smem = static_cast<int>(sizeof(SplitSmem<GQ>)) + kStripes / splits * GQ * kD * 4;
  if (smem > 48 * 1024 &&    // per device and cheap: set on every call that needs it
      cudaFuncSetAttribute(attention_decode_split_kernel<GQ>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) !=
          cudaSuccess)
    return -10;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(batch) * hkv * splits);
  cfg.blockDim = dim3(kDecThreads);
  cfg.dynamicSmemBytes = static_cast<size_t>(smem);
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = static_cast<unsigned>(splits);
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = splits > 1 ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, attention_decode_split_kernel<GQ>, q, k, v, lens, out, hq, hkv, max_len, scale,
                            splits) == cudaSuccess
             ? 0
             : -11;
}

}  // namespace
}  // namespace ka

// q [B, Hq, 128], caches [B, max_len, Hkv, 128] bf16, lens [B] int32 -> out [B, Hq, 128].
extern "C" int ka_attention_decode(const void* q, const void* cache_k, const void* cache_v, const int* lens, void* out,
                                   int batch, int hq, int hkv, int head_dim, int max_len, float scale, void* stream) {
  using namespace ka;
  if (batch <= 0) return 0;
  if (head_dim != kD || hq % hkv != 0 || max_len * 4 > 200 * 1024) return -1;
  const int gq = hq / hkv;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const __nv_bfloat16* qb = static_cast<const __nv_bfloat16*>(q);
  const __nv_bfloat16* kb = static_cast<const __nv_bfloat16*>(cache_k);
  const __nv_bfloat16* vb = static_cast<const __nv_bfloat16*>(cache_v);
  __nv_bfloat16* ob = static_cast<__nv_bfloat16*>(out);
  const bool aligned = ((reinterpret_cast<uintptr_t>(cache_k) | reinterpret_cast<uintptr_t>(cache_v)) & 15u) == 0;
  if (aligned) {
    switch (gq) {
      case 1: return launch_split<1>(qb, kb, vb, lens, ob, batch, hq, hkv, max_len, scale, st);
      case 2: return launch_split<2>(qb, kb, vb, lens, ob, batch, hq, hkv, max_len, scale, st);
      case 4: return launch_split<4>(qb, kb, vb, lens, ob, batch, hq, hkv, max_len, scale, st);
      case 8: return launch_split<8>(qb, kb, vb, lens, ob, batch, hq, hkv, max_len, scale, st);
      default: break;
    }
  }
  const int smem = max_len * 4;
  if (smem > 40 * 1024 && cudaFuncSetAttribute(attention_decode_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               smem) != cudaSuccess)
    return -10;
  attention_decode_kernel<<<batch * hq, kDecThreads, smem, st>>>(qb, kb, vb, lens, ob, hq, hkv, max_len, scale);
  return cudaGetLastError() == cudaSuccess ? 0 : -11;
}
