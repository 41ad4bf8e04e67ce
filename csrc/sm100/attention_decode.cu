// Single-token attention against a KV cache (rollout phase), grouped KV heads, head_dim 128.
//
// What bounds it is the read of the cache, so the keys of a sequence are spread over enough
// CTAs that their loads fill the memory pipe, every K and V row is loaded once, 16 bytes per
// lane, for all query heads of its GQA group, and the instructions per key are kept few.
//
//   * Keys are cut into blocks of 64. Block i belongs to stripe i % 8, and inside a block warp w
//     of the CTA's four takes keys [16 w, 16 w + 16). A warp keeps its own running (max, sum, acc)
//     of a stripe: the loop over blocks has no CTA-wide barrier, and the loads of the next block
//     are in flight while the current one is computed.
//   * Scores: mma.sync m16n8k16 with the 16 keys as rows and the heads of the group as columns
//     (products of bf16 are exact, sums in fp32). The K rows are loaded 16 bytes per lane straight
//     into A fragments: the head dimension is permuted, the same way for K and q, which a dot
//     product does not notice. With the scores on the fp32 pipe (32 sums over 16 lanes per half-warp)
//     the instructions took as long as the bytes: 70 us where this takes 59 us (64 x 875 keys,
//     32 / 8 heads; one CTA per sequence and KV head without any of this took 109 us). P V stays on the fp32 pipe: probabilities and
//     accumulators are fp32.
//   * The states of stripes 0-3 and of stripes 4-7 are folded in stripe order, per warp, and the
//     eight folded states (2 halves x 4 warps) are merged in order. This decomposition depends on
//     the number of keys alone, so a row's bits do not depend on its batch. How many CTAs work on
//     a (sequence, KV head) does: a cluster of S = 2, 4 or 8 takes 8 / S stripes each, the
//     largest S whose CTAs are all resident at once. With S = 2 a CTA folds its own stripes; the
//     rest is read from the other CTAs through distributed shared memory.
//
// The reference has no decode attention (its executor comments defer generation to a future
// vLLM integration, rl_engine/executors/rollout.py:33).
#include <cstdint>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math_constants.h>

#include "common/launch.cuh"
#include "common/ptx.cuh"

namespace ka {
namespace {

constexpr int kD = 128;
constexpr int kDecThreads = 128;
constexpr float kLog2e = 1.4426950408889634f;
constexpr int kMaxScoreBytes = 200 * 1024;             // shared memory for the scores of the general form

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
constexpr int kWarps = kDecThreads / 32;
constexpr int kWarpKeys = 16;                          // keys of a warp in a block: the rows of the MMA
constexpr int kBlockKeys = kWarps * kWarpKeys;

// A warp's state of a stripe (or of a fold of four): per head (max, sum) and the accumulator.
template <int GQ>
struct State {
  float ml[kWarps][GQ][2];
  float acc[kWarps][GQ][kD];
};

template <int GQ>
struct SplitSmem {
  float p[kWarps][kWarpKeys][GQ];
  float alpha[kWarps][GQ];
  // followed by State<GQ>[states per CTA]: one per stripe, or one folded state when splits == 2
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

// D[16 keys, 8 heads] += A[16, 16] * B[16, 8], bf16 in, fp32 out.
__device__ __forceinline__ void mma_16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                          uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
      "{%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
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

// Fold of two states, the same operations wherever it happens: weights first, then value by value.
struct FoldWeights {
  float m, w_old, w_new;
};
__device__ __forceinline__ FoldWeights fold_weights(float m_old, float m_new, float c) {
  FoldWeights f;
  f.m = fmaxf(m_old, m_new);
  f.w_old = state_weight(m_old, f.m, c);
  f.w_new = state_weight(m_new, f.m, c);
  return f;
}
__device__ __forceinline__ float fold_value(const FoldWeights& f, float v_old, float v_new) {
  return __fmaf_rn(f.w_new, v_new, __fmul_rn(f.w_old, v_old));
}

// CTAs of the split kernel that are resident on an SM: its registers are bounded for that many.
template <int GQ>
constexpr int kCtasPerSm = GQ == 8 ? 2 : 3;

template <int GQ>
__global__ void __launch_bounds__(kDecThreads, kCtasPerSm<GQ>)
attention_decode_split_kernel(const __nv_bfloat16* __restrict__ q, const __nv_bfloat16* __restrict__ cache_k,
                              const __nv_bfloat16* __restrict__ cache_v, const int* __restrict__ lens,
                              __nv_bfloat16* __restrict__ out, int hq, int hkv, int max_len, float scale, int splits) {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  SplitSmem<GQ>& sm = *reinterpret_cast<SplitSmem<GQ>*>(smem_raw);
  State<GQ>* states = reinterpret_cast<State<GQ>*>(smem_raw + sizeof(SplitSmem<GQ>));

  const int rank = static_cast<int>(cluster_ctarank());
  const int bh = blockIdx.x / splits;
  const int b = bh / hkv, hk = bh % hkv;
  const int n = lens[b];
  const int per_cta = kStripes / splits;
  const bool folded = splits == 2;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const float c = scale * kLog2e;
  const size_t kv_row = static_cast<size_t>(hkv) * kD;
  const size_t kv_off = (static_cast<size_t>(b) * max_len * hkv + hk) * kD;
  // K fragments: lane (g, t) holds keys g and g + 8, dimensions 32 i + 8 t .. + 7 (two K steps of
  // the MMA per 16-byte load). V: half-warp h holds keys 8 h .. 8 h + 7, lane ln dimensions 8 ln .. + 7.
  const int g8 = lane >> 2, t4 = lane & 3, half = lane >> 4, ln = lane & 15;
  const __nv_bfloat16* kbase = cache_k + kv_off + t4 * 8;
  const __nv_bfloat16* vbase = cache_v + kv_off + ln * 8;
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);

  uint4 qf[4];                     // B fragments: head g8 of the group, the same dimensions
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    qf[i] = zero;
    if (g8 < GQ) {
      const __nv_bfloat16* qp = q + (static_cast<size_t>(b) * hq + hk * GQ + g8) * kD + i * 32 + t4 * 8;
      uint32_t* w = reinterpret_cast<uint32_t*>(&qf[i]);
#pragma unroll
      for (int e = 0; e < 4; ++e)
        w[e] = static_cast<uint32_t>(__bfloat16_as_ushort(qp[2 * e])) |
               (static_cast<uint32_t>(__bfloat16_as_ushort(qp[2 * e + 1])) << 16);
    }
  }

  // The blocks of this CTA: stripes [rank * per_cta, (rank + 1) * per_cta), each stripe's blocks
  // in increasing order.
  const int n_blocks = (n + kBlockKeys - 1) / kBlockKeys;
  const int stripe0 = rank * per_cta, stripe_end = stripe0 + per_cta;
  uint4 kr[8], vr[8];
  auto load_k = [&](int blk) {
    const int key0 = blk * kBlockKeys + warp * kWarpKeys + g8;
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
      for (int i = 0; i < 4; ++i)
        kr[r * 4 + i] = key0 + 8 * r < n
                            ? *reinterpret_cast<const uint4*>(kbase + (key0 + 8 * r) * kv_row + i * 32)
                            : zero;
  };
  auto load_v = [&](int blk) {
    const int key0 = blk * kBlockKeys + warp * kWarpKeys + half * 8;
#pragma unroll
    for (int i = 0; i < 8; ++i)
      vr[i] = key0 + i < n ? *reinterpret_cast<const uint4*>(vbase + (key0 + i) * kv_row) : zero;
  };

  if (stripe0 < n_blocks) {
    load_k(stripe0);
    load_v(stripe0);
  }
  // this lane's two heads of the score fragment (columns 2 t and 2 t + 1) and whether they exist
  const int h0 = 2 * t4;
  const bool has0 = h0 < GQ, has1 = h0 + 1 < GQ;
  for (int stripe = stripe0; stripe < stripe_end; ++stripe) {
    if (stripe >= n_blocks) {      // no keys: an empty state where somebody reads one, nothing to fold otherwise
      if (!folded || stripe == stripe0) {
        State<GQ>& st = states[folded ? 0 : stripe - stripe0];
        if (lane < GQ) {
          st.ml[warp][lane][0] = -CUDART_INF_F;
          st.ml[warp][lane][1] = 0.f;
        }
      }
      continue;
    }
    float acc[GQ][8];
#pragma unroll
    for (int g = 0; g < GQ; ++g)
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[g][e] = 0.f;
    float m_run[2] = {-CUDART_INF_F, -CUDART_INF_F}, l_run[2] = {0.f, 0.f};
    for (int blk = stripe; blk < n_blocks; blk += kStripes) {
      int nblk = blk + kStripes;                    // the block after this one: of this stripe or the next
      if (nblk >= n_blocks) nblk = stripe + 1 < stripe_end ? stripe + 1 : n_blocks;
      float s[4] = {0.f, 0.f, 0.f, 0.f};            // (key g8, heads h0, h0 + 1), (key g8 + 8, the same)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        mma_16816(s, kr[i].x, kr[4 + i].x, kr[i].y, kr[4 + i].y, qf[i].x, qf[i].y);
        mma_16816(s, kr[i].z, kr[4 + i].z, kr[i].w, kr[4 + i].w, qf[i].z, qf[i].w);
      }
      if (nblk < n_blocks) load_k(nblk);
      const int key0 = blk * kBlockKeys + warp * kWarpKeys + g8;
      if (key0 >= n) s[0] = s[1] = -CUDART_INF_F;
      if (key0 + 8 >= n) s[2] = s[3] = -CUDART_INF_F;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        float mb = fmaxf(s[h], s[2 + h]);
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) mb = fmaxf(mb, __shfl_xor_sync(0xffffffffu, mb, o));
        const float m_new = fmaxf(m_run[h], mb);
        const float m_ref = m_new == -CUDART_INF_F ? 0.f : m_new;   // nothing but -inf so far: every weight is 0
        const float al = m_run[h] == -CUDART_INF_F ? 0.f : ex2_approx(__fmul_rn(__fsub_rn(m_run[h], m_ref), c));
        m_run[h] = m_new;
        const float p0 = key0 < n ? ex2_approx(__fmul_rn(__fsub_rn(s[h], m_ref), c)) : 0.f;
        const float p1 = key0 + 8 < n ? ex2_approx(__fmul_rn(__fsub_rn(s[2 + h], m_ref), c)) : 0.f;
        l_run[h] = __fadd_rn(__fmul_rn(l_run[h], al), __fadd_rn(p0, p1));
        if (h == 0 ? has0 : has1) {
          sm.p[warp][g8][h0 + h] = p0;
          sm.p[warp][g8 + 8][h0 + h] = p1;
          if (g8 == 0) sm.alpha[warp][h0 + h] = al;
        }
      }
      __syncwarp();
      float ag[GQ];
#pragma unroll
      for (int g = 0; g < GQ; ++g) ag[g] = sm.alpha[warp][g];
#pragma unroll
      for (int g = 0; g < GQ; ++g)
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[g][e] = __fmul_rn(acc[g][e], ag[g]);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        float vf[8], pg[GQ];
        unpack8(vr[i], vf);
#pragma unroll
        for (int g = 0; g < GQ; ++g) pg[g] = sm.p[warp][half * 8 + i][g];
#pragma unroll
        for (int g = 0; g < GQ; ++g)
#pragma unroll
          for (int e = 0; e < 8; e += 2) fma2(acc[g][e], acc[g][e + 1], pg[g], pg[g], vf[e], vf[e + 1]);
      }
      if (nblk < n_blocks) load_v(nblk);
      __syncwarp();                                 // p and alpha are rewritten by the next block
    }

    // ---- the warp's state of this stripe: sums over the lanes, then stored or folded
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int o = 4; o < 32; o <<= 1) l_run[h] = __fadd_rn(l_run[h], __shfl_xor_sync(0xffffffffu, l_run[h], o));
    // the two half-warps add their accumulators: half h keeps heads [h * GQ / 2, (h + 1) * GQ / 2)
    constexpr int kOwn = GQ == 1 ? 1 : GQ / 2;
    float own[kOwn][8];
#pragma unroll
    for (int g = 0; g < kOwn; ++g)
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        if constexpr (GQ == 1) {
          own[0][e] = __fadd_rn(acc[0][e], __shfl_xor_sync(0xffffffffu, acc[0][e], 16));
        } else {
          const float give = half ? acc[g][e] : acc[kOwn + g][e], keep = half ? acc[kOwn + g][e] : acc[g][e];
          own[g][e] = __fadd_rn(keep, __shfl_xor_sync(0xffffffffu, give, 16));
        }
      }
    State<GQ>& st = states[folded ? 0 : stripe - stripe0];
    const bool first = !folded || stripe == stripe0;
    const int head0 = GQ == 1 ? 0 : half * kOwn;
    float (*dst)[kD] = &st.acc[warp][head0];
    if (first) {
      if (g8 == 0) {
        if (has0) {
          st.ml[warp][h0][0] = m_run[0];
          st.ml[warp][h0][1] = l_run[0];
        }
        if (has1) {
          st.ml[warp][h0 + 1][0] = m_run[1];
          st.ml[warp][h0 + 1][1] = l_run[1];
        }
      }
      if (GQ > 1 || half == 0) {
#pragma unroll
        for (int g = 0; g < kOwn; ++g)
#pragma unroll
          for (int e = 0; e < 8; e += 4)
            *reinterpret_cast<float4*>(&dst[g][ln * 8 + e]) =
                make_float4(own[g][e], own[g][e + 1], own[g][e + 2], own[g][e + 3]);
      }
    } else {
      // every lane needs the maxima of the heads it keeps: head h sits in lanes t4 = h / 2, slot h % 2
      FoldWeights fw[kOwn];
#pragma unroll
      for (int g = 0; g < kOwn; ++g) {
        const int h = head0 + g;
        const float a = __shfl_sync(0xffffffffu, m_run[0], h >> 1), d = __shfl_sync(0xffffffffu, m_run[1], h >> 1);
        fw[g] = fold_weights(st.ml[warp][h][0], (h & 1) ? d : a, c);
      }
      __syncwarp();                                 // the old maxima have been read
      if (g8 == 0) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          if (!(h == 0 ? has0 : has1)) continue;
          float* ml = st.ml[warp][h0 + h];
          const FoldWeights f = fold_weights(ml[0], m_run[h], c);
          ml[0] = f.m;
          ml[1] = fold_value(f, ml[1], l_run[h]);
        }
      }
      if (GQ > 1 || half == 0) {
#pragma unroll
        for (int g = 0; g < kOwn; ++g)
#pragma unroll
          for (int e = 0; e < 8; e += 4) {
            float4* at = reinterpret_cast<float4*>(&dst[g][ln * 8 + e]);
            const float4 old = *at;
            *at = make_float4(fold_value(fw[g], old.x, own[g][e]), fold_value(fw[g], old.y, own[g][e + 1]),
                              fold_value(fw[g], old.z, own[g][e + 2]), fold_value(fw[g], old.w, own[g][e + 3]));
          }
      }
    }
    __syncwarp();                                   // the next stripe of this CTA reads the state
  }

  // ---- merge; CTA r of the cluster writes its share of the outputs
  cluster_arrive();
  cluster_wait();
  const int share = GQ * kD / splits;
  const uint32_t st_base = smem_u32(states);
  for (int i = tid; i < share; i += kDecThreads) {
    const int o = rank * share + i, g = o / kD, d = o % kD;
    float ms[2 * kWarps], ls[2 * kWarps], as[2 * kWarps];
    auto fetch = [&](int stripe, int w, float& m, float& l, float& a) {    // stripe: of the eight, or the fold 0 / 1
      const int owner = folded ? stripe : stripe / per_cta, slot = folded ? 0 : stripe % per_cta;
      const uint32_t at = mapa_u32(st_base + slot * static_cast<uint32_t>(sizeof(State<GQ>)), owner);
      const uint32_t ml = at + ((w * GQ + g) * 2) * 4;
      m = ld_cluster_f32(ml);
      l = ld_cluster_f32(ml + 4);
      a = ld_cluster_f32(at + static_cast<uint32_t>(sizeof(State<GQ>::ml)) + ((w * GQ + g) * kD + d) * 4);
      if (m == -CUDART_INF_F) a = 0.f;      // an empty state has no accumulator
    };
    if (folded) {
#pragma unroll
      for (int f = 0; f < 2; ++f)
#pragma unroll
        for (int w = 0; w < kWarps; ++w) fetch(f, w, ms[f * kWarps + w], ls[f * kWarps + w], as[f * kWarps + w]);
    } else {
#pragma unroll
      for (int f = 0; f < 2; ++f) {
        float m[4][kWarps], l[4][kWarps], a[4][kWarps];                    // all requested before the first is used
#pragma unroll
        for (int k = 0; k < 4; ++k)
#pragma unroll
          for (int w = 0; w < kWarps; ++w) fetch(f * 4 + k, w, m[k][w], l[k][w], a[k][w]);
#pragma unroll
        for (int w = 0; w < kWarps; ++w) {
#pragma unroll
          for (int k = 1; k < 4; ++k) {
            const FoldWeights fw = fold_weights(m[0][w], m[k][w], c);
            m[0][w] = fw.m;
            l[0][w] = fold_value(fw, l[0][w], l[k][w]);
            a[0][w] = fold_value(fw, a[0][w], a[k][w]);
          }
          ms[f * kWarps + w] = m[0][w];
          ls[f * kWarps + w] = l[0][w];
          as[f * kWarps + w] = a[0][w];
        }
      }
    }
    float M = ms[0];
#pragma unroll
    for (int s = 1; s < 2 * kWarps; ++s) M = fmaxf(M, ms[s]);
    float a = 0.f, l = 0.f;
#pragma unroll
    for (int s = 0; s < 2 * kWarps; ++s) {
      const float wt = state_weight(ms[s], M, c);
      l = __fmaf_rn(wt, ls[s], l);
      a = __fmaf_rn(wt, as[s], a);
    }
    out[(static_cast<size_t>(b) * hq + hk * GQ + g) * kD + d] = __float2bfloat16_rn(__fdiv_rn(a, l));
  }
  cluster_arrive();      // nobody leaves while its shared memory may still be read
  cluster_wait();
}

// Shared memory of a CTA that is one of `splits`: the fold (2), or a state per stripe (two with 4).
template <int GQ>
constexpr int split_smem(int splits) {
  return static_cast<int>(sizeof(SplitSmem<GQ>)) +
         (splits == 2 ? 1 : kStripes / splits) * static_cast<int>(sizeof(State<GQ>));
}

// Clusters of `splits` CTAs that are resident at once on the current device. Asked of the runtime, once per device:
// clusters must fit the SMs of a GPC, so there are fewer than kCtasPerSm * SMs / splits of them (64 / 8 heads, 9 x 448
// keys: 72 clusters of four are 288 CTAs for 296 places, but only 71 fit: 19.5 us, as clusters of two 12.2 us).
template <int GQ>
int resident_clusters(int splits) {
  static_assert(split_smem<GQ>(4) <= 48 * 1024, "the largest request, fits without an opt-in");
  static PerDevice once[kStripes + 1];
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  return once[splits].get(dev, [&] {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(splits));
    cfg.blockDim = dim3(kDecThreads);
    cfg.dynamicSmemBytes = static_cast<size_t>(split_smem<GQ>(splits));
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = static_cast<unsigned>(splits);
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, attention_decode_split_kernel<GQ>, &cfg) != cudaSuccess) {
      cudaGetLastError();
      return 0;
    }
    return n;
  });
}

// CTAs per (sequence, KV head): as many as are resident at once, and no more than the cache has blocks: a second wave,
// or CTAs without keys, cost a set-up and two cluster barriers for nothing (32 / 8 heads: 8 x 448 keys 10.0 us with
// S = 4, 13.7 with S = 8; 32 x 100 keys 14 us, 26 us without these limits; 64 / 8 heads, two CTAs per SM: 10 x 448 keys
// 14.6 us with S = 2, 20.2 with S = 4). The result does not depend on this choice.
template <int GQ>
int choose_splits(int batch, int hkv, int max_len) {
  const int blocks = (max_len + kBlockKeys - 1) / kBlockKeys;
  int splits = 2;
  while (splits < kStripes && splits < blocks &&
         static_cast<long long>(batch) * hkv <= resident_clusters<GQ>(splits * 2))
    splits *= 2;
  return splits;
}

template <int GQ>
int launch_split(const __nv_bfloat16* q, const __nv_bfloat16* k, const __nv_bfloat16* v, const int* lens,
                 __nv_bfloat16* out, int batch, int hq, int hkv, int max_len, float scale, cudaStream_t st) {
  const int splits = choose_splits<GQ>(batch, hkv, max_len);
  const int smem = split_smem<GQ>(splits);
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
  cfg.numAttrs = 1;
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
  if (head_dim != kD || hq % hkv != 0 || max_len * 4 > kMaxScoreBytes) return -1;
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
  // the limit and not this call's size: another thread may be about to launch with a longer cache
  static PerDevice once;
  if (smem > 40 * 1024 && !smem_opt_in(once, attention_decode_kernel, kMaxScoreBytes)) return -10;
  attention_decode_kernel<<<batch * hq, kDecThreads, smem, st>>>(qb, kb, vb, lens, ob, hq, hkv, max_len, scale);
  return cudaGetLastError() == cudaSuccess ? 0 : -11;
}

// How many CTAs ka_attention_decode puts on a (sequence, KV head) of an aligned cache on the current device; 1 for a
// grouping that the general form takes.
extern "C" int ka_attention_decode_splits(int batch, int hq, int hkv, int max_len) {
  using namespace ka;
  if (batch <= 0 || hkv <= 0 || hq % hkv != 0) return -1;
  switch (hq / hkv) {
    case 1: return choose_splits<1>(batch, hkv, max_len);
    case 2: return choose_splits<2>(batch, hkv, max_len);
    case 4: return choose_splits<4>(batch, hkv, max_len);
    case 8: return choose_splits<8>(batch, hkv, max_len);
    default: return 1;
  }
}
