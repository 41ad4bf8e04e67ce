// Attention backward for sm_100a (causal / full, GQA, head_dim 128), deterministic: no atomics.
//
//   delta[b, h, i] = sum_d dO[i, d] * O[i, d]
//   P  = exp(scale * Q K^T - lse),   dP = dO V^T,   dS = P * (dP - delta) * scale
//   dQ = dS K            bwd_dq: one CTA per (sequence, q head, q tile),
//                        walks the KV tiles in increasing order, dQ accumulates in TMEM
//   dV = P^T dO, dK = dS^T Q   bwd_dkv: one CTA per (sequence, kv head,
//                        kv tile), walks (q head of the group, q tile) in a fixed order; it
//                        works on S^T = K Q^T so that its threads own KV rows
//
// All five products are tcgen05.mma 128 x 128 tiles; operands that are needed "transposed"
// (K and Q as [d, rows], dO as [d, rows]) are read through MN-major descriptors from the same
// TMA tiles, so nothing is transposed in memory. Every accumulation order is fixed, so the
// gradients are bitwise reproducible and independent of the batch.
//
// The reference has no attention kernel and no backward pass of any kind: it routes the op
// type "attention" to a backend name (rl_engine/kernels/registry.py:41-55).
#include <cstdint>
#include <type_traits>
#include <cuda_bf16.h>
#include <math_constants.h>

#include "common/bounded_wait.cuh"
#include "common/launch.cuh"
#include "common/ptx.cuh"
#include "common/tmap.cuh"
#include "attention_common.cuh"

namespace ka {
namespace {

constexpr int kD = 128;
constexpr int kT = 128;                    // tile rows (queries or keys)
constexpr int kParts = 4;                  // threads per TMEM lane
constexpr int kPartCols = kT / kParts;     // columns of a tile each of them takes
constexpr int kSoftThreads = kT * kParts;  // 16 warps
constexpr int kThreads = kSoftThreads + 64;  // + TMA warp + MMA warp
constexpr int kWarpTma = kSoftThreads / 32, kWarpMma = kSoftThreads / 32 + 1;
constexpr int kTileBytes = 128 * 128 * 2;
constexpr float kLog2e = 1.4426950408889634f;

struct BwdParams {
  const float* lse;     // [B, Hq, L]
  const float* delta;   // [B, Hq, L]
  __nv_bfloat16* dq;    // [B*L, Hq*128], token stride dq_stride
  __nv_bfloat16* dk;    // [B*L, Hkv*128]
  __nv_bfloat16* dv;
  long long dq_stride, dk_stride, dv_stride;
  int batch, seq_len, hq, hkv;
  float scale;
  int causal;
  int* status;
  unsigned long long timeout_ns;
};

// delta[b, h, i] = sum_d dO * O (fp32): 16 lanes x 16 bytes per (token, head), a block takes
// kDeltaTokens consecutive tokens of one head, so that its results are contiguous and every
// thread has four pairs of loads in flight (one 8-byte pair per warp and row took three times
// the time of the bytes: 34 us for 4096 tokens x 32 heads, 67 MB).
constexpr int kDeltaTokens = 64;

__global__ void __launch_bounds__(256)
attention_delta_kernel(const __nv_bfloat16* __restrict__ o, long long o_stride, const __nv_bfloat16* __restrict__ d_o,
                       long long do_stride, float* __restrict__ delta, int seq_len, int hq) {
  constexpr int kPer = kDeltaTokens / 16;
  const int groups = (seq_len + kDeltaTokens - 1) / kDeltaTokens;
  const int b = blockIdx.x / groups, h = blockIdx.y, ln = threadIdx.x & 15;
  const int i0 = (blockIdx.x % groups) * kDeltaTokens + (threadIdx.x >> 4);
  uint4 a[kPer], g[kPer];
#pragma unroll
  for (int n = 0; n < kPer; ++n) {
    const int i = i0 + n * 16;
    const long long tok = static_cast<long long>(b) * seq_len + i;
    if (i < seq_len) {
      a[n] = *reinterpret_cast<const uint4*>(o + tok * o_stride + h * kD + ln * 8);
      g[n] = *reinterpret_cast<const uint4*>(d_o + tok * do_stride + h * kD + ln * 8);
    } else {
      a[n] = g[n] = make_uint4(0u, 0u, 0u, 0u);
    }
  }
#pragma unroll
  for (int n = 0; n < kPer; ++n) {
    const uint32_t x[4] = {a[n].x, a[n].y, a[n].z, a[n].w}, y[4] = {g[n].x, g[n].y, g[n].z, g[n].w};
    float acc = 0.f;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      acc = __fmaf_rn(__uint_as_float(x[e] << 16), __uint_as_float(y[e] << 16), acc);
      acc = __fmaf_rn(__uint_as_float(x[e] & 0xFFFF0000u), __uint_as_float(y[e] & 0xFFFF0000u), acc);
    }
#pragma unroll
    for (int off = 8; off > 0; off >>= 1) acc = __fadd_rn(acc, __shfl_xor_sync(0xffffffffu, acc, off));
    const int i = i0 + n * 16;
    if (ln == 0 && i < seq_len) delta[(static_cast<long long>(b) * hq + h) * seq_len + i] = acc;
  }
}

// (d0, d1) = (a0, a1) * (b0, b1), each lane rounded like mul.rn
__device__ __forceinline__ void mul2(float& d0, float& d1, float a0, float a1, float b0, float b1) {
  asm("{\n\t.reg .b64 ra, rb, rd;\n\tmov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\t"
      "mul.rn.f32x2 rd, ra, rb;\n\tmov.b64 {%0, %1}, rd;\n\t}"
      : "=f"(d0), "=f"(d1)
      : "f"(a0), "f"(a1), "f"(b0), "f"(b1));
}

// 32 consecutive fp32 values of a row, as bf16.
__device__ __forceinline__ void store_row32(__nv_bfloat16* dst, const uint32_t (&v)[32]) {
#pragma unroll
  for (int i = 0; i < 32; i += 8)
    *reinterpret_cast<uint4*>(dst + i) = make_uint4(pack_bf16(__uint_as_float(v[i]), __uint_as_float(v[i + 1])),
                                                    pack_bf16(__uint_as_float(v[i + 2]), __uint_as_float(v[i + 3])),
                                                    pack_bf16(__uint_as_float(v[i + 4]), __uint_as_float(v[i + 5])),
                                                    pack_bf16(__uint_as_float(v[i + 6]), __uint_as_float(v[i + 7])));
}

// Offset (in 16-byte descriptor units) of K step kk of a 128 x 128 tile: K-major, MN-major.
__device__ __forceinline__ constexpr uint64_t kstep(int kk) { return ((kk >> 2) * 16384 + (kk & 3) * 32) >> 4; }
__device__ __forceinline__ constexpr uint64_t mnstep(int kk) { return (kk * 2048) >> 4; }
// Column of K step kk of a bf16 A operand that overlays a 128-column fp32 region: the threads of a
// part write 16 packed columns over the first half of their own 32 fp32 columns.
__device__ __forceinline__ constexpr uint32_t tcol(int kk) { return (kk >> 1) * kPartCols + (kk & 1) * 8; }

// ------------------------------------------------------------------------------------------------
// Both kernels overlap the tensor core with the element-wise work: the operand of the next
// iteration is in a second shared-memory stage, the next S and dP products are issued as soon as
// their TMEM columns have been read, and the 16-bit operand that comes out of S goes back to TMEM
// over the columns of S (the A operand of the product that follows), which leaves shared memory
// to the loaded tiles. Sixteen warps share a tile (eight issued in a quarter of the cycles: with two
// warps per scheduler nothing covers the TMEM loads and barriers), and tiles that need no mask
// run a loop of their own, without comparisons.
// One iteration is three products of 512 cycles (dQ) or four (dK / dV); with a single stage and
// everything in sequence it took about 9000 cycles. B = 2, L = 4000, 32 / 8 heads, causal:
// dQ 891 -> 500 us, dK / dV 1466 -> 530 us; B = 8, L = 512: dQ 114 -> 66 us, dK / dV 173 -> 62 us.
// ------------------------------------------------------------------------------------------------
struct CtlDq {
  uint64_t qdo_full, do_full;        // Q tile loaded, dO tile loaded
  uint64_t kv_full[3], kv_empty[3];  // K tiles: read by S and, an elementwise pass later, by dQ
  uint64_t v_full[2], v_empty[2];    // V tiles: read by dP alone
  uint64_t s_full[2];                // S ready in its TMEM buffer
  uint64_t dp_full, dp_read;         // dP ready / read into registers (count: softmax warps)
  // dS written over S (count: softmax warps), one per S buffer: S(j + 1) and dP(j + 1) are issued before
  // the wait for dS(j), so the warps may finish tile j + 1 before that wait looks. With a single barrier
  // they would have passed two phases by then, and the wait for a parity would never end.
  uint64_t ds_full[2];
  uint64_t acc_full;                 // final dQ ready
  uint32_t tmem_base;
  int abort_flag;
};

// ------------------------------------------------------------------------------------------------
// dQ kernel. TMEM: S (two buffers), dP, dQ. Shared memory: Q, dO, three stages of K, two of V.
// An SM gets about 85 GB/s, so a pair of tiles takes 1400 cycles and the latency on top. With two stages of (K, V)
// that were handed back together, behind dQ(j), the load of tile j + 2 and then S(j + 2) followed one another in the time in which the warps
// took tile j + 1, and an iteration was 3800 cycles; V is handed back by dP(j) now and K has a third stage: 2770
// cycles, what the products of one CTA take to issue (S 590, dP 660, dQ 960: shared memory).
// ------------------------------------------------------------------------------------------------
constexpr int kKStages = 3;
__device__ __forceinline__ void
bwd_dq(const CUtensorMap& tm_q, const CUtensorMap& tm_k, const CUtensorMap& tm_v, const CUtensorMap& tm_do,
       const BwdParams& p, int block) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const uint32_t base = smem_u32(smem_raw);
  const uint32_t q_tile = base, do_tile = base + kTileBytes, k_ring = base + 2 * kTileBytes,
                 v_ring = base + (2 + kKStages) * kTileBytes;
  CtlDq* ctl = reinterpret_cast<CtlDq*>(smem_raw + (4 + kKStages) * kTileBytes);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n_qt = (p.seq_len + kT - 1) / kT;
  const int qt = n_qt - 1 - block % n_qt;
  const int bh = block / n_qt;
  const int h = bh % p.hq, b = bh / p.hq;
  const int hk = h / (p.hq / p.hkv);
  const int q_row0 = qt * kT, tok0 = b * p.seq_len;
  const int kv_end = p.causal ? min(p.seq_len, q_row0 + kT) : p.seq_len;
  const int n_kv = (kv_end + kT - 1) / kT;
  WaitCtx wctx{&ctl->abort_flag, p.status, p.timeout_ns};

  if (threadIdx.x == 0) {
    mbar_init(smem_u32(&ctl->qdo_full), 1);
    mbar_init(smem_u32(&ctl->do_full), 1);
    for (int s = 0; s < kKStages; ++s) {
      mbar_init(smem_u32(&ctl->kv_full[s]), 1);
      mbar_init(smem_u32(&ctl->kv_empty[s]), 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(smem_u32(&ctl->v_full[s]), 1);
      mbar_init(smem_u32(&ctl->v_empty[s]), 1);
      mbar_init(smem_u32(&ctl->s_full[s]), 1);
      mbar_init(smem_u32(&ctl->ds_full[s]), kSoftThreads / 32);
    }
    mbar_init(smem_u32(&ctl->dp_full), 1);
    mbar_init(smem_u32(&ctl->dp_read), kSoftThreads / 32);
    mbar_init(smem_u32(&ctl->acc_full), 1);
    ctl->abort_flag = 0;
    fence_mbar_init_cluster();
  }
  if (warp == kWarpMma) {
    tmem_alloc<1>(smem_u32(&ctl->tmem_base), 512);
    tmem_relinquish<1>();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = ctl->tmem_base;
  const uint32_t tmem_dp = tmem_base + 256, tmem_dq = tmem_base + 384;   // S: tmem_base + 128 * buffer

  if (warp == kWarpTma) {
    if (lane == 0) {
      auto load = [&](uint32_t dst, const CUtensorMap& tm, int col, int row, uint64_t* bar) {
        const uint32_t full = smem_u32(bar);
        mbar_arrive_expect_tx(full, kTileBytes);
        tma_load_2d(dst, &tm, col, row, full);
        tma_load_2d(dst + 16384, &tm, col + 64, row, full);
      };
      load(q_tile, tm_q, h * kD, tok0 + q_row0, &ctl->qdo_full);
      load(k_ring, tm_k, hk * kD, tok0, &ctl->kv_full[0]);
      load(do_tile, tm_do, h * kD, tok0 + q_row0, &ctl->do_full);
      // V(j), then K(j + 1): the products that hand the stages back come in that order
      int ks = 1;
      uint32_t kphase = 1;
      for (int j = 0; j < n_kv; ++j) {
        if (!mbar_wait_bounded(smem_u32(&ctl->v_empty[j & 1]), ((j >> 1) & 1) ^ 1u, wctx, 41, j)) break;
        load(v_ring + (j & 1) * kTileBytes, tm_v, hk * kD, tok0 + j * kT, &ctl->v_full[j & 1]);
        if (j + 1 == n_kv) break;
        if (!mbar_wait_bounded(smem_u32(&ctl->kv_empty[ks]), kphase, wctx, 41, j + 1)) break;
        load(k_ring + ks * kTileBytes, tm_k, hk * kD, tok0 + (j + 1) * kT, &ctl->kv_full[ks]);
        if (++ks == kKStages) {
          ks = 0;
          kphase ^= 1u;
        }
      }
    }
  } else if (warp == kWarpMma) {
    if (lane == 0) {
      const uint32_t idesc_kk = umma_idesc_bf16_f32(kT, kT);             // both operands K-major
      const uint32_t idesc_kmn = umma_idesc_bf16_f32(kT, kD) | (1u << 16);  // B MN-major
      const uint64_t d_q = desc_kmajor(q_tile, 0), d_do = desc_kmajor(do_tile, 0), d_k = desc_kmajor(k_ring, 0),
                     d_k_mn = desc_mnmajor(k_ring, 0), d_v = desc_kmajor(v_ring, 0);
      constexpr uint64_t kTile = kTileBytes >> 4;
      auto issue_s = [&](int j, int ks) {      // S = Q K^T
        const uint64_t dk = d_k + ks * kTile;
#pragma unroll
        for (int kk = 0; kk < kD / 16; ++kk)
          umma_bf16<1>(tmem_base + (j & 1) * 128, d_q + kstep(kk), dk + kstep(kk), idesc_kk, kk > 0 ? 1u : 0u);
        umma_commit<1>(smem_u32(&ctl->s_full[j & 1]));
      };
      auto issue_dp = [&](int j) {     // dP = dO V^T
        const uint64_t dv = d_v + (j & 1) * kTile;
#pragma unroll
        for (int kk = 0; kk < kD / 16; ++kk)
          umma_bf16<1>(tmem_dp, d_do + kstep(kk), dv + kstep(kk), idesc_kk, kk > 0 ? 1u : 0u);
        umma_commit<1>(smem_u32(&ctl->dp_full));
        umma_commit<1>(smem_u32(&ctl->v_empty[j & 1]));
      };
      bool ok = mbar_wait_bounded(smem_u32(&ctl->qdo_full), 0, wctx, 42, 0) &&
                mbar_wait_bounded(smem_u32(&ctl->kv_full[0]), 0, wctx, 43, 0);
      if (ok) {
        tc_fence_after_sync();
        issue_s(0, 0);
        ok = mbar_wait_bounded(smem_u32(&ctl->do_full), 0, wctx, 42, 1) &&
             mbar_wait_bounded(smem_u32(&ctl->v_full[0]), 0, wctx, 43, 0);
      }
      if (ok) {
        tc_fence_after_sync();
        issue_dp(0);
      }
      int ks = 0;                      // stage of K(j)
      uint32_t kphase = 0;             // of K(j + 1)
      for (int j = 0; j < n_kv && ok; ++j) {
        const int ks_next = ks + 1 == kKStages ? 0 : ks + 1;
        if (ks_next == 0) kphase ^= 1u;
        if (j + 1 < n_kv) {
          // S(j + 1) goes over dS(j - 1), whose product was issued an iteration ago; the tensor
          // core executes in issue order
          ok = mbar_wait_bounded(smem_u32(&ctl->kv_full[ks_next]), kphase, wctx, 43, j + 1);
          if (!ok) break;
          tc_fence_after_sync();
          issue_s(j + 1, ks_next);
          ok = mbar_wait_bounded(smem_u32(&ctl->v_full[(j + 1) & 1]), ((j + 1) >> 1) & 1, wctx, 43, j + 1) &&
               mbar_wait_bounded(smem_u32(&ctl->dp_read), j & 1, wctx, 47, j);
          if (!ok) break;
          tc_fence_after_sync();
          issue_dp(j + 1);
        }
        ok = mbar_wait_bounded(smem_u32(&ctl->ds_full[j & 1]), (j >> 1) & 1, wctx, 44, j);
        if (!ok) break;
        tc_fence_after_sync();
        const uint64_t dk = d_k_mn + ks * kTile;
#pragma unroll
        for (int kk = 0; kk < kT / 16; ++kk)  // dQ += dS K
          umma_bf16_ts(tmem_dq, tmem_base + (j & 1) * 128 + tcol(kk), dk + mnstep(kk), idesc_kmn,
                       (j > 0 || kk > 0) ? 1u : 0u);
        umma_commit<1>(smem_u32(&ctl->kv_empty[ks]));
        if (j + 1 == n_kv) umma_commit<1>(smem_u32(&ctl->acc_full));
        ks = ks_next;
      }
    }
  } else {
    const int tid = threadIdx.x;
    const int row = tid & 127, part = tid >> 7;
    const int q_pos = q_row0 + row;
    const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const uint32_t part_base = lane_base + part * kPartCols;
    const float c = p.scale * kLog2e;
    const bool row_ok = q_pos < p.seq_len;
    const long long stat = (static_cast<long long>(b) * p.hq + h) * p.seq_len + q_pos;
    const float neg_lse2 = row_ok ? __fmul_rn(-p.lse[stat], kLog2e) : 0.f;
    const float neg_dlt = row_ok ? -p.delta[stat] : 0.f;
    bool ok = true;
    for (int j = 0; j < n_kv && ok; ++j) {
      bool mine = mbar_wait_bounded(smem_u32(&ctl->s_full[j & 1]), (j >> 1) & 1, wctx, 45, j);
      ok = __all_sync(0xffffffffu, mine) != 0;
      if (!ok) break;
      tc_fence_after_sync();
      const uint32_t tmem_s = tmem_base + static_cast<uint32_t>((j & 1) * 128) + part_base;
      uint32_t sv[32], gv[32], w[16];
      __syncwarp();
      tmem_ld_32x32(tmem_s, sv);
      tmem_ld_wait_dep(sv);
#pragma unroll
      for (int i = 0; i < 32; i += 2) {
        float e0, e1;
        fma2(e0, e1, __uint_as_float(sv[i]), __uint_as_float(sv[i + 1]), c, c, neg_lse2, neg_lse2);
        sv[i] = __float_as_uint(ex2_approx(e0));
        sv[i + 1] = __float_as_uint(ex2_approx(e1));
      }
      mine = mbar_wait_bounded(smem_u32(&ctl->dp_full), j & 1, wctx, 45, j);
      ok = __all_sync(0xffffffffu, mine) != 0;
      if (!ok) break;
      tc_fence_after_sync();
      __syncwarp();
      tmem_ld_32x32(tmem_dp + part_base, gv);
      tmem_ld_wait_dep(gv);
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&ctl->dp_read));
      auto grads = [&](auto masked, int limit) {      // limit: last allowed column of this part
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          float d0, d1;
          add2(d0, d1, __uint_as_float(gv[i]), __uint_as_float(gv[i + 1]), neg_dlt, neg_dlt);
          mul2(d0, d1, __uint_as_float(sv[i]), __uint_as_float(sv[i + 1]), d0, d1);
          mul2(d0, d1, d0, d1, p.scale, p.scale);
          if constexpr (decltype(masked)::value) {
            d0 = i > limit ? 0.f : d0;
            d1 = i + 1 > limit ? 0.f : d1;
          }
          w[i >> 1] = pack_bf16(d0, d1);
        }
      };
      if (p.causal ? j < qt : (j + 1) * kT <= p.seq_len)       // uniform over the CTA
        grads(std::false_type{}, 0);
      else
        grads(std::true_type{},
              row_ok ? (p.causal ? q_pos : p.seq_len - 1) - (j * kT + part * kPartCols) : -1);
      tmem_st_32x16(tmem_s, w);
      tmem_st_wait();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&ctl->ds_full[j & 1]));
    }
    if (ok && n_kv > 0) {
      const bool mine = mbar_wait_bounded(smem_u32(&ctl->acc_full), 0, wctx, 46, 0);
      ok = __all_sync(0xffffffffu, mine) != 0;
    }
    if (ok) {
      tc_fence_after_sync();
      __nv_bfloat16* dst = p.dq + static_cast<long long>(tok0 + q_pos) * p.dq_stride + h * kD + part * kPartCols;
      uint32_t v[32];
      __syncwarp();
      tmem_ld_32x32(tmem_dq + part_base, v);
      tmem_ld_wait_dep(v);
      if (row_ok) store_row32(dst, v);
    }
  }
  if (ctl->abort_flag) drain_in_flight();
  tc_fence_before_sync();
  __syncthreads();
  if (warp == kWarpMma) {
    __syncwarp();
    tc_fence_after_sync();
    tmem_dealloc<1>(tmem_base, 512);
  }
}

// ------------------------------------------------------------------------------------------------
// dK / dV kernel. TMEM: S^T (then P^T as bf16 over it), dP^T, dV, dK. Shared memory: K, V, two
// stages of (Q, dO), dS^T.
// ------------------------------------------------------------------------------------------------
struct CtlDkv {
  uint64_t kv_full, v_full;          // K tile loaded, V tile loaded (once)
  uint64_t qdo_full[2], qdo_empty[2];  // Q tiles: read by S^T and, last of all, by dK
  uint64_t do_full[2], do_empty[2];    // dO tiles: read by dP^T and dV
  uint64_t st_full;                  // S^T ready in TMEM
  uint64_t p_full;                   // P^T written over S^T (count: softmax warps)
  uint64_t dp_full, dp_read;         // dP^T ready / read into registers (count: softmax warps)
  uint64_t ds_full, ds_empty;        // dS^T tile written (count: softmax warps) / consumed
  uint64_t acc_full;
  uint32_t tmem_base;
  int abort_flag;
  alignas(16) float lse2[2][kT];     // -lse * log2(e) of the current q tile, double-buffered by iteration
  alignas(16) float neg_delta[2][kT];
};

__device__ __forceinline__ void
bwd_dkv(const CUtensorMap& tm_q, const CUtensorMap& tm_k, const CUtensorMap& tm_v, const CUtensorMap& tm_do,
        const BwdParams& p, int block) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const uint32_t base = smem_u32(smem_raw);
  const uint32_t k_tile = base, v_tile = base + kTileBytes, ring = base + 2 * kTileBytes,   // stage: Q, dO
                 dst_tile = base + 6 * kTileBytes;
  uint8_t* dst_ptr = smem_raw + 6 * kTileBytes;
  CtlDkv* ctl = reinterpret_cast<CtlDkv*>(smem_raw + 7 * kTileBytes);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n_t = (p.seq_len + kT - 1) / kT;
  // All CTAs of the early (causal: heavy) kv tiles first: the last CTAs to start are the lightest
  // (sequence by sequence the last heavy ones started when the rest was done: 1074 against 833 us).
  const int n_bh = p.batch * p.hkv;
  const int jt = block / n_bh;
  const int bh = block % n_bh;
  const int hk = bh % p.hkv, b = bh / p.hkv;
  const int group = p.hq / p.hkv;
  const int kv_row0 = jt * kT, tok0 = b * p.seq_len;
  const int qt0 = p.causal ? jt : 0;
  const int n_q = n_t - qt0;                                   // q tiles per head
  const int n_iter = group * n_q;
  WaitCtx wctx{&ctl->abort_flag, p.status, p.timeout_ns};

  if (threadIdx.x == 0) {
    mbar_init(smem_u32(&ctl->kv_full), 1);
    mbar_init(smem_u32(&ctl->v_full), 1);
    for (int s = 0; s < 2; ++s) {
      mbar_init(smem_u32(&ctl->qdo_full[s]), 1);
      mbar_init(smem_u32(&ctl->qdo_empty[s]), 1);
      mbar_init(smem_u32(&ctl->do_full[s]), 1);
      mbar_init(smem_u32(&ctl->do_empty[s]), 1);
    }
    mbar_init(smem_u32(&ctl->st_full), 1);
    mbar_init(smem_u32(&ctl->p_full), kSoftThreads / 32);
    mbar_init(smem_u32(&ctl->dp_full), 1);
    mbar_init(smem_u32(&ctl->dp_read), kSoftThreads / 32);
    mbar_init(smem_u32(&ctl->ds_full), kSoftThreads / 32);
    mbar_init(smem_u32(&ctl->ds_empty), 1);
    mbar_init(smem_u32(&ctl->acc_full), 1);
    ctl->abort_flag = 0;
    fence_mbar_init_cluster();
  }
  if (warp == kWarpMma) {
    tmem_alloc<1>(smem_u32(&ctl->tmem_base), 512);
    tmem_relinquish<1>();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = ctl->tmem_base;
  const uint32_t tmem_st = tmem_base, tmem_dpt = tmem_base + 128, tmem_dv = tmem_base + 256, tmem_dk = tmem_base + 384;

  if (warp == kWarpTma) {
    if (lane == 0) {
      auto load = [&](uint32_t dst, const CUtensorMap& tm, int col, int row, uint64_t* bar) {
        const uint32_t full = smem_u32(bar);
        mbar_arrive_expect_tx(full, kTileBytes);
        tma_load_2d(dst, &tm, col, row, full);
        tma_load_2d(dst + 16384, &tm, col + 64, row, full);
      };
      auto load_q = [&](int n) {
        const int h = hk * group + n / n_q, qt = qt0 + n % n_q, s = n & 1;
        if (!mbar_wait_bounded(smem_u32(&ctl->qdo_empty[s]), ((n >> 1) & 1) ^ 1u, wctx, 51, n)) return false;
        load(ring + s * 2 * kTileBytes, tm_q, h * kD, tok0 + qt * kT, &ctl->qdo_full[s]);
        return true;
      };
      auto load_do = [&](int n) {
        const int h = hk * group + n / n_q, qt = qt0 + n % n_q, s = n & 1;
        if (!mbar_wait_bounded(smem_u32(&ctl->do_empty[s]), ((n >> 1) & 1) ^ 1u, wctx, 51, n)) return false;
        load(ring + (s * 2 + 1) * kTileBytes, tm_do, h * kD, tok0 + qt * kT, &ctl->do_full[s]);
        return true;
      };
      load(k_tile, tm_k, hk * kD, tok0 + kv_row0, &ctl->kv_full);
      bool ok = n_iter > 0 && load_q(0);
      load(v_tile, tm_v, hk * kD, tok0 + kv_row0, &ctl->v_full);
      ok = ok && load_do(0);
      // dO(n - 2) is handed back by dV(n - 2), Q(n - 2) by dK(n - 2)
      for (int n = 1; n < n_iter && ok; ++n) ok = load_do(n) && load_q(n);
    }
  } else if (warp == kWarpMma) {
    if (lane == 0) {
      const uint32_t idesc_kk = umma_idesc_bf16_f32(kT, kT);
      const uint32_t idesc_kmn = umma_idesc_bf16_f32(kT, kD) | (1u << 16);
      const uint64_t d_k = desc_kmajor(k_tile, 0), d_v = desc_kmajor(v_tile, 0), d_ring = desc_kmajor(ring, 0),
                     d_ring_mn = desc_mnmajor(ring, 0), d_ds = desc_kmajor(dst_tile, 0);
      constexpr uint64_t kStage = (2 * kTileBytes) >> 4, kTile = kTileBytes >> 4;
      auto issue_st = [&](int n) {     // S^T = K Q^T
        const uint64_t dq = d_ring + (n & 1) * kStage;
#pragma unroll
        for (int kk = 0; kk < kD / 16; ++kk)
          umma_bf16<1>(tmem_st, d_k + kstep(kk), dq + kstep(kk), idesc_kk, kk > 0 ? 1u : 0u);
        umma_commit<1>(smem_u32(&ctl->st_full));
      };
      auto issue_dpt = [&](int n) {    // dP^T = V dO^T
        const uint64_t ddo = d_ring + (n & 1) * kStage + kTile;
#pragma unroll
        for (int kk = 0; kk < kD / 16; ++kk)
          umma_bf16<1>(tmem_dpt, d_v + kstep(kk), ddo + kstep(kk), idesc_kk, kk > 0 ? 1u : 0u);
        umma_commit<1>(smem_u32(&ctl->dp_full));
      };
      bool ok = mbar_wait_bounded(smem_u32(&ctl->kv_full), 0, wctx, 52, 0) &&
                mbar_wait_bounded(smem_u32(&ctl->qdo_full[0]), 0, wctx, 53, 0);
      if (ok) {
        tc_fence_after_sync();
        issue_st(0);
        ok = mbar_wait_bounded(smem_u32(&ctl->v_full), 0, wctx, 52, 1) &&
             mbar_wait_bounded(smem_u32(&ctl->do_full[0]), 0, wctx, 53, 0);
      }
      if (ok) {
        tc_fence_after_sync();
        issue_dpt(0);
      }
      for (int n = 0; n < n_iter && ok; ++n) {
        ok = mbar_wait_bounded(smem_u32(&ctl->p_full), n & 1, wctx, 54, n);
        if (!ok) break;
        tc_fence_after_sync();
        const uint64_t ddo = d_ring_mn + (n & 1) * kStage + kTile;
#pragma unroll
        for (int kk = 0; kk < kT / 16; ++kk)  // dV += P^T dO
          umma_bf16_ts(tmem_dv, tmem_st + tcol(kk), ddo + mnstep(kk), idesc_kmn, (n > 0 || kk > 0) ? 1u : 0u);
        umma_commit<1>(smem_u32(&ctl->do_empty[n & 1]));
        if (n + 1 < n_iter) {
          // S^T(n + 1) goes over P^T(n): the tensor core executes in issue order
          ok = mbar_wait_bounded(smem_u32(&ctl->qdo_full[(n + 1) & 1]), ((n + 1) >> 1) & 1, wctx, 53, n + 1);
          if (!ok) break;
          tc_fence_after_sync();
          issue_st(n + 1);
          ok = mbar_wait_bounded(smem_u32(&ctl->do_full[(n + 1) & 1]), ((n + 1) >> 1) & 1, wctx, 53, n + 1) &&
               mbar_wait_bounded(smem_u32(&ctl->dp_read), n & 1, wctx, 57, n);
          if (!ok) break;
          tc_fence_after_sync();
          issue_dpt(n + 1);
        }
        ok = mbar_wait_bounded(smem_u32(&ctl->ds_full), n & 1, wctx, 58, n);
        if (!ok) break;
        tc_fence_after_sync();
        const uint64_t dq = d_ring_mn + (n & 1) * kStage;
#pragma unroll
        for (int kk = 0; kk < kT / 16; ++kk)  // dK += dS^T Q
          umma_bf16<1>(tmem_dk, d_ds + kstep(kk), dq + mnstep(kk), idesc_kmn, (n > 0 || kk > 0) ? 1u : 0u);
        umma_commit<1>(smem_u32(&ctl->ds_empty));
        umma_commit<1>(smem_u32(&ctl->qdo_empty[n & 1]));
        if (n + 1 == n_iter) umma_commit<1>(smem_u32(&ctl->acc_full));
      }
    }
  } else {
    // Thread (row, part): KV row `row` of the tile, 32 query columns from part * 32.
    // One named barrier per iteration, reached by all threads whatever happened before.
    const int tid = threadIdx.x;
    const int row = tid & 127, part = tid >> 7;
    const int kv_pos = kv_row0 + row;
    const bool row_ok = kv_pos < p.seq_len;
    const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const uint32_t part_base = lane_base + part * kPartCols;
    const float c = p.scale * kLog2e;
    const uint32_t tmem_s = tmem_st + part_base, tmem_g = tmem_dpt + part_base;
    bool ok = true;
    // row statistics of the q tile of iteration n: part 0 fetches the log-sum-exp, part 1 delta
    auto stat_of = [&](int n) {
      const int h = hk * group + n / n_q, qp = (qt0 + n % n_q) * kT + row;
      if (qp >= p.seq_len) return 0.f;
      const long long at = (static_cast<long long>(b) * p.hq + h) * p.seq_len + qp;
      return part == 0 ? __fmul_rn(-p.lse[at], kLog2e) : -p.delta[at];
    };
    float next_stat = n_iter > 0 && part < 2 ? stat_of(0) : 0.f;
    for (int n = 0; n < n_iter; ++n) {
      const int qt = qt0 + n % n_q;
      const int buf = n & 1;
      if (part < 2) (part == 0 ? ctl->lse2[buf] : ctl->neg_delta[buf])[row] = next_stat;
      asm volatile("bar.sync 1, %0;" ::"n"(kSoftThreads) : "memory");
      if (n + 1 < n_iter && part < 2) next_stat = stat_of(n + 1);
      if (ctl->abort_flag) ok = false;
      if (ok) {
        const bool mine = mbar_wait_bounded(smem_u32(&ctl->st_full), n & 1, wctx, 55, n);
        ok = __all_sync(0xffffffffu, mine) != 0;
      }
      if (!ok) continue;
      tc_fence_after_sync();
      const int q0 = qt * kT + part * kPartCols;  // first query column of this thread
      const bool full = (!p.causal || qt > jt) && (qt + 1) * kT <= p.seq_len;   // uniform over the CTA
      // columns [first, end) of this part are allowed for this row
      const int first = p.causal ? kv_pos - q0 : 0, end = row_ok ? p.seq_len - q0 : 0;
      const float4* lse4 = reinterpret_cast<const float4*>(&ctl->lse2[buf][part * kPartCols]);
      const float4* dlt4 = reinterpret_cast<const float4*>(&ctl->neg_delta[buf][part * kPartCols]);
      uint32_t sv[32], w[16];
      __syncwarp();
      tmem_ld_32x32(tmem_s, sv);
      tmem_ld_wait_dep(sv);
      auto probs = [&](auto masked) {             // P, kept in fp32 for dS, packed for the product
#pragma unroll
        for (int i = 0; i < 32; i += 4) {
          const float4 l = lse4[i >> 2];
          float e[4];
          fma2(e[0], e[1], __uint_as_float(sv[i]), __uint_as_float(sv[i + 1]), c, c, l.x, l.y);
          fma2(e[2], e[3], __uint_as_float(sv[i + 2]), __uint_as_float(sv[i + 3]), c, c, l.z, l.w);
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            e[k] = ex2_approx(e[k]);
            if constexpr (decltype(masked)::value) e[k] = i + k >= first && i + k < end ? e[k] : 0.f;
            sv[i + k] = __float_as_uint(e[k]);
          }
          w[i >> 1] = pack_bf16(e[0], e[1]);
          w[(i >> 1) + 1] = pack_bf16(e[2], e[3]);
        }
      };
      if (full)
        probs(std::false_type{});
      else
        probs(std::true_type{});
      tmem_st_32x16(tmem_s, w);
      tmem_st_wait();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&ctl->p_full));
      bool mine = mbar_wait_bounded(smem_u32(&ctl->dp_full), n & 1, wctx, 55, n);
      ok = __all_sync(0xffffffffu, mine) != 0;
      if (!ok) continue;
      tc_fence_after_sync();
      uint32_t gv[32];
      __syncwarp();
      tmem_ld_32x32(tmem_g, gv);
      tmem_ld_wait_dep(gv);
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&ctl->dp_read));
      auto grads = [&](auto masked) {
#pragma unroll
        for (int i = 0; i < 32; i += 4) {
          const float4 d = dlt4[i >> 2];
          float t[4];
          add2(t[0], t[1], __uint_as_float(gv[i]), __uint_as_float(gv[i + 1]), d.x, d.y);
          add2(t[2], t[3], __uint_as_float(gv[i + 2]), __uint_as_float(gv[i + 3]), d.z, d.w);
          mul2(t[0], t[1], __uint_as_float(sv[i]), __uint_as_float(sv[i + 1]), t[0], t[1]);
          mul2(t[2], t[3], __uint_as_float(sv[i + 2]), __uint_as_float(sv[i + 3]), t[2], t[3]);
          mul2(t[0], t[1], t[0], t[1], p.scale, p.scale);
          mul2(t[2], t[3], t[2], t[3], p.scale, p.scale);
          if constexpr (decltype(masked)::value) {       // a masked column may hold anything: 0 * it need not be 0
#pragma unroll
            for (int k = 0; k < 4; ++k) t[k] = i + k >= first && i + k < end ? t[k] : 0.f;
          }
          w[i >> 1] = pack_bf16(t[0], t[1]);
          w[(i >> 1) + 1] = pack_bf16(t[2], t[3]);
        }
      };
      if (full)
        grads(std::false_type{});
      else
        grads(std::true_type{});
      if (n > 0) {           // the product of the previous dS^T has read the tile
        mine = mbar_wait_bounded(smem_u32(&ctl->ds_empty), (n - 1) & 1, wctx, 59, n);
        ok = __all_sync(0xffffffffu, mine) != 0;
        if (!ok) continue;
      }
      store_tile_row32(dst_ptr, row, part * kPartCols, w);
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&ctl->ds_full));
    }
    if (ok && n_iter > 0) {
      const bool mine = mbar_wait_bounded(smem_u32(&ctl->acc_full), 0, wctx, 56, 0);
      ok = __all_sync(0xffffffffu, mine) != 0;
    }
    if (ok) {
      tc_fence_after_sync();
      const long long tok = tok0 + kv_pos;
      const int col = hk * kD + part * kPartCols;
      uint32_t v[32];
      __syncwarp();
      tmem_ld_32x32(tmem_dv + part_base, v);
      tmem_ld_wait_dep(v);
      if (row_ok) store_row32(p.dv + tok * p.dv_stride + col, v);
      __syncwarp();
      tmem_ld_32x32(tmem_dk + part_base, v);
      tmem_ld_wait_dep(v);
      if (row_ok) store_row32(p.dk + tok * p.dk_stride + col, v);
    }
  }
  if (ctl->abort_flag) drain_in_flight();
  tc_fence_before_sync();
  __syncthreads();
  if (warp == kWarpMma) {
    __syncwarp();
    tc_fence_after_sync();
    tmem_dealloc<1>(tmem_base, 512);
  }
}

// Both in one launch: the first n_dkv CTAs do a dK / dV tile each, the others a dQ tile. The two need only
// delta from each other's direction, and a dK / dV CTA walks a whole group of query heads, so a call of few
// sequences or KV heads leaves most SMs idle until the last of them is done, and a call of many its last
// round: dQ tiles fill both. dQ + dK / dV apart, together (us, 32 / 8 heads): 8 x 512 133, 126; 4 x 1000, no mask,
// 310, 290; 1 x 700 82, 61; 2 x 4000 1043, 1037; 4 / 1 heads, 1 x 4000 325, 268.
__global__ void __launch_bounds__(kThreads, 1)
attention_bwd_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                     const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_do,
                     const __grid_constant__ BwdParams p, int n_dkv) {
  const int block = static_cast<int>(blockIdx.x);
  if (block < n_dkv)
    bwd_dkv(tm_q, tm_k, tm_v, tm_do, p, block);
  else
    bwd_dq(tm_q, tm_k, tm_v, tm_do, p, block - n_dkv);
}

}  // namespace
}  // namespace ka

// q, k, v, o, d_o: [B*L, heads*128] bf16 views (token strides in elements); lse: [B, Hq, L];
// delta: scratch [B, Hq, L] fp32; dq / dk / dv: outputs with their own token strides.
extern "C" int ka_attention_bwd(const void* q, long long q_stride, const void* k, long long k_stride, const void* v,
                                long long v_stride, const void* o, long long o_stride, const void* d_o,
                                long long do_stride, const float* lse, float* delta, void* dq, long long dq_stride,
                                void* dk, long long dk_stride, void* dv, long long dv_stride, int batch, int seq_len,
                                int hq, int hkv, int head_dim, float scale, int causal, int* status,
                                unsigned long long timeout_ns, void* stream) {
  using namespace ka;
  if (batch <= 0 || seq_len <= 0) return 0;
  if (head_dim != kD || hq % hkv != 0) return -1;
  // q, k, v and d_o are checked with their tensor maps; o is read by the delta kernel alone
  if ((reinterpret_cast<uintptr_t>(o) & 15u) != 0 || o_stride % 8 != 0) return -2;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  constexpr int kSmemDq = (4 + kKStages) * kTileBytes + 256;
  constexpr int kSmemDkv = 7 * kTileBytes + 2304;
  static_assert(sizeof(CtlDq) <= 256 && sizeof(CtlDkv) <= 2304 && kSmemDkv <= 227 * 1024, "shared memory layout");
  constexpr int kSmem = kSmemDkv > kSmemDq ? kSmemDkv : kSmemDq;
  static PerDevice once;
  if (!smem_opt_in(once, attention_bwd_kernel, kSmem)) return -10;
  const uint64_t tokens = static_cast<uint64_t>(batch) * seq_len;
  CUtensorMap tq, tk, tv, tdo;
  int rc = make_tmap_2d_16bit_sw128(&tq, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, q, tokens, static_cast<uint64_t>(hq) * kD,
                                    q_stride, kT, 64);
  if (rc) return -20 + rc;
  rc = make_tmap_2d_16bit_sw128(&tk, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, k, tokens, static_cast<uint64_t>(hkv) * kD,
                                k_stride, kT, 64);
  if (rc) return -40 + rc;
  rc = make_tmap_2d_16bit_sw128(&tv, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, v, tokens, static_cast<uint64_t>(hkv) * kD,
                                v_stride, kT, 64);
  if (rc) return -60 + rc;
  rc = make_tmap_2d_16bit_sw128(&tdo, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, d_o, tokens, static_cast<uint64_t>(hq) * kD,
                                do_stride, kT, 64);
  if (rc) return -80 + rc;
  const dim3 delta_grid(static_cast<unsigned>((seq_len + kDeltaTokens - 1) / kDeltaTokens) * batch,
                        static_cast<unsigned>(hq));
  attention_delta_kernel<<<delta_grid, 256, 0, st>>>(static_cast<const __nv_bfloat16*>(o), o_stride,
                                                     static_cast<const __nv_bfloat16*>(d_o), do_stride, delta, seq_len,
                                                     hq);
  BwdParams p = {};
  p.lse = lse;
  p.delta = delta;
  p.dq = static_cast<__nv_bfloat16*>(dq);
  p.dk = static_cast<__nv_bfloat16*>(dk);
  p.dv = static_cast<__nv_bfloat16*>(dv);
  p.dq_stride = dq_stride;
  p.dk_stride = dk_stride;
  p.dv_stride = dv_stride;
  p.batch = batch;
  p.seq_len = seq_len;
  p.hq = hq;
  p.hkv = hkv;
  p.scale = scale;
  p.causal = causal;
  p.status = status;
  p.timeout_ns = timeout_ns;
  const int n_t = (seq_len + kT - 1) / kT;
  const int n_dkv = batch * hkv * n_t;
  attention_bwd_kernel<<<static_cast<unsigned>(batch) * (hq + hkv) * n_t, kThreads, kSmem, st>>>(tq, tk, tv, tdo, p, n_dkv);
  return cudaGetLastError() == cudaSuccess ? 0 : -11;
}
