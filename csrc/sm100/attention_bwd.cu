// Attention backward for sm_100a (causal / full, GQA, head_dim 128), deterministic: no atomics.
//
//   delta[b, h, i] = sum_d dO[i, d] * O[i, d]
//   P  = exp(scale * Q K^T - lse),   dP = dO V^T,   dS = P * (dP - delta) * scale
//   dQ = dS K            bwd_dq: a dQ tile per (sequence, q head, q tile), made by one CTA that
//                        walks the KV tiles in increasing order; dQ accumulates in TMEM
//   dV = P^T dO, dK = dS^T Q   bwd_dkv: a dK / dV tile per (sequence, kv head, kv tile), made by one CTA
//                        that walks (q head of the group, q tile) in a fixed order; it
//                        works on S^T = K Q^T so that its threads own KV rows
// One kernel makes both kinds of tiles. With tiles enough a CTA per SM takes one after the other from a counter, with few of
// them each has a CTA of its own; a tile's result does not depend on it.
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
  int* next;            // [2]: the next dK / dV tile, the next dQ tile
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
                       long long do_stride, float* __restrict__ delta, int seq_len, int hq, int* __restrict__ next,
                       int ctas, int n_dkv) {
  // the tiles behind those that the CTAs of the next kernel start with
  if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x < 2)
    next[threadIdx.x] = threadIdx.x == 0 ? min(ctas, n_dkv) : max(ctas - n_dkv, 0);
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
// Both kinds of tiles overlap the tensor core with the element-wise work: the operands of the next
// iteration are in other stages of their rings, the next S and dP products are issued as soon as
// their TMEM columns have been read, and the 16-bit operand that comes out of S goes back to TMEM
// over the columns of S (the A operand of the product that follows), which leaves shared memory
// to the loaded tiles. Sixteen warps share a tile (eight issued in a quarter of the cycles: with two
// warps per scheduler nothing covers the TMEM loads and barriers), and tiles that need no mask
// run a loop of their own, without comparisons.
// One iteration is three products of 512 cycles (dQ) or four (dK / dV); with a single stage and
// everything in sequence it took about 9000 cycles. B = 2, L = 4000, 32 / 8 heads, causal, dQ and dK / dV as launches of their
// own: 891 and 1466 us with a single stage, 500 and 530 so, 902 for both in one launch with a ring for every operand; B = 8,
// L = 512: 114 and 173, 66 and 62, 115.
// ------------------------------------------------------------------------------------------------
// The loading thread takes the next tile of its kind and tells the others, a tile ahead of them.
struct Items {
  uint64_t full[2], empty[2];        // tile number written / read by the MMA thread and the element-wise warps
  int tile[2];                       // -1: there is none any more
};
__device__ __forceinline__ void init_items(Items& it) {
  for (int s = 0; s < 2; ++s) {
    mbar_init(smem_u32(&it.full[s]), 1);
    mbar_init(smem_u32(&it.empty[s]), kSoftThreads / 32 + 1);
  }
}
// The loading thread's side: false if a wait ran out. `first` is the first tile.
__device__ __forceinline__ bool give_item(Items& it, int i, int* next, int first, int n, int& tile, const WaitCtx& wctx, int where) {
  if (!mbar_wait_bounded(smem_u32(&it.empty[i & 1]), ((i >> 1) & 1) ^ 1u, wctx, where, i, 200u)) return false;
  tile = i == 0 ? first : atomicAdd(next, 1);
  if (tile >= n) tile = -1;
  *const_cast<volatile int*>(&it.tile[i & 1]) = tile;
  mbar_arrive(smem_u32(&it.full[i & 1]));
  return true;
}
// The others' side, by one thread or by a whole warp (lane 0 hands the slot back): -2 if the wait ran out.
template <bool kWarp>
__device__ __forceinline__ int take_item(Items& it, int i, const WaitCtx& wctx, int where) {
  bool ok = mbar_wait_bounded(smem_u32(&it.full[i & 1]), (i >> 1) & 1, wctx, where, i);
  if constexpr (kWarp) ok = __all_sync(0xffffffffu, ok) != 0;
  if (!ok) return -2;
  const int tile = *const_cast<volatile int*>(&it.tile[i & 1]);
  if constexpr (kWarp) __syncwarp();
  if (!kWarp || (threadIdx.x & 31) == 0) mbar_arrive(smem_u32(&it.empty[i & 1]));
  return tile;
}

struct CtlDq {
  uint64_t qdo_full, do_full;        // Q tile loaded, dO tile loaded
  uint64_t q_free, do_free;          // the tile's last S has read Q, its last dP dO
  uint64_t kv_full[3], kv_empty[3];  // K tiles: read by S and, an elementwise pass later, by dQ
  uint64_t v_full[2], v_empty[2];    // V tiles: read by dP alone
  uint64_t s_full[2];                // S ready in its TMEM buffer
  uint64_t dp_full, dp_read;         // dP ready / read into registers (count: softmax warps)
  // dS written over S (count: softmax warps), one per S buffer: S(j + 1) and dP(j + 1) are issued before
  // the wait for dS(j), so the warps may finish tile j + 1 before that wait looks. With a single barrier
  // they would have passed two phases by then, and the wait for a parity would never end.
  uint64_t ds_full[2];
  uint64_t acc_full;                 // final dQ ready
  Items items;
};

// ------------------------------------------------------------------------------------------------
// dQ tiles. TMEM: S (two buffers), dP, dQ. Shared memory: Q, dO, three stages of K, two of V.
// An SM gets about 85 GB/s, so a pair of tiles takes 1400 cycles and the latency on top. With two stages of (K, V)
// that were handed back together, behind dQ(j), the load of tile j + 2 and then S(j + 2) followed one another in the time in which the warps
// took tile j + 1, and an iteration was 3800 cycles; V is handed back by dP(j) now and K has a third stage: 2770
// cycles, all of them the issuing thread's: S 590, dP 660 and dQ 960 (512 each at the tensor core's rate) and 560 for its waits, 130
// to 200 for a barrier that is ready and 75 until the tensor core, whose queue has run empty, starts again.
// ------------------------------------------------------------------------------------------------
constexpr int kKStages = 3;
struct DqTile {
  int h, b, hk, qt, q_row0, tok0, n_kv;
};
__device__ __forceinline__ DqTile dq_tile(const BwdParams& p, int tile) {
  const int n_qt = (p.seq_len + kT - 1) / kT, n_bh = p.batch * p.hq;
  DqTile t;
  t.qt = n_qt - 1 - tile / n_bh;            // heavy (late) rows first
  const int bh = tile % n_bh;
  t.h = bh % p.hq;
  t.b = bh / p.hq;
  t.hk = t.h / (p.hq / p.hkv);
  t.q_row0 = t.qt * kT;
  t.tok0 = t.b * p.seq_len;
  const int kv_end = p.causal ? min(p.seq_len, t.q_row0 + kT) : p.seq_len;
  t.n_kv = (kv_end + kT - 1) / kT;
  return t;
}

// All counters (jj: kv tiles so far, i: tiles so far) run on across tiles, so the loads and the first S and dP of the next
// tile overlap the end of this one.
template <bool kOnce>
__device__ __forceinline__ void
bwd_dq(const CUtensorMap& tm_q, const CUtensorMap& tm_k, const CUtensorMap& tm_v, const CUtensorMap& tm_do,
       const BwdParams& p, int n_tiles, int first, CtlDq* ctl, const WaitCtx& wctx, uint32_t tmem_base) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const uint32_t base = smem_u32(smem_raw);
  const uint32_t q_tile = base, do_tile = base + kTileBytes, k_ring = base + 2 * kTileBytes,
                 v_ring = base + (2 + kKStages) * kTileBytes;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t tmem_dp = tmem_base + 256, tmem_dq = tmem_base + 384;   // S: tmem_base + 128 * buffer

  if (warp == kWarpTma) {
    if (lane == 0) {
      auto load = [&](uint32_t dst, const CUtensorMap& tm, int col, int row, uint64_t* bar) {
        const uint32_t full = smem_u32(bar);
        mbar_arrive_expect_tx(full, kTileBytes);
        tma_load_2d(dst, &tm, col, row, full);
        tma_load_2d(dst + 16384, &tm, col + 64, row, full);
      };
      int ks = 0, jj = 0;
      uint32_t kphase = 1;
      auto load_k = [&](const DqTile& t, int j) {
        if (!mbar_wait_bounded(smem_u32(&ctl->kv_empty[ks]), kphase, wctx, 41, j)) return false;
        load(k_ring + ks * kTileBytes, tm_k, t.hk * kD, t.tok0 + j * kT, &ctl->kv_full[ks]);
        if (++ks == kKStages) {
          ks = 0;
          kphase ^= 1u;
        }
        return true;
      };
      int tile = first;
      for (int i = 0; kOnce ? i == 0 : give_item(ctl->items, i, p.next + 1, first, n_tiles, tile, wctx, 40) && tile >= 0; ++i) {
        const DqTile t = dq_tile(p, tile);
        const uint32_t free_phase = (i & 1) ^ 1u;
        bool ok = kOnce || mbar_wait_bounded(smem_u32(&ctl->q_free), free_phase, wctx, 49, i, 200u);
        if (!ok) break;
        load(q_tile, tm_q, t.h * kD, t.tok0 + t.q_row0, &ctl->qdo_full);
        ok = load_k(t, 0) && (kOnce || mbar_wait_bounded(smem_u32(&ctl->do_free), free_phase, wctx, 49, i));
        if (!ok) break;
        load(do_tile, tm_do, t.h * kD, t.tok0 + t.q_row0, &ctl->do_full);
        // V(j), then K(j + 1): the products that hand the stages back come in that order
        for (int j = 0; j < t.n_kv && ok; ++j, ++jj) {
          ok = mbar_wait_bounded(smem_u32(&ctl->v_empty[jj & 1]), ((jj >> 1) & 1) ^ 1u, wctx, 41, j);
          if (!ok) break;
          load(v_ring + (jj & 1) * kTileBytes, tm_v, t.hk * kD, t.tok0 + j * kT, &ctl->v_full[jj & 1]);
          if (j + 1 < t.n_kv) ok = load_k(t, j + 1);
        }
        if (!ok) break;
      }
    }
  } else if (warp == kWarpMma) {
    if (lane == 0) {
      const uint32_t idesc_kk = umma_idesc_bf16_f32(kT, kT);             // both operands K-major
      const uint32_t idesc_kmn = umma_idesc_bf16_f32(kT, kD) | (1u << 16);  // B MN-major
      const uint64_t d_q = desc_kmajor(q_tile, 0), d_do = desc_kmajor(do_tile, 0), d_k = desc_kmajor(k_ring, 0),
                     d_k_mn = desc_mnmajor(k_ring, 0), d_v = desc_kmajor(v_ring, 0);
      constexpr uint64_t kTile = kTileBytes >> 4;
      int ks_s = 0, ks_q = 0;          // stages of K for the next S and the next dQ
      uint32_t kphase = 0;
      auto issue_s = [&](int g) {      // S = Q K^T of kv tile number g
#pragma unroll
        for (int kk = 0; kk < kD / 16; ++kk)
          umma_bf16<1>(tmem_base + (g & 1) * 128, d_q + kstep(kk), d_k + ks_s * kTile + kstep(kk), idesc_kk, kk > 0 ? 1u : 0u);
        umma_commit<1>(smem_u32(&ctl->s_full[g & 1]));
        if (++ks_s == kKStages) {
          ks_s = 0;
          kphase ^= 1u;
        }
      };
      auto issue_dp = [&](int g) {     // dP = dO V^T
        const uint64_t dv = d_v + (g & 1) * kTile;
#pragma unroll
        for (int kk = 0; kk < kD / 16; ++kk)
          umma_bf16<1>(tmem_dp, d_do + kstep(kk), dv + kstep(kk), idesc_kk, kk > 0 ? 1u : 0u);
        umma_commit<1>(smem_u32(&ctl->dp_full));
        umma_commit<1>(smem_u32(&ctl->v_empty[g & 1]));
      };
      bool ok = true;
      int jj = 0;                      // kv tiles so far: number of this tile's first
      for (int i = 0; ok; ++i) {
        const int tile = kOnce ? (i == 0 ? first : -1) : take_item<false>(ctl->items, i, wctx, 40);
        if (tile < 0) break;
        const int n_kv = dq_tile(p, tile).n_kv;
        // S(0) goes over dS of two kv tiles ago and dP(0) over what the warps have read, since dS of the last kv tile
        // has been waited for; the tensor core executes in issue order
        ok = mbar_wait_bounded(smem_u32(&ctl->qdo_full), i & 1, wctx, 42, i) &&
             mbar_wait_bounded(smem_u32(&ctl->kv_full[ks_s]), kphase, wctx, 43, 0);
        if (!ok) break;
        tc_fence_after_sync();
        issue_s(jj);
        if (!kOnce && n_kv == 1) umma_commit<1>(smem_u32(&ctl->q_free));
        ok = mbar_wait_bounded(smem_u32(&ctl->do_full), i & 1, wctx, 42, i) &&
             mbar_wait_bounded(smem_u32(&ctl->v_full[jj & 1]), (jj >> 1) & 1, wctx, 43, 0);
        if (!ok) break;
        tc_fence_after_sync();
        issue_dp(jj);
        if (!kOnce && n_kv == 1) umma_commit<1>(smem_u32(&ctl->do_free));
        for (int j = 0; j < n_kv; ++j) {
          const int g = jj + j;
          if (j + 1 < n_kv) {
            // S(j + 1) goes over dS(j - 1), whose product was issued an iteration ago
            ok = mbar_wait_bounded(smem_u32(&ctl->kv_full[ks_s]), kphase, wctx, 43, j + 1);
            if (!ok) break;
            tc_fence_after_sync();
            issue_s(g + 1);
            if (!kOnce && j + 2 == n_kv) umma_commit<1>(smem_u32(&ctl->q_free));
            ok = mbar_wait_bounded(smem_u32(&ctl->v_full[(g + 1) & 1]), ((g + 1) >> 1) & 1, wctx, 43, j + 1) &&
                 mbar_wait_bounded(smem_u32(&ctl->dp_read), g & 1, wctx, 47, j);
            if (!ok) break;
            tc_fence_after_sync();
            issue_dp(g + 1);
            if (!kOnce && j + 2 == n_kv) umma_commit<1>(smem_u32(&ctl->do_free));
          }
          ok = mbar_wait_bounded(smem_u32(&ctl->ds_full[g & 1]), (g >> 1) & 1, wctx, 44, j);
          if (!ok) break;
          tc_fence_after_sync();
          const uint64_t dk = d_k_mn + ks_q * kTile;
#pragma unroll
          for (int kk = 0; kk < kT / 16; ++kk)  // dQ += dS K
            umma_bf16_ts(tmem_dq, tmem_base + (g & 1) * 128 + tcol(kk), dk + mnstep(kk), idesc_kmn,
                         (j > 0 || kk > 0) ? 1u : 0u);
          umma_commit<1>(smem_u32(&ctl->kv_empty[ks_q]));
          if (j + 1 == n_kv) umma_commit<1>(smem_u32(&ctl->acc_full));
          ks_q = ks_q + 1 == kKStages ? 0 : ks_q + 1;
        }
        jj += n_kv;
      }
    }
  } else {
    const int tid = threadIdx.x;
    const int row = tid & 127, part = tid >> 7;
    const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const uint32_t part_base = lane_base + part * kPartCols;
    const float c = p.scale * kLog2e;
    bool ok = true;
    int g = 0;                         // kv tiles so far
    for (int i = 0; ok; ++i) {
      const int tile = kOnce ? (i == 0 ? first : -1) : take_item<true>(ctl->items, i, wctx, 40);
      if (tile < 0) break;
      const DqTile t = dq_tile(p, tile);
      const int q_pos = t.q_row0 + row;
      const bool row_ok = q_pos < p.seq_len;
      const long long stat = (static_cast<long long>(t.b) * p.hq + t.h) * p.seq_len + q_pos;
      const float neg_lse2 = row_ok ? __fmul_rn(-p.lse[stat], kLog2e) : 0.f;
      const float neg_dlt = row_ok ? -p.delta[stat] : 0.f;
      for (int j = 0; j < t.n_kv && ok; ++j, ++g) {
        bool mine = mbar_wait_bounded(smem_u32(&ctl->s_full[g & 1]), (g >> 1) & 1, wctx, 45, j);
        ok = __all_sync(0xffffffffu, mine) != 0;
        if (!ok) break;
        tc_fence_after_sync();
        const uint32_t tmem_s = tmem_base + static_cast<uint32_t>((g & 1) * 128) + part_base;
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
        mine = mbar_wait_bounded(smem_u32(&ctl->dp_full), g & 1, wctx, 45, j);
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
        if (p.causal ? j < t.qt : (j + 1) * kT <= p.seq_len)       // uniform over the CTA
          grads(std::false_type{}, 0);
        else
          grads(std::true_type{},
                row_ok ? (p.causal ? q_pos : p.seq_len - 1) - (j * kT + part * kPartCols) : -1);
        tmem_st_32x16(tmem_s, w);
        tmem_st_wait();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&ctl->ds_full[g & 1]));
      }
      if (ok) {
        const bool mine = mbar_wait_bounded(smem_u32(&ctl->acc_full), i & 1, wctx, 46, i);
        ok = __all_sync(0xffffffffu, mine) != 0;
      }
      if (ok) {
        tc_fence_after_sync();
        __nv_bfloat16* dst = p.dq + static_cast<long long>(t.tok0 + q_pos) * p.dq_stride + t.h * kD + part * kPartCols;
        uint32_t v[32];
        __syncwarp();
        tmem_ld_32x32(tmem_dq + part_base, v);
        tmem_ld_wait_dep(v);
        if (row_ok) store_row32(dst, v);
        tc_fence_before_sync();        // dQ of the next tile is written behind this warp's next arrival
        __syncwarp();
      }
    }
  }
}

// ------------------------------------------------------------------------------------------------
// dK / dV tiles. TMEM: S^T (then P^T as bf16 over it), dP^T, dV, dK. Shared memory: K, V, two
// stages of (Q, dO), dS^T.
// ------------------------------------------------------------------------------------------------
// Does the condition hold for any element-wise thread? A barrier of all of them.
__device__ __forceinline__ bool soft_any(bool cond) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbarrier.cta.red.or.pred q, 1, %2, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(r)
      : "r"(cond ? 1u : 0u), "n"(kSoftThreads)
      : "memory");
  return r != 0;
}

struct CtlDkv {
  uint64_t kv_full, v_full;          // K tile loaded, V tile loaded
  uint64_t k_free, v_free;           // the tile's last S^T has read K, its last dP^T V
  uint64_t qdo_full[2], qdo_empty[2];  // Q tiles: read by S^T and, last of all, by dK
  uint64_t do_full[2], do_empty[2];    // dO tiles: read by dP^T and dV
  uint64_t st_full;                  // S^T ready in TMEM
  uint64_t p_full;                   // P^T written over S^T (count: softmax warps)
  uint64_t dp_full, dp_read;         // dP^T ready / read into registers (count: softmax warps)
  uint64_t ds_full, ds_empty;        // dS^T tile written (count: softmax warps) / consumed
  uint64_t acc_full;
  Items items;
  alignas(16) float lse2[2][kT];     // -lse * log2(e) of the current q tile, double-buffered by iteration
  alignas(16) float neg_delta[2][kT];
};

struct DkvTile {
  int hk, b, jt, kv_row0, tok0, qt0, n_q, n_iter;
};
__device__ __forceinline__ DkvTile dkv_tile(const BwdParams& p, int tile) {
  const int n_t = (p.seq_len + kT - 1) / kT;
  // All early (causal: heavy) kv tiles first: the last to start are the lightest
  // (sequence by sequence the last heavy ones started when the rest was done: 1074 against 833 us).
  const int n_bh = p.batch * p.hkv;
  DkvTile t;
  t.jt = tile / n_bh;
  const int bh = tile % n_bh;
  t.hk = bh % p.hkv;
  t.b = bh / p.hkv;
  t.kv_row0 = t.jt * kT;
  t.tok0 = t.b * p.seq_len;
  t.qt0 = p.causal ? t.jt : 0;
  t.n_q = n_t - t.qt0;                                         // q tiles per head, at least one
  t.n_iter = p.hq / p.hkv * t.n_q;
  return t;
}

// All counters (nn / g: q tiles so far, i: tiles so far) run on across tiles. The loading thread returns the first dQ tile of
// this CTA, which it takes when the last S^T here is done: not before, a CTA with less to do might have it, and not
// behind the end, which would wait for the answer.
template <bool kOnce>
__device__ __forceinline__ int
bwd_dkv(const CUtensorMap& tm_q, const CUtensorMap& tm_k, const CUtensorMap& tm_v, const CUtensorMap& tm_do,
        const BwdParams& p, int n_tiles, int block, CtlDkv* ctl, const WaitCtx& wctx, uint32_t tmem_base) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const uint32_t base = smem_u32(smem_raw);
  const uint32_t k_tile = base, v_tile = base + kTileBytes, ring = base + 2 * kTileBytes,   // stage: Q, dO
                 dst_tile = base + 6 * kTileBytes;
  uint8_t* dst_ptr = smem_raw + 6 * kTileBytes;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int group = p.hq / p.hkv;
  const uint32_t tmem_st = tmem_base, tmem_dpt = tmem_base + 128, tmem_dv = tmem_base + 256, tmem_dk = tmem_base + 384;

  if (warp == kWarpTma) {
    if (lane == 0) {
      auto load = [&](uint32_t dst, const CUtensorMap& tm, int col, int row, uint64_t* bar) {
        const uint32_t full = smem_u32(bar);
        mbar_arrive_expect_tx(full, kTileBytes);
        tma_load_2d(dst, &tm, col, row, full);
        tma_load_2d(dst + 16384, &tm, col + 64, row, full);
      };
      int nn = 0;                      // q tiles so far: number of this tile's first
      auto load_q = [&](const DkvTile& t, int n) {
        const int h = t.hk * group + n / t.n_q, qt = t.qt0 + n % t.n_q, s = (nn + n) & 1;
        if (!mbar_wait_bounded(smem_u32(&ctl->qdo_empty[s]), (((nn + n) >> 1) & 1) ^ 1u, wctx, 51, n)) return false;
        load(ring + s * 2 * kTileBytes, tm_q, h * kD, t.tok0 + qt * kT, &ctl->qdo_full[s]);
        return true;
      };
      auto load_do = [&](const DkvTile& t, int n) {
        const int h = t.hk * group + n / t.n_q, qt = t.qt0 + n % t.n_q, s = (nn + n) & 1;
        if (!mbar_wait_bounded(smem_u32(&ctl->do_empty[s]), (((nn + n) >> 1) & 1) ^ 1u, wctx, 51, n)) return false;
        load(ring + (s * 2 + 1) * kTileBytes, tm_do, h * kD, t.tok0 + qt * kT, &ctl->do_full[s]);
        return true;
      };
      int tile = block, i = 0;
      for (; kOnce ? i == 0 : give_item(ctl->items, i, p.next, block, n_tiles, tile, wctx, 50) && tile >= 0; ++i) {
        const DkvTile t = dkv_tile(p, tile);
        const uint32_t free_phase = (i & 1) ^ 1u;
        bool ok = kOnce || mbar_wait_bounded(smem_u32(&ctl->k_free), free_phase, wctx, 61, i, 200u);
        if (!ok) break;
        load(k_tile, tm_k, t.hk * kD, t.tok0 + t.kv_row0, &ctl->kv_full);
        ok = load_q(t, 0) && (kOnce || mbar_wait_bounded(smem_u32(&ctl->v_free), free_phase, wctx, 61, i));
        if (!ok) break;
        load(v_tile, tm_v, t.hk * kD, t.tok0 + t.kv_row0, &ctl->v_full);
        ok = load_do(t, 0);
        // dO(n - 2) is handed back by dV(n - 2), Q(n - 2) by dK(n - 2)
        for (int n = 1; n < t.n_iter && ok; ++n) ok = load_do(t, n) && load_q(t, n);
        if (!ok) break;
        nn += t.n_iter;
      }
      if (kOnce) return 0;
      if (i == 0) return block - n_tiles;
      if (mbar_wait_bounded(smem_u32(&ctl->k_free), (i - 1) & 1, wctx, 62, i, 500u)) return atomicAdd(p.next + 1, 1);
    }
  } else if (warp == kWarpMma) {
    if (lane == 0) {
      const uint32_t idesc_kk = umma_idesc_bf16_f32(kT, kT);
      const uint32_t idesc_kmn = umma_idesc_bf16_f32(kT, kD) | (1u << 16);
      const uint64_t d_k = desc_kmajor(k_tile, 0), d_v = desc_kmajor(v_tile, 0), d_ring = desc_kmajor(ring, 0),
                     d_ring_mn = desc_mnmajor(ring, 0), d_ds = desc_kmajor(dst_tile, 0);
      constexpr uint64_t kStage = (2 * kTileBytes) >> 4, kTile = kTileBytes >> 4;
      auto issue_st = [&](int g) {     // S^T = K Q^T of q tile number g
        const uint64_t dq = d_ring + (g & 1) * kStage;
#pragma unroll
        for (int kk = 0; kk < kD / 16; ++kk)
          umma_bf16<1>(tmem_st, d_k + kstep(kk), dq + kstep(kk), idesc_kk, kk > 0 ? 1u : 0u);
        umma_commit<1>(smem_u32(&ctl->st_full));
      };
      auto issue_dpt = [&](int g) {    // dP^T = V dO^T
        const uint64_t ddo = d_ring + (g & 1) * kStage + kTile;
#pragma unroll
        for (int kk = 0; kk < kD / 16; ++kk)
          umma_bf16<1>(tmem_dpt, d_v + kstep(kk), ddo + kstep(kk), idesc_kk, kk > 0 ? 1u : 0u);
        umma_commit<1>(smem_u32(&ctl->dp_full));
      };
      bool ok = true;
      int nn = 0;
      for (int i = 0; ok; ++i) {
        const int tile = kOnce ? (i == 0 ? block : -1) : take_item<false>(ctl->items, i, wctx, 50);
        if (tile < 0) break;
        const int n_iter = dkv_tile(p, tile).n_iter;
        // S^T(0) goes over the last tile's P^T and dP^T(0) over its dP^T, which the warps have read, since its dS^T
        // has been waited for; the tensor core executes in issue order
        ok = mbar_wait_bounded(smem_u32(&ctl->kv_full), i & 1, wctx, 52, i) &&
             mbar_wait_bounded(smem_u32(&ctl->qdo_full[nn & 1]), (nn >> 1) & 1, wctx, 53, 0);
        if (!ok) break;
        tc_fence_after_sync();
        issue_st(nn);
        if (!kOnce && n_iter == 1) umma_commit<1>(smem_u32(&ctl->k_free));
        ok = mbar_wait_bounded(smem_u32(&ctl->v_full), i & 1, wctx, 52, i) &&
             mbar_wait_bounded(smem_u32(&ctl->do_full[nn & 1]), (nn >> 1) & 1, wctx, 53, 0);
        if (!ok) break;
        tc_fence_after_sync();
        issue_dpt(nn);
        if (!kOnce && n_iter == 1) umma_commit<1>(smem_u32(&ctl->v_free));
        for (int n = 0; n < n_iter; ++n) {
          const int g = nn + n;
          ok = mbar_wait_bounded(smem_u32(&ctl->p_full), g & 1, wctx, 54, n);
          if (!ok) break;
          tc_fence_after_sync();
          const uint64_t ddo = d_ring_mn + (g & 1) * kStage + kTile;
#pragma unroll
          for (int kk = 0; kk < kT / 16; ++kk)  // dV += P^T dO
            umma_bf16_ts(tmem_dv, tmem_st + tcol(kk), ddo + mnstep(kk), idesc_kmn, (n > 0 || kk > 0) ? 1u : 0u);
          umma_commit<1>(smem_u32(&ctl->do_empty[g & 1]));
          if (n + 1 < n_iter) {
            // S^T(n + 1) goes over P^T(n): the tensor core executes in issue order
            ok = mbar_wait_bounded(smem_u32(&ctl->qdo_full[(g + 1) & 1]), ((g + 1) >> 1) & 1, wctx, 53, n + 1);
            if (!ok) break;
            tc_fence_after_sync();
            issue_st(g + 1);
            if (!kOnce && n + 2 == n_iter) umma_commit<1>(smem_u32(&ctl->k_free));
            ok = mbar_wait_bounded(smem_u32(&ctl->do_full[(g + 1) & 1]), ((g + 1) >> 1) & 1, wctx, 53, n + 1) &&
                 mbar_wait_bounded(smem_u32(&ctl->dp_read), g & 1, wctx, 57, n);
            if (!ok) break;
            tc_fence_after_sync();
            issue_dpt(g + 1);
            if (!kOnce && n + 2 == n_iter) umma_commit<1>(smem_u32(&ctl->v_free));
          }
          ok = mbar_wait_bounded(smem_u32(&ctl->ds_full), g & 1, wctx, 58, n);
          if (!ok) break;
          tc_fence_after_sync();
          const uint64_t dq = d_ring_mn + (g & 1) * kStage;
#pragma unroll
          for (int kk = 0; kk < kT / 16; ++kk)  // dK += dS^T Q
            umma_bf16<1>(tmem_dk, d_ds + kstep(kk), dq + mnstep(kk), idesc_kmn, (n > 0 || kk > 0) ? 1u : 0u);
          umma_commit<1>(smem_u32(&ctl->ds_empty));
          umma_commit<1>(smem_u32(&ctl->qdo_empty[g & 1]));
          if (n + 1 == n_iter) umma_commit<1>(smem_u32(&ctl->acc_full));
        }
        nn += n_iter;
      }
    }
  } else {
    // Thread (row, part): KV row `row` of the tile, 32 query columns from part * 32.
    // One named barrier per iteration, reached by all threads whatever happened before; whether there is another tile
    // is one decision of all of them.
    const int tid = threadIdx.x;
    const int row = tid & 127, part = tid >> 7;
    const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const uint32_t part_base = lane_base + part * kPartCols;
    const float c = p.scale * kLog2e;
    const uint32_t tmem_s = tmem_st + part_base, tmem_g = tmem_dpt + part_base;
    bool ok = true;
    int g = 0;                         // q tiles so far
    for (int i = 0;; ++i) {
      const int tile = kOnce ? block : take_item<true>(ctl->items, i, wctx, 50);
      if (kOnce ? i > 0 : soft_any(tile < 0 || !ok)) break;
      // few values live through the loop: the others are worked out again behind it
      const int jt = tile / (p.batch * p.hkv), qt0 = p.causal ? jt : 0, n_t = (p.seq_len + kT - 1) / kT;
      const int kv_pos = jt * kT + row;
      const bool row_ok = kv_pos < p.seq_len;
      // row statistics of the next q tile: part 0 fetches the log-sum-exp, part 1 delta
      const float* stat_head = (part == 0 ? p.lse : p.delta) + row;
      {
        const DkvTile t = dkv_tile(p, tile);
        stat_head += (static_cast<long long>(t.b) * p.hq + t.hk * group) * p.seq_len;
      }
      auto stat_of = [&](int qt) {
        return qt * kT + row < p.seq_len ? __fmul_rn(stat_head[qt * kT], part == 0 ? -kLog2e : -1.f) : 0.f;
      };
      float next_stat = part < 2 ? stat_of(qt0) : 0.f;
      int next_qt = qt0;               // the q tile whose statistics are in next_stat, of the head at stat_head
      for (int left = group * (n_t - qt0); left > 0; --left, ++g) {
        const int qt = next_qt;
        if (++next_qt == n_t) {
          next_qt = qt0;
          stat_head += p.seq_len;
        }
        const int buf = g & 1;
        if (part < 2) (part == 0 ? ctl->lse2[buf] : ctl->neg_delta[buf])[row] = next_stat;
        asm volatile("bar.sync 1, %0;" ::"n"(kSoftThreads) : "memory");
        if (left > 1 && part < 2) next_stat = stat_of(next_qt);
        if (*wctx.abort_flag) ok = false;
        if (ok) {
          const bool mine = mbar_wait_bounded(smem_u32(&ctl->st_full), g & 1, wctx, 55, g);
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
        bool mine = mbar_wait_bounded(smem_u32(&ctl->dp_full), g & 1, wctx, 55, g);
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
        if (g > 0) {           // the product of the previous dS^T has read the tile
          mine = mbar_wait_bounded(smem_u32(&ctl->ds_empty), (g - 1) & 1, wctx, 59, g);
          ok = __all_sync(0xffffffffu, mine) != 0;
          if (!ok) continue;
        }
        store_tile_row32(dst_ptr, row, part * kPartCols, w);
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&ctl->ds_full));
      }
      if (ok) {
        const bool mine = mbar_wait_bounded(smem_u32(&ctl->acc_full), i & 1, wctx, 56, i);
        ok = __all_sync(0xffffffffu, mine) != 0;
      }
      if (ok) {
        tc_fence_after_sync();
        const DkvTile t = dkv_tile(p, tile);
        const long long tok = t.tok0 + kv_pos;
        const int col = t.hk * kD + part * kPartCols;
        uint32_t v[32];
        __syncwarp();
        tmem_ld_32x32(tmem_dv + part_base, v);
        tmem_ld_wait_dep(v);
        if (row_ok) store_row32(p.dv + tok * p.dv_stride + col, v);
        __syncwarp();
        tmem_ld_32x32(tmem_dk + part_base, v);
        tmem_ld_wait_dep(v);
        if (row_ok) store_row32(p.dk + tok * p.dk_stride + col, v);
        tc_fence_before_sync();        // dV and dK of the next tile are written behind this warp's next arrivals
        __syncwarp();
      }
    }
  }
  return 0;
}

struct Ctl {
  CtlDkv dkv;
  CtlDq dq;
  uint32_t tmem_base;
  int abort_flag;
};
constexpr int kSmemBwd = 7 * kTileBytes + static_cast<int>(sizeof(Ctl));
static_assert(4 + kKStages == 7 && kSmemBwd <= 227 * 1024, "shared memory layout");

// One CTA per SM, which takes dK / dV tiles until there are none and then dQ tiles: the two need only
// delta from each other's direction. A dK / dV tile walks a whole group of query heads, so a call of few
// sequences or KV heads leaves most SMs idle until the last of them is done, and a call of many its last
// round: dQ tiles fill both. As CTAs of their own the tiles cost 7 us each on top of their iterations (start, TMEM, first
// loads, last product and stores, all in sequence), half of the time of short
// sequences: 8 x 512, 32 / 8 heads 131 us, 115 as one walk, in which the next tile's loads and first products overlap the end of this one.
template <bool kOnce>
__global__ void __launch_bounds__(kThreads, 1)
attention_bwd_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                     const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_do,
                     const __grid_constant__ BwdParams p, int n_dkv, int n_dq) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  Ctl* ctl = reinterpret_cast<Ctl*>(smem_raw + 7 * kTileBytes);
  const int warp = threadIdx.x >> 5;
  const WaitCtx wctx{&ctl->abort_flag, p.status, p.timeout_ns};
  if (threadIdx.x == 0) {
    auto init = [](uint64_t* bar, int n, int count) {
      for (int i = 0; i < n; ++i) mbar_init(smem_u32(bar + i), count);
    };
    constexpr int kWarps = kSoftThreads / 32;
    CtlDkv& a = ctl->dkv;
    init(&a.kv_full, 1, 1);
    init(&a.v_full, 1, 1);
    init(&a.k_free, 1, 1);
    init(&a.v_free, 1, 1);
    init(a.qdo_full, 2, 1);
    init(a.qdo_empty, 2, 1);
    init(a.do_full, 2, 1);
    init(a.do_empty, 2, 1);
    init(&a.st_full, 1, 1);
    init(&a.p_full, 1, kWarps);
    init(&a.dp_full, 1, 1);
    init(&a.dp_read, 1, kWarps);
    init(&a.ds_full, 1, kWarps);
    init(&a.ds_empty, 1, 1);
    init(&a.acc_full, 1, 1);
    init_items(a.items);
    CtlDq& b = ctl->dq;
    init(&b.qdo_full, 1, 1);
    init(&b.do_full, 1, 1);
    init(&b.q_free, 1, 1);
    init(&b.do_free, 1, 1);
    init(b.kv_full, kKStages, 1);
    init(b.kv_empty, kKStages, 1);
    init(b.v_full, 2, 1);
    init(b.v_empty, 2, 1);
    init(b.s_full, 2, 1);
    init(b.ds_full, 2, kWarps);
    init(&b.dp_full, 1, 1);
    init(&b.dp_read, 1, kWarps);
    init(&b.acc_full, 1, 1);
    init_items(b.items);
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
  const int block = static_cast<int>(blockIdx.x);
  if constexpr (kOnce) {
    if (block < n_dkv)
      bwd_dkv<true>(tm_q, tm_k, tm_v, tm_do, p, n_dkv, block, &ctl->dkv, wctx, tmem_base);
    else
      bwd_dq<true>(tm_q, tm_k, tm_v, tm_do, p, n_dq, block - n_dkv, &ctl->dq, wctx, tmem_base);
  } else {
    const int first = bwd_dkv<false>(tm_q, tm_k, tm_v, tm_do, p, n_dkv, block, &ctl->dkv, wctx, tmem_base);
    // the dQ tiles use the same shared memory and TMEM: every product and store of the others is done
    if (ctl->abort_flag) drain_in_flight();
    fence_proxy_async_smem();
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    if (ctl->abort_flag == 0) bwd_dq<false>(tm_q, tm_k, tm_v, tm_do, p, n_dq, first, &ctl->dq, wctx, tmem_base);
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

}  // namespace
}  // namespace ka

// q, k, v, o, d_o: [B*L, heads*128] bf16 views (token strides in elements); lse: [B, Hq, L];
// delta: scratch of B * Hq * L + 2 floats; dq / dk / dv: outputs with their own token strides.
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
  static PerDevice once;
  static PerDevice once_each;
  if (!smem_opt_in(once, attention_bwd_kernel<false>, kSmemBwd) || !smem_opt_in(once_each, attention_bwd_kernel<true>, kSmemBwd))
    return -10;
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
  const int n_t = (seq_len + kT - 1) / kT;
  const int n_dkv = batch * hkv * n_t, n_dq = batch * hq * n_t;
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  // A CTA per tile while the longest dK / dV tile (a group of heads, n_t q tiles each) takes longer than all work shared by the
  // SMs: its iterations then count, and they take 4 % less in the kernel without the walk. Pairs of tiles: 2.1 us in dK / dV,
  // 1.45 in dQ. us, walk / CTA per tile: 1 x 700, 32 / 8 heads 73.8 / 69.0; 1 x 1500 116 / 112; 1 x 4000, 4 / 1 heads 284 / 269;
  // 3 x 700, 32 / 8 heads 80 / 88; 8 x 512 115 / 131; 2 x 2048, 16 / 16 heads 152 / 167; 2 x 4000, 32 / 8 heads 902 / 928.
  const long long pairs = static_cast<long long>(batch) * hq * (causal ? n_t * (n_t + 1ll) / 2 : static_cast<long long>(n_t) * n_t);
  const bool each = 2 * pairs < static_cast<long long>(hq / hkv) * n_t * sms;
  const int ctas = each ? n_dkv + n_dq : sms;
  int* next = reinterpret_cast<int*>(delta + static_cast<size_t>(batch) * hq * seq_len);
  const dim3 delta_grid(static_cast<unsigned>((seq_len + kDeltaTokens - 1) / kDeltaTokens) * batch,
                        static_cast<unsigned>(hq));
  attention_delta_kernel<<<delta_grid, 256, 0, st>>>(static_cast<const __nv_bfloat16*>(o), o_stride,
                                                     static_cast<const __nv_bfloat16*>(d_o), do_stride, delta, seq_len,
                                                     hq, next, ctas, n_dkv);
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
  p.next = next;
  p.status = status;
  p.timeout_ns = timeout_ns;
  auto* kernel = each ? attention_bwd_kernel<true> : attention_bwd_kernel<false>;
  kernel<<<static_cast<unsigned>(ctas), kThreads, kSmemBwd, st>>>(tq, tk, tv, tdo, p, n_dkv, n_dq);
  return cudaGetLastError() == cudaSuccess ? 0 : -11;
}
