// Batch-invariant bf16 GEMM for sm_100a: persistent CTA pairs, TMA operand ring,
// tcgen05.mma (cta_group::2, M=256 N=256 K=16) into double-buffered TMEM accumulators, and an
// epilogue that either stores the tile or emits fp32 K-slice partials for the tensor-parallel
// reduce-scatter (see gemm.h). Operands may be K-major or MN-major (the latter serves the
// backward GEMMs without transposes).
//
// The reference has no GEMM of its own; its registry only names backends
// (rl_engine/kernels/registry.py:20-30).
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cuda_bf16.h>

#include "common/bounded_wait.cuh"
#include "common/launch.cuh"
#include "common/ptx.cuh"
#include "common/tmap.cuh"
#include "gemm.h"

namespace ka {
namespace {

constexpr int kG = 2;              // CTAs per tile
constexpr int kBM = 128;           // rows per CTA
constexpr int kBN = 256;           // columns per tile
constexpr int kBK = 64;            // K per stage
constexpr int kUmmaK = 16;
constexpr int kEpiWarps = 8;        // two per TMEM lane quarter: columns [0,128) and [128,256)
constexpr int kEpiThreads = kEpiWarps * 32;
constexpr int kWarpTma = kEpiWarps, kWarpMma = kEpiWarps + 1, kWarpPub = kEpiWarps + 2;
constexpr int kThreads = kEpiThreads + 96;  // epilogue warps, TMA producer, MMA issuer, one spare warp
constexpr int kMaxStages = 8;
constexpr int kABytes = kBM * kBK * 2;            // 16 KiB
constexpr int kTileBytes = 192 * 1024;            // the operand ring
constexpr int kEpiBufWords = 32 * 33;     // per epilogue warp: 32 rows x 32 words, padded
constexpr int kSmemBytes = kTileBytes + 1024 + 512 + kEpiWarps * kEpiBufWords * 4;
constexpr int kGroupM = 8;         // row tiles that share a column tile in the schedule

struct Control {
  uint64_t full[kMaxStages];
  uint64_t empty[kMaxStages];
  uint64_t tfull[2];
  uint64_t tempty[2];
  uint32_t tmem_base;
  int abort_flag;
};

// Columns per tile: BN = kBN, or half of it for small products (see narrow_tiles).
template <int BN>
struct Cfg {
  static constexpr int kBBytes = (BN / kG) * kBK * 2;
  static constexpr int kStageBytes = kABytes + kBBytes;
  static constexpr int kTxBytes = kStageBytes * kG;
  static constexpr int kStages = kTileBytes / kStageBytes;      // 6, or 8 for the narrow tile
  static_assert(kStages <= kMaxStages, "barriers of the ring");
};

enum Where : int { kWProducer = 11, kWMmaFull = 12, kWMmaTmem = 13, kWEpi = 14, kWReduceFlag = 15, kWGatherFlag = 16 };

// MN-major operand tile written by TMA as 64-element (128 B) wide boxes of 64 K-rows each:
// 16-byte chunks along MN are contiguous (swizzled), 8 K-rows form a 1024 B group (SBO), the
// next 64 MN elements start one box (8 KiB) further (LBO).
__device__ __forceinline__ uint64_t umma_desc_mn_sw128(uint32_t smem_addr) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((smem_addr & 0x3FFFFu) >> 4);
  d |= static_cast<uint64_t>(8192 >> 4) << 16;
  d |= static_cast<uint64_t>(1024 >> 4) << 32;
  d |= static_cast<uint64_t>(1) << 46;
  d |= static_cast<uint64_t>(2) << 61;
  return d;
}

struct Unit {
  int m_blk, n_blk, slice;
};

__device__ __forceinline__ void decode_unit(const GemmParams& p, int tiles_m, int tiles_n, int u, Unit& out) {
  int t = u / p.k_slices;
  out.slice = u - t * p.k_slices;
  if (p.c_slice_stride != 0) {
    // slices apart: all tiles of one slice follow one another, so that pairs that run together share operands
    // (2048 x 4096 x 14336: 183 us, 198 us with all slices of one tile following one another)
    const int tiles = tiles_m * tiles_n;
    out.slice = u / tiles;
    t = u - out.slice * tiles;
  }
  const int per_group = kGroupM * tiles_n;
  const int g = t / per_group;
  const int gm = min(kGroupM, tiles_m - g * kGroupM);
  const int r = t - g * per_group;
  out.n_blk = r / gm;
  out.m_blk = g * kGroupM + (r - out.n_blk * gm);
  // all-gather mode: start with the row tiles whose source is this rank, they need no wait
  if (p.a_gather) out.m_blk = (out.m_blk + (p.rank * p.a_rows_per_rank) / (kBM * kG)) % tiles_m;
  // reduce-scatter mode: start with the row tiles this rank owns, then the next rank's, ... so
  // that at any time every rank stores to a different owner; with one order for all ranks
  // everybody would send to rank 0 first, then to rank 1, ... and each owner's link in turn
  // would carry the whole traffic while the others idle (o_proj of 32768 tokens on 8 GPUs:
  // 1.20 ms with one order, 0.70 ms rotated)
  if (p.epilogue == kEpiPartialF32 && p.world > 1)
    out.m_blk = (out.m_blk + static_cast<int>((static_cast<long long>(p.rank) * p.rows_per_rank) / (kBM * kG))) % tiles_m;
}

// The units of a CTA pair, in order. Plain modes deal units (tile, slice) round robin over the
// pairs; tree mode (kTree) deals whole tiles, so that all slices of a tile follow one another on
// the pair that combines them.
template <bool kTree>
__device__ __forceinline__ int first_unit(int pair_id, int k_slices) {
  return kTree ? pair_id * k_slices : pair_id;
}
template <bool kTree>
__device__ __forceinline__ int next_unit(int u, int n_pairs, int k_slices) {
  if (!kTree) return u + n_pairs;
  return (u + 1) % k_slices != 0 ? u + 1 : u + 1 + (n_pairs - 1) * k_slices;
}

__device__ __forceinline__ void epi_bar() { asm volatile("bar.sync 1, %0;" ::"n"(kEpiThreads) : "memory"); }

__device__ __forceinline__ void tmem_ld_wait_dep(uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.wait::ld.sync.aligned;"
      : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]),
        "+r"(v[7]), "+r"(v[8]), "+r"(v[9]), "+r"(v[10]), "+r"(v[11]), "+r"(v[12]), "+r"(v[13]),
        "+r"(v[14]), "+r"(v[15]), "+r"(v[16]), "+r"(v[17]), "+r"(v[18]), "+r"(v[19]),
        "+r"(v[20]), "+r"(v[21]), "+r"(v[22]), "+r"(v[23]), "+r"(v[24]), "+r"(v[25]),
        "+r"(v[26]), "+r"(v[27]), "+r"(v[28]), "+r"(v[29]), "+r"(v[30]), "+r"(v[31])
      :
      : "memory");
}

__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}

struct RowCtx {
  float neg_lse2;  // -lse * log2(e)
  float gs;        // upstream gradient * scale
  long long tgt;   // target column inside this shard (or out of range)
};

// Layout of the reduce-scatter staging buffer of one owner rank. A partial tile is not stored
// row-major: the 32 rows x 64 columns that one epilogue warp stores at a time are one contiguous
// 4 KiB fragment, [slice][row block][column tile][row quarter][column half][column pair], so
// that a warp's stores to the owner (another GPU for 7/8 of the tiles at TP = 8) cover whole
// contiguous kilobytes instead of 128-byte pieces 8 KiB apart (which reached 160 GB/s over
// NVLink). The reduce tail reads with the same function.
constexpr int kFragElems = 32 * 64;                  // bf16 elements of a fragment
constexpr int kTileElems = kBM * kBN;                // 16 fragments
__device__ __forceinline__ long long stage_offset(int slice, int rblks, int tiles_n, int lr, int col) {
  const int rblk = lr / kBM, r = lr - rblk * kBM;
  const int nb = col / kBN, c = col - nb * kBN;
  const int frag = ((r >> 5) * 2 + (c >> 7)) * 2 + ((c >> 6) & 1);
  return ((static_cast<long long>(slice) * rblks + rblk) * tiles_n + nb) * kTileElems +
         static_cast<long long>(frag) * kFragElems + (r & 31) * 64 + (c & 63);
}

// Store 32 consecutive accumulator columns of the warp's 32 rows. Each lane holds one row
// (that is how tcgen05.ld hands out TMEM lanes); the values are transposed through a padded
// shared-memory tile so that the global stores are whole 64 / 128-byte row segments: eight
// (fp32) or four (bf16) lanes cover one row segment contiguously. This matters most for the
// partial tiles that go to another GPU, where every store instruction becomes NVLink packets.
//
// bf16 outputs are staged two 32-column groups at a time (`half` 0 then 1) and stored after the
// second, so that a row segment is 128 bytes: a whole line for the peer's memory system instead
// of two half-line writes (64-byte segments reached about 140 GB/s over NVLink).
__device__ __forceinline__ void store_group_warp(const GemmParams& p, const uint32_t (&v)[32], uint32_t* wbuf,
                                                 long long row_w0, int col, int slice_global, const RowCtx& rc,
                                                 int lane, int half) {
  const bool f32 = p.epilogue == kEpiStoreF32;
  if (f32 && col >= p.n) return;  // uniform over the warp
  uint32_t* mine = wbuf + lane * 33 + (f32 ? 0 : half * 16);
  if (f32) {
#pragma unroll
    for (int j = 0; j < 32; ++j) mine[j] = v[j];
  } else if (p.epilogue == kEpiLogitsGrad) {
    const float s2 = p.scale * 1.4426950408889634f;
    float d[32];
#pragma unroll
    for (int j = 0; j < 32; ++j) {
      const float pr = ex2_approx(__fmaf_rn(__uint_as_float(v[j]), s2, rc.neg_lse2));
      const float one = (col + j == rc.tgt) ? 1.f : 0.f;
      d[j] = __fmul_rn(rc.gs, __fsub_rn(one, pr));
    }
#pragma unroll
    for (int j = 0; j < 16; ++j) mine[j] = pack_bf16(d[2 * j], d[2 * j + 1]);
  } else {
#pragma unroll
    for (int j = 0; j < 16; ++j) mine[j] = pack_bf16(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1]));
  }
  __syncwarp();
  if (!f32) {
    if (half == 0) return;   // stored together with the next group
    col -= 32;               // first column of the staged pair of groups
    if (col >= p.n) return;  // uniform over the warp
  }
  if (f32) {
    float* base = static_cast<float*>(p.c) + row_w0 * p.ldc + col;
    const long long ld = p.ldc;
    const int c = lane & 7, r0 = lane >> 3;
    const bool col_ok = col + c * 4 + 4 <= p.n;
#pragma unroll
    for (int it = 0; it < 8; ++it) {
      const int r = r0 + 4 * it;
      if (col_ok && row_w0 + r < p.m) {
        const uint32_t* src = wbuf + r * 33 + c * 4;
        *reinterpret_cast<uint4*>(base + r * ld + c * 4) = make_uint4(src[0], src[1], src[2], src[3]);
      }
    }
  } else {
    __nv_bfloat16* base;
    long long ld;
    if (p.epilogue == kEpiPartialF32) {
      const int owner = static_cast<int>(row_w0 / p.rows_per_rank);
      const int lr = static_cast<int>(row_w0 - static_cast<long long>(owner) * p.rows_per_rank);
      base = static_cast<__nv_bfloat16*>(p.stage[owner]) +
             stage_offset(slice_global, p.rows_per_rank / kBM, (p.n + kBN - 1) / kBN, lr, col);
      ld = 64;  // rows of a fragment are 64 elements apart
    } else {
      base = static_cast<__nv_bfloat16*>(p.c) + slice_global * p.c_slice_stride + row_w0 * p.ldc + col;
      ld = p.ldc;
    }
    const int c = lane & 7, r0 = lane >> 3;   // eight lanes cover the 128 bytes of one row
    const bool col_ok = col + c * 8 + 8 <= p.n;
#pragma unroll
    for (int it = 0; it < 8; ++it) {
      const int r = r0 + 4 * it;
      if (col_ok && row_w0 + r < p.m) {
        const uint32_t* src = wbuf + r * 33 + c * 4;
        *reinterpret_cast<uint4*>(base + r * ld + c * 8) = make_uint4(src[0], src[1], src[2], src[3]);
      }
    }
  }
  __syncwarp();
}

__device__ __forceinline__ float4 ld_f4_sys(const float* p) {
  return ld_relaxed_sys_f4(reinterpret_cast<const float4*>(p));
}
__device__ __forceinline__ float4 add4(float4 a, float4 b) {
  return make_float4(__fadd_rn(a.x, b.x), __fadd_rn(a.y, b.y), __fadd_rn(a.z, b.z), __fadd_rn(a.w, b.w));
}

// ---- tree mode: the eight canonical K slices of a tile summed where they are computed.
// A thread of the epilogue owns one row and 128 columns of the tile. Slice partials are rounded
// to bf16 once and added in fp32 as ((0+1)+(2+3))+((4+5)+(6+7)), the reduce-scatter tail's
// order, so the bits are those of the staged path. Even slices stay in registers as packed
// bf16; (0+1), then (0+1)+(2+3), and (4+5) wait in two fp32 slots of a per-CTA scratch block
// (2 x 128 KiB, 38 MB over the device: it stays in L2) that only this thread reads back.
constexpr int kTreeSlices = 8;
constexpr int kTreeSlotFloats = kBM * kBN;

template <int BN>
__device__ __forceinline__ float4* tree_slot(float* scratch, int cta, int slot, int warp, int g, int lane) {
  return reinterpret_cast<float4*>(scratch + (static_cast<size_t>(cta) * 2 + slot) * kTreeSlotFloats) +
         (warp * (BN / 64) + g) * 8 * 32 + lane;   // eight float4 per thread and group, 32 apart
}

__device__ __forceinline__ float bf16_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t w) { return __uint_as_float(w & 0xFFFF0000u); }

// One 32-column group of slice `s`. `v`: the accumulators; `leaf`: the packed even slice of the
// pair. Returns true when the tile is finished: `v` then holds 32 sums.
template <int BN>
__device__ __forceinline__ bool tree_group(float* scratch, int s, int warp, int g, int lane, uint32_t (&v)[32],
                                           uint32_t (&leaf)[16]) {
  if ((s & 1) == 0) {
#pragma unroll
    for (int j = 0; j < 16; ++j) leaf[j] = pack_bf16(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1]));
    return false;
  }
  float4* s0 = tree_slot<BN>(scratch, blockIdx.x, 0, warp, g, lane);
  float4* s1 = tree_slot<BN>(scratch, blockIdx.x, 1, warp, g, lane);
  float4 t[8];
  if (s == 3 || s == 7) {
    const float4* src = s == 3 ? s0 : s1;
#pragma unroll
    for (int i = 0; i < 8; ++i) t[i] = src[i * 32];
  }
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    const uint32_t w = pack_bf16(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1]));
    v[2 * j] = __float_as_uint(__fadd_rn(bf16_lo(leaf[j]), bf16_lo(w)));
    v[2 * j + 1] = __float_as_uint(__fadd_rn(bf16_hi(leaf[j]), bf16_hi(w)));
  }
  if (s == 3 || s == 7) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float4 a = add4(t[i], make_float4(__uint_as_float(v[4 * i]), __uint_as_float(v[4 * i + 1]),
                                              __uint_as_float(v[4 * i + 2]), __uint_as_float(v[4 * i + 3])));
      v[4 * i] = __float_as_uint(a.x);
      v[4 * i + 1] = __float_as_uint(a.y);
      v[4 * i + 2] = __float_as_uint(a.z);
      v[4 * i + 3] = __float_as_uint(a.w);
    }
  }
  if (s == 7) {
#pragma unroll
    for (int i = 0; i < 8; ++i) t[i] = s0[i * 32];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float4 a = add4(t[i], make_float4(__uint_as_float(v[4 * i]), __uint_as_float(v[4 * i + 1]),
                                              __uint_as_float(v[4 * i + 2]), __uint_as_float(v[4 * i + 3])));
      v[4 * i] = __float_as_uint(a.x);
      v[4 * i + 1] = __float_as_uint(a.y);
      v[4 * i + 2] = __float_as_uint(a.z);
      v[4 * i + 3] = __float_as_uint(a.w);
    }
    return true;
  }
  float4* dst = s == 5 ? s1 : s0;
#pragma unroll
  for (int i = 0; i < 8; ++i)
    dst[i * 32] = make_float4(__uint_as_float(v[4 * i]), __uint_as_float(v[4 * i + 1]), __uint_as_float(v[4 * i + 2]),
                              __uint_as_float(v[4 * i + 3]));
  return false;
}

// Store two finished 32-column groups (`half` 0 stages, 1 stores) with the optional residual:
// the sum is rounded to bf16 first, as a separate bf16 linear + add would.
__device__ __forceinline__ void tree_store(const GemmParams& p, const uint32_t (&v)[32], uint32_t* wbuf,
                                           long long row_w0, int col, int lane, int half) {
  uint32_t* mine = wbuf + lane * 33 + half * 16;
#pragma unroll
  for (int j = 0; j < 16; ++j) mine[j] = pack_bf16(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1]));
  __syncwarp();
  if (half == 0) return;
  const int c = lane & 7, r0 = lane >> 3;
  const bool col_ok = col + c * 8 + 8 <= p.n;
#pragma unroll
  for (int it = 0; it < 8; ++it) {
    const int r = r0 + 4 * it;
    if (col_ok && row_w0 + r < p.m) {
      const uint32_t* src = wbuf + r * 33 + c * 4;
      const long long off = (row_w0 + r) * p.n + col + c * 8;
      uint4 o = make_uint4(src[0], src[1], src[2], src[3]);
      if (p.residual) {
        const uint4 rr = *reinterpret_cast<const uint4*>(static_cast<const __nv_bfloat16*>(p.residual) + off);
        o.x = pack_bf16(__fadd_rn(bf16_lo(o.x), bf16_lo(rr.x)), __fadd_rn(bf16_hi(o.x), bf16_hi(rr.x)));
        o.y = pack_bf16(__fadd_rn(bf16_lo(o.y), bf16_lo(rr.y)), __fadd_rn(bf16_hi(o.y), bf16_hi(rr.y)));
        o.z = pack_bf16(__fadd_rn(bf16_lo(o.z), bf16_lo(rr.z)), __fadd_rn(bf16_hi(o.z), bf16_hi(rr.z)));
        o.w = pack_bf16(__fadd_rn(bf16_lo(o.w), bf16_lo(rr.w)), __fadd_rn(bf16_hi(o.w), bf16_hi(rr.w)));
      }
      *reinterpret_cast<uint4*>(static_cast<__nv_bfloat16*>(p.out) + off) = o;
    }
  }
  __syncwarp();
}

template <bool kTree, int BN>
__global__ void __launch_bounds__(kThreads, 1)
gemm_bf16_kernel(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_b,
                 const __grid_constant__ GemmParams p) {
  using C = Cfg<BN>;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = smem_u32(smem_raw);
  const uint32_t tiles_addr = (raw_addr + 1023u) & ~1023u;
  uint8_t* tiles = smem_raw + (tiles_addr - raw_addr);
  Control* ctl = reinterpret_cast<Control*>(tiles + kTileBytes);
  uint32_t* epi_buf = reinterpret_cast<uint32_t*>(tiles + kTileBytes + 512);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t cta_rank = cluster_ctarank();
  const bool leader = cta_rank == 0;
  const int pair_id = blockIdx.x / kG;
  const int n_pairs = gridDim.x / kG;
  const int tiles_m = (p.m + kBM * kG - 1) / (kBM * kG);
  const int tiles_n = (p.n + BN - 1) / BN;
  const int n_units = tiles_m * tiles_n * p.k_slices;
  const int k_per_slice = p.k / p.k_slices;
  const int num_kb = (k_per_slice + kBK - 1) / kBK;

  WaitCtx wctx{&ctl->abort_flag, p.status, p.timeout_ns};

  if (threadIdx.x == 0) {
    for (int s = 0; s < C::kStages; ++s) {
      mbar_init(smem_u32(&ctl->full[s]), 1);
      mbar_init(smem_u32(&ctl->empty[s]), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(smem_u32(&ctl->tfull[b]), 1);
      mbar_init(smem_u32(&ctl->tempty[b]), kEpiWarps * kG);
    }
    ctl->abort_flag = 0;
    fence_mbar_init_cluster();
  }
  if (warp == kWarpMma) {
    tmem_alloc<kG>(smem_u32(&ctl->tmem_base), 2 * BN);
    tmem_relinquish<kG>();
  }
  if (warp == kWarpTma && lane == 0) {
    tma_prefetch_desc(&tm_a);
    tma_prefetch_desc(&tm_b);
  }
  tc_fence_before_sync();
  __syncthreads();
  cluster_arrive();
  cluster_wait();
  tc_fence_after_sync();
  const uint32_t tmem_base = ctl->tmem_base;

  if (warp == kWarpTma) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int u = first_unit<kTree>(pair_id, p.k_slices); u < n_units && ok; u = next_unit<kTree>(u, n_pairs, p.k_slices)) {
        Unit un;
        decode_unit(p, tiles_m, tiles_n, u, un);
        const int row0 = un.m_blk * (kBM * kG) + static_cast<int>(cta_rank) * kBM;
        const int col0 = un.n_blk * BN + static_cast<int>(cta_rank) * (BN / kG);
        const int kbase = un.slice * k_per_slice;
        if (p.a_gather) {
          // rows of another rank become readable when that rank's push has been flagged
          const int src = row0 / p.a_rows_per_rank;
          const int blk = (row0 - src * p.a_rows_per_rank) / kBM;
          const int blocks = p.a_rows_per_rank / kBM;
          if (row0 < p.m)
            ok = flag_wait_bounded(p.a_flags[p.rank] + static_cast<size_t>(src) * blocks + blk, p.epoch, wctx,
                                   kWGatherFlag, src * 65536 + blk);
          if (!ok) break;
        }
        for (int kb = 0; kb < num_kb; ++kb) {
          ok = mbar_wait_bounded(smem_u32(&ctl->empty[stage]), phase ^ 1u, wctx, kWProducer, stage);
          if (!ok) break;
          const uint32_t a_dst = tiles_addr + stage * C::kStageBytes;
          const uint32_t b_dst = a_dst + kABytes;
          const uint32_t full = smem_u32(&ctl->full[stage]);
          if (leader) mbar_arrive_expect_tx(full, C::kTxBytes);
          const uint32_t full_leader = mapa_u32(full, 0);
          const int k0 = kbase + kb * kBK;
          if (p.a_major == 0) {
            tma_load_2d_pair(a_dst, &tm_a, k0, row0, full_leader);
          } else {
            tma_load_2d_pair(a_dst, &tm_a, row0, k0, full_leader);
            tma_load_2d_pair(a_dst + 8192, &tm_a, row0 + 64, k0, full_leader);
          }
          if (p.b_major == 0) {
            tma_load_2d_pair(b_dst, &tm_b, k0, col0, full_leader);
          } else {
            tma_load_2d_pair(b_dst, &tm_b, col0, k0, full_leader);
            if constexpr (BN / kG > 64) tma_load_2d_pair(b_dst + 8192, &tm_b, col0 + 64, k0, full_leader);
          }
          if (++stage == C::kStages) {
            stage = 0;
            phase ^= 1u;
          }
        }
      }
    }
  } else if (warp == kWarpMma) {
    // ------------------------------------------------------------------ MMA issuer
    if (lane == 0 && leader) {
      const uint32_t idesc = umma_idesc_bf16_f32(kBM * kG, BN) | (static_cast<uint32_t>(p.a_major) << 15) |
                             (static_cast<uint32_t>(p.b_major) << 16);
      const uint32_t a_step = p.a_major == 0 ? 2u : 128u;  // descriptor units (16 B) per K=16
      const uint32_t b_step = p.b_major == 0 ? 2u : 128u;
      int stage = 0;
      uint32_t phase = 0;
      int abuf = 0;
      uint32_t aphase = 0;
      bool ok = true;
      for (int u = first_unit<kTree>(pair_id, p.k_slices); u < n_units && ok; u = next_unit<kTree>(u, n_pairs, p.k_slices)) {
        ok = mbar_wait_bounded(smem_u32(&ctl->tempty[abuf]), aphase ^ 1u, wctx, kWMmaTmem, abuf);
        if (!ok) break;
        tc_fence_after_sync();
        const uint32_t d_tmem = tmem_base + static_cast<uint32_t>(abuf * BN);
        for (int kb = 0; kb < num_kb; ++kb) {
          ok = mbar_wait_bounded(smem_u32(&ctl->full[stage]), phase, wctx, kWMmaFull, stage);
          if (!ok) break;
          tc_fence_after_sync();
          const uint32_t a_addr = tiles_addr + stage * C::kStageBytes;
          const uint64_t a_desc = p.a_major == 0 ? umma_desc_k_sw128(a_addr) : umma_desc_mn_sw128(a_addr);
          const uint64_t b_desc =
              p.b_major == 0 ? umma_desc_k_sw128(a_addr + kABytes) : umma_desc_mn_sw128(a_addr + kABytes);
#pragma unroll
          for (int k = 0; k < kBK / kUmmaK; ++k) {
            umma_bf16<kG>(d_tmem, a_desc + a_step * k, b_desc + b_step * k, idesc, (kb > 0 || k > 0) ? 1u : 0u);
          }
          umma_commit<kG>(smem_u32(&ctl->empty[stage]));
          if (++stage == C::kStages) {
            stage = 0;
            phase ^= 1u;
          }
        }
        if (!ok) break;
        umma_commit<kG>(smem_u32(&ctl->tfull[abuf]));
        abuf ^= 1;
        if (abuf == 0) aphase ^= 1u;
      }
    }
  } else if (warp == kWarpPub) {
    // (spare warp: the flags of the partial tiles are raised by the epilogue warps once, after
    // the CTA's last unit; a system-scope fence and a flag per unit made every unit wait for the
    // round trip of its own peer stores: 1.47 ms against 1.20 ms for o_proj of 32768 tokens)
  } else {
    // ------------------------------------------------------------------ epilogue (warps 0-7)
    // Warp w reads TMEM lanes 32 * (w & 3) .. +31 (its rows) and columns 128 * (w >> 2) .. +127.
    // The unit loop has no CTA-wide barrier: a warp whose wait runs out simply leaves it. The
    // named barriers of the copy and reduce phases are reached by all 256 threads.
    const int tid = threadIdx.x;
    const int wq = warp & 3, wh = warp >> 2;
    bool ok = true;

    if (p.a_gather) {
      // ---- all-gather: push this rank's rows of A into every peer's gather buffer, one
      // 128-row block at a time, then raise the block's flag on that peer.
      const int blocks = p.a_rows_per_rank / kBM;
      const int vec_per_row = p.k / 8;  // 16-byte vectors
      const uint4* src = static_cast<const uint4*>(p.a_local);
      const long long nv = static_cast<long long>(kBM) * vec_per_row;
      // work item = (destination, 128-row block), destination-major starting with this rank, so
      // the local copy (which this rank's own GEMM needs first) leaves first
      for (int it = blockIdx.x; it < blocks * p.world; it += gridDim.x) {
        const int d = it / blocks, blk = it - d * blocks;
        const int dst_rank = (p.rank + d) % p.world;
        const long long v0 = static_cast<long long>(blk) * nv;
        uint4* dst = static_cast<uint4*>(p.a_bufs[dst_rank]) +
                     static_cast<long long>(p.rank) * p.a_rows_per_rank * vec_per_row + v0;
        constexpr int kS = kEpiThreads;
        for (long long i = tid; i < nv; i += 4 * kS) {
          // four independent 16-byte copies in flight per thread
          uint4 t0 = src[v0 + i], t1, t2, t3;
          const bool b1 = i + kS < nv, b2 = i + 2 * kS < nv, b3 = i + 3 * kS < nv;
          if (b1) t1 = src[v0 + i + kS];
          if (b2) t2 = src[v0 + i + 2 * kS];
          if (b3) t3 = src[v0 + i + 3 * kS];
          dst[i] = t0;
          if (b1) dst[i + kS] = t1;
          if (b2) dst[i + 2 * kS] = t2;
          if (b3) dst[i + 3 * kS] = t3;
        }
        epi_bar();
        if (tid == 0) {
          __threadfence_system();
          st_release_sys_u32(p.a_flags[dst_rank] + static_cast<size_t>(p.rank) * blocks + blk, p.epoch);
        }
      }
    }

    int abuf = 0;
    uint32_t aphase = 0;
    const uint32_t tempty_leader = mapa_u32(smem_u32(&ctl->tempty[0]), 0);
    uint32_t leaf[kTree ? BN / 64 : 1][16];
    for (int u = first_unit<kTree>(pair_id, p.k_slices); u < n_units; u = next_unit<kTree>(u, n_pairs, p.k_slices)) {
      Unit un;
      decode_unit(p, tiles_m, tiles_n, u, un);
      const long long row_w0 = static_cast<long long>(un.m_blk) * (kBM * kG) + cta_rank * kBM + wq * 32;
      const long long row = row_w0 + lane;
      const bool mine = mbar_wait_bounded(smem_u32(&ctl->tfull[abuf]), aphase, wctx, kWEpi, abuf);
      ok = __all_sync(0xffffffffu, mine) != 0;
      if (!ok) break;
      tc_fence_after_sync();
      const uint32_t trow = tmem_base + (static_cast<uint32_t>(wq * 32) << 16) +
                            static_cast<uint32_t>(abuf * BN + wh * (BN / 2));
      const int col0 = un.n_blk * BN + wh * (BN / 2);
      const int slice_global = p.slice_base + un.slice;
      RowCtx rc = {0.f, 0.f, -1};
      if (p.epilogue == kEpiLogitsGrad && row < p.m) {
        rc.neg_lse2 = __fmul_rn(-p.row_lse[row], 1.4426950408889634f);
        rc.gs = __fmul_rn(p.row_g[row], p.scale);
        rc.tgt = p.row_ids[row] - p.col_offset;
      }
      uint32_t* wbuf = epi_buf + warp * kEpiBufWords;
      if constexpr (kTree) {
#pragma unroll
        for (int g = 0; g < BN / 64; ++g) {
          uint32_t v[32];
          __syncwarp();
          tmem_ld_32x32(trow + g * 32, v);
          tmem_ld_wait_dep(v);
          if (tree_group<BN>(p.tree_scratch, un.slice, warp, g, lane, v, leaf[g]))
            tree_store(p, v, wbuf, row_w0, col0 + (g & ~1) * 32, lane, g & 1);
        }
      } else {
      uint32_t va[32], vb[32];
      tmem_ld_32x32(trow, va);
      tmem_ld_wait_dep(va);
#pragma unroll
      for (int g = 0; g < BN / 64; g += 2) {
        __syncwarp();
        tmem_ld_32x32(trow + (g + 1) * 32, vb);
        store_group_warp(p, va, wbuf, row_w0, col0 + g * 32, slice_global, rc, lane, 0);
        __syncwarp();
        tmem_ld_wait_dep(vb);
        if (g + 2 < BN / 64) tmem_ld_32x32(trow + (g + 2) * 32, va);
        store_group_warp(p, vb, wbuf, row_w0, col0 + (g + 1) * 32, slice_global, rc, lane, 1);
        __syncwarp();
        if (g + 2 < BN / 64) tmem_ld_wait_dep(va);
      }
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(tempty_leader + static_cast<uint32_t>(abuf) * 8u);
      abuf ^= 1;
      if (abuf == 0) aphase ^= 1u;
    }

    if (BN == kBN && p.epilogue == kEpiPartialF32) {
      // Publish the partial tiles: every thread makes its own stores visible system-wide, the
      // CTA meets, then the flags of all units this CTA computed are raised (the owners read
      // them in their reduce tails, which start after their own last unit anyway).
      __threadfence_system();
      epi_bar();  // every epilogue thread gets here, whether or not its loop ran to the end
      if (ctl->abort_flag) ok = false;
      if (ok) {
        const int rblks = p.rows_per_rank / kBM;
        int k = 0;
        for (int u = pair_id; u < n_units; u += n_pairs, ++k) {
          if ((k % kEpiThreads) != tid) continue;
          Unit un;
          decode_unit(p, tiles_m, tiles_n, u, un);
          const long long row0 = static_cast<long long>(un.m_blk) * (kBM * kG) + cta_rank * kBM;
          if (row0 < p.m) {
            const int owner = static_cast<int>(row0 / p.rows_per_rank);
            const int rblk = static_cast<int>((row0 - static_cast<long long>(owner) * p.rows_per_rank) / kBM);
            st_release_sys_u32(p.flags[owner] + (static_cast<size_t>(p.slice_base + un.slice) * rblks + rblk) * tiles_n +
                                   un.n_blk,
                               p.epoch);
          }
        }
      }
    }
    if (BN == kBN && p.epilogue == kEpiPartialF32 && ok && p.out != nullptr) {
      // ---- reduce-scatter tail (skipped when the caller only wants the partials staged): the rows this rank owns, slices combined by a balanced tree
      const int rblks = p.rows_per_rank / kBM;
      const int items = rblks * tiles_n;
      const int rows_valid = min(p.rows_per_rank, p.m - p.rank * p.rows_per_rank);
      for (int it = blockIdx.x; it < items; it += gridDim.x) {
        const int rblk = it / tiles_n, nb = it - rblk * tiles_n;
        if (rblk * kBM >= rows_valid) continue;  // block past the end of the matrix: nobody writes it
        if (tid < p.total_slices)
          flag_wait_bounded(p.flags[p.rank] + (static_cast<size_t>(tid) * rblks + rblk) * tiles_n + nb, p.epoch, wctx,
                            kWReduceFlag, it);
        epi_bar();
        if (ctl->abort_flag) break;
        const int ncols = min(kBN, p.n - nb * kBN);
        const int vec_per_row = ncols / 8;  // 8 bf16 = 16 bytes
        const size_t slice_stride = static_cast<size_t>(rblks) * tiles_n * kTileElems;
#pragma unroll 2
        for (int i = tid; i < kBM * vec_per_row; i += kEpiThreads) {
          const int r = i / vec_per_row, c8 = i - r * vec_per_row;
          const int lr = rblk * kBM + r;
          if (lr >= rows_valid) continue;
          const size_t off = static_cast<size_t>(lr) * p.n + nb * kBN + c8 * 8;  // in out / residual (row-major)
          const __nv_bfloat16* base = static_cast<const __nv_bfloat16*>(p.stage[p.rank]) +
                                      stage_offset(0, rblks, tiles_n, lr, nb * kBN + c8 * 8);
          float4 lo[8], hi[8];
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            if (q < p.total_slices) {
              // weak L2 loads: the acquire on the flags (and the barrier) orders them after the peers'
              // stores, and unlike system-scope strong loads they pipeline
              const float4 raw = __ldcg(reinterpret_cast<const float4*>(base + q * slice_stride));
              const uint32_t w0 = __float_as_uint(raw.x), w1 = __float_as_uint(raw.y), w2 = __float_as_uint(raw.z),
                             w3 = __float_as_uint(raw.w);
              lo[q] = make_float4(__uint_as_float(w0 << 16), __uint_as_float(w0 & 0xFFFF0000u),
                                  __uint_as_float(w1 << 16), __uint_as_float(w1 & 0xFFFF0000u));
              hi[q] = make_float4(__uint_as_float(w2 << 16), __uint_as_float(w2 & 0xFFFF0000u),
                                  __uint_as_float(w3 << 16), __uint_as_float(w3 & 0xFFFF0000u));
            } else {
              lo[q] = make_float4(0.f, 0.f, 0.f, 0.f);
              hi[q] = lo[q];
            }
          }
          float4 a0 = add4(add4(add4(lo[0], lo[1]), add4(lo[2], lo[3])), add4(add4(lo[4], lo[5]), add4(lo[6], lo[7])));
          float4 a1 = add4(add4(add4(hi[0], hi[1]), add4(hi[2], hi[3])), add4(add4(hi[4], hi[5]), add4(hi[6], hi[7])));
          if (p.residual) {
            // residual add in bf16 arithmetic order: round the GEMM result first, as a separate
            // bf16 linear + add would
            const uint4 rr = *reinterpret_cast<const uint4*>(static_cast<const __nv_bfloat16*>(p.residual) + off);
            auto addr = [](float g, uint32_t rbits) {
              return __fadd_rn(__bfloat162float(__float2bfloat16_rn(g)), __uint_as_float(rbits));
            };
            a0.x = addr(a0.x, rr.x << 16);
            a0.y = addr(a0.y, rr.x & 0xFFFF0000u);
            a0.z = addr(a0.z, rr.y << 16);
            a0.w = addr(a0.w, rr.y & 0xFFFF0000u);
            a1.x = addr(a1.x, rr.z << 16);
            a1.y = addr(a1.y, rr.z & 0xFFFF0000u);
            a1.z = addr(a1.z, rr.w << 16);
            a1.w = addr(a1.w, rr.w & 0xFFFF0000u);
          }
          uint4 o;
          o.x = pack_bf16(a0.x, a0.y);
          o.y = pack_bf16(a0.z, a0.w);
          o.z = pack_bf16(a1.x, a1.y);
          o.w = pack_bf16(a1.z, a1.w);
          *reinterpret_cast<uint4*>(static_cast<__nv_bfloat16*>(p.out) + off) = o;
        }
      }
    }
  }

  // ------------------------------------------------------------------ common exit
  if (ctl->abort_flag) {
    st_shared_cluster_u32(mapa_u32(smem_u32(&ctl->abort_flag), cta_rank ^ 1u), 1u);
    drain_in_flight();
  }
  tc_fence_before_sync();
  __syncthreads();
  cluster_arrive();
  cluster_wait();
  if (warp == kWarpMma) {
    __syncwarp();
    tc_fence_after_sync();
    tmem_dealloc<kG>(tmem_base, 2 * BN);
  }
}

// Resident CTAs of the kernel on the current device, with its shared memory opted in there.
template <bool kTree, int BN>
int setup_ctas(int num_sms) {
  if (cudaFuncSetAttribute(gemm_bf16_kernel<kTree, BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes) != cudaSuccess)
    return -1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(num_sms / 2 * 2));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = kSmemBytes;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int clusters = 0;
  if (cudaOccupancyMaxActiveClusters(&clusters, gemm_bf16_kernel<kTree, BN>, &cfg) != cudaSuccess || clusters <= 0) {
    cudaGetLastError();
    clusters = num_sms / 2;
  }
  int n = clusters * 2;
  if (n > num_sms / 2 * 2) n = num_sms / 2 * 2;
  return n;
}

template <bool kTree, int BN>
int max_ctas(int num_sms) {
  static PerDevice once;
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess) return -1;
  return once.get(dev, [&] { return setup_ctas<kTree, BN>(num_sms); });
}

// Whether a product takes tiles of 128 columns instead of 256: when the narrow tiles still fit the
// CTA pairs in one round, so that twice as many SMs run the epilogue and the last tile's drain. What
// that saves is the same for every K (about 1 us, 8 us where the slices are kept in the kernel), while
// the narrow tiles load a third more per product, so a plain product with a long K takes the wide ones.
// Measured wide / narrow in us, 4 to 36 wide tiles on 74 pairs: plain, 464 x 4096 (32 tiles): 8.1 / 6.9
// (K = 128), 27.8 / 26.9 (4096), 76.4 / 76.1 (14336), 103.6 / 103.5 (20000), 160.4 / 161.3 (32000), 629 / 648
// (128256: the hidden gradient of the LM head); slices kept in the kernel, 512 x 4096: 43.4 / 35.2 (4096),
// 93.2 / 88.4 (14336), 167 / 162 (28672). More narrow tiles than pairs would need another round.
constexpr int kNarrowMaxK = 16384;

inline bool narrow_tiles(int tiles_m, int tiles_n, int k, bool tree, int pairs) {
  return static_cast<long long>(tiles_m) * tiles_n * 2 <= pairs && (tree || k <= kNarrowMaxK);
}

// ---- split mode (ka_gemm_split8). A pair that keeps a tile walks its eight slices one after the other, so few
// tiles with a long K leave most pairs idle; the times of both are with the rule (_split_pays in
// parallel/tp_gemm.py). The price is a pass over the partials, 3 to 6 us (they stay in L2). A unit is always a
// tile of 256 columns: with 128 there are twice as many, and one takes 0.7 (K = 4096) to 0.9 (28672) of the
// time. Wide / narrow units in us: 512 x 1024 19.6 / 19.3 (K = 4096), 34.3 / 50.3 (28672), 128 x 5120 24.1 / 28.1,
// 79.3 / 105.5; 512 x 4096 32.2 / 36.8, 101.5 / 143.8; 768 x 4096 44.7 / 52.7, 148.6 / 218.6; 128 x 1024, where
// both are one round, 19.3 / 19.2, 32.3 / 31.5. Second half: the eight bf16 partials
// of every element summed in the order of the reduce-scatter tail, ((0+1)+(2+3))+((4+5)+(6+7)) in fp32,
// rounded, the residual added after that.
constexpr int kSumThreads = 256;

__global__ void __launch_bounds__(kSumThreads)
slice_sum_kernel(const uint4* __restrict__ part, long long vecs, const uint4* __restrict__ residual, uint4* __restrict__ out) {
  const long long i = static_cast<long long>(blockIdx.x) * kSumThreads + threadIdx.x;
  if (i >= vecs) return;
  uint4 v[kTreeSlices];
#pragma unroll
  for (int s = 0; s < kTreeSlices; ++s) v[s] = __ldcg(part + s * vecs + i);
  uint4 r = make_uint4(0u, 0u, 0u, 0u);
  if (residual) r = __ldg(residual + i);
  auto word = [&](auto get) {
    float lo[kTreeSlices], hi[kTreeSlices];
#pragma unroll
    for (int s = 0; s < kTreeSlices; ++s) {
      lo[s] = bf16_lo(get(v[s]));
      hi[s] = bf16_hi(get(v[s]));
    }
    auto tree = [](const float(&a)[kTreeSlices]) {
      return __fadd_rn(__fadd_rn(__fadd_rn(a[0], a[1]), __fadd_rn(a[2], a[3])),
                       __fadd_rn(__fadd_rn(a[4], a[5]), __fadd_rn(a[6], a[7])));
    };
    uint32_t o = pack_bf16(tree(lo), tree(hi));
    if (residual) o = pack_bf16(__fadd_rn(bf16_lo(o), bf16_lo(get(r))), __fadd_rn(bf16_hi(o), bf16_hi(get(r))));
    return o;
  };
  out[i] = make_uint4(word([](const uint4& a) { return a.x; }), word([](const uint4& a) { return a.y; }),
                      word([](const uint4& a) { return a.z; }), word([](const uint4& a) { return a.w; }));
}

}  // namespace

// Shared by the plain entry point and the tensor-parallel ones (tp_gemm.cu): build the
// tensor maps for the operand layouts in `p` and launch.
int gemm_launch(const void* a, long long lda, const void* b, long long ldb, const GemmParams& p, int num_sms,
                bool full_grid, cudaStream_t stream) {
  if (p.m <= 0 || p.n <= 0 || p.k <= 0) return 0;
  if (p.k % 8 != 0 || p.n % 8 != 0 || lda % 8 != 0 || ldb % 8 != 0) return -1;
  if (p.k_slices < 1 || p.k % p.k_slices != 0 || (p.k_slices > 1 && (p.k / p.k_slices) % kBK != 0)) return -2;
  if (p.a_major == 1 && p.m % 8 != 0) return -3;
  const bool tree = p.epilogue == kEpiTreeBf16;
  if (tree && (p.k_slices != kTreeSlices || !p.tree_scratch)) return -4;
  int ctas = tree ? max_ctas<true, kBN>(num_sms) : max_ctas<false, kBN>(num_sms);
  if (ctas <= 0) return -10;
  const int tiles_m = (p.m + kBM * kG - 1) / (kBM * kG);
  const bool narrow = !full_grid && p.c_slice_stride == 0 &&
                      narrow_tiles(tiles_m, (p.n + kBN - 1) / kBN, p.k, tree, ctas / kG);
  if (narrow) ctas = tree ? max_ctas<true, kBN / 2>(num_sms) : max_ctas<false, kBN / 2>(num_sms);
  if (ctas <= 0) return -10;
  const int bn = narrow ? kBN / 2 : kBN;
  const int tiles_n = (p.n + bn - 1) / bn;
  CUtensorMap tm_a, tm_b;
  int rc;
  if (p.a_major == 0)
    rc = make_tmap_2d_16bit_sw128(&tm_a, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, a, p.m, p.k, lda, kBM, kBK);
  else
    rc = make_tmap_2d_16bit_sw128(&tm_a, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, a, p.k, p.m, lda, kBK, 64);
  if (rc != 0) return -20 + rc;
  if (p.b_major == 0)
    rc = make_tmap_2d_16bit_sw128(&tm_b, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, b, p.n, p.k, ldb, bn / kG, kBK);
  else
    rc = make_tmap_2d_16bit_sw128(&tm_b, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, b, p.k, p.n, ldb, kBK, 64);
  if (rc != 0) return -40 + rc;
  const int units = tiles_m * tiles_n * (tree ? 1 : p.k_slices);
  if (!full_grid && units * kG < ctas) ctas = units * kG;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(ctas));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = kSmemBytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = kG;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  auto* kernel = narrow ? (tree ? gemm_bf16_kernel<true, kBN / 2> : gemm_bf16_kernel<false, kBN / 2>)
                        : (tree ? gemm_bf16_kernel<true, kBN> : gemm_bf16_kernel<false, kBN>);
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, tm_a, tm_b, p);
  if (e != cudaSuccess) {
    fprintf(stderr, "[kernel_align_b200] gemm launch failed: %s\n", cudaGetErrorString(e));
    return -11;
  }
  return 0;
}

}  // namespace ka

// Columns per tile that an m x n x k product takes on a device where `pairs` CTA pairs are resident;
// tree: with its eight K slices summed in the kernel.
extern "C" int ka_gemm_tile_columns(int m, int n, int k, int tree, int pairs) {
  using namespace ka;
  return narrow_tiles((m + kBM * kG - 1) / (kBM * kG), (n + kBN - 1) / kBN, k, tree != 0, pairs) ? kBN / 2 : kBN;
}

extern "C" int ka_gemm_bf16(const void* a, long long lda, int a_major, const void* b, long long ldb, int b_major,
                            void* c, long long ldc, int out_f32, int m, int n, int k, int* status, int num_sms,
                            unsigned long long timeout_ns, void* stream) {
  ka::GemmParams p = {};
  p.m = m;
  p.n = n;
  p.k = k;
  p.a_major = a_major ? 1 : 0;
  p.b_major = b_major ? 1 : 0;
  p.epilogue = out_f32 ? ka::kEpiStoreF32 : ka::kEpiStoreBf16;
  p.c = c;
  p.ldc = ldc;
  p.k_slices = 1;
  p.total_slices = 1;
  p.world = 1;
  p.status = status;
  p.timeout_ns = timeout_ns;
  return ka::gemm_launch(a, lda, b, ldb, p, num_sms, false, static_cast<cudaStream_t>(stream));
}

// Bytes of scratch ka_gemm_tree8 needs on a device with num_sms SMs (uninitialised memory).
extern "C" size_t ka_gemm_tree8_scratch_bytes(int num_sms) {
  return static_cast<size_t>(num_sms) * 2 * ka::kTreeSlotFloats * sizeof(float);
}

// out[m, n] (bf16, row-major) = a[m, k] times b^T (+ residual) with K cut into the eight
// canonical slices of the tensor-parallel linears, every slice rounded to bf16 once and summed in
// fp32 in the fixed tree order: what ka_gemm_reduce_scatter computes on one rank, bit for bit,
// without its staging buffers. b: [n, k] (b_major = 0) or [k, n] (b_major = 1).
extern "C" int ka_gemm_tree8(const void* a, long long lda, const void* b, long long ldb, int b_major, void* out,
                             const void* residual, void* scratch, int m, int n, int k, int* status, int num_sms,
                             unsigned long long timeout_ns, void* stream) {
  if (n % 8 != 0) return -51;
  if (((reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(residual)) & 15u) != 0) return -54;
  ka::GemmParams p = {};
  p.m = m;
  p.n = n;
  p.k = k;
  p.b_major = b_major ? 1 : 0;
  p.epilogue = ka::kEpiTreeBf16;
  p.out = out;
  p.residual = residual;
  p.tree_scratch = static_cast<float*>(scratch);
  p.k_slices = ka::kTreeSlices;
  p.total_slices = ka::kTreeSlices;
  p.world = 1;
  p.status = status;
  p.timeout_ns = timeout_ns;
  return ka::gemm_launch(a, lda, b, ldb, p, num_sms, false, static_cast<cudaStream_t>(stream));
}

// Elements (bf16) of scratch ka_gemm_split8 needs.
extern "C" size_t ka_gemm_split8_scratch_elems(int m, int n) { return static_cast<size_t>(ka::kTreeSlices) * m * n; }

// The same result as ka_gemm_tree8, for products of few tiles: the slices are units of their own, spread
// over all CTA pairs, their bf16 partials go to `scratch` ([8, m, n], 16-byte aligned; it stays in L2) and a
// second kernel sums them.
extern "C" int ka_gemm_split8(const void* a, long long lda, const void* b, long long ldb, int b_major, void* out,
                              const void* residual, void* scratch, int m, int n, int k, int* status, int num_sms,
                              unsigned long long timeout_ns, void* stream) {
  if (m <= 0 || n <= 0) return 0;
  if (n % 8 != 0) return -51;
  if (((reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(residual) | reinterpret_cast<uintptr_t>(scratch)) & 15u) != 0)
    return -54;
  ka::GemmParams p = {};
  p.m = m;
  p.n = n;
  p.k = k;
  p.b_major = b_major ? 1 : 0;
  p.epilogue = ka::kEpiStoreBf16;
  p.c = scratch;
  p.ldc = n;
  p.c_slice_stride = static_cast<long long>(m) * n;
  p.k_slices = ka::kTreeSlices;
  p.total_slices = ka::kTreeSlices;
  p.world = 1;
  p.status = status;
  p.timeout_ns = timeout_ns;
  const cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int rc = ka::gemm_launch(a, lda, b, ldb, p, num_sms, false, st);
  if (rc != 0) return rc;
  const long long vecs = p.c_slice_stride / 8;
  ka::slice_sum_kernel<<<static_cast<unsigned>((vecs + ka::kSumThreads - 1) / ka::kSumThreads), ka::kSumThreads, 0, st>>>(
      static_cast<const uint4*>(scratch), vecs, static_cast<const uint4*>(residual), static_cast<uint4*>(out));
  return cudaGetLastError() == cudaSuccess ? 0 : -11;
}

namespace ka {
namespace {

// d_logits from kept logits: the arithmetic of the kEpiLogitsGrad epilogue, so the bits are those of the
// recomputed ones. A stream: 4 bytes read and 2 written per logit.
constexpr int kGradThreads = 256, kGradVecs = 4;   // vectors of 8 columns per thread

__global__ void __launch_bounds__(kGradThreads)
kept_logits_grad_kernel(const float* __restrict__ logits, const long long* __restrict__ ids, const float* __restrict__ lse,
                        const float* __restrict__ g, __nv_bfloat16* __restrict__ out, int n, float scale) {
  const int row = blockIdx.y;
  const float s2 = scale * 1.4426950408889634f, neg_lse2 = __fmul_rn(-lse[row], 1.4426950408889634f);
  const float gs = __fmul_rn(g[row], scale);
  const long long tgt = ids[row];
  const float* src = logits + static_cast<long long>(row) * n;
  __nv_bfloat16* dst = out + static_cast<long long>(row) * n;
  const int c0 = (blockIdx.x * kGradThreads * kGradVecs + threadIdx.x) * 8;
  float4 a[kGradVecs], b[kGradVecs];
#pragma unroll
  for (int u = 0; u < kGradVecs; ++u) {
    const int c = c0 + u * kGradThreads * 8;
    if (c < n) {
      a[u] = __ldcs(reinterpret_cast<const float4*>(src + c));
      b[u] = __ldcs(reinterpret_cast<const float4*>(src + c + 4));
    }
  }
#pragma unroll
  for (int u = 0; u < kGradVecs; ++u) {
    const int c = c0 + u * kGradThreads * 8;
    if (c >= n) break;
    const float v[8] = {a[u].x, a[u].y, a[u].z, a[u].w, b[u].x, b[u].y, b[u].z, b[u].w};
    float d[8];
#pragma unroll
    for (int j = 0; j < 8; ++j)
      d[j] = __fmul_rn(gs, __fsub_rn(c + j == tgt ? 1.f : 0.f, ex2_approx(__fmaf_rn(v[j], s2, neg_lse2))));
    *reinterpret_cast<uint4*>(dst + c) = make_uint4(pack_bf16(d[0], d[1]), pack_bf16(d[2], d[3]), pack_bf16(d[4], d[5]),
                                                    pack_bf16(d[6], d[7]));
  }
}

}  // namespace
}  // namespace ka

// d_logits [m, n] bf16 from logits [m, n] fp32 that ka_lmhead_logp_forward_keep wrote; n % 8 == 0, 16-byte aligned.
extern "C" int ka_lmhead_kept_logits_grad(const float* logits, const long long* ids, const float* lse, const float* g,
                                          void* d_logits, int m, int n, float scale, void* stream) {
  if (m <= 0 || n <= 0) return 0;
  if (n % 8 != 0 || m > 65535 || ((reinterpret_cast<uintptr_t>(logits) | reinterpret_cast<uintptr_t>(d_logits)) & 15u) != 0)
    return -1;
  constexpr int per = ka::kGradThreads * ka::kGradVecs * 8;
  ka::kept_logits_grad_kernel<<<dim3((n + per - 1) / per, m), ka::kGradThreads, 0, static_cast<cudaStream_t>(stream)>>>(
      logits, ids, lse, g, static_cast<__nv_bfloat16*>(d_logits), n, scale);
  return cudaGetLastError() == cudaSuccess ? 0 : -11;
}

extern "C" int ka_lmhead_logits_grad(const void* hidden, const void* weight, const long long* ids, const float* lse,
                                     const float* g, void* d_logits, long long ldd, int m, int n, int k, float scale,
                                     int col_offset, int* status, int num_sms, unsigned long long timeout_ns,
                                     void* stream) {
  ka::GemmParams p = {};
  p.m = m;
  p.n = n;
  p.k = k;
  p.epilogue = ka::kEpiLogitsGrad;
  p.c = d_logits;
  p.ldc = ldd;
  p.k_slices = 1;
  p.total_slices = 1;
  p.world = 1;
  p.row_lse = lse;
  p.row_g = g;
  p.row_ids = ids;
  p.scale = scale;
  p.col_offset = col_offset;
  p.status = status;
  p.timeout_ns = timeout_ns;
  return ka::gemm_launch(hidden, k, weight, k, p, num_sms, false, static_cast<cudaStream_t>(stream));
}
