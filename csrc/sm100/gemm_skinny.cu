// Skinny bf16 GEMM for decode-sized batches on sm_100a: C[M, N] = A[M, K] * W[N, K]^T with
// M <= 64 (one new token per sequence), bitwise equal to the tiled kernel of gemm.cu.
//
// With a handful of rows the product is a stream of the weight matrix, so the operands are
// swapped: the WEIGHTS are the 128-row A operand of tcgen05.mma and the activations the narrow
// B operand (N = the batch padded to 16 / 32 / 64), D^T[n, m] accumulating in TMEM. An output
// element is one accumulation chain over K (no split-K: the order of the sum over K is the one
// the tiled kernel uses, so a row's result does not depend on which of the two kernels its batch
// size selects).
//
// What bounds it is the weight stream, and an SM pulls at most about 80 GB/s, so every SM has
// to have its share of the rows: the N rows are cut into tiles of R rows (R a multiple of 8, at
// most 128) such that the tiles fill the SMs evenly, N = 4096 into 128 tiles of 32 rows instead
// of 32 tiles of 128. The MMA reads 64 or 128 rows of shared memory (M = 64 for tiles of at most
// 64 rows); what lies behind a shorter tile (the next stage, or slack at the end) only reaches
// accumulator rows that nobody stores. M = 64 matters because those reads share the shared-memory
// port with the arriving tiles: 39 cycles per MMA at M = 128, N = 16, 23 at M = 64, and N = 4096,
// K = 14336 took 32.6 us with M = 128, 27.1 us with M = 64.
// A CTA walks its tiles persistently; the ring of K blocks (128 to 512 columns, see launch) runs on across
// tiles and the accumulator is double-buffered.
// Measured, 8 rows (64 rows): the four products of a Llama-3-8B decoder layer (436 MB of weights)
// take 83 us (98 us), 90 us (102 us) with K blocks of 128 columns throughout; with 128 weight rows per CTA
// everywhere they took 157 us (164 us).
//
// The reference has no GEMM of its own (it names backends in rl_engine/kernels/registry.py:41-55).
#include <cstdint>
#include <cuda_bf16.h>

#include "common/bounded_wait.cuh"
#include "common/ptx.cuh"
#include "common/tmap.cuh"

namespace ka {
namespace {

constexpr int kMaxRows = 128;  // largest M of the MMA (rows of shared memory it reads per K step)
constexpr int kBox = 64;       // K columns of a TMA box: one 128-byte swizzled row
constexpr int kThreads = 192;  // four epilogue warps, one TMA warp, one MMA warp
constexpr int kMaxStages = 32;
constexpr int kRingBytes = 192 * 1024;
constexpr int kSmemBytes = kRingBytes + kMaxRows * kBox * 2 + 2048;   // ring, slack behind it, control

struct Control {
  uint64_t full[kMaxStages];
  uint64_t empty[kMaxStages];
  uint64_t acc_full[2];
  uint64_t acc_empty[2];
  uint32_t tmem_base;
  int abort_flag;
};

struct SkinnyParams {
  __nv_bfloat16* out;   // [M, N], row stride ldc
  long long ldc;
  int m, n, k;
  int tile_rows, n_tiles, stages;
  bool joined;          // K is whole boxes: one copy per operand and stage
  int* status;
  unsigned long long timeout_ns;
};

__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
  return p != 0;
}

// NB: batch rows padded (the MMA's N); MR: weight rows of the MMA (its M); kBoxes: boxes per stage
template <int NB, int MR, int kBoxes>
__global__ void __launch_bounds__(kThreads, 1)
gemm_skinny_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_x,
                   const __grid_constant__ SkinnyParams p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = smem_u32(smem_raw);
  const uint32_t base = (raw_addr + 1023u) & ~1023u;
  uint8_t* smem = smem_raw + (base - raw_addr);
  Control* ctl = reinterpret_cast<Control*>(smem + kRingBytes + kMaxRows * kBox * 2);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int w_bytes = p.tile_rows * kBox * 2;                 // one box of the weight tile
  constexpr int kXBytes = NB * kBox * 2;
  const int box_bytes = w_bytes + kXBytes, stage_bytes = kBoxes * box_bytes;
  const int n_boxes = (p.k + kBox - 1) / kBox, num_kb = (n_boxes + kBoxes - 1) / kBoxes;
  constexpr int kTmemCols = 2 * NB < 32 ? 32 : 2 * NB;

  WaitCtx wctx{&ctl->abort_flag, p.status, p.timeout_ns};
  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(smem_u32(&ctl->full[s]), 1);
      mbar_init(smem_u32(&ctl->empty[s]), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(smem_u32(&ctl->acc_full[b]), 1);
      mbar_init(smem_u32(&ctl->acc_empty[b]), 4);
    }
    ctl->abort_flag = 0;
    fence_mbar_init_cluster();
  }
  if (warp == 5) {
    tmem_alloc<1>(smem_u32(&ctl->tmem_base), kTmemCols);
    tmem_relinquish<1>();
  }
  if (warp == 4 && lane == 0) {
    tma_prefetch_desc(&tm_w);
    tma_prefetch_desc(&tm_x);
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = ctl->tmem_base;

  if (warp == 4) {
    // ------------------------------------------------------------------ TMA producer
    if (elect_one()) {
      int s = 0;
      uint32_t phase = 1;
      bool ok = true;
      for (int t = blockIdx.x; t < p.n_tiles && ok; t += gridDim.x) {
        for (int kb = 0; kb < num_kb; ++kb) {
          ok = mbar_wait_bounded(smem_u32(&ctl->empty[s]), phase, wctx, 61, s);
          if (!ok) break;
          const uint32_t full = smem_u32(&ctl->full[s]);
          const uint32_t dst = base + s * stage_bytes;
          const int boxes = min(kBoxes, n_boxes - kb * kBoxes);
          if (p.joined) {
            // boxes behind the last one are filled with zeros and counted like the others
            mbar_arrive_expect_tx(full, kBoxes * box_bytes);
            tma_load_3d(dst, &tm_w, 0, t * p.tile_rows, kb * kBoxes, full);
            tma_load_3d(dst + kBoxes * w_bytes, &tm_x, 0, 0, kb * kBoxes, full);
          } else {
            mbar_arrive_expect_tx(full, boxes * box_bytes);
            for (int x = 0; x < boxes; ++x) {
              const int k0 = (kb * kBoxes + x) * kBox;
              tma_load_2d(dst + x * w_bytes, &tm_w, k0, t * p.tile_rows, full);
              tma_load_2d(dst + kBoxes * w_bytes + x * kXBytes, &tm_x, k0, 0, full);
            }
          }
          if (++s == p.stages) {
            s = 0;
            phase ^= 1u;
          }
        }
      }
    }
  } else if (warp == 5) {
    // ------------------------------------------------------------------ MMA issuer
    if (elect_one()) {
      constexpr uint32_t idesc = umma_idesc_bf16_f32(MR, NB);
      const uint64_t d0 = umma_desc_k_sw128(base);
      int s = 0, i = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < p.n_tiles && ok; t += gridDim.x, ++i) {
        const int b = i & 1;
        ok = mbar_wait_bounded(smem_u32(&ctl->acc_empty[b]), ((i >> 1) & 1) ^ 1u, wctx, 64, i);
        if (!ok) break;
        tc_fence_after_sync();
        const uint32_t acc = tmem_base + static_cast<uint32_t>(b * NB);
        for (int kb = 0; kb < num_kb; ++kb) {
          ok = mbar_wait_bounded(smem_u32(&ctl->full[s]), phase, wctx, 62, s);
          if (!ok) break;
          tc_fence_after_sync();
          const uint64_t dw = d0 + static_cast<uint64_t>((s * stage_bytes) >> 4);
          const uint64_t dx = dw + static_cast<uint64_t>((kBoxes * w_bytes) >> 4);
          const int boxes = min(kBoxes, n_boxes - kb * kBoxes);
#pragma unroll
          for (int x = 0; x < kBoxes; ++x) {
            if (x >= boxes) break;
#pragma unroll
            for (int k = 0; k < kBox / 16; ++k)
              umma_bf16<1>(acc, dw + static_cast<uint64_t>((x * w_bytes) >> 4) + k * 2,
                           dx + static_cast<uint64_t>((x * kXBytes) >> 4) + k * 2, idesc,
                           (kb > 0 || x > 0 || k > 0) ? 1u : 0u);
          }
          umma_commit<1>(smem_u32(&ctl->empty[s]));
          if (++s == p.stages) {
            s = 0;
            phase ^= 1u;
          }
        }
        if (ok) umma_commit<1>(smem_u32(&ctl->acc_full[b]));
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue
    // TMEM column = batch row m. TMEM lane = weight row (output column n); with M = 64 the rows
    // 16 w .. 16 w + 15 sit in the first half of warp w's 32 lanes.
    constexpr int kWarpRows = MR / 4;
    int i = 0;
    for (int t = blockIdx.x; t < p.n_tiles; t += gridDim.x, ++i) {
      const int b = i & 1;
      const bool mine = mbar_wait_bounded(smem_u32(&ctl->acc_full[b]), (i >> 1) & 1, wctx, 63, i);
      if (__all_sync(0xffffffffu, mine) == 0) break;
      tc_fence_after_sync();
      const int r = warp * kWarpRows + lane, n = t * p.tile_rows + r;
      const bool row_ok = lane < kWarpRows && r < p.tile_rows && n < p.n;
      const uint32_t taddr = tmem_base + static_cast<uint32_t>(b * NB) + (static_cast<uint32_t>(warp * 32) << 16);
      if (warp * kWarpRows < p.tile_rows) {
#pragma unroll
        for (int c0 = 0; c0 < NB; c0 += 16) {
          if (c0 >= p.m) break;
          uint32_t v[16];
          __syncwarp();
          tmem_ld_32x16(taddr + c0, v);
          // the wait names the registers, so that no use of them moves in front of it
          asm volatile("tcgen05.wait::ld.sync.aligned;"
                       : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7]),
                         "+r"(v[8]), "+r"(v[9]), "+r"(v[10]), "+r"(v[11]), "+r"(v[12]), "+r"(v[13]), "+r"(v[14]),
                         "+r"(v[15])
                       :
                       : "memory");
          if (row_ok) {
#pragma unroll
            for (int j = 0; j < 16; ++j)
              if (c0 + j < p.m)
                p.out[static_cast<long long>(c0 + j) * p.ldc + n] = __float2bfloat16_rn(__uint_as_float(v[j]));
          }
        }
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&ctl->acc_empty[b]));
    }
  }

  if (ctl->abort_flag) drain_in_flight();
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 5) {
    __syncwarp();
    tc_fence_after_sync();
    tmem_dealloc<1>(tmem_base, kTmemCols);
  }
}

template <int NB, int MR, int kBoxes>
int launch_boxes(const void* a, long long lda, const void* w, long long ldw, SkinnyParams p, int sms, cudaStream_t stream) {
  if (cudaFuncSetAttribute(gemm_skinny_kernel<NB, MR, kBoxes>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes) !=
      cudaSuccess)
    return -10;
  const int stage_bytes = kBoxes * (p.tile_rows + NB) * kBox * 2;
  p.stages = kRingBytes / stage_bytes < kMaxStages ? kRingBytes / stage_bytes : kMaxStages;
  CUtensorMap tw, tx;
  p.joined = p.k % kBox == 0 && p.k >= kBoxes * kBox;   // K = 64: nobody waits for a box of zeros (0.1 us of 3.9, 64 rows)
  auto map = [&](CUtensorMap* t, const void* base, int rows, long long ld, int box_rows) {
    return p.joined ? make_tmap_3d_16bit_sw128(t, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, base, static_cast<uint64_t>(rows),
                                               static_cast<uint64_t>(p.k), ld, static_cast<uint32_t>(box_rows), kBoxes)
                    : make_tmap_2d_16bit_sw128(t, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, base, static_cast<uint64_t>(rows),
                                               static_cast<uint64_t>(p.k), ld, static_cast<uint32_t>(box_rows), kBox);
  };
  int rc = map(&tw, w, p.n, ldw, p.tile_rows);
  if (rc) return -20 + rc;
  rc = map(&tx, a, p.m, lda, NB);
  if (rc) return -40 + rc;
  const unsigned grid = static_cast<unsigned>(p.n_tiles < sms ? p.n_tiles : sms);
  gemm_skinny_kernel<NB, MR, kBoxes><<<grid, kThreads, kSmemBytes, stream>>>(tw, tx, p);
  return cudaGetLastError() == cudaSuccess ? 0 : -11;
}

// Boxes per stage: the most that leave four stages in the ring and that K fills. A stage costs the MMA warp about
// 220 cycles on top of its MMAs (27 cycles each for 16 batch rows: 8 rows x 1184 columns, K = 4096, where only the
// chain of MMAs counts, takes 10.6 us with two boxes, 8.9 with four, 8.2 with eight), but with fewer than four
// stages the loads no longer keep ahead. us, boxes 2 / 4 / 8: 8 rows, 4096 columns, K = 14336 28.1 / 23.5 / 22.9, K = 4096
// 10.8 / 9.8 / 9.4; 6144 columns 12.3 / 11.6 / 11.7; 28672 columns 39.9 / 39.5 / 51.9 (six, three and one stage);
// 64 rows, 4096 columns, K = 14336 32.4 / 29.5 / 36.7; 6144 columns 14.2 / 14.5 / 20.8.
template <int NB, int MR>
int launch(const void* a, long long lda, const void* w, long long ldw, SkinnyParams p, int sms, cudaStream_t stream) {
  const int bytes = (p.tile_rows + NB) * kBox * 2;
  auto fits = [&](int boxes) { return 4 * boxes * bytes <= kRingBytes && boxes * kBox <= p.k; };
  if (fits(8)) return launch_boxes<NB, MR, 8>(a, lda, w, ldw, p, sms, stream);
  if (fits(4)) return launch_boxes<NB, MR, 4>(a, lda, w, ldw, p, sms, stream);
  return launch_boxes<NB, MR, 2>(a, lda, w, ldw, p, sms, stream);
}

}  // namespace
}  // namespace ka

// out[M, N] (bf16, row stride ldc) = a[M, K] (row stride lda) times w[N, K]^T (row stride ldw),
// for 1 <= M <= 64. Strides in elements, multiples of 8; pointers 16-byte aligned.
extern "C" int ka_gemm_skinny_bf16(const void* a, long long lda, const void* w, long long ldw, void* out,
                                   long long ldc, int m, int n, int k, int* status,
                                   unsigned long long timeout_ns, void* stream) {
  using namespace ka;
  if (m <= 0 || n <= 0) return 0;
  if (m > 64 || k <= 0) return -1;
  SkinnyParams p = {};
  p.out = static_cast<__nv_bfloat16*>(out);
  p.ldc = ldc;
  p.m = m;
  p.n = n;
  p.k = k;
  p.status = status;
  p.timeout_ns = timeout_ns;
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0)
    return -12;
  // Rows per tile: as many tiles as SMs, or a whole multiple of that when a tile would exceed the
  // MMA's 128 rows, rounded up to the 8 rows of a swizzle atom.
  const int rounds = (p.n + sms * kMaxRows - 1) / (sms * kMaxRows);
  const int per = (p.n + sms * rounds - 1) / (sms * rounds);
  p.tile_rows = (per + 7) / 8 * 8;
  p.n_tiles = (p.n + p.tile_rows - 1) / p.tile_rows;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (p.tile_rows <= 64) {
    if (m <= 16) return launch<16, 64>(a, lda, w, ldw, p, sms, st);
    if (m <= 32) return launch<32, 64>(a, lda, w, ldw, p, sms, st);
    return launch<64, 64>(a, lda, w, ldw, p, sms, st);
  }
  if (m <= 16) return launch<16, 128>(a, lda, w, ldw, p, sms, st);
  if (m <= 32) return launch<32, 128>(a, lda, w, ldw, p, sms, st);
  return launch<64, 128>(a, lda, w, ldw, p, sms, st);
}
