// Fused temperature / top-k / top-p token sampling for sm_100a: one CTA per row, one launch
// per call, the logits row is read once from HBM (later passes hit L2).
//
// Semantics (the order the reference gets from FlashInfer's default "top_k_first",
// rl_engine/kernels/sampling.py:61-64, with the temperature applied once):
//   1. y = logits / temperature
//   2. keep the k largest y; ties at the k-th value are kept in increasing token-id order
//   3. softmax over the survivors, sorted by (y descending, token id ascending); keep token i
//      while the probability mass of the tokens before it is <= top_p
//   4. draw u from Philox4x32-10 keyed by (seed, row id, step) and invert the CDF
// Probability masses are 32.32 fixed-point integers (csrc/common/detmath.h), so every sum is
// exact and order-free: the token depends only on (row contents, seed, row id, step), not on
// the batch size, the launch shape or the schedule, and the C++ CPU path reproduces it bit
// for bit.
//
// Four kernels:
//   sample_topk_kernel     top_k in [1, 1024] (greedy = top_k 1), optional top_p
//   sample_topk_held_kernel  the same for 16-bit rows that 1, 2 or 4 CTAs hold in registers
//                          (a cluster; candidates exchanged through distributed shared memory)
//   sample_general_kernel  no top_k (or k > 1024), optional top_p: 16-bit rows by one histogram of
//                          counts per key (sample_row16), fp32 rows and the few 16-bit rows that
//                          does not take by radix descent on (count, mass) histograms
//   sample_parts_kernel    the same for bf16 rows with a filter where part_ctas says so: a histogram for every
//                          part of the row, one to eight CTAs per row
#include <cstdint>
#include <cstdlib>
#include <type_traits>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "../common/detmath.h"
#include "common/launch.cuh"
#include "sampling.h"

namespace ka {
namespace {

constexpr int kThreads = 1024;
constexpr int kWarps = kThreads / 32;
constexpr int kCandCap = 10240;
constexpr int kMaxTopK = 1024;

// `wmax` / `any_ge` work on a 32-bit register word as it was loaded (two 16-bit floats or one fp32):
// a NaN loses against every number, fails every comparison and -0 counts as +0 in a comparison.
template <typename T>
struct Elem;
template <>
struct Elem<float> {
  static constexpr int kVec = 4;
  static constexpr int kLowBit = 0;
  static constexpr bool kPacked = false;
  static constexpr uint32_t kInf2 = 0;
  __device__ static float to_float(float v) { return v; }
  __device__ static uint32_t wmax(uint32_t a, uint32_t b) {
    return __float_as_uint(fmaxf(__uint_as_float(a), __uint_as_float(b)));
  }
  static __device__ bool any_ge(uint32_t a, uint32_t b) { return __uint_as_float(a) >= __uint_as_float(b); }
};
template <>
struct Elem<__nv_bfloat16> {
  static constexpr int kVec = 8;
  static constexpr int kLowBit = 16;
  static constexpr bool kPacked = true;
  static constexpr uint32_t kInf2 = 0x7F807F80u;  // +inf bit pattern, twice
  __device__ static float to_float(__nv_bfloat16 v) { return __bfloat162float(v); }
  __device__ static uint32_t wmax(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("max.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
  }
  static __device__ bool any_ge(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("{\n\t.reg .pred p, q;\n\tsetp.ge.bf16x2 p|q, %1, %2;\n\tor.pred p, p, q;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(d)
        : "r"(a), "r"(b));
    return d != 0;
  }
};
template <>
struct Elem<__half> {
  static constexpr int kVec = 8;
  static constexpr int kLowBit = 13;
  static constexpr bool kPacked = true;
  static constexpr uint32_t kInf2 = 0x7C007C00u;
  __device__ static float to_float(__half v) { return __half2float(v); }
  __device__ static uint32_t wmax(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("max.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
  }
  static __device__ bool any_ge(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("{\n\t.reg .pred p, q;\n\tsetp.ge.f16x2 p|q, %1, %2;\n\tor.pred p, p, q;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(d)
        : "r"(a), "r"(b));
    return d != 0;
  }
};

template <typename T>
__device__ __forceinline__ uint32_t vec_max(const uint4& r) {
  return Elem<T>::wmax(Elem<T>::wmax(r.x, r.y), Elem<T>::wmax(r.z, r.w));
}

// Elements of a row in front of its first 16-byte boundary (rows of an odd width start anywhere).
template <typename T>
__device__ __forceinline__ int row_head(const T* rp, int v) {
  const int bytes = static_cast<int>((16u - (reinterpret_cast<uintptr_t>(rp) & 15u)) & 15u);
  return min(v, bytes / static_cast<int>(sizeof(T)));
}

// Visit every element of a row once, in any order: scalars up to the first 16-byte boundary and
// behind the last, vectors between, four of them in flight per thread (a single CTA that walks a row
// is bound by the latency of its loads).
template <typename T, typename F>
__device__ __forceinline__ void for_each_key(const T* __restrict__ row, int v, F&& f) {
  constexpr int kVec = Elem<T>::kVec;
  const int tid = threadIdx.x, stride = blockDim.x;
  const int head = row_head(row, v), nvec = (v - head) / kVec, scal = v - nvec * kVec;
  const uint4* p = reinterpret_cast<const uint4*>(row + head);
  int i = tid;
  for (; i + 3 * stride < nvec; i += 4 * stride) {
    uint4 raw[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) raw[u] = p[i + u * stride];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const T* e = reinterpret_cast<const T*>(&raw[u]);
#pragma unroll
      for (int j = 0; j < kVec; ++j) f(float_to_key(Elem<T>::to_float(e[j])), head + (i + u * stride) * kVec + j);
    }
  }
  for (; i < nvec; i += stride) {
    const uint4 raw = p[i];
    const T* e = reinterpret_cast<const T*>(&raw);
#pragma unroll
    for (int j = 0; j < kVec; ++j) f(float_to_key(Elem<T>::to_float(e[j])), head + i * kVec + j);
  }
  for (int k = tid; k < scal; k += stride) {
    const int idx = k < head ? k : nvec * kVec + k;
    f(float_to_key(Elem<T>::to_float(row[idx])), idx);
  }
}

__device__ __forceinline__ int block_sum_int(int v, int* s_warp) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();
  if (lane == 0) s_warp[warp] = v;
  __syncthreads();
  int t = (lane < static_cast<int>(blockDim.x >> 5)) ? s_warp[lane] : 0;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  return t;
}

// Exclusive prefix sum over the block in thread order; `total` receives the block sum.
__device__ __forceinline__ unsigned long long block_exscan_u64(unsigned long long v, unsigned long long* s_warp,
                                                             unsigned long long& total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned long long inc = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long n = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += n;
  }
  __syncthreads();
  if (lane == 31) s_warp[warp] = inc;
  __syncthreads();
  unsigned long long w = (lane < static_cast<int>(blockDim.x >> 5)) ? s_warp[lane] : 0ull;
  unsigned long long winc = w;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long n = __shfl_up_sync(0xffffffffu, winc, o);
    if (lane >= o) winc += n;
  }
  total = __shfl_sync(0xffffffffu, winc, 31);
  const unsigned long long warp_off = __shfl_sync(0xffffffffu, winc - w, warp);
  return warp_off + inc - v;
}

constexpr int kWarpTops = 128;    // keys that the warps of a block bring to the search for a small k

struct TopkSmem {
  unsigned long long cand[kCandCap];          // key in the high word, ~token id in the low: descending = sorted order
  unsigned long long sorted[kMaxTopK];
  unsigned long long mass[kMaxTopK];
  unsigned long long scan[kWarps];
  unsigned long long kept_mass;
  unsigned int hits[2][kWarps];
  unsigned int top[kWarpTops];                // the largest keys of every warp
  unsigned int bound;
  int red[kWarps];
  int count;
  int n_sorted;
  int n_ties;
  int keep;
  int pick;
};

__device__ __forceinline__ unsigned long long cand_of(uint32_t key, int idx) {
  return (static_cast<unsigned long long>(key) << 32) | (~static_cast<uint32_t>(idx));
}

// Block totals of three counts, packed by thread in fields of 10 bits that a warp's sum must fit; a total
// is at most 65535. One barrier: `hits` alternates between two rows, and the row is read before the next
// call's barrier.
__device__ __forceinline__ void block_count3(uint32_t packed, unsigned int (&hits)[2][kWarps], int parity, int& c1, int& c2,
                                             int& c3) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  packed = __reduce_add_sync(0xffffffffu, packed);
  if (lane == 0) hits[parity][warp] = packed;
  __syncthreads();
  const uint32_t w = lane < static_cast<int>(blockDim.x >> 5) ? hits[parity][lane] : 0u;
  const uint32_t a = __reduce_add_sync(0xffffffffu, (w & 1023u) | (((w >> 10) & 1023u) << 16));
  c3 = static_cast<int>(__reduce_add_sync(0xffffffffu, w >> 20));
  c1 = static_cast<int>(a & 0xFFFFu);
  c2 = static_cast<int>(a >> 16);
}

// Final step of the top-k path for at most 64 survivors, run by one warp: lane l holds the masses q0, q1
// of the survivors 2 l and 2 l + 1 in sorted order; apply top-p, draw, return the position picked. All
// sums are integers, so the warp-parallel prefix sums give exactly the result of a serial walk.
__device__ __forceinline__ int pick_sorted_warp(unsigned long long q0, unsigned long long q1, int n, float top_p,
                                                uint32_t u24) {
  const int lane = threadIdx.x & 31, i = 2 * lane;
  unsigned long long inc = q0 + q1;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long t = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += t;
  }
  const unsigned long long z = __shfl_sync(0xffffffffu, inc, 31);
  const unsigned long long mid = inc - q1, before = mid - q0;
  // position of the first survivor for which a (the even one of a lane) or b (the odd one) holds, else n
  auto first_of = [&](bool a, bool b) {
    const uint32_t ma = __ballot_sync(0xffffffffu, a), mb = __ballot_sync(0xffffffffu, b);
    if ((ma | mb) == 0) return n;
    const int l = __ffs(static_cast<int>(ma | mb)) - 1;
    return 2 * l + ((ma >> l) & 1u ? 0 : 1);
  };
  int keep = n;
  unsigned long long zk = z;
  if (top_p < 1.0f) {
    // keep = first i > 0 with (mass before i) > limit, else n
    const unsigned long long limit = mass_fraction(static_cast<double>(top_p), z);
    keep = first_of(i > 0 && i < n && before > limit, i + 1 < n && mid > limit);
    zk = __shfl_sync(0xffffffffu, (keep & 1) ? mid : inc, (keep - 1) >> 1);
  }
  const unsigned long long target = mass_scale_u24(u24, zk);
  const int pick = first_of(i < keep && mid > target, i + 1 < keep && inc > target);
  return pick < keep ? pick : keep - 1;
}

// Bits that a search among keys between lo and hi has to decide, rounded up to pairs.
__device__ __forceinline__ int open_bits(uint32_t lo, uint32_t hi) { return (33 - __clz(static_cast<int>(lo ^ hi))) & ~1; }
__device__ __forceinline__ uint32_t above_bits(uint32_t key, int bits) { return bits >= 32 ? 0u : key >> bits << bits; }

// The largest key that at least kk of the block's keys reach (0 if there are fewer above 0), two bits per
// step; bits that all keys share need no step. A thread brings NW words: two 16-bit keys each, or one key
// of 32 bits.
template <int NW, int kBits>
__device__ __forceinline__ uint32_t kth_key(const uint32_t (&w)[NW], int kk, unsigned int (&hits)[2][kWarps]) {
  uint32_t top = 0, bottom = ~0u;
#pragma unroll
  for (int i = 0; i < NW; ++i) {
    if constexpr (kBits == 16) {
      top = max(top, max(w[i] >> 16, w[i] & 0xFFFFu));
      bottom = min(bottom, min(w[i] >> 16, w[i] & 0xFFFFu));
    } else {
      top = max(top, w[i]);
      bottom = min(bottom, w[i]);
    }
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  top = __reduce_max_sync(0xffffffffu, top);
  bottom = __reduce_min_sync(0xffffffffu, bottom);
  if (lane == 0) {
    hits[0][warp] = top;
    hits[1][warp] = bottom;
  }
  __syncthreads();
  const bool in = lane < static_cast<int>(blockDim.x >> 5);
  top = __reduce_max_sync(0xffffffffu, in ? hits[0][lane] : 0u);
  bottom = __reduce_min_sync(0xffffffffu, in ? hits[1][lane] : ~0u);
  __syncthreads();
  const int bits = open_bits(bottom, top);
  uint32_t low = above_bits(top, bits);
#pragma unroll 1
  for (int shift = bits - 2, st = 0; shift >= 0; shift -= 2, ++st) {
    uint32_t packed = 0;
#pragma unroll
    for (uint32_t t = 1; t <= 3; ++t) {
      const uint32_t cand = low | (t << shift);
      uint32_t n = 0;
#pragma unroll
      for (int i = 0; i < NW; ++i) {
        if constexpr (kBits == 16)
          n += (w[i] >= (cand << 16) ? 1u : 0u) + ((w[i] << 16) >= (cand << 16) ? 1u : 0u);
        else
          n += w[i] >= cand ? 1u : 0u;
      }
      packed += n << (10 * (t - 1));
    }
    int c1, c2, c3;
    block_count3(packed, hits, st & 1, c1, c2, c3);
    low |= static_cast<uint32_t>(c3 >= kk ? 3 : (c2 >= kk ? 2 : (c1 >= kk ? 1 : 0))) << shift;
  }
  __syncthreads();
  return low;
}

// The same for kk <= 64 without a block-wide step per bit: the warps bring their largest keys, 128 in all,
// and one warp searches among those. They are keys of the block, so at least kk of the block's reach the
// result; it is the kk-th largest of all unless a warp holds more of those than it brings. With 1024 threads
// 2.4k cycles; a block-wide step per two bits took 7.3k.
template <int kBits, int kBlockWarps>
__device__ __forceinline__ uint32_t kth_of_warp_tops(uint32_t w, int kk, TopkSmem& s) {
  constexpr int kTops = kWarpTops / kBlockWarps;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t hi = w, lo = 0;
  if constexpr (kBits == 16) {
    hi = max(w >> 16, w & 0xFFFFu);
    lo = min(w >> 16, w & 0xFFFFu);
  }
  uint32_t mine = 0;
#pragma unroll
  for (int r = 0; r < kTops; ++r) {
    const uint32_t m = __reduce_max_sync(0xffffffffu, hi);
    const int owner = __ffs(static_cast<int>(__ballot_sync(0xffffffffu, hi == m))) - 1;
    if (lane == owner) {
      hi = lo;
      lo = 0;
    }
    if (lane == r) mine = m;
  }
  if (lane < kTops) s.top[warp * kTops + lane] = mine;
  __syncthreads();
  if (warp == 0) {
    uint32_t v[kWarpTops / 32], top = 0, bottom = ~0u;
#pragma unroll
    for (int i = 0; i < kWarpTops / 32; ++i) {
      v[i] = s.top[lane + 32 * i];
      top = max(top, v[i]);
      bottom = min(bottom, v[i]);
    }
    top = __reduce_max_sync(0xffffffffu, top);
    bottom = __reduce_min_sync(0xffffffffu, bottom);
    const int bits = open_bits(bottom, top);
    uint32_t low = above_bits(top, bits);
#pragma unroll 1
    for (int bit = bits - 1; bit >= 0; --bit) {
      const uint32_t cand = low | (1u << bit);
      uint32_t c = 0;
#pragma unroll
      for (int i = 0; i < kWarpTops / 32; ++i) c += v[i] >= cand ? 1u : 0u;
      if (__reduce_add_sync(0xffffffffu, c) >= static_cast<uint32_t>(kk)) low = cand;
    }
    if (lane == 0) s.bound = low;
  }
  __syncthreads();
  return s.bound;
}

// How a block finds the bound: from the keys that the warps bring (one word per thread), or by a search among
// all its maxima, one or four words per thread.
enum BoundFrom : int { kWarpKeys = 0, kOneWord = 1, kFourWords = 4 };
constexpr int words_of(int from) { return from == kFourWords ? 4 : 1; }

// A bound that at least kk of the keys in the block's words reach.
template <int kFrom, int kBits, int kBlockWarps>
__device__ __forceinline__ uint32_t bound_of(const uint32_t (&w)[words_of(kFrom)], int kk, TopkSmem& s) {
  if constexpr (kFrom == kWarpKeys)
    return kth_of_warp_tops<kBits, kBlockWarps>(w[0], kk, s);
  else
    return kth_key<words_of(kFrom), kBits>(w, kk, s.hits);
}

// The search of one word, out of line: for a path that is rarely taken (inline it costs the one-CTA cluster 0.3 us
// of 6.7, out of line it costs two CTAs 0.3 us of 9.1).
__device__ __noinline__ uint32_t kth_key16_far(uint32_t w, int kk, TopkSmem& s) {
  const uint32_t words[1] = {w};
  return kth_key<1, 16>(words, kk, s.hits);
}

// s.sorted[0 .. 1023] descending, by 256 threads that hold four neighbours each: partners at distance 1
// and 2 are in the same thread, up to 64 in the same warp (shuffles), farther ones go through shared memory.
// Run by all threads of the block.
__device__ __forceinline__ void sort_1024(TopkSmem& s) {
  constexpr int kT = 256, kE = 4;
  const int tid = threadIdx.x;
  if (tid < kT) {
    unsigned long long v[kE];
#pragma unroll
    for (int r = 0; r < kE; ++r) v[r] = s.sorted[tid * kE + r];
    auto swap_if = [](unsigned long long& a, unsigned long long& b, bool desc) {
      const bool sw = (a < b) == desc;
      const unsigned long long t = sw ? b : a;
      b = sw ? a : b;
      a = t;
    };
#pragma unroll 1
    for (int wb = 1; wb <= 10; ++wb) {
#pragma unroll 1
      for (int b = wb - 1; b >= 2; --b) {
        // this thread's elements are the upper or the lower partners together
        const bool upper = (tid * kE >> b) & 1, desc = ((tid * kE >> wb) & 1) == 0;
        unsigned long long o[kE];
        if (b >= 7) {
          asm volatile("bar.sync 1, 256;" ::: "memory");      // the partners have read what the last exchange left
#pragma unroll
          for (int r = 0; r < kE; ++r) s.sorted[tid * kE + r] = v[r];
          asm volatile("bar.sync 1, 256;" ::: "memory");
          const int partner = (tid * kE) ^ (1 << b);
#pragma unroll
          for (int r = 0; r < kE; ++r) o[r] = s.sorted[partner + r];
        } else {
#pragma unroll
          for (int r = 0; r < kE; ++r) o[r] = __shfl_xor_sync(0xffffffffu, v[r], 1 << (b - 2));
        }
#pragma unroll
        for (int r = 0; r < kE; ++r) {
          const bool larger = v[r] > o[r];
          v[r] = larger == (upper != desc) ? v[r] : o[r];
        }
      }
      const bool desc = ((tid * kE >> wb) & 1) == 0;
      if (wb >= 2) {
        swap_if(v[0], v[2], desc);
        swap_if(v[1], v[3], desc);
      }
      swap_if(v[0], v[1], wb == 1 ? true : desc);
      swap_if(v[2], v[3], wb == 1 ? false : desc);
    }
    asm volatile("bar.sync 1, 256;" ::: "memory");
#pragma unroll
    for (int r = 0; r < kE; ++r) s.sorted[tid * kE + r] = v[r];
  }
  __syncthreads();
}

constexpr int kTopkThreads = 512;

// Two 16-bit floats (bf16 or fp16 bit patterns) -> two order-preserving 16-bit keys; NaN -> 0.
template <typename T>
__device__ __forceinline__ uint32_t key16x2(uint32_t w) {
  const uint32_t nan = __vcmpgtu2(w & 0x7FFF7FFFu, Elem<T>::kInf2);
  const uint32_t sign = (w >> 15) & 0x00010001u;
  const uint32_t k = w ^ (sign * 0xFFFFu | 0x80008000u);
  return k & ~nan;
}

template <typename T>
__device__ __forceinline__ T from_bits16(uint32_t h) {
  const unsigned short us = static_cast<unsigned short>(h);
  return *reinterpret_cast<const T*>(&us);
}

// k up to which the bound may come from what the warps bring (bound_from has the rule)
constexpr int kFewK = 64;
// Candidates that are ranked by counting, from more the k largest are searched first: eight steps over 16-bit keys,
// sixteen over 32-bit ones, so the line lies higher there. On the GPU, us, counting / search: bf16, 500 candidates, 200
// rows, k = 200: 26.0 / 15.9; 64 rows of 128256 columns, k = 200: 20.6 / 18.1; 8 rows of 8000, k = 400:
// 17.9 / 16.9; fp32, 8 rows of 16000, k = 200: 12.6 / 14.4, k = 400 18.8 / 20.8; 200 rows
// of 500, k = 200 (500): 27.0 / 20.0.
template <typename T>
constexpr int kRankSort = Elem<T>::kPacked ? 256 : 480;

// Key of an element given as the low bits of a register word.
template <typename T>
__device__ __forceinline__ uint32_t key_of_bits(uint32_t bits) {
  if constexpr (Elem<T>::kPacked)
    return float_to_key(Elem<T>::to_float(from_bits16<T>(bits & 0xFFFFu)));
  else
    return float_to_key(__uint_as_float(bits));
}

// A bound on keys in the two forms the collection uses: `thr` (the same number, in every half of a word) for
// a quick look at a vector's maximum, `low` for the exact comparison of a 32-bit key. A bound below -inf's
// key means that NaNs qualify as well, so the quick look must let everything through.
template <typename T>
struct Bound {
  uint32_t low, thr;
  bool all;
  __device__ __forceinline__ explicit Bound(uint32_t k) {   // k: the leading 16 bits of the key, or all 32
    if constexpr (Elem<T>::kPacked) {
      const uint32_t bits = (k & 0x8000u) ? (k & 0x7FFFu) : (~k & 0xFFFFu);
      thr = bits * 0x00010001u;
      all = k <= (~(Elem<T>::kInf2 | 0x8000u) & 0xFFFFu);
      low = all && k == 0 ? 0u : float_to_key(Elem<T>::to_float(from_bits16<T>(bits)));
    } else {
      thr = __float_as_uint(key_to_float(k));
      all = k <= ~0xFF800000u;
      low = k;
    }
  }
  __device__ __forceinline__ bool maybe(uint32_t word) const { return all || Elem<T>::any_ge(word, thr); }
};

// Keys of a thread's maxima, in place: two 16-bit keys per word, or one of 32 bits.
template <typename T, int NW>
__device__ __forceinline__ void words_to_keys(uint32_t (&w)[NW]) {
#pragma unroll
  for (int i = 0; i < NW; ++i) {
    if constexpr (Elem<T>::kPacked)
      w[i] = key16x2<T>(w[i]);
    else
      w[i] = float_to_key(__uint_as_float(w[i]));
  }
}

// Calls f(key, idx) for the elements of `raw` that reach the bound; vector u's first element is token
// i0 + u * step, vectors from n on are left out. Hits are rare, so a thread first notes which of its vectors
// have one; the code behind that exists once and runs as often as the busiest lane has hits, not once per
// vector (straight-line code that runs once per launch costs instruction fetches). Returns false, with the
// visit cut short, once a vector takes the thread past `most` hits.
template <typename T, int N, typename F>
__device__ __forceinline__ bool visit_hits(const uint4 (&raw)[N], int n, int i0, int step, const Bound<T>& b, int most,
                                           F&& f) {
  constexpr int kVec = Elem<T>::kVec;
  uint32_t vecs = 0;
#pragma unroll
  for (int u = 0; u < N; ++u) vecs |= (u < n && b.maybe(vec_max<T>(raw[u])) ? 1u : 0u) << u;
  while (vecs) {
    const int u = __ffs(static_cast<int>(vecs)) - 1;
    vecs &= vecs - 1;
    uint4 r = raw[0];
#pragma unroll
    for (int x = 1; x < N; ++x) r = u == x ? raw[x] : r;
    const uint32_t w[4] = {r.x, r.y, r.z, r.w};
    uint32_t elems = 0;
#pragma unroll
    for (int j = 0; j < kVec; ++j)
      elems |= (key_of_bits<T>(Elem<T>::kPacked ? w[j / 2] >> (16 * (j & 1)) : w[j & 3]) >= b.low ? 1u : 0u) << j;
    most -= __popc(elems);
    if (most < 0) return false;
    while (elems) {
      const int j = __ffs(static_cast<int>(elems)) - 1;
      elems &= elems - 1;
      const int wi = Elem<T>::kPacked ? j >> 1 : j;
      const uint32_t word = wi == 0 ? w[0] : (wi == 1 ? w[1] : (wi == 2 ? w[2] : w[3]));
      f(key_of_bits<T>(Elem<T>::kPacked ? word >> (16 * (j & 1)) : word), i0 + u * step + j);
    }
  }
  return true;
}

// Second half of the top-k path, shared by the one-CTA and the cluster kernel: n_cand candidates
// sit in s.cand (in any order; if there are more than the buffer holds the row is searched
// exactly), the kk largest by (key desc, id asc) are the survivors; masses, top-p and the draw
// follow. Run by all threads of one CTA. Few candidates are ranked by counting; from many the kk
// largest are selected by a bit search and sorted by a bitonic network (counting grows with the square:
// the 2100 candidates of k = 1000 in two parts of a row took 300 us that way, 12 us now).
template <typename T>
__device__ __forceinline__ void topk_finish(TopkSmem& s, int n_cand, const T* __restrict__ rp, int v, int kk,
                                            float inv_temp, float top_p, uint32_t u24, int row, int* __restrict__ out) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nt = blockDim.x;
  constexpr int kLow = Elem<T>::kLowBit;
  if (n_cand > kCandCap) {
    // ---- rare: more ties / near-ties than the candidate buffer holds. Exact radix select by
    // counting passes, then an index-ordered pick among the ties at the threshold.
    uint32_t tau = 0;
    for (int bit = 31; bit >= kLow; --bit) {
      const uint32_t cand = tau | (1u << bit);
      int local = 0;
      for_each_key<T>(rp, v, [&](uint32_t key, int) { local += (key >= cand) ? 1 : 0; });
      if (block_sum_int(local, s.red) >= kk) tau = cand;
    }
    // the low bits of a widened 16-bit value's key are ones below zero (and 0 is NaN's key)
    if (tau != 0 && !(tau & 0x80000000u)) tau |= (1u << kLow) - 1u;
    int local_gt = 0;
    for_each_key<T>(rp, v, [&](uint32_t key, int) { local_gt += (key > tau) ? 1 : 0; });
    const int n_gt = block_sum_int(local_gt, s.red);
    const int quota = kk - n_gt;
    if (tid == 0) s.count = 0;
    __syncthreads();
    for_each_key<T>(rp, v, [&](uint32_t key, int i) {
      if (key > tau) s.cand[atomicAdd(&s.count, 1)] = cand_of(key, i);
    });
    __syncthreads();
    unsigned long long tie_base = 0;
    constexpr int kPer = 8;
    for (int base = 0; base < v && tie_base < static_cast<unsigned long long>(quota); base += nt * kPer) {
      const int i0 = base + tid * kPer;
      int mine = 0;
      for (int j = 0; j < kPer; ++j) {
        const int i = i0 + j;
        if (i < v && float_to_key(Elem<T>::to_float(rp[i])) == tau) ++mine;
      }
      unsigned long long total;
      unsigned long long off = tie_base + block_exscan_u64(static_cast<unsigned long long>(mine), s.scan, total);
      for (int j = 0; j < kPer; ++j) {
        const int i = i0 + j;
        if (i < v && float_to_key(Elem<T>::to_float(rp[i])) == tau) {
          if (off < static_cast<unsigned long long>(quota)) s.cand[n_gt + off] = cand_of(tau, i);
          ++off;
        }
      }
      tie_base += total;
    }
    __syncthreads();
    n_cand = kk;
  }

  // ---- the kk survivors, sorted by (key desc, id asc)
  if (n_cand <= kRankSort<T>) {
    // eight lanes count for one candidate
    for (int i0 = 0; i0 < n_cand; i0 += nt >> 3) {
      const int i = i0 + (tid >> 3);
      const unsigned long long mine = i < n_cand ? s.cand[i] : ~0ull;
      uint32_t rank = 0;
#pragma unroll 4
      for (int j = tid & 7; j < n_cand; j += 8) rank += s.cand[j] > mine ? 1u : 0u;
#pragma unroll
      for (int o = 1; o < 8; o <<= 1) rank += __shfl_xor_sync(0xffffffffu, rank, o);
      if ((tid & 7) == 0 && i < n_cand && rank < static_cast<uint32_t>(kk)) s.sorted[rank] = mine;
    }
    __syncthreads();
  } else {
    // the kk-th largest key (its leading bits name it), then the kk-th largest (key, ~id) among its ties;
    // a warp counts at most 32 * 20 candidates, which fits the fields of block_count3
    static_assert(kCandCap <= 20 * 512, "counts per warp");
    constexpr uint32_t kMask = ~((1u << (kLow & ~1)) - 1u);
    uint32_t top = 0, bottom = ~0u;
    for (int i = tid; i < n_cand; i += nt) {
      const uint32_t key = static_cast<uint32_t>(s.cand[i] >> 32);
      top = max(top, key);
      bottom = min(bottom, key);
    }
    top = __reduce_max_sync(0xffffffffu, top);
    bottom = __reduce_min_sync(0xffffffffu, bottom);
    if (lane == 0) {
      s.hits[0][warp] = top;
      s.hits[1][warp] = bottom;
    }
    if (tid == 0) s.n_sorted = s.n_ties = 0;
    __syncthreads();
    top = __reduce_max_sync(0xffffffffu, lane < nt >> 5 ? s.hits[0][lane] : 0u);
    bottom = __reduce_min_sync(0xffffffffu, lane < nt >> 5 ? s.hits[1][lane] : ~0u);
    __syncthreads();
    const int bits = open_bits(bottom, top);
    int c1, c2, c3, st = 0;
    uint32_t tau = above_bits(top, bits) & kMask;
    for (int bit = bits - 2; bit >= (kLow & ~1); bit -= 2, ++st) {
      uint32_t packed = 0;
      for (int i = tid; i < n_cand; i += nt) {
        const uint32_t key = static_cast<uint32_t>(s.cand[i] >> 32);
        packed += (key >= (tau | (1u << bit)) ? 1u : 0u) + (key >= (tau | (2u << bit)) ? 1u << 10 : 0u) +
                  (key >= (tau | (3u << bit)) ? 1u << 20 : 0u);
      }
      block_count3(packed, s.hits, st & 1, c1, c2, c3);
      tau |= static_cast<uint32_t>(c3 >= kk ? 3 : (c2 >= kk ? 2 : (c1 >= kk ? 1 : 0))) << bit;
    }
    // ---- what is above it survives, its ties go to a list of their own
    // (in s.mass, which is not in use yet) and are ranked by counting if they are few; a search for the last id
    // that survives takes the same time for any number of them (fp32, one row of 1000 columns of which one is not
    // -inf, k = 50: 69 us with a thousand ties ranked, 18 with the search)
    constexpr int kTieCap = 256;
    for (int i = tid; i < n_cand; i += nt) {
      const unsigned long long c = s.cand[i];
      const uint32_t key = static_cast<uint32_t>(c >> 32) & kMask;
      if (key > tau) s.sorted[atomicAdd(&s.n_sorted, 1)] = c;
      if (key == tau) {
        const int slot = atomicAdd(&s.n_ties, 1);
        if (slot < kTieCap) s.mass[slot] = c;
      }
    }
    __syncthreads();
    const int n_gt = s.n_sorted, n_ties = s.n_ties, quota = kk - n_gt;   // ties that survive: the smallest ids
    if (n_ties <= kTieCap) {
      for (int i = warp; i < n_ties; i += nt >> 5) {
        const unsigned long long mine = s.mass[i];
        uint32_t rank = 0;
        for (int j = lane; j < n_ties; j += 32) rank += s.mass[j] > mine ? 1u : 0u;
        rank = __reduce_add_sync(0xffffffffu, rank);
        if (lane == 0 && rank < static_cast<uint32_t>(quota)) s.sorted[n_gt + rank] = mine;
      }
    } else {
      uint32_t tie = 0;                          // the smallest ~id among those that survive
      const int top_bit = (31 - __clz(v)) & ~1;
      const uint32_t id_mask = top_bit == 30 ? ~0u : (4u << top_bit) - 1u;
      for (int bit = top_bit; bit >= 0; bit -= 2, ++st) {
        uint32_t packed = 0;
        for (int i = tid; i < n_cand; i += nt) {
          const unsigned long long c = s.cand[i];
          if ((static_cast<uint32_t>(c >> 32) & kMask) != tau) continue;
          const uint32_t id = static_cast<uint32_t>(c) & id_mask;
          packed += (id >= (tie | (1u << bit)) ? 1u : 0u) + (id >= (tie | (2u << bit)) ? 1u << 10 : 0u) +
                    (id >= (tie | (3u << bit)) ? 1u << 20 : 0u);
        }
        block_count3(packed, s.hits, st & 1, c1, c2, c3);
        tie |= static_cast<uint32_t>(c3 >= quota ? 3 : (c2 >= quota ? 2 : (c1 >= quota ? 1 : 0))) << bit;
      }
      tie |= ~id_mask;
      for (int i = tid; i < n_cand; i += nt) {
        const unsigned long long c = s.cand[i];
        if ((static_cast<uint32_t>(c >> 32) & kMask) == tau && static_cast<uint32_t>(c) >= tie)
          s.sorted[atomicAdd(&s.n_sorted, 1)] = c;
      }
    }
    if (kk <= nt >> 1) {
      // eight lanes count for up to four survivors, in place
      __syncthreads();
      const int group = tid >> 3, groups = nt >> 3;
      unsigned long long mine[4];
      uint32_t rank[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        mine[c] = group + c * groups < kk ? s.sorted[group + c * groups] : ~0ull;
        rank[c] = 0;
      }
      for (int j = tid & 7; j < kk; j += 8) {
        const unsigned long long other = s.sorted[j];
#pragma unroll
        for (int c = 0; c < 4; ++c) rank[c] += other > mine[c] ? 1u : 0u;
      }
#pragma unroll
      for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) rank[c] += __shfl_xor_sync(0xffffffffu, rank[c], o);
      __syncthreads();
#pragma unroll
      for (int c = 0; c < 4; ++c)
        if ((tid & 7) == 0 && group + c * groups < kk) s.sorted[rank[c]] = mine[c];
      __syncthreads();
    } else {
      for (int i = kk + tid; i < kMaxTopK; i += nt) s.sorted[i] = 0;   // sorts behind every candidate
      __syncthreads();
      sort_1024(s);
    }
  }

  // ---- masses, top-p, draw
  auto key_at = [&](int i) { return static_cast<uint32_t>(s.sorted[i] >> 32); };
  const float y0 = mul_rn(key_to_float(key_at(0)), inv_temp);
  auto mass_at = [&](int i) {
    return static_cast<unsigned long long>(mass_fixed(exp_det(sub_rn(mul_rn(key_to_float(key_at(i)), inv_temp), y0))));
  };
  int pos = 0;
  if (kk <= 64) {
    // one warp does it all
    if (warp != 0) return;
    const int i = 2 * lane;
    pos = pick_sorted_warp(i < kk ? mass_at(i) : 0ull, i + 1 < kk ? mass_at(i + 1) : 0ull, kk, top_p, u24);
  } else {
    // thread t owns the survivors [t * per, t * per + per), per is 1 or 2
    const int per = (kk + nt - 1) / nt, i0 = tid * per;
    const unsigned long long q0 = i0 < kk ? mass_at(i0) : 0ull, q1 = per == 2 && i0 + 1 < kk ? mass_at(i0 + 1) : 0ull;
    if (tid == 0) {
      s.keep = kk;
      s.pick = -1;
    }
    unsigned long long z;
    const unsigned long long before = block_exscan_u64(q0 + q1, s.scan, z);
    if (top_p < 1.0f) {
      // keep = first i > 0 with (mass before i) > limit
      const unsigned long long limit = mass_fraction(static_cast<double>(top_p), z);
      int first = kk;
      if (i0 > 0 && i0 < kk && before > limit)
        first = i0;
      else if (per == 2 && i0 + 1 < kk && before + q0 > limit)
        first = i0 + 1;
      first = __reduce_min_sync(0xffffffffu, first);
      if (lane == 0 && first < kk) atomicMin(&s.keep, first);
      __syncthreads();
    }
    const int keep = s.keep;
    if (i0 < keep && i0 + per >= keep) s.kept_mass = before + q0 + (i0 + 1 < keep ? q1 : 0ull);
    __syncthreads();
    const unsigned long long target = mass_scale_u24(u24, s.kept_mass);
    if (i0 < keep && before <= target && before + q0 > target)
      s.pick = i0;
    else if (per == 2 && i0 + 1 < keep && before + q0 <= target && before + q0 + q1 > target)
      s.pick = i0 + 1;
    __syncthreads();
    pos = s.pick < 0 ? keep - 1 : s.pick;
  }
  if (tid == 0) out[row] = static_cast<int>(~static_cast<uint32_t>(s.sorted[pos]));
}

// One CTA per row, two passes: the first (HBM) finds a bound that at least kk elements reach, the second (L2)
// collects the elements that do. Each thread keeps the largest elements of NW groups of the row in NW words
// as they were loaded (packed maxima: one instruction per two 16-bit elements); the kk-th largest of the
// block's maxima bounds the kk-th largest element from below. Bound by the two passes: bf16 [256, 128256],
// k = 50, 33 us (49 us with the keys of all elements computed); fp32 [256, 128256] 66 us (70 us), 128255
// columns 76 us (255 us when rows off a 16-byte boundary were read by scalars).
template <typename T, int kFrom>
__global__ void __launch_bounds__(kTopkThreads, 2)
sample_topk_kernel(const T* __restrict__ logits, long long row_stride, int v, const long long* __restrict__ row_ids,
                   float inv_temp, int top_k, float top_p, unsigned long long seed, unsigned long long step,
                   int* __restrict__ out) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  TopkSmem& s = *reinterpret_cast<TopkSmem*>(smem_raw);
  constexpr int kVec = Elem<T>::kVec, nt = kTopkThreads, NW = words_of(kFrom);
  constexpr int kU = 8;                       // 16-byte loads in flight per thread
  static_assert(kU % NW == 0, "every word gets its share of a batch");
  const int tid = threadIdx.x;
  const int row = blockIdx.x;
  const T* rp = logits + static_cast<long long>(row) * row_stride;
  const int kk = min(min(top_k, kMaxTopK), v);
  const int head = row_head(rp, v), nvec = (v - head) / kVec, scal = v - nvec * kVec;
  const uint4* vp = reinterpret_cast<const uint4*>(rp + head);
  const int scal_idx = tid < head ? tid : nvec * kVec + tid;     // thread's scalar element, if tid < scal
  uint32_t scal_word = ~0u;                                      // NaN
  if (tid < scal) {
    if constexpr (Elem<T>::kPacked)
      scal_word = 0xFFFF0000u | reinterpret_cast<const unsigned short*>(rp)[scal_idx];
    else
      scal_word = __float_as_uint(rp[scal_idx]);
  }
  if (tid == 0) s.count = 0;
  uint32_t mx[NW];
#pragma unroll
  for (int i = 0; i < NW; ++i) mx[i] = ~0u;
  mx[0] = scal_word;
  for (int i = tid; i < nvec; i += kU * nt) {
    uint4 raw[kU];
#pragma unroll
    for (int u = 0; u < kU; ++u) raw[u] = i + u * nt < nvec ? __ldg(vp + i + u * nt) : make_uint4(~0u, ~0u, ~0u, ~0u);
#pragma unroll
    for (int u = 0; u < kU; ++u) mx[u % NW] = Elem<T>::wmax(mx[u % NW], vec_max<T>(raw[u]));
  }
  const unsigned long long rid = row_ids ? static_cast<unsigned long long>(row_ids[row])
                                         : static_cast<unsigned long long>(row);
  const uint32_t u24 = uniform_u24(seed, rid, step);
  words_to_keys<T>(mx);
  const Bound<T> bound(bound_of<kFrom, Elem<T>::kPacked ? 16 : 32, kTopkThreads / 32>(mx, kk, s));
  auto push = [&](uint32_t key, int idx) {
    const int slot = atomicAdd(&s.count, 1);
    if (slot < kCandCap) s.cand[slot] = cand_of(key, idx);
  };
  for (int i = tid; i < nvec; i += kU * nt) {
    uint4 raw[kU];
#pragma unroll
    for (int u = 0; u < kU; ++u) raw[u] = i + u * nt < nvec ? __ldg(vp + i + u * nt) : make_uint4(~0u, ~0u, ~0u, ~0u);
    visit_hits<T>(raw, (nvec - i + nt - 1) / nt, head + i * kVec, nt * kVec, bound, kU * kVec, push);
  }
  if (tid < scal) {
    const uint32_t key = key_of_bits<T>(scal_word);
    if (key >= bound.low) push(key, scal_idx);
  }
  __syncthreads();
  const int n_cand = s.count;
  __syncthreads();

  topk_finish<T>(s, n_cand, rp, v, kk, inv_temp, top_p, u24, row, out);
}

// ------------------------------------------------------------------------------------------
// Top-k kernel for rows of 16-bit logits that fit the registers of a few SMs: a cluster of
// C CTAs (1, 2 or 4) shares a row, every thread requests its whole part (eight 16-byte vectors) at
// once and keeps it, so the row is read once and the collection costs no second pass. One CTA
// with eight loads per thread and step needs several round trips to memory and the same again to L2.
//   1. CTA r keeps its 1/C of the row and finds, as above, a bound that at least kk of its own
//      elements reach. One from a search is exchanged through distributed shared memory and the largest
//      serves the whole row (the part that produced it alone holds kk elements at or above it); with the
//      warps' keys, for a small k, the few more candidates cost less than the exchange.
//   2. Every CTA collects the elements of its part that reach its bound; the others store theirs into
//      CTA 0's shared memory, all meet at the cluster barrier, the others leave and CTA 0 finishes as the
//      one-CTA kernel does. If the candidates of a small k do not fit, there is a second try with a bound
//      from all maxima.
// The survivors are the kk largest by (key desc, id asc) of a candidate set that contains them
// all, so the token is the one the one-CTA kernel and the CPU library return. No multicast.
// What bounds it is the chain, 18.5k cycles for bf16 [64, 128256], k = 50: load of the row 6.3k, bound 2.4k,
// collection 1.5k, exchange 4.2k, sort 2.1k, masses and draw 1.4k (27.3k before: bound 7.4k, sort 3.6k, draw
// 3.4k; 22.6 us a call then, 16.4 us now, the L2 flushed before each). Packed 16-bit maxima and comparisons
// look at a vector in five instructions instead of about eighty, and rows may start anywhere: what lies
// before the first 16-byte boundary is read as scalars (128255 columns, 64 rows: 72 us scalar, 16.4 us now).
// ------------------------------------------------------------------------------------------
constexpr int kMaxCluster = 4;

struct ClusterXchg {
  uint32_t low[kMaxCluster];   // bound found by each CTA of the cluster
  int cnt[kMaxCluster];        // candidates collected by each CTA (CTA 0's copy)
};

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t map_to_cta(const void* p, uint32_t rank) {
  uint32_t a = static_cast<uint32_t>(__cvta_generic_to_shared(p)), r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}
__device__ __forceinline__ void st_remote_u32(uint32_t cluster_addr, uint32_t v) {
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(cluster_addr), "r"(v) : "memory");
}
__device__ __forceinline__ void st_remote_u64(uint32_t cluster_addr, unsigned long long v) {
  asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(cluster_addr), "l"(v) : "memory");
}
__device__ __forceinline__ void cluster_arrive_release() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait_acquire() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }

constexpr int kHeldThreads = 1024;
constexpr int kHeldVecs = 8;                                          // 16-byte vectors a thread keeps
constexpr int kHeldElems = kHeldThreads * kHeldVecs * 8;              // 16-bit elements a CTA keeps

template <typename T, int C, int kFrom>
__global__ void __launch_bounds__(kHeldThreads, 1)
sample_topk_held_kernel(const T* __restrict__ logits, long long row_stride, int v,
                        const long long* __restrict__ row_ids, float inv_temp, int top_k, float top_p,
                        unsigned long long seed, unsigned long long step, int* __restrict__ out) {
  static_assert(Elem<T>::kPacked, "the kernel takes 16-bit logits");
  constexpr int NW = words_of(kFrom);
  static_assert(kHeldVecs % NW == 0, "every word gets its share of the vectors");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  TopkSmem& s = *reinterpret_cast<TopkSmem*>(smem_raw);
  ClusterXchg& x = *reinterpret_cast<ClusterXchg*>(smem_raw + sizeof(TopkSmem));
  const int tid = threadIdx.x;
  const int row = blockIdx.x / C;
  const int cr = C == 1 ? 0 : static_cast<int>(cluster_rank());
  const T* rp = logits + static_cast<long long>(row) * row_stride;
  const int kk = min(min(top_k, kMaxTopK), v);
  if (tid == 0) s.count = 0;
  if constexpr (C > 1) cluster_arrive_release();   // waited for before the first remote access

  // ---- this CTA's part: vectors [v0, v1) of the row, the scalars at its ends go to the last CTA
  const int head = row_head(rp, v), nvec = (v - head) / 8, scal = v - nvec * 8;
  const int v0 = static_cast<int>(static_cast<long long>(nvec) * cr / C);
  const int v1 = static_cast<int>(static_cast<long long>(nvec) * (cr + 1) / C);
  const uint4* mine_p = reinterpret_cast<const uint4*>(rp + head) + v0 + tid;   // this thread's vectors, kHeldThreads apart
  const int left = v1 - v0 - tid;
  uint4 raw[kHeldVecs];
#pragma unroll
  for (int u = 0; u < kHeldVecs; ++u)
    raw[u] = u * kHeldThreads < left ? __ldg(mine_p + u * kHeldThreads) : make_uint4(~0u, ~0u, ~0u, ~0u);   // NaN: key 0
  const bool has_scal = cr == C - 1 && tid < scal;
  const int scal_idx = tid < head ? tid : nvec * 8 + tid;
  const uint32_t scal_word = 0xFFFF0000u | (has_scal ? reinterpret_cast<const unsigned short*>(rp)[scal_idx] : 0xFFFFu);
  const unsigned long long rid = row_ids ? static_cast<unsigned long long>(row_ids[row])
                                         : static_cast<unsigned long long>(row);
  const uint32_t u24 = uniform_u24(seed, rid, step);   // while the loads are under way
  uint32_t mx[NW];
#pragma unroll
  for (int i = 0; i < NW; ++i) mx[i] = i == 0 ? scal_word : ~0u;
#pragma unroll
  for (int u = 0; u < kHeldVecs; ++u) mx[u % NW] = Elem<T>::wmax(mx[u % NW], vec_max<T>(raw[u]));
  words_to_keys<T>(mx);
  uint32_t low16 = bound_of<kFrom, 16, kHeldThreads / 32>(mx, kk, s);
  if constexpr (C > 1) {
    cluster_wait_acquire();                            // every CTA of the cluster runs, its counter is zero
    if constexpr (kFrom != kWarpKeys) {
      if (tid < C) st_remote_u32(map_to_cta(&x.low[cr], static_cast<uint32_t>(tid)), low16);
      cluster_arrive_release();
      cluster_wait_acquire();
#pragma unroll
      for (int r = 0; r < C; ++r) low16 = max(low16, x.low[r]);
    }
  }

  // ---- collect this part's elements at or above the bound. The warps' keys may bound a part far too low: one
  // that has few finite elements, or has its largest in a few warps. If the candidates then do not fit, the
  // block searches all its maxima, the largest bound of all parts serves the row and the parts, which
  // are still in registers, are looked at again (bf16, 40 rows of 128256 columns, k = 50: 99.9 % -inf 195 us when
  // such rows were searched exactly, 22 now; sorted 153 us, 22 now).
  constexpr int kPart = C > 1 ? 1536 : 0, kList = kCandCap - (C - 1) * kPart;
  int total;
#pragma unroll 1
  for (bool again = kFrom != kWarpKeys;; again = true) {
    const Bound<T> bound(low16);
    auto push = [&](uint32_t key, int idx) {
      const int slot = atomicAdd(&s.count, 1);
      if (slot < kCandCap) s.cand[slot] = cand_of(key, idx);
    };
    // with room for 1536 candidates a part, a thread with more than a few says that the bound is too low
    if (!visit_hits<T>(raw, (left + kHeldThreads - 1) / kHeldThreads, head + (v0 + tid) * 8, kHeldThreads * 8, bound,
                       again || C == 1 ? kHeldVecs * 8 : 8, push))
      atomicAdd(&s.count, kCandCap + 1);
    if (has_scal) {
      const uint32_t key = key_of_bits<T>(scal_word);
      if (key >= bound.low) push(key, scal_idx);
    }
    __syncthreads();
    total = s.count;
    bool fits = total <= kList;
    if constexpr (C > 1) {
      // the others' candidates go to parts of CTA 0's buffer that its own do not reach; one-way stores, no
      // round trip for a place in the list. Every CTA learns all counts, so that all decide alike.
      if (cr != 0) {
        const uint32_t dst = map_to_cta(&s.cand[kCandCap - cr * kPart], 0u);
        for (int j = tid; j < total && j < kPart; j += kHeldThreads)
          st_remote_u64(dst + 8u * static_cast<uint32_t>(j), s.cand[j]);
      }
      if (tid < C) st_remote_u32(map_to_cta(&x.cnt[cr], static_cast<uint32_t>(tid)), static_cast<uint32_t>(total));
      cluster_arrive_release();
      cluster_wait_acquire();
      int sum = x.cnt[0];
      fits = true;
#pragma unroll
      for (int r = 1; r < C; ++r) {
        fits = fits && x.cnt[r] <= kPart;
        sum += x.cnt[r];
      }
      fits = fits && sum <= kList;
    }
    if (fits || again) {
      if (!fits) total = kCandCap + 1;         // the row is searched exactly
      break;
    }
    uint32_t wide;
    if constexpr (C == 1) {
      wide = kth_key16_far(mx[0], kk, s);
    } else {
      const uint32_t word[1] = {mx[0]};
      wide = kth_key<1, 16>(word, kk, s.hits);
    }
    const uint32_t best = max(low16, wide);    // the search has barriers: everybody has read s.count
    bool better = best > low16;
    if (tid == 0) s.count = 0;
    if constexpr (C > 1) {
      if (tid < C) st_remote_u32(map_to_cta(&x.low[cr], static_cast<uint32_t>(tid)), (low16 << 16) | best);
      cluster_arrive_release();
      cluster_wait_acquire();                  // everybody has read x.cnt as well
      low16 = best;
#pragma unroll
      for (int r = 0; r < C; ++r) low16 = max(low16, x.low[r] & 0xFFFFu);
      better = false;
#pragma unroll
      for (int r = 0; r < C; ++r) better = better || low16 > (x.low[r] >> 16);
    } else {
      low16 = best;
    }
    if (!better) {                             // ties: no bound leaves fewer
      total = kCandCap + 1;
      break;
    }
    __syncthreads();
  }
  if constexpr (C > 1) {
    if (cr != 0) return;                       // nobody touches another CTA's shared memory any more
    if (total <= kCandCap) {
#pragma unroll
      for (int r = 1; r < C; ++r) {            // close the gap
        const int n = x.cnt[r];
        for (int j = tid; j < n; j += kHeldThreads) s.cand[total + j] = s.cand[kCandCap - r * kPart + j];
        total += n;
      }
    }
  }
  __syncthreads();
  topk_finish<T>(s, total, rp, v, kk, inv_temp, top_p, u24, row, out);
}

// ------------------------------------------------------------------------------------------
// General kernel: no top-k bound small enough for the candidate list.
//
// The kept set is a prefix of the order (key desc, id asc): the first n* elements with
//   n* = min(k, smallest n with mass(first n) > top_p * Z_k)      (Z_k = mass of the first k)
// The prefix is located by radix descent over the key bits (11, 11, 10) with exact integer
// histograms of element counts and fixed-point masses (fp32 rows, and fp16 rows that sample_row16
// hands back), or at full key resolution from two half histograms of counts per key (such bf16
// rows, descend16 below); ties at the threshold key are cut in token-id order. The draw inverts
// the CDF over the kept set in token-id order: every thread owns a contiguous piece of the row,
// two block scans give it the ties and the kept mass before its piece.
// ------------------------------------------------------------------------------------------
constexpr int kBins = 2048;

struct GeneralSmem {
  unsigned int cnt[kBins];
  unsigned long long mass[kBins];
  unsigned long long scan[kWarps];
  int red[kWarps];
  uint32_t max_key;
  // results of a descent
  unsigned long long above_cnt;
  unsigned long long above_mass;
  int sel_bin;
  int pick;
};

constexpr int kGeneralSmemBytes = (static_cast<int>(sizeof(GeneralSmem)) + 15) / 16 * 16;

// One descent: find key tau and the (count, mass) strictly above it such that the element
// that crosses `limit` lies among the keys equal to tau. `by_mass` selects the criterion:
//   by count: first key where count_above + count(key) >  limit  (limit = k - 1)
//   by mass : first key where mass_above  + mass(key)  >  limit
template <typename T>
__device__ void descend(const T* rp, int v, float inv_temp, float y_max, bool by_mass,
                        unsigned long long limit, GeneralSmem& s, uint32_t& tau, unsigned long long& above_cnt,
                        unsigned long long& above_mass) {
  const int tid = threadIdx.x;
  uint32_t prefix = 0;
  int known_bits = 0;
  above_cnt = 0;
  above_mass = 0;
  const int widths[3] = {11, 11, 10};
  for (int round = 0; round < 3; ++round) {
    const int w = widths[round];
    const int shift = 32 - known_bits - w;
    for (int b = tid; b < kBins; b += kThreads) {
      s.cnt[b] = 0;
      s.mass[b] = 0;
    }
    __syncthreads();
    for_each_key<T>(rp, v, [&](uint32_t key, int) {
      const bool match = known_bits == 0 || (key >> (32 - known_bits)) == (prefix >> (32 - known_bits));
      if (match) {
        const int bin = (key >> shift) & ((1 << w) - 1);
        atomicAdd(&s.cnt[bin], 1u);
        const float y = mul_rn(key_to_float(key), inv_temp);
        atomicAdd(&s.mass[bin], mass_fixed(exp_det(sub_rn(y, y_max))));
      }
    });
    __syncthreads();
    if (tid == 0) {
      unsigned long long c = above_cnt, m = above_mass;
      int sel = 0;
      for (int b = (1 << w) - 1; b >= 0; --b) {
        const unsigned long long nc = c + s.cnt[b], nm = m + s.mass[b];
        const bool crosses = by_mass ? (nm > limit) : (nc > limit);
        if (crosses || b == 0) {
          sel = b;
          break;
        }
        c = nc;
        m = nm;
      }
      s.sel_bin = sel;
      s.above_cnt = c;
      s.above_mass = m;
    }
    __syncthreads();
    prefix |= static_cast<uint32_t>(s.sel_bin) << shift;
    above_cnt = s.above_cnt;
    above_mass = s.above_mass;
    known_bits += w;
    __syncthreads();
  }
  tau = prefix;
}

// ---- bf16 rows: one descent at full key resolution ------------------------------------------
// A bf16 value has 16 significant bits, so key >> 16 names the key and the mass of a key is a
// function of the key alone: a histogram of element COUNTS per key gives every (count, mass)
// the search needs, mass(key) * count(key) being the exact integer sum the element-wise walk
// would produce. The 65536 keys are taken in two halves of 32768 counters (128 KiB of shared
// memory), upper half (non-negative values) first; the second pass over the row only happens
// when the threshold lies among the negative values. No 64-bit atomics, and the counters of a
// row spread over hundreds of keys instead of a few dozen coarse bins.
constexpr int kHalfBins = 32768;
constexpr int kHistBytes = kHalfBins * 4;

__device__ __forceinline__ uint32_t key16_to_key(uint32_t k16) {
  if (k16 == 0) return 0u;  // NaN
  return (k16 << 16) | ((k16 & 0x8000u) ? 0u : 0xFFFFu);
}

__device__ __forceinline__ unsigned long long key16_mass(uint32_t k16, float inv_temp, float y_max) {
  const float y = mul_rn(key_to_float(key16_to_key(k16)), inv_temp);
  return mass_fixed(exp_det(sub_rn(y, y_max)));
}

// Same contract as descend(); `present` additionally receives the number of elements equal to tau.
template <typename T>
__device__ void descend16(const T* rp, int v, float inv_temp, float y_max, bool by_mass,
                          unsigned long long limit, GeneralSmem& s, unsigned int* hist, uint32_t& tau,
                          unsigned long long& above_cnt, unsigned long long& above_mass,
                          unsigned long long& present) {
  const int tid = threadIdx.x;
  constexpr int kPer = kHalfBins / kThreads;  // bins per thread, walked from the top down
  unsigned long long carry_cnt = 0, carry_mass = 0;
  for (int half = 1; half >= 0; --half) {
    for (int b = tid; b < kHalfBins; b += kThreads) hist[b] = 0;
    if (tid == 0) s.sel_bin = -1;
    __syncthreads();
    for_each_key<T>(rp, v, [&](uint32_t key, int) {
      const uint32_t k16 = key >> 16;
      if (static_cast<int>(k16 >> 15) == half) atomicAdd(&hist[k16 & 0x7FFFu], 1u);
    });
    __syncthreads();
    const int top = kHalfBins - 1 - tid * kPer;
    const uint32_t hi_bit = static_cast<uint32_t>(half) << 15;
    // totals of this thread's bins; the walk starts at a different bin in every lane, so that
    // the lanes of a warp (whose ranges are kPer words apart) read different banks
    static_assert(kPer == 32, "the rotation below assumes one bin per bank and lane");
    unsigned long long my_cnt = 0, my_mass = 0;
    for (int j = 0; j < kPer; ++j) {
      const int b = top - ((j + tid) & (kPer - 1));
      const unsigned int c = hist[b];
      if (c) {
        my_cnt += c;
        my_mass += c * key16_mass(hi_bit | static_cast<uint32_t>(b), inv_temp, y_max);
      }
    }
    unsigned long long tot_cnt, tot_mass;
    const unsigned long long pre_cnt = carry_cnt + block_exscan_u64(my_cnt, s.scan, tot_cnt);
    const unsigned long long pre_mass = carry_mass + block_exscan_u64(my_mass, s.scan, tot_mass);
    const unsigned long long crit_pre = by_mass ? pre_mass : pre_cnt;
    const unsigned long long crit_mine = by_mass ? my_mass : my_cnt;
    if (crit_pre <= limit && crit_pre + crit_mine > limit) {  // the crossing is in this thread's bins
      unsigned long long c = pre_cnt, m = pre_mass;
      for (int j = 0; j < kPer; ++j) {
        const unsigned int n = hist[top - j];
        const unsigned long long nc = c + n;
        const unsigned long long nm =
            m + (n ? n * key16_mass(hi_bit | static_cast<uint32_t>(top - j), inv_temp, y_max) : 0ull);
        if (by_mass ? (nm > limit) : (nc > limit)) {
          s.sel_bin = top - j;
          s.above_cnt = c;
          s.above_mass = m;
          break;
        }
        c = nc;
        m = nm;
      }
    }
    __syncthreads();
    if (s.sel_bin >= 0) {
      tau = key16_to_key(hi_bit | static_cast<uint32_t>(s.sel_bin));
      above_cnt = s.above_cnt;
      above_mass = s.above_mass;
      present = hist[s.sel_bin];
      __syncthreads();
      return;
    }
    carry_cnt += tot_cnt;
    carry_mass += tot_mass;
    __syncthreads();
  }
  // nothing crossed: the lowest key (NaN, mass 0), as the bitwise descent ends in bin 0 of every level
  tau = 0u;
  present = hist[0];
  above_cnt = carry_cnt - hist[0];
  above_mass = carry_mass;
  __syncthreads();
}

// ---- masses by arithmetic -------------------------------------------------------------------
// mass_fixed(exp_det(x * inv_temp - y_max)) of two elements at a time, the same integers without the
// conversion instructions (a quarter of the rate of the others): rounding to an integer by adding and
// subtracting 1.5 * 2^23, the exponent taken from that sum's bits, the float-to-integer step by a shift of
// the mantissa. The products and sums are the packed two-element instructions, which round each half as the
// scalar ones do. 19 instructions an element: a draw over
// all 128256 elements (temperature only) takes 25 us for one row, with a histogram and a table in front of it
// it took 62 us; fp32 25 us, with exp_det per element 168 us.
struct MassArgs {
  float inv_temp, neg_y_max;
};

__device__ __forceinline__ unsigned long long pack2(float a, float b) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpack2(unsigned long long v, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ unsigned long long mul2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ unsigned long long both(float a) { return pack2(a, a); }

__device__ __forceinline__ void mass_pair(float x0, float x1, const MassArgs& a, unsigned long long& sum) {
  constexpr float kRound = 12582912.0f;                       // 1.5 * 2^23
  // the first product is scalar: the assembler joins a packed product and the packed sum behind it into one
  // rounding, .rn or not
  const unsigned long long y = pack2(__fmul_rn(x0, a.inv_temp), __fmul_rn(x1, a.inv_temp));
  unsigned long long t = mul2(add2(y, both(a.neg_y_max)), both(1.4426950408889634f));
  float t0, t1;
  unpack2(t, t0, t1);
  t = pack2(fmaxf(t0, -64.f), fmaxf(t1, -64.f));              // below 2^-33 the mass is 0; NaN becomes -64
  const unsigned long long r = add2(t, both(kRound));
  const unsigned long long f = fma2(add2(r, both(-kRound)), both(-1.f), t);
  unsigned long long p = both(1.5403530393381609e-4f);
  p = fma2(p, f, both(1.3333558146428443e-3f));
  p = fma2(p, f, both(9.6181291076284772e-3f));
  p = fma2(p, f, both(5.5504108664821580e-2f));
  p = fma2(p, f, both(2.4022650695910071e-1f));
  p = fma2(p, f, both(6.9314718055994531e-1f));
  p = fma2(p, f, both(1.0f));
  float r0, r1, p0, p1;
  unpack2(r, r0, r1);
  unpack2(p, p0, p1);
  auto add = [&](float rr, float pp) {
    const uint32_t pb = __float_as_uint(pp);
    // floor(p 2^(n + 32)) = mantissa (bit 31 down) >> shift, with n in the low bits of rr
    const uint32_t shift = 126u + 0x4B400000u - (pb >> 23) - __float_as_uint(rr);
    const uint32_t m = __funnelshift_rc((pb << 8) | 0x80000000u, 0u, shift);   // a shift of 32 or more gives 0
    sum += (static_cast<unsigned long long>(shift >> 31) << 32) | m;           // shift -1: p = 1, n = 0
  };
  add(r0, p0);
  add(r1, p1);
}

__device__ __forceinline__ unsigned long long warp_sum_u64(unsigned long long v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ unsigned long long warp_incl_u64(unsigned long long v) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long n = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += n;
  }
  return v;
}

// ---- 16-bit rows: everything from one histogram of counts per key -----------------------------
// A bf16 or fp16 value has 65536 keys and the mass of a key is a function of the key, so one
// pass that counts elements per key answers every question about (count, mass) prefixes: the
// maximum, the total mass and both thresholds cost one exponential per distinct value instead
// of one per element and pass.
//   * Counters are 16 bits, two per word (128 KiB), named by the value's bits as they are; only what reads
//     them puts them in the order of keys, by groups of 32. An overflow loses at least 65535 from the sum
//     of the counters, so "sum == v" says that none happened; a row in which one value fills more than
//     65535 places takes the older search. NaNs, which have many bit patterns and one key, are moved to that
//     key's counter, if there are any, and the groups are counted once more.
//   * Only groups that occur are visited when masses are added up (150 of 2048 for bf16 logits).
//   * The masses of the keys above the threshold go to a table in the counters' place if there are fewer
//     than 16384 of them (a few hundred for top-p on bf16 logits). Its entries are 64 bits, so that a tie at
//     the threshold counts itself in the high bits and a lookup needs no branch.
// What bounds it: bf16 [148, 128256] ~ N(0, 2), T = 1, top_p = 0.9 takes a CTA 52.9k cycles: 18k for the
// histogram (a shared-memory atomic per element, about four conflicting lanes each), 17k for the draw (a
// table lookup per element), 10k for the searches between, 7k for clearing, table and the end of the draw.
// 107k before: groups that do not occur were visited, lookups went through two tables and behind a branch
// (33k for the draw with one table and the branch). 62 us a call then, 35 us now.
constexpr int kGroups = 2048;                 // of 32 keys; GeneralSmem::cnt / mass hold their sums
constexpr int kTable = 16384;
constexpr int kTieShift = 48;                 // a thread's masses add up to less than 2^48 (at most 2^15 elements of 2^32)
constexpr int kTableMaxVocab = 1 << 25;       // ... which 32 warps' lanes see in rows of at most this many elements
constexpr int kHistWords = 32768;
static_assert(kGroups == kBins && kGroups == 2 * kThreads, "two groups per thread, sums kept in the descent's bins");

struct FastSmem {
  union {
    unsigned int words[kHistWords];             // 16-bit counters
    unsigned long long table[kTable];           // then masses by distance from the largest key
  };
  unsigned short list[kGroups];               // groups that occur
  unsigned int n_list;
  unsigned int total;
  unsigned int nans;
  unsigned int top_group;
  // result of a search
  int sel;
  unsigned int sel_key;
  unsigned long long above_cnt, above_mass, present;
};

// What the draw keeps: keys above tau, and of the ties at tau the first tie_keep in token-id order.
struct Kept {
  uint32_t tau;                  // 32-bit key
  unsigned long long tie_keep, q_tau;
  MassArgs args;
  const unsigned long long* table;   // kByTable: masses by distance from the largest key, a tie, 0
  uint32_t top2, last2;              // in both halves of a word: the largest 16-bit key + 1, the distance of what has no mass
};
struct DrawSmem {
  unsigned long long seg_ties[kWarps];
  unsigned long long seg_mass[kWarps];
  unsigned long long ties_before, target;
  int sel;
};
enum : int { kAll = 0, kByExp = 1, kByTable = 2, kByCount = 3 };   // all are kept / masses computed / looked up / 1 each

template <typename T>
__device__ __forceinline__ float key16_float(uint32_t k16) {
  if (k16 == 0) return key_to_float(0u);  // NaN
  return Elem<T>::to_float(from_bits16<T>((k16 & 0x8000u) ? (k16 & 0x7FFFu) : (~k16 & 0xFFFFu)));
}
template <typename T>
__device__ __forceinline__ unsigned long long key16_mass_of(uint32_t k16, float inv_temp, float y_max) {
  return mass_fixed(exp_det(sub_rn(mul_rn(key16_float<T>(k16), inv_temp), y_max)));
}

__device__ __forceinline__ unsigned int key_count(const FastSmem& f, uint32_t k16) {
  const uint32_t bits = (k16 & 0x8000u) ? (k16 & 0x7FFFu) : (0xFFFFu - k16);
  return (f.words[bits >> 1] >> ((bits & 1u) * 16u)) & 0xFFFFu;
}

// descend()'s contract on the histogram, from the prefix sums of this thread's two groups (pre_c / pre_m: what
// lies above them): the group that holds the crossing, then the key inside it by one warp. above_cnt is only
// valid if counts were summed.
template <typename T>
__device__ void search_groups(bool by_mass, unsigned long long limit, float inv_temp, float y_max,
                              unsigned long long pre_c, unsigned long long pre_m, unsigned long long tot_c,
                              unsigned long long tot_m, const GeneralSmem& s, FastSmem& f) {
  const int tid = threadIdx.x, lane = tid & 31;
  if (tid == 0) f.sel = -1;
  __syncthreads();
  const int g0 = kGroups - 1 - 2 * tid;       // this thread's groups, from the top: g0, g0 - 1
  const unsigned long long c0 = s.cnt[g0], c1 = s.cnt[g0 - 1], m0 = s.mass[g0], m1 = s.mass[g0 - 1];
  const unsigned long long pre = by_mass ? pre_m : pre_c, mid = pre + (by_mass ? m0 : c0), end = mid + (by_mass ? m1 : c1);
  if (pre <= limit && end > limit) {
    const bool second = mid <= limit;
    f.sel = second ? g0 - 1 : g0;
    f.above_cnt = second ? pre_c + c0 : pre_c;
    f.above_mass = second ? pre_m + m0 : pre_m;
  }
  __syncthreads();
  const int g = f.sel;
  if (g < 0) {
    // nothing crossed: the lowest key (NaN, mass 0), as the bitwise descent ends in bin 0
    if (tid == 0) {
      f.present = key_count(f, 0);
      f.sel_key = 0;
      f.above_cnt = tot_c - f.present;
      f.above_mass = tot_m;
    }
  } else if (tid < 32) {
    const uint32_t key = static_cast<uint32_t>(g) * 32u + 31u - lane;   // from the top
    const unsigned long long kc = key_count(f, key);
    const unsigned long long km = kc ? kc * key16_mass_of<T>(key, inv_temp, y_max) : 0ull;
    const unsigned long long ic = warp_incl_u64(kc), im = warp_incl_u64(km);
    const unsigned long long above_c = f.above_cnt, above_m = f.above_mass;
    const bool crosses = by_mass ? above_m + im > limit : above_c + ic > limit;
    const int first = __ffs(static_cast<int>(__ballot_sync(0xffffffffu, crosses))) - 1;
    if (lane == first) {
      f.sel_key = key;
      f.above_cnt = above_c + ic - kc;
      f.above_mass = above_m + im - km;
      f.present = kc;
    }
  }
  __syncthreads();
}

// Kept mass and ties of the elements [begin, end) of the row, summed by one warp (any order).
template <typename T, int kMode>
__device__ __forceinline__ void sum_range(const T* rp, int begin, int end, const Kept& k, unsigned long long& mass,
                                          unsigned long long& ties) {
  constexpr int kVec = Elem<T>::kVec, kU = 4;
  static_assert(kMode != kByTable || Elem<T>::kPacked, "the table is indexed by 16-bit keys");
  const int lane = threadIdx.x & 31;
  const T* p = rp + begin;
  const int n = end - begin, head = row_head(p, n), nvec = (n - head) / kVec, scal = n - nvec * kVec;
  unsigned long long m = 0;
  unsigned int n_ties = 0;
  const int tau_o = static_cast<int>(k.tau ^ 0x80000000u);    // keys as signed numbers
  auto ordered = [](float x) {
    const int b = __float_as_int(x);
    return b ^ ((b >> 31) & 0x7FFFFFFF);
  };
  auto take2 = [&](float x0, float x1) {
    if constexpr (kMode != kAll) {
      const int o0 = ordered(x0), o1 = ordered(x1);
      n_ties += (o0 == tau_o ? 1u : 0u) + (o1 == tau_o ? 1u : 0u);
      x0 = o0 > tau_o ? x0 : __uint_as_float(0xFF800000u);
      x1 = o1 > tau_o ? x1 : __uint_as_float(0xFF800000u);
    }
    mass_pair(x0, x1, k.args, m);
  };
  auto take_word = [&](uint32_t w) {
    if constexpr (kMode == kByTable) {
      // distance of both keys from the largest one, cut off behind the tie's: min(top - key, last)
      const uint32_t not_key = ~(w ^ (((w >> 15) & 0x00010001u) * 0x7FFFu));   // keys as signed numbers
      const uint32_t i2 = __viaddmin_u16x2(not_key, k.top2, k.last2);
      m += k.table[i2 & 0xFFFFu];
      m += k.table[i2 >> 16];
    } else if constexpr (Elem<T>::kPacked) {
      take2(Elem<T>::to_float(from_bits16<T>(w & 0xFFFFu)), Elem<T>::to_float(from_bits16<T>(w >> 16)));
    }
  };
  const uint4* vp = reinterpret_cast<const uint4*>(p + head);
  for (int j = lane; j < nvec; j += 32 * kU) {
    uint4 raw[kU];
#pragma unroll
    for (int u = 0; u < kU; ++u)
      if (j + 32 * u < nvec) raw[u] = __ldg(vp + j + 32 * u);
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      if (j + 32 * u >= nvec) break;
      if constexpr (Elem<T>::kPacked) {
        take_word(raw[u].x);
        take_word(raw[u].y);
        take_word(raw[u].z);
        take_word(raw[u].w);
      } else {
        take2(__uint_as_float(raw[u].x), __uint_as_float(raw[u].y));
        take2(__uint_as_float(raw[u].z), __uint_as_float(raw[u].w));
      }
    }
  }
  if (lane < scal) {
    // one element; its partner is -inf, which has no mass and is no tie (-inf as a threshold has mass 0)
    const T e = p[lane < head ? lane : nvec * kVec + lane];
    if constexpr (kMode == kByTable) {
      const uint32_t w = *reinterpret_cast<const unsigned short*>(&e);
      m += k.table[__viaddmin_u16x2(~(w ^ ((w >> 15) * 0x7FFFu)), k.top2, k.last2) & 0xFFFFu];
    } else {
      const float x = Elem<T>::to_float(e);
      const unsigned int before = n_ties;
      take2(x, __uint_as_float(0xFF800000u));
      n_ties = before + (kMode != kAll && ordered(x) == tau_o ? 1u : 0u);
    }
  }
  if constexpr (kMode == kByTable) {
    n_ties = static_cast<unsigned int>(m >> kTieShift);
    m &= (1ull << kTieShift) - 1;
  }
  mass = warp_sum_u64(m);
  ties = kMode == kAll ? 0ull : __reduce_add_sync(0xffffffffu, n_ties);
}

// First element, in token-id order, whose cumulative kept mass exceeds the target: the row is cut into
// 32 contiguous segments, one per warp, whose kept masses are order-free integer sums (coalesced loads),
// the segment that holds the target is cut into 32 again, and only the last hundred elements are walked
// in order. With kAll the kept mass is what the first level adds up; false if it is 0.
template <typename T, int kMode>
__device__ bool draw(const T* rp, int v, const Kept& k, unsigned long long kept_mass, uint32_t u24, DrawSmem& d, int* out) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int begin = 0, end = v;
  if (tid == 0) {
    d.target = mass_scale_u24(u24, kept_mass);
    d.ties_before = 0;
    d.sel = -1;
  }
#pragma unroll 1
  for (int level = 0; level < 2; ++level) {
    const int len = ((end - begin + kWarps - 1) / kWarps + 7) / 8 * 8;
    const int b = min(end, begin + warp * len), e = min(end, b + len);
    unsigned long long mass, ties;
    sum_range<T, kMode>(rp, b, e, k, mass, ties);
    if (lane == 0) {
      d.seg_mass[warp] = mass;
      d.seg_ties[warp] = ties;
    }
    __syncthreads();
    if (warp == 0) {
      const unsigned long long t = d.seg_ties[lane];
      const unsigned long long t0 = d.ties_before + warp_incl_u64(t) - t;
      const unsigned long long left = k.tie_keep > t0 ? k.tie_keep - t0 : 0ull;
      const unsigned long long m = d.seg_mass[lane] + (t < left ? t : left) * k.q_tau;
      const unsigned long long inc = warp_incl_u64(m);
      unsigned long long target = d.target;
      if (kMode == kAll && level == 0) target = mass_scale_u24(u24, __shfl_sync(0xffffffffu, inc, 31));
      const int first = __ffs(static_cast<int>(__ballot_sync(0xffffffffu, inc > target))) - 1;
      if (lane == first) {
        d.sel = first;
        d.target = target - (inc - m);
        d.ties_before = t0;
      }
    }
    __syncthreads();
    if (d.sel < 0) return false;
    begin = min(end, begin + d.sel * len);
    end = min(end, begin + len);
  }
  if (warp == 0) {
    const unsigned long long target = d.target;
    const float y_max = -k.args.neg_y_max;
    unsigned long long acc = 0, t0 = d.ties_before;
    for (int i0 = begin; i0 < end; i0 += 32) {
      const int i = i0 + lane;
      const float x = i < end ? Elem<T>::to_float(rp[i]) : 0.f;
      const uint32_t key = float_to_key(x);
      const bool tie = i < end && kMode != kAll && key == k.tau;
      const unsigned int tie_mask = __ballot_sync(0xffffffffu, tie);
      const unsigned long long rank = t0 + __popc(tie_mask & ((1u << lane) - 1u));
      unsigned long long q = 0;
      if (i < end && (kMode == kAll || key > k.tau))
        q = mass_fixed(exp_det(sub_rn(mul_rn(key_to_float(key), k.args.inv_temp), y_max)));
      else if (tie && rank < k.tie_keep)
        q = k.q_tau;
      const unsigned long long inc = acc + warp_incl_u64(q);
      const unsigned int hit = __ballot_sync(0xffffffffu, inc > target);
      if (hit) {
        if (lane == __ffs(static_cast<int>(hit)) - 1) *out = i;
        break;
      }
      acc = __shfl_sync(0xffffffffu, inc, 31);
      t0 += __popc(tie_mask);
    }
  }
  return true;
}

// One row of 16-bit logits with a top-p or a large top-k. Returns false (for the whole block) if the row
// needs the older search.
template <typename T>
__device__ bool sample_row16(const T* rp, int v, float inv_temp, int top_k, float top_p, uint32_t u24, GeneralSmem& s,
                             FastSmem& f, DrawSmem& d, int* out) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned short* hp = reinterpret_cast<const unsigned short*>(rp);
  // ---- count
  for (int i = tid; i < kHistWords / 4; i += kThreads) reinterpret_cast<uint4*>(f.words)[i] = make_uint4(0u, 0u, 0u, 0u);
  s.mass[2 * tid] = s.mass[2 * tid + 1] = 0;
  if (tid == 0) f.n_list = f.total = f.nans = f.top_group = 0;
  __syncthreads();
  {
    // the counter of bits b is half b & 1 of word b >> 1
    auto add_word = [&](uint32_t w) {
      unsigned char* base = reinterpret_cast<unsigned char*>(f.words);
      atomicAdd(reinterpret_cast<unsigned int*>(base + ((w << 1) & 0x1FFFCu)), max((w << 16) & 0x10000u, 1u));
      atomicAdd(reinterpret_cast<unsigned int*>(base + ((w >> 15) & 0x1FFFCu)), max(w & 0x10000u, 1u));
    };
    const int head = row_head(rp, v), nvec = (v - head) / 8, scal = v - nvec * 8;
    const uint4* vp = reinterpret_cast<const uint4*>(hp + head);
    constexpr int kU = 4;
    for (int j = tid; j < nvec; j += kThreads * kU) {
      uint4 raw[kU];
#pragma unroll
      for (int u = 0; u < kU; ++u)
        if (j + kThreads * u < nvec) raw[u] = __ldg(vp + j + kThreads * u);
#pragma unroll
      for (int u = 0; u < kU; ++u) {
        if (j + kThreads * u >= nvec) break;
        add_word(raw[u].x);
        add_word(raw[u].y);
        add_word(raw[u].z);
        add_word(raw[u].w);
      }
    }
    if (tid < scal) {
      const uint32_t w = hp[tid < head ? tid : nvec * 8 + tid];
      atomicAdd(&f.words[w >> 1], 1u << ((w & 1u) * 16u));
    }
  }
  __syncthreads();
  // ---- counts per group of 32 keys (four threads' vectors of eight counters), their sum, which groups occur
  constexpr uint32_t kInf = Elem<T>::kInf2 & 0xFFFFu;
#pragma unroll 1
  for (bool again = false;; again = true) {
    constexpr int kN = kHistWords / 4 / kThreads;
    unsigned int n[kN], occurs[kN], sum = 0, nans = 0, top = 0, found = 0;
    const bool lead = (lane & 3) == 0;
    auto group_of = [&](int i) {
      const int bg = (i * kThreads + tid) >> 2;
      return bg < kGroups / 2 ? kGroups / 2 + bg : kGroups - 1 - bg;
    };
#pragma unroll
    for (int i = 0; i < kN; ++i) {
      const int at = i * kThreads + tid;
      const uint4 q = reinterpret_cast<const uint4*>(f.words)[at];
      n[i] = (q.x & 0xFFFFu) + (q.x >> 16) + (q.y & 0xFFFFu) + (q.y >> 16) + (q.z & 0xFFFFu) + (q.z >> 16) +
             (q.w & 0xFFFFu) + (q.w >> 16);
      const uint32_t mag = static_cast<uint32_t>(at * 8) & 0x7FFFu;
      if (mag >= kInf) nans += n[i] - (mag == kInf ? q.x & 0xFFFFu : 0u);
    }
#pragma unroll
    for (int i = 0; i < kN; ++i) {
      n[i] += __shfl_xor_sync(0xffffffffu, n[i], 1);
      n[i] += __shfl_xor_sync(0xffffffffu, n[i], 2);
      occurs[i] = __ballot_sync(0xffffffffu, lead && n[i] != 0);
      found += __popc(occurs[i]);
    }
    unsigned int slot = 0;
    if (lane == 0 && found) slot = atomicAdd(&f.n_list, found);
    slot = __shfl_sync(0xffffffffu, slot, 0);
#pragma unroll
    for (int i = 0; i < kN; ++i) {
      if (lead) {
        const int g = group_of(i);
        s.cnt[g] = n[i];
        sum += n[i];
        if (n[i]) {
          f.list[slot + __popc(occurs[i] & ((1u << lane) - 1u))] = static_cast<unsigned short>(g);
          top = max(top, static_cast<unsigned int>(g));
        }
      }
      slot += __popc(occurs[i]);
    }
    sum = __reduce_add_sync(0xffffffffu, sum);
    nans = __reduce_add_sync(0xffffffffu, nans);
    top = __reduce_max_sync(0xffffffffu, top);
    if (lane == 0) {
      atomicAdd(&f.total, sum);
      if (nans) atomicAdd(&f.nans, nans);
      atomicMax(&f.top_group, top);
    }
    __syncthreads();
    if (f.total != static_cast<unsigned int>(v)) return false;   // a counter overflowed
    const unsigned int n_nan = f.nans;
    if (again || n_nan == 0) break;
    if (n_nan > 0xFFFFu) return false;
    __syncthreads();
    // the patterns above infinity's, of both signs, hold nothing any more; key 0 (0xFFFF's counter) holds them all
    for (uint32_t w = (kInf >> 1) + tid; w < 0x4000u; w += kThreads) {
      const bool inf = w == kInf >> 1;         // infinity's own counter is the lower half
      f.words[w] = inf ? f.words[w] & 0xFFFFu : 0u;
      f.words[w + 0x4000u] = (inf ? f.words[w + 0x4000u] & 0xFFFFu : 0u) | (w == 0x3FFFu ? n_nan << 16 : 0u);
    }
    if (tid == 0) f.n_list = f.total = f.top_group = 0;
    __syncthreads();
  }
  uint32_t max_key;
  {
    const uint32_t key = f.top_group * 32u + static_cast<uint32_t>(lane);
    max_key = f.top_group * 32u + 31u - __clz(static_cast<int>(__ballot_sync(0xffffffffu, key_count(f, key) != 0)));
  }
  const float y_max = mul_rn(key16_float<T>(max_key), inv_temp);
  // four groups per warp at a time, eight lanes with four keys each
  for (unsigned int j0 = warp * 4; j0 < f.n_list; j0 += kWarps * 4) {
    const unsigned int j = j0 + (lane >> 3);
    unsigned long long m = 0;
    if (j < f.n_list) {
      const uint32_t key0 = f.list[j] * 32u + static_cast<uint32_t>(lane & 7) * 4u;
      // four neighbours' counters are one 64-bit word, in rising order of bits: falling keys below zero
      const bool neg = key0 < 0x8000u;
      const uint32_t bits0 = neg ? 0xFFFCu - key0 : key0 - 0x8000u;
      const uint2 c = *reinterpret_cast<const uint2*>(&f.words[bits0 >> 1]);
      const uint32_t cnt[4] = {c.x & 0xFFFFu, c.x >> 16, c.y & 0xFFFFu, c.y >> 16};
#pragma unroll
      for (int e = 0; e < 4; ++e) m += cnt[e] * key16_mass_of<T>(neg ? key0 + 3 - e : key0 + e, inv_temp, y_max);
    }
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) m += __shfl_xor_sync(0xffffffffu, m, o);
    if (j < f.n_list && (lane & 7) == 0) s.mass[f.list[j]] = m;
  }
  __syncthreads();

  // ---- where the kept prefix ends: the same decisions as in sample_general_kernel
  uint32_t tau = 0;
  unsigned long long tie_keep = ~0ull, kept_mass = 0;
  {
    uint32_t k_tau = 0;
    unsigned long long k_ties = ~0ull;
    const bool has_k = top_k > 0 && top_k < v;
    const int g0 = kGroups - 1 - 2 * tid;
    unsigned long long tot_m, tot_c = v, pre_c = 0;
    const unsigned long long pre_m = block_exscan_u64(s.mass[g0] + s.mass[g0 - 1], s.scan, tot_m);
    kept_mass = tot_m;
    if (has_k) {
      pre_c = block_exscan_u64(s.cnt[g0] + s.cnt[g0 - 1], s.scan, tot_c);
      search_groups<T>(false, static_cast<unsigned long long>(top_k - 1), inv_temp, y_max, pre_c, pre_m, tot_c, tot_m, s, f);
      k_tau = f.sel_key;
      k_ties = static_cast<unsigned long long>(top_k) - f.above_cnt;
      kept_mass = f.above_mass + k_ties * key16_mass_of<T>(k_tau, inv_temp, y_max);
    }
    tau = k_tau;
    tie_keep = k_ties;
    if (top_p < 1.0f) {
      const unsigned long long limit = mass_fraction(static_cast<double>(top_p), kept_mass);
      __syncthreads();
      search_groups<T>(true, limit, inv_temp, y_max, pre_c, pre_m, tot_c, tot_m, s, f);
      const uint32_t p_tau = f.sel_key;
      const unsigned long long above = f.above_mass, q = key16_mass_of<T>(p_tau, inv_temp, y_max);
      const unsigned long long p_ties = above > limit ? 0ull : (q == 0 ? ~0ull : (limit - above) / q + 1);
      if (!has_k || (p_tau != k_tau ? p_tau > k_tau : p_ties < k_ties)) {
        tau = p_tau;
        tie_keep = p_ties < f.present ? p_ties : f.present;
        kept_mass = above + tie_keep * q;
      }
    }
  }
  if (kept_mass == 0) return false;           // nothing has a mass: the older path picks by position

  Kept k;
  k.tau = float_to_key(key16_float<T>(tau));
  k.tie_keep = tie_keep;
  k.q_tau = key16_mass_of<T>(tau, inv_temp, y_max);
  k.args = {inv_temp, -y_max};
  const uint32_t range = max_key - tau;       // keys above the threshold
  if (range + 2 <= kTable && v <= kTableMaxVocab) {
    // table[i]: the key max_key - i; tau's entry counts ties, what is below has nothing
    for (unsigned int i = tid; i < range; i += kThreads) f.table[i] = key16_mass_of<T>(max_key - i, inv_temp, y_max);
    if (tid == 0) {
      f.table[range] = 1ull << kTieShift;
      f.table[range + 1] = 0;
    }
    k.table = f.table;
    k.top2 = ((max_key + 0x8001u) & 0xFFFFu) * 0x00010001u;   // as a signed number, + 1: ~key + 1 = -key
    k.last2 = (range + 1) * 0x00010001u;
    __syncthreads();
    return draw<T, kByTable>(rp, v, k, kept_mass, u24, d, out);
  }
  return draw<T, kByExp>(rp, v, k, kept_mass, u24, d, out);
}

// The last kept element of a row in which nothing has a mass (-1: none is kept).
template <typename T>
__device__ int last_kept(const T* rp, int v, uint32_t tau, unsigned long long tie_keep, GeneralSmem& s) {
  const int tid = threadIdx.x;
  const int chunk = (v + kThreads - 1) / kThreads;
  const int begin = min(v, tid * chunk), end = min(v, begin + chunk);
  unsigned long long ties = 0, total;
  for (int i = begin; i < end; ++i) ties += float_to_key(Elem<T>::to_float(rp[i])) == tau ? 1u : 0u;
  unsigned long long rank = block_exscan_u64(ties, s.scan, total);
  int last = -1;
  for (int i = begin; i < end; ++i) {
    const uint32_t key = float_to_key(Elem<T>::to_float(rp[i]));
    if (key > tau || (key == tau && rank < tie_keep)) last = i;
    rank += key == tau ? 1u : 0u;
  }
  last = __reduce_max_sync(0xffffffffu, last);
  __syncthreads();
  if (tid == 0) s.pick = -1;
  __syncthreads();
  if ((tid & 31) == 0) atomicMax(&s.pick, last);
  __syncthreads();
  return s.pick;
}

// Largest key of the row, for the whole block.
template <typename T>
__device__ uint32_t row_max_key(const T* rp, int v, GeneralSmem& s) {
  constexpr int kVec = Elem<T>::kVec, kU = 8;
  const int tid = threadIdx.x;
  const int head = row_head(rp, v), nvec = (v - head) / kVec, scal = v - nvec * kVec;
  const uint4* vp = reinterpret_cast<const uint4*>(rp + head);
  uint32_t w[1] = {~0u};                      // NaN: key 0
  for (int j = tid; j < nvec; j += kThreads * kU) {
    uint4 raw[kU];
#pragma unroll
    for (int u = 0; u < kU; ++u) raw[u] = j + kThreads * u < nvec ? __ldg(vp + j + kThreads * u) : make_uint4(~0u, ~0u, ~0u, ~0u);
#pragma unroll
    for (int u = 0; u < kU; ++u) w[0] = Elem<T>::wmax(w[0], vec_max<T>(raw[u]));
  }
  words_to_keys<T>(w);
  uint32_t top;
  if constexpr (Elem<T>::kPacked) {
    top = max(w[0] >> 16, w[0] & 0xFFFFu);
    top = top == 0 ? 0u : float_to_key(key16_float<T>(top));
  } else {
    top = w[0];
  }
  if (tid < scal) top = max(top, float_to_key(Elem<T>::to_float(rp[tid < head ? tid : nvec * kVec + tid])));
  top = __reduce_max_sync(0xffffffffu, top);
  if (tid == 0) s.max_key = 0;
  __syncthreads();
  if ((tid & 31) == 0) atomicMax(&s.max_key, top);
  __syncthreads();
  return s.max_key;
}

template <typename T>
__global__ void __launch_bounds__(kThreads, 1)
sample_general_kernel(const T* __restrict__ logits, long long row_stride, int v, const long long* __restrict__ row_ids,
                      float inv_temp, int top_k, float top_p, unsigned long long seed, unsigned long long step,
                      int* __restrict__ out) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ DrawSmem d;
  GeneralSmem& s = *reinterpret_cast<GeneralSmem*>(smem_raw);
  constexpr bool kKey16 = std::is_same<T, __nv_bfloat16>::value;
  unsigned int* hist = reinterpret_cast<unsigned int*>(smem_raw + kGeneralSmemBytes);  // kKey16 only
  const int tid = threadIdx.x;
  const int row = blockIdx.x;
  const T* rp = logits + static_cast<long long>(row) * row_stride;
  const unsigned long long rid = row_ids ? static_cast<unsigned long long>(row_ids[row])
                                         : static_cast<unsigned long long>(row);
  const uint32_t u24 = uniform_u24(seed, rid, step);
  const bool has_k = top_k > 0 && top_k < v;
  if constexpr (Elem<T>::kPacked) {
    FastSmem& f = *reinterpret_cast<FastSmem*>(smem_raw + kGeneralSmemBytes);
    if ((has_k || top_p < 1.0f) && sample_row16<T>(rp, v, inv_temp, top_k, top_p, u24, s, f, d, out + row)) return;
    __syncthreads();
  }
  const float y_max = mul_rn(key_to_float(row_max_key(rp, v, s)), inv_temp);
  Kept k;
  k.args = {inv_temp, -y_max};
  k.q_tau = 0;
  if (!has_k && top_p >= 1.0f) {              // everything is kept: the sums of the draw are the only pass
    k.tie_keep = 0;
    if (!draw<T, kAll>(rp, v, k, 0, u24, d, out + row) && tid == 0) out[row] = v - 1;
    return;
  }

  // ---- where the kept prefix ends: (tau, number of ties at tau that are kept)
  uint32_t tau = 0;                     // threshold key
  unsigned long long tie_keep = ~0ull;  // ties at tau kept, in id order
  unsigned long long kept_mass = 0;     // mass of the kept set
  {
    // total mass and, if top_k is set, the top-k prefix
    unsigned long long k_above_cnt = 0, k_above_mass = 0;
    uint32_t k_tau = 0;
    unsigned long long k_ties = ~0ull;
    unsigned long long zk;
    if (has_k) {
      if constexpr (kKey16) {
        unsigned long long unused;
        descend16<T>(rp, v, inv_temp, y_max, false, static_cast<unsigned long long>(top_k - 1), s, hist, k_tau,
                     k_above_cnt, k_above_mass, unused);
      } else {
        descend<T>(rp, v, inv_temp, y_max, false, static_cast<unsigned long long>(top_k - 1), s, k_tau, k_above_cnt,
                   k_above_mass);
      }
      k_ties = static_cast<unsigned long long>(top_k) - k_above_cnt;
      const float y = mul_rn(key_to_float(k_tau), inv_temp);
      zk = k_above_mass + k_ties * mass_fixed(exp_det(sub_rn(y, y_max)));
    } else {
      // everything is kept by the count criterion: Z = total mass
      const int len = ((v + kWarps - 1) / kWarps + 7) / 8 * 8;
      const int b = min(v, (tid >> 5) * len);
      unsigned long long part, unused, total;
      sum_range<T, kAll>(rp, b, min(v, b + len), k, part, unused);
      block_exscan_u64((tid & 31) == 0 ? part : 0ull, s.scan, total);
      zk = total;
    }
    tau = has_k ? k_tau : 0u;
    tie_keep = k_ties;
    kept_mass = zk;
    if (top_p < 1.0f) {
      const unsigned long long limit = mass_fraction(static_cast<double>(top_p), zk);
      uint32_t p_tau;
      unsigned long long p_above_cnt, p_above_mass, p_present = 0;
      if constexpr (kKey16) {
        descend16<T>(rp, v, inv_temp, y_max, true, limit, s, hist, p_tau, p_above_cnt, p_above_mass, p_present);
      } else {
        descend<T>(rp, v, inv_temp, y_max, true, limit, s, p_tau, p_above_cnt, p_above_mass);
      }
      // element i (in sorted order) is kept while the mass before it is <= limit
      const float y = mul_rn(key_to_float(p_tau), inv_temp);
      const unsigned long long q = mass_fixed(exp_det(sub_rn(y, y_max)));
      unsigned long long p_ties;
      if (p_above_mass > limit) {
        p_ties = 0;  // cannot happen: the descent stops at the first crossing key
      } else if (q == 0) {
        p_ties = ~0ull;
      } else {
        p_ties = (limit - p_above_mass) / q + 1;
      }
      // the tighter of the two prefixes wins
      bool p_tighter;
      if (!has_k) {
        p_tighter = true;
      } else if (p_tau != k_tau) {
        p_tighter = p_tau > k_tau;
      } else {
        p_tighter = p_ties < k_ties;
      }
      if (p_tighter) {
        tau = p_tau;
        tie_keep = p_ties;
        // the kept mass follows from the number of ties actually present
        unsigned long long present;
        if constexpr (kKey16) {
          present = p_present;  // the histogram had the count
        } else {
          int local = 0;
          for_each_key<T>(rp, v, [&](uint32_t key, int) { local += (key == p_tau) ? 1 : 0; });
          present = static_cast<unsigned long long>(block_sum_int(local, s.red));
        }
        const unsigned long long used = p_ties < present ? p_ties : present;
        tie_keep = used;
        kept_mass = p_above_mass + used * q;
      }
    }
  }

  // ---- draw: invert the CDF over the kept set in token-id order
  k.tau = tau;
  k.tie_keep = tie_keep;
  k.q_tau = mass_fixed(exp_det(sub_rn(mul_rn(key_to_float(tau), inv_temp), y_max)));
  if (draw<T, kByExp>(rp, v, k, kept_mass, u24, d, out + row)) return;
  // target == kept_mass can only happen when kept_mass is 0 (all masses underflowed):
  // fall back to the last kept element
  const int last = last_kept<T>(rp, v, tau, tie_keep, s);
  if (tid == 0) out[row] = last < 0 ? 0 : last;
}

// ---- bf16 rows: histograms per part of the row -------------------------------------------------
// What bounds the general path is one shared-memory atomic per element: a histogram of 148 rows of
// 128256 columns, one row per SM, takes 14.5 us whatever the counters' width, 12.5 of them atomics (5.9 cycles per
// warp, the conflicts of 32 random banks), and nothing else has to be done per element:
//   * A row is cut into C * 2 contiguous sub-parts, C CTAs (a cluster) with a histogram for each of their
//     two. The kept mass of a sub-part follows from its histogram, so only the one that holds the target is
//     read again by the draw (a sixteenth to a half of the row; the draw over whole rows took as long as the counting).
//   * C is chosen by part_ctas: few rows fill the GPU, and 200 rows are 400 CTAs, at most three half rows per SM, where one CTA
//     of 1024 threads per row and SM takes two rounds.
//   * For three CTAs per SM the two histograms must fit 64 KiB: 16-bit counters (a sub-part has at most 65535 elements) of the
//     values whose magnitude lies in 64 binades, [2^-51, 2^13) at first. What lies outside is sorted out element by
//     element: NaN has no mass, what is low enough to have none (-inf, the type's lowest value) need not be counted, and zeros
//     and "small" values below the 64 binades have four counters, one per kind and sign: they weigh the same to the last bit
//     while the maximum is far larger than they are or all of them are next to nothing (part_small_alike). A look at the row's
//     first elements moves the 64 binades for rows of large or of small values; if they turn out not to serve the row, it is
//     counted again with those that its maximum asks for, which always do.
//     The 64 binades end at 2^13 because of finite masks: 200 rows of 128256 columns, 90 % of them -1e4, 49 us, and 118 if these
//     are counted (one counter for all). One value of 1e-18 in each of 8 / 64 / 200 rows: 18 / 25 / 41 us, as
//     without it (31 / 31 / 59 by one CTA per row; 243 / 260 / 502 when such a row was searched by radix descent); zeros or NaN
//     in 1 % / 10 % of the places 62 / 49 us for 200 rows (70 / 66).
//   * A threshold among the small values, whose order their counters do not tell, is found by rank (part_select), and so is
//     the last kept element of a row in which nothing has a mass.
// [200, 128256] ~ N(0, 2), T = 1, top_p = 0.9: 58.4 us with one CTA per row, 41.2 us now: counting takes 31k cycles of an
// SM with three half rows, the rest is latency (searches, barriers, the draw).
// With 512 threads (40 registers each, three CTAs) the loops spilled: 46.8 us for 200 rows of 128256, 41.6 with 384; 320 41.9, 288 41.8.
constexpr int kPartThreads = 384, kPartWarps = kPartThreads / 32;
constexpr int kPartsPerCta = 2;
constexpr int kMaxPartCtas = 8;
constexpr int kPartBinades = 64;
constexpr int kPartMags = kPartBinades * 128;                        // magnitudes counted per sign
constexpr int kPartBase = (127 + 13 - kPartBinades) * 128;           // bits of the smallest of them: 2^-51
constexpr int kPartHistBytes = kPartMags * 2 * 2;
constexpr int kPartGroups = 2 * kPartMags / 32 + 1;                  // descending: positive values, small ones, negative values
constexpr int kPartSmallGroup = kPartMags / 32;
constexpr int kPartSmall = 4;                                        // small and positive, +0, -0, small and negative
constexpr int kPartMaxElems = 65535;                                 // of a sub-part: what a counter holds
constexpr int kNothing = 0x7FFFFFFF;                                 // below every counted value

constexpr int kPartMaxBlocks = kPartMaxElems / 256 + 3;              // of 256 elements, and the scalars at both ends

constexpr int kPartUnits = 2 * kPartMags / 128;                      // of 128 neighbouring counters

struct PartInfo {
  uint32_t max_key;             // 16-bit key of the largest element, 0 if there is no number
  uint32_t any_small;           // a nonzero value below the counted magnitudes
  uint32_t units[kPartUnits / 32];   // which units of counters are not empty
};
constexpr int kInfoWords = static_cast<int>(sizeof(PartInfo) / 4);
constexpr int kPartBins = kPartsPerCta * kPartHistBytes / 4;         // of part_select: 32-bit counters of four keys each
static_assert(kPartBins == 65536 / 4, "every key has a counter");

struct PartSmem {
  unsigned long long mass[kPartGroups];
  unsigned int cnt[kPartGroups];
  unsigned int small[kPartsPerCta][kPartSmall];
  PartInfo mine;
  PartInfo info[kMaxPartCtas];
  unsigned long long scan[kPartWarps];
  unsigned long long sub_mass[kMaxPartCtas * kPartsPerCta], sub_ties[kMaxPartCtas * kPartsPerCta];
  unsigned long long acc[kPartsPerCta];
  // result of a search
  unsigned long long above_cnt, above_mass, present;
  int group, sel;
  int owner, n_units;
  unsigned char units[kPartUnits];   // those of the row that are not empty
  uint32_t u24;
  uint32_t look[kPartWarps];
  unsigned long long target, ties_before;      // of the draw inside the owner's sub-part
  unsigned long long blocks[kPartMaxBlocks];   // ties << kTieShift | mass
  // part_select: elements in each CTA's slice of the bins, the bin that holds the rank and what lies above it, and
  // per sub-part the elements above that bin and those of its keys
  unsigned int slice[kMaxPartCtas], bin, above_bin, sel_above;
  uint32_t sel_key;
  unsigned int mine_keys[kPartsPerCta][5], keys[kMaxPartCtas * kPartsPerCta][5];
};
constexpr int kPartSmemBytes = kPartsPerCta * kPartHistBytes + static_cast<int>(sizeof(PartSmem));
static_assert(kPartGroups <= 2 * kPartThreads, "a thread sums two groups");

// Counted values in descending order: d = 0 .. kPartMags - 1 are the positive ones, then the four kinds of small ones (which
// all weigh what a zero does), then the negative ones.
__device__ __forceinline__ uint32_t part_bits(int d, uint32_t base) {
  if (d < kPartMags) return base + static_cast<uint32_t>(kPartMags - 1 - d);
  return d < kPartMags + kPartSmall ? (d == kPartMags + 2 ? 0x8000u : 0u)
                                    : 0x8000u + base + static_cast<uint32_t>(d - kPartMags - kPartSmall);
}
__device__ __forceinline__ uint32_t part_offset(int d) {             // of its counter; not for small ones
  return d < kPartMags ? static_cast<uint32_t>(kPartMags - 1 - d) * 2 : static_cast<uint32_t>(d - kPartSmall) * 2;
}
__device__ __forceinline__ int part_rank(uint32_t bits, uint32_t base) {   // d of the largest value
  const uint32_t mag = bits & 0x7FFFu;
  if (mag < base) return kPartMags;          // the first of the small ones
  return bits & 0x8000u ? kPartMags + kPartSmall + static_cast<int>(mag - base) : kPartMags - 1 - static_cast<int>(mag - base);
}
__device__ __forceinline__ uint32_t key16_of_bits(uint32_t bits) {        // NaN: 0
  return (bits & 0x7FFFu) > 0x7F80u ? 0u : (bits & 0x8000u ? 0xFFFFu - bits : bits + 0x8000u);
}
__device__ __forceinline__ float bits16_float(uint32_t bits) { return __uint_as_float(bits << 16); }
__device__ __forceinline__ unsigned long long bits16_mass(uint32_t bits, float inv_temp, float y_max) {
  return mass_fixed(exp_det(sub_rn(mul_rn(bits16_float(bits), inv_temp), y_max)));
}
__device__ __forceinline__ uint32_t ld_remote_u16(uint32_t a) {
  unsigned short v;
  asm volatile("ld.shared::cluster.u16 %0, [%1];" : "=h"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ uint32_t ld_remote_u32(uint32_t a) {
  uint32_t v;
  asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ uint2 ld_remote_u32x2(uint32_t a) {
  uint2 v;
  asm volatile("ld.shared::cluster.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ uint32_t map_addr(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}

// Sub-part q of n_sub in token order: scalars in front of the row's first 16-byte boundary (q = 0), whole vectors,
// scalars behind the last one (the last sub-part).
struct PartRange {
  int n_head;                   // scalars, from the row's start
  int first, n_vec;             // first element of the vectors, vectors
  int tail, n_tail;
};
__device__ __forceinline__ PartRange part_range(int q, int n_sub, int head, int v) {
  const int nvec = (v - head) / 8, per = (nvec + n_sub - 1) / n_sub;
  const int v0 = min(nvec, q * per), v1 = q == n_sub - 1 ? nvec : min(nvec, (q + 1) * per);
  PartRange r;
  r.n_head = q == 0 ? head : 0;
  r.first = head + 8 * v0;
  r.n_vec = v1 - v0;
  r.tail = head + 8 * nvec;
  r.n_tail = q == n_sub - 1 ? v - r.tail : 0;
  return r;
}

// The largest magnitude that can have a mass if the largest value is x, and the 64 binades up to it.
__device__ __forceinline__ float part_reach(float x, float inv_temp) {
  return fminf(fmaxf(fabsf(x), fabsf(x - 24.f / inv_temp)), 3.0e38f);
}
__device__ __forceinline__ uint32_t part_base(float reach) {
  const uint32_t top = min(((__float_as_uint(reach) >> 23) + 1u) << 7, 0x7F80u);
  return top > kPartMags ? top - kPartMags : 1u;
}

// Do all values below magnitude `base` weigh the same as a zero, to the last bit? They do if their weights have one
// argument, and if the arguments are so close to 0 that the weight is 1 (exp_det rounds to it below 2^-26).
__device__ __forceinline__ bool part_small_alike(uint32_t base, float inv_temp, float y_max) {
  const float y = mul_rn(bits16_float(base - 1), inv_temp);
  return sub_rn(y, y_max) == sub_rn(-y, y_max) || (fabsf(y) <= 0x1p-28f && fabsf(y_max) <= 0x1p-28f);
}

// Histogram of this CTA's sub-parts (zeroed before), its largest element, its small values.
__device__ __forceinline__ void part_count(const __nv_bfloat16* rp, int v, uint32_t base, int rank, int ctas, unsigned char* hist,
                                           PartSmem& s) {
  using T = __nv_bfloat16;
  // Vectors in flight per thread, us with two / three / four: 64 rows of 128256 27.3 / 25.6 / 25.6, 200 rows 41.4 / 41.2 / 42.3,
  // 256 rows 49.9 / 47.8 / 48.5; short rows do not care (256 x 8000: 18.2 / 18.4 / 18.5).
  constexpr int kTs = kPartThreads / kPartsPerCta, kU = 3;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, sub = tid / kTs, t = tid % kTs;
  static_assert(kTs % 32 == 0, "a warp works on one sub-part");
  const PartRange pr = part_range(rank * kPartsPerCta + sub, ctas * kPartsPerCta, row_head(rp, v), v);
  const int n_vec = pr.n_vec;
  unsigned char* mine = hist + sub * kPartHistBytes;
  uint32_t top = 0xFFFFFFFFu;
  uint32_t below2 = 0, below_pos2 = 0, zero2 = 0, zero_pos2 = 0;     // values below base, zeros; of both signs / positive ones
  auto count = [&](uint32_t a) {       // a: bits - base in the low half; a counter of 16 bits is half a word
    const uint32_t off = ((a << 1) & 0x3FFCu) | ((a >> 1) & 0x4000u);
    atomicAdd(reinterpret_cast<unsigned int*>(mine + off), max((a << 16) & 0x10000u, 1u));
  };
  // the same under a predicate: eight branches a vector cost more than the atomics
  const uint32_t mine_addr = static_cast<uint32_t>(__cvta_generic_to_shared(mine));
  auto count_if = [&](bool inside, uint32_t a) {
    const uint32_t off = ((a << 1) & 0x3FFCu) | ((a >> 1) & 0x4000u);
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %0, 0;\n\t@p red.shared.add.u32 [%1], %2;\n\t}" ::"r"(inside ? 1u : 0u),
                 "r"(mine_addr + off), "r"(max((a << 16) & 0x10000u, 1u))
                 : "memory");
  };
  const uint32_t base2 = (base + 1) * 0x00010001u;
  // per half of a word: 1 where the magnitude is below the limit (limit2: limit + 1 in both halves)
  auto below = [](uint32_t w, uint32_t limit2) { return __viaddmin_s16x2_relu(~w | 0x80008000u, limit2, 0x00010001u); };
  auto positive = [](uint32_t w, uint32_t ones) { return ones & ~(w >> 15); };
  auto note = [&](uint32_t w, uint32_t small) {
    const uint32_t zero = below(w, 0x00020002u);
    below2 += small;
    below_pos2 += positive(w, small);
    zero2 += zero;
    zero_pos2 += positive(w, zero);
  };
  const uint4* vp = reinterpret_cast<const uint4*>(rp + pr.first);
  for (int j0 = t - lane; j0 < n_vec; j0 += kTs * kU) {
    uint4 raw[kU];
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      const int j = j0 + kTs * u + lane;
      raw[u] = j < n_vec ? __ldg(vp + j) : make_uint4(~0u, ~0u, ~0u, ~0u);     // NaN: neither counted nor noted
    }
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      if (j0 + kTs * u >= n_vec) break;
      const uint32_t w[4] = {raw[u].x, raw[u].y, raw[u].z, raw[u].w};
      uint32_t a[8], out = 0;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        a[2 * i] = w[i] - base;
        a[2 * i + 1] = (w[i] >> 16) - base;
        out |= (a[2 * i] | a[2 * i + 1]) & 0x6000u;
      }
      top = Elem<T>::wmax(top, vec_max<T>(raw[u]));
      const bool have = j0 + kTs * u + lane < n_vec;
      if (__any_sync(0xffffffffu, have && out != 0) == 0) {     // one path for the warp: lanes apart would take both
        if (have) {
#pragma unroll
          for (int i = 0; i < 8; ++i) count(a[i]);
        }
      } else {
        uint32_t small[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) small[i] = below(w[i], base2);
#pragma unroll
        for (int i = 0; i < 8; ++i) count_if((a[i] & 0x6000u) == 0, a[i]);
        if (__any_sync(0xffffffffu, (small[0] | small[1] | small[2] | small[3]) != 0)) {
#pragma unroll
          for (int i = 0; i < 4; ++i) note(w[i], small[i]);
        }
      }
    }
  }
  // scalars in front of the first vector and behind the last one (fewer than eight each)
  const unsigned short* hp = reinterpret_cast<const unsigned short*>(rp);
  if (t < pr.n_head + pr.n_tail) {
    const uint32_t h = hp[t < pr.n_head ? t : pr.tail + (t - pr.n_head)] | 0xFFFF0000u;
    if (((h - base) & 0x6000u) == 0) count(h - base);
    note(h, below(h, base2));
    top = Elem<T>::wmax(top, h);
  }
  top = key16x2<T>(top);
  top = __reduce_max_sync(0xffffffffu, max(top >> 16, top & 0xFFFFu));
  auto total = [](uint32_t c) { return __reduce_add_sync(0xffffffffu, (c & 0xFFFFu) + (c >> 16)); };
  const unsigned int n_below = total(below2), n_pos = total(below_pos2), n_zero = total(zero2), n_zero_pos = total(zero_pos2);
  if (lane == 0) {
    atomicMax(&s.mine.max_key, top);
    if (n_below) {
      if (n_below != n_zero) s.mine.any_small = 1u;
      const unsigned int n[kPartSmall] = {n_pos - n_zero_pos, n_zero_pos, n_zero - n_zero_pos, n_below - n_pos - (n_zero - n_zero_pos)};
#pragma unroll
      for (int i = 0; i < kPartSmall; ++i)
        if (n[i]) atomicAdd(&s.small[sub][i], n[i]);
    }
  }
  __syncthreads();
  // which units of 128 counters are not empty
#pragma unroll 4
  for (int u = warp; u < kPartUnits; u += kPartWarps) {
    const uint2 c0 = *reinterpret_cast<const uint2*>(hist + u * 256 + lane * 8);
    const uint2 c1 = *reinterpret_cast<const uint2*>(hist + kPartHistBytes + u * 256 + lane * 8);
    if (__any_sync(0xffffffffu, (c0.x | c0.y | c1.x | c1.y) != 0) && lane == 0)
      atomicOr(&s.mine.units[u >> 5], 1u << (u & 31));
  }
}
static_assert(kPartsPerCta == 2, "both histograms of a CTA");

// Small values of one kind in the whole row.
__device__ __forceinline__ unsigned int part_smalls(int kind, int ctas, const PartSmem& s) {
  unsigned int n = 0;
#pragma unroll
  for (int r = 0; r < kMaxPartCtas; ++r)
    if (r < ctas)
#pragma unroll
      for (int sub = 0; sub < kPartsPerCta; ++sub) n += ld_remote_u32(map_to_cta(&s.small[sub][kind], r));
  return n;
}

__device__ __forceinline__ void part_barrier(int ctas) {
  if (ctas == 1) {
    __syncthreads();
  } else {
    cluster_arrive_release();
    cluster_wait_acquire();
  }
}

// The counted value that crosses `limit`, by count or by mass, from the prefix sums of this thread's two groups (what
// lies above them); s.sel = kNothing if none does. above_cnt is only valid if counts were summed.
__device__ void part_search(bool by_mass, unsigned long long limit, float inv_temp, float y_max, uint32_t base, int ctas,
                            unsigned long long pre_c, unsigned long long pre_m, uint32_t hist, PartSmem& s) {
  const int tid = threadIdx.x, lane = tid & 31, g0 = 2 * tid, g1 = g0 + 1;
  if (tid == 0) s.group = -1;
  __syncthreads();
  const unsigned long long c0 = g0 < kPartGroups ? s.cnt[g0] : 0, c1 = g1 < kPartGroups ? s.cnt[g1] : 0;
  const unsigned long long m0 = g0 < kPartGroups ? s.mass[g0] : 0, m1 = g1 < kPartGroups ? s.mass[g1] : 0;
  const unsigned long long pre = by_mass ? pre_m : pre_c, mid = pre + (by_mass ? m0 : c0), end = mid + (by_mass ? m1 : c1);
  if (pre <= limit && end > limit) {
    const bool second = mid <= limit;
    s.group = second ? g1 : g0;
    s.above_cnt = second ? pre_c + c0 : pre_c;
    s.above_mass = second ? pre_m + m0 : pre_m;
  }
  __syncthreads();
  const int g = s.group;
  if (g < 0) {
    if (tid == 0) s.sel = kNothing;
  } else if (tid < 32) {
    const bool small = g == kPartSmallGroup;
    const int d = (g <= kPartSmallGroup ? 32 * g : 32 * g - (32 - kPartSmall)) + lane;
    unsigned int n = 0;
    if (small) {
      if (lane < kPartSmall) n = part_smalls(lane, ctas, s);
    } else {
      const uint32_t a = hist + part_offset(d);
#pragma unroll
      for (int r = 0; r < kMaxPartCtas; ++r)
        if (r < ctas)
#pragma unroll
          for (int sub = 0; sub < kPartsPerCta; ++sub) n += ld_remote_u16(map_addr(a + sub * kPartHistBytes, r));
    }
    const unsigned long long kc = n, km = n ? n * bits16_mass(part_bits(d, base), inv_temp, y_max) : 0ull;
    const unsigned long long ic = warp_incl_u64(kc), im = warp_incl_u64(km);
    const unsigned long long above_c = s.above_cnt, above_m = s.above_mass;
    const bool crosses = by_mass ? above_m + im > limit : above_c + ic > limit;
    const int first = __ffs(static_cast<int>(__ballot_sync(0xffffffffu, crosses))) - 1;
    if (lane == first) {
      s.sel = d;
      s.above_cnt = above_c + ic - kc;
      s.above_mass = above_m + im - km;
      s.present = kc;
    }
  }
  __syncthreads();
}

// First element of the sub-part, in token-id order, whose cumulative kept mass exceeds s.target. The kept mass of every
// 256 elements (a vector per lane) is summed, order-free, and the block that holds the target is walked by one warp,
// so the sub-part is read once and that block again.
template <int kMode>
__device__ __forceinline__ void part_draw(const __nv_bfloat16* rp, const PartRange& r, const Kept& k, PartSmem& s, int* out) {
  using T = __nv_bfloat16;
  constexpr int kU = 4;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned short* hp = reinterpret_cast<const unsigned short*>(rp);
  const uint4* vp = reinterpret_cast<const uint4*>(rp + r.first);
  const int n_blocks = (r.n_vec + 31) / 32;
  const float y_max = -k.args.neg_y_max;
  auto mass_of = [&](uint32_t h) {         // ties << kTieShift | mass
    const uint32_t key = float_to_key(bits16_float(h));
    if (kMode != kAll && key <= k.tau) return key == k.tau ? 1ull << kTieShift : 0ull;
    if (kMode == kByCount) return 1ull;
    return static_cast<unsigned long long>(mass_fixed(exp_det(sub_rn(mul_rn(key_to_float(key), k.args.inv_temp), y_max))));
  };
  const int tau_o = static_cast<int>(k.tau ^ 0x80000000u);
  auto take_word = [&](uint32_t w, unsigned long long& m) {
    if constexpr (kMode == kByTable) {
      const uint32_t not_key = ~(w ^ (((w >> 15) & 0x00010001u) * 0x7FFFu));
      const uint32_t i2 = __viaddmin_u16x2(not_key, k.top2, k.last2);
      m += k.table[i2 & 0xFFFFu];
      m += k.table[i2 >> 16];
    } else if constexpr (kMode == kByCount) {
      m += mass_of(w & 0xFFFFu) + mass_of(w >> 16);
    } else {
      float x0 = __uint_as_float(w << 16), x1 = __uint_as_float(w & 0xFFFF0000u);
      if constexpr (kMode != kAll) {
        auto ordered = [](float x) {
          const int b = __float_as_int(x);
          return b ^ ((b >> 31) & 0x7FFFFFFF);
        };
        const int o0 = ordered(x0), o1 = ordered(x1);
        m += static_cast<unsigned long long>((o0 == tau_o ? 1u : 0u) + (o1 == tau_o ? 1u : 0u)) << kTieShift;
        x0 = o0 > tau_o ? x0 : __uint_as_float(0xFF800000u);
        x1 = o1 > tau_o ? x1 : __uint_as_float(0xFF800000u);
      }
      mass_pair(x0, x1, k.args, m);
    }
  };
#pragma unroll 1
  for (int b0 = warp; b0 < n_blocks; b0 += kPartWarps * kU) {
    uint4 raw[kU];
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      const int j = (b0 + u * kPartWarps) * 32 + lane;
      if (j < r.n_vec) raw[u] = __ldg(vp + j);
    }
    unsigned long long m[kU] = {};
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      if ((b0 + u * kPartWarps) * 32 + lane < r.n_vec) {
        take_word(raw[u].x, m[u]);
        take_word(raw[u].y, m[u]);
        take_word(raw[u].z, m[u]);
        take_word(raw[u].w, m[u]);
      }
    }
    // the sums of four blocks together: lanes 8 i .. 8 i + 7 end up with block i's
    static_assert(kU == 4, "two exchanges of halves");
    const bool hi = lane & 16, odd = lane & 8;
    unsigned long long a = (hi ? m[2] : m[0]) + __shfl_xor_sync(0xffffffffu, hi ? m[0] : m[2], 16);
    unsigned long long c = (hi ? m[3] : m[1]) + __shfl_xor_sync(0xffffffffu, hi ? m[1] : m[3], 16);
    a = (odd ? c : a) + __shfl_xor_sync(0xffffffffu, odd ? a : c, 8);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    const int b = b0 + (lane >> 3) * kPartWarps;
    if ((lane & 7) == 0 && b < n_blocks) s.blocks[1 + b] = a;
  }
  if (warp >= kPartWarps - 2) {            // the scalars at the ends: first and last block
    const bool last = warp == kPartWarps - 1;
    const unsigned long long m =
        warp_sum_u64(last ? (lane < r.n_tail ? mass_of(hp[r.tail + lane]) : 0ull) : (lane < r.n_head ? mass_of(hp[lane]) : 0ull));
    if (lane == 0) s.blocks[last ? 1 + n_blocks : 0] = m;
  }
  __syncthreads();
  if (warp != 0) return;
  const int n = n_blocks + 2, per = (n + 31) / 32;
  constexpr unsigned long long kMassMask = (1ull << kTieShift) - 1;
  unsigned long long target = s.target, t0 = s.ties_before;
  int sel = -1;
  {
    // ties in front of this lane's blocks, then their kept mass
    const int e0 = min(n, lane * per), e1 = min(n, e0 + per);
    unsigned long long ties = 0, mass = 0;
    for (int e = e0; e < e1; ++e) ties += s.blocks[e] >> kTieShift;
    unsigned long long t = t0 + warp_incl_u64(ties) - ties;
    const unsigned long long t_lane = t;
    auto kept = [&](unsigned long long m) {
      const unsigned long long left = k.tie_keep > t ? k.tie_keep - t : 0ull, here = m >> kTieShift;
      t += here;
      return (m & kMassMask) + (here < left ? here : left) * k.q_tau;
    };
    for (int e = e0; e < e1; ++e) mass += kept(s.blocks[e]);
    const unsigned long long inc = warp_incl_u64(mass);
    const int first = __ffs(static_cast<int>(__ballot_sync(0xffffffffu, inc > target))) - 1;
    unsigned long long before = inc - mass;
    if (lane == first) {
      t = t_lane;
      for (int e = e0; e < e1; ++e) {
        const unsigned long long tb = t, m = kept(s.blocks[e]);
        if (before + m > target) {
          sel = e;
          t0 = tb;
          break;
        }
        before += m;
      }
    }
    if (first < 0) return;                 // cannot happen: the sub-part holds the target
    sel = __shfl_sync(0xffffffffu, sel, first);
    t0 = __shfl_sync(0xffffffffu, t0, first);
    target -= __shfl_sync(0xffffffffu, before, first);
  }
  // the block: eight elements per lane, or a scalar
  uint32_t w[4] = {0u, 0u, 0u, 0u};
  int have = 0, i0;
  if (sel == 0 || sel == n - 1) {
    const bool last = sel != 0;
    i0 = (last ? r.tail : 0) + lane;
    if (lane < (last ? r.n_tail : r.n_head)) {
      w[0] = hp[i0];
      have = 1;
    }
  } else {
    const int j = (sel - 1) * 32 + lane;
    i0 = r.first + 8 * j;
    if (j < r.n_vec) {
      const uint4 raw = __ldg(vp + j);
      w[0] = raw.x;
      w[1] = raw.y;
      w[2] = raw.z;
      w[3] = raw.w;
      have = 8;
    }
  }
  unsigned long long q[8], ties = 0;
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    q[e] = e < have ? mass_of((w[e >> 1] >> (16 * (e & 1))) & 0xFFFFu) : 0ull;
    ties += q[e] >> kTieShift;
  }
  unsigned long long rank = t0 + warp_incl_u64(ties) - ties, mass = 0;
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    if (q[e] >> kTieShift) {
      q[e] = rank < k.tie_keep ? k.q_tau : 0ull;
      ++rank;
    }
    mass += q[e];
  }
  const unsigned long long inc = warp_incl_u64(mass);
  const int first = __ffs(static_cast<int>(__ballot_sync(0xffffffffu, inc > target))) - 1;
  if (lane == first) {
    unsigned long long acc = inc - mass;
    int at = -1;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      acc += q[e];
      if (at < 0 && acc > target) at = e;
    }
    *out = i0 + at;
  }
}

// The sub-part that holds s.target of the kept mass, from s.sub_mass and s.sub_ties; the target and the ties in front inside it.
// By one warp.
__device__ __forceinline__ void part_owner(int n_sub, const Kept& k, unsigned long long target, PartSmem& s) {
  const int lane = threadIdx.x & 31;
  const unsigned long long t = lane < n_sub ? s.sub_ties[lane] : 0ull, t0 = warp_incl_u64(t) - t;
  const unsigned long long left = k.tie_keep > t0 ? k.tie_keep - t0 : 0ull;
  const unsigned long long m = (lane < n_sub ? s.sub_mass[lane] : 0ull) + (t < left ? t : left) * k.q_tau;
  const unsigned long long inc = warp_incl_u64(m);
  const int first = __ffs(static_cast<int>(__ballot_sync(0xffffffffu, inc > target))) - 1;
  if (lane == first) {
    s.owner = first;
    s.target = target - (inc - m);
    s.ties_before = t0;
  }
}

// By rank: the key of the n-th largest of the row's elements whose 16-bit keys lie in [lo, hi] (there are that many), and
// how many of these elements lie above that key. s.sub_mass gets, per sub-part, `each` for every one of them on top of what
// it holds, s.sub_ties the elements of that key. Out of line, by all CTAs of the row: bins of four keys, of which each
// CTA adds up a slice, then a look at the four keys of the bin that holds the rank. The histograms are overwritten.
// What bounds it is its instructions, two passes of about 15 per element, and no earnest row comes here: half of the values
// nonzero and below 2^-51, us, one CTA of 1024 threads per row / here: 8 rows of 128256 34.6 / 36.8, 64 rows 35.2 / 70.7, 200 rows
// 65.9 / 128; rows with an infinity, k = 2000: 148 / 40, 150 / 64, 296 / 116.
__device__ __noinline__ void part_select(const __nv_bfloat16* rp, int v, int rank, int ctas, uint32_t lo, uint32_t hi, unsigned int n,
                                         unsigned long long each, unsigned int* bins, PartSmem& s) {
  constexpr int kTs = kPartThreads / kPartsPerCta;
  const int tid = threadIdx.x, lane = tid & 31, sub = tid / kTs, t = tid % kTs;
  const PartRange pr = part_range(rank * kPartsPerCta + sub, ctas * kPartsPerCta, row_head(rp, v), v);
  const uint4* vp = reinterpret_cast<const uint4*>(rp + pr.first);
  const unsigned short* hp = reinterpret_cast<const unsigned short*>(rp);
  auto each_key = [&](auto&& f) {        // keys of this thread's elements that lie in [lo, hi]
    auto one = [&](uint32_t h) {
      const uint32_t key = key16_of_bits(h);
      if (key >= lo && key <= hi) f(key);
    };
    for (int j = t; j < pr.n_vec; j += kTs) {
      const uint4 raw = __ldg(vp + j);
      const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        one(w[i] & 0xFFFFu);
        one(w[i] >> 16);
      }
    }
    if (t < pr.n_head + pr.n_tail) one(hp[t < pr.n_head ? t : pr.tail + (t - pr.n_head)]);
  };
  part_barrier(ctas);                    // nobody reads the histograms any more
  for (int i = tid; i < kPartBins / 4; i += kPartThreads) reinterpret_cast<uint4*>(bins)[i] = make_uint4(0u, 0u, 0u, 0u);
  if (tid < kPartsPerCta * 5) s.mine_keys[tid / 5][tid % 5] = 0;
  __syncthreads();
  each_key([&](uint32_t key) { atomicAdd(&bins[key >> 2], 1u); });
  part_barrier(ctas);
  // this CTA's slice: bins top - from ... top - (to - 1), each thread a run of them, summed over the row's CTAs
  const int top = static_cast<int>(hi >> 2), n_bins = top - static_cast<int>(lo >> 2) + 1, per = (n_bins + ctas - 1) / ctas;
  const int from = min(n_bins, rank * per), to = min(n_bins, from + per), run = (to - from + kPartThreads - 1) / kPartThreads;
  const int b0 = min(to, from + tid * run), b1 = min(to, b0 + run);
  auto bin_sum = [&](int b) {
    unsigned int c = 0;
#pragma unroll
    for (int r = 0; r < kMaxPartCtas; ++r)
      if (r < ctas) c += ld_remote_u32(map_to_cta(bins + (top - b), r));
    return c;
  };
  unsigned int mine = 0;
  for (int b = b0; b < b1; ++b) mine += bin_sum(b);
  unsigned long long all;
  unsigned long long before = block_exscan_u64(mine, s.scan, all);
  if (tid < ctas) st_remote_u32(map_to_cta(&s.slice[rank], tid), static_cast<unsigned int>(all));
  part_barrier(ctas);
  for (int r = 0; r < rank; ++r) before += s.slice[r];
  if (before < n && n <= before + mine) {
    for (int b = b0; b < b1; ++b) {
      const unsigned int c = bin_sum(b);
      if (n <= before + c) {
        for (int r = 0; r < ctas; ++r) {
          st_remote_u32(map_to_cta(&s.bin, r), static_cast<uint32_t>(top - b));
          st_remote_u32(map_to_cta(&s.above_bin, r), static_cast<uint32_t>(before));
        }
        break;
      }
      before += c;
    }
  }
  part_barrier(ctas);
  const uint32_t bin = s.bin;
  unsigned int c[5] = {0, 0, 0, 0, 0};   // above the bin, then its keys from the top
  each_key([&](uint32_t key) {
    c[0] += (key >> 2) > bin ? 1u : 0u;
#pragma unroll
    for (int i = 0; i < 4; ++i) c[1 + i] += key == 4 * bin + 3 - i ? 1u : 0u;
  });
#pragma unroll
  for (int i = 0; i < 5; ++i) {
    c[i] = __reduce_add_sync(0xffffffffu, c[i]);
    if (lane == 0 && c[i]) atomicAdd(&s.mine_keys[sub][i], c[i]);
  }
  __syncthreads();
  if (tid < ctas * kPartsPerCta * 5) {
    const int to_cta = tid / (kPartsPerCta * 5), at = tid % (kPartsPerCta * 5);
    st_remote_u32(map_to_cta(&s.keys[rank * kPartsPerCta + at / 5][at % 5], to_cta), s.mine_keys[at / 5][at % 5]);
  }
  part_barrier(ctas);
  unsigned int above = s.above_bin;
  int at = 0;
  for (;; ++at) {                        // the key of the four that holds the rank
    unsigned int here = 0;
    for (int q = 0; q < ctas * kPartsPerCta; ++q) here += s.keys[q][1 + at];
    if (at == 3 || n <= above + here) break;
    above += here;
  }
  if (tid == 0) {
    s.sel_key = 4 * bin + 3 - at;
    s.sel_above = above;
  }
  if (tid < ctas * kPartsPerCta) {
    unsigned int kept = 0;
    for (int i = 0; i <= at; ++i) kept += s.keys[tid][i];
    s.sub_mass[tid] += kept * each;
    s.sub_ties[tid] = s.keys[tid][1 + at];
  }
  __syncthreads();
}

// The draw where the kept elements end among the small ones of one sign, of which the first n by rank are kept: the rest of
// the kernel, with q the mass of a small value and s.sub_mass what is kept above them.
__device__ __noinline__ void part_draw_small(const __nv_bfloat16* rp, int v, int rank, int ctas, uint32_t base, bool neg, unsigned int n,
                                             unsigned long long q, MassArgs args, unsigned long long target, unsigned int* bins,
                                             PartSmem& s, int* out) {
  part_select(rp, v, rank, ctas, neg ? 0x8000u - base : 0x8001u, neg ? 0x7FFEu : 0x7FFFu + base, n, q, bins, s);
  Kept k;
  k.tau = float_to_key(key16_float<__nv_bfloat16>(s.sel_key));
  k.tie_keep = n - s.sel_above;
  k.q_tau = q;
  k.args = args;
  const int n_sub = ctas * kPartsPerCta;
  if (threadIdx.x < 32) part_owner(n_sub, k, target, s);
  __syncthreads();
  if (s.owner / kPartsPerCta != rank) return;
  part_draw<kByExp>(rp, part_range(s.owner, n_sub, row_head(rp, v), v), k, s, out);
}

// A row in which nothing has a mass (its maximum is infinite or there is no number): the last of its top_k largest elements in
// token-id order.
__device__ __noinline__ void part_last(const __nv_bfloat16* rp, int v, int rank, int ctas, int top_k, unsigned int* bins,
                                       PartSmem& s, int* out) {
  const int n_sub = ctas * kPartsPerCta;
  if (threadIdx.x < n_sub) s.sub_mass[threadIdx.x] = 0;
  part_select(rp, v, rank, ctas, 0u, 0xFFFFu, static_cast<unsigned int>(top_k), 1ull, bins, s);
  Kept k;
  k.tau = s.sel_key == 0 ? 0u : float_to_key(key16_float<__nv_bfloat16>(s.sel_key));
  k.tie_keep = static_cast<unsigned int>(top_k) - s.sel_above;
  k.q_tau = 1;
  k.args = {0.f, 0.f};
  if (threadIdx.x < 32) part_owner(n_sub, k, static_cast<unsigned long long>(top_k) - 1, s);
  __syncthreads();
  if (s.owner / kPartsPerCta != rank) return;
  part_draw<kByCount>(rp, part_range(s.owner, n_sub, row_head(rp, v), v), k, s, out);
}

__global__ void __launch_bounds__(kPartThreads, 3)
sample_parts_kernel(const __nv_bfloat16* __restrict__ logits, long long row_stride, int v,
                    const long long* __restrict__ row_ids, float inv_temp, int top_k, float top_p, unsigned long long seed,
                    unsigned long long step, int ctas, int* __restrict__ out) {
  using T = __nv_bfloat16;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  unsigned char* hist = smem_raw;
  PartSmem& s = *reinterpret_cast<PartSmem*>(smem_raw + kPartsPerCta * kPartHistBytes);
  const uint32_t hist_addr = static_cast<uint32_t>(__cvta_generic_to_shared(hist));
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int rank = static_cast<int>(cluster_rank()), row = static_cast<int>(blockIdx.x) / ctas;
  const T* rp = logits + static_cast<long long>(row) * row_stride;
  const bool has_k = top_k > 0 && top_k < v;
  if (ctas > 1) cluster_arrive_release();          // waited for before the first remote access

  // a look at the row's first 8 * kPartThreads elements, for the magnitudes to count
  uint32_t look = 0xFFFFFFFFu;
  {
    const int head = row_head(rp, v);
    if (tid < (v - head) / 8) look = vec_max<T>(__ldg(reinterpret_cast<const uint4*>(rp + head) + tid));
  }
  // ---- count; the largest element and what was left out are known to all CTAs of the row behind the barrier
  uint32_t base = kPartBase;
  float y_max = 0.f;
  uint32_t max_key = 0, max_bits = 0;
#pragma unroll 1
  for (int attempt = 0;; ++attempt) {
    for (int i = tid; i < kPartsPerCta * kPartHistBytes / 16; i += kPartThreads)
      reinterpret_cast<uint4*>(hist)[i] = make_uint4(0u, 0u, 0u, 0u);
    for (int i = tid; i < kPartGroups; i += kPartThreads) {
      s.mass[i] = 0;
      s.cnt[i] = 0;
    }
    if (tid < kPartsPerCta * kPartSmall) s.small[tid / kPartSmall][tid % kPartSmall] = 0;
    if (tid < kPartsPerCta) s.acc[tid] = 0;
    if (tid < kInfoWords) reinterpret_cast<uint32_t*>(&s.mine)[tid] = 0;
    if (attempt == 0) {
      look = Elem<T>::wmax(look, __byte_perm(look, 0, 0x1032));
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) look = Elem<T>::wmax(look, __shfl_xor_sync(0xffffffffu, look, o));
      if (lane == 0) s.look[warp] = look | 0xFFFF0000u;
    }
    __syncthreads();
    if (attempt == 0) {
      uint32_t m = 0xFFFFFFFFu;
#pragma unroll
      for (int w = 0; w < kPartWarps; ++w) m = Elem<T>::wmax(m, s.look[w]);
      const float x = bits16_float(m & 0xFFFFu), reach = 2.f * part_reach(x, inv_temp);
      if (reach >= 0x1p13f && reach < 1e38f) base = part_base(reach);     // no number, an infinity: as usual
      if (x > 0.f && x < 0x1p-51f) base = part_base(4.f * x);
    }
    part_count(rp, v, base, rank, ctas, hist, s);
    __syncthreads();
    if (attempt == 0 && ctas > 1) cluster_wait_acquire();            // every CTA of the cluster runs
    if (tid < ctas * kInfoWords)
      st_remote_u32(map_to_cta(reinterpret_cast<uint32_t*>(&s.info[rank]) + tid % kInfoWords, tid / kInfoWords),
                    reinterpret_cast<const uint32_t*>(&s.mine)[tid % kInfoWords]);
    if (tid == kPartThreads - 1)
      s.u24 = uniform_u24(seed, row_ids ? static_cast<unsigned long long>(row_ids[row]) : static_cast<unsigned long long>(row), step);
    part_barrier(ctas);
    bool small = false;
    max_key = 0;
    for (int r = 0; r < ctas; ++r) {
      small |= s.info[r].any_small != 0;
      max_key = max(max_key, s.info[r].max_key);
    }
    max_bits = max_key == 0 ? 0x7FFFu : (max_key & 0x8000u ? max_key & 0x7FFFu : 0xFFFFu - max_key);
    const float x_max = bits16_float(max_bits);
    y_max = mul_rn(x_max, inv_temp);
    if (!(fabsf(y_max) <= 3.402823466e38f)) {
      // no number, or an infinite one: nothing has a mass, the last kept element is the answer
      if (has_k)
        part_last(rp, v, rank, ctas, top_k, reinterpret_cast<unsigned int*>(hist), s, out + row);
      else if (rank == 0 && tid == 0)
        out[row] = v - 1;
      return;
    }
    if (attempt > 0) break;              // the second 64 binades serve every row
    // What the first ones may miss: the largest value; values below all of them that have a mass, which is 0 below
    // 2^-33 of the maximum's (2^-32 is the smallest that counts); small values that weigh other than a zero
    const uint32_t max_mag = max_bits & 0x7FFFu;
    const float lowest = -bits16_float(base + kPartMags);
    const bool big = max_mag >= base + kPartMags, low = (lowest * inv_temp - y_max) * 1.4426950408889634f > -33.f;
    const bool differ = small && !part_small_alike(base, inv_temp, y_max);
    if (!big && !low && !differ) break;
    base = part_base(part_reach(x_max, inv_temp));
    part_barrier(ctas);               // s.info is written again
  }

  // ---- masses of the groups: units of four groups are dealt over the CTAs, whose sums go to all of them
  if (tid < kPartUnits) {
    unsigned int before = 0, word = 0;
#pragma unroll
    for (int i = 0; i < kPartUnits / 32; ++i) {
      unsigned int w = 0;
      for (int r = 0; r < ctas; ++r) w |= s.info[r].units[i];
      if (i < warp) before += __popc(w);
      if (i == warp) word = w;
    }
    if (word >> lane & 1u) s.units[before + __popc(word & ((1u << lane) - 1u))] = static_cast<unsigned char>(tid);
    if (tid == kPartUnits - 1) s.n_units = before + __popc(word);
  }
  __syncthreads();
#pragma unroll 1
  for (int i = rank + ctas * warp; i < s.n_units; i += ctas * kPartWarps) {
    const int u = s.units[i];
    const int at = u * 128 + lane * 4;                      // four neighbours' counters, in rising order of magnitude
    unsigned int n[4] = {0, 0, 0, 0};
#pragma unroll 1
    for (int r0 = 0; r0 < ctas; r0 += 4) {                  // four CTAs' counters in flight
      uint2 c[4 * kPartsPerCta];
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int sub = 0; sub < kPartsPerCta; ++sub) {
          c[r * kPartsPerCta + sub] = make_uint2(0u, 0u);
          if (r0 + r < ctas)
            c[r * kPartsPerCta + sub] =
                ld_remote_u32x2(map_addr(hist_addr + static_cast<uint32_t>(at) * 2 + sub * kPartHistBytes, r0 + r));
        }
#pragma unroll
      for (int i = 0; i < 4 * kPartsPerCta; ++i) {
        n[0] += c[i].x & 0xFFFFu;
        n[1] += c[i].x >> 16;
        n[2] += c[i].y & 0xFFFFu;
        n[3] += c[i].y >> 16;
      }
    }
    unsigned int cnt = n[0] + n[1] + n[2] + n[3];
    const bool neg = at >= kPartMags;
    const uint32_t bits = neg ? 0x8000u + base + static_cast<uint32_t>(at - kPartMags) : base + static_cast<uint32_t>(at);
    unsigned long long m = 0;
#pragma unroll
    for (int e = 0; e < 4; ++e) m += n[e] * bits16_mass(bits + e, inv_temp, y_max);
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) {
      m += __shfl_xor_sync(0xffffffffu, m, o);
      cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
    }
    const int g = neg ? kPartSmallGroup + 1 + (at - kPartMags) / 32 : kPartSmallGroup - 1 - at / 32;
    if ((lane & 7) < ctas && cnt) {
      st_remote_u64(map_to_cta(&s.mass[g], lane & 7), m);
      st_remote_u32(map_to_cta(&s.cnt[g], lane & 7), cnt);
    }
  }
  if (rank == 0 && warp == kPartWarps - 1) {
    const unsigned int n = __reduce_add_sync(0xffffffffu, lane < kPartSmall ? part_smalls(lane, ctas, s) : 0u);
    if (lane < ctas && n) {
      st_remote_u64(map_to_cta(&s.mass[kPartSmallGroup], lane), n * bits16_mass(0u, inv_temp, y_max));
      st_remote_u32(map_to_cta(&s.cnt[kPartSmallGroup], lane), n);
    }
  }
  part_barrier(ctas);

  // ---- where the kept prefix ends, in every CTA: the same decisions as in sample_general_kernel
  int tau = kNothing;
  unsigned long long tie_keep = ~0ull, kept_mass;
  {
    const int g0 = 2 * tid, g1 = g0 + 1;
    unsigned long long pre_c = 0, tot_c;
    const unsigned long long pre_m = block_exscan_u64((g0 < kPartGroups ? s.mass[g0] : 0ull) + (g1 < kPartGroups ? s.mass[g1] : 0ull),
                                                      s.scan, kept_mass);
    if (has_k) {
      pre_c = block_exscan_u64((g0 < kPartGroups ? s.cnt[g0] : 0u) + (g1 < kPartGroups ? s.cnt[g1] : 0u), s.scan, tot_c);
      // if fewer elements than that are counted, every element with a mass is among the k largest
      part_search(false, static_cast<unsigned long long>(top_k - 1), inv_temp, y_max, base, ctas, pre_c, pre_m, hist_addr, s);
      if (s.sel != kNothing) {
        tau = s.sel;
        tie_keep = static_cast<unsigned long long>(top_k) - s.above_cnt;
        kept_mass = s.above_mass + tie_keep * bits16_mass(part_bits(tau, base), inv_temp, y_max);
      }
    }
    if (top_p < 1.0f) {
      const unsigned long long limit = mass_fraction(static_cast<double>(top_p), kept_mass);
      __syncthreads();
      part_search(true, limit, inv_temp, y_max, base, ctas, pre_c, pre_m, hist_addr, s);
      if (s.sel != kNothing) {
        const int p_tau = s.sel;
        const unsigned long long q = bits16_mass(part_bits(p_tau, base), inv_temp, y_max);   // not 0: it crosses
        const unsigned long long p_ties = (limit - s.above_mass) / q + 1;
        if (p_tau != tau ? p_tau < tau : p_ties < tie_keep) {
          tau = p_tau;
          tie_keep = p_ties < s.present ? p_ties : s.present;
          kept_mass = s.above_mass + tie_keep * q;
        }
      }
    }
  }

  // small values without a mass: everything that has one is kept
  const bool among_small = tau == kPartMags || tau == kPartMags + kPartSmall - 1;
  const unsigned long long q_small = among_small ? bits16_mass(0u, inv_temp, y_max) : 0ull;
  if (among_small && q_small == 0) tau = kNothing;

  // ---- kept mass and ties of this CTA's sub-parts, from their histograms
  {
    unsigned long long m[kPartsPerCta] = {};
    const int d_end = min(tau, 2 * kPartMags + kPartSmall);
#pragma unroll 1
    for (int i = part_rank(max_bits, base) + tid; i < d_end; i += kPartThreads) {
      unsigned int n[kPartsPerCta], any = 0;
      const bool small = i >= kPartMags && i < kPartMags + kPartSmall;
#pragma unroll
      for (int sub = 0; sub < kPartsPerCta; ++sub) {
        n[sub] = small ? s.small[sub][i - kPartMags]
                       : *reinterpret_cast<const unsigned short*>(hist + sub * kPartHistBytes + part_offset(i));
        any |= n[sub];
      }
      if (any == 0) continue;
      const unsigned long long q = bits16_mass(part_bits(i, base), inv_temp, y_max);
#pragma unroll
      for (int sub = 0; sub < kPartsPerCta; ++sub) m[sub] += n[sub] * q;
    }
#pragma unroll
    for (int sub = 0; sub < kPartsPerCta; ++sub) {
      m[sub] = warp_sum_u64(m[sub]);
      if (lane == 0 && m[sub]) atomicAdd(&s.acc[sub], m[sub]);
    }
    __syncthreads();
    if (tid < ctas * kPartsPerCta) {
      const int to = tid / kPartsPerCta, sub = tid % kPartsPerCta, q = rank * kPartsPerCta + sub;
      unsigned long long ties = 0;
      if (tau != kNothing)
        ties = tau >= kPartMags && tau < kPartMags + kPartSmall
                   ? s.small[sub][tau - kPartMags]
                   : *reinterpret_cast<const unsigned short*>(hist + sub * kPartHistBytes + part_offset(tau));
      st_remote_u64(map_to_cta(&s.sub_mass[q], to), s.acc[sub]);
      st_remote_u64(map_to_cta(&s.sub_ties[q], to), ties);
    }
    part_barrier(ctas);
  }

  // ---- the sub-part that holds the target; its CTA draws, nobody reads another CTA's memory any more
  Kept k;
  const uint32_t tau_bits = tau == kNothing ? 0u : part_bits(tau, base);
  const uint32_t tau16 = tau == kNothing ? 0u : key16_of_bits(tau_bits);
  if (q_small != 0) {
    part_draw_small(rp, v, rank, ctas, base, tau != kPartMags, static_cast<unsigned int>(tie_keep), q_small, {inv_temp, -y_max},
                    mass_scale_u24(s.u24, kept_mass), reinterpret_cast<unsigned int*>(hist), s, out + row);
    return;
  }
  k.tau = tau == kNothing ? 0u : float_to_key(key16_float<T>(tau16));
  k.tie_keep = tau == kNothing ? 0ull : tie_keep;
  k.q_tau = tau == kNothing ? 0ull : bits16_mass(tau_bits, inv_temp, y_max);
  k.args = {inv_temp, -y_max};
  const int n_sub = ctas * kPartsPerCta;
  if (warp == 0) part_owner(n_sub, k, mass_scale_u24(s.u24, kept_mass), s);
  __syncthreads();
  const int q = s.owner;
  if (q / kPartsPerCta != rank) return;
  const PartRange r = part_range(q, n_sub, row_head(rp, v), v);
  if (tau == kNothing) {
    part_draw<kAll>(rp, r, k, s, out + row);
    return;
  }
  const uint32_t range = max_key - tau16;
  unsigned long long* table = reinterpret_cast<unsigned long long*>(hist);
  if (range + 2 <= kPartsPerCta * kPartHistBytes / 8) {
    for (uint32_t i = tid; i < range; i += kPartThreads) table[i] = key16_mass_of<T>(max_key - i, inv_temp, y_max);
    if (tid == 0) {
      table[range] = 1ull << kTieShift;
      table[range + 1] = 0;
    }
    k.table = table;
    k.top2 = ((max_key + 0x8001u) & 0xFFFFu) * 0x00010001u;
    k.last2 = (range + 1) * 0x00010001u;
    __syncthreads();
    part_draw<kByTable>(rp, r, k, s, out + row);
    return;
  }
  part_draw<kByExp>(rp, r, k, s, out + row);
}

// How many CTAs share a row, 0 for the one of 1024 threads that counts and draws by itself. Counting is bound by the
// atomics an SM can do, so more CTAs than SMs help only to deal rows that do not fill a whole number of rounds, and what is behind the
// counting (searches, two barriers of the cluster, the draw: 14 us) is paid by any number of CTAs. us, top_p = 0.9, the CTA
// of 1024 threads / one / two / four / eight CTAs:
//   128256 columns, rows of 9: 29.2 / 31.5 / 22.5 / 18.4 / 16.7; 18: 29.4 / 31.4 / 22.6 / 18.4 / 19.0; 37: 29.4 / 31.8 / 22.9 / 21.8;
//     64: 30.1 / 36.3 / 25.4 / 23.9; 100: 31.1 / 36.9 / 31.4; 148: 31.5 / 37.3 / 32.0. So as many as leave an eighth of the SMs free, and from
//     65 rows on the one of 1024 (two would still win up to 74, 30.3 / 25.9).
//   8 rows, four or eight CTAs only in rows of 28672 columns and more: 16384 13.7 / 14.5 (eight), 24576 14.9 / 15.0, 28672 15.3 / 15.0,
//     32000 15.7 / 15.0, 49152 18.2 / 15.5. 64 rows, two CTAs only from 49152 on: 32000 15.7 / 16.7, 40960 17.1 / 17.1, 49152 18.5 / 17.7.
//   More rows than SMs: the CTA of 1024 threads needs another round, parts have them all resident, three per SM. 149 rows of 128256
//     56.6 / 45.9 / 39.9; 222 58.9 / 47.3 / 41.4; 223, where two CTAs per row are more than three per SM, 58.9 / 47.1 / 54.8; 200 rows of 4096
//     22.9 / 16.7 / 18.8, 28672 29.4 / 23.3 / 23.3, 49152 36.6 / 29.3 / 27.9, 65536 40.6 / 33.1 / 31.1: two from 65536 on, which leaves
//     1 to 2 us between 32000 and there.
inline int part_ctas(int rows, int v, int sms) {
  // a sub-part's vectors are rounded up, its ends have up to seven scalars each
  auto fits = [&](int ctas) { return v / (ctas * kPartsPerCta) + 32 <= kPartMaxElems; };
  int ctas = 1;
  if (rows > sms) {
    if (v >= 65536 && 2ll * rows <= 3ll * sms) ctas = 2;
  } else {
    // an eighth of the SMs stays free: clusters of eight do not find a place on all of them
    while (ctas < kMaxPartCtas && 16ll * ctas * rows <= 7ll * sms) ctas *= 2;
    if (v < (ctas >= 4 ? 28672 : 49152) || ctas == 1) return 0;
  }
  while (ctas < kMaxPartCtas && !fits(ctas)) ctas *= 2;
  return fits(ctas) ? ctas : 0;
}

inline int launch_parts(const __nv_bfloat16* lp, long long row_stride, int rows, int v, const long long* row_ids, float inv_temp,
                        int top_k, float top_p, unsigned long long seed, unsigned long long step, int ctas, int* out,
                        cudaStream_t stream) {
  static PerDevice once;
  if (!smem_opt_in(once, sample_parts_kernel, kPartSmemBytes)) return -10;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(rows) * ctas);
  cfg.blockDim = dim3(kPartThreads);
  cfg.dynamicSmemBytes = kPartSmemBytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = static_cast<unsigned>(ctas);
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, sample_parts_kernel, lp, row_stride, v, row_ids, inv_temp, top_k, top_p, seed, step, ctas, out) ==
                 cudaSuccess
             ? 0
             : -11;
}

// Which maxima bound a row of which a block of `threads` holds `elems` elements. The warps' keys (eight or four
// each, kth_of_warp_tops) take the least time, but in a short row only a few warps have any, and with fewer than
// k the bound is 0 and every element a candidate. One word per thread is enough while its maxima are
// four times k or more (about a quarter more candidates than k then; with as many maxima as k the bound would be the
// smallest of them), or if a thread has no more than one vector anyway. On the GPU, us: k = 50, 200 bf16 rows of 1000 columns: warps' keys 20.6, four words 10.7, one 8.1; 8
// rows 17.2, 11.5, 8.5; k = 100, four words / one: 200 rows of 4000 columns, bf16 13.8 / 11.3, fp32 15.4 / 13.3,
// 64 bf16 rows of 128256 16.8 / 14.3; k = 1000, 64 rows: 28 / 345 (ranked by counting). 64 bf16 rows of 128256
// columns, k = 50, with the warps' keys: 9.0.
template <typename T>
BoundFrom bound_from(int elems, int threads, int k) {
  const int with_keys = min(threads, elems / Elem<T>::kVec), warps = (with_keys + 31) / 32;
  if (k <= kFewK && warps * (kWarpTops / (threads / 32)) >= k) return kWarpKeys;
  return elems / Elem<T>::kVec <= threads || 4 * k <= with_keys * (Elem<T>::kPacked ? 2 : 1) ? kOneWord : kFourWords;
}

template <typename T>
int launch_topk(const T* lp, long long row_stride, int rows, int v, const long long* row_ids, float inv_temp, int top_k,
                float top_p, unsigned long long seed, unsigned long long step, int* out, cudaStream_t stream) {
  // 16-bit rows that 1, 2 or 4 CTAs can keep in registers take the kernel that reads them once, as long as
  // all CTAs (one per SM) are resident at once; otherwise they would come in waves where the other kernel,
  // two CTAs per SM, needs one. KA_SAMPLE_CLUSTER = 1 keeps the other one, 2 and 4 ask for that many CTAs
  // per row.
  if constexpr (Elem<T>::kPacked) {
    int cluster = v <= kHeldElems ? 1 : (v <= 2 * kHeldElems ? 2 : (v <= 4 * kHeldElems ? 4 : 0));
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const char* env = getenv("KA_SAMPLE_CLUSTER");
    const int asked = env ? atoi(env) : 0;
    if (asked == 2 || asked == 4)
      cluster = cluster != 0 && asked > cluster ? asked : cluster;
    else if (asked == 1 || static_cast<long long>(rows) * cluster > sms)
      cluster = 0;
    if (cluster > 0) {
      const int smem = static_cast<int>(sizeof(TopkSmem) + sizeof(ClusterXchg));
      auto of = [&](auto from) {
        constexpr int kFrom = decltype(from)::value;
        return cluster == 1 ? sample_topk_held_kernel<T, 1, kFrom>
                            : (cluster == 2 ? sample_topk_held_kernel<T, 2, kFrom> : sample_topk_held_kernel<T, 4, kFrom>);
      };
      const BoundFrom from = bound_from<T>(v / cluster, kHeldThreads, min(top_k, v));
      auto* kernel = from == kWarpKeys  ? of(std::integral_constant<int, kWarpKeys>{})
                     : from == kOneWord ? of(std::integral_constant<int, kOneWord>{})
                                        : of(std::integral_constant<int, kFourWords>{});
      static PerDevice once[9];
      if (!smem_opt_in(once[cluster / 2 * 3 + (from + 1) / 2], kernel, smem)) return -10;
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(static_cast<unsigned>(rows) * cluster);
      cfg.blockDim = dim3(kHeldThreads);
      cfg.dynamicSmemBytes = smem;
      cfg.stream = stream;
      cudaLaunchAttribute attr[1];
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = static_cast<unsigned>(cluster);
      attr[0].val.clusterDim.y = 1;
      attr[0].val.clusterDim.z = 1;
      cfg.attrs = attr;
      cfg.numAttrs = cluster > 1 ? 1 : 0;
      return cudaLaunchKernelEx(&cfg, kernel, lp, row_stride, v, row_ids, inv_temp, top_k, top_p, seed, step, out) ==
                     cudaSuccess
                 ? 0
                 : -11;
    }
  }
  const BoundFrom from = bound_from<T>(v, kTopkThreads, min(top_k, v));
  auto* kernel = from == kWarpKeys  ? sample_topk_kernel<T, kWarpKeys>
                 : from == kOneWord ? sample_topk_kernel<T, kOneWord>
                                    : sample_topk_kernel<T, kFourWords>;
  static PerDevice once[3];
  if (!smem_opt_in(once[(from + 1) / 2], kernel, static_cast<int>(sizeof(TopkSmem)))) return -10;
  kernel<<<rows, kTopkThreads, sizeof(TopkSmem), stream>>>(lp, row_stride, v, row_ids, inv_temp, top_k, top_p, seed, step, out);
  return cudaGetLastError() == cudaSuccess ? 0 : -11;
}

template <typename T>
int launch_sampling(const void* logits, long long row_stride, int rows, int v, const long long* row_ids,
                    float inv_temp, int top_k, float top_p, unsigned long long seed, unsigned long long step,
                    int* out, cudaStream_t stream) {
  const T* lp = static_cast<const T*>(logits);
  if (top_k >= 1 && top_k <= kMaxTopK) {
    return launch_topk<T>(lp, row_stride, rows, v, row_ids, inv_temp, top_k, top_p, seed, step, out, stream);
  } else {
    if constexpr (std::is_same<T, __nv_bfloat16>::value) {
      // without a filter the sums of the draw are the only pass, and less work than counting
      int dev = 0, sms = 0;
      cudaGetDevice(&dev);
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
      const int ctas = (top_k > 0 && top_k < v) || top_p < 1.0f ? part_ctas(rows, v, sms) : 0;
      if (ctas > 0) return launch_parts(lp, row_stride, rows, v, row_ids, inv_temp, top_k, top_p, seed, step, ctas, out, stream);
    }
    constexpr int smem = kGeneralSmemBytes + (Elem<T>::kPacked ? static_cast<int>(sizeof(FastSmem)) : 0);
    static_assert(sizeof(FastSmem) >= kHistBytes, "the older search keeps its histogram there");
    static PerDevice once;
    if (!smem_opt_in(once, sample_general_kernel<T>, smem)) return -10;
    sample_general_kernel<T><<<rows, kThreads, smem, stream>>>(lp, row_stride, v, row_ids, inv_temp, top_k, top_p,
                                                              seed, step, out);
  }
  return cudaGetLastError() == cudaSuccess ? 0 : -11;
}

}  // namespace
}  // namespace ka

extern "C" int ka_sample(const void* logits, int dtype, long long row_stride, int rows, int vocab,
                         const long long* row_ids, float inv_temperature, int top_k, float top_p,
                         unsigned long long seed, unsigned long long step, int* out, void* stream) {
  using namespace ka;
  if (rows <= 0) return 0;
  if (vocab <= 0 || !(inv_temperature > 0.f) || !(top_p > 0.f)) return -1;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  switch (dtype) {
    case KA_DTYPE_F32:
      return launch_sampling<float>(logits, row_stride, rows, vocab, row_ids, inv_temperature, top_k, top_p, seed,
                                    step, out, st);
    case KA_DTYPE_BF16:
      return launch_sampling<__nv_bfloat16>(logits, row_stride, rows, vocab, row_ids, inv_temperature, top_k, top_p,
                                            seed, step, out, st);
    case KA_DTYPE_F16:
      return launch_sampling<__half>(logits, row_stride, rows, vocab, row_ids, inv_temperature, top_k, top_p, seed,
                                     step, out, st);
    default:
      return -2;
  }
}
