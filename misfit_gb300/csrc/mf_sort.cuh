// mf_sort.cuh -- the one-block stable radix sort in registers and shared memory,
// and the ranking it shares with the multi-block sort (mf_prims.cu).
#pragma once

#include "mf_internal.cuh"

namespace mf {
namespace sort_detail {

// Sort digits come from the key itself, or from a mixed copy of it when the
// caller only needs equal keys to end up in one run of equal mixed bits.
__device__ __forceinline__ uint32_t sort_digit(bool mixed, uint64_t key, int shift) {
  return (uint32_t)((mixed ? mix_key(key) : key) >> shift) & 255u;
}

constexpr int kDigits = 256;

// Rank of each of the warp's items among the warp's items of the same digit
// (in item order), and the digit counts of the warp (cnt[256], zeroed here).
// A thread's items are at warp base + r * 32 + lane.
template <int Items>
__device__ __forceinline__ void warp_rank(const uint32_t (&d)[Items], int (&rank)[Items], uint32_t* cnt) {
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
#pragma unroll
  for (int j = 0; j < kDigits / 32; ++j) cnt[lane + 32 * j] = 0;
  __syncwarp();
#pragma unroll
  for (int r = 0; r < Items; ++r) {
    const unsigned peers = __match_any_sync(0xffffffffu, d[r]);
    const int lead = __ffs(peers) - 1;
    int old = 0;
    if (lane == lead) {
      old = (int)cnt[d[r]];
      cnt[d[r]] = (uint32_t)(old + __popc(peers));
    }
    rank[r] = __shfl_sync(0xffffffffu, old, lead) + __popc(peers & lt);
    __syncwarp();
  }
}

// Thread d < 256: the warps' counts of digit d become exclusive prefixes over
// the warps; returns the digit's total.
__device__ __forceinline__ uint32_t digit_columns(uint32_t* cnt, int warps) {
  uint32_t acc = 0;
#pragma unroll 8
  for (int j = 0; j < warps; ++j) {
    const uint32_t t = cnt[j * kDigits + threadIdx.x];
    cnt[j * kDigits + threadIdx.x] = acc;
    acc += t;
  }
  return acc;
}

// Exclusive scan over the 256 digits, by the first eight warps (every thread
// of the block calls it; the others pass anything).
__device__ __forceinline__ uint32_t digit_scan(uint32_t total, uint32_t* sw) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  uint32_t inc = total;
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += t;
  }
  if (lane == 31 && w < kDigits / 32) sw[w] = inc;
  __syncthreads();
  uint32_t before = 0;
  for (int j = 0; j < w && j < kDigits / 32; ++j) before += sw[j];
  return before + inc - total;
}

// One block sorts up to Items * blockDim.x pairs held in registers: one pass
// per digit ranks them (warp_rank) and moves them through shared memory.
// Positions from n on are padding: their digit counts as 255 and they come
// last in item order, so they stay behind every pair.
template <int Items>
__device__ __forceinline__ void block_sort(bool mixed, uint64_t (&key)[Items], uint32_t (&val)[Items], int n, int first_bit, int end_bit,
                           uint64_t* sk, uint32_t* sv, uint32_t* cnt, uint32_t* dbase, uint32_t* sw) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const int at = w * 32 * Items + lane;
  for (int shift = first_bit; shift < end_bit; shift += 8) {
    uint32_t d[Items];
    int rank[Items];
#pragma unroll
    for (int r = 0; r < Items; ++r) d[r] = at + r * 32 < n ? sort_digit(mixed, key[r], shift) : 255u;
    warp_rank<Items>(d, rank, cnt + w * kDigits);
    __syncthreads();
    uint32_t total = 0;
    if (threadIdx.x < kDigits) total = digit_columns(cnt, warps);
    const uint32_t base = digit_scan(total, sw);
    if (threadIdx.x < kDigits) dbase[threadIdx.x] = base;
    __syncthreads();
#pragma unroll
    for (int r = 0; r < Items; ++r) {
      const uint32_t pos = dbase[d[r]] + cnt[w * kDigits + d[r]] + (uint32_t)rank[r];
      sk[pos] = key[r];
      sv[pos] = val[r];
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < Items; ++r) {
      key[r] = sk[at + r * 32];
      val[r] = sv[at + r * 32];
    }
    __syncthreads();
  }
}

}  // namespace sort_detail
}  // namespace mf
