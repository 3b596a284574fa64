// mf_prims.cu -- device scans and a stable LSD radix sort.
//
// Scans: one launch.  Small inputs in one block; larger ones with the
// single-pass decoupled look-back scan (k_scan_lookback, mf_scan.cuh).
// Radix sort: 8-bit digits, stable (equal keys keep their input order, which
// is what the callers rely on).  Up to kBlockSortMax pairs the whole sort is one
// block's work in shared memory (block_sort); longer inputs take one launch
// per digit, each tile finding its place by a decoupled look-back per digit
// (Adinets and Merrill, "Onesweep", 2022).
#include <algorithm>

#include "mf_scan.cuh"
#include "mf_sort.cuh"

namespace mf {

namespace {

using namespace scan_detail;
using namespace sort_detail;

// ---- radix sort --------------------------------------------------------------

template <int Items, bool Mixed>
__global__ void __launch_bounds__(1024) k_sort_block(uint64_t* keys, uint32_t* vals, int n, int first_bit,
                                                     int end_bit) {
  pdl_wait();
  pdl_trigger();
  extern __shared__ __align__(16) unsigned char sort_smem[];
  __shared__ uint32_t dbase[kDigits];
  __shared__ uint32_t sw[kDigits / 32];
  const int cap = Items * (int)blockDim.x;
  uint64_t* sk = reinterpret_cast<uint64_t*>(sort_smem);
  uint32_t* sv = reinterpret_cast<uint32_t*>(sk + cap);
  uint32_t* cnt = sv + cap;
  const int at = (threadIdx.x >> 5) * 32 * Items + (threadIdx.x & 31);
  uint64_t key[Items];
  uint32_t val[Items];
#pragma unroll
  for (int r = 0; r < Items; ++r) {
    key[r] = at + r * 32 < n ? keys[at + r * 32] : 0;
    val[r] = at + r * 32 < n ? vals[at + r * 32] : 0;
  }
  block_sort<Items>(Mixed, key, val, n, first_bit, end_bit, sk, sv, cnt, dbase, sw);
#pragma unroll
  for (int r = 0; r < Items; ++r) {
    if (at + r * 32 < n) {
      keys[at + r * 32] = key[r];
      vals[at + r * 32] = val[r];
    }
  }
}

// Registers bound one block: eight 12-byte pairs, their digits and ranks in the
// 64 registers a thread of a 1,024-thread block has.
constexpr int kBlockSortMax = 8192;

template <int Items, bool Mixed>
void sort_block(uint64_t* keys, uint32_t* vals, int n, int threads, int first_bit, int end_bit, Scratch& ws,
                cudaStream_t s) {
  const size_t smem = (size_t)Items * threads * 12 + (size_t)(threads / 32) * kDigits * 4;
  if (smem > 48 * 1024) ws.smem.raise(k_sort_block<Items, Mixed>, Items * 1024 * 12 + 32 * kDigits * 4);
  MF_K(launch_pdl(k_sort_block<Items, Mixed>, 1, (unsigned)threads, smem, s, keys, vals, n, first_bit, end_bit));
}

// Digit counts of every pass over the whole input (hist zeroed before).
constexpr int kMaxPasses = 8;

template <bool Mixed>
__global__ void __launch_bounds__(kThreads) k_sort_hist(const uint64_t* keys, int64_t n, int first_bit, int passes,
                                                        uint32_t* hist) {
  pdl_wait();
  pdl_trigger();
  __shared__ uint32_t h[kMaxPasses * kDigits];
  for (int i = threadIdx.x; i < passes * kDigits; i += blockDim.x) h[i] = 0;
  __syncthreads();
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const uint64_t k = Mixed ? mix_key(keys[i]) : keys[i];
    for (int p = 0; p < passes; ++p) atomicAdd(&h[p * kDigits + ((k >> (first_bit + 8 * p)) & 255u)], 1u);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < passes * kDigits; i += blockDim.x)
    if (h[i]) atomicAdd(hist + i, h[i]);
}

// One digit of the sort: tiles of 256 threads x 8 items.  A tile ranks its
// items, publishes its digit counts and sums its predecessors' (thread d looks
// back for digit d, eight tiles' words in flight), then writes its pairs out in
// digit runs.  Status word: seq << 34 | flag << 32 | count (flag 1: the tile's
// count, 2: the count up to and including the tile); `seq` is new for every
// pass, so the words are never reset.  A wait gives up after kLookbackSpin
// reads, and the thread then counts its digit over all earlier items itself.
//
// A pass over 200,000 pairs moves 4.8 MB; what bounds it is latency (two loads,
// the ranking, the look-back, the store).  It replaces three launches (digit
// histogram, scan, scatter) of 19 us together at 2,000-4,000 pairs.
template <bool Mixed>
__global__ void __launch_bounds__(kThreads) k_sort_pass(const uint64_t* keys, const uint32_t* vals, int64_t n, int shift,
                                                        const uint32_t* hist, unsigned long long* status,
                                                        unsigned long long seq, uint64_t* okeys, uint32_t* ovals) {
  pdl_wait();
  pdl_trigger();
  __shared__ uint64_t sk[kTile];
  __shared__ uint32_t sv[kTile];
  __shared__ uint32_t cnt[(kThreads / 32) * kDigits];
  __shared__ uint32_t dbase[kDigits];
  __shared__ int64_t gofs[kDigits];
  __shared__ uint32_t sw[kDigits / 32];
  __shared__ uint32_t sw2[kDigits / 32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t t = blockIdx.x;
  const int64_t base = t * kTile;
  const int cap = (int)min((int64_t)kTile, n - base);
  const int at = w * 32 * kItems + lane;
  uint64_t key[kItems];
  uint32_t val[kItems];
  uint32_t d[kItems];
  int rank[kItems];
#pragma unroll
  for (int r = 0; r < kItems; ++r) {
    const bool ok = at + r * 32 < cap;
    key[r] = ok ? keys[base + at + r * 32] : 0;
    val[r] = ok ? vals[base + at + r * 32] : 0;
  }
#pragma unroll
  for (int r = 0; r < kItems; ++r) d[r] = at + r * 32 < cap ? sort_digit(Mixed, key[r], shift) : 255u;
  warp_rank<kItems>(d, rank, cnt + w * kDigits);
  __syncthreads();
  const uint32_t padded = digit_columns(cnt, kThreads / 32);
  // the padding sits in digit 255
  const uint32_t mine = threadIdx.x == 255 ? padded - (uint32_t)(kTile - cap) : padded;
  unsigned long long* my = status + t * kDigits + threadIdx.x;
  *(volatile unsigned long long*)my = (seq << 34) | (t == 0 ? 2ull << 32 : 1ull << 32) | mine;
  const uint32_t local = digit_scan(padded, sw);
  dbase[threadIdx.x] = local;
  const uint32_t global = digit_scan(hist[threadIdx.x], sw2);
  int64_t excl = 0;
  bool found = t == 0, lost = false;
  for (int64_t q = t - 1; q >= 0 && !found && !lost; q -= 8) {
    unsigned long long x[8];
#pragma unroll
    for (int j = 0; j < 8; ++j)
      x[j] = q - j >= 0 ? *(volatile const unsigned long long*)(status + (q - j) * kDigits + threadIdx.x) : 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      if (found || lost || q - j < 0) continue;
      int64_t spins = 0;
      while ((x[j] >> 34) != seq && ++spins < kLookbackSpin)
        x[j] = *(volatile const unsigned long long*)(status + (q - j) * kDigits + threadIdx.x);
      if ((x[j] >> 34) != seq) {
        lost = true;
        continue;
      }
      excl += (int64_t)(x[j] & 0xffffffffull);
      found = ((x[j] >> 32) & 3ull) == 2ull;
    }
  }
  if (lost) {
    excl = 0;
    for (int64_t i = 0; i < base; ++i) excl += sort_digit(Mixed, keys[i], shift) == threadIdx.x;
  }
  if (t > 0) *(volatile unsigned long long*)my = (seq << 34) | (2ull << 32) | (unsigned long long)(excl + mine);
  gofs[threadIdx.x] = (int64_t)global + excl - (int64_t)local;
#pragma unroll
  for (int r = 0; r < kItems; ++r) {
    if (r == 0) __syncthreads();
    const uint32_t pos = dbase[d[r]] + cnt[w * kDigits + d[r]] + (uint32_t)rank[r];
    sk[pos] = key[r];
    sv[pos] = val[r];
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < kItems; ++r) {
    const int i = r * kThreads + threadIdx.x;
    if (i < cap) {
      const uint64_t k = sk[i];
      const int64_t pos = gofs[sort_digit(Mixed, k, shift)] + i;
      okeys[pos] = k;
      ovals[pos] = sv[i];
    }
  }
}

void reserve_passes(Scratch& ws, int64_t n, cudaStream_t s) {
  const int64_t tiles = (n + kTile - 1) / kTile;
  ws.keys_alt.reserve(n);
  ws.vals_alt.reserve(n);
  ws.hist.reserve(kMaxPasses * kDigits);
  if (ws.sort_status.cap < tiles * kDigits) {
    ws.sort_status.reserve(tiles * kDigits);
    // fresh memory may hold anything: no tag may match a later sequence number
    MF_CUDA(cudaMemsetAsync(ws.sort_status.p, 0, sizeof(unsigned long long) * (size_t)ws.sort_status.cap, s));
    ws.sort_seq = 0;
  }
}

template <bool Mixed>
SortedPairs sort_pairs(uint64_t* keys, uint32_t* vals, int64_t n, int first_bit, int end_bit, Scratch& ws,
                       cudaStream_t s) {
  if (n <= 1) return {keys, vals};
  if (n <= kBlockSortMax) {
    // one to eight items a thread; 256 threads at least, one per digit
    if (n <= 256) sort_block<1, Mixed>(keys, vals, (int)n, 256, first_bit, end_bit, ws, s);
    else if (n <= 1024) sort_block<1, Mixed>(keys, vals, (int)n, 1024, first_bit, end_bit, ws, s);
    else if (n <= 2048) sort_block<2, Mixed>(keys, vals, (int)n, 1024, first_bit, end_bit, ws, s);
    else if (n <= 4096) sort_block<4, Mixed>(keys, vals, (int)n, 1024, first_bit, end_bit, ws, s);
    else sort_block<8, Mixed>(keys, vals, (int)n, 1024, first_bit, end_bit, ws, s);
    MF_CUDA(cudaGetLastError());
    return {keys, vals};
  }
  const int64_t tiles = (n + kTile - 1) / kTile;
  const int passes = (end_bit - first_bit + 7) / 8;
  reserve_passes(ws, n, s);
  if (ws.sort_seq + kMaxPasses >= (1ull << 30)) {   // the tag's 30 bits are used up
    MF_CUDA(cudaMemsetAsync(ws.sort_status.p, 0, sizeof(unsigned long long) * (size_t)ws.sort_status.cap, s));
    ws.sort_seq = 0;
  }
  MF_CUDA(cudaMemsetAsync(ws.hist.p, 0, sizeof(uint32_t) * (size_t)passes * kDigits, s));
  MF_K(launch_pdl(k_sort_hist<Mixed>, (unsigned)std::min<int64_t>(tiles, 304), kThreads, 0, s, keys, n, first_bit, passes,
                  ws.hist.p));
  SortedPairs a{keys, vals}, b{ws.keys_alt.p, ws.vals_alt.p};
  for (int pass = 0; pass < passes; ++pass) {
    const unsigned long long seq = ++ws.sort_seq;
    MF_K(launch_pdl(k_sort_pass<Mixed>, (unsigned)tiles, kThreads, 0, s, a.keys, a.vals, n, first_bit + 8 * pass,
                    ws.hist.p + pass * kDigits, ws.sort_status.p, seq, b.keys, b.vals));
    std::swap(a, b);
  }
  MF_CUDA(cudaGetLastError());
  return a;
}

}  // namespace

int bits_for(int64_t v) {
  int b = 1;
  while (b < 63 && (v >> b) != 0) ++b;
  return b;
}

void scan_exclusive_i64(const int64_t* in, int64_t* out, int64_t n, Scratch& ws, cudaStream_t s) {
  scan_exclusive(Loader<int64_t>{in}, out, n, ws, s);
}
void scan_exclusive_i32(const int32_t* in, int64_t* out, int64_t n, Scratch& ws, cudaStream_t s) {
  scan_exclusive(Loader<int32_t>{in}, out, n, ws, s);
}
void scan_exclusive_u8(const uint8_t* in, int64_t* out, int64_t n, Scratch& ws, cudaStream_t s) {
  scan_exclusive(Loader<uint8_t>{in}, out, n, ws, s);
}

void reserve_sort(Scratch& ws, int64_t n, cudaStream_t s) {
  if (n > kBlockSortMax) reserve_passes(ws, n, s);
}

SortedPairs radix_sort_pairs(uint64_t* keys, uint32_t* vals, int64_t n, int first_bit, int end_bit, Scratch& ws,
                             cudaStream_t s) {
  return sort_pairs<false>(keys, vals, n, first_bit, end_bit, ws, s);
}

void radix_sort_pairs_in_place(uint64_t* keys, uint32_t* vals, int64_t n, int first_bit, int end_bit, Scratch& ws,
                               cudaStream_t s) {
  const SortedPairs r = radix_sort_pairs(keys, vals, n, first_bit, end_bit, ws, s);
  if (r.keys != keys) {
    MF_CUDA(cudaMemcpyAsync(keys, r.keys, sizeof(uint64_t) * n, cudaMemcpyDeviceToDevice, s));
    MF_CUDA(cudaMemcpyAsync(vals, r.vals, sizeof(uint32_t) * n, cudaMemcpyDeviceToDevice, s));
  }
}

SortedPairs radix_group_pairs(uint64_t* keys, uint32_t* vals, int64_t n, int bits, Scratch& ws, cudaStream_t s) {
  return sort_pairs<true>(keys, vals, n, 64 - bits, 64, ws, s);
}

}  // namespace mf
