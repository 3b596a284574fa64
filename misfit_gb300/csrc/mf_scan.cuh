// mf_scan.cuh -- the library's exclusive scan, as a template over the item
// loader, so that a caller can scan values it computes on the fly (the row
// counts of the load-balanced traversals) without writing them first.
// Included by mf_prims.cu (the plain-array scans) and mf_repair.cu.
#pragma once

#include "mf_internal.cuh"

namespace mf {
namespace scan_detail {

constexpr int kThreads = 256;   // block of the radix sort (mf_prims.cu)
constexpr int kItems = 8;
constexpr int kTile = kThreads * kItems;

template <typename T>
struct Loader {
  const T* p;
  __device__ __forceinline__ int64_t operator()(int64_t i) const { return (int64_t)p[i]; }
};

// Where the prefix goes: out(i, prefix) for i in [0, n].
struct Store {
  int64_t* p;
  __device__ __forceinline__ void operator()(int64_t i, int64_t v) const { p[i] = v; }
};

__device__ __forceinline__ int64_t block_sum(int64_t v, int64_t* smem_warp) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  if (lane == 0) smem_warp[w] = v;
  __syncthreads();
  int64_t t = 0;
  if (threadIdx.x < 32) {
    t = threadIdx.x < (blockDim.x >> 5) ? smem_warp[threadIdx.x] : 0;
    for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
  }
  __syncthreads();
  return t;  // valid in thread 0
}

// Exclusive scan across the block of one value per thread; returns the
// thread's prefix and writes the block total to *total.
__device__ __forceinline__ int64_t block_exclusive(int64_t v, int64_t* smem_warp, int64_t* total) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int64_t inc = v;
  for (int o = 1; o < 32; o <<= 1) {
    int64_t t = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += t;
  }
  if (lane == 31) smem_warp[w] = inc;
  __syncthreads();
  if (threadIdx.x < 32) {
    const int nw = blockDim.x >> 5;
    int64_t x = threadIdx.x < nw ? smem_warp[threadIdx.x] : 0;
    int64_t xi = x;
    for (int o = 1; o < 32; o <<= 1) {
      int64_t t = __shfl_up_sync(0xffffffffu, xi, o);
      if (threadIdx.x >= o) xi += t;
    }
    if (threadIdx.x < nw) smem_warp[threadIdx.x] = xi - x;
    if (threadIdx.x == nw - 1) smem_warp[32] = xi;
  }
  __syncthreads();
  const int64_t r = smem_warp[w] + inc - v;
  *total = smem_warp[32];
  __syncthreads();
  return r;
}

// One block, one item per thread, for inputs of up to kSingleThreads items.
constexpr int kSingleThreads = 1024;

template <typename L, typename O>
__global__ void __launch_bounds__(kSingleThreads) k_scan_single(L load, int64_t n, O out) {
  pdl_wait();
  pdl_trigger();
  __shared__ int64_t sw[33];
  const int64_t i = threadIdx.x;
  const int64_t v = i < n ? load(i) : 0;
  int64_t tot;
  const int64_t pre = block_exclusive(v, sw, &tot);
  if (i < n) out(i, pre);
  if (i == 0) out(n, tot);
}

// A tile's status: {value, tag}, tag = seq << 2 | flag (1: value is the
// tile's aggregate, 2: its inclusive prefix), read and written as one 16-byte
// word, so that a matching tag vouches for the value beside it.
__device__ __forceinline__ ulonglong2 status_load(const ulonglong2* p) {
  ulonglong2 r;
  asm volatile("{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\tmov.b128 {%0, %1}, t;\n\t}"
               : "=l"(r.x), "=l"(r.y) : "l"(p) : "memory");
  return r;
}
__device__ __forceinline__ void status_store(ulonglong2* p, unsigned long long value, unsigned long long tag) {
  asm volatile("{\n\t.reg .b128 t;\n\tmov.b128 t, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], t;\n\t}"
               :: "l"(p), "l"(value), "l"(tag) : "memory");
}

// Single-pass scan with decoupled look-back (Merrill and Garland, "Single-pass
// Parallel Prefix Scan with Decoupled Look-back", 2016): one launch, one
// tile of Threads x Items items per block.  Tile t publishes its aggregate,
// then one warp looks back over its predecessors 32 at a time (the sum of the
// aggregates up to the nearest inclusive prefix), and publishes its own
// inclusive prefix.  `seq` is new for every call, so the status words are never
// reset (a stale tag never matches).  Blocks are dispatched in index order, so
// a tile's predecessors are running or done; still, a wait on one gives up
// after kLookbackSpin reads, and the tile then sums its predecessors' inputs
// itself, so the result is right and the wait ends either way.
//
// Latency bounds it: a tile is a chain of loads (the row counts: list entry,
// tag, row bounds), the block scan and the look-back.  With 2,048-item tiles
// and one thread reading one predecessor at a time, 320,000 row counts took
// 42 us and 24,000 took 27 us (12 of 152 SMs busy); see scan_exclusive for the
// split that replaced it.
constexpr int64_t kLookbackSpin = (int64_t)1 << 22;

template <int Threads, int Items, typename L, typename O>
__global__ void __launch_bounds__(Threads) k_scan_lookback(L load, int64_t n, O out, ulonglong2* st,
                                                           unsigned long long seq) {
  pdl_wait();
  pdl_trigger();
  constexpr int kSpan = Threads * Items;
  __shared__ int64_t tile[Items > 1 ? kSpan : 1];
  __shared__ int64_t sw[33];
  __shared__ int64_t s_excl;
  __shared__ int s_fallback;
  const int64_t t = blockIdx.x;
  const int64_t base = t * kSpan;
  // all of the thread's items are loaded before any is stored: a loader's
  // generic loads may not pass a store to shared memory, so interleaved they
  // would run one dependent chain (list entry -> row bounds) at a time
  int64_t v[Items];
#pragma unroll
  for (int k = 0; k < Items; ++k) {
    const int64_t i = base + k * Threads + threadIdx.x;
    v[k] = i < n ? load(i) : 0;
  }
  int64_t local = v[0];
  if (Items > 1) {
#pragma unroll
    for (int k = 0; k < Items; ++k) tile[k * Threads + threadIdx.x] = v[k];
    __syncthreads();
    local = 0;
#pragma unroll
    for (int k = 0; k < Items; ++k) local += tile[threadIdx.x * Items + k];
  }
  int64_t tot;
  int64_t pre = block_exclusive(local, sw, &tot);
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
    int64_t excl = 0;
    int fb = 0;
    if (t > 0) {
      if (lane == 0) status_store(st + t, (unsigned long long)tot, (seq << 2) | 1ull);
      for (int64_t q = t - 1; q >= 0; q -= 32) {
        ulonglong2 w = make_ulonglong2(0ull, (seq << 2) | 2ull);   // before tile 0: an empty prefix
        if (q - lane >= 0) {
          int64_t spins = 0;
          do {
            w = status_load(st + (q - lane));
          } while ((w.y >> 2) != seq && ++spins < kLookbackSpin);
        }
        if (__any_sync(0xffffffffu, (w.y >> 2) != seq)) {
          fb = 1;
          break;
        }
        const unsigned full = __ballot_sync(0xffffffffu, (w.y & 3ull) == 2ull);
        const int last = full ? __ffs(full) - 1 : 31;
        int64_t x = lane <= last ? (int64_t)w.x : 0;
        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        excl += x;
        if (full) break;
      }
    }
    if (lane == 0) {
      if (!fb) status_store(st + t, (unsigned long long)(excl + tot), (seq << 2) | 2ull);
      s_excl = excl;
      s_fallback = fb;
    }
  }
  __syncthreads();
  if (s_fallback) {
    int64_t acc = 0;
    for (int64_t i = threadIdx.x; i < base; i += blockDim.x) acc += load(i);
    const int64_t sum = block_sum(acc, sw);
    if (threadIdx.x == 0) {
      s_excl = sum;
      status_store(st + t, (unsigned long long)(sum + tot), (seq << 2) | 2ull);
    }
    __syncthreads();
  }
  const int64_t excl = s_excl;
  pre += excl;
  if (Items > 1) {
#pragma unroll
    for (int k = 0; k < Items; ++k) {
      const int idx = threadIdx.x * Items + k;
      const int64_t x = tile[idx];
      tile[idx] = pre;
      pre += x;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < Items; ++k) {
      const int idx = k * Threads + threadIdx.x;
      const int64_t i = base + idx;
      if (i < n) out(i, tile[idx]);
    }
  } else {
    const int64_t i = base + threadIdx.x;
    if (i < n) out(i, pre);
  }
  if (t == (int64_t)gridDim.x - 1 && threadIdx.x == 0) out(n, excl + tot);
}

inline void reserve_tiles(Scratch& ws, int64_t nb, cudaStream_t s) {
  if (ws.scan_status.cap < 2 * nb) {
    ws.scan_status.reserve(2 * nb);
    // fresh memory may hold anything: no tag may match a later sequence number
    MF_CUDA(cudaMemsetAsync(ws.scan_status.p, 0, sizeof(unsigned long long) * (size_t)ws.scan_status.cap, s));
  }
}

template <int Threads, int Items, typename L, typename O>
void scan_lookback(L load, O out, int64_t n, Scratch& ws, cudaStream_t s) {
  const int64_t nb = (n + Threads * Items - 1) / (Threads * Items);
  reserve_tiles(ws, nb, s);
  const unsigned long long seq = ++ws.scan_seq;
  MF_K(launch_pdl(k_scan_lookback<Threads, Items, L, O>, (unsigned)nb, Threads, 0, s, load, n, out,
                  reinterpret_cast<ulonglong2*>(ws.scan_status.p), seq));
}

// How the items are split.  Up to one block's threads: one block, no
// look-back.  Up to kSmallTiles tiles of 256: one item per thread, so that a
// short list of expensive items (row counts) is spread over as many SMs as it
// can fill and the look-back still takes at most six steps of 32 tiles.
// Longer inputs: 2,048-item tiles, 512 threads with four items each.
// Before the split the row counts of a sub-batch took 27 to 42 us (see
// k_scan_lookback).  R-MAT scale 22 with it (ncu): the seeds' row counts by one
// block 4.0 us, 131,072 bitmap words by 256-item tiles 14.8 us (each writes its
// vertices), 330,000 creation flags by 2,048-item tiles 9.8 us.
constexpr int64_t kSmallTiles = 192;

// Room for the status words of any scan of up to n items with the default
// split, so that the scan itself allocates nothing.
inline void reserve_scan(Scratch& ws, int64_t n, cudaStream_t s) {
  reserve_tiles(ws, std::max<int64_t>(kSmallTiles, (n + 2047) / 2048), s);
}

// `small_tiles`: how many tiles of 256 before the 2,048-item ones (callers whose
// items write lists of their own want more blocks).
template <typename L, typename O>
void scan_exclusive_to(L load, O out, int64_t n, Scratch& ws, cudaStream_t s, int64_t small_tiles = kSmallTiles) {
  if (n <= kSingleThreads) {
    const unsigned threads = (unsigned)((n + 31) & ~(int64_t)31);
    MF_K(launch_pdl(k_scan_single<L, O>, 1, threads, 0, s, load, n, out));
  } else if (n <= small_tiles * 256) {
    scan_lookback<256, 1>(load, out, n, ws, s);
  } else {
    scan_lookback<512, 4>(load, out, n, ws, s);
  }
  MF_CUDA(cudaGetLastError());
}

template <typename L>
void scan_exclusive(L load, int64_t* out, int64_t n, Scratch& ws, cudaStream_t s) {
  if (n <= 0) MF_CUDA(cudaMemsetAsync(out, 0, sizeof(int64_t), s));
  else scan_exclusive_to(load, Store{out}, n, ws, s);
}

}  // namespace scan_detail

// out[i] = sum_{j<i} load(j) for i in [0, n]; one launch.
template <typename L>
void scan_exclusive_with(L load, int64_t* out, int64_t n, Scratch& ws, cudaStream_t s) {
  scan_detail::scan_exclusive(load, out, n, ws, s);
}

}  // namespace mf
