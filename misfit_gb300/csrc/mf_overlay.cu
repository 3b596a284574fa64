// mf_overlay.cu -- device-resident base CSR + delta overlay.
//
// The reference keeps the overlay as hash maps of vectors and sets on the
// host (core/FlashGraph.h:172-276).  Here:
//   * a tombstone of (x, y) clears the live bits of every copy of y in the
//     base row of x (and of x in the row of y) and counts into rcnt[x],
//     rcnt[y] -- the size of removed_adj[x] that DeltaOverlay::degree uses;
//   * added neighbours live in a CSR (aoff/aadj) that keeps each vertex's
//     entries in insertion order; it is rebuilt after every batch from the
//     surviving entries followed by the new ones in batch order.
// A batch is applied in parallel by grouping its updates per unordered pair:
// different pairs touch disjoint overlay entries, so only the updates of one
// pair have to run in batch order (one thread walks them through the
// three-state machine none / added / tombstoned that insertEdge, removeEdge,
// un_tombstone and forget_delta_edge implement, core/FlashGraph.h:196-275).
#include <algorithm>
#include <mutex>

#include "mf_internal.cuh"
#include "mf_scan.cuh"
#include "mf_sort.cuh"

namespace mf {

using scan_detail::scan_exclusive_to;

namespace {

constexpr int kTB = 256;

inline unsigned grid_for(int64_t n, int per = kTB) {
  int64_t g = (n + per - 1) / per;
  if (g < 1) g = 1;
  if (g > (1 << 30)) g = 1 << 30;
  return (unsigned)g;
}

__global__ void k_base_degree(const int64_t* nindex, int32_t n, int32_t* deg) {
  int64_t x = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (x < n) deg[x] = (int32_t)(nindex[x + 1] - nindex[x]);
}

// The longest row (base and added positions).
__global__ void k_max_row(GraphView g, unsigned long long* out) {
  const int64_t x = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  long long len = x < g.n ? (long long)row_positions(g, (int32_t)x) : 0;
  for (int o = 16; o > 0; o >>= 1) len = max(len, __shfl_xor_sync(0xffffffffu, len, o));
  __shared__ long long s_len[kTB / 32];
  if ((threadIdx.x & 31) == 0) s_len[threadIdx.x >> 5] = len;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < kTB / 32; ++w) len = max(len, s_len[w]);
    atomicMax(out, (unsigned long long)len);
  }
}

// Rows non-decreasing?  (Sorted rows allow binary search for a neighbour.)
// Load-balanced over all entries: each entry compares with its predecessor
// in the same row.  flags[0] cleared on a descent.
__global__ void k_check_sorted(GraphView g, const int32_t* list, const int64_t* offs, int32_t n, int* ok) {
  lb_rows_pos(g, list, offs, n, 0, [&](int64_t, int32_t x, int32_t y, int64_t j) {
    if (j > 0 && g.nlist[g.nindex[x] + j - 1] > y) atomicAnd(ok, 0);
  });
}

// Every entry x -> y has its reverse y -> x (rows sorted: binary search).
__global__ void k_check_symmetric(GraphView g, const int32_t* list, const int64_t* offs, int32_t n, int* ok) {
  lb_rows(g, list, offs, n, [&](int64_t, int32_t x, int32_t y) {
    int64_t lo = g.nindex[y], hi = g.nindex[y + 1];
    while (lo < hi) {
      const int64_t mid = (lo + hi) >> 1;
      if (g.nlist[mid] < x) lo = mid + 1; else hi = mid;
    }
    if (lo >= g.nindex[y + 1] || g.nlist[lo] != x) atomicAnd(ok, 0);
  });
}

__global__ void k_iota_n(int32_t* out, int32_t n) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = (int32_t)i;
}

__global__ void k_base_positions(const int64_t* nindex, int32_t n, int64_t* out) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = nindex[i + 1] - nindex[i];
}

__global__ void k_check_ids(const int32_t* nlist, int64_t nnz, int32_t n, int* ok) {
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < nnz;
       k += (int64_t)gridDim.x * blockDim.x) {
    const int32_t y = nlist[k];
    if (y < 0 || y >= n) { atomicAnd(ok, 0); return; }
  }
}

__global__ void k_check_index(const int64_t* nindex, int32_t n, int64_t nnz, int* ok) {
  int64_t x = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (x > n) return;
  const int64_t a = nindex[x];
  if (a < 0 || a > nnz || (x < n && nindex[x + 1] < a) || (x == 0 && a != 0)) atomicAnd(ok, 0);
}

// Copies of y in the base row of x, split by live/tombstoned.
__device__ void base_copies(const GraphView& g, bool sorted, int32_t x, int32_t y, int32_t* nlive, int32_t* ndead) {
  int32_t l = 0, d = 0;
  int64_t b = g.nindex[x], e = g.nindex[x + 1];
  if (sorted) {
    int64_t lo = b, hi = e;
    while (lo < hi) {
      int64_t mid = (lo + hi) >> 1;
      if (g.nlist[mid] < y) lo = mid + 1; else hi = mid;
    }
    for (int64_t k = lo; k < e && g.nlist[k] == y; ++k) {
      if (live_at(g.live, k)) ++l; else ++d;
    }
  } else {
    for (int64_t k = b; k < e; ++k)
      if (g.nlist[k] == y) { if (live_at(g.live, k)) ++l; else ++d; }
  }
  *nlive = l;
  *ndead = d;
}

// Live bits of the copies of y among the base positions [k, e) (sorted rows: k is
// the first copy).
__device__ __forceinline__ void base_mark(const GraphView& g, uint32_t* live, bool sorted, int64_t k, int64_t e,
                                          int32_t y, bool on) {
  for (; k < e; ++k) {
    const int32_t z = g.nlist[k];
    if (sorted && z != y) break;
    if (z != y) continue;
    const uint32_t bit = 1u << (k & 31);
    if (on) atomicOr(live + (k >> 5), bit); else atomicAnd(live + (k >> 5), ~bit);
  }
}

__device__ int64_t added_find(const GraphView& g, int32_t x, int32_t y) {
  for (int64_t k = g.aoff[x]; k < g.aoff[x + 1]; ++k)
    if (g.aadj[k] == y) return k;
  return -1;
}

// ---- batch input -----------------------------------------------------------------

__device__ __forceinline__ uint64_t pair_key(int32_t x, int32_t y, int nbits) {
  return ((uint64_t)(uint32_t)min(x, y) << nbits) | (uint64_t)(uint32_t)max(x, y);
}

__device__ __forceinline__ bool bad_line(int32_t x, int32_t y, int32_t n) {
  return x < 0 || x >= n || y < 0 || y >= n || x == y;
}

// The lines into the context's arrays (unless they are there), checked; the
// pair keys and the endpoint slots' vertices for the sorts.
__global__ void k_stage(BatchIn in, int64_t m, int32_t n, int nbits, int32_t* u, int32_t* v, uint8_t* ins,
                        uint8_t* app_line, uint64_t* pair_keys, uint32_t* pair_vals, uint64_t* slot_keys,
                        uint32_t* slot_vals, unsigned long long* bad) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= m) return;
  const int32_t x = in.u[i], y = in.v[i];
  if (in.u != u) {
    u[i] = x;
    v[i] = y;
    ins[i] = in.ins[i];
  }
  app_line[i] = 0;
  if (bad_line(x, y, n)) atomicAdd(bad, 1ull);
  pair_keys[i] = pair_key(x, y, nbits);
  pair_vals[i] = (uint32_t)i;
  reinterpret_cast<ulonglong2*>(slot_keys)[i] = make_ulonglong2((uint32_t)x, (uint32_t)y);
  reinterpret_cast<uint2*>(slot_vals)[i] = make_uint2((uint32_t)(2 * i), (uint32_t)(2 * i + 1));
}

// Previous edge index of every endpoint slot's vertex (sorted slots: each
// vertex's in slot order).
__global__ void k_prev(const uint64_t* keys, const uint32_t* vals, int64_t cnt, int32_t* prev) {
  pdl_wait();
  pdl_trigger();
  const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= cnt) return;
  prev[vals[j]] = j > 0 && keys[j - 1] == keys[j] ? (int32_t)(vals[j - 1] >> 1) : -1;
}

// A small batch's input in one launch: block 0 stages and checks the lines and
// groups the pairs, block 1 sorts the endpoint slots and finds the previous
// occurrences.  Both read the lines where they are (pinned host memory, the
// caller's device arrays, or the context's).  Latency of one block's sort bounds
// it; as separate launches (three copies, a check, key kernels, three sorts,
// k_prev) the same work took 16 launches and two round trips to the host.
template <int Items>
__global__ void __launch_bounds__(1024) k_small_input(BatchIn in, int m, int32_t n, int nbits, int gbits, int32_t* u,
                                                      int32_t* v, uint8_t* ins, uint8_t* app_line, uint64_t* pair_keys,
                                                      uint32_t* pair_vals, uint64_t* slot_keys, uint32_t* slot_vals,
                                                      int32_t* prev, unsigned long long* bad) {
  extern __shared__ __align__(16) unsigned char in_smem[];
  __shared__ uint32_t dbase[sort_detail::kDigits];
  __shared__ uint32_t sw[sort_detail::kDigits / 32];
  const int cap = Items * (int)blockDim.x;
  uint64_t* sk = reinterpret_cast<uint64_t*>(in_smem);
  uint32_t* sv = reinterpret_cast<uint32_t*>(sk + cap);
  uint32_t* cnt = sv + cap;
  const int at = (threadIdx.x >> 5) * 32 * Items + (threadIdx.x & 31);
  uint64_t key[Items];
  uint32_t val[Items];
  if (blockIdx.x == 0) {
#pragma unroll
    for (int r = 0; r < Items; ++r) {
      const int i = at + r * 32;
      key[r] = 0;
      val[r] = (uint32_t)i;
      if (i < m) {
        const int32_t x = in.u[i], y = in.v[i];
        if (in.u != u) {
          u[i] = x;
          v[i] = y;
          ins[i] = in.ins[i];
        }
        app_line[i] = 0;
        if (bad_line(x, y, n)) atomicAdd(bad, 1ull);
        key[r] = pair_key(x, y, nbits);
      }
    }
    sort_detail::block_sort<Items>(true, key, val, m, 64 - gbits, 64, sk, sv, cnt, dbase, sw);
#pragma unroll
    for (int r = 0; r < Items; ++r) {
      const int i = at + r * 32;
      if (i < m) {
        pair_keys[i] = key[r];
        pair_vals[i] = val[r];
      }
    }
  } else {
#pragma unroll
    for (int r = 0; r < Items; ++r) {
      const int i = at + r * 32;
      val[r] = (uint32_t)i;
      key[r] = i < 2 * m ? (uint32_t)((i & 1) ? in.v[i >> 1] : in.u[i >> 1]) : 0;
    }
    sort_detail::block_sort<Items>(false, key, val, 2 * m, 0, nbits, sk, sv, cnt, dbase, sw);
#pragma unroll
    for (int r = 0; r < Items; ++r) {
      const int i = at + r * 32;
      if (i < 2 * m) {
        slot_keys[i] = key[r];
        slot_vals[i] = val[r];
        prev[val[r]] = i > 0 && sk[i - 1] == key[r] ? (int32_t)(sv[i - 1] >> 1) : -1;
      }
    }
  }
}

template <int Items>
void small_input(mf_ctx* c, const BatchIn& in, int m, int threads, int nbits, int gbits) {
  const size_t smem = (size_t)Items * threads * 12 + (size_t)(threads / 32) * sort_detail::kDigits * 4;
  if (smem > 48 * 1024) c->ws.smem.raise(k_small_input<Items>, Items * 1024 * 12 + 32 * sort_detail::kDigits * 4);
  MF_K(k_small_input<Items><<<2, threads, smem, c->stream>>>(
      in, m, c->n, nbits, gbits, c->bu.p, c->bv.p, c->bins.p, c->app_line.p, c->keys.p, c->vals.p, c->slot_keys.p,
      c->slot_vals.p, c->prev.p, c->work.p + kCntBad));
}

enum : int { kStN = 0, kStA = 1, kStR = 2 };

// The updates of one unordered pair lie in one run of equal mixed key bits, in
// batch order, seldom with another pair's between them; the thread of the
// pair's first update walks them.  Two updates are in one run when the top
// `gbits` of their mixed keys agree.
__device__ __forceinline__ bool same_run(uint64_t a, uint64_t b, int gbits) {
  return a == b || ((mix_key(a) ^ mix_key(b)) >> (64 - gbits)) == 0;
}

// Both directions of a pair: the entry of each vertex in the other's added part,
// and the other's copies in each base row.  The two rows' searches go step by
// step together, so their loads overlap.
struct PairState {
  int64_t pos[2];           // added entry, or -1
  int64_t first[2], end[2]; // base positions to look at: from the first copy (sorted rows) to the row's end
  int32_t live[2], dead[2];
};

// Live and dead copies of y in the base positions [k, e) of an unsorted row: read
// whole, a hub's of 10^4 entries by one thread, so eight loads are in flight (one
// at a time a batch on unsorted R-MAT scale 17 took 4.7 ms; so 3.7).
__device__ __noinline__ int2 unsorted_copies(const int32_t* nlist, const uint32_t* live, int64_t k, int64_t e, int32_t y) {
  constexpr int kStep = 8;
  int2 c = make_int2(0, 0);
  for (; k < e; k += kStep) {
    int32_t z[kStep];
#pragma unroll
    for (int j = 0; j < kStep; ++j) z[j] = k + j < e ? __ldg(nlist + k + j) : -1;
#pragma unroll
    for (int j = 0; j < kStep; ++j)
      if (z[j] == y) {
        if (live_at(live, k + j)) ++c.x; else ++c.y;
      }
  }
  return c;
}

__device__ __forceinline__ PairState pair_state(const GraphView& g, bool sorted, int32_t a, int32_t b) {
  PairState r;
  const int32_t x[2] = {a, b}, y[2] = {b, a};
  int64_t lo[2], hi[2], e[2], ab[2], ae[2];
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    lo[q] = g.nindex[x[q]];
    hi[q] = e[q] = g.nindex[x[q] + 1];
    ab[q] = g.aoff[x[q]];
    ae[q] = g.aoff[x[q] + 1];
    r.pos[q] = -1;
    r.live[q] = r.dead[q] = 0;
  }
  if (sorted) {
    while (lo[0] < hi[0] || lo[1] < hi[1]) {
      int32_t z[2];
      int64_t mid[2];
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        mid[q] = (lo[q] + hi[q]) >> 1;
        z[q] = lo[q] < hi[q] ? __ldg(g.nlist + mid[q]) : 0;
      }
#pragma unroll
      for (int q = 0; q < 2; ++q)
        if (lo[q] < hi[q]) {
          if (z[q] < y[q]) lo[q] = mid[q] + 1; else hi[q] = mid[q];
        }
    }
  }
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    r.first[q] = lo[q];
    r.end[q] = e[q];
    if (!sorted) {
      const int2 c = unsorted_copies(g.nlist, g.live, lo[q], e[q], y[q]);
      r.live[q] = c.x;
      r.dead[q] = c.y;
    } else {
      for (int64_t k = lo[q]; k < e[q] && __ldg(g.nlist + k) == y[q]; ++k) {
        if (live_at(g.live, k)) ++r.live[q]; else ++r.dead[q];
      }
    }
    for (int64_t k = ab[q]; k < ae[q]; ++k)
      if (g.aadj[k] == y[q]) {
        r.pos[q] = k;
        break;
      }
  }
  return r;
}

// What a pair's updates have done so far.
struct PairWalk {
  int st;
  bool appended, old_killed;
  uint32_t last_seq;
};

__device__ __forceinline__ void pair_update(PairWalk& w, bool insert, bool base_xy, uint32_t line) {
  const bool adj = w.st == kStA || (w.st == kStN && base_xy);
  if (insert && !adj) {
    if (w.st == kStR) w.st = kStN;
    else { w.st = kStA; w.appended = true; w.last_seq = line; }
  } else if (!insert && adj) {
    if (w.st == kStA) {
      w.st = kStN;
      if (w.appended) w.appended = false; else w.old_killed = true;
    } else {
      w.st = kStR;
    }
  }
}

// The pair's further updates, from position j of its run on, four read at a
// time: thousands of them are one thread's work (100,000 of one pair took
// 25.3 ms one at a time; so 18.6).  Seldom reached, so it stays out of line.
__device__ __noinline__ PairWalk pair_updates(PairWalk w, const uint64_t* keys, const uint32_t* vals, int64_t j,
                                              int64_t m, int gbits, uint64_t key, const int32_t* u, const uint8_t* ins,
                                              int32_t a, bool in_base_ab, bool in_base_ba) {
  constexpr int kAhead = 4;
  for (; j < m; j += kAhead) {
    uint64_t k[kAhead];
    uint32_t i[kAhead];
    int32_t x[kAhead];
    bool insert[kAhead];
#pragma unroll
    for (int q = 0; q < kAhead; ++q) k[q] = j + q < m ? keys[j + q] : ~key;
#pragma unroll
    for (int q = 0; q < kAhead; ++q) i[q] = k[q] == key ? vals[j + q] : 0;
#pragma unroll
    for (int q = 0; q < kAhead; ++q) {
      x[q] = k[q] == key ? u[i[q]] : 0;
      insert[q] = k[q] == key && ins[i[q]] != 0;
    }
#pragma unroll
    for (int q = 0; q < kAhead; ++q) {
      if (k[q] == key) pair_update(w, insert[q], x[q] == a ? in_base_ab : in_base_ba, i[q]);
      else if (j + q >= m || !same_run(k[q], key, gbits)) return w;
    }
  }
  return w;
}

// One thread per unordered pair.  Besides the base tombstones it records what
// the added arrays' rebuild needs: the change of the added counts (adelta),
// the entries that go (akill) and the line whose pair is appended
// (app_line).  cnt = the batch counters from kCntBad; with invalid lines
// nothing is touched.  The counters are one address for the whole batch, so a
// block adds to them once (25,000 lines' own atomics took 45 of 66 us).
__global__ void __launch_bounds__(kTB) k_apply_pairs(GraphView g, uint32_t* live, int32_t* dead, int32_t* rcnt,
                                                     int32_t* deg, bool sorted, const uint64_t* keys,
                                                     const uint32_t* vals, int64_t m, int nbits, int gbits,
                                                     const int32_t* u, const int32_t* v, const uint8_t* ins,
                                                     int32_t* adelta, uint8_t* akill, uint8_t* app_line,
                                                     unsigned long long* cnt) {
  pdl_wait();
  pdl_trigger();
  __shared__ int s_appended, s_killed;
  __shared__ long long s_longest;
  if (*cnt != 0) return;
  if (threadIdx.x == 0) {
    s_appended = s_killed = 0;
    s_longest = 0;
  }
  __syncthreads();
  const int64_t j0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  bool head = j0 < m;
  const uint64_t key = head ? keys[j0] : 0;
  for (int64_t j = j0 - 1; head && j >= 0; --j) {
    const uint64_t k = keys[j];
    if (k == key) head = false;   // not the pair's first update
    else if (!same_run(k, key, gbits)) break;
  }
  if (head) {
    const int32_t a = (int32_t)(key >> nbits);
    const int32_t b = (int32_t)(key & ((1ull << nbits) - 1));
    const PairState ps = pair_state(g, sorted, a, b);
    const bool in_base_ab = ps.live[0] + ps.dead[0] > 0, in_base_ba = ps.live[1] + ps.dead[1] > 0;
    const int st0 = (ps.pos[0] >= 0 || ps.pos[1] >= 0) ? kStA : ((ps.dead[0] + ps.dead[1]) > 0 ? kStR : kStN);
    PairWalk w{st0, false, false, 0};
    pair_update(w, ins[vals[j0]] != 0, u[vals[j0]] == a ? in_base_ab : in_base_ba, vals[j0]);
    if (j0 + 1 < m && same_run(keys[j0 + 1], key, gbits))
      w = pair_updates(w, keys, vals, j0 + 1, m, gbits, key, u, ins, a, in_base_ab, in_base_ba);
    const int st = w.st;
    const bool appended = w.appended, old_killed = w.old_killed;
    const uint32_t last_seq = w.last_seq;
    int da = 0, db = 0;   // degree = base - tombstones + added (DeltaOverlay::degree)
    if ((st0 == kStR) != (st == kStR)) {
      const bool on = st0 == kStR;  // untombstone -> set live again
      base_mark(g, live, sorted, ps.first[0], ps.end[0], b, on);
      base_mark(g, live, sorted, ps.first[1], ps.end[1], a, on);
      const int32_t sgn = on ? -1 : 1;
      atomicAdd(rcnt + a, sgn);
      atomicAdd(rcnt + b, sgn);
      atomicAdd(dead + a, sgn * (ps.live[0] + ps.dead[0]));
      atomicAdd(dead + b, sgn * (ps.live[1] + ps.dead[1]));
      da = db = -sgn;
    }
    if (old_killed) {
      if (ps.pos[0] >= 0) { akill[ps.pos[0]] = 1; atomicSub(adelta + a, 1); --da; }
      if (ps.pos[1] >= 0) { akill[ps.pos[1]] = 1; atomicSub(adelta + b, 1); --db; }
      atomicAdd(&s_killed, 2);
    }
    if (appended) {
      app_line[last_seq] = 1;
      // at least the new length of either row (other pairs may take entries yet)
      const long long la = row_positions(g, a) + atomicAdd(adelta + a, 1) + 1;
      const long long lb = row_positions(g, b) + atomicAdd(adelta + b, 1) + 1;
      const long long longest = max(la, lb);
      if (*(volatile long long*)&s_longest < longest)
        atomicMax(reinterpret_cast<unsigned long long*>(&s_longest), (unsigned long long)longest);
      ++da;
      ++db;
      atomicAdd(&s_appended, 2);
    }
    if (da) atomicAdd(deg + a, da);
    if (db) atomicAdd(deg + b, db);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    if (s_killed) atomicAdd(cnt + (kCntKilled - kCntBad), (unsigned long long)s_killed);
    if (s_appended) atomicAdd(cnt + (kCntAppended - kCntBad), (unsigned long long)s_appended);
    if (s_longest) atomicMax(cnt + (kCntMaxRow - kCntBad), (unsigned long long)s_longest);
  }
}

// ---- rebuild of the added arrays -----------------------------------------------------
// One scan over three segments: the n new added counts (prefix = the new
// offsets), the a_total kill marks, and the 2m endpoint slots (by vertex, in
// slot order) whose line appends its pair.  The last two give every survivor
// and every new entry its rank, so one more launch places them all.

struct RebuildCounts {
  int64_t n, a_total;
  const int64_t* aoff;
  const int32_t* adelta;
  const uint8_t* akill;
  const uint32_t* slot_vals;
  const uint8_t* app_line;
  __device__ __forceinline__ int64_t operator()(int64_t i) const {
    if (i < n) return aoff[i + 1] - aoff[i] + adelta[i];
    if (i < n + a_total) return akill[i - n];
    return app_line[slot_vals[i - n - a_total] >> 1];
  }
};

struct RebuildOut {   // tail[j]: prefix at item n + j
  int64_t n;
  int64_t* noff;
  int64_t* tail;
  __device__ __forceinline__ void operator()(int64_t i, int64_t v) const {
    if (i <= n) noff[i] = v;
    if (i >= n) tail[i - n] = v;
  }
};

__global__ void k_rebuild_added(const int64_t* aoff, const int32_t* aadj, const int32_t* aown, int64_t a_total,
                                const int64_t* noff, const int64_t* tail, const uint64_t* slot_keys,
                                const uint32_t* slot_vals, int64_t slots, const int32_t* u, const int32_t* v,
                                const uint8_t* app_line, const unsigned long long* bad, uint8_t* akill,
                                int32_t* adelta, int32_t* nadj, int32_t* nown) {
  pdl_wait();
  pdl_trigger();
  if (*bad != 0) return;
  const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (j < a_total) {
    // a surviving entry: behind the row's earlier survivors
    if (akill[j]) {
      akill[j] = 0;
      return;
    }
    const int32_t x = aown[j];
    const int64_t s = aoff[x];
    const int64_t pos = noff[x] + (j - s) - (tail[j] - tail[s]);
    nadj[pos] = aadj[j];
    nown[pos] = x;
    return;
  }
  const int64_t k = j - a_total;
  if (k >= slots) return;
  const int32_t x = (int32_t)slot_keys[k];
  adelta[x] = 0;
  const uint32_t slot = slot_vals[k];
  if (!app_line[slot >> 1]) return;
  // a new entry: behind the row's survivors and the vertex's earlier new ones;
  // the vertex's first slot is found by doubling steps back, then bisection
  int64_t lo = k, step = 1;
  while (lo > 0 && slot_keys[max(lo - step, (int64_t)0)] == (uint64_t)(uint32_t)x) {
    lo = max(lo - step, (int64_t)0);
    step *= 2;
  }
  if (lo > 0) {
    int64_t out = max(lo - step, (int64_t)0);   // another vertex's
    while (lo - out > 1) {
      const int64_t mid = (lo + out) >> 1;
      if (slot_keys[mid] == (uint64_t)(uint32_t)x) lo = mid; else out = mid;
    }
  }
  const int64_t b = aoff[x], e = aoff[x + 1];
  const int64_t survivors = (e - b) - (tail[e] - tail[b]);
  const int64_t pos = noff[x] + survivors + (tail[a_total + k] - tail[a_total + lo]);
  nadj[pos] = (slot & 1) ? u[slot >> 1] : v[slot >> 1];
  nown[pos] = x;
}

// isAdjacent (core/FlashGraph.h:291-301) for every update.
__global__ void k_flags(GraphView g, bool sorted, const int32_t* u, const int32_t* v, int64_t m, uint8_t* ins) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= m) return;
  const int32_t x = u[i], y = v[i];
  bool adj = added_find(g, x, y) >= 0;
  if (!adj) {
    int32_t l, d;
    base_copies(g, sorted, x, y, &l, &d);
    adj = l > 0;
  }
  ins[i] = adj ? 0 : 1;
}

// k_flags with the endpoint check folded in, for flag_updates_noalloc: a pair
// with an endpoint outside [0, n) or u == v is counted into *bad and gets no
// flag (the host then reports the batch as invalid and copies nothing out).
__global__ void k_flags_checked(GraphView g, bool sorted, const int32_t* u, const int32_t* v, int64_t m,
                                uint8_t* ins, unsigned long long* bad) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= m) return;
  const int32_t x = u[i], y = v[i];
  if (x < 0 || x >= g.n || y < 0 || y >= g.n || x == y) {
    atomicAdd(bad, 1ull);
    return;
  }
  bool adj = added_find(g, x, y) >= 0;
  if (!adj) {
    int32_t l, d;
    base_copies(g, sorted, x, y, &l, &d);
    adj = l > 0;
  }
  ins[i] = adj ? 0 : 1;
}

// ---- compaction --------------------------------------------------------------

__global__ void k_compact_check(GraphView g, const int32_t* deg, int64_t* counters) {
  int64_t x = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (x >= g.n) return;
  const int32_t d = deg[x];
  if (d < 0) atomicAdd((unsigned long long*)(counters + 0), 1ull);
  else if ((int64_t)d != row_len(g, x)) atomicAdd((unsigned long long*)(counters + 1), 1ull);
}

__global__ void k_compact_gather(GraphView g, const int64_t* noff, int32_t* out) {
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (warp >= g.n) return;
  const int32_t x = (int32_t)warp;
  int64_t o = noff[x];
  const int64_t b = g.nindex[x], e = g.nindex[x + 1];
  const bool filt = g.dead[x] != 0;
  for (int64_t k0 = b; k0 < e; k0 += 32) {
    const int64_t k = k0 + lane;
    const bool ok = k < e && (!filt || live_at(g.live, k));
    const unsigned msk = __ballot_sync(0xffffffffu, ok);
    if (ok) out[o + __popc(msk & ((1u << lane) - 1u))] = g.nlist[k];
    o += __popc(msk);
  }
  for (int64_t k0 = g.aoff[x]; k0 < g.aoff[x + 1]; k0 += 32) {
    const int64_t k = k0 + lane;
    if (k < g.aoff[x + 1]) out[o + lane] = g.aadj[k];
    o += min((int64_t)32, g.aoff[x + 1] - k0);
  }
}

// ---- greedy MIS in vertex order ------------------------------------------------
// x joins iff no lower-id neighbour joined.  States: 0 undecided, 1 in, 2 out.
// Warps take 32 vertices at a time in ascending id (list null), or 32 entries
// of a list (in the order in which the last pass gave them up).  A lane reads its row from the first lower neighbour that
// was not out yet: one that is in settles x out, an undecided one makes it try
// again, the row's end settles it in.  The lower vertices belong to tiles that
// other warps have already taken, so most settle while the lane waits; a tile
// gives up after kGreedyTries tries, and what it leaves undecided goes to the
// next pass's list.  The smallest undecided vertex waits for nobody, wherever
// it stands, so every pass settles some.
//
// Rounds that every vertex walks whole (its lower part up to a member) took 405,
// 173, 91, ... us on R-MAT scale 21, 950 us in twelve rounds: next to hubs most
// rows end at their first member, but in the first round there is none yet.
constexpr int kGreedyTries = 64;
constexpr int kGreedyStep = 4;   // entries read at once

struct GreedyRow {
  int64_t k, e;     // base positions from the cursor on
  int64_t ak, ae;   // added positions from the cursor on
  bool filt;
};

// Advances x's cursor; true once x is settled.
__device__ __forceinline__ bool greedy_try(const GraphView& g, bool sorted, int32_t x, GreedyRow& r, uint8_t* st) {
  volatile uint8_t* vst = st;
  while (r.k < r.e) {
    int32_t y[kGreedyStep];
    uint8_t s[kGreedyStep];
#pragma unroll
    for (int q = 0; q < kGreedyStep; ++q) y[q] = r.k + q < r.e ? __ldg(g.nlist + r.k + q) : x;
#pragma unroll
    for (int q = 0; q < kGreedyStep; ++q)
      s[q] = y[q] < x && (!r.filt || live_at(g.live, r.k + q)) ? vst[y[q]] : 2;
    int wait = kGreedyStep;
#pragma unroll
    for (int q = kGreedyStep - 1; q >= 0; --q) {
      if (s[q] == 1) {
        vst[x] = 2;
        return true;
      }
      if (s[q] == 0) wait = q;
    }
    if (wait < kGreedyStep) {
      r.k += wait;
      return false;
    }
    // sorted rows: the lower part ends at the first entry that is not lower
    r.k = sorted && y[kGreedyStep - 1] >= x ? r.e : r.k + kGreedyStep;
  }
  while (r.ak < r.ae) {
    const int32_t y = g.aadj[r.ak];
    const uint8_t s = y < x ? vst[y] : 2;
    if (s == 1) {
      vst[x] = 2;
      return true;
    }
    if (s == 0) return false;
    ++r.ak;
  }
  vst[x] = 1;
  return true;
}

// c[0]: next entry of the pass, c[1]: entries left for the next one.
__global__ void __launch_bounds__(kTB) k_greedy_pass(GraphView g, bool sorted, uint8_t* st, const int32_t* list,
                                                     int64_t cnt, int32_t* left, unsigned long long* c) {
  const int lane = threadIdx.x & 31;
  for (;;) {
    unsigned long long base = 0;
    if (lane == 0) base = atomicAdd(c, 32ull);
    base = __shfl_sync(0xffffffffu, base, 0);
    if ((int64_t)base >= cnt) return;
    const int64_t i = (int64_t)base + lane;
    const int32_t x = i < cnt ? (list ? list[i] : (int32_t)i) : 0;
    bool done = i >= cnt || *(volatile uint8_t*)(st + x) != 0;
    GreedyRow r{};
    if (!done) r = GreedyRow{g.nindex[x], g.nindex[x + 1], g.aoff[x], g.aoff[x + 1], g.dead[x] != 0};
    for (int t = 0; t < kGreedyTries; ++t) {
      if (!done) done = greedy_try(g, sorted, x, r, st);
      if (__all_sync(0xffffffffu, done)) break;
    }
    const unsigned open = __ballot_sync(0xffffffffu, !done);
    if (open) {
      unsigned long long at = 0;
      if (lane == 0) at = atomicAdd(c + 1, (unsigned long long)__popc(open));
      at = __shfl_sync(0xffffffffu, at, 0);
      if (!done) left[at + __popc(open & ((1u << lane) - 1u))] = x;
    }
  }
}

// ---- exact-MIS mode (no reference counterpart) -----------------------------------
// After a batch's repair: a member with a smaller-id member neighbour leaves
// (decided on the set the repair left), then the vertices with no member
// neighbour are completed in ascending id by the greedy rounds (state 1 in,
// 2 out, 0 undecided; non-members next to a member start out).

__global__ void k_exact_leave(GraphView g, bool sorted, const uint8_t* mis, uint8_t* leave) {
  const int64_t xi = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (xi >= g.n) return;
  const int32_t x = (int32_t)xi;
  bool found = false;
  if (mis[x] & 1) {
    const int64_t b = g.nindex[x], e = g.nindex[x + 1];
    const bool filt = g.dead[x] != 0;
    for (int64_t k = b; k < e && !found; ++k) {
      const int32_t y = g.nlist[k];
      if (sorted && y >= x) break;
      if (y >= x || (filt && !live_at(g.live, k))) continue;
      found = (mis[y] & 1) != 0;
    }
    for (int64_t k = g.aoff[x]; k < g.aoff[x + 1] && !found; ++k) {
      const int32_t y = g.aadj[k];
      found = y < x && (mis[y] & 1) != 0;
    }
  }
  leave[x] = found ? 1 : 0;
}

__global__ void k_exact_init(GraphView g, const uint8_t* mis, const uint8_t* leave, uint8_t* st) {
  const int64_t xi = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (xi >= g.n) return;
  const int32_t x = (int32_t)xi;
  auto member = [&](int32_t y) { return (mis[y] & 1) != 0 && leave[y] == 0; };
  if (member(x)) {
    st[x] = 1;
    return;
  }
  const bool covered = thread_row_until(g, x, [&](int32_t y) { return member(y); });
  st[x] = covered ? 2 : 0;
}

__global__ void k_exact_out(const uint8_t* st, int32_t n, uint8_t* mis) {
  const int64_t x = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (x < n) mis[x] = st[x] == 1 ? 1 : 0;
}

__global__ void k_greedy_out(const uint8_t* st, int32_t n, uint8_t* out) {
  int64_t x = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (x < n) out[x] = st[x] == 1 ? 1 : 0;
}

__global__ void k_check_mis(GraphView g, const uint8_t* mis, int64_t* counters) {
  int64_t xi = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (xi >= g.n) return;
  const int32_t x = (int32_t)xi;
  const bool in = mis[x] != 0;
  bool covered = in;
  int64_t viol = 0;
  thread_row_until(g, x, [&](int32_t y) {
    if (mis[y]) {
      covered = true;
      if (in && x < y) ++viol;
    }
    return false;
  });
  if (viol) atomicAdd((unsigned long long*)(counters + 0), (unsigned long long)viol);
  if (!covered) atomicAdd((unsigned long long*)(counters + 1), 1ull);
}

}  // namespace

void upload_base(mf_ctx* c, int32_t n, const int64_t* nindex, const int32_t* nlist, int64_t nnz) {
  cudaStream_t s = c->stream;
  c->n = n;
  c->nnz = nnz;
  c->nindex.reserve((int64_t)n + 1);
  c->nlist.reserve(nnz + kNlistPad);
  if (nindex) MF_CUDA(cudaMemcpyAsync(c->nindex.p, nindex, sizeof(int64_t) * ((size_t)n + 1), cudaMemcpyHostToDevice, s));
  if (nlist && nnz > 0) MF_CUDA(cudaMemcpyAsync(c->nlist.p, nlist, sizeof(int32_t) * (size_t)nnz, cudaMemcpyHostToDevice, s));
  const int64_t words = (nnz + 31) / 32;
  c->live.reserve(words);
  MF_CUDA(cudaMemsetAsync(c->live.p, 0xFF, sizeof(uint32_t) * (size_t)std::max<int64_t>(words, 1), s));
  c->dead.reserve(n);
  c->rcnt.reserve(n);
  c->deg.reserve(n);
  c->aoff.reserve((int64_t)n + 1);
  c->mis.reserve(n);
  c->cid.reserve(n);
  MF_CUDA(cudaMemsetAsync(c->dead.p, 0, sizeof(int32_t) * (size_t)n, s));
  MF_CUDA(cudaMemsetAsync(c->rcnt.p, 0, sizeof(int32_t) * (size_t)n, s));
  MF_CUDA(cudaMemsetAsync(c->aoff.p, 0, sizeof(int64_t) * ((size_t)n + 1), s));
  MF_CUDA(cudaMemsetAsync(c->mis.p, 0, (size_t)n, s));
  MF_CUDA(cudaMemsetAsync(c->cid.p, 0xFF, sizeof(int32_t) * (size_t)n, s));
  c->a_total = 0;
  alloc_vertex_scratch(c);
  if (n > 0) {
    MF_K(k_base_degree<<<grid_for(n), kTB, 0, s>>>(c->nindex.p, n, c->deg.p));
  }
  // validate and detect sorted rows
  MF_CUDA(cudaMemsetAsync(c->counters.p, 0xFF, sizeof(int64_t) * 4, s));
  int* okp = reinterpret_cast<int*>(c->counters.p);
  MF_K(k_check_index<<<grid_for((int64_t)n + 1), kTB, 0, s>>>(c->nindex.p, n, nnz, okp));
  if (nnz > 0) MF_K(k_check_ids<<<grid_for(std::min<int64_t>(nnz, (int64_t)1 << 22)), kTB, 0, s>>>(c->nlist.p, nnz, n, okp + 1));
  MF_CUDA(cudaStreamSynchronize(s));
  int ok[2] = {0, 0};
  MF_CUDA(cudaMemcpy(ok, okp, sizeof(ok), cudaMemcpyDeviceToHost));
  if (!ok[0]) MF_FAIL(MF_EFORMAT, "nindex is not a valid offset array (non-monotone or outside [0, entries])");
  if (!ok[1]) MF_FAIL(MF_EFORMAT, "nlist holds a vertex id outside [0, nodes)");
  // sorted rows and symmetry (both enable the pull form of the clustering write)
  if (n > 0) {
    DBuf<int32_t> all;
    DBuf<int64_t> offs;
    all.reserve(n);
    offs.reserve(2 * (int64_t)n + 1);
    MF_K(k_iota_n<<<grid_for(n), kTB, 0, s>>>(all.p, n));
    MF_K(k_base_positions<<<grid_for(n), kTB, 0, s>>>(c->nindex.p, n, offs.p + n + 1));
    scan_exclusive_i64(offs.p + n + 1, offs.p, n, c->ws, s);
    int sms = 0;
    MF_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c->device));
    MF_K(k_check_sorted<<<(unsigned)(sms * 8), kTB, 0, s>>>(c->view(), all.p, offs.p, n, okp + 2));
    MF_CUDA(cudaMemcpyAsync(ok, okp + 2, sizeof(int), cudaMemcpyDeviceToHost, s));
    MF_CUDA(cudaStreamSynchronize(s));
    c->rows_sorted = ok[0] != 0;
    c->symmetric = false;
    if (c->rows_sorted) {
      MF_K(k_check_symmetric<<<(unsigned)(sms * 8), kTB, 0, s>>>(c->view(), all.p, offs.p, n, okp + 3));
      MF_CUDA(cudaMemcpyAsync(ok, okp + 3, sizeof(int), cudaMemcpyDeviceToHost, s));
      MF_CUDA(cudaStreamSynchronize(s));
      c->symmetric = ok[0] != 0;
    }
    all.release();
    offs.release();
  } else {
    c->rows_sorted = true;
    c->symmetric = true;
  }
  c->tails.release();   // of another base
  c->max_csr = initial_max_csr(n, c->header_edges);
  c->max_row = -1;
}

// The n-sized scratch with its initial values: no row mapped (v2i = -1),
// epoch-tagged arrays at epoch 0, plus the device counters.
void alloc_vertex_scratch(mf_ctx* c) {
  cudaStream_t s = c->stream;
  const int32_t n = c->n;
  c->aoff_alt.reserve((int64_t)n + 1);
  c->v2i.reserve(n);
  c->bval.reserve(n);
  c->wval.reserve(n);
  c->f1.reserve(n);
  c->nlist_need.reserve(n);
  c->touched.reserve(n);
  c->hlist.reserve(n);
  c->adelta.reserve(n);
  if (n > 0) {
    MF_CUDA(cudaMemsetAsync(c->v2i.p, 0xFF, sizeof(int32_t) * (size_t)n, s));
    MF_CUDA(cudaMemsetAsync(c->bval.p, 0, sizeof(uint32_t) * (size_t)n, s));
    MF_CUDA(cudaMemsetAsync(c->wval.p, 0, sizeof(uint32_t) * (size_t)n, s));
    MF_CUDA(cudaMemsetAsync(c->adelta.p, 0, sizeof(int32_t) * (size_t)n, s));
  }
  c->epoch = 0;
  c->counters.reserve(kCounterWords);
}

void flag_updates(mf_ctx* c, int64_t m) {
  if (m <= 0) return;
  MF_K(k_flags<<<grid_for(m), kTB, 0, c->stream>>>(c->view(), c->rows_sorted, c->bu.p, c->bv.p, m, c->bins.p));
  MF_CUDA(cudaGetLastError());
}

void reserve_overlay(mf_ctx* c, int64_t m, Group& sized) {
  cudaStream_t s = c->stream;
  const int64_t n = c->n, a = c->a_total, slots = 2 * m;
  sized.add(c->bu, m);   // these three not again where the lines were copied to them
  sized.add(c->bv, m);
  sized.add(c->bins, m);
  sized.add(c->app_line, m);
  sized.add(c->keys, slots);
  sized.add(c->vals, slots);
  sized.add(c->slot_keys, slots);
  sized.add(c->slot_vals, slots);
  sized.add(c->prev, slots);
  // grown with every mark cleared: the rebuild clears the ones it used
  if (c->akill.grow(std::max<int64_t>(a, 1)))
    MF_CUDA(cudaMemsetAsync(c->akill.p, 0, (size_t)c->akill.cap, s));
  c->aadj_alt.grow(a + slots);
  c->aown_alt.grow(a + slots);
  c->aadj.reserve(std::max<int64_t>(a, 1));
  c->aown.reserve(std::max<int64_t>(a, 1));
  c->atail.grow(a + slots + 1);
  reserve_sort(c->ws, slots, s);
  scan_detail::reserve_scan(c->ws, n + a + slots, s);
}

void apply_overlay(mf_ctx* c, const BatchIn& in, int64_t m) {
  cudaStream_t s = c->stream;
  const int nbits = bits_for(std::max<int32_t>(c->n - 1, 1));
  // pairs are grouped on mixed bits, three to ten more than the line count
  // needs: two 8-bit digits up to 2^13 lines and three up to 2^21, where the
  // pair itself has 2 * nbits bits (six digits at 2^22 vertices)
  const int gbits = std::min(64, (bits_for(m) + 3 + 7) / 8 * 8);
  SortedPairs pairs{c->keys.p, c->vals.p};
  if (m <= kSmallBatch) {
    const int slots = (int)(2 * m);
    if (slots <= 256) small_input<1>(c, in, (int)m, 256, nbits, gbits);
    else if (slots <= 1024) small_input<1>(c, in, (int)m, 1024, nbits, gbits);
    else if (slots <= 2048) small_input<2>(c, in, (int)m, 1024, nbits, gbits);
    else if (slots <= 4096) small_input<4>(c, in, (int)m, 1024, nbits, gbits);
    else small_input<8>(c, in, (int)m, 1024, nbits, gbits);
  } else {
    MF_K(k_stage<<<grid_for(m), kTB, 0, s>>>(in, m, c->n, nbits, c->bu.p, c->bv.p, c->bins.p, c->app_line.p, c->keys.p,
                                             c->vals.p, c->slot_keys.p, c->slot_vals.p, c->work.p + kCntBad));
    pairs = radix_group_pairs(c->keys.p, c->vals.p, m, gbits, c->ws, s);
  }
  if (c->max_row < 0) MF_K(k_max_row<<<grid_for(c->n), kTB, 0, s>>>(c->view(), c->work.p + kCntMaxRow));
  MF_K(launch_pdl(k_apply_pairs, grid_for(m), kTB, 0, s, c->view(), c->live.p, c->dead.p, c->rcnt.p, c->deg.p,
                  c->rows_sorted, pairs.keys, pairs.vals, m, nbits, gbits, c->bu.p, c->bv.p, c->bins.p, c->adelta.p,
                  c->akill.p, c->app_line.p, c->work.p + kCntBad));
  if (m > kSmallBatch) {
    radix_sort_pairs_in_place(c->slot_keys.p, c->slot_vals.p, 2 * m, 0, nbits, c->ws, s);
    MF_K(launch_pdl(k_prev, grid_for(2 * m), kTB, 0, s, c->slot_keys.p, c->slot_vals.p, 2 * m, c->prev.p));
  }
  MF_CUDA(cudaGetLastError());
}

void rebuild_added(mf_ctx* c, int64_t m) {
  cudaStream_t s = c->stream;
  const int64_t n = c->n, a = c->a_total, slots = 2 * m;
  scan_exclusive_to(RebuildCounts{n, a, c->aoff.p, c->adelta.p, c->akill.p, c->slot_vals.p, c->app_line.p},
                    RebuildOut{n, c->aoff_alt.p, c->atail.p}, n + a + slots, c->ws, s);
  MF_K(launch_pdl(k_rebuild_added, grid_for(a + slots), kTB, 0, s, c->aoff.p, c->aadj.p, c->aown.p, a, c->aoff_alt.p,
                  c->atail.p, c->slot_keys.p, c->slot_vals.p, slots, c->bu.p, c->bv.p, c->app_line.p,
                  c->work.p + kCntBad, c->akill.p, c->adelta.p, c->aadj_alt.p, c->aown_alt.p));
  MF_CUDA(cudaGetLastError());
}

void swap_overlay(mf_ctx* c, int64_t appended, int64_t killed) {
  std::swap(c->aoff, c->aoff_alt);
  std::swap(c->aadj, c->aadj_alt);
  std::swap(c->aown, c->aown_alt);
  c->a_total += appended - killed;
}

void compact_graph(mf_ctx* c, std::vector<int64_t>& nindex_out, std::vector<int32_t>& nlist_out) {
  cudaStream_t s = c->stream;
  const int32_t n = c->n;
  MF_CUDA(cudaMemsetAsync(c->counters.p, 0, sizeof(int64_t) * 2, s));
  if (n > 0) MF_K(k_compact_check<<<grid_for(n), kTB, 0, s>>>(c->view(), c->deg.p, c->counters.p));
  MF_CUDA(cudaMemcpyAsync(c->h_counters, c->counters.p, sizeof(int64_t) * 2, cudaMemcpyDeviceToHost, s));
  MF_CUDA(cudaStreamSynchronize(s));
  if (c->h_counters[0] > 0) MF_FAIL(MF_ESTATE, "compaction computed a negative degree: delta is inconsistent with the base graph");
  if (c->h_counters[1] > 0) MF_FAIL(MF_ESTATE, "compaction degree mismatch: tombstones without base entries (asymmetric base graph)");
  c->i64b.reserve((int64_t)n + 1);
  scan_exclusive_i32(c->deg.p, c->i64b.p, n, c->ws, s);
  int64_t total = 0;
  MF_CUDA(cudaMemcpyAsync(&total, c->i64b.p + n, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
  MF_CUDA(cudaStreamSynchronize(s));
  DBuf<int32_t> out;
  out.reserve(std::max<int64_t>(total, 1));
  if (n > 0) MF_K(k_compact_gather<<<grid_for((int64_t)n * 32), kTB, 0, s>>>(c->view(), c->i64b.p, out.p));
  MF_CUDA(cudaGetLastError());
  nindex_out.resize((size_t)n + 1);
  nlist_out.resize((size_t)total);
  MF_CUDA(cudaMemcpyAsync(nindex_out.data(), c->i64b.p, sizeof(int64_t) * ((size_t)n + 1), cudaMemcpyDeviceToHost, s));
  if (total > 0) MF_CUDA(cudaMemcpyAsync(nlist_out.data(), out.p, sizeof(int32_t) * (size_t)total, cudaMemcpyDeviceToHost, s));
  MF_CUDA(cudaStreamSynchronize(s));
  out.release();
}

namespace {

// Settles every undecided vertex of st, pass by pass.  A pass settles at least
// the smallest undecided one.  Lists alternate between two n-sized scratch
// arrays that nothing uses between batches.
void greedy_settle(mf_ctx* c, uint8_t* st, const char* failure) {
  cudaStream_t s = c->stream;
  const int64_t n = c->n;
  int sms = 0;
  MF_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c->device));
  unsigned long long* cnt = reinterpret_cast<unsigned long long*>(c->counters.p);
  const int32_t* list = nullptr;
  int32_t* left = c->touched.p;
  int64_t todo = n;
  for (int64_t pass = 0;; ++pass) {
    MF_CUDA(cudaMemsetAsync(cnt, 0, 2 * sizeof(unsigned long long), s));
    MF_K(k_greedy_pass<<<(unsigned)std::min<int64_t>(grid_for(todo), (int64_t)8 * sms), kTB, 0, s>>>(
        c->view(), c->rows_sorted, st, list, todo, left, cnt));
    MF_CUDA(cudaMemcpyAsync(c->h_counters, cnt, 2 * sizeof(int64_t), cudaMemcpyDeviceToHost, s));
    MF_CUDA(cudaStreamSynchronize(s));
    todo = c->h_counters[1];
    if (todo == 0) return;
    if (pass > n + 2) MF_FAIL(MF_ESTATE, failure);
    list = left;
    left = left == c->touched.p ? c->nlist_need.p : c->touched.p;
  }
}

}  // namespace

void greedy_mis(mf_ctx* c, uint8_t* out) {
  cudaStream_t s = c->stream;
  const int32_t n = c->n;
  if (n <= 0) return;
  c->xst.reserve(n);
  c->xleave.reserve(n);
  MF_CUDA(cudaMemsetAsync(c->xst.p, 0, (size_t)n, s));
  greedy_settle(c, c->xst.p, "greedy MIS did not settle");
  MF_K(k_greedy_out<<<grid_for(n), kTB, 0, s>>>(c->xst.p, n, c->xleave.p));
  MF_CUDA(cudaMemcpyAsync(out, c->xleave.p, (size_t)n, cudaMemcpyDeviceToHost, s));
  MF_CUDA(cudaStreamSynchronize(s));
}

void exact_fixup(mf_ctx* c) {
  cudaStream_t s = c->stream;
  const int32_t n = c->n;
  if (n <= 0) return;
  c->xst.reserve(n);
  c->xleave.reserve(n);
  MF_K(k_exact_leave<<<grid_for(n), kTB, 0, s>>>(c->view(), c->rows_sorted, c->mis.p, c->xleave.p));
  MF_K(k_exact_init<<<grid_for(n), kTB, 0, s>>>(c->view(), c->mis.p, c->xleave.p, c->xst.p));
  greedy_settle(c, c->xst.p, "exact-MIS completion did not settle");
  MF_K(k_exact_out<<<grid_for(n), kTB, 0, s>>>(c->xst.p, n, c->mis.p));
  MF_CUDA(cudaGetLastError());
}

void check_mis(mf_ctx* c, int64_t* viol, int64_t* uncovered) {
  cudaStream_t s = c->stream;
  MF_CUDA(cudaMemsetAsync(c->counters.p, 0, sizeof(int64_t) * 2, s));
  if (c->n > 0) MF_K(k_check_mis<<<grid_for(c->n), kTB, 0, s>>>(c->view(), c->mis.p, c->counters.p));
  MF_CUDA(cudaMemcpyAsync(c->h_counters, c->counters.p, sizeof(int64_t) * 2, cudaMemcpyDeviceToHost, s));
  MF_CUDA(cudaStreamSynchronize(s));
  *viol = c->h_counters[0];
  *uncovered = c->h_counters[1];
}

void rebase(mf_ctx* c) {
  std::vector<int64_t> ni;
  std::vector<int32_t> nl;
  compact_graph(c, ni, nl);
  // keep membership and cluster ids; the base becomes the compacted graph
  DBuf<uint8_t> mis_keep;
  DBuf<int32_t> cid_keep;
  cudaStream_t s = c->stream;
  const int32_t n = c->n;
  mis_keep.reserve(std::max(n, 1));
  cid_keep.reserve(std::max(n, 1));
  MF_CUDA(cudaMemcpyAsync(mis_keep.p, c->mis.p, (size_t)n, cudaMemcpyDeviceToDevice, s));
  MF_CUDA(cudaMemcpyAsync(cid_keep.p, c->cid.p, sizeof(int32_t) * (size_t)n, cudaMemcpyDeviceToDevice, s));
  c->nlist.release();
  c->live.release();
  c->header_edges = (uint64_t)nl.size();
  const int64_t keep_max = c->max_csr;
  upload_base(c, n, ni.data(), nl.data(), (int64_t)nl.size());
  c->max_csr = keep_max;
  MF_CUDA(cudaMemcpyAsync(c->mis.p, mis_keep.p, (size_t)n, cudaMemcpyDeviceToDevice, s));
  MF_CUDA(cudaMemcpyAsync(c->cid.p, cid_keep.p, sizeof(int32_t) * (size_t)n, cudaMemcpyDeviceToDevice, s));
  MF_CUDA(cudaStreamSynchronize(s));
  mis_keep.release();
  cid_keep.release();
}

}  // namespace mf

// ---- update flags without allocation ------------------------------------------
// mf_flag_updates stages the endpoints in the context's buffers, which grow
// to the largest batch seen (cudaFree of the old buffer + cudaMalloc).  This
// variant stages them in one fixed device array instead, so that it never
// allocates: every call on a device uses the same array, found once per
// device with cudaGetSymbolAddress.
//
// Layout of the array (byte offsets, each part 256-byte aligned):
//   [0, 256)                     invalid-pair counter (u64; zeroed every call)
//   [256, 256 + 4K)              u endpoints (int32, K = MF_NOALLOC_MAX_UPDATES)
//   [256 + 4K, 256 + 8K)         v endpoints
//   [256 + 8K, 256 + 9K)         flags (u8)
// K = 65536 gives 590,080 bytes.
namespace {
constexpr size_t kNaCounterBytes = 256;
constexpr size_t kNaEndpointBytes = sizeof(int32_t) * (size_t)MF_NOALLOC_MAX_UPDATES;
constexpr size_t kNaScratchBytes = kNaCounterBytes + 2 * kNaEndpointBytes + (size_t)MF_NOALLOC_MAX_UPDATES;
constexpr int kNaMaxDevices = 64;
static_assert(kNaEndpointBytes % 256 == 0, "each part of the scratch starts on a 256-byte boundary");
}  // namespace

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNaScratchBytes];

namespace mf {
namespace {

std::mutex g_na_mutex;
unsigned char* g_na_base[kNaMaxDevices] = {};

// Device address of the scratch array on the current device (which must be
// `device`).  The first call for a device looks it up; later calls read the
// table.
unsigned char* noalloc_scratch(int device) {
  if (device < 0 || device >= kNaMaxDevices) MF_FAIL(MF_ELIMIT, "device id beyond the no-allocation table (64)");
  std::lock_guard<std::mutex> lock(g_na_mutex);
  if (g_na_base[device] == nullptr) {
    void* p = nullptr;
    MF_CUDA(cudaGetSymbolAddress(&p, g_noalloc_scratch));
    if (p == nullptr) MF_FAIL(MF_ECUDA, "cudaGetSymbolAddress returned a null scratch address");
    g_na_base[device] = static_cast<unsigned char*>(p);
  }
  return g_na_base[device];
}

}  // namespace

// Looks the scratch address up again for `device` (current on the calling
// thread).  Contexts call this when they are created, so that a device
// whose primary context was reset and re-created gets the new address.
void noalloc_refresh(int device) {
  if (device < 0 || device >= kNaMaxDevices) return;
  void* p = nullptr;
  MF_CUDA(cudaGetSymbolAddress(&p, g_noalloc_scratch));
  std::lock_guard<std::mutex> lock(g_na_mutex);
  g_na_base[device] = static_cast<unsigned char*>(p);
}

void flag_updates_noalloc(mf_ctx* c, const int32_t* u, const int32_t* v, int64_t m, uint8_t* ins_out) {
  if (m > (int64_t)MF_NOALLOC_MAX_UPDATES)
    MF_FAIL(MF_ELIMIT, "mf_flag_updates_noalloc takes at most 65536 updates per call");
  unsigned char* base = noalloc_scratch(c->device);
  if (m <= 0) return;
  cudaStream_t s = c->stream;
  auto* bad = reinterpret_cast<unsigned long long*>(base);
  auto* du = reinterpret_cast<int32_t*>(base + kNaCounterBytes);
  auto* dv = reinterpret_cast<int32_t*>(base + kNaCounterBytes + kNaEndpointBytes);
  auto* dins = base + kNaCounterBytes + 2 * kNaEndpointBytes;
  // the counter is the only part read before it is written
  MF_CUDA(cudaMemsetAsync(bad, 0, sizeof(unsigned long long), s));
  MF_CUDA(cudaMemcpyAsync(du, u, sizeof(int32_t) * (size_t)m, cudaMemcpyHostToDevice, s));
  MF_CUDA(cudaMemcpyAsync(dv, v, sizeof(int32_t) * (size_t)m, cudaMemcpyHostToDevice, s));
  MF_K(k_flags_checked<<<grid_for(m), kTB, 0, s>>>(c->view(), c->rows_sorted, du, dv, m, dins, bad));
  MF_CUDA(cudaGetLastError());
  unsigned long long nbad = 0;
  MF_CUDA(cudaMemcpyAsync(&nbad, bad, sizeof(nbad), cudaMemcpyDeviceToHost, s));
  MF_CUDA(cudaStreamSynchronize(s));
  if (nbad != 0) MF_FAIL(MF_EINVAL, "update endpoints must be distinct vertex ids in [0, n)");
  MF_CUDA(cudaMemcpyAsync(ins_out, dins, (size_t)m, cudaMemcpyDeviceToHost, s));
  MF_CUDA(cudaStreamSynchronize(s));
}

}  // namespace mf
