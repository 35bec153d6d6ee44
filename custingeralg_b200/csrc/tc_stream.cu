// Streaming triangle counting: batch preparation, structural updates of the slack-managed
// adjacency and the triangle delta of a batch (sm_100a).
//
// Replaces the reference's three streaming kernels devicecuStingerNewTriangles,
// deviceBUThreeTriangles and deviceBUTwoCUOneTriangles (src/streaming_triangle_counting/
// cct_upd.cu:231-410), whose inclusion-exclusion nets +2 per vertex of every new triangle on a
// symmetric batch (K1 counts a triangle with k new edges k times, K2 and K3 correct the
// overcount). Here a triangle is attributed once, to the smallest of its changed edges in the
// (min id, max id) order: N(x) and N(y) are intersected for each changed edge {x, y}, which keeps
// a common neighbour w unless (x, w) or (y, w) is a changed edge with a smaller key. Whether an
// edge is changed comes either from a per-slot mark array parallel to the adjacency pool
// (tc_apply_batch) or from a lookup in the sorted batch (the cuStinger-style path).
//
// With marks, an edge whose longer list belongs to a hub of the batch is counted there
// (k_delta_hub); the others by a warp each (k_delta_fused), which searches the shorter list's entries
// in the longer one ("search") or, where the strategy table asks for it, stages the longer list into
// shared memory piece by piece with cp.async and searches it there ("stage"). The cuStinger-style path
// (k_delta, k_delta_split) chooses by the lengths or the table between search and, for balanced
// pairs, a partitioned merge in which each lane owns a contiguous slice of the shorter list and
// merges it against the longer one from a binary-searched start ("merge").
#include <cub/cub.cuh>

#include <algorithm>
#include <condition_variable>
#include <cstring>
#include <mutex>

#include "tc_graph.cuh"
#include "tc_pipe_tune.h"

namespace tc {

namespace {

constexpr int kThreads = 256;
constexpr uint64_t kSentinel = ~0ull;
constexpr int kLongList = 2048;  // lists longer than this are rewritten in pieces, by many CTAs
constexpr int64_t kDeltaItems = 1 << 20;  // capacity of the split-item queue
constexpr unsigned long long kNoItem = ~0ull;
constexpr int kGrab = 4;  // most changed edges a warp takes per grab from the delta kernel's queue
// Bound of the wait in which the persistent delta kernel's CTAs meet (a wait that runs out reports
// kErrTimeout).
constexpr unsigned long long kSpinNs = 2000000000ull;  // 2 s
constexpr unsigned kSpinMaxIters = 1u << 24;

enum : unsigned { kErrRange = 1u, kErrPool = 2u, kErrTimeout = 4u, kErrScratch = 8u };
constexpr unsigned kLastSelfLoop = 16u;  // not an error: an entry with the sentinels' low bits (tc_insert_sorted)
// first_del[v] between batches: no deletion marked in v's list (0x7f7f7f7f, a byte memset)
constexpr int32_t kNoDel = 0x7f7f7f7f;
constexpr unsigned long long kNoLongItem = ~0ull;

struct BatchStatus {
  unsigned long long n_del;       // effective deletions
  unsigned long long n_ins;       // effective insertions
  unsigned long long n_dir;       // directed insert entries (2 n_ins)
  unsigned long long n_runs;      // affected source vertices of insertions
  unsigned long long demand;      // pool slots relocations may take
  unsigned long long tri_removed;
  unsigned long long tri_added;
  unsigned long long pool_top;    // device copy of the bump pointer
  unsigned long long dir_added;   // directed entries inserted (cuStinger path)
  unsigned long long dir_removed; // directed entries deleted (cuStinger path)
  unsigned long long not_fitting;
  unsigned long long n_long;      // insertion runs whose list is long (plan_long_run)
  unsigned long long long_scr;    // scratch entries and work items of the long-list insertion
  unsigned long long long_items;
  unsigned long long n_cmp;       // long lists compacted, their scratch entries and work items
  unsigned long long cmp_scr;
  unsigned long long cmp_items;
  unsigned long long n_split[2];  // split-intersection items queued (deletions, insertions)
  unsigned long long delta_bytes; // algorithmic bytes of the batch's intersections (4(deg x + deg y) + 8 each)
  unsigned int arrived[2];        // CTAs of the persistent delta kernel done with the count
  unsigned int err;
  unsigned int pad;
  unsigned long long n_hubs[2];   // hub groups of the delta count (deletions, insertions)
  unsigned long long hub_total[2];  // changed edges placed in hub groups
  unsigned long long hub_q[2];    // work-queue heads of the hub kernel
  unsigned long long hub_items[2];  // hub work items queued
  unsigned long long n_desc[2];   // changed edges left to the per-edge kernel
  unsigned long long e_next[2];   // work-queue heads of the delta kernel's edges and of its split items
  unsigned long long i_next[2];
};

__device__ __forceinline__ uint64_t ekey(int32_t a, int32_t b) {
  const uint32_t lo = (uint32_t)min(a, b), hi = (uint32_t)max(a, b);
  return ((uint64_t)lo << 32) | hi;
}

template <typename T>
__device__ __forceinline__ T warp_sum(T x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(kFull, x, o);
  return x;
}

// First index in [lo, hi) of list with list[i] >= key.
__device__ __forceinline__ int64_t lower_bound(const int32_t* __restrict__ list, int64_t lo, int64_t hi, int32_t key) {
  while (lo < hi) {
    const int64_t mid = lo + ((hi - lo) >> 1);
    if (__ldg(list + mid) < key) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

// First index of the ascending list lst[0 .. len) whose entry is >= key, found by the warp: 32
// evenly spaced samples per round (one load each lane), so a list of up to 32^r entries takes r
// rounds. Every lane returns the same index.
__device__ __forceinline__ int32_t warp_lower_bound(const int32_t* __restrict__ lst, int32_t len, int32_t key) {
  const int lane = threadIdx.x & 31;
  int32_t lo = 0, hi = len;  // the answer lies in [lo, hi]
  while (hi - lo > 32) {
    const int32_t step = (hi - lo + 31) / 32;
    const int32_t p = lo + lane * step;
    const int32_t v = p < hi ? lst[p] : INT32_MAX;
    const int c = __popc(__ballot_sync(kFull, v < key));  // the samples below key are a prefix
    const int32_t nlo = c > 0 ? lo + (c - 1) * step + 1 : lo;
    hi = c < 32 ? min(hi, lo + c * step) : hi;
    lo = nlo;
  }
  const int32_t p = lo + lane;
  const int32_t v = p < hi ? lst[p] : INT32_MAX;
  return lo + __popc(__ballot_sync(kFull, v < key));
}

// Asynchronous 4-byte copy from global to shared memory (cp.async, no register round trip); the
// copies of a thread complete at cp_async_wait_all.
__device__ __forceinline__ void cp_async4(int32_t* smem_dst, const int32_t* gsrc) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(smem_dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// GPU-scope relaxed load (a poll of another CTA's arrival).
__device__ __forceinline__ unsigned ld_relaxed(const unsigned* p) {
  unsigned v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

int grid_for(int64_t items, int per_block) {
  const int64_t want = std::max<int64_t>(1, (items + per_block - 1) / per_block);
  return (int)std::min<int64_t>(want, (int64_t)device_info().sms * 16);
}

// ---- batch preparation (canonical undirected updates) --------------------------------------

// key = (min << (L+1)) | (max << 1) | is_insert; self-loops and bad ids become the sentinel
// (1 << (2L+1)) - 1, and so do the entries [b, cap) of a padded batch.
__device__ __forceinline__ uint64_t update_key(const int32_t* __restrict__ src, const int32_t* __restrict__ dst,
                                               const uint8_t* __restrict__ is_del, const int64_t i, const int64_t b,
                                               const int32_t n, const int L, BatchStatus* __restrict__ st) {
  const uint64_t sent = (1ull << (2 * L + 1)) - 1;
  if (i >= b) return sent;
  const int32_t s = src[i], d = dst[i];
  if (s < 0 || s >= n || d < 0 || d >= n) {
    atomicOr(&st->err, kErrRange);
    return sent;
  }
  if (s == d) return sent;
  const uint64_t lo = (uint64_t)min(s, d), hi = (uint64_t)max(s, d);
  return (lo << (L + 1)) | (hi << 1) | (uint64_t)((is_del && is_del[i]) ? 0 : 1);
}

// The keys of a batch of b updates, padded to cap entries, and the directed keys' padding.
__global__ void __launch_bounds__(kThreads) k_load_keys(const int32_t* __restrict__ src, const int32_t* __restrict__ dst,
                                                        const uint8_t* __restrict__ is_del, const int64_t b,
                                                        const int64_t cap, const int32_t n, const int L,
                                                        uint64_t* __restrict__ keys, uint64_t* __restrict__ dirkeys,
                                                        BatchStatus* __restrict__ st) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < cap; i += (int64_t)gridDim.x * blockDim.x) {
    keys[i] = update_key(src, dst, is_del, i, b, n, L, st);
    reinterpret_cast<ulonglong2*>(dirkeys)[i] = make_ulonglong2(kSentinel, kSentinel);
  }
}

// ---- small batches: sorted by one CTA ------------------------------------------------------
//
// A batch of at most kSmallBatch updates is bound by its launches: each of the library sort's is 13 us
// or more here, between kernels of a few dependent loads. One CTA sorts its keys in shared memory
// instead, in the kernels that make them and use them.
constexpr int64_t kSmallBatch = 2048;
constexpr int kSortThreads = 1024;

// Ascending bitonic sort of P >= 32 (a power of two) keys in shared memory by the CTA. Exchanges at a
// distance below 32 stay in registers (shuffles), so P = 1024 takes 21 block barriers, not 55.
__device__ __forceinline__ void cta_sort(uint64_t* __restrict__ k, const int P) {
  auto exchange = [](const uint64_t x, const int i, const int h, const int size) {
    const uint64_t y = __shfl_xor_sync(kFull, x, h);
    return (((i & h) == 0) == ((i & size) == 0)) == (x < y) ? x : y;  // equal keys: either
  };
  for (int i = threadIdx.x; i < P; i += kSortThreads) {  // P a multiple of 32: whole warps
    uint64_t x = k[i];
#pragma unroll
    for (int size = 2; size <= 32; size <<= 1)
#pragma unroll
      for (int h = size >> 1; h > 0; h >>= 1) x = exchange(x, i, h, size);
    k[i] = x;
  }
  __syncthreads();
  for (int size = 64; size <= P; size <<= 1) {
    for (int h = size >> 1; h >= 32; h >>= 1) {
      for (int p = threadIdx.x; p < P / 2; p += kSortThreads) {
        const int i = ((p & ~(h - 1)) << 1) | (p & (h - 1)), j = i | h;
        const uint64_t x = k[i], y = k[j];
        if ((x > y) == ((i & size) == 0)) {
          k[i] = y;
          k[j] = x;
        }
      }
      __syncthreads();
    }
    for (int i = threadIdx.x; i < P; i += kSortThreads) {
      uint64_t x = k[i];
#pragma unroll
      for (int h = 16; h > 0; h >>= 1) x = exchange(x, i, h, size);
      k[i] = x;
    }
    __syncthreads();
  }
}

__device__ __forceinline__ int pow2_at_least(const int64_t n) {
  int P = 32;
  while (P < n) P <<= 1;
  return P;
}

// The sorted keys of a batch of b <= cap <= kSmallBatch updates, padded to cap.
__global__ void __launch_bounds__(kSortThreads) k_load_sorted(const int32_t* __restrict__ src,
                                                              const int32_t* __restrict__ dst,
                                                              const uint8_t* __restrict__ is_del, const int64_t b,
                                                              const int64_t cap, const int32_t n, const int L,
                                                              uint64_t* __restrict__ sorted, BatchStatus* __restrict__ st) {
  __shared__ uint64_t k[kSmallBatch];
  const int P = pow2_at_least(b);
  for (int i = threadIdx.x; i < P; i += kSortThreads) k[i] = update_key(src, dst, is_del, i, b, n, L, st);
  __syncthreads();
  cta_sort(k, P);
  const uint64_t sent = (1ull << (2 * L + 1)) - 1;
  for (int i = threadIdx.x; i < cap; i += kSortThreads) sorted[i] = i < P ? k[i] : sent;
}

// ---- classification ------------------------------------------------------------------------

// The run of equal edges starting at i, if one does: does it delete, does it insert.
__device__ __forceinline__ bool edge_run(const uint64_t* __restrict__ keys, const int64_t i, const int64_t b, const int L,
                                         bool& del_any, bool& ins_any) {
  const uint64_t k = keys[i], e = k >> 1;
  if (k == (1ull << (2 * L + 1)) - 1 || (i > 0 && (keys[i - 1] >> 1) == e)) return false;
  int64_t j = i;
  while (j + 1 < b && (keys[j + 1] >> 1) == e) ++j;
  del_any = (k & 1ull) == 0;        // deletions sort before insertions of the same edge
  ins_any = (keys[j] & 1ull) == 1;
  return true;
}

// Append an effective deletion (the edge's places in both lists) or insertion (its directed keys,
// (src << L) | dst).
__device__ __forceinline__ void append_change(const bool is_del, const int32_t x, const int32_t y, const int32_t px,
                                              const int32_t py, const int L, int4* __restrict__ dlist,
                                              int2* __restrict__ ilist, uint64_t* __restrict__ dirkeys,
                                              BatchStatus* __restrict__ st) {
  if (is_del) {
    dlist[atomicAdd(&st->n_del, 1ull)] = make_int4(x, y, px, py);
  } else {
    const unsigned long long at = atomicAdd(&st->n_ins, 1ull);
    ilist[at] = make_int2(x, y);
    dirkeys[2 * at] = ((uint64_t)(uint32_t)x << L) | (uint32_t)y;
    dirkeys[2 * at + 1] = ((uint64_t)(uint32_t)y << L) | (uint32_t)x;
  }
}

// Each unique undirected edge: classify against the graph and append to the deletion or the
// insertion list. A thread per key; a deletion records the edge's places in both lists.
__global__ void k_classify(const SlackView g, const uint64_t* __restrict__ keys, const int64_t b, const int L,
                           int4* __restrict__ dlist, int2* __restrict__ ilist, uint64_t* __restrict__ dirkeys,
                           BatchStatus* __restrict__ st) {
  const uint64_t maxmask = (1ull << L) - 1;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < b; i += (int64_t)gridDim.x * blockDim.x) {
    bool del_any, ins_any;
    if (!edge_run(keys, i, b, L, del_any, ins_any)) continue;
    const uint64_t e = keys[i] >> 1;
    const int32_t x = (int32_t)(e >> L), y = (int32_t)(e & maxmask);
    // presence: search the shorter list
    const int32_t lx = g.len(x), ly = g.len(y);
    const int64_t sx = g.start(x), sy = g.start(y);
    int64_t px = -1, py = -1;
    if (lx <= ly) {
      const int64_t p = lower_bound(g.ind, sx, sx + lx, y);
      if (p < sx + lx && g.ind[p] == y) px = p - sx;
    } else {
      const int64_t p = lower_bound(g.ind, sy, sy + ly, x);
      if (p < sy + ly && g.ind[p] == x) py = p - sy;
    }
    const bool present = px >= 0 || py >= 0;
    if (del_any && !ins_any && present) {
      if (px < 0) px = lower_bound(g.ind, sx, sx + lx, y) - sx;
      if (py < 0) py = lower_bound(g.ind, sy, sy + ly, x) - sy;
      append_change(true, x, y, (int32_t)px, (int32_t)py, L, dlist, ilist, dirkeys, st);
    } else if (ins_any && !present) {
      append_change(false, x, y, 0, 0, L, dlist, ilist, dirkeys, st);
    }
  }
}

// The same, a warp per key: 32 samples a round, so a list of 10^5 entries takes four dependent loads
// instead of seventeen. For batches that leave most warps idle otherwise.
__global__ void k_classify_warp(const SlackView g, const uint64_t* __restrict__ keys, const int64_t b, const int L,
                                int4* __restrict__ dlist, int2* __restrict__ ilist, uint64_t* __restrict__ dirkeys,
                                BatchStatus* __restrict__ st) {
  const uint64_t maxmask = (1ull << L) - 1;
  const int lane = threadIdx.x & 31;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < b; i += nw) {
    bool del_any, ins_any;
    if (!edge_run(keys, i, b, L, del_any, ins_any)) continue;
    const uint64_t e = keys[i] >> 1;
    const int32_t x = (int32_t)(e >> L), y = (int32_t)(e & maxmask);
    const int32_t lx = g.len(x), ly = g.len(y);
    const int32_t* const nx = g.ind + g.start(x);
    const int32_t* const ny = g.ind + g.start(y);
    const bool x_short = lx <= ly;
    const int32_t ps = x_short ? warp_lower_bound(nx, lx, y) : warp_lower_bound(ny, ly, x);
    const bool present = x_short ? ps < lx && nx[ps] == y : ps < ly && ny[ps] == x;
    if (del_any && !ins_any && present) {
      const int32_t pl = x_short ? warp_lower_bound(ny, ly, x) : warp_lower_bound(nx, lx, y);
      if (lane == 0) append_change(true, x, y, x_short ? ps : pl, x_short ? pl : ps, L, dlist, ilist, dirkeys, st);
    } else if (ins_any && !present) {
      if (lane == 0) append_change(false, x, y, 0, 0, L, dlist, ilist, dirkeys, st);
    }
    __syncwarp();
  }
}

// ---- insertion planning / application ------------------------------------------------------

__device__ __forceinline__ int32_t dir_src(const uint64_t k, const int L) { return (int32_t)(k >> L); }
__device__ __forceinline__ int32_t dir_dst(const uint64_t k, const int L) {
  return (int32_t)((uint32_t)k & (uint32_t)((1ull << L) - 1));
}

// Heads of source-vertex runs in the sorted directed entries ((src << L) | dst), and the pool slots
// the lists that must move could take (computed on the pre-deletion lengths, an upper bound).
// A run is stored as (start, length), one whose list will be long (used + new > kLongList) as
// (-1 - start, length).
__device__ __forceinline__ void dir_run(const uint64_t* __restrict__ dk, const int64_t i, const int64_t nd_cap, const int L,
                                        const int32_t* __restrict__ used, const int32_t* __restrict__ cap,
                                        const int32_t slack_q10, int2* __restrict__ runs,
                                        BatchStatus* __restrict__ st) {
  const uint64_t k = dk[i];
  if (k == kSentinel) return;
  const uint32_t v = (uint32_t)(k >> L);
  if (i > 0 && (uint32_t)(dk[i - 1] >> L) == v) return;
  // the run's end: doubling steps, then a binary search (a hub's run can hold 10^4 entries; a
  // sentinel's source is 2^32 - 1)
  int64_t end = i + 1, step = 1;
  while (end + step <= nd_cap && (uint32_t)(dk[end + step - 1] >> L) == v) {
    end += step;
    step *= 2;
  }
  for (int64_t hi = min(nd_cap, end + step - 1); end < hi;) {
    const int64_t mid = (end + hi) >> 1;
    if ((uint32_t)(dk[mid] >> L) == v) end = mid + 1;
    else hi = mid;
  }
  const int32_t c = (int32_t)(end - i);
  const unsigned long long r = atomicAdd(&st->n_runs, 1ull);
  const int32_t need = used[v] + c;
  runs[r] = make_int2(need > kLongList ? -1 - (int32_t)i : (int32_t)i, c);
  if (need > cap[v]) atomicAdd(&st->demand, (unsigned long long)slack_capacity(need, max(slack_q10, 256)));
}

__global__ void k_dir_runs(const uint64_t* __restrict__ dk, const int64_t nd_cap, const int L,
                           const int32_t* __restrict__ used, const int32_t* __restrict__ cap, const int32_t slack_q10,
                           int2* __restrict__ runs, BatchStatus* __restrict__ st) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nd_cap; i += (int64_t)gridDim.x * blockDim.x)
    dir_run(dk, i, nd_cap, L, used, cap, slack_q10, runs, st);
}

// A small batch's directed keys sorted by one CTA (padded with sentinels to 2 * cap), and their runs.
__global__ void __launch_bounds__(kSortThreads) k_sort_runs(const uint64_t* __restrict__ dk, const int64_t cap, const int L,
                                                            uint64_t* __restrict__ sorted, const int32_t* __restrict__ used,
                                                            const int32_t* __restrict__ vcap, const int32_t slack_q10,
                                                            int2* __restrict__ runs, BatchStatus* __restrict__ st) {
  __shared__ uint64_t k[2 * kSmallBatch];
  const int64_t n = 2 * (int64_t)st->n_ins;
  const int P = pow2_at_least(n);
  for (int i = threadIdx.x; i < P; i += kSortThreads) k[i] = i < n ? dk[i] : kSentinel;
  __syncthreads();
  cta_sort(k, P);
  for (int i = threadIdx.x; i < 2 * cap; i += kSortThreads) sorted[i] = i < P ? k[i] : kSentinel;
  for (int i = threadIdx.x; i < n; i += kSortThreads)
    dir_run(k, i, n, L, used, vcap, slack_q10, runs, st);
}

// The long-list insertion's plan of one run (see k_long_stage).
struct LongPlan {
  int64_t s_old;   // list start before the batch
  int64_t s_new;   // list start after it (s_old unless relocated)
  int64_t soff;    // the run's range in the scratch buffer
  int32_t a;       // entries before the batch
  int32_t c;       // new entries
  int32_t first;   // first moving entry (0 when relocated)
  int32_t len;     // entries staged: a - first + c (0 = nothing to do)
  int32_t i0;      // the run's first entry in the sorted directed keys
  int32_t pad;
};
constexpr int kLongChunk = 4096;  // entries per work item of the long-list kernels

struct InsertArgs {
  const uint64_t* dk;        // sorted directed keys
  int L;
  const int2* runs;
  int64_t* start;
  int32_t* used;
  int32_t* cap;
  int32_t* pool;
  int64_t pool_cap;
  uint8_t* mark;             // new slots are marked when given
  int64_t* slot;             // absolute slots of the new entries
  unsigned long long* pool_top;
  int32_t slack_q10;
  LongPlan* plan;            // long runs: their plans and work items
  unsigned long long* items;
  int64_t item_cap;
  int64_t scr_cap;
};

// A long run's plan, by the warp: relocation (done by insert_runs) or the first moving entry, the
// list's new length, a range of the scratch buffer and work items of kLongChunk entries.
__device__ __forceinline__ void plan_long_run(const InsertArgs& I, const int32_t v, const int64_t i0, const int32_t a,
                                              const int32_t c, const int64_t s_old, const int64_t s_new,
                                              BatchStatus* __restrict__ st) {
  const int lane = threadIdx.x & 31;
  LongPlan P;
  P.s_old = s_old;
  P.s_new = s_new;
  P.a = a;
  P.c = c;
  P.i0 = (int32_t)i0;
  P.pad = 0;
  P.first = s_new == s_old ? warp_lower_bound(I.pool + s_old, a, dir_dst(I.dk[i0], I.L)) : 0;
  P.len = a - P.first + c;
  const int32_t nch = (P.len + kLongChunk - 1) / kLongChunk;
  unsigned long long so = 0, ib = 0, r = 0;
  if (lane == 0) {
    so = atomicAdd(&st->long_scr, (unsigned long long)P.len);
    ib = atomicAdd(&st->long_items, (unsigned long long)nch);
    r = atomicAdd(&st->n_long, 1ull);
  }
  so = __shfl_sync(kFull, so, 0);
  ib = __shfl_sync(kFull, ib, 0);
  r = __shfl_sync(kFull, r, 0);
  const bool ok = (int64_t)(so + P.len) <= I.scr_cap && (int64_t)(ib + nch) <= I.item_cap;
  for (int32_t j = lane; j < nch; j += 32)
    if ((int64_t)(ib + j) < I.item_cap) I.items[ib + j] = ok ? (r << 32) | (unsigned)j : kNoLongItem;
  if (!ok) {  // unreachable while the scratch follows the pool's size
    for (int32_t j = lane; j < c; j += 32) I.slot[i0 + j] = -1;
    P.len = 0;
  }
  P.soff = (int64_t)so;
  if (lane == 0) {
    if (ok) {
      I.used[v] = a + c;
      atomicAdd(&st->dir_added, (unsigned long long)c);
    } else {
      atomicOr(&st->err, kErrScratch);
    }
    I.plan[r] = P;
  }
  __syncwarp();
}

// One warp per affected source vertex: merge its sorted new neighbours into its list, in place
// (backwards) when the capacity allows, else into a fresh block at the pool top. New slots are
// marked (mark = 1) when `mark` is given; their absolute slots go to slot[]. A list that will be
// long is planned here and merged by k_long_stage / k_long_write.
__global__ void __launch_bounds__(kThreads) k_insert_runs(const InsertArgs I, BatchStatus* __restrict__ st) {
  const int lane = threadIdx.x & 31;
  const int64_t gw = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const int64_t nruns = (int64_t)st->n_runs;
  for (int64_t r = gw; r < nruns; r += nw) {
    const int2 run = I.runs[r];
    const bool is_long = run.x < 0;
    const int64_t i0 = is_long ? -1 - run.x : run.x;
    const int32_t c = run.y;
    const int64_t i1 = i0 + c;
    const int32_t v = dir_src(I.dk[i0], I.L);
    const int32_t a = I.used[v];
    const int64_t s_old = I.start[v];
    int64_t s_new = s_old;
    bool moved = false;
    if (a + c > I.cap[v]) {
      const int32_t nc = slack_capacity(a + c, max(I.slack_q10, 256));
      unsigned long long at = 0;
      if (lane == 0) at = atomicAdd(I.pool_top, (unsigned long long)nc);
      __syncwarp();
      at = __shfl_sync(kFull, at, 0);
      __syncwarp();
      if ((int64_t)at + nc > I.pool_cap) {
        if (lane == 0) atomicOr(&st->err, kErrPool);
        for (int64_t j = i0 + lane; j < i1; j += 32) I.slot[j] = -1;  // nothing to clear later
        continue;  // cannot happen when the host sized the pool from the demand pass
      }
      s_new = (int64_t)at;
      moved = true;
      if (lane == 0) {
        I.cap[v] = nc;
        I.start[v] = s_new;
        atomicAdd(&st->not_fitting, (unsigned long long)c);
      }
    }
    if (is_long) {
      plan_long_run(I, v, i0, a, c, s_old, s_new, st);
      continue;
    }
    const int32_t* A = I.pool + s_old;
    // New entries first, while A is intact: final position j + #(old < B[j]) (relative). The
    // first five levels of each search come from 32 evenly spaced samples of A held in the lanes.
    int32_t first_new = a;  // old entries below the smallest new entry keep their slots
    int32_t mine = INT32_MAX;  // this lane's new entry (runs of at most 32)
    {
      const int32_t step = (a + 31) / 32;
      const int32_t smp = lane * step < a ? A[lane * step] : INT32_MAX;
      const int32_t s31 = __shfl_sync(kFull, smp, 31);
      for (int64_t jb = i0; jb < i1; jb += 32) {
        const int64_t j = jb + lane;
        const bool act = j < i1;
        const int32_t val = act ? dir_dst(I.dk[j], I.L) : INT32_MAX;
        mine = val;
        int pos = 0;  // samples below val (they ascend with the lane)
#pragma unroll
        for (int h = 16; h > 0; h >>= 1)
          if (__shfl_sync(kFull, smp, pos + h - 1) < val) pos += h;
        if (pos == 31 && s31 < val) pos = 32;
        int32_t lo = pos > 0 ? (pos - 1) * step + 1 : 0;
        int32_t hi = pos < 32 ? min(pos * step, a) : a;
        if (act) {
          while (lo < hi) {
            const int32_t mid = (lo + hi) >> 1;
            if (A[mid] < val) lo = mid + 1;
            else hi = mid;
          }
          I.slot[j] = (j - i0) + lo;
          if (j == i0) first_new = lo;
        }
        __syncwarp();
      }
    }
    __syncwarp();
    // In place, old entries below the first new entry do not move; relocated, all of them do.
    const int32_t keep_below = moved ? 0 : __shfl_sync(kFull, first_new, 0);
    const int32_t m31 = __shfl_sync(kFull, mine, 31);
    // Old entries: final position i + #(new < A[i]); backwards in steps of 128 entries, each read whole
    // before its first write, so that, in place, no unread entry is overwritten (targets never
    // precede sources). The new entries below an old one are counted from the lanes: one by one for
    // runs of at most 8 (the usual case), by a search over the lanes up to 32; else by a search of
    // the keys.
    const int32_t low = (keep_below / 128) * 128;
    for (int32_t base = a > 0 ? ((a - 1) / 128) * 128 : -1; base >= low; base -= 128) {
      int32_t val[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int32_t i = base + 32 * q + lane;
        val[q] = i < a && i >= keep_below ? A[i] : -1;
      }
      __syncwarp();
      int32_t few[4] = {0, 0, 0, 0};
      if (c <= 8) {
        for (int j = 0; j < c; ++j) {
          const int32_t x = __shfl_sync(kFull, mine, j);
#pragma unroll
          for (int q = 0; q < 4; ++q) few[q] += x < val[q];
        }
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        int32_t below = few[q];
        if (c <= 8) {
        } else if (c <= 32) {
#pragma unroll
          for (int h = 16; h > 0; h >>= 1)
            if (__shfl_sync(kFull, mine, below + h - 1) < val[q]) below += h;
          if (below == 31 && m31 < val[q]) below = 32;
        } else if (val[q] >= 0) {
          int64_t lo = i0, hi = i1;
          while (lo < hi) {
            const int64_t mid = (lo + hi) >> 1;
            if (dir_dst(I.dk[mid], I.L) < val[q]) lo = mid + 1;
            else hi = mid;
          }
          below = (int32_t)(lo - i0);
        }
        if (val[q] >= 0) {
          const int64_t pos = s_new + base + 32 * q + lane + below;
          I.pool[pos] = val[q];
          if (I.mark) I.mark[pos] = 0;
        }
      }
      __syncwarp();
    }
    // New entries into the holes.
    for (int64_t j = i0 + lane; j < i1; j += 32) {
      const int64_t pos = s_new + I.slot[j];
      I.pool[pos] = dir_dst(I.dk[j], I.L);
      if (I.mark) I.mark[pos] = 1;
      I.slot[j] = pos;
    }
    __syncwarp();
    if (lane == 0) {
      I.used[v] = a + c;
      atomicAdd(&st->dir_added, (unsigned long long)c);
    }
  }
}

// ---- deletion -------------------------------------------------------------------------------

// Mark the slots of the batch's deletions and keep each list's smallest marked slot (the
// compaction leaves the entries below it in place); opens the compaction epoch.
__global__ void k_mark_deletions(const int4* __restrict__ dlist, const BatchStatus* __restrict__ st,
                                 const int64_t* __restrict__ start, uint8_t* __restrict__ mark,
                                 int32_t* __restrict__ first_del, unsigned* __restrict__ epoch) {
  const int64_t nd = (int64_t)st->n_del;
  if (blockIdx.x == 0 && threadIdx.x == 0) *epoch += 1u;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nd; i += (int64_t)gridDim.x * blockDim.x) {
    const int4 d = dlist[i];
    mark[start[d.x] + d.z] = 1;
    mark[start[d.y] + d.w] = 1;
    atomicMin(&first_del[d.x], d.z);
    atomicMin(&first_del[d.y], d.w);
  }
}

// The long-list compaction's plan of one list (see k_cmp_stage).
struct CmpPlan {
  int64_t s;       // list start
  int64_t soff;    // the list's range in the scratch buffer (chunks j0 on)
  int64_t ib;      // its first work item
  int32_t v;
  int32_t a;       // entries before the deletions
  int32_t nch;     // work items: chunks j0 .. j0 + nch - 1
  int32_t j0;      // the chunk of the first marked slot; the chunks below it stay in place
  int32_t done;    // chunks staged so far
  int32_t pad;
};

struct CompactArgs {
  const int64_t* start;
  int32_t* used;
  int32_t* pool;
  uint8_t* mark;
  unsigned* claim;
  const unsigned* epoch;
  int32_t* first_del;
  CmpPlan* plan;             // long lists: their plans and work items
  unsigned long long* items;
  int64_t item_cap;
  int64_t scr_cap;
};

// Remove the marked slots from the list of v (each vertex once: the first warp to claim it with this
// epoch) and clear its marks, by the warp. The entries below the list's first marked slot
// (first_del, reset here to kNoDel) stay where they are; the rest move down in steps of 128
// entries, each read whole before its first write. A long list is only planned (k_cmp_stage).
__device__ __forceinline__ void compact_vertex(const CompactArgs& C, const int32_t v, BatchStatus* __restrict__ st) {
  const int lane = threadIdx.x & 31;
  const unsigned epoch = *C.epoch;
  const int32_t a = C.used[v];
  unsigned old = 0;
  if (lane == 0) old = atomicMax(&C.claim[v], epoch);
  __syncwarp();
  old = __shfl_sync(kFull, old, 0);
  if (old >= epoch) return;
  const int64_t s = C.start[v];
  const int32_t f = min(C.first_del[v], a);
  __syncwarp();
  if (lane == 0) C.first_del[v] = kNoDel;
  if (a > kLongList) {
    CmpPlan P;
    P.s = s;
    P.v = v;
    P.a = a;
    P.j0 = f / kLongChunk;
    P.nch = f < a ? (a + kLongChunk - 1) / kLongChunk - P.j0 : 0;
    P.done = 0;
    P.pad = 0;
    const int32_t span = a - P.j0 * kLongChunk;  // entries from chunk j0 on
    unsigned long long so = 0, ib = 0, r = 0;
    if (lane == 0) {
      so = atomicAdd(&st->cmp_scr, (unsigned long long)span);
      ib = atomicAdd(&st->cmp_items, (unsigned long long)P.nch);
      r = atomicAdd(&st->n_cmp, 1ull);
    }
    so = __shfl_sync(kFull, so, 0);
    ib = __shfl_sync(kFull, ib, 0);
    r = __shfl_sync(kFull, r, 0);
    const bool ok = (int64_t)(so + span) <= C.scr_cap && (int64_t)(ib + P.nch) <= C.item_cap;
    for (int32_t j = lane; j < P.nch; j += 32)
      if ((int64_t)(ib + j) < C.item_cap) C.items[ib + j] = ok ? (r << 32) | (unsigned)(P.j0 + j) : kNoLongItem;
    if (lane == 0) {
      if (!ok) {  // unreachable while the scratch follows the pool's size
        atomicOr(&st->err, kErrScratch);
        P.nch = 0;
      }
      P.soff = (int64_t)so;
      P.ib = (int64_t)ib;
      C.plan[r] = P;
    }
    __syncwarp();
    return;
  }
  const unsigned lt = (1u << lane) - 1u;
  int32_t wp = f;
  for (int32_t base = f; base < a; base += 128) {
    int32_t val[4];
    bool keep[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int32_t i = base + 32 * q + lane;
      val[q] = i < a ? C.pool[s + i] : 0;
      keep[q] = i < a && C.mark[s + i] == 0;
    }
    __syncwarp();
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int32_t i = base + 32 * q + lane;
      const unsigned m = __ballot_sync(kFull, keep[q]);
      if (keep[q]) C.pool[s + wp + __popc(m & lt)] = val[q];
      else if (i < a) C.mark[s + i] = 0;
      wp += __popc(m);
    }
    __syncwarp();
  }
  if (lane == 0) {
    C.used[v] = wp;
    atomicAdd(&st->dir_removed, (unsigned long long)(a - wp));
  }
  __syncwarp();
}

// The lists of the vertices vlist[0 .. *nv) (the cuStinger-style deletion).
__global__ void __launch_bounds__(kThreads) k_compact(const CompactArgs C, const int32_t* __restrict__ vlist,
                                                      const unsigned long long* __restrict__ nv,
                                                      BatchStatus* __restrict__ st) {
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t k = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; k < (int64_t)*nv; k += nw)
    compact_vertex(C, vlist[k], st);
}

// Insertion into long lists (more than kLongList entries after the batch), over all of the batch's
// long runs at once, from the plans of k_insert_runs:
//   k_long_stage  one CTA per item: each moving old entry and each new entry computes its place
//                 in the merged suffix (an old entry shifts by the number of new entries below it,
//                 a new entry lands after the old entries below it) and writes there in scratch;
//   k_long_write  one CTA per item: the merged suffix back into the list, with the new entries'
//                 marks.
// The launch boundary between staging and writing takes the place of an in-place merge's block
// barriers: every source is read before any target is written, so a hub list of 10^5 entries is
// spread over many CTAs instead of being one CTA's chain of steps.
__global__ void __launch_bounds__(kThreads) k_long_stage(
    const uint64_t* __restrict__ dk, const int L, const int32_t* __restrict__ pool,
    const LongPlan* __restrict__ plan, const unsigned long long* __restrict__ items, const int64_t item_cap,
    int32_t* __restrict__ scr, uint8_t* __restrict__ smark, int64_t* __restrict__ slot, const BatchStatus* __restrict__ st) {
  // The new entries whose values fall inside the item's old entries, staged in shared memory,
  // so that each old entry counts the new ones below it there instead of in global memory.
  __shared__ int32_t s_run[kLongChunk];
  __shared__ int32_t s_lo, s_n;
  const int64_t n_items = min((int64_t)st->long_items, item_cap);
  for (int64_t q = blockIdx.x; q < n_items; q += gridDim.x) {
    const unsigned long long item = items[q];
    if (item == kNoLongItem) continue;
    const LongPlan P = plan[item >> 32];
    const int32_t k0 = (int32_t)(uint32_t)item * kLongChunk, k1 = min(P.len, k0 + kLongChunk);
    const int32_t suffix = P.a - P.first;
    const int32_t ko1 = min(k1, suffix);  // the item's old entries: [k0, ko1)
    int32_t run_lo = 0, run_n = -1;       // run_n < 0: not staged
    if (k0 < ko1) {
      if (threadIdx.x == 0) {
        // new entries below the item's first old value, and below its last: the ones between
        // are the only ones that tell its old entries apart
        const int32_t v0 = pool[P.s_old + P.first + k0], v1 = pool[P.s_old + P.first + ko1 - 1];
        int32_t lo = 0, hi = P.c;
        while (lo < hi) {
          const int32_t mid = (lo + hi) >> 1;
          if (dir_dst(dk[P.i0 + mid], L) < v0) lo = mid + 1;
          else hi = mid;
        }
        int32_t lo2 = lo, hi2 = P.c;
        while (lo2 < hi2) {
          const int32_t mid = (lo2 + hi2) >> 1;
          if (dir_dst(dk[P.i0 + mid], L) < v1) lo2 = mid + 1;
          else hi2 = mid;
        }
        s_lo = lo;
        s_n = lo2 - lo;
      }
      __syncthreads();
      run_lo = s_lo;
      run_n = s_n <= kLongChunk ? s_n : -1;
      for (int32_t t = threadIdx.x; t < run_n; t += kThreads) s_run[t] = dir_dst(dk[P.i0 + run_lo + t], L);
      __syncthreads();
    }
    for (int32_t k = k0 + (int32_t)threadIdx.x; k < k1; k += kThreads) {
      int32_t val, pos;
      uint8_t mk;
      if (k < suffix) {  // an old entry: shifts by the new entries below it
        val = pool[P.s_old + P.first + k];
        int32_t lo, hi;
        if (run_n >= 0) {
          lo = 0;
          hi = run_n;
          while (lo < hi) {
            const int32_t mid = (lo + hi) >> 1;
            if (s_run[mid] < val) lo = mid + 1;
            else hi = mid;
          }
          lo += run_lo;
        } else {
          lo = 0;
          hi = P.c;
          while (lo < hi) {
            const int32_t mid = (lo + hi) >> 1;
            if (dir_dst(dk[P.i0 + mid], L) < val) lo = mid + 1;
            else hi = mid;
          }
        }
        pos = k + lo;
        mk = 0;
      } else {  // a new entry: lands after the old entries below it
        const int32_t j = k - suffix;
        val = dir_dst(dk[P.i0 + j], L);
        pos = j + (int32_t)(lower_bound(pool, P.s_old, P.s_old + P.a, val) - P.s_old) - P.first;
        slot[P.i0 + j] = P.s_new + P.first + pos;
        mk = 1;
      }
      scr[P.soff + pos] = val;
      smark[P.soff + pos] = mk;
    }
    __syncthreads();  // the next item restages s_run
  }
}

__global__ void __launch_bounds__(kThreads) k_long_write(
    const LongPlan* __restrict__ plan, const unsigned long long* __restrict__ items, const int64_t item_cap,
    const int32_t* __restrict__ scr, const uint8_t* __restrict__ smark, int32_t* __restrict__ pool,
    uint8_t* __restrict__ mark, const BatchStatus* __restrict__ st) {
  const int64_t n_items = min((int64_t)st->long_items, item_cap);
  for (int64_t q = blockIdx.x; q < n_items; q += gridDim.x) {
    const unsigned long long item = items[q];
    if (item == kNoLongItem) continue;
    const LongPlan P = plan[item >> 32];
    const int32_t k0 = (int32_t)(uint32_t)item * kLongChunk, k1 = min(P.len, k0 + kLongChunk);
#pragma unroll 4
    for (int32_t k = k0 + (int32_t)threadIdx.x; k < k1; k += kThreads) {
      const int64_t dest = P.s_new + P.first + k;
      pool[dest] = scr[P.soff + k];
      if (mark) mark[dest] = smark[P.soff + k];
    }
  }
}

// Deletions from long lists (more than kLongList entries), over all of the batch's long lists at
// once, from the plans of compact_vertex and through the insertion's scratch buffer:
//   k_cmp_stage   one CTA per item: the chunk's kept entries, compacted within the chunk, into
//                 scratch, and their count; the chunk's marks cleared. The CTA that stages a list's
//                 last chunk turns the counts into output offsets and sets the new length;
//   k_cmp_write   one CTA per item: the chunk's kept entries from scratch to their place.
// The scratch keeps sources and targets apart, so chunks of one list proceed on many CTAs.

// Each thread holds kCmpPer consecutive entries of the chunk (256 threads x 16 = kLongChunk).
constexpr int kCmpPer = kLongChunk / kThreads;
static_assert(kCmpPer % 4 == 0, "a thread's run of entries is whole 16-byte units");

__global__ void __launch_bounds__(kThreads) k_cmp_stage(
    CmpPlan* __restrict__ plan, const unsigned long long* __restrict__ items, const int64_t item_cap,
    const int32_t* __restrict__ pool, uint8_t* __restrict__ mark, int32_t* __restrict__ scr,
    int2* __restrict__ chunk, int32_t* __restrict__ used, BatchStatus* __restrict__ st) {
  __shared__ int32_t sh_wsum[kThreads / 32];
  __shared__ int32_t sh_kept[kLongChunk];  // the chunk's kept entries, for coalesced writes
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int64_t n_items = min((int64_t)st->cmp_items, item_cap);
  for (int64_t q = blockIdx.x; q < n_items; q += gridDim.x) {
    const unsigned long long item = items[q];
    if (item == kNoLongItem) continue;
    const CmpPlan P = plan[item >> 32];
    const int32_t j = (int32_t)(uint32_t)item;
    const int32_t c0 = j * kLongChunk;
    const int32_t r0 = (j - P.j0) * kLongChunk;  // the chunk's place in the list's scratch range
    const int32_t i0 = c0 + (int32_t)threadIdx.x * kCmpPer;
    int32_t val[kCmpPer];
    unsigned keepm = 0;
    int32_t kept = 0;
    if (i0 + kCmpPer <= P.a) {
      // a full run of kCmpPer entries: 16-byte loads of the entries (list starts are multiples of
      // 4 entries and i0 of kCmpPer) and 4-byte loads of their marks, all independent
      const int4* e4 = reinterpret_cast<const int4*>(pool + P.s + i0);
      uint32_t* m4 = reinterpret_cast<uint32_t*>(mark + P.s + i0);
#pragma unroll
      for (int u = 0; u < kCmpPer / 4; ++u) {
        const int4 v = e4[u];
        const uint32_t m = m4[u];
        val[4 * u] = v.x;
        val[4 * u + 1] = v.y;
        val[4 * u + 2] = v.z;
        val[4 * u + 3] = v.w;
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          const bool keep = ((m >> (8 * b)) & 0xffu) == 0;
          keepm |= (unsigned)keep << (4 * u + b);
          kept += keep;
        }
        if (m) m4[u] = 0u;  // the deleted slots' marks are cleared (kept slots' are zero)
      }
    } else {
#pragma unroll
      for (int t = 0; t < kCmpPer; ++t) {
        const int32_t i = i0 + t;
        bool keep = false;
        val[t] = 0;
        if (i < P.a) {
          keep = mark[P.s + i] == 0;
          if (keep) val[t] = pool[P.s + i];
          else mark[P.s + i] = 0;
        }
        keepm |= (unsigned)keep << t;
        kept += keep;
      }
    }
    int32_t incl = kept;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int32_t y = __shfl_up_sync(kFull, incl, o);
      if (lane >= o) incl += y;
    }
    if (lane == 31) sh_wsum[wid] = incl;
    __syncthreads();
    int32_t before = 0, total = 0;
    for (int w = 0; w < kThreads / 32; ++w) {
      const int32_t x = sh_wsum[w];
      if (w < wid) before += x;
      total += x;
    }
    int32_t at = before + incl - kept;
#pragma unroll
    for (int t = 0; t < kCmpPer; ++t)
      if (keepm >> t & 1u) sh_kept[at++] = val[t];
    __syncthreads();
    for (int32_t t = threadIdx.x; t < total; t += kThreads) scr[P.soff + r0 + t] = sh_kept[t];
    if (threadIdx.x == 0) {
      __stcg(&chunk[P.ib + (j - P.j0)], make_int2(0, total));
      __threadfence();
      if (atomicAdd(&plan[item >> 32].done, 1) == P.nch - 1) {
        __threadfence();
        int32_t off = P.j0 * kLongChunk;  // the chunks below j0 keep their entries in place
        for (int32_t x = 0; x < P.nch; ++x) {
          const int32_t c = __ldcg(&chunk[P.ib + x]).y;
          __stcg(&chunk[P.ib + x], make_int2(off, c));
          off += c;
        }
        used[P.v] = off;
        atomicAdd(&st->dir_removed, (unsigned long long)(P.a - off));
      }
    }
    __syncthreads();
  }
}

__global__ void __launch_bounds__(kThreads) k_cmp_write(
    const CmpPlan* __restrict__ plan, const unsigned long long* __restrict__ items, const int64_t item_cap,
    const int32_t* __restrict__ scr, const int2* __restrict__ chunk, int32_t* __restrict__ pool,
    const BatchStatus* __restrict__ st) {
  const int64_t n_items = min((int64_t)st->cmp_items, item_cap);
  for (int64_t q = blockIdx.x; q < n_items; q += gridDim.x) {
    const unsigned long long item = items[q];
    if (item == kNoLongItem) continue;
    const CmpPlan P = plan[item >> 32];
    const int32_t j = (int32_t)(uint32_t)item - P.j0;
    const int2 oc = chunk[P.ib + j];
#pragma unroll 4
    for (int32_t t = threadIdx.x; t < oc.y; t += kThreads) pool[P.s + oc.x + t] = scr[P.soff + j * kLongChunk + t];
  }
}

// ---- the triangle delta of changed edges -----------------------------------------------------

enum { kPredMark = 0, kPredBatch = 1 };

struct BatchLists {
  const int32_t* src;    // sorted directed entries (cuStinger path)
  const int32_t* dst;
  const int32_t* off;    // batch CSR over src, int32[nv+1]
  const int32_t* dup;
};

// A changed edge as the per-edge kernel takes it: its lists, the shorter one first. kSplitFlag in la:
// its intersection is queued as split items.
constexpr int32_t kSplitFlag = INT32_MIN;
struct __align__(16) DeltaDesc {
  int32_t oa, ob, la, lb;  // owners and lengths
  int64_t sa, sb;          // starts
};

struct DeltaArgs {
  SlackView g;
  const uint8_t* mark;
  // entries: either int2/int4 canonical lists (mark predicate) or the batch arrays
  const int2* ilist;
  const int4* dlist;
  const unsigned long long* count_dev;  // number of entries (device), or NULL with count_host
  int64_t count_host;
  BatchLists bl;
  int sign;          // +1 insertions, -1 deletions
  uint32_t weight;   // per-vertex increment per counted triangle
  int search_ratio_x16;
  int only_present;  // skip entries whose edge is absent (cuStinger deletion count)
  int use_table;     // per-cell strategy table: 0 = search, 1 = merge
  int cell_filter;   // -1 all, -2 none, c >= 0 only edges of cell c (timing mode)
  // split queue: (edge << 24 | chunk) items of long intersections
  unsigned long long* split_items;
  unsigned long long* split_cnt;  // zero before the items are queued
  int split_min;     // intersections whose shorter list is longer than this are split ...
  int chunk;         // ... into items of this many entries of the shorter list
  int shard;         // this rank counts the entries e with e % nshards == shard
  int nshards;
  unsigned long long* bytes_out;  // algorithmic bytes of the intersections run (NULL = not kept)
  // persistent kernel (k_delta_fused): its CTAs meet once, between the count and the update that
  // needs the count done. arrived counts them (zero at launch; kMeetLeft). A wait that runs out
  // reports kErrTimeout in err; bar_extra is added to the CTAs waited for (0; a test sets 1 to make the
  // wait run out); spin_ns bounds the wait.
  unsigned* arrived;
  unsigned* err;
  unsigned bar_extra;
  unsigned long long spin_ns;
  // hub-centred counting (k_delta_hub): changed edges whose longer endpoint holds at least
  // hub_min of the phase's changed edges are counted at that endpoint (0 = never)
  int hub_min;
  // the changed edges not counted at a hub (k_hub_place) and their number
  const DeltaDesc* desc;
  const unsigned long long* n_desc;
  // dynamic work queues of k_delta_fused's two passes (zero at launch)
  unsigned long long* e_next;
  unsigned long long* i_next;
  int stage_ok;      // the launch has kStageSmem of dynamic shared memory: staged cells may stage
  uint8_t table[256];
};

__device__ __forceinline__ int cell_of(int a, int b) {
  const int ca = min(31 - __clz(max(a, 1)), 15), cb = min(31 - __clz(max(b, 1)), 15);
  return ca * 16 + cb;
}

// Does the batch hold the non-duplicate entry (x, y)?
__device__ __forceinline__ bool batch_has(const BatchLists& bl, const int32_t x, const int32_t y) {
  const int32_t hi = bl.off[x + 1];
  int32_t l = bl.off[x], h = hi;
  while (l < h) {
    const int32_t mid = (l + h) >> 1;
    if (bl.dst[mid] < y) l = mid + 1;
    else h = mid;
  }
  return l < hi && bl.dst[l] == y && bl.dup[l] == 0;
}

template <int PRED>
__device__ __forceinline__ bool changed(const DeltaArgs& A, int32_t owner, int64_t slot_abs, int32_t w) {
  if (PRED == kPredMark) return A.mark[slot_abs] != 0;
  return batch_has(A.bl, owner, w);
}

// Entry e of the changed-edge list: its endpoints and whether it adds to the total (the
// cuStinger-style batch holds both directions of every edge; the total counts one).
template <int PRED>
__device__ __forceinline__ bool delta_entry(const DeltaArgs& A, int64_t e, int32_t& x, int32_t& y, bool& count_total) {
  count_total = true;
  if (PRED == kPredMark) {
    if (A.dlist) {
      const int4 d = A.dlist[e];
      x = d.x;
      y = d.y;
    } else {
      const int2 d = A.ilist[e];
      x = d.x;
      y = d.y;
    }
    return true;
  }
  if (A.bl.dup[e]) return false;
  x = A.bl.src[e];
  y = A.bl.dst[e];
  count_total = x < y;
  return x != y;
}

// Intersection strategies of the delta count (the streaming strategy table's values).
enum : int { kStratSearch = 0, kStratMerge = 1, kStratStage = 2 };
constexpr int kStageEntries = 1024;  // entries of the longer list a warp stages per piece
// Dynamic shared memory of a delta kernel launch that may stage (one buffer per warp); a launch
// without it searches the staged cells (with marks) or merges them.
constexpr size_t kStageSmem = sizeof(int32_t) * kStageEntries * (kThreads / 32);

// The two lists of edge {x, y} as the intersection takes them: A the shorter, B the longer.
struct DeltaPair {
  int32_t oa, ob, la, lb;
  int64_t sa, sb;
  uint64_t key;
  int strat;
  int cell;
};

// How the pair's lists are intersected. With marks (PRED = kPredMark) every cell that does not stage
// searches: a merge's lanes each walk a chain of dependent loads, and searching was never slower
// (whole streaming passes, ratio rule -> search everywhere: 3-1000 updates on R-MAT 22
// 14.1 -> 6.7 ms, 20,011 on BA n = 2^20 3.8 -> 2.0 ms, 10^6 on R-MAT 22 16.3 -> 14.4 ms).
template <int PRED>
__device__ __forceinline__ int pair_strategy(const DeltaArgs& A, const DeltaPair& P) {
  const int t = A.use_table ? A.table[P.cell] : -1;
  if (t == kStratStage && A.stage_ok) return kStratStage;
  if (PRED == kPredMark || t == kStratSearch) return kStratSearch;
  if (t >= 0) return kStratMerge;
  const int lg = 32 - __clz(P.lb);
  return 16LL * P.lb > (long long)A.search_ratio_x16 * P.la * lg ? kStratSearch : kStratMerge;
}

template <int PRED>
__device__ __forceinline__ DeltaPair delta_pair(const DeltaArgs& A, int32_t x, int32_t y, int32_t lx, int32_t ly,
                                                int64_t sx, int64_t sy) {
  DeltaPair P;
  const bool xs = lx <= ly;
  P.oa = xs ? x : y;
  P.ob = xs ? y : x;
  P.sa = xs ? sx : sy;
  P.sb = xs ? sy : sx;
  P.la = xs ? lx : ly;
  P.lb = xs ? ly : lx;
  P.key = ekey(x, y);
  P.cell = cell_of(P.la, P.lb);
  P.strat = pair_strategy<PRED>(A, P);
  return P;
}

// The warp intersects entries [i_begin, i_end) of the shorter list with the longer one and
// returns (in every lane) the triangles kept there; each kept common neighbour w gets its
// per-vertex update here, the endpoints get theirs from the caller. With marks the lists are read by
// plain loads: the launch rewrites them later (k_delta_fused), and the read-only path is only for what
// no thread writes during the launch.
template <int PRED>
__device__ __forceinline__ uint32_t delta_range(const DeltaArgs& A, const DeltaPair& P, int32_t i_begin,
                                                int32_t i_end, const uint32_t inc, uint32_t* __restrict__ pv) {
  const int lane = threadIdx.x & 31;
  const int32_t* L = A.g.ind;
  uint32_t c = 0;
  auto match = [&](const bool ca, int64_t ib, int32_t w) {
    const bool cb = changed<PRED>(A, P.ob, P.sb + ib, w);
    const bool keep = (!ca || P.key < ekey(P.oa, w)) && (!cb || P.key < ekey(P.ob, w));
    if (keep) {
      ++c;
      atomicAdd(&pv[w], inc);
    }
  };
  auto on_match = [&](int64_t ia, int64_t ib, int32_t w) { match(changed<PRED>(A, P.oa, P.sa + ia, w), ib, w); };
  const int64_t sb = P.sb, eb = P.sb + P.lb;
  if (P.strat == kStratStage) {
    // The part of the longer list that can meet entries [i_begin, i_end) of the shorter one,
    // [lo, hi), is staged into this warp's shared-memory buffer in pieces of kStageEntries
    // (cp.async: every copy of a piece in flight at once); each lane then binary-searches one
    // shorter-list entry in the piece. A piece takes the shorter-list entries up to its last
    // entry (the last piece takes the rest), so each is searched once.
    extern __shared__ __align__(16) int32_t s_stage[];  // kStageSmem bytes (A.stage_ok)
    int32_t* buf = s_stage + (threadIdx.x >> 5) * kStageEntries;
    const int32_t a_first = L[P.sa + i_begin], a_last = L[P.sa + i_end - 1];
    const int32_t lo = warp_lower_bound(L + sb, P.lb, a_first);
    const int32_t hi = warp_lower_bound(L + sb, P.lb, a_last + 1);
    int32_t ia = i_begin;
    for (int32_t cb = lo; cb < hi && ia < i_end; cb += kStageEntries) {
      const int32_t n = min(hi - cb, kStageEntries);
      __syncwarp();  // the previous piece's searches are done with the buffer
      for (int32_t k = lane; k < n; k += 32) cp_async4(buf + k, L + sb + cb + k);
      cp_async_wait_all();
      __syncwarp();
      const int32_t bmax = buf[n - 1];
      const bool last = cb + n >= hi;
      while (ia < i_end) {
        const int32_t i = ia + lane;
        const int32_t w = i < i_end ? L[P.sa + i] : INT32_MAX;
        // the lanes that take part are a prefix (the shorter list ascends with the lane)
        const bool in = i < i_end && (last || w <= bmax);
        const int k = __popc(__ballot_sync(kFull, in));
        if (in) {
          int32_t l = 0, h = n;
          while (l < h) {
            const int32_t mid = (l + h) >> 1;
            if (buf[mid] < w) l = mid + 1;
            else h = mid;
          }
          if (l < n && buf[l] == w) on_match(i, (int64_t)cb + l, w);
        }
        __syncwarp();
        ia += k;
        if (k < 32) break;
      }
    }
  } else if (P.strat == kStratSearch) {
    // The first seven search levels come from 128 evenly spaced samples of the longer list, four
    // per lane in ascending order (one round of loads): a lane counts the samples below its key
    // with shuffles, then searches memory only inside that bucket, two entries at once (two
    // independent chains of loads in flight). Bound by the rounds of those chains and, in the
    // fused kernel, by registers: with 32 samples, 64-bit positions and 6 CTAs an SM (40
    // registers, 140 bytes spilled) 10^6 updates on R-MAT 22 took 9.89 ms a pass, with 32-bit positions
    // 9.57, with 128 samples as well 9.45 (256: 9.74), and 1000 updates 1.56, 1.54, 1.50 (5 CTAs: 1.47;
    // one call's figures: the same pass takes 1.5 to 1.6 ms from call to call).
    constexpr int kS = 4;  // samples per lane
    const int32_t* const B = L + sb;
    const int32_t step = (int32_t)(((unsigned)P.lb + 32 * kS - 1) / (32 * kS));
    int32_t smp[kS];
#pragma unroll
    for (int r = 0; r < kS; ++r) {
      const unsigned at = (unsigned)(lane * kS + r) * (unsigned)step;
      smp[r] = at < (unsigned)P.lb ? B[at] : INT32_MAX;
    }
    const int32_t s31 = __shfl_sync(kFull, smp[0], 31);
    // [lo, hi): the part of the longer list between the samples around w
    auto bucket = [&](const int32_t w, const bool in, int32_t& lo, int32_t& hi) {
      int pos = 0;  // lanes whose first sample is below w (they ascend with the lane)
#pragma unroll
      for (int st = 16; st > 0; st >>= 1)
        if (__shfl_sync(kFull, smp[0], pos + st - 1) < w) pos += st;
      if (pos == 31 && s31 < w) pos = 32;
      int cnt = (pos - 1) * kS + 1;  // samples below w (below 1: none)
#pragma unroll
      for (int r = 1; r < kS; ++r) cnt += __shfl_sync(kFull, smp[r], pos - 1) < w;
      if (pos == 0) cnt = 0;
      hi = (int32_t)min((unsigned)cnt * (unsigned)step, (unsigned)P.lb);
      lo = cnt > 0 ? min((cnt - 1) * step + 1, hi) : 0;
      if (!in) lo = hi;
    };
    const int32_t* const Q = L + P.sa;
    const uint8_t* const MQ = A.mark + P.sa;
    for (int32_t i = i_begin + lane; i < i_end + lane; i += 64) {
      const bool in = i < i_end, in2 = i + 32 < i_end;
      const int32_t w = in ? Q[i] : INT32_MAX;
      const int32_t w2 = in2 ? Q[i + 32] : INT32_MAX;
      // the shorter list's marks are read beside its entries, not after a match
      const bool ca = PRED == kPredMark && in && MQ[i] != 0;
      const bool ca2 = PRED == kPredMark && in2 && MQ[i + 32] != 0;
      int32_t lo, hi, lo2, hi2;
      bucket(w, in, lo, hi);
      bucket(w2, in2, lo2, hi2);
      while (lo < hi || lo2 < hi2) {  // two lower bounds, one step of each per round
        if (lo < hi) {
          const int32_t mid = (int32_t)(((unsigned)lo + (unsigned)hi) >> 1);
          if (B[mid] < w) lo = mid + 1;
          else hi = mid;
        }
        if (lo2 < hi2) {
          const int32_t mid = (int32_t)(((unsigned)lo2 + (unsigned)hi2) >> 1);
          if (B[mid] < w2) lo2 = mid + 1;
          else hi2 = mid;
        }
      }
      const bool m = in && lo < P.lb && B[lo] == w, m2 = in2 && lo2 < P.lb && B[lo2] == w2;
      if (PRED == kPredMark) {
        if (m) match(ca, lo, w);
        if (m2) match(ca2, lo2, w2);
      } else {
        if (m) on_match(i, lo, w);
        if (m2) on_match(i + 32, lo2, w2);
      }
    }
  } else if (PRED == kPredBatch) {
    const int32_t len = i_end - i_begin;
    const int32_t per = (len + 31) / 32;
    const int32_t i0 = i_begin + min(len, lane * per), i1 = min(i_end, i0 + per);
    if (i0 < i1) {
      int64_t p = lower_bound(L, sb, eb, L[P.sa + i0]);
      for (int32_t i = i0; i < i1 && p < eb; ++i) {
        const int32_t w = L[P.sa + i];
        while (p < eb && L[p] < w) ++p;
        if (p < eb && L[p] == w) on_match(i, p - sb, w);
      }
    }
  }
  __syncwarp();
  return warp_sum(c);
}

// Per-CTA flush of the kept-triangle total and the algorithmic bytes: one atomic each per CTA.
__device__ __forceinline__ void delta_flush(unsigned long long tri_acc, unsigned long long bytes_acc,
                                            unsigned long long* __restrict__ tri_out,
                                            unsigned long long* __restrict__ bytes_out) {
  __shared__ unsigned long long s_tri[kThreads / 32], s_bytes[kThreads / 32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) {
    s_tri[wid] = tri_acc;
    s_bytes[wid] = bytes_acc;
  }
  __syncwarp();
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long t = 0, b = 0;
    for (int w = 0; w < kThreads / 32; ++w) {
      t += s_tri[w];
      b += s_bytes[w];
    }
    if (t) atomicAdd(tri_out, t);
    if (b && bytes_out) atomicAdd(bytes_out, b);
  }
}

// Rank that counts the changed edge {x, y} of a sharded count: a hash of the edge's canonical
// key, so every rank assigns each edge alike whatever the order of its own lists.
__device__ __forceinline__ int edge_shard(int32_t x, int32_t y, int nshards) {
  uint64_t z = ekey(x, y) + 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return (int)((z ^ (z >> 31)) % (uint64_t)nshards);
}

// Flags of its split items: the edge counts for both directions; its triangles enter the total.
constexpr unsigned long long kItemTwice = 1ull << 62, kItemTotal = 1ull << 61;

// The cuStinger-style count (tc_count_batch): the triangle delta of the batch's edges, one warp per
// edge (warp-strided; with shards, only this rank's edges). Both directions of an edge keep the same
// triangles, so where the batch holds both (as a symmetric batch does) the one from the smaller
// id counts for both: its increments are doubled and the other one is skipped. An edge whose shorter list is longer
// than A.split_min (two hubs) would be one warp's serial tail of the whole launch: it is queued
// instead as items of A.chunk entries of its shorter list, which the second launch spreads over
// all warps (a full queue leaves the edge to this warp). Lane 0 of each warp accumulates the kept
// triangles and the edge's algorithmic bytes.
__device__ __forceinline__ void batch_entries(const DeltaArgs& A, uint32_t* __restrict__ pv, const int64_t gw,
                                              const int64_t nw, unsigned long long& tri_acc,
                                              unsigned long long& bytes_acc) {
  const int lane = threadIdx.x & 31;
  for (int64_t e = gw; e < A.count_host; e += nw) {
    int32_t x, y;
    bool count_total;
    if (!delta_entry<kPredBatch>(A, e, x, y, count_total)) continue;
    const bool both = batch_has(A.bl, y, x);
    if (both && x > y) continue;  // counted from (y, x)
    uint32_t times = both ? 2 : 1;
    if (A.nshards > 1 && edge_shard(x, y, A.nshards) != A.shard) continue;
    const int32_t lx = A.g.len(x), ly = A.g.len(y);
    if (lx < 2 || ly < 2) continue;
    const int64_t sx = A.g.start(x), sy = A.g.start(y);
    if (A.only_present) {
      // the edge must exist for its triangles to be destroyed: each direction is looked up in its list
      bool pres = false;
      if (lane == 0 || (lane == 1 && both)) {
        const int64_t p = lane == 0 ? lower_bound(A.g.ind, sx, sx + lx, y) : lower_bound(A.g.ind, sy, sy + ly, x);
        pres = lane == 0 ? p < sx + lx && A.g.ind[p] == y : p < sy + ly && A.g.ind[p] == x;
      }
      __syncwarp();
      const unsigned m = __ballot_sync(kFull, pres);
      if (m == 0) continue;
      times = __popc(m);
      count_total = count_total && (m & 1u);
    }
    const uint32_t inc = A.weight * (uint32_t)A.sign * times;
    const DeltaPair P = delta_pair<kPredBatch>(A, x, y, lx, ly, sx, sy);
    if (A.cell_filter == -2 || (A.cell_filter >= 0 && P.cell != A.cell_filter)) continue;
    if (lane == 0 && count_total) bytes_acc += 4ull * (unsigned long long)(lx + ly) + 8ull;
    if (P.la > A.split_min) {
      const int nch = (P.la + A.chunk - 1) / A.chunk;
      unsigned long long at = 0;
      if (lane == 0) at = atomicAdd(A.split_cnt, (unsigned long long)nch);
      at = __shfl_sync(kFull, at, 0);
      const bool fits = at + (unsigned long long)nch <= (unsigned long long)kDeltaItems;
      for (int j = lane; j < nch; j += 32)
        if (at + j < (unsigned long long)kDeltaItems)
          A.split_items[at + j] = fits ? ((unsigned long long)e << 24) | (unsigned long long)j |
                                             (times == 2 ? kItemTwice : 0) | (count_total ? kItemTotal : 0)
                                       : kNoItem;
      if (fits) continue;
    }
    const uint32_t c = delta_range<kPredBatch>(A, P, 0, P.la, inc, pv);
    if (lane == 0 && c) {
      atomicAdd(&pv[x], c * inc);
      atomicAdd(&pv[y], c * inc);
      if (count_total) tri_acc += c;
    }
  }
}

// Its queued chunks, one warp per item (the second launch). An item's edge passed every check of
// the first; its endpoints' per-vertex updates and the total add up per chunk.
__device__ __forceinline__ void batch_items(const DeltaArgs& A, uint32_t* __restrict__ pv, const int64_t gw,
                                            const int64_t nw, unsigned long long& tri_acc) {
  const int lane = threadIdx.x & 31;
  const int64_t n_items = (int64_t)min(*A.split_cnt, (unsigned long long)kDeltaItems);
  for (int64_t q = gw; q < n_items; q += nw) {
    const unsigned long long item = A.split_items[q];
    if (item == kNoItem) continue;
    const int64_t e = (int64_t)((item & ~(kItemTwice | kItemTotal)) >> 24);
    int32_t x, y;
    bool count_total;
    if (!delta_entry<kPredBatch>(A, e, x, y, count_total)) continue;
    count_total = (item & kItemTotal) != 0;
    const DeltaPair P =
        delta_pair<kPredBatch>(A, x, y, A.g.len(x), A.g.len(y), A.g.start(x), A.g.start(y));
    const int32_t i0 = (int32_t)(item & 0xffffffu) * A.chunk;
    if (i0 >= P.la) continue;
    const uint32_t inc = A.weight * (uint32_t)A.sign * (item & kItemTwice ? 2u : 1u);
    const uint32_t c = delta_range<kPredBatch>(A, P, i0, min(P.la, i0 + A.chunk), inc, pv);
    if (lane == 0 && c) {
      atomicAdd(&pv[x], c * inc);
      atomicAdd(&pv[y], c * inc);
      if (count_total) tri_acc += c;
    }
  }
}

// The pair of a described edge.
__device__ __forceinline__ DeltaPair described_pair(const DeltaArgs& A, const DeltaDesc& d) {
  DeltaPair P;
  P.oa = d.oa;
  P.ob = d.ob;
  P.la = d.la;
  P.lb = d.lb;
  P.sa = d.sa;
  P.sb = d.sb;
  P.key = ekey(d.oa, d.ob);
  P.cell = A.use_table ? cell_of(d.la, d.lb) : 0;
  P.strat = pair_strategy<kPredMark>(A, P);
  return P;
}

// Entries [i0, i1) of a described edge's shorter list, run by the warp.
__device__ __forceinline__ void delta_part(const DeltaArgs& A, uint32_t* __restrict__ pv, const DeltaDesc& d,
                                           const int32_t i0, const int32_t i1, unsigned long long& tri_acc) {
  const uint32_t inc = A.weight * (uint32_t)A.sign;
  const uint32_t c = delta_range<kPredMark>(A, described_pair(A, d), i0, i1, inc, pv);
  if ((threadIdx.x & 31) == 0 && c) {
    atomicAdd(&pv[d.oa], c * inc);
    atomicAdd(&pv[d.ob], c * inc);
    tri_acc += c;
  }
}

// Field-wise broadcast of lane k's description.
__device__ __forceinline__ DeltaDesc desc_from(const DeltaDesc& m, const int k) {
  return DeltaDesc{__shfl_sync(kFull, m.oa, k), __shfl_sync(kFull, m.ob, k), __shfl_sync(kFull, m.la, k),
                   __shfl_sync(kFull, m.lb, k), __shfl_sync(kFull, m.sa, k), __shfl_sync(kFull, m.sb, k)};
}

// Elements a warp takes per grab of a queue of cnt: up to kGrab, whose descriptions its lanes read
// together; one where that would leave warps without work.
__device__ __forceinline__ int grab_size(const int64_t cnt) {
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  return (int)max((int64_t)1, min((int64_t)kGrab, cnt / (2 * nw)));
}

// A queue of cnt elements taken `grab` at a time by the grid's warps: each warp's first piece by its
// index, the rest from a shared counter (zero at launch). 7104 warps asking one counter for work
// take longer than a small batch's count.
struct Queue {
  unsigned long long* next;
  int64_t cnt, at, warps;
  int grab;
  __device__ __forceinline__ Queue(unsigned long long* n, const int64_t c) : next(n), cnt(c) {
    warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    grab = grab_size(c);
    at = (((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * grab;
  }
  // Advance to the next piece; `at` is past the end when there is none.
  __device__ __forceinline__ void advance() {
    if (cnt <= warps * grab) {
      at = cnt;
      return;
    }
    unsigned long long g = 0;
    if ((threadIdx.x & 31) == 0) g = atomicAdd(next, (unsigned long long)grab);
    at = warps * grab + (int64_t)__shfl_sync(kFull, g, 0);
  }
};

// The count of the persistent kernel: the queued items of split intersections, then the other
// described edges, one warp each. Both queues are complete before the launch (k_hub_place).
__device__ __forceinline__ void delta_count(const DeltaArgs& A, uint32_t* __restrict__ pv, unsigned long long& tri_acc,
                                            unsigned long long& bytes_acc) {
  const int lane = threadIdx.x & 31;
  const int64_t n_items = (int64_t)min(*A.split_cnt, (unsigned long long)kDeltaItems);
  const int64_t n_desc = (int64_t)*A.n_desc;
  for (Queue q(A.i_next, n_items); q.at < n_items; q.advance()) {
    const int64_t g = q.at;
    const int have = (int)min((int64_t)q.grab, n_items - g);
    DeltaDesc mine = {};
    int32_t i0_l = -1;
    if (lane < have) {
      const unsigned long long item = A.split_items[g + lane];
      if (item != kNoItem) {
        mine = A.desc[item >> 24];
        i0_l = (int32_t)(item & 0xffffffu) * A.chunk;
      }
    }
    __syncwarp();
    for (int k = 0; k < have; ++k) {
      DeltaDesc d = desc_from(mine, k);
      const int32_t i0 = __shfl_sync(kFull, i0_l, k);
      if (i0 < 0) continue;
      d.la &= ~kSplitFlag;
      delta_part(A, pv, d, i0, min(d.la, i0 + A.chunk), tri_acc);
    }
  }
  for (Queue q(A.e_next, n_desc); q.at < n_desc; q.advance()) {
    const int64_t g = q.at;
    const int have = (int)min((int64_t)q.grab, n_desc - g);
    DeltaDesc mine = {};
    if (lane < have) {
      mine = A.desc[g + lane];
      bytes_acc += 4ull * ((unsigned long long)(mine.la & ~kSplitFlag) + (unsigned long long)mine.lb) + 8ull;
    }
    __syncwarp();
    for (int k = 0; k < have; ++k) {
      const DeltaDesc d = desc_from(mine, k);
      if (d.la >= 0) delta_part(A, pv, d, 0, d.la, tri_acc);
    }
  }
}

// Which part of a phase's end a CTA does once the CTAs of its grid have met.
enum : int { kShareOwn, kShareNone, kShareAll };
constexpr unsigned kMeetLeft = 1u << 31;  // of the arrivals: a CTA left before the last one arrived

// All CTAs of a resident grid meet: each waits (spin_ns of device time, at most kSpinMaxIters polls)
// until every other has arrived. The phase's end rewrites what the count reads, so no CTA starts on
// it while another still counts: a CTA whose wait runs out (kErrTimeout) before the last arrival
// leaves its share undone, and the last CTA to arrive then does all of it. kMeetLeft is set only
// below that last arrival, in the word that counts them, so all CTAs see the same outcome.
__device__ __forceinline__ int grid_meet(const DeltaArgs& A) {
  __shared__ int s_share;
  __syncthreads();
  if (threadIdx.x == 0) {
    const unsigned wanted = gridDim.x + A.bar_extra;
    __threadfence();
    unsigned seen = atomicAdd(A.arrived, 1u) + 1u;
    if (!(seen & kMeetLeft)) {
      unsigned long long t0, t;
      asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
      for (unsigned it = 0; (seen & ~kMeetLeft) < wanted; ++it, seen = ld_relaxed(A.arrived)) {
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
        if (it >= kSpinMaxIters || t - t0 > A.spin_ns) {
          atomicOr(A.err, kErrTimeout);
          while ((seen & ~kMeetLeft) < gridDim.x) {
            const unsigned was = atomicCAS(A.arrived, seen, seen | kMeetLeft);
            if (was == seen) break;
            seen = was;
          }
          break;
        }
        __nanosleep(64);
      }
      // here either every CTA of the grid has arrived or this one has left
      s_share = (seen & ~kMeetLeft) < gridDim.x || (seen & kMeetLeft) ? kShareNone : kShareOwn;
    } else {
      s_share = (seen & ~kMeetLeft) == gridDim.x ? kShareAll : kShareNone;
    }
    __threadfence();
  }
  __syncthreads();
  return s_share;
}

// Two launches: the edges, then the items of the split ones (the cuStinger-style count, tc_count_batch).
// Bound by chains of dependent loads, so warps in flight count for more than the few spills that 32
// registers cost. Both directions of present edges of R-MAT 20, counted for deletion, with 6 CTAs an SM
// under a grid of 8 -> 8 CTAs -> and a grid of up to 32 (5 CTAs: + 3 %): 19,996 entries 158 -> 147 -> 141 us,
// 99,912 849 -> 744 -> 668 us, 398,774 2.96 -> 2.37 -> 2.19 ms; up to 2000 entries unchanged.
constexpr int kBatchCtasPerSm = 8;
__global__ void __launch_bounds__(kThreads, kBatchCtasPerSm) k_delta(const DeltaArgs A, uint32_t* __restrict__ pv,
                                                                     unsigned long long* __restrict__ tri_out) {
  const int64_t gw = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  unsigned long long tri_acc = 0, bytes_acc = 0;
  batch_entries(A, pv, gw, nw, tri_acc, bytes_acc);
  delta_flush(tri_acc, bytes_acc, tri_out, A.bytes_out);
}

__global__ void __launch_bounds__(kThreads, kBatchCtasPerSm) k_delta_split(const DeltaArgs A, uint32_t* __restrict__ pv,
                                                                           unsigned long long* __restrict__ tri_out) {
  const int64_t gw = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  unsigned long long tri_acc = 0;
  batch_items(A, pv, gw, nw, tri_acc);
  delta_flush(tri_acc, 0ull, tri_out, nullptr);
}

// What a phase does once its count is done: deletions compact their lists, insertions clear the
// marks of the new slots and add the batch's triangles to the running delta (NULL = not here).
struct PhaseEnd {
  const int4* dlist;               // deletions (phase 0)
  const unsigned long long* n_del;
  CompactArgs cmp;
  const int64_t* slot;             // insertions (phase 1): slots of the 2 * *n_ins new entries
  const unsigned long long* n_ins;
  uint8_t* mark;
  int64_t* delta;
  const unsigned long long* added;
  const unsigned long long* removed;
  BatchStatus* st;
};

// One persistent launch per phase (a resident grid, at most the occupancy limit of CTAs per SM): the
// per-edge count, then, once every CTA has met (grid_meet), the phase's end, so that a small
// batch does not pay a launch for each. The batch's sizes are read from device memory, so one
// captured launch serves every batch of a bin. A meeting that runs out (the grid was not
// resident, or a test forces it) sets kErrTimeout, which the host reports as TC_ERR_TIMEOUT; the
// batch's count and update still complete.
#ifndef TC_DELTA_MIN_BLOCKS
#define TC_DELTA_MIN_BLOCKS 5
#endif
constexpr int kDeltaCtasPerSm = TC_DELTA_MIN_BLOCKS;  // 48 registers; 1000 updates on R-MAT 22: 6 CTAs
                                                      // + 2 %; 10^6: 4 CTAs + 1.3 %
__global__ void __launch_bounds__(kThreads, kDeltaCtasPerSm) k_delta_fused(const DeltaArgs A, const PhaseEnd E,
                                                                           uint32_t* __restrict__ pv,
                                                                           unsigned long long* __restrict__ tri_out) {
  unsigned long long tri_acc = 0, bytes_acc = 0;
  delta_count(A, pv, tri_acc, bytes_acc);
  bytes_acc = warp_sum(bytes_acc);
  delta_flush(tri_acc, bytes_acc, tri_out, A.bytes_out);
  const int share = grid_meet(A);
  if (share == kShareNone) return;
  const int64_t thread = share == kShareAll ? threadIdx.x : (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t threads = share == kShareAll ? blockDim.x : (int64_t)gridDim.x * blockDim.x;
  if (E.dlist) {
    const int64_t ends = 2 * (int64_t)*E.n_del;
    for (int64_t k = thread >> 5; k < ends; k += threads >> 5) {
      const int4 d = E.dlist[k >> 1];
      compact_vertex(E.cmp, k & 1 ? d.y : d.x, E.st);
    }
  } else {
    const int64_t n = 2 * (int64_t)*E.n_ins;
    for (int64_t i = thread; i < n; i += threads) {
      const int64_t at = E.slot[i];
      if (at >= 0) E.mark[at] = 0;
    }
    if (E.delta && thread == 0) *E.delta += (int64_t)__ldcg(E.added) - (int64_t)__ldcg(E.removed);
  }
}

// ---- hub-centred delta count ------------------------------------------------------------------
//
// The changed edges of a batch phase concentrate on few endpoints (R-MAT insertions draw both
// endpoints by degree). An edge {h, s} whose longer-list endpoint h (ties to the smaller id) holds
// at least hub_min of the phase's changed edges is counted at h: a CTA hashes N(h) into shared
// memory, each key with bit 31 set when the edge (h, key) is itself changed (the mark array), and
// its warps stream the partner lists N(s) through the table with coalesced loads, in units of
// kHubUnit entries that the warps take one at a time (a long partner list, another hub's, is
// many units, so no warp holds the others up). Per partner entry that is one shared-memory probe,
// where the per-edge kernel binary-searches it into the longer list. A hub longer than one table
// (kHubPass entries) is hashed in value-range passes: pass pk holds the entries of N(h) in
// [vlo, vhi), and a unit is walked only over its entries in that range (its first and last
// entries tell whether it meets the range; a warp-cooperative sampled search finds where it
// enters), so every partner entry is probed once over the passes. A hub's work is cut into items
// (pass, chunk of its units), each one CTA's table build plus walks, sized so the build is a small
// part of the item; the items of all hubs share one queue, so no hub is a serial tail.
// The keep rule is the per-edge kernel's: a common neighbour w is kept unless (h, w) or (s, w) is
// a changed edge with a smaller key, so every triangle is still attributed to exactly one changed
// edge whichever kernel counts it. Grouping takes three passes over the changed edges: count the
// edges, units and partner entries per longer endpoint, where a vertex becomes a hub when its
// edge count reaches hub_min; give each hub a range of unit slots and its items; place the units
// and describe the other edges for the per-edge kernel. A hub whose units or items do not fit is left
// to that kernel.

#ifndef TC_HUB_THREADS
#define TC_HUB_THREADS 512
#endif
constexpr int kHubThreads = TC_HUB_THREADS;
constexpr int kHubCtasPerSm = 1536 / kHubThreads;
// log2 of the slots of each half of the largest table: 32 slots a thread, 64 KB of keys for 512 threads
constexpr int kHubSlotBits = kHubThreads <= 256 ? 12 : kHubThreads <= 512 ? 13 : 14;
#ifndef TC_HUB_UNIT
#define TC_HUB_UNIT 512
#endif
// Partner entries per unit of work of a warp. Smaller units shorten the wait at the end of an
// item for the warp with the last unit; on the streaming workload 512 entries measured 5 % less
// time than 1024 over the whole run (prefetching the next 128 entries changed nothing).
constexpr int kHubUnit = TC_HUB_UNIT;
constexpr int kHubPass = 3 << (kHubSlotBits - 2);  // entries of N(h) per pass (load <= 3/8)
constexpr int32_t kHubMarkBit = INT32_MIN;    // bit 31 of a stored key: the edge (h, key) is changed
constexpr int64_t kHubSearchCost = 64;        // an item's estimate of one range search, in probes
#ifndef TC_HUB_ITEM_LOG2
#define TC_HUB_ITEM_LOG2 19
#endif
// probes of work per item at least (a build and three block barriers each; 2 x 10^6 updates on R-MAT
// 22: 2^17 10.90 ms a pass, 2^18 10.67, 2^19 10.57, 2^20 10.63) ...
constexpr int64_t kHubItemMin = 1ll << TC_HUB_ITEM_LOG2;
constexpr int64_t kHubBuildShare = 16;        // ... and at least this many times its table build
constexpr int64_t kHubItemsPerUpdate = 4;     // item queue capacity per batch update
constexpr int64_t kHubUnitsPerUpdate = kHubUnit >= 1024 ? 4 : 4 * 1024 / kHubUnit;  // unit slots per update

struct HubWs {
  int32_t* cnt;      // [n] changed edges per longer endpoint in this phase (zero between phases)
  int32_t* uni;      // [n] their partner units (zero between phases)
  long long* sum;    // [n] sum of their partner list lengths (zero between phases)
  int32_t* of;       // [n] hub id + 1 of a vertex (zero between phases)
  int32_t* list;     // [cap] hub vertices
  int32_t* off;      // [cap] first slot of a hub's units in `units`
  int32_t* len;      // [cap] number of units of the hub
  int32_t* chunks;   // [cap] unit chunks of the hub (items per pass)
  int32_t* fill;     // [cap]
  int2* units;       // [unit_cap] (partner s, unit r: entries [r kHubUnit, (r + 1) kHubUnit) of N(s))
  int64_t unit_cap;
  DeltaDesc* desc;   // [cap] the edges not counted at a hub
  unsigned long long* n_desc;
  int on;            // hub groups are formed (0: every edge is described)
  unsigned long long* items;  // [item_cap] (hub id << 32 | item index within the hub)
  int64_t item_cap;
  unsigned long long* n_hubs;
  unsigned long long* total;
  unsigned long long* n_items;
  unsigned long long* q;
};

// Changed edge e as the delta count sees it: false unless this rank counts it and both lists have
// at least two entries; h = the endpoint with the longer list, s = the other one.
__device__ __forceinline__ bool hub_entry(const DeltaArgs& A, int64_t e, int32_t& h, int32_t& s, int32_t& lh,
                                          int32_t& ls) {
  int32_t x, y;
  bool count_total;
  if (!delta_entry<kPredMark>(A, e, x, y, count_total)) return false;
  if (A.nshards > 1 && edge_shard(x, y, A.nshards) != A.shard) return false;
  const int32_t lx = A.g.len(x), ly = A.g.len(y);
  if (lx < 2 || ly < 2) return false;
  const bool x_long = lx > ly || (lx == ly && x < y);
  h = x_long ? x : y;
  s = x_long ? y : x;
  lh = x_long ? lx : ly;
  ls = x_long ? ly : lx;
  return true;
}

__global__ void __launch_bounds__(kThreads) k_hub_count(const DeltaArgs A, const HubWs H) {
  const int64_t cnt = (int64_t)*A.count_dev;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < cnt; e += (int64_t)gridDim.x * blockDim.x) {
    int32_t h, s, lh, ls;
    if (!hub_entry(A, e, h, s, lh, ls)) continue;
    atomicAdd(reinterpret_cast<unsigned long long*>(&H.sum[h]), (unsigned long long)ls);
    atomicAdd(&H.uni[h], (ls + kHubUnit - 1) / kHubUnit);
    if (atomicAdd(&H.cnt[h], 1) + 1 == A.hub_min) {  // exactly one edge sees the count reach hub_min
      const unsigned long long hid = atomicAdd(H.n_hubs, 1ull);
      H.list[hid] = h;
      H.of[h] = (int32_t)hid + 1;
    }
  }
}

// Passes of a hub of lh entries, and the value range of pass pk: its entries are N(h)[cb, cb_next).
__device__ __forceinline__ int hub_passes(int32_t lh) { return (lh + kHubPass - 1) / kHubPass; }

// Unit slots and items per hub, allocated by atomics; a hub whose units or items do not fit drops
// out (its edges go to the per-edge kernel).
__global__ void __launch_bounds__(kThreads) k_hub_alloc(const DeltaArgs A, const HubWs H) {
  const int64_t nh = (int64_t)*H.n_hubs;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nh; i += (int64_t)gridDim.x * blockDim.x) {
    const int32_t h = H.list[i];
    const int32_t k = H.uni[h];
    const int32_t lh = A.g.len(h);
    H.len[i] = 0;
    const unsigned long long off = atomicAdd(H.total, (unsigned long long)k);
    if (off + k > (unsigned long long)H.unit_cap) {
      H.of[h] = 0;
      continue;
    }
    const int P = hub_passes(lh);
    // probes of the hub's walks and searches, over the items' target size
    const long long work = H.sum[h] + (long long)(P - 1) * k * kHubSearchCost;
    const long long build = kHubBuildShare * ((long long)lh / P);
    const long long target = build > (long long)kHubItemMin ? build : (long long)kHubItemMin;
    const long long want = (work + target - 1) / target;
    const int C = (int)(want < 1 ? 1 : want > k ? k : want);
    const long long nitems = (long long)P * C;
    const unsigned long long base = atomicAdd(H.n_items, (unsigned long long)nitems);
    if (base + nitems > (unsigned long long)H.item_cap) {
      for (long long j = 0; j < nitems && base + j < (unsigned long long)H.item_cap; ++j) H.items[base + j] = kNoItem;
      H.of[h] = 0;
      continue;
    }
    for (long long j = 0; j < nitems; ++j) H.items[base + j] = ((unsigned long long)i << 32) | (unsigned long long)j;
    H.len[i] = k;
    H.chunks[i] = C;
    H.off[i] = (int32_t)off;
    H.fill[i] = 0;
  }
}

// Place the units of every hub edge in its hub's range and describe every other edge for the per-edge
// kernel (its lists looked up here once, by a thread per edge, so that a warp of that kernel starts
// with one load), queueing the chunks of long intersections (an edge with a shorter list past
// A.split_min, two hubs, would be one warp's serial tail; a full queue leaves it whole); clears the
// per-vertex counts.
__global__ void __launch_bounds__(kThreads) k_hub_place(const DeltaArgs A, const HubWs H) {
  const int64_t cnt = (int64_t)*A.count_dev;
  const int lane = threadIdx.x & 31;
  for (int64_t e0 = (int64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31); e0 < cnt;
       e0 += (int64_t)gridDim.x * blockDim.x) {
    const int64_t e = e0 + lane;
    int32_t h = 0, s = 0, lh = 0, ls = 0;
    bool left = e < cnt && hub_entry(A, e, h, s, lh, ls);  // counted by the per-edge kernel
    if (left && H.on) {
      const int32_t hid1 = H.of[h];
      if (hid1 > 0) {
        const int32_t u = (ls + kHubUnit - 1) / kHubUnit;
        const int32_t pos = H.off[hid1 - 1] + atomicAdd(&H.fill[hid1 - 1], u);
        for (int32_t r = 0; r < u; ++r) H.units[pos + r] = make_int2(s, r);
        left = false;
      }
      H.cnt[h] = 0;
      H.uni[h] = 0;
      H.sum[h] = 0;
    }
    if (A.cell_filter != -1 && (A.cell_filter == -2 || cell_of(ls, lh) != A.cell_filter)) left = false;
    __syncwarp();
    const unsigned m = __ballot_sync(kFull, left);
    if (m == 0) continue;
    unsigned long long at = 0;
    if (lane == 0) at = atomicAdd(H.n_desc, (unsigned long long)__popc(m));
    at = __shfl_sync(kFull, at, 0);
    const unsigned long long mine = at + __popc(m & ((1u << lane) - 1u));
    int nch = 0;  // items of a split edge
    unsigned long long q = 0;
    if (left) {
      int32_t la = ls;
      if (ls > A.split_min) {
        nch = (ls + A.chunk - 1) / A.chunk;
        q = atomicAdd(A.split_cnt, (unsigned long long)nch);
        if (q + (unsigned long long)nch <= (unsigned long long)kDeltaItems) la |= kSplitFlag;
      }
      H.desc[mine] = DeltaDesc{s, h, la, lh, A.g.start(s), A.g.start(h)};
    }
    __syncwarp();
    for (unsigned split = __ballot_sync(kFull, nch > 0); split; split &= split - 1) {
      const int k = __ffs(split) - 1;
      const int cnt_k = __shfl_sync(kFull, nch, k);
      const unsigned long long q_k = __shfl_sync(kFull, q, k), d_k = __shfl_sync(kFull, mine, k);
      const bool fits = q_k + (unsigned long long)cnt_k <= (unsigned long long)kDeltaItems;
      for (int c = lane; c < cnt_k && q_k + c < (unsigned long long)kDeltaItems; c += 32)
        A.split_items[q_k + c] = fits ? (d_k << 24) | (unsigned long long)c : kNoItem;
    }
  }
}

// A hub's hash set in shared memory: 2 * 2^bits slots of 4 bytes, every key (an id, with kHubMarkBit
// when the edge to it is changed) at one of its two slots, one in each half (cuckoo hashing): a
// lookup is two loads and two comparisons with no loop. Addressed by 32-bit shared addresses.
struct HubSet {
  uint32_t base;
  int bits;
  __device__ __forceinline__ uint32_t slot1(const uint32_t x) const { return ((x >> (30 - bits)) & ~3u) + base; }
  __device__ __forceinline__ uint32_t slot2(const uint32_t x) const {
    return ((x >> (30 - 2 * bits)) & ((4u << bits) - 4u)) + (base + (4u << bits));
  }
};
constexpr int32_t kHubFree = -1;  // no key: ids are below INT32_MAX
constexpr int32_t kHubNone = -2;  // an entry that is not there: equals no id
constexpr int kHubKicks = 64;

__device__ __forceinline__ uint32_t hub_hash(const int32_t id) { return (uint32_t)id * 0x9E3779B1u; }
__device__ __forceinline__ int32_t hub_lds(const uint32_t at) {
  int32_t v;
  asm volatile("ld.shared.s32 %0, [%1];" : "=r"(v) : "r"(at));
  return v;
}

// Insert a key (concurrently with others): into its first slot, the key found there into its other
// one, and so on; false when a key is left over. A key that meets its like is dropped, so the repeats
// of a list that was never checked do not fail the build.
__device__ __forceinline__ bool hub_insert(const HubSet& t, int32_t key) {
  uint32_t at = t.slot1(hub_hash(key & INT32_MAX));
  for (int it = 0; it < kHubKicks; ++it) {
    int32_t old;
    asm volatile("atom.shared.exch.b32 %0, [%1], %2;" : "=r"(old) : "r"(at), "r"(key) : "memory");
    if (old == kHubFree || old == key) return true;
    key = old;
    const uint32_t x = hub_hash(key & INT32_MAX), s1 = t.slot1(x);
    at = at == s1 ? t.slot2(x) : s1;
  }
  return false;
}

// Work items of the hubs from one queue: item (hub, j) is pass j / C over unit chunk j % C of the
// hub's C chunks; its warps walk one unit each. A pass whose table cannot be built (ids chosen
// against the hash) is taken in halves. Bound by its instructions and the partner lists' loads: with
// 16-byte buckets of four keys and the marks read after a hit, a pass of 2 x 10^6 updates on R-MAT 22
// spent 6.98 ms here, with two-slot sets and the marks beside the entries 4.96 ms.
__global__ void __launch_bounds__(kHubThreads, kHubCtasPerSm) k_delta_hub(const DeltaArgs A, const HubWs H,
                                                                          uint32_t* __restrict__ pv,
                                                                          unsigned long long* __restrict__ tri_out) {
  extern __shared__ __align__(16) int32_t hub_keys[];
  __shared__ unsigned long long s_item;
  __shared__ int s_next;
  __shared__ unsigned long long s_red[kHubThreads / 32][2];
  uint32_t table;
  asm volatile("mov.u32 %0, %1;" : "=r"(table) : "r"((uint32_t)__cvta_generic_to_shared(hub_keys)));
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int64_t n_items = (int64_t)min(*H.n_items, (unsigned long long)H.item_cap);
  const uint32_t inc = A.weight * (uint32_t)A.sign;
  unsigned long long tri_acc = 0, bytes_acc = 0;
  while (true) {
    if (threadIdx.x == 0) {
      const unsigned long long q = atomicAdd(H.q, 1ull);
      s_item = q < (unsigned long long)n_items ? H.items[q] : ~1ull;
    }
    __syncthreads();
    const unsigned long long item = s_item;
    if (item == ~1ull) break;
    if (item == kNoItem) {  // a slot of a hub that did not fit
      __syncthreads();
      continue;
    }
    const int32_t hid = (int32_t)(item >> 32), j = (int32_t)(item & 0xffffffffu);
    const int32_t h = H.list[hid], base = H.off[hid], k = H.len[hid], C = H.chunks[hid];
    const int32_t lh = A.g.len(h);
    const int64_t sh = A.g.start(h);
    const int P = hub_passes(lh);
    const int pk = j / C, ci = j % C;
    const int32_t per = (k + C - 1) / C;
    const int32_t e0 = ci * per, e1 = min(k, e0 + per);
    const int cb_end = (int)(((int64_t)(pk + 1) * lh) / P);
    uint32_t hub_c = 0;  // triangles kept at h in this item (lane 0 of each warp)
    int cb = (int)(((int64_t)pk * lh) / P);
    int clen = cb_end - cb;
    HubSet t{table, 4};
    while ((3 << t.bits) < 4 * clen && t.bits < kHubSlotBits) ++t.bits;  // load <= 3/8
    for (; cb < cb_end; cb += clen) {
      clen = min(clen, cb_end - cb);
      while (true) {
        for (int i = threadIdx.x; i < (2 << t.bits) / 4; i += kHubThreads)
          reinterpret_cast<int4*>(hub_keys)[i] = make_int4(kHubFree, kHubFree, kHubFree, kHubFree);
        if (threadIdx.x == 0) s_next = 0;
        __syncthreads();
        bool ok = true;
        for (int i = threadIdx.x; i < clen; i += kHubThreads) {
          const int32_t w = A.g.ind[sh + cb + i];
          ok &= hub_insert(t, A.mark[sh + cb + i] ? (w | kHubMarkBit) : w);
        }
        if (__syncthreads_and(ok)) break;
        clen = (clen + 1) / 2;
      }
      const bool ranged = clen < lh;
      const int32_t vlo = cb == 0 ? INT32_MIN : A.g.ind[sh + cb];
      const int32_t vhi = cb + clen == lh ? INT32_MAX : A.g.ind[sh + cb + clen];
      while (true) {
        int i = 0;
        if (lane == 0) i = atomicAdd(&s_next, 1);
        i = e0 + __shfl_sync(kFull, i, 0);
        if (i >= e1) break;
        const int2 un = H.units[base + i];
        const int32_t s = un.x;
        const int32_t ls = A.g.len(s);
        const int64_t ss = A.g.start(s);
        if (cb == 0 && un.y == 0 && lane == 0) bytes_acc += 4ull * (unsigned long long)(lh + ls) + 8ull;
        int32_t cur = un.y * kHubUnit, end = min(ls, cur + kHubUnit);
        if (ranged) {  // the unit's part in [vlo, vhi), if any
          const int32_t* const u = A.g.ind + ss + cur;
          const int32_t len = end - cur, first = u[0], last = u[len - 1];
          if (last < vlo || first >= vhi) continue;
          if (last >= vhi) end = cur + warp_lower_bound(u, len, vhi);
          if (first < vlo) cur += warp_lower_bound(u, len, vlo);
        }
        const int32_t* lst = A.g.ind + ss + cur + lane;
        const uint8_t* mrk = A.mark + ss + cur + lane;
        uint32_t c = 0;
        // N(s)[cur, end), 128 entries per step: four loads per lane, and the entries' marks beside them
        // (eight loads: 1 % slower; marks read after a hit: 7 %)
        for (int32_t left = end - cur - lane; left > -lane; left -= 128, lst += 128, mrk += 128) {
          int32_t w[4];
          uint32_t m[4];
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            w[r] = left > 32 * r ? lst[32 * r] : kHubNone;
            m[r] = left > 32 * r ? mrk[32 * r] : 0;
          }
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            const uint32_t x = hub_hash(w[r]);
            const int32_t q1 = hub_lds(t.slot1(x)), q2 = hub_lds(t.slot2(x));
            const bool f = (q1 & INT32_MAX) == w[r], g = (q2 & INT32_MAX) == w[r];
            bool keep = f | g;
            if (keep) {
              const bool ch = (f ? q1 : q2) < 0;  // (h, w) is changed
              if (ch || m[r]) {  // or (s, w) is: the triangle is the smallest changed edge's
                const uint64_t key_hs = ekey(h, s);
                keep = (!ch || key_hs < ekey(h, w[r])) && (!m[r] || key_hs < ekey(s, w[r]));
              }
              if (keep) {
                ++c;
                atomicAdd(&pv[w[r]], inc);
              }
            }
          }
          __syncwarp();
        }
        c = __reduce_add_sync(kFull, c);
        if (lane == 0 && c) {
          atomicAdd(&pv[s], c * inc);
          hub_c += c;
          tri_acc += c;
        }
      }
      __syncthreads();
    }
    // h's per-vertex count: one atomic per item
    if (lane == 0) s_red[wid][0] = hub_c;
    __syncthreads();
    if (threadIdx.x == 0) {
      unsigned long long sum = 0;
      for (int w = 0; w < kHubThreads / 32; ++w) sum += s_red[w][0];
      if (sum) atomicAdd(&pv[h], (uint32_t)sum * inc);
      if (j == 0) H.of[h] = 0;  // zero between phases (k_hub_place, its last reader, is done)
    }
    __syncthreads();
  }
  if (lane == 0) {
    s_red[wid][0] = tri_acc;
    s_red[wid][1] = bytes_acc;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long t = 0, b = 0;
    for (int w = 0; w < kHubThreads / 32; ++w) {
      t += s_red[w][0];
      b += s_red[w][1];
    }
    if (t) atomicAdd(tri_out, t);
    if (b && A.bytes_out) atomicAdd(A.bytes_out, b);
  }
}

// ---- cuStinger-style batch helpers ------------------------------------------------------------

__global__ void k_pack_dir(const int32_t* __restrict__ s, const int32_t* __restrict__ d, const int64_t b,
                           uint64_t* __restrict__ keys) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < b; i += (int64_t)gridDim.x * blockDim.x)
    keys[i] = ((uint64_t)(uint32_t)s[i] << 32) | (uint32_t)d[i];
}

__global__ void k_unpack_dir(const uint64_t* __restrict__ keys, const int64_t b, const int32_t nv, int32_t* __restrict__ s,
                             int32_t* __restrict__ d, int32_t* __restrict__ dup, int32_t* __restrict__ cnt,
                             unsigned* __restrict__ err) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < b; i += (int64_t)gridDim.x * blockDim.x) {
    const uint64_t k = keys[i];
    const int32_t a = (int32_t)(k >> 32), c = (int32_t)(uint32_t)k;
    s[i] = a;
    d[i] = c;
    const bool bad = a < 0 || a >= nv || c < 0 || c >= nv;
    if (bad) {
      atomicOr(err, kErrRange);
      dup[i] = 1;
      continue;
    }
    dup[i] = (a == c) || (i > 0 && keys[i - 1] == k);
    atomicAdd(&cnt[a], 1);
  }
}

// Entries with dup == 0 that are already in the graph become duplicates; the rest are packed
// as directed insertion keys (sentinel elsewhere).
__global__ void k_flag_present(const SlackView g, const int32_t* __restrict__ s, const int32_t* __restrict__ d,
                               int32_t* __restrict__ dup, const int64_t b, const int L, uint64_t* __restrict__ dk,
                               BatchStatus* __restrict__ st) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < b; i += (int64_t)gridDim.x * blockDim.x) {
    uint64_t k = kSentinel;
    if (!dup[i]) {
      const int32_t x = s[i], y = d[i];
      const int64_t sx = g.start(x);
      const int32_t lx = g.len(x);
      const int64_t p = lower_bound(g.ind, sx, sx + lx, y);
      if (p < sx + lx && g.ind[p] == y) dup[i] = 1;
      else k = ((uint64_t)(uint32_t)x << L) | (uint32_t)y;
      if (k == (1ull << (2 * L)) - 1) atomicOr(&st->err, kLastSelfLoop);
    }
    dk[i] = k;
  }
}

// Mark the slots of present, non-duplicate entries for deletion; list their source vertices.
__global__ void k_mark_dir_deletions(const SlackView g, const int32_t* __restrict__ s, const int32_t* __restrict__ d,
                                     const int32_t* __restrict__ dup, const int64_t b, uint8_t* __restrict__ mark,
                                     int32_t* __restrict__ first_del, int32_t* __restrict__ vlist,
                                     unsigned long long* __restrict__ nvl) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < b; i += (int64_t)gridDim.x * blockDim.x) {
    if (dup[i]) continue;
    const int32_t x = s[i], y = d[i];
    const int64_t sx = g.start(x);
    const int32_t lx = g.len(x);
    const int64_t p = lower_bound(g.ind, sx, sx + lx, y);
    if (p < sx + lx && g.ind[p] == y) {
      mark[p] = 1;
      atomicMin(&first_del[x], (int32_t)(p - sx));
      vlist[atomicAdd(nvl, 1ull)] = x;
    }
  }
}

// The compaction epoch lives on the device so that a captured launch sequence advances it.
__global__ void k_bump_epoch(unsigned* __restrict__ epoch) {
  if (threadIdx.x == 0 && blockIdx.x == 0) *epoch += 1u;
}

__global__ void k_add_delta(int64_t* __restrict__ delta, const unsigned long long* __restrict__ add,
                            const unsigned long long* __restrict__ sub) {
  if (threadIdx.x == 0 && blockIdx.x == 0) *delta += (int64_t)(add ? *add : 0ull) - (int64_t)(sub ? *sub : 0ull);
}

__global__ void k_to_int32(const int64_t* __restrict__ in, const int64_t n, int32_t* __restrict__ out) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i <= n; i += (int64_t)gridDim.x * blockDim.x)
    out[i] = (int32_t)in[i];
}

}  // namespace

// ---- per-graph streaming workspace -----------------------------------------------------------

struct StreamWs {
  int64_t b_cap = 0;
  int64_t n_cap = 0;
  int32_t* src = nullptr;       // host batches staged here
  int32_t* dst = nullptr;
  uint8_t* isdel = nullptr;
  uint64_t* keys = nullptr;     // [b]
  uint64_t* keys2 = nullptr;    // [b]
  int4* dlist = nullptr;        // [b]
  int2* ilist = nullptr;        // [b]
  uint64_t* dk = nullptr;       // [2b]
  uint64_t* dk2 = nullptr;      // [2b]
  int2* runs = nullptr;         // [2b]
  LongPlan* long_plan = nullptr;  // [2b]
  CmpPlan* cmp_plan = nullptr;    // [2b] long lists with deletions
  // long-list insertion scratch, sized with the pool (ensure_long_scratch)
  int32_t* long_scr = nullptr;
  uint8_t* long_smark = nullptr;
  unsigned long long* long_items = nullptr;
  int2* long_chunk = nullptr;     // per work item: (output offset, kept entries) of a compacted chunk
  int64_t scr_cap = 0;
  int64_t long_item_cap = 0;
  int64_t* ins_slot = nullptr;  // [2b]
  int32_t* vlist = nullptr;     // [2b]
  unsigned* claim = nullptr;    // [n]
  int32_t* first_del = nullptr; // [n] smallest marked slot of a list in this batch (kNoDel otherwise)
  unsigned* d_epoch = nullptr;  // [1] compaction epoch
  uint64_t version = 0;         // bumped when the batch-sized buffers are reallocated
  void* cub_tmp = nullptr;
  size_t cub_bytes = 0;
  BatchStatus* st = nullptr;
  BatchStatus* st_host = nullptr;  // pinned
  unsigned long long* counter = nullptr;
  int32_t* cnt = nullptr;       // [n+1] per-source counts (cuStinger sort)
  int64_t* scan64 = nullptr;    // [n+1]
  int64_t* tiles = nullptr;
  unsigned long long* split_items = nullptr;  // [kDeltaItems] queued chunks of long intersections
  // hub groups of the delta count (k_delta_hub)
  int32_t* hub_cnt = nullptr;     // [n] zero between phases
  long long* hub_sum = nullptr;   // [n] zero between phases
  int32_t* hub_uni = nullptr;     // [n] zero between phases
  int32_t* hub_of = nullptr;      // [n] zero between phases
  int32_t* hub_list = nullptr;    // [b]
  int32_t* hub_off = nullptr;     // [b]
  int32_t* hub_len = nullptr;     // [b]
  int32_t* hub_fill = nullptr;    // [b]
  int32_t* hub_chunks = nullptr;  // [b]
  int2* hub_units = nullptr;      // [kHubUnitsPerUpdate * b]
  DeltaDesc* desc = nullptr;      // [b] changed edges of the per-edge kernel
  unsigned long long* hub_items = nullptr;  // [kHubItemsPerUpdate * b]
  void release();
};

void StreamWs::release() {
  cudaFree(src); cudaFree(dst); cudaFree(isdel); cudaFree(keys); cudaFree(keys2);
  cudaFree(dlist); cudaFree(ilist); cudaFree(dk); cudaFree(dk2); cudaFree(runs);
  cudaFree(long_plan); cudaFree(long_scr); cudaFree(long_smark); cudaFree(long_items);
  cudaFree(cmp_plan); cudaFree(long_chunk);
  cudaFree(ins_slot);
  cudaFree(vlist); cudaFree(claim); cudaFree(first_del); cudaFree(d_epoch); cudaFree(cub_tmp); cudaFree(st); cudaFreeHost(st_host); cudaFree(counter);
  cudaFree(cnt); cudaFree(scan64); cudaFree(tiles); cudaFree(split_items);
  cudaFree(hub_cnt); cudaFree(hub_sum); cudaFree(hub_uni); cudaFree(hub_of); cudaFree(hub_list); cudaFree(hub_off);
  cudaFree(hub_len); cudaFree(hub_fill); cudaFree(hub_chunks); cudaFree(hub_units); cudaFree(desc);
  cudaFree(hub_items);
  *this = StreamWs();
}

void release_stream_ws(StreamWs* w) {
  if (!w) return;
  w->release();
  delete w;
}

namespace {

// Allocate (or grow) the batch workspace. Each group of arrays is replaced as a whole: a failed
// allocation frees the group and leaves its capacity at 0, so a later call allocates it again and
// no kernel sees a freed or missing array (the graph itself is untouched).
tc_status ensure_stream_ws(tc_graph* g, int64_t b) {
  if (!g->sw) g->sw = new StreamWs();
  StreamWs& w = *g->sw;
  if (!g->mark) {
    uint8_t* mk = nullptr;
    if (::tc::dev_malloc(&mk, (size_t)std::max<int64_t>(g->pool_cap, 1)) != cudaSuccess)
      return fail(TC_ERR_OOM, "edge marks: device allocation failed");
    const cudaError_t e = cudaMemset(mk, 0, (size_t)std::max<int64_t>(g->pool_cap, 1));
    if (e != cudaSuccess) {
      cudaFree(mk);
      return fail(TC_ERR_CUDA, "edge marks: %s", cudaGetErrorString(e));
    }
    g->mark = mk;
  }
  if (w.n_cap < (int64_t)g->n + 1) {
    auto free_pv = [&w]() {
      cudaFree(w.claim); cudaFree(w.first_del); cudaFree(w.cnt); cudaFree(w.scan64); cudaFree(w.tiles);
      cudaFree(w.d_epoch);
      cudaFree(w.hub_cnt); cudaFree(w.hub_sum); cudaFree(w.hub_uni); cudaFree(w.hub_of);
      w.claim = nullptr; w.first_del = nullptr; w.cnt = nullptr; w.scan64 = nullptr; w.tiles = nullptr;
      w.d_epoch = nullptr;
      w.hub_cnt = nullptr; w.hub_sum = nullptr; w.hub_uni = nullptr; w.hub_of = nullptr;
      w.n_cap = 0;
    };
    free_pv();
    ++w.version;
    const size_t n1 = (size_t)g->n + 1;
    if (::tc::dev_malloc(&w.claim, sizeof(unsigned) * n1) != cudaSuccess ||
        ::tc::dev_malloc(&w.first_del, sizeof(int32_t) * n1) != cudaSuccess ||
        ::tc::dev_malloc(&w.d_epoch, sizeof(unsigned)) != cudaSuccess ||
        ::tc::dev_malloc(&w.cnt, sizeof(int32_t) * n1) != cudaSuccess ||
        ::tc::dev_malloc(&w.scan64, sizeof(int64_t) * (n1 + 1)) != cudaSuccess ||
        ::tc::dev_malloc(&w.tiles, sizeof(int64_t) * (size_t)(scan_tiles(g->n + 1) + 1)) != cudaSuccess ||
        ::tc::dev_malloc(&w.hub_cnt, sizeof(int32_t) * n1) != cudaSuccess ||
        ::tc::dev_malloc(&w.hub_sum, sizeof(long long) * n1) != cudaSuccess ||
        ::tc::dev_malloc(&w.hub_uni, sizeof(int32_t) * n1) != cudaSuccess ||
        ::tc::dev_malloc(&w.hub_of, sizeof(int32_t) * n1) != cudaSuccess) {
      free_pv();
      return fail(TC_ERR_OOM, "batch workspace (per vertex): device allocation failed");
    }
    TC_CUDA_TRY(cudaMemset(w.claim, 0, sizeof(unsigned) * n1));
    TC_CUDA_TRY(cudaMemset(w.first_del, 0x7f, sizeof(int32_t) * n1));  // kNoDel
    TC_CUDA_TRY(cudaMemset(w.d_epoch, 0, sizeof(unsigned)));
    TC_CUDA_TRY(cudaMemset(w.hub_cnt, 0, sizeof(int32_t) * n1));
    TC_CUDA_TRY(cudaMemset(w.hub_sum, 0, sizeof(long long) * n1));
    TC_CUDA_TRY(cudaMemset(w.hub_uni, 0, sizeof(int32_t) * n1));
    TC_CUDA_TRY(cudaMemset(w.hub_of, 0, sizeof(int32_t) * n1));
    w.n_cap = g->n + 1;
  }
  if (!w.st || !w.st_host || !w.counter || !w.split_items) {
    auto free_st = [&w]() {
      cudaFree(w.st); cudaFreeHost(w.st_host); cudaFree(w.counter); cudaFree(w.split_items);
      w.st = nullptr; w.st_host = nullptr; w.counter = nullptr; w.split_items = nullptr;
    };
    free_st();
    if (::tc::dev_malloc(&w.st, sizeof(BatchStatus)) != cudaSuccess ||
        cudaMallocHost(&w.st_host, sizeof(BatchStatus)) != cudaSuccess ||
        ::tc::dev_malloc(&w.counter, sizeof(unsigned long long)) != cudaSuccess ||
        ::tc::dev_malloc(&w.split_items, sizeof(unsigned long long) * kDeltaItems) != cudaSuccess) {
      free_st();
      return fail(TC_ERR_OOM, "batch status: allocation failed");
    }
    ++w.version;
  }
  if (b <= w.b_cap) return TC_OK;
  const int64_t nb = std::max<int64_t>(b, 1024);
  auto free_batch = [&w]() {
    cudaFree(w.src); cudaFree(w.dst); cudaFree(w.isdel); cudaFree(w.keys); cudaFree(w.keys2);
    cudaFree(w.dlist); cudaFree(w.ilist); cudaFree(w.dk); cudaFree(w.dk2); cudaFree(w.runs);
    cudaFree(w.ins_slot); cudaFree(w.vlist); cudaFree(w.cub_tmp);
    cudaFree(w.long_plan); cudaFree(w.cmp_plan);
    w.long_plan = nullptr; w.cmp_plan = nullptr;
    cudaFree(w.hub_list); cudaFree(w.hub_off); cudaFree(w.hub_len); cudaFree(w.hub_fill); cudaFree(w.hub_chunks);
    cudaFree(w.hub_units); cudaFree(w.desc); cudaFree(w.hub_items);
    w.src = nullptr; w.dst = nullptr; w.isdel = nullptr; w.keys = nullptr; w.keys2 = nullptr;
    w.dlist = nullptr; w.ilist = nullptr; w.dk = nullptr; w.dk2 = nullptr; w.runs = nullptr;
    w.ins_slot = nullptr; w.vlist = nullptr; w.cub_tmp = nullptr;
    w.hub_list = nullptr; w.hub_off = nullptr; w.hub_len = nullptr; w.hub_fill = nullptr; w.hub_chunks = nullptr;
    w.hub_units = nullptr; w.desc = nullptr; w.hub_items = nullptr;
    w.b_cap = 0;
    w.cub_bytes = 0;
  };
  free_batch();
  ++w.version;
  size_t t1 = 0, t2 = 0;
  bool ok = ::tc::dev_malloc(&w.src, sizeof(int32_t) * nb) == cudaSuccess &&
            ::tc::dev_malloc(&w.dst, sizeof(int32_t) * nb) == cudaSuccess &&
            ::tc::dev_malloc(&w.isdel, nb) == cudaSuccess &&
            ::tc::dev_malloc(&w.keys, sizeof(uint64_t) * nb) == cudaSuccess &&
            ::tc::dev_malloc(&w.keys2, sizeof(uint64_t) * nb) == cudaSuccess &&
            ::tc::dev_malloc(&w.dlist, sizeof(int4) * nb) == cudaSuccess &&
            ::tc::dev_malloc(&w.ilist, sizeof(int2) * nb) == cudaSuccess &&
            ::tc::dev_malloc(&w.dk, sizeof(uint64_t) * 2 * nb) == cudaSuccess &&
            ::tc::dev_malloc(&w.dk2, sizeof(uint64_t) * 2 * nb) == cudaSuccess &&
            ::tc::dev_malloc(&w.runs, sizeof(int2) * 2 * nb) == cudaSuccess &&
            ::tc::dev_malloc(&w.long_plan, sizeof(LongPlan) * 2 * nb) == cudaSuccess &&
            ::tc::dev_malloc(&w.cmp_plan, sizeof(CmpPlan) * 2 * nb) == cudaSuccess &&
            ::tc::dev_malloc(&w.ins_slot, sizeof(int64_t) * 2 * nb) == cudaSuccess &&
            ::tc::dev_malloc(&w.vlist, sizeof(int32_t) * 2 * nb) == cudaSuccess &&
            ::tc::dev_malloc(&w.hub_list, sizeof(int32_t) * nb) == cudaSuccess &&
            ::tc::dev_malloc(&w.hub_off, sizeof(int32_t) * nb) == cudaSuccess &&
            ::tc::dev_malloc(&w.hub_len, sizeof(int32_t) * nb) == cudaSuccess &&
            ::tc::dev_malloc(&w.hub_fill, sizeof(int32_t) * nb) == cudaSuccess &&
            ::tc::dev_malloc(&w.hub_chunks, sizeof(int32_t) * nb) == cudaSuccess &&
            ::tc::dev_malloc(&w.hub_units, sizeof(int2) * kHubUnitsPerUpdate * nb) == cudaSuccess &&
            ::tc::dev_malloc(&w.desc, sizeof(DeltaDesc) * nb) == cudaSuccess &&
            ::tc::dev_malloc(&w.hub_items, sizeof(unsigned long long) * kHubItemsPerUpdate * nb) == cudaSuccess &&
            cub::DeviceRadixSort::SortKeys(nullptr, t1, w.keys, w.keys2, (int)(2 * nb)) == cudaSuccess &&
            cub::DeviceRadixSort::SortKeys(nullptr, t2, w.dk, w.dk2, (int)(2 * nb)) == cudaSuccess &&
            ::tc::dev_malloc(&w.cub_tmp, std::max(t1, t2)) == cudaSuccess;
  if (!ok) {
    free_batch();
    return fail(TC_ERR_OOM, "batch workspace for %lld updates: device allocation failed", (long long)nb);
  }
  w.cub_bytes = std::max(t1, t2);
  w.b_cap = nb;
  return TC_OK;
}

// Scratch of the long-list insertion: the merged suffixes of one batch's long lists, at most every
// entry of the pool plus the batch's new ones (pool_cap + 2 b), and their work items. Follows the
// pool's capacity; a reallocation bumps the workspace version (captured graphs hold the pointers).
tc_status ensure_long_scratch(tc_graph* g) {
  if (!g->sw) return TC_OK;
  StreamWs& w = *g->sw;
  const int64_t need = g->pool_cap + 2 * w.b_cap;
  if (w.scr_cap >= need && w.long_scr && w.long_smark && w.long_items && w.long_chunk) return TC_OK;
  cudaFree(w.long_scr);
  cudaFree(w.long_smark);
  cudaFree(w.long_items);
  cudaFree(w.long_chunk);
  w.long_scr = nullptr;
  w.long_smark = nullptr;
  w.long_items = nullptr;
  w.long_chunk = nullptr;
  w.scr_cap = 0;
  w.long_item_cap = 0;
  ++w.version;
  const int64_t cap = need + need / 4;
  const int64_t icap = cap / kLongChunk + 2 * w.b_cap + 1;
  if (::tc::dev_malloc(&w.long_scr, sizeof(int32_t) * (size_t)cap) != cudaSuccess ||
      ::tc::dev_malloc(&w.long_smark, (size_t)cap) != cudaSuccess ||
      ::tc::dev_malloc(&w.long_items, sizeof(unsigned long long) * (size_t)icap) != cudaSuccess ||
      ::tc::dev_malloc(&w.long_chunk, sizeof(int2) * (size_t)icap) != cudaSuccess) {
    cudaFree(w.long_scr);
    cudaFree(w.long_smark);
    cudaFree(w.long_items);
    cudaFree(w.long_chunk);
    w.long_scr = nullptr;
    w.long_smark = nullptr;
    w.long_items = nullptr;
    w.long_chunk = nullptr;
    return fail(TC_ERR_OOM, "long-list insertion scratch: device allocation failed");
  }
  w.scr_cap = cap;
  w.long_item_cap = icap;
  return TC_OK;
}

// Make room for `extra` slots past pool_top (grow the pool and the mark array by copying), and
// size the long-list insertion scratch to the pool.
tc_status ensure_pool(tc_graph* g, int64_t extra, cudaStream_t s) {
  const int64_t need = g->pool_top + extra;
  if (need <= g->pool_cap) return ensure_long_scratch(g);
  const int64_t ncap = std::max<int64_t>(need + need / 4, g->pool_cap * 3 / 2);
  int32_t* np = nullptr;
  uint8_t* nm = nullptr;
  if (::tc::dev_malloc(&np, sizeof(int32_t) * (size_t)ncap) != cudaSuccess ||
      ::tc::dev_malloc(&nm, (size_t)ncap) != cudaSuccess) {
    cudaFree(np);
    cudaFree(nm);
    return fail(TC_ERR_OOM, "adjacency pool growth to %lld slots: device allocation failed", (long long)ncap);
  }
  TC_CUDA_TRY(cudaMemcpyAsync(np, g->pool, sizeof(int32_t) * (size_t)g->pool_top, cudaMemcpyDeviceToDevice, s));
  TC_CUDA_TRY(cudaMemsetAsync(nm, 0, (size_t)ncap, s));
  if (g->mark) TC_CUDA_TRY(cudaMemcpyAsync(nm, g->mark, (size_t)g->pool_top, cudaMemcpyDeviceToDevice, s));
  TC_CUDA_TRY(cudaStreamSynchronize(s));
  cudaFree(g->pool);
  cudaFree(g->mark);
  g->pool = np;
  g->mark = nm;
  g->pool_cap = ncap;
  g->view_version++;
  return ensure_long_scratch(g);
}

int bits_for(int32_t n) {
  int L = 1;
  while (L < 31 && ((int64_t)1 << L) < (int64_t)n) ++L;
  return L;
}

DeltaArgs delta_args(tc_graph* g, const SchedParams& sp) {
  DeltaArgs A;
  memset(&A, 0, sizeof(A));
  A.g = SlackView{g->start, g->used, g->pool};
  A.mark = g->mark;
  A.search_ratio_x16 = sp.search_ratio_x16;
  A.use_table = sp.use_table;
  A.cell_filter = sp.cell_filter;
  A.shard = sp.shard;
  A.nshards = sp.nshards;
  A.spin_ns = kSpinNs;
  A.hub_min = sp.hub_min;
  memcpy(A.table, sp.table, sizeof(A.table));
  // staging buffers only for launches whose strategy table stages somewhere
  if (A.use_table)
    for (int c = 0; c < 256; ++c) A.stage_ok |= A.table[c] == kStratStage;
  return A;
}

struct PipeCand {
  int ctas;       // persistent delta kernel CTAs per SM (0 = the occupancy limit)
  int chunk;      // split-item size: entries of the shorter list
  int split_min;  // intersections whose shorter list is longer than this are split
};
constexpr PipeCand kPipeCand[kPipeCands] = {
    {0, 1024, 2048}, {0, 512, 1024}, {0, 256, 512}, {0, 128, 256}, {0, 64, 128}};

// The shape without tuning, for a phase of about `edges` changed edges: small items where few edges
// share the chip (a warp searching 1024 entries into a hub's list is a chain of hundreds of
// dependent loads: batches of 3-1000 updates on R-MAT 22 6.7 ms with items of 1024, 3.2 ms with 64,
// a pass of 12 batches), larger ones where the items' own look-ups count (10^6 updates: 13.4 ms a
// pass with 256, 14.1 with 64, 14.4 with 1024).
int default_cand(int64_t edges) { return edges <= ((int64_t)1 << 15) ? 4 : 2; }

// Dynamic shared memory of a delta-kernel launch with these arguments.
size_t delta_smem(const DeltaArgs& A) { return A.stage_ok ? kStageSmem : 0; }

// CTAs of the cuStinger-style count over a batch of `entries`: a warp per entry up to four times the
// resident grid (8 CTAs an SM), which evens out warps whose edges are long; at least the resident
// grid, as the split items of few entries can fill it.
int delta_grid(int64_t entries) {
  const int64_t few = device_info().sms * 8, many = device_info().sms * 32;
  return (int)std::min(many, std::max(few, (entries + kThreads / 32 - 1) / (kThreads / 32)));
}
int long_grid() { return device_info().sms * 8; }

CompactArgs compact_args(tc_graph* g, StreamWs& w) {
  return CompactArgs{g->start, g->used,      g->pool,       g->mark,         w.claim,  w.d_epoch,
                     w.first_del, w.cmp_plan, w.long_items, w.long_item_cap, w.scr_cap};
}

// The long lists that a compaction (compact_vertex) planned. The scratch must be sized
// (ensure_long_scratch).
void long_compact(tc_graph* g, StreamWs& w, cudaStream_t s) {
  k_cmp_stage<<<long_grid(), kThreads, 0, s>>>(w.cmp_plan, w.long_items, w.long_item_cap, g->pool, g->mark, w.long_scr,
                                               w.long_chunk, g->used, w.st);
  k_cmp_write<<<long_grid(), kThreads, 0, s>>>(w.cmp_plan, w.long_items, w.long_item_cap, w.long_scr, w.long_chunk,
                                               g->pool, w.st);
}

// Insertion of the sorted directed keys w.dk2, in at most `runs` runs; the scratch
// must be sized (ensure_pool).
void insert_sorted_keys(tc_graph* g, StreamWs& w, int64_t runs, int L, uint8_t* mark, cudaStream_t s) {
  const InsertArgs I{w.dk2,      L,           w.runs,    g->start,     g->used,      g->cap,         g->pool,
                     g->pool_cap, mark,    w.ins_slot,  g->d_pool_top,  g->slack_q10, w.long_plan,  w.long_items,
                     w.long_item_cap, w.scr_cap};
  k_insert_runs<<<grid_for(runs * 32, kThreads), kThreads, 0, s>>>(I, w.st);
  k_long_stage<<<long_grid(), kThreads, 0, s>>>(w.dk2, L, g->pool, w.long_plan, w.long_items, w.long_item_cap, w.long_scr,
                                                w.long_smark, w.ins_slot, w.st);
  k_long_write<<<long_grid(), kThreads, 0, s>>>(w.long_plan, w.long_items, w.long_item_cap, w.long_scr, w.long_smark,
                                                g->pool, mark, w.st);
}

// Batches of at most kWarpClassify updates are classified by a warp per key (k_classify_warp).
constexpr int64_t kWarpClassify = 8192;

// From the sorted keys w.keys2 (cap of them) to the changed-edge lists and the sorted directed keys
// w.dk2 with their runs.
cudaError_t classify_and_sort(tc_graph* g, StreamWs& w, int64_t cap, int L, cudaStream_t s) {
  const SlackView view{g->start, g->used, g->pool};
  if (cap <= kWarpClassify)
    k_classify_warp<<<grid_for(cap * 32, kThreads), kThreads, 0, s>>>(view, w.keys2, cap, L, w.dlist, w.ilist, w.dk, w.st);
  else
    k_classify<<<grid_for(cap, kThreads), kThreads, 0, s>>>(view, w.keys2, cap, L, w.dlist, w.ilist, w.dk, w.st);
  if (cap <= kSmallBatch) {
    k_sort_runs<<<1, kSortThreads, 0, s>>>(w.dk, cap, L, w.dk2, g->used, g->cap, g->slack_q10, w.runs, w.st);
    return cudaSuccess;
  }
  // the sentinels' low 2L bits are all ones, which no edge has (it would be a self-loop)
  size_t tb = w.cub_bytes;
  const cudaError_t e = cub::DeviceRadixSort::SortKeys(w.cub_tmp, tb, w.dk, w.dk2, (int)(2 * cap), 0, 2 * L, s);
  if (e != cudaSuccess) return e;
  k_dir_runs<<<grid_for(2 * cap, kThreads), kThreads, 0, s>>>(w.dk2, 2 * cap, L, g->used, g->cap, g->slack_q10,
                                                              w.runs, w.st);
  return cudaSuccess;
}

// The keys of a device batch of b <= cap updates into w.keys2, sorted, or (cap > kSmallBatch) into
// w.keys, to be sorted; the status starts at zero.
cudaError_t load_batch(tc_graph* g, StreamWs& w, const int32_t* src, const int32_t* dst, const uint8_t* is_del, int64_t b,
                       int64_t cap, int L, cudaStream_t s) {
  const cudaError_t e = cudaMemsetAsync(w.st, 0, sizeof(BatchStatus), s);
  if (e != cudaSuccess) return e;
  if (cap <= kSmallBatch)
    k_load_sorted<<<1, kSortThreads, 0, s>>>(src, dst, is_del, b, cap, g->n, L, w.keys2, w.st);
  else
    k_load_keys<<<grid_for(cap, kThreads), kThreads, 0, s>>>(src, dst, is_del, b, cap, g->n, L, w.keys, w.dk, w.st);
  return cudaGetLastError();
}

cudaError_t sort_batch(StreamWs& w, int64_t cap, int L, cudaStream_t s) {
  if (cap <= kSmallBatch) return cudaSuccess;  // k_load_sorted did
  size_t tb = w.cub_bytes;
  return cub::DeviceRadixSort::SortKeys(w.cub_tmp, tb, w.keys, w.keys2, (int)cap, 0, 2 * L + 1, s);
}

// Grid of the persistent delta kernel: ctas_per_sm CTAs per SM (0 = the occupancy limit), never
// more than can be resident at once (its CTAs meet before the phase's end).
tc_status fused_grid(int ctas_per_sm, size_t smem, int* grid) {
  constexpr int kMaxDev = 64;
  static int occ[kMaxDev][2] = {};  // without, with the staging buffers
  int dev = 0;
  TC_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxDev) return fail(TC_ERR_INVALID_ARG, "device %d out of range", dev);
  const int k = smem > 0 ? 1 : 0;
  if (occ[dev][k] == 0) {
    int b = 0;
    TC_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_delta_fused, kThreads, k ? kStageSmem : 0));
    occ[dev][k] = std::max(1, b);
  }
  const int per_sm = ctas_per_sm > 0 ? std::min(ctas_per_sm, occ[dev][k]) : occ[dev][k];
  *grid = device_info().sms * per_sm;
  return TC_OK;
}

constexpr size_t kHubSmem = sizeof(int32_t) * (2 << kHubSlotBits);

// Grid of the hub kernel: its occupancy limit of CTAs per SM (64 KB of shared memory each).
tc_status hub_grid(int* grid) {
  constexpr int kMaxDev = 64;
  static int occ[kMaxDev] = {};
  int dev = 0;
  TC_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxDev) return fail(TC_ERR_INVALID_ARG, "device %d out of range", dev);
  if (occ[dev] == 0) {
    TC_CUDA_TRY(cudaFuncSetAttribute(k_delta_hub, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kHubSmem));
    int b = 0;
    TC_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_delta_hub, kHubThreads, kHubSmem));
    occ[dev] = std::max(1, b);
  }
  *grid = device_info().sms * occ[dev];
  return TC_OK;
}

// Phases of at most this many changed edges form no hub groups, which saves three launches (k_hub_count,
// k_hub_alloc and k_delta_hub; k_hub_place describes the edges in any case).
constexpr int64_t kHubBatchMin = kSmallBatch;

// Hub groups and their count for one phase of a batch (deletions: phase 0, insertions: 1) on a
// grid of `grid` hub CTAs, and the descriptions of the edges left to the per-edge kernel that
// follows (all of them when the hub count is off: hub_min <= 0, a small batch, or a timing run of
// one degree cell); `cap` bounds the phase's changed edges. Launches only (it can run inside a stream capture).
void hub_kernels(DeltaArgs& A, StreamWs& w, int phase, int64_t cap, int grid, uint32_t* pv,
                 unsigned long long* tri_out, cudaStream_t s) {
  HubWs H;
  H.cnt = w.hub_cnt;
  H.sum = w.hub_sum;
  H.uni = w.hub_uni;
  H.of = w.hub_of;
  H.list = w.hub_list;
  H.off = w.hub_off;
  H.len = w.hub_len;
  H.chunks = w.hub_chunks;
  H.fill = w.hub_fill;
  H.units = w.hub_units;
  H.unit_cap = kHubUnitsPerUpdate * w.b_cap;
  H.desc = w.desc;
  H.n_desc = &w.st->n_desc[phase];
  H.on = A.hub_min > 0 && A.cell_filter == -1 && cap > kHubBatchMin;
  H.items = w.hub_items;
  H.item_cap = kHubItemsPerUpdate * w.b_cap;
  H.n_hubs = &w.st->n_hubs[phase];
  H.total = &w.st->hub_total[phase];
  H.n_items = &w.st->hub_items[phase];
  H.q = &w.st->hub_q[phase];
  A.desc = w.desc;
  A.n_desc = H.n_desc;
  const int gb = grid_for(cap, kThreads);
  if (H.on) {
    k_hub_count<<<gb, kThreads, 0, s>>>(A, H);
    k_hub_alloc<<<gb, kThreads, 0, s>>>(A, H);
  }
  k_hub_place<<<gb, kThreads, 0, s>>>(A, H);
  if (H.on) k_delta_hub<<<grid, kHubThreads, kHubSmem, s>>>(A, H, pv, tri_out);
}

// The delta of one phase of a batch (deletions: phase 0, insertions: 1) on the batch workspace's
// counters: hub groups, then the persistent kernel with the phase's end, on grids found outside
// (launches only: it can run inside a stream capture).
void delta_phase(tc_graph* g, StreamWs& w, const SchedParams& sp, int phase, int64_t cap, const PipeCand& shape,
                 int ghub, int gdelta, uint32_t* pv, int64_t* delta, unsigned long long spin_ns, unsigned bar_extra,
                 cudaStream_t s) {
  DeltaArgs A = delta_args(g, sp);
  unsigned long long* const tri = phase ? &w.st->tri_added : &w.st->tri_removed;
  if (phase) A.ilist = w.ilist;
  else A.dlist = w.dlist;
  A.count_dev = phase ? &w.st->n_ins : &w.st->n_del;
  A.sign = phase ? 1 : -1;
  A.weight = 2;
  A.chunk = shape.chunk;
  A.split_min = shape.split_min;
  A.spin_ns = spin_ns;
  A.bar_extra = bar_extra;
  A.split_items = w.split_items;
  A.split_cnt = &w.st->n_split[phase];
  A.arrived = &w.st->arrived[phase];
  A.err = &w.st->err;
  A.bytes_out = &w.st->delta_bytes;
  A.e_next = &w.st->e_next[phase];
  A.i_next = &w.st->i_next[phase];
  hub_kernels(A, w, phase, cap, ghub, pv, tri, s);
  PhaseEnd E;
  memset(&E, 0, sizeof(E));
  E.st = w.st;
  if (phase) {
    E.slot = w.ins_slot;
    E.n_ins = &w.st->n_ins;
    E.mark = g->mark;
    E.delta = delta;
    E.added = &w.st->tri_added;
    E.removed = &w.st->tri_removed;
  } else {
    E.dlist = w.dlist;
    E.n_del = &w.st->n_del;
    E.cmp = compact_args(g, w);
  }
  k_delta_fused<<<gdelta, kThreads, delta_smem(A), s>>>(A, E, pv, tri);
}

// Working memory of tc_batch_sort. Each device keeps one, used by one call at a time (the call waits
// for its stream before it returns it); a call that finds it taken, or needs more than kSortWsKeep
// bytes, works on memory of its own. Allocating and freeing seven arrays per call took longer than
// sorting the batch (100,000 entries of a graph of 2^20 vertices: 1-10 ms against 0.2 ms).
constexpr size_t kSortWsKeep = (size_t)256 << 20;

struct SortWs {
  int64_t n_cap = -1, b_cap = -1;
  uint64_t *k1 = nullptr, *k2 = nullptr;  // [b]
  void* tmp = nullptr;
  size_t tmp_bytes = 0;
  int32_t* cnt = nullptr;                 // [n + 1]
  int64_t *off64 = nullptr, *tiles = nullptr;
  unsigned* err = nullptr;

  void release() {
    cudaFree(k1); cudaFree(k2); cudaFree(tmp); cudaFree(cnt); cudaFree(off64); cudaFree(tiles); cudaFree(err);
    *this = SortWs();
  }
  size_t bytes() const {
    return 16 * (size_t)std::max<int64_t>(b_cap, 0) + tmp_bytes + 12 * (size_t)std::max<int64_t>(n_cap, 0);
  }
  // n vertices, b entries, and what is held already where both fit; after a failure nothing is held.
  tc_status ensure(int64_t n, int64_t b) {
    if (n <= n_cap && b <= b_cap) return TC_OK;
    const int64_t nn = std::max(n, n_cap), nb = std::max(b, b_cap);
    release();
    if (allocate(nn, nb) || ((nn > n || nb > b) && allocate(n, b))) return TC_OK;
    return fail(TC_ERR_OOM, "batch sort: allocation failed");
  }

 private:
  bool allocate(int64_t nn, int64_t nb) {
    size_t tb = 0;
    const size_t bb = (size_t)std::max<int64_t>(nb, 1);
    const bool ok = ::tc::dev_malloc(&k1, sizeof(uint64_t) * bb) == cudaSuccess &&
                    ::tc::dev_malloc(&k2, sizeof(uint64_t) * bb) == cudaSuccess &&
                    ::tc::dev_malloc(&cnt, sizeof(int32_t) * ((size_t)nn + 1)) == cudaSuccess &&
                    ::tc::dev_malloc(&off64, sizeof(int64_t) * ((size_t)nn + 2)) == cudaSuccess &&
                    ::tc::dev_malloc(&tiles, sizeof(int64_t) * (size_t)(scan_tiles(nn) + 1)) == cudaSuccess &&
                    ::tc::dev_malloc(&err, sizeof(unsigned)) == cudaSuccess &&
                    cub::DeviceRadixSort::SortKeys(nullptr, tb, k1, k2, (int)bb, 0, 64) == cudaSuccess &&
                    ::tc::dev_malloc(&tmp, std::max<size_t>(tb, 1)) == cudaSuccess;
    if (!ok) {
      cudaGetLastError();
      release();
      return false;
    }
    tmp_bytes = tb;
    n_cap = nn;
    b_cap = nb;
    return true;
  }
};

// The kept workspaces and who uses them (not a lock held through the call: the call's own allocations
// may ask for what is kept here).
struct SortWsPool {
  std::mutex mu;
  std::condition_variable given_back;
  bool taken[64] = {};
  SortWs ws[64];
  bool take(int dev, bool wait) {
    std::unique_lock<std::mutex> lk(mu);
    if (wait) given_back.wait(lk, [&] { return !taken[dev]; });
    if (taken[dev]) return false;
    return taken[dev] = true;
  }
  void give_back(int dev) {
    {
      std::lock_guard<std::mutex> lk(mu);
      taken[dev] = false;
    }
    given_back.notify_all();
  }
};
SortWsPool& sort_ws_pool() {
  static SortWsPool* p = new SortWsPool();  // intentionally leaked: outlives CUDA teardown
  return *p;
}

// One call's use of a workspace: the device's, or its own. Unless done() says that the call's work on
// it has ended, leaving waits for the device first.
class SortWsLease {
 public:
  SortWsLease() {
    if (cudaGetDevice(&dev_) != cudaSuccess || dev_ < 0 || dev_ >= 64) dev_ = -1;
    if (dev_ >= 0 && !sort_ws_pool().take(dev_, false)) dev_ = -1;
  }
  ~SortWsLease() {
    if (!done_) cudaDeviceSynchronize();
    SortWs& w = ws();
    if (dev_ < 0 || w.bytes() > kSortWsKeep) w.release();
    if (dev_ >= 0) sort_ws_pool().give_back(dev_);
  }
  SortWsLease(const SortWsLease&) = delete;
  SortWsLease& operator=(const SortWsLease&) = delete;
  SortWs& ws() { return dev_ >= 0 ? sort_ws_pool().ws[dev_] : own_; }
  void done() { done_ = true; }

 private:
  int dev_ = -1;
  bool done_ = false;
  SortWs own_;
};

}  // namespace

bool release_sort_ws(int dev, bool wait) {
  SortWsPool& p = sort_ws_pool();
  if (!p.take(dev, wait)) return false;
  const bool held = p.ws[dev].bytes() > 0;
  p.ws[dev].release();
  p.give_back(dev);
  return held;
}

}  // namespace tc

using namespace tc;

extern "C" {

tc_status tc_apply_batch(tc_graph* g, const int32_t* src, const int32_t* dst, const uint8_t* is_delete, int64_t b,
                         int mem, int32_t* per_vertex, int64_t* delta_dev, tc_batch_info* info, const tc_sched* sched,
                         void* stream) {
  tc::TraceRange trace_range("tc_apply_batch");
  if (!g) return fail(TC_ERR_INVALID_ARG, "graph is NULL");
  if (b < 0 || (b > 0 && (!src || !dst)) || (mem != TC_MEM_HOST && mem != TC_MEM_DEVICE))
    return fail(TC_ERR_INVALID_ARG, "invalid batch arguments");
  if (b > (int64_t)INT32_MAX / 2) return fail(TC_ERR_CAPACITY, "batch of %lld pairs exceeds 2^30", (long long)b);
  cudaStream_t s = (cudaStream_t)stream;
  TC_TRY(ensure_stream_ws(g, b));
  StreamWs& w = *g->sw;
  const SchedParams sp = to_params(sched);
  const int32_t* d_src = src;
  const int32_t* d_dst = dst;
  const uint8_t* d_del = is_delete;
  if (mem == TC_MEM_HOST && b > 0) {
    TC_CUDA_TRY(cudaMemcpyAsync(w.src, src, sizeof(int32_t) * b, cudaMemcpyHostToDevice, s));
    TC_CUDA_TRY(cudaMemcpyAsync(w.dst, dst, sizeof(int32_t) * b, cudaMemcpyHostToDevice, s));
    if (is_delete) TC_CUDA_TRY(cudaMemcpyAsync(w.isdel, is_delete, b, cudaMemcpyHostToDevice, s));
    d_src = w.src;
    d_dst = w.dst;
    d_del = is_delete ? w.isdel : nullptr;
  }
  const int L = bits_for(std::max(g->n, 2));
  // 1. canonical keys, sort, unique + classify
  if (b > 0) {
    TC_CUDA_TRY(load_batch(g, w, d_src, d_dst, d_del, b, b, L, s));
    TC_CUDA_TRY(sort_batch(w, b, L, s));
    TC_CUDA_TRY(classify_and_sort(g, w, b, L, s));
    TC_CUDA_TRY(cudaGetLastError());
  } else {
    TC_CUDA_TRY(cudaMemsetAsync(w.st, 0, sizeof(BatchStatus), s));
  }
  // 2. one synchronisation: sizes and the pool demand
  TC_CUDA_TRY(cudaMemcpyAsync(w.st_host, w.st, sizeof(BatchStatus), cudaMemcpyDeviceToHost, s));
  TC_CUDA_TRY(cudaMemcpyAsync(&w.st_host->pool_top, g->d_pool_top, sizeof(unsigned long long), cudaMemcpyDeviceToHost, s));
  TC_CUDA_TRY(cudaStreamSynchronize(s));
  const BatchStatus h = *w.st_host;
  g->pool_top = (int64_t)h.pool_top;
  if (h.err & kErrRange) return fail(TC_ERR_INVALID_ARG, "batch has vertex ids outside [0, %d)", g->n);
  TC_TRY(ensure_pool(g, (int64_t)h.demand, s));
  uint32_t* pv = reinterpret_cast<uint32_t*>(per_vertex);
  uint32_t* pv_use = pv;
  uint32_t* scratch_pv = nullptr;
  if (!pv_use) {
    // counts only: route per-vertex updates to a scratch array
    if (!g->pv_scratch && ::tc::dev_malloc(&g->pv_scratch, sizeof(uint32_t) * ((size_t)g->n + 1)) != cudaSuccess) {
      g->pv_scratch = nullptr;
      return fail(TC_ERR_OOM, "per-vertex scratch: device allocation failed");
    }
    scratch_pv = reinterpret_cast<uint32_t*>(g->pv_scratch);
    pv_use = scratch_pv;
  }
  int ghub = 0, gdelta = 0;
  TC_TRY(hub_grid(&ghub));
  TC_TRY(fused_grid(0, delta_smem(delta_args(g, sp)), &gdelta));
  // 3. deletions: mark, count on the pre-deletion graph, compact
  if (h.n_del > 0) {
    const int64_t nd = (int64_t)h.n_del;
    k_mark_deletions<<<grid_for(nd, kThreads), kThreads, 0, s>>>(w.dlist, w.st, g->start, g->mark, w.first_del, w.d_epoch);
    delta_phase(g, w, sp, 0, nd, kPipeCand[default_cand(nd)], ghub, gdelta, pv_use, nullptr, kSpinNs, 0, s);
    long_compact(g, w, s);
    TC_CUDA_TRY(cudaGetLastError());
  }
  // 4. insertions: merge into the lists, count on the post-insertion graph, clear marks
  if (h.n_ins > 0) {
    const int64_t ni = (int64_t)h.n_ins;
    insert_sorted_keys(g, w, (int64_t)h.n_runs, L, g->mark, s);
    delta_phase(g, w, sp, 1, ni, kPipeCand[default_cand(ni)], ghub, gdelta, pv_use, nullptr, kSpinNs, 0, s);
    TC_CUDA_TRY(cudaGetLastError());
  }
  g->m += 2 * ((int64_t)h.n_ins - (int64_t)h.n_del);
  g->pool_top += (int64_t)h.demand;  // host bound until the next read of the device counter
  g->view_version++;
  if (delta_dev) k_add_delta<<<1, 32, 0, s>>>(delta_dev, &w.st->tri_added, &w.st->tri_removed);
  if (info) {
    TC_CUDA_TRY(cudaMemcpyAsync(w.st_host, w.st, sizeof(BatchStatus), cudaMemcpyDeviceToHost, s));
    TC_CUDA_TRY(cudaStreamSynchronize(s));
    const BatchStatus& f = *w.st_host;
    if (f.err & (kErrPool | kErrScratch)) return fail(TC_ERR_CAPACITY, "adjacency pool or insertion scratch exhausted");
    if (f.err & kErrTimeout)
      return fail(TC_ERR_TIMEOUT, "a delta kernel's CTAs did not meet in time (the batch is applied and counted)");
    info->updates = b;
    info->inserted = (int64_t)f.n_ins;
    info->deleted = (int64_t)f.n_del;
    info->ignored = b - (int64_t)f.n_ins - (int64_t)f.n_del;
    info->triangles_added = (int64_t)f.tri_added;
    info->triangles_removed = (int64_t)f.tri_removed;
    info->status = TC_OK;
  }
  return TC_OK;
}

tc_status tc_batch_sort(int32_t nv, int32_t* d_src, int32_t* d_dst, int64_t b, int32_t* d_offsets, int32_t* d_dup,
                        void* stream) {
  if (nv < 0 || b < 0 || (b > 0 && (!d_src || !d_dst || !d_dup)) || !d_offsets)
    return fail(TC_ERR_INVALID_ARG, "invalid batch arguments");
  if (b > (int64_t)INT32_MAX / 2) return fail(TC_ERR_CAPACITY, "batch too large");
  cudaStream_t s = (cudaStream_t)stream;
  SortWsLease lease;
  SortWs& w = lease.ws();
  TC_TRY(w.ensure(nv, b));
  unsigned herr = 0;
  TC_CUDA_TRY(cudaMemsetAsync(w.cnt, 0, sizeof(int32_t) * ((size_t)nv + 1), s));
  TC_CUDA_TRY(cudaMemsetAsync(w.err, 0, sizeof(unsigned), s));
  if (b > 0) {
    k_pack_dir<<<grid_for(b, kThreads), kThreads, 0, s>>>(d_src, d_dst, b, w.k1);
    size_t tb = w.tmp_bytes;
    TC_CUDA_TRY(cub::DeviceRadixSort::SortKeys(w.tmp, tb, w.k1, w.k2, (int)b, 0, 64, s));
    k_unpack_dir<<<grid_for(b, kThreads), kThreads, 0, s>>>(w.k2, b, nv, d_src, d_dst, d_dup, w.cnt, w.err);
  }
  TC_TRY(scan_counts(w.cnt, nv, w.off64, w.tiles, s));
  k_to_int32<<<grid_for((int64_t)nv + 1, kThreads), kThreads, 0, s>>>(w.off64, nv, d_offsets);
  TC_CUDA_TRY(cudaGetLastError());
  TC_CUDA_TRY(cudaMemcpyAsync(&herr, w.err, sizeof(unsigned), cudaMemcpyDeviceToHost, s));
  TC_CUDA_TRY(cudaStreamSynchronize(s));  // the working memory is free again
  lease.done();
  if (herr) return fail(TC_ERR_INVALID_ARG, "batch has vertex ids outside [0, %d)", nv);
  return TC_OK;
}

tc_status tc_insert_sorted(tc_graph* g, const int32_t* d_src, const int32_t* d_dst, int64_t b, int32_t* d_dup,
                           int64_t* not_fitting, void* stream) {
  if (!g || b < 0 || (b > 0 && (!d_src || !d_dst || !d_dup))) return fail(TC_ERR_INVALID_ARG, "invalid arguments");
  cudaStream_t s = (cudaStream_t)stream;
  TC_TRY(ensure_stream_ws(g, (b + 1) / 2 + 1));
  StreamWs& w = *g->sw;
  TC_CUDA_TRY(cudaMemsetAsync(w.st, 0, sizeof(BatchStatus), s));
  if (not_fitting) *not_fitting = 0;
  if (b == 0) return TC_OK;
  SlackView view{g->start, g->used, g->pool};
  // entries come sorted by (src, dst): the packed keys of the new ones stay sorted, sentinel
  // elsewhere; sort once more to push the sentinels to the end.
  const int L = bits_for(std::max(g->n, 2));
  k_flag_present<<<grid_for(b, kThreads), kThreads, 0, s>>>(view, d_src, d_dst, d_dup, b, L, w.dk, w.st);
  for (int bits = 2 * L;; ++bits) {
    size_t tb = w.cub_bytes;
    TC_CUDA_TRY(cub::DeviceRadixSort::SortKeys(w.cub_tmp, tb, w.dk, w.dk2, (int)b, 0, bits, s));
    k_dir_runs<<<grid_for(b, kThreads), kThreads, 0, s>>>(w.dk2, b, L, g->used, g->cap, g->slack_q10, w.runs, w.st);
    TC_CUDA_TRY(cudaMemcpyAsync(w.st_host, w.st, sizeof(BatchStatus), cudaMemcpyDeviceToHost, s));
    TC_CUDA_TRY(cudaMemcpyAsync(&w.st_host->pool_top, g->d_pool_top, sizeof(unsigned long long), cudaMemcpyDeviceToHost, s));
    TC_CUDA_TRY(cudaStreamSynchronize(s));
    // The caller says what is a duplicate, so a self-loop can come, and that of the last of 2^L ids has the
    // sentinels' low 2L bits: it may lie apart from its vertex's run. Then once more with one bit more.
    if (!(w.st_host->err & kLastSelfLoop) || bits > 2 * L) break;
    TC_CUDA_TRY(cudaMemsetAsync(w.st, 0, sizeof(BatchStatus), s));
  }
  const BatchStatus h = *w.st_host;
  g->pool_top = (int64_t)h.pool_top;
  TC_TRY(ensure_pool(g, (int64_t)h.demand, s));
  if (h.n_runs > 0) {
    insert_sorted_keys(g, w, (int64_t)h.n_runs, L, nullptr, s);
    TC_CUDA_TRY(cudaGetLastError());
  }
  TC_CUDA_TRY(cudaMemcpyAsync(w.st_host, w.st, sizeof(BatchStatus), cudaMemcpyDeviceToHost, s));
  TC_CUDA_TRY(cudaStreamSynchronize(s));
  if (w.st_host->err & (kErrPool | kErrScratch)) return fail(TC_ERR_CAPACITY, "adjacency pool or insertion scratch exhausted");
  g->m += (int64_t)w.st_host->dir_added;
  g->pool_top += (int64_t)h.demand;  // host bound until the next read of the device counter
  g->view_version++;
  if (not_fitting) *not_fitting = (int64_t)w.st_host->not_fitting;
  return TC_OK;
}

tc_status tc_delete_sorted(tc_graph* g, const int32_t* d_src, const int32_t* d_dst, const int32_t* d_dup, int64_t b,
                           void* stream) {
  if (!g || b < 0 || (b > 0 && (!d_src || !d_dst || !d_dup))) return fail(TC_ERR_INVALID_ARG, "invalid arguments");
  cudaStream_t s = (cudaStream_t)stream;
  TC_TRY(ensure_stream_ws(g, (b + 1) / 2 + 1));
  TC_TRY(ensure_long_scratch(g));
  StreamWs& w = *g->sw;
  TC_CUDA_TRY(cudaMemsetAsync(w.st, 0, sizeof(BatchStatus), s));
  if (b == 0) return TC_OK;
  TC_CUDA_TRY(cudaMemsetAsync(w.counter, 0, sizeof(unsigned long long), s));
  SlackView view{g->start, g->used, g->pool};
  k_mark_dir_deletions<<<grid_for(b, kThreads), kThreads, 0, s>>>(view, d_src, d_dst, d_dup, b, g->mark, w.first_del,
                                                                   w.vlist, w.counter);
  k_bump_epoch<<<1, 32, 0, s>>>(w.d_epoch);
  k_compact<<<grid_for(b * 32, kThreads), kThreads, 0, s>>>(compact_args(g, w), w.vlist, w.counter, w.st);
  long_compact(g, w, s);
  TC_CUDA_TRY(cudaGetLastError());
  TC_CUDA_TRY(cudaMemcpyAsync(w.st_host, w.st, sizeof(BatchStatus), cudaMemcpyDeviceToHost, s));
  TC_CUDA_TRY(cudaStreamSynchronize(s));
  g->m -= (int64_t)w.st_host->dir_removed;
  g->view_version++;
  return TC_OK;
}

tc_status tc_count_batch(tc_graph* g, const int32_t* d_src, const int32_t* d_dst, const int32_t* d_offsets,
                         const int32_t* d_dup, int64_t b, int sign, int32_t* per_vertex, int64_t* delta_dev,
                         const tc_sched* sched, void* stream) {
  tc::TraceRange trace_range("tc_count_batch");
  if (!g || b < 0 || (b > 0 && (!d_src || !d_dst || !d_dup || !d_offsets)) || (sign != 1 && sign != -1) || !per_vertex)
    return fail(TC_ERR_INVALID_ARG, "invalid arguments");
  cudaStream_t s = (cudaStream_t)stream;
  TC_TRY(ensure_stream_ws(g, 1));
  StreamWs& w = *g->sw;
  TC_CUDA_TRY(cudaMemsetAsync(w.counter, 0, sizeof(unsigned long long), s));
  if (b > 0) {
    DeltaArgs A = delta_args(g, to_params(sched));
    A.bl = BatchLists{d_src, d_dst, d_offsets, d_dup};
    A.count_host = b;
    A.sign = sign;
    A.weight = 1;
    A.only_present = sign < 0;
    const PipeCand& shape = kPipeCand[default_cand(b / 2)];
    A.chunk = shape.chunk;
    A.split_min = shape.split_min;
    A.split_items = w.split_items;
    A.split_cnt = &w.st->n_split[0];
    TC_CUDA_TRY(cudaMemsetAsync(A.split_cnt, 0, sizeof(unsigned long long), s));
    k_delta<<<delta_grid(b), kThreads, delta_smem(A), s>>>(A, reinterpret_cast<uint32_t*>(per_vertex),
                                                                     w.counter);
    k_delta_split<<<delta_grid(b), kThreads, delta_smem(A), s>>>(A, reinterpret_cast<uint32_t*>(per_vertex),
                                                                           w.counter);
    TC_CUDA_TRY(cudaGetLastError());
  }
  if (delta_dev) {
    if (sign > 0) k_add_delta<<<1, 32, 0, s>>>(delta_dev, w.counter, nullptr);
    else k_add_delta<<<1, 32, 0, s>>>(delta_dev, nullptr, w.counter);
    TC_CUDA_TRY(cudaGetLastError());
  }
  return TC_OK;
}

}  // extern "C"

// ---- captured streaming pipeline ---------------------------------------------------------------
//
// tc_apply_batch reads the batch's sizes and the pool demand on the host halfway through (one
// synchronisation) and sizes each launch from them. The pipeline below runs the same steps as
// one CUDA graph per batch-size bin instead: every launch is sized for the bin's capacity and
// reads the batch's real counts from device memory (grid-stride loops over device counts, the
// batch padded with sentinel keys), so a batch is one small launch that loads it and its size
// into the bin's buffers (sorted as well where one CTA can) and one graph launch, with no host
// synchronisation inside. The delta count of each phase (deletions, insertions) is one
// persistent kernel (k_delta_fused). The pool headroom the relocations of one batch can take is
// bounded ahead (every touched list moving: (m + 2b)(1 + slack) slots) and reserved before the
// launch, so the device bump allocator cannot run out. The graphs capture the graph's pool and
// workspace pointers and the caller's per-vertex and delta arrays; they are captured again when
// any of these change.
//
// Autotuner (tc_pipeline_autotune): the bins start as a fine ladder of capacities (2^10, 2^11,
// ... up to max_batch). Over the next k batches each batch runs under one "arm" of its natural
// bin (the smallest that holds it): one of the candidate tile shapes of the delta kernel (CTAs
// per SM, split threshold and split-item size) in that bin's graph, or the fastest of them so far in
// the next bin's graph. Each arm's time per update is measured with events, the load of the batch
// included. At the end every bin keeps its fastest shape, and a bin to whose batches the padding adds no
// more than 3 % (merge_bins) is merged into the next one: its threshold is dropped and its batches use
// the graph that serves that bin (fewer graphs where padding costs nothing, the fine ladder where it
// does).

namespace tc {
namespace {
constexpr int kPipeBins = 16;
constexpr int64_t kPipeMinBin = 1 << 10;
}  // namespace
}  // namespace tc

struct tc_pipeline {
  tc_graph* g = nullptr;
  int device = -1;
  int64_t b_max = 0;
  int nbins = 0;
  int64_t bin_cap[tc::kPipeBins] = {};
  int cand[tc::kPipeBins] = {};                      // chosen tile-shape candidate per bin
  int serve[tc::kPipeBins] = {};                     // bin whose graph runs this bin's batches
  cudaGraphExec_t exec[tc::kPipeBins][tc::kPipeCands] = {};
  tc::BinTimes tune[tc::kPipeBins];                  // autotuning: per natural bin
  int tune_left = 0;                                 // batches still spent exploring
  // what the captured graphs hold
  const void* key_pool = nullptr;
  const void* key_mark = nullptr;
  const void* key_pv = nullptr;
  const void* key_delta = nullptr;
  uint64_t key_ws = 0;
  int64_t key_pool_cap = 0;
  tc::SchedParams sp;
  unsigned long long spin_ns = tc::kSpinNs;          // bound of the wait in which the delta kernels' CTAs meet
  unsigned bar_extra = 0;                            // (test hook: arrivals that never come)
  cudaStream_t cs = nullptr;     // capture stream
  tc::BatchStatus* h_st = nullptr;          // pinned: status of the last batch
  unsigned long long* h_top = nullptr;      // pinned: pool bump pointer after it
  uint32_t* pv_scratch = nullptr;
  int64_t* delta_scratch = nullptr;
  cudaEvent_t done = nullptr, t0 = nullptr, t1 = nullptr;
  cudaEvent_t pev[4] = {};       // profiling: around the two delta kernels, inside the graphs
  bool profile = false;
  int64_t prof_batches = 0;
  double prof_delta_ms = 0.0;
  int64_t prof_delta_bytes = 0;
  bool pending = false;
  int pending_bin = -1, pending_cand = -1, pending_arm = -1, pending_nat = -1;
  int64_t pending_b = 0;
  bool timing = false;
  tc_batch_info last{};
};

namespace tc {
namespace {

void drop_graphs(tc_pipeline* p) {
  for (int i = 0; i < kPipeBins; ++i)
    for (int j = 0; j < kPipeCands; ++j)
      if (p->exec[i][j]) {
        cudaGraphExecDestroy(p->exec[i][j]);
        p->exec[i][j] = nullptr;
      }
}

// Fold the finished batch's device status into the host view of the graph.
tc_status pipe_settle(tc_pipeline* p) {
  if (!p->pending) return TC_OK;
  TC_CUDA_TRY(cudaEventSynchronize(p->done));
  p->pending = false;
  tc_graph* g = p->g;
  const BatchStatus& f = *p->h_st;
  g->pool_top = (int64_t)*p->h_top;
  g->m += 2 * ((int64_t)f.n_ins - (int64_t)f.n_del);
  g->view_version++;
  p->last.updates = p->pending_b;
  p->last.inserted = (int64_t)f.n_ins;
  p->last.deleted = (int64_t)f.n_del;
  p->last.ignored = p->pending_b - (int64_t)f.n_ins - (int64_t)f.n_del;
  p->last.triangles_added = (int64_t)f.tri_added;
  p->last.triangles_removed = (int64_t)f.tri_removed;
  p->last.status = TC_OK;
  if (p->timing) {
    float ms = 0.f;
    TC_CUDA_TRY(cudaEventElapsedTime(&ms, p->t0, p->t1));
    p->tune[p->pending_nat].add(p->pending_arm, ms, p->pending_b);
    p->timing = false;
  }
  if (p->profile && p->prof_delta_ms >= 0.0) {
    // a failed read (no event recorded by the graph) turns the profile off, not the batch
    float d0 = 0.f, d1 = 0.f;
    if (cudaEventElapsedTime(&d0, p->pev[0], p->pev[1]) != cudaSuccess ||
        cudaEventElapsedTime(&d1, p->pev[2], p->pev[3]) != cudaSuccess) {
      cudaGetLastError();
      p->prof_delta_ms = -1.0;
    } else {
      p->prof_batches += 1;
      p->prof_delta_ms += (double)d0 + (double)d1;
      p->prof_delta_bytes += (int64_t)f.delta_bytes;
    }
  }
  if (f.err & kErrRange) {
    p->last.status = TC_ERR_INVALID_ARG;
    return fail(TC_ERR_INVALID_ARG, "batch had vertex ids outside [0, %d); they were ignored", g->n);
  }
  if (f.err & (kErrPool | kErrScratch)) {
    p->last.status = TC_ERR_CAPACITY;
    return fail(TC_ERR_CAPACITY, "adjacency pool or insertion scratch exhausted");
  }
  if (f.err & kErrTimeout) {
    p->last.status = TC_ERR_TIMEOUT;
    return fail(TC_ERR_TIMEOUT, "a delta kernel's CTAs did not meet in time (the batch is applied and counted)");
  }
  return TC_OK;
}

int64_t pipe_worst_demand(const tc_graph* g, int64_t b) {
  const int64_t q = std::max<int64_t>(g->slack_q10, 256);
  return ((g->m + 2 * b) * (1024 + q) + 1023) / 1024 + 16 * b + 64;
}

// Drop the captured graphs when what they hold (pool, marks, workspace, outputs) has changed.
void pipe_check_keys(tc_pipeline* p, const void* pv, const void* delta) {
  tc_graph* g = p->g;
  const StreamWs& w = *g->sw;
  if (p->key_pool != g->pool || p->key_mark != g->mark || p->key_pv != pv || p->key_delta != delta ||
      p->key_ws != w.version || p->key_pool_cap != g->pool_cap) {
    drop_graphs(p);
    p->key_pool = g->pool;
    p->key_mark = g->mark;
    p->key_pv = pv;
    p->key_delta = delta;
    p->key_ws = w.version;
    p->key_pool_cap = g->pool_cap;
  }
}

// Record the whole batch pipeline for a bin of capacity cap, with tile shape `cand`, on the
// capture stream.
tc_status pipe_capture(tc_pipeline* p, int bin, int cand, uint32_t* pv, int64_t* delta) {
  tc_graph* g = p->g;
  StreamWs& w = *g->sw;
  const int64_t cap = p->bin_cap[bin];
  const PipeCand& pc = kPipeCand[cand];
  cudaStream_t s = p->cs;
  const int L = bits_for(std::max(g->n, 2));
  int gdelta = 0, ghub = 0;
  TC_TRY(fused_grid(pc.ctas, delta_smem(delta_args(g, p->sp)), &gdelta));
  TC_TRY(hub_grid(&ghub));
  cudaGraph_t graph = nullptr;
  TC_CUDA_TRY(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
  cudaError_t e = cudaSuccess;
  do {
    if ((e = sort_batch(w, cap, L, s)) != cudaSuccess) break;
    if ((e = classify_and_sort(g, w, cap, L, s)) != cudaSuccess) break;
    // deletions: mark, count on the pre-deletion graph, compact
    k_mark_deletions<<<grid_for(cap, kThreads), kThreads, 0, s>>>(w.dlist, w.st, g->start, g->mark, w.first_del,
                                                                  w.d_epoch);
    if (p->profile) cudaEventRecordWithFlags(p->pev[0], s, cudaEventRecordExternal);
    delta_phase(g, w, p->sp, 0, cap, pc, ghub, gdelta, pv, nullptr, p->spin_ns, p->bar_extra, s);
    if (p->profile) cudaEventRecordWithFlags(p->pev[1], s, cudaEventRecordExternal);
    long_compact(g, w, s);
    // insertions: merge, count on the post-insertion graph, clear the marks
    insert_sorted_keys(g, w, 2 * cap, L, g->mark, s);
    if (p->profile) cudaEventRecordWithFlags(p->pev[2], s, cudaEventRecordExternal);
    delta_phase(g, w, p->sp, 1, cap, pc, ghub, gdelta, pv, delta, p->spin_ns, p->bar_extra, s);
    if (p->profile) cudaEventRecordWithFlags(p->pev[3], s, cudaEventRecordExternal);
    cudaMemcpyAsync(p->h_st, w.st, sizeof(BatchStatus), cudaMemcpyDeviceToHost, s);
    cudaMemcpyAsync(p->h_top, g->d_pool_top, sizeof(unsigned long long), cudaMemcpyDeviceToHost, s);
    e = cudaGetLastError();
  } while (0);
  const cudaError_t e2 = cudaStreamEndCapture(s, &graph);
  if (e == cudaSuccess) e = e2;
  if (e == cudaSuccess) e = cudaGraphInstantiate(&p->exec[bin][cand], graph, 0);
  if (graph) cudaGraphDestroy(graph);
  if (e != cudaSuccess) {
    p->exec[bin][cand] = nullptr;
    return fail(TC_ERR_CUDA, "pipeline capture: %s", cudaGetErrorString(e));
  }
  return TC_OK;
}

// End of the exploration: the fastest shape per bin, then the merges (top bin down, so a chain
// of merged bins resolves to the graph that serves the highest of them).
void pipe_finish_tuning(tc_pipeline* p) {
  for (int i = 0; i < p->nbins; ++i) p->cand[i] = p->tune[i].best(p->cand[i]);
  merge_bins(p->tune, p->nbins, p->serve);
}

int pipe_natural_bin(const tc_pipeline* p, int64_t b) {
  int bin = 0;
  while (bin + 1 < p->nbins && p->bin_cap[bin] < b) ++bin;
  return bin;
}

}  // namespace
}  // namespace tc

extern "C" {

tc_status tc_pipeline_create(tc_graph* g, int64_t max_batch, const tc_sched* sched, tc_pipeline** out) {
  if (!g || !out || max_batch < 1) return fail(TC_ERR_INVALID_ARG, "invalid pipeline arguments");
  if (max_batch > (int64_t)INT32_MAX / 4) return fail(TC_ERR_CAPACITY, "pipeline batch capacity exceeds 2^29");
  *out = nullptr;
  tc_pipeline* p = new tc_pipeline();
  p->g = g;
  p->sp = to_params(sched);
  TC_CUDA_TRY(cudaGetDevice(&p->device));
  // fine ladder: 2^10, 2^11, ... (the last bin holds max_batch; past kPipeBins bins the ladder
  // doubles its step)
  int64_t step = 2;
  {
    int64_t levels = 1;
    for (int64_t c = kPipeMinBin; c < max_batch; c *= 2) ++levels;
    while (levels > kPipeBins) {
      step *= 2;
      levels = (levels + 1) / 2;
    }
  }
  for (int64_t c = kPipeMinBin; p->nbins < kPipeBins; c *= step) {
    p->bin_cap[p->nbins++] = std::min(c, std::max(max_batch, kPipeMinBin));
    if (c >= max_batch) break;
  }
  p->b_max = p->bin_cap[p->nbins - 1];
  for (int i = 0; i < kPipeBins; ++i) {
    p->cand[i] = i < p->nbins ? default_cand(p->bin_cap[i]) : 0;
    p->serve[i] = i;
  }
  tc_status rc = TC_OK;
  do {
    if ((rc = ensure_stream_ws(g, p->b_max)) != TC_OK) break;
    if (cudaStreamCreateWithFlags(&p->cs, cudaStreamNonBlocking) != cudaSuccess ||
        cudaMallocHost(&p->h_st, sizeof(BatchStatus)) != cudaSuccess ||
        cudaMallocHost(&p->h_top, sizeof(unsigned long long)) != cudaSuccess ||
        ::tc::dev_malloc(&p->pv_scratch, sizeof(uint32_t) * ((size_t)g->n + 1)) != cudaSuccess ||
        ::tc::dev_malloc(&p->delta_scratch, sizeof(int64_t)) != cudaSuccess ||
        cudaEventCreate(&p->done) != cudaSuccess || cudaEventCreate(&p->t0) != cudaSuccess ||
        cudaEventCreate(&p->t1) != cudaSuccess || cudaEventCreate(&p->pev[0]) != cudaSuccess ||
        cudaEventCreate(&p->pev[1]) != cudaSuccess || cudaEventCreate(&p->pev[2]) != cudaSuccess ||
        cudaEventCreate(&p->pev[3]) != cudaSuccess) {
      rc = fail(TC_ERR_OOM, "pipeline: allocation failed");
      break;
    }
    if (cudaMemset(p->pv_scratch, 0, sizeof(uint32_t) * ((size_t)g->n + 1)) != cudaSuccess ||
        cudaMemset(p->delta_scratch, 0, sizeof(int64_t)) != cudaSuccess)
      rc = fail(TC_ERR_CUDA, "pipeline: set-up failed");
  } while (0);
  if (rc != TC_OK) {
    tc_pipeline_destroy(p);
    return rc;
  }
  *out = p;
  return TC_OK;
}

tc_status tc_pipeline_destroy(tc_pipeline* p) {
  if (!p) return TC_OK;
  if (p->pending) cudaEventSynchronize(p->done);
  drop_graphs(p);
  if (p->cs) cudaStreamDestroy(p->cs);
  cudaFreeHost(p->h_st);
  cudaFreeHost(p->h_top);
  cudaFree(p->pv_scratch);
  cudaFree(p->delta_scratch);
  if (p->done) cudaEventDestroy(p->done);
  if (p->t0) cudaEventDestroy(p->t0);
  if (p->t1) cudaEventDestroy(p->t1);
  for (int i = 0; i < 4; ++i)
    if (p->pev[i]) cudaEventDestroy(p->pev[i]);
  delete p;
  return TC_OK;
}

tc_status tc_pipeline_apply(tc_pipeline* p, const int32_t* d_src, const int32_t* d_dst, const uint8_t* d_is_delete,
                            int64_t b, int32_t* per_vertex, int64_t* delta_dev, void* stream) {
  tc::TraceRange trace_range("tc_pipeline_apply");
  if (!p || b < 0 || (b > 0 && (!d_src || !d_dst))) return fail(TC_ERR_INVALID_ARG, "invalid batch arguments");
  if (b > p->b_max)
    return fail(TC_ERR_CAPACITY, "batch of %lld updates exceeds the pipeline's %lld", (long long)b,
                (long long)p->b_max);
  int dev = 0;
  TC_CUDA_TRY(cudaGetDevice(&dev));
  if (dev != p->device) return fail(TC_ERR_INVALID_ARG, "pipeline used on device %d, created on %d", dev, p->device);
  TC_TRY(pipe_settle(p));
  tc_graph* g = p->g;
  cudaStream_t s = (cudaStream_t)stream;
  if (b == 0) return TC_OK;
  // Headroom for the worst case: every list the batch touches moves to the pool top.
  const int64_t worst = pipe_worst_demand(g, b);
  if (g->pool_cap - g->pool_top < worst) TC_TRY(ensure_pool(g, worst + worst / 2, s));
  TC_TRY(ensure_stream_ws(g, p->b_max));
  TC_TRY(ensure_long_scratch(g));
  uint32_t* pv = per_vertex ? reinterpret_cast<uint32_t*>(per_vertex) : p->pv_scratch;
  int64_t* delta = delta_dev ? delta_dev : p->delta_scratch;
  StreamWs& w = *g->sw;
  pipe_check_keys(p, pv, delta);
  const int nat = pipe_natural_bin(p, b);
  int bin = p->serve[nat];
  int cand = p->cand[bin];
  int arm = -1;
  if (p->tune_left > 0) {
    // explore: the arm of this natural bin with the fewest samples
    arm = p->tune[nat].next(nat + 1 < p->nbins ? kPipeArms : kPipeCands);
    bin = arm < kPipeCands ? nat : nat + 1;
    cand = arm < kPipeCands ? arm : p->tune[nat].best(p->cand[nat]);
  }
  if (!p->exec[bin][cand]) TC_TRY(pipe_capture(p, bin, cand, pv, delta));
  p->timing = false;
  if (arm >= 0) TC_CUDA_TRY(cudaEventRecord(p->t0, s));
  // the batch's keys, padded to the bin's capacity, where the graph reads them
  TC_CUDA_TRY(load_batch(g, w, d_src, d_dst, d_is_delete, b, p->bin_cap[bin], bits_for(std::max(g->n, 2)), s));
  TC_CUDA_TRY(cudaGraphLaunch(p->exec[bin][cand], s));
  if (arm >= 0) TC_CUDA_TRY(cudaEventRecord(p->t1, s));
  p->timing = arm >= 0;
  TC_CUDA_TRY(cudaEventRecord(p->done, s));
  p->pending = true;
  p->pending_bin = bin;
  p->pending_cand = cand;
  p->pending_arm = arm;
  p->pending_nat = nat;
  p->pending_b = b;
  if (p->tune_left > 0 && --p->tune_left == 0) {
    // exploration over: settle the last sample, keep the fastest shape per bin, merge bins
    TC_TRY(pipe_settle(p));
    pipe_finish_tuning(p);
  }
  return TC_OK;
}

tc_status tc_pipeline_prepare(tc_pipeline* p, int32_t* per_vertex, int64_t* delta_dev, void* stream) {
  if (!p) return fail(TC_ERR_INVALID_ARG, "pipeline is NULL");
  TC_TRY(pipe_settle(p));
  tc_graph* g = p->g;
  const int64_t worst = pipe_worst_demand(g, p->b_max);
  if (g->pool_cap - g->pool_top < worst) TC_TRY(ensure_pool(g, 2 * worst, (cudaStream_t)stream));
  TC_TRY(ensure_stream_ws(g, p->b_max));
  TC_TRY(ensure_long_scratch(g));
  uint32_t* pv = per_vertex ? reinterpret_cast<uint32_t*>(per_vertex) : p->pv_scratch;
  int64_t* delta = delta_dev ? delta_dev : p->delta_scratch;
  pipe_check_keys(p, pv, delta);
  for (int i = 0; i < p->nbins; ++i) {
    const int bin = p->serve[i];
    if (!p->exec[bin][p->cand[bin]]) TC_TRY(pipe_capture(p, bin, p->cand[bin], pv, delta));
  }
  return TC_OK;
}

tc_status tc_pipeline_sync(tc_pipeline* p, tc_batch_info* last) {
  if (!p) return fail(TC_ERR_INVALID_ARG, "pipeline is NULL");
  TC_TRY(pipe_settle(p));
  if (last) *last = p->last;
  return TC_OK;
}

tc_status tc_pipeline_autotune(tc_pipeline* p, int32_t batches) {
  if (!p || batches < 0) return fail(TC_ERR_INVALID_ARG, "invalid autotune arguments");
  TC_TRY(pipe_settle(p));
  for (int i = 0; i < kPipeBins; ++i) {
    p->tune[i] = BinTimes();
    p->serve[i] = i;
  }
  p->tune_left = batches;
  return TC_OK;
}

tc_status tc_pipeline_info(const tc_pipeline* p, int32_t* nbins, int64_t* bin_cap, int32_t* delta_blocks_per_sm) {
  if (!p) return fail(TC_ERR_INVALID_ARG, "pipeline is NULL");
  if (nbins) *nbins = p->nbins;
  for (int i = 0; i < p->nbins; ++i) {
    const int bin = p->serve[i];
    if (bin_cap) bin_cap[i] = p->bin_cap[i];
    if (delta_blocks_per_sm) {
      int grid = 0;
      if (fused_grid(kPipeCand[p->cand[bin]].ctas, delta_smem(delta_args(p->g, p->sp)), &grid) != TC_OK)
        return TC_ERR_CUDA;
      delta_blocks_per_sm[i] = grid / device_info().sms;
    }
  }
  return TC_OK;
}

tc_status tc_pipeline_plan_get(const tc_pipeline* p, tc_pipeline_plan* plan) {
  if (!p || !plan) return fail(TC_ERR_INVALID_ARG, "invalid arguments");
  memset(plan, 0, sizeof(*plan));
  plan->nbins = p->nbins;
  for (int i = 0; i < p->nbins; ++i) {
    const PipeCand& c = kPipeCand[p->cand[p->serve[i]]];
    plan->bin_cap[i] = p->bin_cap[i];
    plan->serve[i] = p->serve[i];
    plan->ctas_per_sm[i] = c.ctas;
    plan->chunk[i] = c.chunk;
    plan->split_min[i] = c.split_min;
  }
  return TC_OK;
}

tc_status tc_pipeline_plan_set(tc_pipeline* p, const tc_pipeline_plan* plan) {
  if (!p || !plan) return fail(TC_ERR_INVALID_ARG, "invalid arguments");
  if (plan->nbins != p->nbins) return fail(TC_ERR_INVALID_ARG, "plan has %d bins, the pipeline %d", plan->nbins, p->nbins);
  int cand[kPipeBins], serve[kPipeBins];
  for (int i = 0; i < p->nbins; ++i) {
    if (plan->bin_cap[i] != p->bin_cap[i]) return fail(TC_ERR_INVALID_ARG, "plan bin %d capacity differs", i);
    if (plan->serve[i] < i || plan->serve[i] >= p->nbins || (i > 0 && plan->serve[i] < plan->serve[i - 1]))
      return fail(TC_ERR_INVALID_ARG, "plan bin %d is served by bin %d", i, plan->serve[i]);
    cand[i] = -1;
    for (int j = 0; j < kPipeCands; ++j)
      if (kPipeCand[j].ctas == plan->ctas_per_sm[i] && kPipeCand[j].chunk == plan->chunk[i] &&
          kPipeCand[j].split_min == plan->split_min[i])
        cand[i] = j;
    if (cand[i] < 0) return fail(TC_ERR_INVALID_ARG, "plan bin %d: tile shape is not one of the candidates", i);
    serve[i] = plan->serve[i];
  }
  TC_TRY(pipe_settle(p));
  for (int i = 0; i < p->nbins; ++i) {
    p->serve[i] = serve[i];
    p->cand[serve[i]] = cand[i];
  }
  p->tune_left = 0;
  return TC_OK;
}

tc_status tc_pipeline_profile(tc_pipeline* p, int on) {
  if (!p) return fail(TC_ERR_INVALID_ARG, "pipeline is NULL");
  TC_TRY(pipe_settle(p));
  if ((on != 0) != p->profile) drop_graphs(p);  // the event records live inside the graphs
  p->profile = on != 0;
  p->prof_batches = 0;
  p->prof_delta_ms = 0.0;
  p->prof_delta_bytes = 0;
  return TC_OK;
}

tc_status tc_pipeline_stats(tc_pipeline* p, int64_t* batches, double* delta_ms, int64_t* delta_bytes) {
  if (!p) return fail(TC_ERR_INVALID_ARG, "pipeline is NULL");
  TC_TRY(pipe_settle(p));
  if (batches) *batches = p->prof_batches;
  if (delta_ms) *delta_ms = p->prof_delta_ms;
  if (delta_bytes) *delta_bytes = p->prof_delta_bytes;
  return TC_OK;
}

tc_status tc_pipeline_set_wait_bound(tc_pipeline* p, uint64_t wait_ns, int32_t extra_arrivals) {
  if (!p || wait_ns == 0 || extra_arrivals < 0) return fail(TC_ERR_INVALID_ARG, "invalid wait bound");
  TC_TRY(pipe_settle(p));
  p->spin_ns = wait_ns;
  p->bar_extra = (unsigned)extra_arrivals;
  drop_graphs(p);  // the bound is an argument of the captured launches
  return TC_OK;
}

}  // extern "C"
