// Static triangle count: degree orientation + vertex-grouped intersections (sm_100a).
//
// Replaces the reference's devicecuStingerAllTriangles (src/static_triangle_counting/cct.cu:216-270)
// and count_all_trianglesGPU (tests/cct_csr.cu:228-276). The reference intersects the full
// lists of every directed edge with a merge path split across 1-32 lanes and one block
// reduction per source vertex. Here:
//
//  1. Orientation (one pass). k_find_hubs registers the vertices with more than kHubMin = 256
//     neighbours (hubs); k_orient then builds the degree orientation G+ (u -> v iff
//     (deg u, u) < (deg v, v)) in the input's own index space: N+(u) is written, ascending by
//     id, at indp[start(u) ...], so no offsets scan is needed. Every triangle {x < y < z in
//     that order} is found exactly once: at x, on edge x->y, as the common element z of N+(x)
//     and N+(y). Warps take hub chunks of up to 2048 entries from one queue (the warp that
//     finishes a hub's last chunk moves the pieces together), then tiles of up to 32 vertex ids from
//     another, walking a tile's concatenated lists (at most 32 x 256 entries), so neither a
//     degree-64k hub nor a run of low-id vertices of degree 2000 (R-MAT) is one warp's serial
//     tail. The same pass
//     checks the input (ids in range, strictly ascending lists, no self-loops, a signed edge
//     checksum for symmetry) and fills the work queues of the count.
//  2. Counting. Every edge {c, o} is intersected once, at its centre c: the endpoint with the
//     larger out-degree (ties to the smaller id). The centre's N+(c) is a shared-memory hash set
//     with two possible slots per key; the other list N+(o), the shorter one, goes through it, so the probe
//     work is the sum over edges of min(d+u, d+v). k_count is a persistent grid; a centre walks
//     its original neighbour list N(c) in groups of 32 and takes the neighbours it is centre
//     for. Tiers by a = d+(c):
//       CTA   a > warp_max: one CTA per item of up to 4096 neighbours, N+(c) staged in a 2048-slot
//             table in passes of at most 768 entries split evenly; a pass holds a value range of
//             N+(c), and each streamed list is cut to that range by binary search, so no list
//             entry is probed twice;
//       warp  1 <= a <= warp_max (at most 128): one warp per centre (items of up to 256 neighbours
//             for centres with more), a warp-private set of up to 512 slots.
//     CTAs of 4 warps, 10 resident per SM (48 registers, 16.5 KB of shared memory each).
//     Per edge, the warp streams N+(o) with coalesced loads (four per lane in flight); or, for
//     short lists, one lane walks it while the other lanes walk theirs; or, for mid-size lists,
//     several such lists are walked at once by a few lanes each (packed); the scheduler
//     (thresholds or learned per-degree-cell table) picks.
//  3. Attribution. Per-vertex counts never take a global atomic per triangle: the centre's count
//     stays in registers, the other endpoint's is reduced once per list (one redux.sync), and
//     the third vertex's is a shared-memory counter beside the hash slot that the probe found;
//     they flush with at most one global atomic per edge or staged entry. The triangle total
//     takes one global atomic per CTA.
#include <algorithm>
#include <climits>
#include <cstring>

#include "tc_internal.cuh"

#ifdef TC_DEBUG_PROGRESS
extern "C" void* tc_dbg_progress_host_dev;
extern "C" size_t tc_dbg_progress_bytes;
#endif

namespace tc {

namespace {

constexpr int kThreads = 128;      // 4 warps: a CTA's warps wait for one another at each item's end
                                   // (256 threads on the same table: 6 % slower on R-MAT 20)
constexpr int kWarps = kThreads / kWarp;
constexpr int kCtasPerSm = 10;     // k_count: 48 registers a thread, 56 to 80 bytes of them spilled with
                                   // per-vertex output (12 CTAs at 40 spill more: R-MAT 24 + 19 %,
                                   // BA n = 2^22 + 24 %; 8 CTAs: R-MAT 20 + 8 %)
constexpr int kHashMaxBits = 11;
constexpr int kHashMax = 1 << kHashMaxBits;  // hash slots of the CTA tier's table
constexpr int kChunk = 768;        // entries of N+(c) staged per pass (load <= 3/8)
constexpr int kWarpSlots = kHashMax / kWarps;  // of a warp-private table (load <= 0.25)
static_assert(kWarpSlots >= 4 * kWarpTierMax, "load of the warp tables");
constexpr int kTableBytes = 2 * 4 * kHashMax;  // keys and counters
constexpr int kUnroll = 4;         // list elements a lane loads before probing (independent loads)
constexpr int kScanThreads = 256;
constexpr int kScanPer = 8;
constexpr int kScanTile = kScanThreads * kScanPer;

#ifdef TC_DEBUG_PROGRESS
// Debug builds only: per-warp progress words and per-kernel entry/exit counters in host-mapped
// memory, readable while a kernel runs.
__device__ unsigned long long* tc_dbg_progress = nullptr;
__device__ unsigned long long* tc_dbg_kern = nullptr;
#define TC_DBG_MARK(idx, val)                                                              \
  do {                                                                                     \
    if (tc_dbg_progress) ((volatile unsigned long long*)tc_dbg_progress)[(idx)] = (val);  \
  } while (0)
#define TC_DBG_ENTER(id)                                                                     \
  do {                                                                                       \
    if (tc_dbg_kern && threadIdx.x == 0) atomicAdd_system(&tc_dbg_kern[2 * (id)], 1ull);      \
  } while (0)
#define TC_DBG_EXIT(id)                                                                      \
  do {                                                                                       \
    if (tc_dbg_kern && threadIdx.x == 0) atomicAdd_system(&tc_dbg_kern[2 * (id) + 1], 1ull);  \
  } while (0)
#else
#define TC_DBG_MARK(idx, val) \
  do {                        \
  } while (0)
#define TC_DBG_ENTER(id) \
  do {                   \
  } while (0)
#define TC_DBG_EXIT(id) \
  do {                  \
  } while (0)
#endif

// Hash sets of staged entries of N+(c): every entry sits at one of its two slots (cuckoo hashing, one
// slot in each half of the table, both from one multiplicative hash), so a lookup reads two 4-byte
// slots and compares twice, with no loop and no divergence. The third-vertex counter of an entry
// sits beside its slot: cnt[s] counts the triangles found through the key keys[s], so a hit adds
// to the slot it found with no indirection. A build that finds no place for an entry in kKicks
// moves fails (at these loads that takes ids chosen against the hash), and the caller stages half
// as many entries; two entries always fit. A list that repeats an id is refused (kBadOrder), but only
// once the count is done, so repeats must not fail builds: an entry that meets its like is dropped.
//
// The kernel is bound by the instructions around each lookup and by the shared-memory pipe. On R-MAT
// 20 (1.97 G lookups, 2 t(v) per vertex): 16-byte buckets of four slots, 62 warp instructions per
// 32 lookups, 4.46 ms; one 4-byte slot with a scan past collisions, which some lane of nearly every
// row takes, 4.4 ms; two slots 2.65 G instructions and 632 M shared wavefronts, 3.19 ms (total only:
// 3.87 -> 2.61 ms; CSR weights: 5.39 -> 3.66 ms). R-MAT 24: 180 -> 124 ms for the whole count.
constexpr int32_t kFreeSlot = -1;
constexpr int32_t kNoKey = -2;  // an entry that is not there: equals no slot's key
constexpr int kKicks = 64;

// Dynamic shared memory of k_count: the tables, then CountSmem. Tables are addressed by 32-bit
// shared addresses and read and updated with inline ld.shared / red.shared, so that a slot's address
// is 32-bit arithmetic on the hash.
constexpr int kWarpTableBytes = kTableBytes / kWarps;
extern __shared__ __align__(16) unsigned char smem_raw[];

struct CountSmem {
  unsigned long long tri[kWarps];
  unsigned long long item;
  int gctr;
  // Value range [vlo, vhi) of the CTA-tier pass in flight when its centre takes several passes
  // (ranged = 1; 0 for a centre of one pass). Only the CTA tier reads them.
  int ranged;
  int32_t vlo, vhi;
};
constexpr size_t kCountSmem = kTableBytes + sizeof(CountSmem);

__device__ __forceinline__ uint32_t table_base() {
  uint32_t base;  // volatile, so that it is computed once
  asm volatile("mov.u32 %0, %1;" : "=r"(base) : "r"((uint32_t)__cvta_generic_to_shared(smem_raw)));
  return base;
}
__device__ __forceinline__ int32_t lds(const uint32_t at) {
  int32_t v;
  asm volatile("ld.shared.s32 %0, [%1];" : "=r"(v) : "r"(at));
  return v;
}
__device__ __forceinline__ int4 lds4(const uint32_t at) {
  int4 v;
  asm volatile("ld.shared.v4.s32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(at));
  return v;
}
__device__ __forceinline__ void sts4(const uint32_t at, const int32_t v) {
  asm volatile("st.shared.v4.s32 [%0], {%1, %1, %1, %1};" ::"r"(at), "r"(v) : "memory");
}
__device__ __forceinline__ int32_t exchange(const uint32_t at, const int32_t v) {
  int32_t old;
  asm volatile("atom.shared.exch.b32 %0, [%1], %2;" : "=r"(old) : "r"(at), "r"(v) : "memory");
  return old;
}
__device__ __forceinline__ int lane_id() {
  int lane;
  asm volatile("mov.u32 %0, %%laneid;" : "=r"(lane));
  return lane;
}

__device__ __forceinline__ unsigned lanemask_lt() {
  unsigned r;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(r));
  return r;
}

__device__ __forceinline__ uint64_t sym_hash(uint32_t x, uint32_t y) {
  uint64_t z = ((uint64_t)x << 32) | y;
  z += 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

template <typename T>
__device__ __forceinline__ T warp_sum(T x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(kFull, x, o);
  return x;
}

// A set of 2 * 2^bits slots, 2^bits in each half, at the shared address keys; its counters lie kCnt
// bytes after its keys.
template <int kCnt>
struct Set {
  uint32_t keys;
  int bits;
  __device__ __forceinline__ int slots() const { return 2 << bits; }
  // Addresses of the two slots of a key: the top bits of its hash, and the next ones in the upper
  // half.
  __device__ __forceinline__ uint32_t slot1(const uint32_t h) const { return ((h >> (30 - bits)) & ~3u) + keys; }
  __device__ __forceinline__ uint32_t slot2(const uint32_t h) const {
    return ((h >> (30 - 2 * bits)) & ((4u << bits) - 4u)) + (keys + (4u << bits));
  }
};
using CtaSet = Set<kHashMax * 4>;
using WarpSet = Set<kWarpSlots * 4>;

__device__ __forceinline__ uint32_t hash_of(const int32_t key) { return (uint32_t)key * 0x9E3779B1u; }

// Insert a key (concurrently with others): into its first slot, the key found there into its other
// one, and so on; false when a key is left over after kKicks moves.
template <class S>
__device__ __forceinline__ bool insert(const S& t, int32_t key) {
  uint32_t at = t.slot1(hash_of(key));
  for (int it = 0; it < kKicks; ++it) {
    const int32_t old = exchange(at, key);
    if (old == kFreeSlot || old == key) return true;
    key = old;
    const uint32_t h = hash_of(key), s1 = t.slot1(h);
    at = at == s1 ? t.slot2(h) : s1;
  }
  return false;
}

// Free slots and zero counters, by `threads` threads of index `at`.
template <int kCnt>
__device__ __forceinline__ void clear_set(const Set<kCnt>& t, const int at, const int threads) {
  for (int s = at; s < t.slots() / 4; s += threads) {
    sts4(t.keys + 16 * s, kFreeSlot);
    sts4(t.keys + kCnt + 16 * s, 0);
  }
}

// Add x to the shared counter at `at` where `take` holds.
__device__ __forceinline__ void count_if(const bool take, const uint32_t at, const uint32_t x) {
  asm volatile("{ .reg .pred p; setp.ne.u32 p, %0, 0; @p red.shared.add.u32 [%1], %2; }" ::"r"((unsigned)take),
               "r"(at), "r"(x));
}

__device__ __forceinline__ int log2_cell(int x) {
  const int c = 31 - __clz(max(x, 1));
  return min(c, 15);
}

// Weights of a found triangle in the per-vertex output. Handle conventions: 1 per vertex, doubled
// at flush (out = 2 t(v)). TC_PV_CSR: the reference's raw-CSR kernel counts a triangle at every
// edge (x, y) with y > x whose lists share the third vertex, crediting x: the smallest id gets 2,
// the middle 1.
template <int PV>
__host__ __device__ constexpr uint32_t flush_mult() {
  return PV == TC_PV_HANDLE || PV == TC_PV_HANDLE64 ? 2u : 1u;
}

// Handle conventions (every triangle weighs 1 per vertex, doubled at flush): int32 or int64 output.
template <int PV>
__host__ __device__ constexpr bool handle_like() {
  return PV == TC_PV_HANDLE || PV == TC_PV_HANDLE64;
}

// Flush x triangles (weights) of vertex v into the per-vertex output: int32 entries, or int64
// entries for TC_PV_HANDLE64 (the output pointer then addresses int64[nv]).
template <int PV>
__device__ __forceinline__ void out_add(uint32_t* __restrict__ out, const int32_t v, const uint32_t x) {
  if (PV == TC_PV_HANDLE64)
    atomicAdd(reinterpret_cast<unsigned long long*>(out) + v, (unsigned long long)x * flush_mult<PV>());
  else
    atomicAdd(out + v, x * flush_mult<PV>());
}

// Is the edge {c, o} intersected at c? At the endpoint with the larger out-degree (its list is
// the hash set, the other one is streamed), ties to the smaller id. Both endpoints read the same
// dplus values, so exactly one of them takes the edge.
__device__ __forceinline__ bool centre_of(int32_t c, int a, int32_t o, int b) {
  return b < a || (b == a && c < o);
}

// What a walk of (part of) one list found: the hits and, for TC_PV_CSR, how many of the third
// vertices have smaller ids than the centre and than the list's owner (the weights of a triangle
// depend on the order of its ids alone).
struct Hits {
  uint32_t n = 0, below_c = 0, below_o = 0;
};

// Look up two entries of the list owned by o (kNoKey where there is none); their slots are read
// before either is counted.
template <int PV, int kCnt>
__device__ __forceinline__ void probe2(const int32_t k0, const int32_t k1, const int32_t c, const int32_t o,
                                       const Set<kCnt>& t, Hits& h) {
  const uint32_t x0 = hash_of(k0), x1 = hash_of(k1);
  const uint32_t a0 = t.slot1(x0), b0 = t.slot2(x0), a1 = t.slot1(x1), b1 = t.slot2(x1);
  const int32_t p0 = lds(a0), q0 = lds(b0), p1 = lds(a1), q1 = lds(b1);
  const bool f0 = p0 == k0, f1 = p1 == k1;
  const bool h0 = f0 | (q0 == k0), h1 = f1 | (q1 == k1);
  h.n += h0;
  h.n += h1;
  if (handle_like<PV>()) {
    count_if(h0, (f0 ? a0 : b0) + kCnt, 1u);
    count_if(h1, (f1 ? a1 : b1) + kCnt, 1u);
  } else if (PV == TC_PV_CSR) {
    const uint32_t c0 = h0 & (k0 < c), c1 = h1 & (k1 < c), o0 = h0 & (k0 < o), o1 = h1 & (k1 < o);
    h.below_c += c0 + c1;
    h.below_o += o0 + o1;
    count_if(c0 | o0, (f0 ? a0 : b0) + kCnt, c0 + o0);
    count_if(c1 | o1, (f1 ? a1 : b1) + kCnt, c1 + o1);
  }
}

// The weights of a walk's hits for the centre (added to c_acc) and the owner (returned).
template <int PV>
__device__ __forceinline__ uint32_t credit(const Hits& h, const int32_t c, const int32_t o, uint32_t& tri,
                                           uint32_t& c_acc) {
  tri += h.n;
  if (handle_like<PV>()) {
    c_acc += h.n;
    return h.n;
  }
  if (PV == TC_PV_CSR) {  // the smallest id of a triangle gets 2, the middle one 1
    c_acc += h.n * (1u + (c < o)) - h.below_c;
    return h.n * (1u + (o < c)) - h.below_o;
  }
  return 0;
}

// kLanes lanes walk the list lst[0 .. len) together, lane `at` of them taking every kLanes-th
// entry, kUnroll per lane in flight: the whole warp with coalesced loads (kLanes = 32), or one lane
// alone (kLanes = 1; the lanes of a warp then walk different short lists at once).
template <int PV, int kLanes, int kCnt>
__device__ __forceinline__ void walk_list(const int32_t* __restrict__ lst, const int len, const int at, const int32_t c,
                                          const int32_t o, const Set<kCnt>& t, Hits& h) {
  static_assert(kUnroll == 4, "the last step is cut to half of its rows");
  lst += at;
  int left = len;
  for (; left >= kUnroll * kLanes; left -= kUnroll * kLanes, lst += kUnroll * kLanes) {
    int32_t w[kUnroll];
#pragma unroll
    for (int j = 0; j < kUnroll; ++j) w[j] = __ldg(lst + j * kLanes);
#pragma unroll
    for (int j = 0; j < kUnroll; j += 2) probe2<PV>(w[j], w[j + 1], c, o, t, h);
  }
  if (left > 0) {
    const int mine = left - at;
    int32_t w[kUnroll];
#pragma unroll
    for (int j = 0; j < kUnroll; ++j) w[j] = mine > j * kLanes ? __ldg(lst + j * kLanes) : kNoKey;
    probe2<PV>(w[0], w[1], c, o, t, h);
    if (left > 2 * kLanes) probe2<PV>(w[2], w[3], c, o, t, h);
  }
}

// First index of the ascending list lst[0 .. len) whose entry is >= key (one lane, binary search).
__device__ __forceinline__ int lower_bound_list(const int32_t* __restrict__ lst, int len, const int32_t key) {
  int lo = 0;
  while (len > 0) {
    const int half = len >> 1;
    if (__ldg(lst + lo + half) < key) {
      lo += half + 1;
      len -= half + 1;
    } else {
      len = half;
    }
  }
  return lo;
}

// Lanes that walk one packed list. Handle conventions: 4 (8 lists at a time; 8 lanes: BA n = 2^22
// + 2.6 %); without per-vertex output or with CSR weights 8 (4 lanes: Erdos-Renyi n = 10^6 total
// + 6 %, R-MAT 20 + 1.5 %).
template <int PV>
__host__ __device__ constexpr int pack_lanes() {
  return handle_like<PV>() ? 4 : 8;
}

// Lists at most this long are walked whole in a value-range pass (entries outside the pass's
// range just miss the hash set); longer ones are first cut to the range by two binary searches.
constexpr int kRangeSearchMin = 32;

// offp[u] holds where N+(u) starts and, in its upper bits, how long it is (dplus[u], cut at
// kHeadMax), so that a neighbour's list is looked up with one 8-byte load. The warp tiers wait on
// chains of dependent loads (58 % of their cycles on BA n = 2^22: neighbour, out-degree, start where
// the edge is the centre's, list); with one load for both, the first neighbours read beside the
// entries and the centres' heads read by the chunk: BA 6.72 -> 6.05 ms, Erdos-Renyi n = 10^6 1.353 ->
// 1.256, R-MAT 24 125.1 -> 121.4, R-MAT 20 3.95 -> 3.88. Not kept: the next centre's or group's
// loads a step ahead (BA + 3 %, registers), neighbours' heads before the set is built (BA + 1 %).
constexpr int kHeadShift = 40;
constexpr int kHeadMax = (1 << 23) - 1;
__device__ __forceinline__ int64_t head_of(const int64_t start, const int32_t a) {
  return start | ((int64_t)min(a, kHeadMax) << kHeadShift);
}
__device__ __forceinline__ int64_t head_start(const int64_t head) { return head & (((int64_t)1 << kHeadShift) - 1); }

__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// A lane's neighbour o (-1: none), its out-degree and its oriented list (b = 0 where there is none).
struct Group {
  int32_t o;
  int b;
  const int32_t* lst;
};
__device__ __forceinline__ Group fetch_group(const int32_t n, int32_t o, const int32_t* __restrict__ dplus,
                                             const int64_t* __restrict__ offp, const int32_t* __restrict__ indp) {
  const bool valid = o >= 0 && o < n;  // ids out of range were flagged by the orientation
  if (!valid) o = 0;
  const int64_t head = __ldg(offp + o);
  int b = (int)(head >> kHeadShift);
  if (b == kHeadMax) b = __ldg(dplus + o);
  return {o, valid ? b : 0, indp + head_start(head)};
}

// Position of the n-th (from 0) set bit of m.
__device__ __forceinline__ int nth_bit(const unsigned m, int n) {
  int at = 0;
#pragma unroll
  for (int step = kWarp / 2; step > 0; step >>= 1) {
    const int below = __popc((m >> at) & ((1u << step) - 1u));
    if (n >= below) {
      n -= below;
      at += step;
    }
  }
  return at;
}

// One warp takes a group of up to 32 neighbours o of centre c (out-degree a), one per lane, and
// intersects every edge {c, o} whose centre is c: N+(o), the shorter list (b <= a entries), goes
// through the hash set of the staged chunk of N+(c). Per edge the scheduler picks how (table cell,
// else the thresholds b <= lane_max, b <= packed_max):
//   lane:   each such lane walks its own list, all at once (short lists);
//   packed: several such lists at a time, pack_lanes() lanes each, so mid-size lists neither leave
//           most of the warp idle nor need a search for the owner of each entry;
//   warp:   the lists are taken one at a time and the warp streams each with coalesced loads,
//           so o, its list and its count stay warp-uniform.
// When the hash set holds only the entries of N+(c) in [vlo, vhi) (one pass of a centre whose
// N+(c) is larger than a table), only the part of each N+(o) inside that range is walked: both
// lists are ascending, so no entry outside it can hit. The range sits in shared memory
// (CountSmem::ranged, vlo, vhi), so it holds no register across the group loop; the CTA tier
// compiles the cut in, the warp tiers leave it out.
template <int PV, int kCnt>
__device__ __forceinline__ void process_group(Group f, const int32_t c, const int a,
                                              const Set<kCnt>& t, const CountSmem& sm, const int lane,
                                              uint32_t* __restrict__ out, const SchedParams& sp, uint32_t& tri,
                                              uint32_t& c_acc) {
  constexpr bool kMayRange = kCnt == kHashMax * 4;  // the CTA tier
  const int32_t o = f.o;
  const int b = f.b;
  const int32_t* lst = f.lst;
  const bool mine = b > 0 && centre_of(c, a, o, b) &&
                    (sp.cell_filter == -1 ||
                     (sp.cell_filter >= 0 && log2_cell(a) * 16 + log2_cell(b) == sp.cell_filter));
  int strat = !mine ? -1
              : sp.use_table ? sp.table[log2_cell(a)][log2_cell(b)]
                             : (b <= sp.lane_max ? 1 : b <= sp.packed_max ? 2 : 0);
  int len = b;  // entries of N+(o) walked, from lst
  if (kMayRange && sm.ranged) {  // uniform over the CTA
    if (strat >= 0 && b > kRangeSearchMin) {
      const int32_t vlo = sm.vlo, vhi = sm.vhi;
      const int p0 = vlo == INT_MIN ? 0 : lower_bound_list(lst, b, vlo);
      const int p1 = vhi == INT_MAX ? b : p0 + lower_bound_list(lst + p0, b - p0, vhi);
      lst += p0;
      len = p1 - p0;
      if (len == 0) strat = -1;
    }
    __syncwarp();
  }
  const bool by_lane = strat == 1;
  if (__any_sync(kFull, by_lane)) {
    if (by_lane) {
      Hits h;
      walk_list<PV, 1>(lst, len, 0, c, o, t, h);
      const uint32_t vacc = credit<PV>(h, c, o, tri, c_acc);
      if (PV != TC_PV_NONE && vacc) out_add<PV>(out, o, vacc);
    }
    __syncwarp();
  }
  // The lists are on their way from DRAM while the first ones are walked (first and last line: a
  // packed list is seldom longer than two). BA n = 2^22 6.05 -> 5.69 ms, Erdos-Renyi n = 10^6 1.257
  // -> 1.222, R-MAT 24 121.5 -> 121.0; R-MAT 20, whose lists are in L2, 3.883 -> 3.895.
  if (strat >= 0) prefetch_l2(lst);
  if (strat == 2) prefetch_l2(lst + len - 1);
  const unsigned packed = __ballot_sync(kFull, strat == 2);
  if (packed) {
    // the packed lists' fields, moved to the first lanes: lane r holds the r-th such list
    const int count = __popc(packed);
    const int from = nth_bit(packed, lane);
    constexpr int kPackLanes = pack_lanes<PV>();
    const int32_t po_l = __shfl_sync(kFull, o, from);
    const int plen_l = __shfl_sync(kFull, len, from);
    const unsigned long long plst_l = __shfl_sync(kFull, (unsigned long long)lst, from);
    for (int r0 = 0; r0 < count; r0 += kWarp / kPackLanes) {
      const int r = r0 + lane / kPackLanes;
      const int32_t po = __shfl_sync(kFull, po_l, r);
      const int32_t* plst = (const int32_t*)__shfl_sync(kFull, plst_l, r);
      const int plen_r = __shfl_sync(kFull, plen_l, r);
      const int plen = r < count ? plen_r : 0;
      Hits h;
      walk_list<PV, kPackLanes>(plst, plen, lane % kPackLanes, c, po, t, h);
      __syncwarp();
      uint32_t vacc = credit<PV>(h, c, po, tri, c_acc);
      if (PV != TC_PV_NONE) {
#pragma unroll
        for (int d = kPackLanes / 2; d > 0; d >>= 1) vacc += __shfl_xor_sync(kFull, vacc, d);
        if (lane % kPackLanes == 0 && vacc) out_add<PV>(out, po, vacc);
      }
    }
    __syncwarp();
  }
  unsigned todo = __ballot_sync(kFull, strat == 0);
  uint32_t o_acc = 0;  // what this lane's neighbour gets from its own list's walk
  while (todo) {
    const int sl = __ffs(todo) - 1;
    todo &= todo - 1;
    const int32_t so = __shfl_sync(kFull, o, sl);
    const int sb = __shfl_sync(kFull, len, sl);
    const int32_t* slst = (const int32_t*)__shfl_sync(kFull, (unsigned long long)lst, sl);
    Hits h;
    walk_list<PV, kWarp>(slst, sb, lane, c, so, t, h);
    __syncwarp();
    uint32_t vacc = credit<PV>(h, c, so, tri, c_acc);
    if (PV != TC_PV_NONE) {
      vacc = __reduce_add_sync(kFull, vacc);
      if (lane == sl) o_acc = vacc;
    }
  }
  if (PV != TC_PV_NONE && o_acc) out_add<PV>(out, o, o_acc);
  __syncwarp();
}

// Flush a set's counters into the per-vertex output, by `threads` threads of index `at`.
template <int PV, int kCnt>
__device__ __forceinline__ void flush_set(const Set<kCnt>& t, const int at, const int threads, uint32_t* __restrict__ out) {
  for (int s = at; s < t.slots() / 4; s += threads) {
    const int4 x = lds4(t.keys + kCnt + 16 * s);
    if (!(x.x | x.y | x.z | x.w)) continue;
    const int4 k = lds4(t.keys + 16 * s);
    if (x.x) out_add<PV>(out, k.x, x.x);
    if (x.y) out_add<PV>(out, k.y, x.y);
    if (x.z) out_add<PV>(out, k.z, x.z);
    if (x.w) out_add<PV>(out, k.w, x.w);
  }
}

// One warp counts the edges of centre c (out-degree a <= kWarpTierMax) among its neighbours
// N(c)[k0 .. k1).
template <int PV>
__device__ __forceinline__ void warp_centre(const int32_t n, const int32_t c, const int a, const int64_t start,
                                            const int k0, const int k1, const uint32_t table,
                                            const CountSmem& sm, const int lane,
                                            const int32_t* __restrict__ ind, const int32_t* __restrict__ dplus,
                                            const int64_t* __restrict__ offp, const int32_t* __restrict__ indp,
                                            uint32_t* __restrict__ out, const SchedParams& sp, uint32_t& tri) {
  int bits = 6;  // 2^(bits + 1) slots, at least 4a (load <= 0.25; one 16-byte store per lane clears 128)
  while ((2 << bits) < 4 * a && (2 << bits) < kWarpSlots) ++bits;
  const WarpSet t{table, bits};
  uint32_t c_acc = 0;
  int clen = a;  // entries staged at a time: all of them, fewer only after a failed build
  // The first neighbours and entries are in flight together, while the set is cleared.
  int32_t nbr = lane < k1 - k0 ? __ldg(ind + start + k0 + lane) : -1;
  const int32_t first = lane < a ? __ldg(indp + start + lane) : kNoKey;
  for (int cb = 0; cb < a; cb += clen) {
    clen = min(clen, a - cb);
    while (true) {
      clear_set(t, lane, kWarp);
      __syncwarp();
      bool ok = true;
      int j = lane;
      if (cb == 0 && j < clen) {
        ok = insert(t, first);
        j += kWarp;
      }
      for (; j < clen; j += kWarp) ok &= insert(t, __ldg(indp + start + cb + j));
      __syncwarp();
      if (__all_sync(kFull, ok)) break;
      clen = (clen + 1) / 2;
    }
    for (int g = k0; g < k1; g += kWarp) {
      if (g > k0 || cb > 0) nbr = lane < k1 - g ? __ldg(ind + start + g + lane) : -1;
      const Group f = fetch_group(n, nbr, dplus, offp, indp);
      process_group<PV>(f, c, a, t, sm, lane, out, sp, tri, c_acc);
    }
    if (PV != TC_PV_NONE) {
      flush_set<PV>(t, lane, kWarp, out);
      __syncwarp();
    }
  }
  if (PV != TC_PV_NONE) {
    c_acc = __reduce_add_sync(kFull, c_acc);
    if (lane == 0 && c_acc) out_add<PV>(out, c, c_acc);
  }
  __syncwarp();
}

// Work items of the queues: centre c and the first neighbour index k0 of its range of N(c).
__device__ __forceinline__ unsigned long long make_item(int32_t c, int32_t k0) {
  return ((unsigned long long)(uint32_t)c << 32) | (uint32_t)k0;
}

template <int PV>
__global__ void __launch_bounds__(kThreads, kCtasPerSm) k_count(const int32_t n, const int32_t* __restrict__ ind,
                                                    const int32_t* __restrict__ degv,
                                                    const int32_t* __restrict__ dplus,
                                                    const int64_t* __restrict__ offp,
                                                    const int32_t* __restrict__ indp,
                                                    const unsigned long long* __restrict__ large,
                                                    const unsigned long long* __restrict__ medium,
                                                    uint32_t* __restrict__ out, DevStatus* __restrict__ st,
                                                    const SchedParams sp) {
  TC_DBG_ENTER(6);
  const uint32_t table = table_base();
  CountSmem& sm = *reinterpret_cast<CountSmem*>(smem_raw + kTableBytes);
  const int lane = lane_id();
  const int wid = threadIdx.x / kWarp;
  uint32_t tri = 0;
  const unsigned n_large = st->n_large;
  const unsigned n_medium = st->n_medium;

  // An empty queue is not asked: thousands of warps at one counter take longer than a small graph's
  // count (256x256 torus with orient's queues by index: 107 -> 93 us; R-MAT 20 is unchanged).

  // CTA tier: one CTA per item (centre with a > warp_max, sp.cta_range of its neighbours), over
  // chunks of kChunk entries of N+(c).
  const CtaSet L{table, kHashMaxBits - 1};
  if (threadIdx.x == 0) sm.ranged = 0;
  while (n_large != 0) {
    if (threadIdx.x == 0) {
      const unsigned q = atomicAdd(&st->q_large, 1u);
      sm.item = q < n_large ? large[q] : ~0ull;
    }
    __syncwarp();
    __syncthreads();
    const unsigned long long item = sm.item;
    __syncthreads();
    if (item == ~0ull) break;
    const int32_t c = (int32_t)(item >> 32);
    const int32_t k0 = (int32_t)(uint32_t)item;
    const int32_t a = dplus[c];
    const int64_t start = head_start(offp[c]);
    const int32_t k1 = min(degv[c], k0 + sp.cta_range);
    uint32_t c_acc = 0;
    // N+(c) in passes of at most kChunk entries, split evenly; a pass holds the entries of N+(c) in
    // [vlo, vhi), and only that part of each streamed list is walked in it.
    const int passes = (a + kChunk - 1) / kChunk;
    int clen = (a + passes - 1) / passes;
    for (int cb = 0; cb < a; cb += clen) {
      clen = min(clen, a - cb);
      while (true) {
        // this thread's entries, in flight while the table is cleared
        int32_t mine[kChunk / kThreads];
#pragma unroll
        for (int j = 0; j < kChunk / kThreads; ++j) {
          const int e = (int)threadIdx.x + j * kThreads;
          mine[j] = e < clen ? __ldg(indp + start + cb + e) : kNoKey;
        }
        clear_set(L, threadIdx.x, kThreads);
        if (threadIdx.x == 0) {
          sm.gctr = 0;
          sm.ranged = clen < a;
          sm.vlo = cb == 0 ? INT_MIN : mine[0];
          sm.vhi = cb + clen == a ? INT_MAX : __ldg(indp + start + cb + clen);
        }
        __syncwarp();
        __syncthreads();
        bool ok = true;
#pragma unroll
        for (int j = 0; j < kChunk / kThreads; ++j)
          if (mine[j] != kNoKey) ok &= insert(L, mine[j]);
        __syncwarp();
        if (__syncthreads_and(ok)) break;
        clen = (clen + 1) / 2;
      }
      const int ngroups = (k1 - k0 + kWarp - 1) / kWarp;
      while (true) {
        int g = 0;
        if (lane == 0) g = atomicAdd(&sm.gctr, 1);
        __syncwarp();
        g = __shfl_sync(kFull, g, 0);
        if (g >= ngroups) break;
        const int gk = k0 + g * kWarp;
        const Group f = fetch_group(n, lane < k1 - gk ? __ldg(ind + start + gk + lane) : -1, dplus, offp, indp);
        process_group<PV>(f, c, a, L, sm, lane, out, sp, tri, c_acc);
      }
      __syncwarp();
      __syncthreads();
      if (PV != TC_PV_NONE)
        flush_set<PV>(L, threadIdx.x, kThreads, out);
      __syncwarp();
      __syncthreads();
    }
    if (threadIdx.x == 0) sm.ranged = 0;  // the next item sets it again before its first group
    if (PV != TC_PV_NONE) {
      c_acc = __reduce_add_sync(kFull, c_acc);
      if (lane == 0 && c_acc) out_add<PV>(out, c, c_acc);
    }
  }

  // From here every warp works alone, on its own slice of the (now free) staging area.
  const uint32_t W = table + wid * kWarpTableBytes;

  // Warp tier, centres with many neighbours: one warp per item (sp.warp_range neighbours).
  while (n_medium != 0) {
    unsigned long long item = ~0ull;
    if (lane == 0) {
      const unsigned q = atomicAdd(&st->q_medium, 1u);
      if (q < n_medium) item = medium[q];
    }
    __syncwarp();
    item = __shfl_sync(kFull, item, 0);
    if (item == ~0ull) break;
    const int32_t c = (int32_t)(item >> 32);
    const int32_t k0 = (int32_t)(uint32_t)item;
    const int a = __ldg(dplus + c);
    const int64_t start = head_start(__ldg(offp + c));
    const int k1 = min(__ldg(degv + c), k0 + sp.warp_range);
    warp_centre<PV>(n, c, a, start, k0, k1, W, sm, lane, ind, dplus, offp, indp, out, sp, tri);
  }

  // Warp tier, the rest (1 <= a <= warp_max, degree <= sp.warp_range): one warp per centre,
  // claimed in chunks of vertex ids.
  while (true) {
    unsigned long long c0 = 0;
    if (lane == 0) c0 = atomicAdd(&st->q_small, (unsigned long long)sp.chunk);
    __syncwarp();
    c0 = __shfl_sync(kFull, c0, 0);
    if (c0 >= (unsigned long long)n) break;
    const int32_t cend = (int32_t)min((unsigned long long)n, c0 + (unsigned long long)sp.chunk);
    // this count's centres (all of them unless sharded), read per claimed chunk
    const bool sharded = st->sharded != 0;
    const int32_t s_lo = (int32_t)st->shard_lo, s_hi = (int32_t)st->shard_hi;
    for (int32_t ub = (int32_t)c0; ub < cend; ub += kWarp) {
      const int32_t uu = ub + lane;
      const bool in = uu < cend;
      const int64_t head = in ? __ldg(offp + uu) : 0;
      const int aa = (int)(head >> kHeadShift);  // a centre of this tier has a <= warp_max < kHeadMax
      const int dd = in ? __ldg(degv + uu) : 0;
      unsigned elig = __ballot_sync(
          kFull, aa >= 1 && aa <= sp.warp_max && dd <= sp.warp_range && (!sharded || (uu >= s_lo && uu < s_hi)));
      if (aa >= 1) {  // the rows of the chunk's later centres
        prefetch_l2(ind + head_start(head));
        prefetch_l2(indp + head_start(head));
      }
      while (elig) {
        const int sl = __ffs(elig) - 1;
        elig &= elig - 1;
        const int32_t c = ub + sl;
        const int a = __shfl_sync(kFull, aa, sl);
        const int d = __shfl_sync(kFull, dd, sl);
        const int64_t start = head_start(__shfl_sync(kFull, head, sl));
        warp_centre<PV>(n, c, a, start, 0, d, W, sm, lane, ind, dplus, offp, indp, out, sp, tri);
      }
    }
  }

  // One global atomic per CTA for the triangle total.
  __syncwarp();
  const unsigned long long t = warp_sum((unsigned long long)tri);
  if (lane == 0) sm.tri[wid] = t;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long s = 0;
    for (int w = 0; w < kWarps; ++w) s += sm.tri[w];
    if (s) atomicAdd(&st->triangles, s);
  }
  TC_DBG_EXIT(6);
}

// ---- orientation ------------------------------------------------------------------------

__device__ __forceinline__ bool precedes(int32_t du, int32_t u, int32_t dv, int32_t v) {
  return du < dv || (du == dv && u < v);
}

// One warp orients entries [k_begin, k_end) of u's list (s = its start, d = its degree): it
// checks each entry (id in range, strictly ascending, no self-loop, signed symmetry checksum)
// and, when kWrite, writes the out-neighbours (in list order) to indp[out_base ...]. Returns
// their number (warp-uniform).
template <class View, bool kWrite>
__device__ __forceinline__ int orient_range(const View& g, const int32_t n, const int32_t u, const int32_t d,
                                            const int64_t s, const int32_t k_begin, const int32_t k_end,
                                            int32_t* __restrict__ indp, const int64_t out_base,
                                            unsigned long long& chk, unsigned& bad) {
  const int lane = threadIdx.x & (kWarp - 1);
  const unsigned lt = lanemask_lt();
  int cnt = 0;
  int32_t last = k_begin > 0 ? g.ind[s + k_begin - 1] : INT32_MIN;
  for (int32_t k0 = k_begin; k0 < k_end; k0 += kWarp) {
    const int32_t k = k0 + lane;
    const bool in = k < k_end;
    const int32_t v = in ? g.ind[s + k] : INT32_MAX;
    int32_t prev = __shfl_up_sync(kFull, v, 1);
    if (lane == 0) prev = last;
    last = __shfl_sync(kFull, v, kWarp - 1);
    bool pred = false;
    if (in) {
      if (v < 0 || v >= n) {
        bad |= kBadRange;
      } else {
        if (k > 0 && prev >= v) bad |= kBadOrder;
        if (v == u) bad |= kBadSelfLoop;
        pred = precedes(d, u, g.len(v), v);
        const uint64_t h = (u < v) ? sym_hash((uint32_t)u, (uint32_t)v) : sym_hash((uint32_t)v, (uint32_t)u);
        chk += (u < v) ? h : (0ull - h);
      }
    }
    __syncwarp();
    const unsigned msk = __ballot_sync(kFull, pred);
    if (kWrite && pred) indp[out_base + cnt + __popc(msk & lt)] = v;
    cnt += __popc(msk);
  }
  return cnt;
}

// Orientation bookkeeping of a finished vertex u with degree d and out-degree a (warp-uniform
// call): its offset, degree and out-degree and the work figures.
struct OrientAcc {
  unsigned long long work = 0, ei = 0;
  unsigned mx = 0;
};

__device__ __forceinline__ void finish_vertex(const int32_t u, const int32_t d, const int64_t s, const int32_t a,
                                              int32_t* __restrict__ dplus, int64_t* __restrict__ offp,
                                              int32_t* __restrict__ degv, OrientAcc& acc) {
  const int lane = threadIdx.x & (kWarp - 1);
  if (lane == 0) {
    dplus[u] = a;
    offp[u] = head_of(s, a);
    degv[u] = d;
    if (d >= 2) acc.ei += (unsigned long long)a;
    // sum over u -> v of d+(u) + d+(v) = sum over v of d+(v) deg(v)
    acc.work += (unsigned long long)a * (unsigned long long)d;
    acc.mx = max(acc.mx, (unsigned)a);
  }
}

// Register the vertices whose list is longer than kHubMin: they are oriented in chunks of up to
// kHubChunk entries that separate warps take. One thread per vertex. A hub starts with
// out-degree 0, so a hub that is never completed (capacity error) leaves nothing for the count
// to read.
template <class View>
__global__ void __launch_bounds__(256) k_find_hubs(const View g, const int32_t n, int32_t* __restrict__ dplus,
                                                   int64_t* __restrict__ offp, int32_t* __restrict__ degv,
                                                   int32_t* __restrict__ hub_u,
                                                   int32_t* __restrict__ hub_base, int32_t* __restrict__ hub_done,
                                                   int32_t* __restrict__ chunk_hub, const int64_t hub_cap,
                                                   const int64_t chunk_cap, const int32_t hub_chunk,
                                                   DevStatus* __restrict__ st) {
  for (int64_t uu = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; uu < n; uu += (int64_t)gridDim.x * blockDim.x) {
    const int32_t u = (int32_t)uu;
    const int32_t d = g.len(u);
    if (d <= kHubMin) continue;
    dplus[u] = 0;
    offp[u] = 0;
    degv[u] = 0;
    const int nch = (d + hub_chunk - 1) / hub_chunk;
    const unsigned h = atomicAdd(&st->n_hubs, 1u);
    const unsigned base = atomicAdd(&st->n_hub_chunks, (unsigned)nch);
    const bool ok = h < hub_cap && (int64_t)base + nch <= chunk_cap;
    if (ok) {
      hub_u[h] = u;
      hub_base[h] = (int32_t)base;
      hub_done[h] = 0;
    } else {
      atomicOr(&st->bad_flags, kBadCapacity);
    }
    for (int c = 0; c < nch && (int64_t)base + c < chunk_cap; ++c) chunk_hub[base + c] = ok ? (int32_t)h : -1;
  }
}

// Single-pass orientation into the input's own index space: N+(u) is written at
// indp[start(u) ...], so no offsets scan is needed (offp[u] = start(u) and the length). A persistent grid of
// warps first takes hub chunks from one queue, then tiles of vertex ids from another. A hub
// chunk is written at its own position in the hub's list; the warp that finishes a hub's last
// chunk (a counter per hub) moves the pieces together and completes the vertex.
constexpr int kOrientCtasPerSm = 5;  // 48 registers, 8 bytes spilled (6 CTAs: Erdos-Renyi n = 10^6 count + 1.4 %)
template <class View, bool kWrite>
__global__ void __launch_bounds__(256, kOrientCtasPerSm) k_orient(const View g, const int32_t n, int32_t* __restrict__ dplus,
                                                int64_t* __restrict__ offp, int32_t* __restrict__ degv,
                                                int32_t* __restrict__ indp, const int64_t e_cap,
                                                const int32_t* __restrict__ hub_u,
                                                const int32_t* __restrict__ hub_base, int32_t* __restrict__ hub_cnt,
                                                int32_t* __restrict__ hub_done, const int32_t* __restrict__ chunk_hub,
                                                const int64_t hub_cap, const int64_t chunk_cap, const int32_t hub_chunk,
                                                const int32_t tile, DevStatus* __restrict__ st) {
  const int lane = threadIdx.x & (kWarp - 1);
  const unsigned nchunks = (unsigned)min((long long)st->n_hub_chunks, (long long)chunk_cap);
  const unsigned nhubs = (unsigned)min((long long)st->n_hubs, (long long)hub_cap);
  unsigned long long chk = 0;
  unsigned bad = 0;
  OrientAcc acc;

  // Hub chunks. A queue of at most one piece per warp goes by index instead of by its counter (the
  // tiles only where no hub chunk holds some warps back): R-MAT 16 count 225 -> 219 us.
  const unsigned warps = (gridDim.x * blockDim.x) / kWarp, gw = (blockIdx.x * blockDim.x + threadIdx.x) / kWarp;
  const bool hubs_by_index = nchunks <= warps;
  for (bool first = true; first || !hubs_by_index; first = false) {
    unsigned q = gw;
    if (!hubs_by_index) {
      if (lane == 0) q = atomicAdd(&st->q_orient_hub, 1u);
      __syncwarp();
      q = __shfl_sync(kFull, q, 0);
    }
    if (q >= nchunks) break;
    const int h = chunk_hub[q];
    if (h < 0 || h >= (int)nhubs) continue;
    const int hb = hub_base[h];
    const int32_t u = hub_u[h];
    const int64_t s = g.start(u);
    const int32_t d = g.len(u);
    const int nch = (d + hub_chunk - 1) / hub_chunk;
    const int c = (int)q - hb;
    if (c < 0 || c >= nch) continue;
    if (s < 0 || s + d > e_cap) {
      bad |= kBadCapacity;
      continue;
    }
    const int32_t k_begin = c * hub_chunk, k_end = min(d, k_begin + hub_chunk);
    const int cnt = orient_range<View, kWrite>(g, n, u, d, s, k_begin, k_end, indp, s + k_begin, chk, bad);
    // Publish this chunk (entries written by every lane, then its count), then count it done.
    if (lane == 0) hub_cnt[q] = cnt;
    __threadfence();
    __syncwarp();
    int done = 0;
    if (lane == 0) done = atomicAdd(&hub_done[h], 1);
    __syncwarp();
    done = __shfl_sync(kFull, done, 0);
    if (done != nch - 1) continue;
    // Last chunk of this hub: gather the pieces (each chunk's out-neighbours start at the
    // chunk's own position; moving them down in chunk order never overwrites an unread entry).
    __threadfence();
    int a = 0;
    for (int cc = 0; cc < nch; ++cc) {
      const int cn = __ldcg(hub_cnt + hb + cc);
      if (kWrite && cc > 0 && cn > 0) {
        const int64_t src = s + (int64_t)cc * hub_chunk, dst = s + a;
        for (int k0 = 0; k0 < cn; k0 += kWarp) {
          const int k = k0 + lane;
          const int32_t x = k < cn ? __ldcg(indp + src + k) : 0;
          __syncwarp();
          if (k < cn) indp[dst + k] = x;
          __syncwarp();
        }
      }
      a += cn;
    }
    finish_vertex(u, d, s, a, dplus, offp, degv, acc);
  }

  // Vertex tiles (hubs skipped: done above). The warp walks the concatenated lists of a tile's
  // vertices (at most 32), 32 entries per step and two steps in flight: short lists leave no lane idle,
  // and a step is one round of coalesced loads instead of one dependent round per vertex. Lane i
  // keeps the i-th list that has entries. The lists that start in a step are one bit each of a word
  // or-ed over the lanes, so an entry's owner is a population count. An out-neighbour's rank in
  // N+(u) is the count carried from earlier steps (of the list that goes on into this one) plus the
  // predecessors in its segment. Bound by issue (68 % on BA n = 2^22) and by the round trip to
  // each neighbour's length. With a binary search over the lanes for the owner, one step in flight and
  // the ranks' counters in shared memory the whole count took, both timed in one call: R-MAT 16 215 us
  // (with it 206), Erdos-Renyi n = 10^6 1.230 ms (1.217), BA n = 2^22 5.76 ms (5.71), R-MAT 20 3.906 ms
  // (3.895).
  constexpr int kTile = 32, kUnr = 2;
  __shared__ int32_t s_out[256 / kWarp][kTile];
  int32_t* const my_out = s_out[threadIdx.x / kWarp];
  const unsigned lt = lanemask_lt();
  const bool tiles_by_index = nchunks == 0 && (unsigned long long)n <= (unsigned long long)warps * (unsigned)tile;
  for (bool first = true; first || !tiles_by_index; first = false) {
    unsigned t0 = gw * (unsigned)tile;
    if (!tiles_by_index) {
      if (lane == 0) t0 = atomicAdd(&st->q_orient_vtx, (unsigned)tile);
      __syncwarp();
      t0 = __shfl_sync(kFull, t0, 0);
    }
    if (t0 >= (unsigned)n) break;
    const int32_t u_l = (int32_t)t0 + lane;
    const bool in_t = lane < tile && u_l < n;
    const int32_t d_l = in_t ? g.len(u_l) : 0;
    const int64_t s_l = in_t ? g.start(u_l) : 0;
    const bool own_l = in_t && d_l <= kHubMin;  // hubs were completed by the chunk loop
    const bool cap_bad = own_l && (s_l < 0 || s_l + d_l > e_cap);
    if (cap_bad) bad |= kBadCapacity;
    const int32_t len_l = own_l && !cap_bad ? d_l : 0;
    int32_t incl = len_l;
#pragma unroll
    for (int o = 1; o < kWarp; o <<= 1) {
      const int32_t y = __shfl_up_sync(kFull, incl, o);
      if (lane >= o) incl += y;
    }
    const int32_t excl_l = incl - len_l;
    const int32_t total = __shfl_sync(kFull, incl, kWarp - 1);
    my_out[lane] = 0;
    // The lists that have entries, moved to the first lanes: where entry k = 0 of the tile would be if
    // it were this list's, and the list's degree, lane and first k in one word.
    const unsigned full = __ballot_sync(kFull, len_l > 0);
    const int from = nth_bit(full, lane);
    const int64_t c_at = __shfl_sync(kFull, s_l - excl_l, from);
    static_assert(kHubMin <= 256 && kTile <= 32, "fields of c_word");
    const uint32_t word_l = (uint32_t)excl_l << 14 | (uint32_t)lane << 9 | (uint32_t)(len_l & 511);
    const uint32_t c_word = __shfl_sync(kFull, word_l, from);
    const int32_t c_first = lane < __popc(full) ? (int32_t)(c_word >> 14) : INT32_MAX;
    int started = 0;  // lists that started before the step
    int carry = 0;    // out-neighbours so far of the list that goes on into the step
    int32_t last = INT32_MIN;
    __syncwarp();
    for (int32_t k0 = 0; k0 < total; k0 += kUnr * kWarp) {
      unsigned heads[kUnr];
      uint32_t word[kUnr];
      int64_t at[kUnr];
      int32_t vs[kUnr], lens[kUnr];
#pragma unroll
      for (int j = 0; j < kUnr; ++j) {
        const int32_t k = k0 + j * kWarp;
        const unsigned rel = (unsigned)(c_first - k);
        heads[j] = __reduce_or_sync(kFull, rel < kWarp ? 1u << rel : 0u);
        const int i = started + __popc(heads[j] & (lt | (1u << lane))) - 1;
        started += __popc(heads[j]);
        at[j] = __shfl_sync(kFull, c_at, i);
        word[j] = __shfl_sync(kFull, c_word, i);
        vs[j] = k + lane < total ? g.ind[at[j] + (k + lane)] : INT32_MAX;
      }
#pragma unroll
      for (int j = 0; j < kUnr; ++j) lens[j] = (uint32_t)vs[j] < (uint32_t)n ? g.len(vs[j]) : 0;
#pragma unroll
      for (int j = 0; j < kUnr; ++j) {
        const bool in = k0 + j * kWarp + lane < total;
        const bool starts = (heads[j] >> lane) & 1u;
        const int slot = (word[j] >> 9) & 31;
        const int32_t u = (int32_t)t0 + slot;
        const int32_t v = vs[j];
        int32_t prev = __shfl_up_sync(kFull, v, 1);
        if (lane == 0) prev = last;
        last = __shfl_sync(kFull, v, kWarp - 1);
        bool pred = false;
        if (in) {
          if (v < 0 || v >= n) {
            bad |= kBadRange;
          } else {
            if (!starts && prev >= v) bad |= kBadOrder;
            if (v == u) bad |= kBadSelfLoop;
            pred = precedes((int32_t)(word[j] & 511), u, lens[j], v);
            const uint64_t h = (u < v) ? sym_hash((uint32_t)u, (uint32_t)v) : sym_hash((uint32_t)v, (uint32_t)u);
            chk += (u < v) ? h : (0ull - h);
          }
        }
        const unsigned msk = __ballot_sync(kFull, pred);
        const unsigned mine = heads[j] & (lt | (1u << lane));  // the lists that start up to this lane
        const int prior = mine ? 0 : carry;
        const unsigned seg = mine ? ~0u << (31 - __clz(mine)) : ~0u;  // from this list's first lane on
        if (kWrite && pred) indp[at[j] + (int32_t)((word[j] >> 14) + prior + __popc(msk & lt & seg))] = v;
        if (in && (starts || lane == 0)) {
          const unsigned above = heads[j] & ~(lt | (1u << lane));
          my_out[slot] = prior + __popc(msk & ~lt & (above ? (above & (0u - above)) - 1u : ~0u));
        }
        carry = heads[j] ? __popc(msk >> (31 - __clz(heads[j]))) : carry + __popc(msk);
        __syncwarp();
      }
    }
    const int32_t a_l = own_l ? my_out[lane] : 0;
    __syncwarp();
    // Finish the tile's vertices, one per lane (the bookkeeping of finish_vertex).
    if (own_l) {
      dplus[u_l] = a_l;
      offp[u_l] = head_of(cap_bad ? 0 : s_l, a_l);
      degv[u_l] = cap_bad ? 0 : d_l;
      const int32_t dd = cap_bad ? 0 : d_l;
      if (dd >= 2) acc.ei += (unsigned long long)a_l;
      acc.work += (unsigned long long)a_l * (unsigned long long)dd;
      acc.mx = max(acc.mx, (unsigned)a_l);
    }
  }

  __syncwarp();
  chk = warp_sum(chk);
  acc.work = warp_sum(acc.work);
  acc.ei = warp_sum(acc.ei);
  acc.mx = __reduce_max_sync(kFull, acc.mx);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) bad |= __shfl_xor_sync(kFull, bad, o);
  if (lane == 0) {
    if (chk) atomicAdd(&st->sym_checksum, chk);
    if (bad) atomicOr(&st->bad_flags, bad);
    if (acc.work) atomicAdd(&st->oriented_work, acc.work);
    if (acc.ei) atomicAdd(&st->edges_intersected, acc.ei);
    if (acc.mx) atomicMax(&st->max_dplus, acc.mx);
  }
}

// The count's work queues, filled after the orientation. A centre with out-degree a > warp_max
// gets CTA items of cta_range neighbours; one with a <= warp_max and more than warp_range
// neighbours gets warp items of warp_range (the other centres are claimed by id ranges). The CTA
// queue is ordered by estimated item work, largest first, so the persistent grid does not end
// on a few long items: the work class of a centre's items is log2(a * min(d, cta_range)), and
// classes are laid out in decreasing order, each in vertex-id order (which on R-MAT keeps
// centres with shared neighbours together). k_push_items counts the items per class and fills
// the warp queue; k_fill_items places the CTA items.
constexpr int kWorkClasses = 32;

__device__ __forceinline__ int work_class(const int32_t a, const int32_t d, const int32_t range) {
  const unsigned long long w = (unsigned long long)a * (unsigned long long)min(d, range);
  return min(kWorkClasses - 1, 63 - __clzll(max(w, 1ull)));
}

// Is u a centre of this count's shard (every centre when the count is not sharded)?
__device__ __forceinline__ bool in_shard(const DevStatus* __restrict__ st, const int32_t u) {
  return !st->sharded || (u >= (int32_t)st->shard_lo && u < (int32_t)st->shard_hi);
}

__device__ __forceinline__ bool cta_centre(const DevStatus* __restrict__ st, const int32_t u, const int32_t a,
                                           const int warp_max) {
  return a > warp_max && in_shard(st, u);
}

__global__ void __launch_bounds__(256) k_push_items(const int32_t n, const int32_t* __restrict__ dplus,
                                                    const int32_t* __restrict__ degv,
                                                    unsigned long long* __restrict__ medium, const int64_t item_cap,
                                                    DevStatus* __restrict__ st, const int warp_max,
                                                    const int cta_range, const int warp_range) {
  const int lane = threadIdx.x & (kWarp - 1);
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) / kWarp;
  unsigned bad = 0;
  for (int64_t t = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / kWarp; t * kWarp < n; t += nwarps) {
    const int64_t uu = t * kWarp + lane;
    const bool in = uu < n;
    const int32_t u = (int32_t)uu;
    const int32_t a = in ? dplus[u] : 0;
    const int32_t d = in ? degv[u] : 0;
    if (in && cta_centre(st, u, a, warp_max))
      atomicAdd(&st->cls_cnt[work_class(a, d, cta_range)], (unsigned)((d + cta_range - 1) / cta_range));
    const bool wrp = in && a > 0 && a <= warp_max && d > warp_range && in_shard(st, u);
    const int x = wrp ? (d + warp_range - 1) / warp_range : 0;
    int incl = x;
#pragma unroll
    for (int o = 1; o < kWarp; o <<= 1) {
      const int y = __shfl_up_sync(kFull, incl, o);
      if (lane >= o) incl += y;
    }
    const int tot = __shfl_sync(kFull, incl, kWarp - 1);
    if (tot == 0) continue;
    unsigned base = 0;
    if (lane == 0) base = atomicAdd(&st->n_medium, (unsigned)tot);
    base = __shfl_sync(kFull, base, 0);
    if ((int64_t)base + tot > item_cap) {
      bad |= kBadCapacity;
      continue;
    }
    for (int j = 0; j < x; ++j) medium[base + (incl - x) + j] = make_item(u, j * warp_range);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) bad |= __shfl_xor_sync(kFull, bad, o);
  if (lane == 0 && bad) atomicOr(&st->bad_flags, bad);
}

__global__ void __launch_bounds__(256) k_fill_items(const int32_t n, const int32_t* __restrict__ dplus,
                                                    const int32_t* __restrict__ degv,
                                                    unsigned long long* __restrict__ large, const int64_t item_cap,
                                                    DevStatus* __restrict__ st, const int warp_max,
                                                    const int cta_range, const int warp_range) {
  __shared__ unsigned cls_base[kWorkClasses];
  __shared__ unsigned total;
  if (threadIdx.x < kWarp) {
    // exclusive scan over the classes in decreasing order: class c starts after all classes > c
    const int lane = threadIdx.x;
    const unsigned x = st->cls_cnt[kWorkClasses - 1 - lane];
    unsigned incl = x;
#pragma unroll
    for (int o = 1; o < kWarp; o <<= 1) {
      const unsigned y = __shfl_up_sync(kFull, incl, o);
      if (lane >= o) incl += y;
    }
    cls_base[kWorkClasses - 1 - lane] = incl - x;
    if (lane == kWarp - 1) total = incl;
  }
  __syncthreads();
  const unsigned n_items = (unsigned)min((long long)total, (long long)item_cap);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    st->n_large = n_items;
    if ((long long)total > item_cap) atomicOr(&st->bad_flags, kBadCapacity);
  }
  for (int64_t uu = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; uu < n; uu += (int64_t)gridDim.x * blockDim.x) {
    const int32_t u = (int32_t)uu;
    const int32_t a = dplus[u];
    if (!cta_centre(st, u, a, warp_max)) continue;
    const int32_t d = degv[u];
    const int cls = work_class(a, d, cta_range);
    const int nit = (d + cta_range - 1) / cta_range;
    const unsigned at = cls_base[cls] + atomicAdd(&st->cls_pos[cls], (unsigned)nit);
    if ((int64_t)at + nit > (int64_t)n_items) continue;  // only past a capacity error
    for (int j = 0; j < nit; ++j) large[at + j] = make_item(u, j * cta_range);
  }
}

// ---- multi-GPU split of the static count -------------------------------------------------

// Predicted intersection work of each centre c (needs the orientation): one probe per entry of
// the other endpoint's list for every edge {c, o} that c is the centre of, plus 2 per such edge
// and 1 per neighbour scanned, in units of 16 (int32, clamped). One warp per vertex.
template <class View>
__global__ void __launch_bounds__(256) k_shard_cost(const View g, const int32_t n, const int32_t* __restrict__ dplus,
                                                    int32_t* __restrict__ cost) {
  const int lane = threadIdx.x & (kWarp - 1);
  const int64_t gw = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / kWarp;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) / kWarp;
  for (int64_t uu = gw; uu < n; uu += nw) {
    const int32_t u = (int32_t)uu;
    const int32_t d = g.len(u), a = dplus[u];
    const int64_t s = g.start(u);
    unsigned long long w = 0;
    for (int32_t k = lane; k < d; k += kWarp) {
      const int32_t o = g.ind[s + k];
      if (o < 0 || o >= n) continue;
      const int32_t b = dplus[o];
      if (b > 0 && centre_of(u, a, o, b)) w += (unsigned long long)b + 2ull;
    }
    w = warp_sum(w);
    if (lane == 0) cost[u] = (int32_t)min((w + (unsigned long long)d + 15ull) / 16ull, (unsigned long long)INT32_MAX);
  }
}

// This count's range of centres (shard_start over the exclusive prefix of the costs).
__global__ void k_shard_bounds(const int64_t* __restrict__ prefix, const int32_t n, const int32_t shard,
                               const int32_t nshards, DevStatus* __restrict__ st) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  const int32_t lo = shard_start(prefix, n, shard, nshards), hi = shard_start(prefix, n, shard + 1, nshards);
  st->shard_lo = (unsigned)lo;
  st->shard_hi = (unsigned)hi;
  st->shard_work = (unsigned long long)(prefix[hi] - prefix[lo]);
  st->total_work = (unsigned long long)prefix[n];
  st->sharded = 1;
}

// ---- exclusive scan of int32 counts into int64 offsets ------------------------------------

__global__ void __launch_bounds__(kScanThreads) k_scan_tile_sums(const int32_t* __restrict__ in, const int64_t n,
                                                                 int64_t* __restrict__ tile_sums) {
  TC_DBG_ENTER(2);
  __shared__ long long red[kScanThreads / kWarp];
  const int64_t base = (int64_t)blockIdx.x * kScanTile;
  long long s = 0;
  for (int k = 0; k < kScanPer; ++k) {
    const int64_t i = base + (int64_t)k * kScanThreads + threadIdx.x;
    if (i < n) s += in[i];
  }
  s = warp_sum(s);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x / kWarp] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    long long t = 0;
    for (int w = 0; w < kScanThreads / kWarp; ++w) t += red[w];
    tile_sums[blockIdx.x] = t;
  }
  TC_DBG_EXIT(2);
}

// Single CTA: exclusive scan of tile_sums[0..ntiles) in place, total into tile_sums[ntiles].
__global__ void __launch_bounds__(1024) k_scan_tile_prefix(int64_t* __restrict__ tile_sums, const int64_t ntiles) {
  TC_DBG_ENTER(3);
  __shared__ long long wsum[32];
  __shared__ long long carry_s;
  const int lane = threadIdx.x & 31, wid = threadIdx.x / 32;
  if (threadIdx.x == 0) carry_s = 0;
  __syncthreads();
  for (int64_t b0 = 0; b0 < ntiles; b0 += 1024) {
    const int64_t i = b0 + threadIdx.x;
    const long long x = (i < ntiles) ? tile_sums[i] : 0;
    long long incl = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const long long t = __shfl_up_sync(kFull, incl, o);
      if (lane >= o) incl += t;
    }
    if (lane == 31) wsum[wid] = incl;
    __syncthreads();
    if (wid == 0) {
      long long w = wsum[lane];
      long long wi = w;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const long long t = __shfl_up_sync(kFull, wi, o);
        if (lane >= o) wi += t;
      }
      wsum[lane] = wi - w;
    }
    __syncthreads();
    const long long c = carry_s;
    if (i < ntiles) tile_sums[i] = c + wsum[wid] + incl - x;
    __syncthreads();
    if (threadIdx.x == 1023) carry_s = c + wsum[wid] + incl;
    __syncthreads();
  }
  if (threadIdx.x == 0) tile_sums[ntiles] = carry_s;
  TC_DBG_EXIT(3);
}

__global__ void __launch_bounds__(kScanThreads) k_scan_tiles(const int32_t* __restrict__ in, const int64_t n,
                                                             const int64_t* __restrict__ tile_sums,
                                                             int64_t* __restrict__ out, const int64_t ntiles) {
  TC_DBG_ENTER(4);
  __shared__ long long wsum[kScanThreads / kWarp];
  const int lane = threadIdx.x & 31, wid = threadIdx.x / 32;
  const int64_t base = (int64_t)blockIdx.x * kScanTile + (int64_t)threadIdx.x * kScanPer;
  long long v[kScanPer];
  long long s = 0;
#pragma unroll
  for (int k = 0; k < kScanPer; ++k) {
    const int64_t i = base + k;
    v[k] = (i < n) ? in[i] : 0;
    s += v[k];
  }
  long long incl = s;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const long long t = __shfl_up_sync(kFull, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) wsum[wid] = incl;
  __syncthreads();
  long long wpre = 0;
  for (int w = 0; w < wid; ++w) wpre += wsum[w];
  long long run = tile_sums[blockIdx.x] + wpre + incl - s;
#pragma unroll
  for (int k = 0; k < kScanPer; ++k) {
    const int64_t i = base + k;
    if (i < n) out[i] = run;
    run += v[k];
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) out[n] = tile_sums[ntiles];
  TC_DBG_EXIT(4);
}

int orient_grid(int64_t n) {
  const int64_t want = (n + kWarps - 1) / kWarps;
  const int64_t cap = (int64_t)device_info().sms * 16;
  return (int)std::max<int64_t>(1, std::min(want, cap));
}

int hubs_grid(int64_t n) {
  const int64_t want = (n + 255) / 256;
  return (int)std::max<int64_t>(1, std::min<int64_t>(want, (int64_t)device_info().sms * 8));
}

template <int PV>
tc_status launch_count(int32_t n, const int32_t* ind, const Workspace& ws, uint32_t* out, const SchedParams& sp,
                       cudaStream_t stream) {
  constexpr int kMaxDev = 64;
  static int blocks_per_sm[kMaxDev] = {};  // 0 = not configured on that device yet
  const size_t smem = kCountSmem;
  int dev = 0;
  TC_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxDev) return fail(TC_ERR_INVALID_ARG, "device %d out of range", dev);
  if (blocks_per_sm[dev] == 0) {
    TC_CUDA_TRY(cudaFuncSetAttribute(k_count<PV>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int b = 0;
    TC_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_count<PV>, kThreads, smem));
    blocks_per_sm[dev] = std::max(1, b);
  }
  const int bps = sp.blocks_per_sm > 0 ? std::min(sp.blocks_per_sm, blocks_per_sm[dev]) : blocks_per_sm[dev];
  const int grid = device_info().sms * bps;
#ifdef TC_DEBUG_PROGRESS
  if (tc_dbg_progress_host_dev) cudaMemsetAsync(tc_dbg_progress_host_dev, 0, tc_dbg_progress_bytes, stream);
#endif
  k_count<PV><<<grid, kThreads, smem, stream>>>(n, ind, ws.degv, ws.dplus, ws.offp, ws.indp, ws.large, ws.medium, out,
                                                ws.st, sp);
  TC_CUDA_TRY(cudaGetLastError());
  return TC_OK;
}

// Grid of a persistent kernel: every CTA resident at once (occupancy looked up once per device).
template <auto kernel>
tc_status resident_grid(int threads, int* grid) {
  constexpr int kMaxDev = 64;
  static int per_sm[kMaxDev] = {};
  int dev = 0;
  TC_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxDev) return fail(TC_ERR_INVALID_ARG, "device %d out of range", dev);
  if (per_sm[dev] == 0) {
    int b = 0;
    TC_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, kernel, threads, 0));
    per_sm[dev] = std::max(1, b);
  }
  *grid = device_info().sms * per_sm[dev];
  return TC_OK;
}

template <class View>
tc_status orient(const View& view, int32_t n, Workspace& ws, const SchedParams& sp, bool write, cudaStream_t stream) {
  k_find_hubs<View><<<hubs_grid(n), 256, 0, stream>>>(view, n, ws.dplus, ws.offp, ws.degv, ws.hub_u, ws.hub_base,
                                                      ws.hub_done, ws.chunk_hub, ws.hub_cap, ws.chunk_cap, sp.hub_chunk, ws.st);
  TC_CUDA_TRY(cudaGetLastError());
  int grid = 0;
  if (write) TC_TRY((resident_grid<k_orient<View, true>>(256, &grid)));
  else TC_TRY((resident_grid<k_orient<View, false>>(256, &grid)));
  if (write)
    k_orient<View, true><<<grid, 256, 0, stream>>>(view, n, ws.dplus, ws.offp, ws.degv, ws.indp, ws.e_cap,
                                                   ws.hub_u, ws.hub_base, ws.hub_cnt, ws.hub_done, ws.chunk_hub,
                                                   ws.hub_cap, ws.chunk_cap, sp.hub_chunk, sp.tile, ws.st);
  else
    k_orient<View, false><<<grid, 256, 0, stream>>>(view, n, ws.dplus, ws.offp, ws.degv, ws.indp, ws.e_cap,
                                                    ws.hub_u, ws.hub_base, ws.hub_cnt, ws.hub_done, ws.chunk_hub,
                                                    ws.hub_cap, ws.chunk_cap, sp.hub_chunk, sp.tile, ws.st);
  TC_CUDA_TRY(cudaGetLastError());
  if (write) {
    if (sp.nshards > 1) {
      // this count's range of centres: predicted work per centre, its prefix, the range
      if (!ws.shard_cost || ws.shard_cap < (int64_t)n + 1)
        return fail(TC_ERR_STATE, "sharded count without its shard workspace");
      k_shard_cost<View><<<orient_grid(n), 256, 0, stream>>>(view, n, ws.dplus, ws.shard_cost);
      TC_CUDA_TRY(cudaGetLastError());
      TC_TRY(scan_counts(ws.shard_cost, n, ws.shard_prefix, ws.shard_tiles, stream));
      k_shard_bounds<<<1, 32, 0, stream>>>(ws.shard_prefix, n, sp.shard, sp.nshards, ws.st);
      TC_CUDA_TRY(cudaGetLastError());
    }
    // the count's work queues (only a count reads them)
    k_push_items<<<hubs_grid(n), 256, 0, stream>>>(n, ws.dplus, ws.degv, ws.medium, ws.item_cap, ws.st, sp.warp_max,
                                              sp.cta_range, sp.warp_range);
    TC_CUDA_TRY(cudaGetLastError());
    k_fill_items<<<hubs_grid(n), 256, 0, stream>>>(n, ws.dplus, ws.degv, ws.large, ws.item_cap, ws.st, sp.warp_max,
                                              sp.cta_range, sp.warp_range);
    TC_CUDA_TRY(cudaGetLastError());
  }
  return TC_OK;
}

}  // namespace

int64_t scan_tiles(int64_t n) { return (n + kScanTile - 1) / kScanTile; }

tc_status scan_counts(const int32_t* in, int64_t n, int64_t* out, int64_t* tile_sums, cudaStream_t stream) {
  const int64_t nt = scan_tiles(n);
  if (nt == 0) {
    TC_CUDA_TRY(cudaMemsetAsync(out, 0, sizeof(int64_t), stream));
    return TC_OK;
  }
  k_scan_tile_sums<<<(unsigned)nt, kScanThreads, 0, stream>>>(in, n, tile_sums);
  k_scan_tile_prefix<<<1, 1024, 0, stream>>>(tile_sums, nt);
  k_scan_tiles<<<(unsigned)nt, kScanThreads, 0, stream>>>(in, n, tile_sums, out, nt);
  TC_CUDA_TRY(cudaGetLastError());
  return TC_OK;
}

SchedParams to_params(const tc_sched* s) {
  tc_sched d;
  if (!s) {
    tc_sched_default(&d);
    s = &d;
  }
  SchedParams p;
  p.warp_max = std::min(kWarpTierMax, std::max(2, s->warp_max_deg));
  p.search_ratio_x16 = std::max(0, s->search_ratio_x16);
  p.use_table = s->use_table ? 1 : 0;
  p.chunk = s->chunk > 0 ? (std::min(s->chunk, 1 << 30) + 31) / 32 * 32 : 0;
  p.blocks_per_sm = std::max(0, s->blocks_per_sm);
  p.nshards = std::max(1, s->nshards);
  p.shard = std::min(std::max(0, s->shard), p.nshards - 1);
  p.cell_filter = s->cell_filter < -2 ? -1 : s->cell_filter;
  p.lane_max = std::min(64, std::max(0, s->lane_max_deg));
  p.packed_max = std::max(0, s->packed_max_deg);
  p.hub_min = std::max(0, s->stream_hub_min);
  memcpy(p.table, s->table, sizeof(p.table));
  return p;
}

// How a count's work is cut. On a graph that keeps every warp busy for long the pieces are large
// (fewer grabs and table builds); on a small one (below 2^23 directed edges, where a count takes
// under about half a millisecond) a large piece is the tail: one warp's chain of dependent steps.
// Measured on R-MAT 16 (1.8 M directed edges): centres claimed 5 instead of 64 at a time 527 -> 291 us
// for the whole count, items of 512 and 64 edges instead of 4096 and 256 -> 264 us, orientation tiles
// of 8 vertices instead of 32 and hub chunks of 512 entries -> 222 us. On R-MAT 20 the same small items
// cost 1 % and tiles of 8 nothing, on Barabasi-Albert n = 2^22 3 % and 2 %.
void set_work_sizes(SchedParams& sp, int64_t n, int64_t m, int64_t item_cap) {
  const bool small = m < kSmallEdges;
  sp.cta_range = small ? 512 : 4096;
  sp.warp_range = small && item_cap >= Workspace::items_for(n, m, kItemRangeMin) ? kItemRangeMin : kItemRange;
  sp.hub_chunk = small ? kHubChunkMin : kHubChunk;
  // Vertices claimed at a time, where the caller gives no number: at least two claims per warp, at most
  // 16 (64: R-MAT 20 + 2 %, Erdos-Renyi n = 2^20 + 6 %; 1: 16384 vertices + 2 %, 90601 + 25 %).
  const int64_t warps = (int64_t)device_info().sms * kCtasPerSm * kWarps;
  if (sp.chunk == 0) sp.chunk = (int32_t)std::max<int64_t>(1, std::min<int64_t>(16, n / (2 * warps)));
  // Orientation tiles: 32 vertices, or on a graph of fewer tiles than warps as many as hold about 128
  // entries (four steps).
  sp.tile = kWarp;
  if (n < kWarp * warps)
    while (sp.tile > 4 && (int64_t)sp.tile / 2 * m >= 128 * n) sp.tile /= 2;
}

template <class View>
tc_status static_count(const View& view, int32_t n, int64_t m, Workspace& ws, int pv_mode, int32_t* per_vertex,
                       int64_t* triangles_dev, const SchedParams& sp0, cudaStream_t stream) {
  SchedParams sp = sp0;
  set_work_sizes(sp, n, m, ws.item_cap);
  if (sp.nshards > 1 && n > 0) TC_TRY(ws.ensure_shards(n));
  TC_CUDA_TRY(cudaMemsetAsync(ws.st, 0, sizeof(DevStatus), stream));
  if (pv_mode != TC_PV_NONE && n > 0)
    TC_CUDA_TRY(cudaMemsetAsync(per_vertex, 0, (pv_mode == TC_PV_HANDLE64 ? 8 : 4) * (size_t)n, stream));
  if (n > 0) {
    prof_mark(0, stream);
    TC_TRY(orient(view, n, ws, sp, true, stream));
    prof_mark(1, stream);
    uint32_t* out = reinterpret_cast<uint32_t*>(per_vertex);
    switch (pv_mode) {
      case TC_PV_NONE: TC_TRY(launch_count<TC_PV_NONE>(n, view.ind, ws, out, sp, stream)); break;
      case TC_PV_HANDLE: TC_TRY(launch_count<TC_PV_HANDLE>(n, view.ind, ws, out, sp, stream)); break;
      case TC_PV_CSR: TC_TRY(launch_count<TC_PV_CSR>(n, view.ind, ws, out, sp, stream)); break;
      case TC_PV_HANDLE64: TC_TRY(launch_count<TC_PV_HANDLE64>(n, view.ind, ws, out, sp, stream)); break;
      default: return fail(TC_ERR_INVALID_ARG, "unknown per-vertex mode %d", pv_mode);
    }
    prof_mark(2, stream);
    // k_find_hubs, k_orient, k_push_items, k_fill_items, k_count (+ k_shard_cost, three scan
    // kernels and k_shard_bounds when sharded)
    prof_launches(sp.nshards > 1 ? 10 : 5);
  }
  (void)m;
  if (triangles_dev)
    TC_CUDA_TRY(cudaMemcpyAsync(triangles_dev, &ws.st->triangles, sizeof(int64_t), cudaMemcpyDeviceToDevice, stream));
  return TC_OK;
}

template tc_status static_count<Csr32View>(const Csr32View&, int32_t, int64_t, Workspace&, int, int32_t*, int64_t*,
                                           const SchedParams&, cudaStream_t);
template tc_status static_count<Csr64View>(const Csr64View&, int32_t, int64_t, Workspace&, int, int32_t*, int64_t*,
                                           const SchedParams&, cudaStream_t);
template tc_status static_count<SlackView>(const SlackView&, int32_t, int64_t, Workspace&, int, int32_t*, int64_t*,
                                           const SchedParams&, cudaStream_t);

tc_status read_info(const Workspace& ws, cudaStream_t stream, tc_count_info* info) {
  DevStatus h;
  TC_CUDA_TRY(cudaMemcpyAsync(&h, ws.st, sizeof(DevStatus), cudaMemcpyDeviceToHost, stream));
  TC_CUDA_TRY(cudaStreamSynchronize(stream));
  info->triangles = (int64_t)h.triangles;
  info->edges_intersected = (int64_t)h.edges_intersected;
  info->oriented_work = (int64_t)h.oriented_work;
  info->max_out_degree = (int32_t)h.max_dplus;
  info->shard_lo = h.sharded ? (int32_t)h.shard_lo : 0;
  info->shard_hi = h.sharded ? (int32_t)h.shard_hi : -1;
  info->shard_work = (int64_t)h.shard_work;
  info->total_work = (int64_t)h.total_work;
  if (h.bad_flags & (kBadRange | kBadOrder | kBadSelfLoop)) {
    info->status = TC_ERR_BAD_GRAPH;
    return fail(TC_ERR_BAD_GRAPH, "graph check failed:%s%s%s", (h.bad_flags & kBadRange) ? " id out of range" : "",
                (h.bad_flags & kBadOrder) ? " list not strictly ascending" : "",
                (h.bad_flags & kBadSelfLoop) ? " self-loop" : "");
  }
  if (h.bad_flags & kBadCapacity) {
    info->status = TC_ERR_CAPACITY;
    return fail(TC_ERR_CAPACITY, "oriented graph exceeded its workspace");
  }
  if (h.sym_checksum != 0) {
    info->status = TC_ERR_NOT_SYMMETRIC;
    return fail(TC_ERR_NOT_SYMMETRIC, "adjacency is not symmetric");
  }
  info->status = TC_OK;
  return TC_OK;
}

namespace {
// Warp per source vertex: per degree-cell sums over its oriented edges, in shared memory, then
// one atomic per touched cell per CTA.
__global__ void __launch_bounds__(256) k_cell_stats(const int32_t n, const int32_t* __restrict__ dplus,
                                                    const int64_t* __restrict__ offp, const int32_t* __restrict__ indp,
                                                    double* __restrict__ out) {
  __shared__ double acc[256 * 4];
  for (int i = threadIdx.x; i < 256 * 4; i += blockDim.x) acc[i] = 0.0;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int64_t gw = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t uu = gw; uu < n; uu += nw) {
    const int32_t du = dplus[uu];
    const int64_t s = head_start(offp[uu]);
    for (int32_t k = lane; k < du; k += 32) {
      // the cell the count files the edge under: (centre's out-degree, the other endpoint's)
      const int32_t dv = dplus[indp[s + k]];
      const int32_t a = max(du, dv), b = min(du, dv);
      const int c = log2_cell(a) * 16 + log2_cell(b);
      atomicAdd(&acc[4 * c + 0], 1.0);
      atomicAdd(&acc[4 * c + 1], log2(1.0 + a));
      atomicAdd(&acc[4 * c + 2], log2(1.0 + b));
      atomicAdd(&acc[4 * c + 3], (double)b / (double)max(a, 1));
    }
  }
  __syncwarp();
  __syncthreads();
  for (int i = threadIdx.x; i < 256 * 4; i += blockDim.x)
    if (acc[i] != 0.0) atomicAdd(&out[i], acc[i]);
}
}  // namespace

tc_status cell_stats(int32_t n, Workspace& ws, double* out_host, cudaStream_t stream) {
  double* d = nullptr;
  TC_CUDA_TRY(::tc::dev_malloc(&d, sizeof(double) * 1024));
  cudaMemsetAsync(d, 0, sizeof(double) * 1024, stream);
  if (n > 0) k_cell_stats<<<orient_grid(n), 256, 0, stream>>>(n, ws.dplus, ws.offp, ws.indp, d);
  cudaError_t e = cudaMemcpyAsync(out_host, d, sizeof(double) * 1024, cudaMemcpyDeviceToHost, stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
  cudaFree(d);
  if (e != cudaSuccess) return fail(TC_ERR_CUDA, "cell stats: %s", cudaGetErrorString(e));
  return TC_OK;
}

template <class View>
tc_status validate_view(const View& view, int32_t n, int64_t m, Workspace& ws, cudaStream_t stream) {
  TC_CUDA_TRY(cudaMemsetAsync(ws.st, 0, sizeof(DevStatus), stream));
  SchedParams sp = to_params(nullptr);
  set_work_sizes(sp, n, m, ws.item_cap);
  if (n > 0) TC_TRY(orient(view, n, ws, sp, false, stream));
  return TC_OK;
}

template tc_status validate_view<SlackView>(const SlackView&, int32_t, int64_t, Workspace&, cudaStream_t);
template tc_status validate_view<Csr64View>(const Csr64View&, int32_t, int64_t, Workspace&, cudaStream_t);

}  // namespace tc

#ifdef TC_DEBUG_PROGRESS
extern "C" {
volatile int tc_dbg_host_stage = 0;
void* tc_dbg_progress_host_dev = nullptr;
size_t tc_dbg_progress_bytes = 0;
int tc_debug_get_stage(void) { return tc_dbg_host_stage; }
int tc_debug_set_progress(void* dev_ptr, size_t bytes, void* kern_dev_ptr) {
  unsigned long long* p = (unsigned long long*)dev_ptr;
  unsigned long long* k = (unsigned long long*)kern_dev_ptr;
  tc_dbg_progress_host_dev = dev_ptr;
  tc_dbg_progress_bytes = bytes;
  int e = (int)cudaMemcpyToSymbol(tc::tc_dbg_progress, &p, sizeof(p));
  if (e) return e;
  return (int)cudaMemcpyToSymbol(tc::tc_dbg_kern, &k, sizeof(k));
}
}
#endif
