// Triangle counting over an oriented adjacency (each edge kept once, at its
// lower-ranked end), shared by the PMA graph (traverse.cu) and the
// byte-width snapshot (compact.cu), which build the orientation each from
// their own rows.
#pragma once
#include <algorithm>
#include <cstdint>
#include <cuda_runtime.h>

#include "common.cuh"
#include "primitives.cuh"

namespace sst {
namespace {

// rank order used to orient each undirected edge once: (degree, id).  Each
// vertex keeps the neighbours that rank above it (N+), so a hub keeps only
// the few neighbours of even higher degree and the lists stay short; every
// triangle is counted once, at its lowest-ranked vertex.
__device__ __forceinline__ bool rank_less(const uint32_t *deg, uint32_t a,
                                          uint32_t b) {
  uint32_t da = deg[a], db = deg[b];
  return da < db || (da == db && a < b);
}
__device__ __forceinline__ bool ranks_above(const uint32_t *deg, uint32_t w,
                                            uint32_t u) {
  return rank_less(deg, u, w);
}

__device__ __forceinline__ bool sorted_has(const uint32_t *a, uint64_t n,
                                           uint32_t x) {
  uint64_t lo = 0, hi = n;
  while (lo < hi) {
    uint64_t mid = (lo + hi) >> 1;
    if (a[mid] < x)
      lo = mid + 1;
    else
      hi = mid;
  }
  return lo < n && a[lo] == x;
}

// A triangle is a common entry of the lists N+(x) and N+(y) of the ends of one
// of its edges (the end w above both), so the count is the sum, over edges, of
// |N+(x) n N+(y)|: one list goes into a hash set, the other is streamed past
// it.  The set is the longer list (its vertex x), the stream the shorter one:
// on an RMAT graph of 2^18 vertices that streams 96e6 entries where hashing
// the lower-ranked end's list streamed 204e6 (k_tc_count 678 -> 399 us).
// A list too long for the set is streamed past the other end's set if that one
// fits (tc_key), else probed by binary search.
//
// The count runs over work items: up to 32 neighbours y of one x.  A warp takes
// kTcGrab consecutive items at a time from a global cursor, so the serial work
// a warp can be left with at the end is a few items', whatever the degree
// distribution.  For an item the warp puts N+(x) into a hash set in its shared
// memory (kept while the next item has the same x), then reads the lists N+(y)
// of the item's edges that x counts as one flattened stream: lane i holds
// y_i's list bounds and the warp's inclusive prefix P of their lengths; stream
// item k lies in the first list i with P_i > k, which each lane tracks with a
// cursor that only moves forward (every lane's k grows by 32 a step); each
// lane issues kTcAhead loads before it probes the set, so a warp keeps
// kTcAhead * 32 list entries in flight.
constexpr uint32_t kTcSlots = 2048;  // set slots per warp (8 KiB)
constexpr int kTcBucketBits = 9;     // up to 2^9 buckets of 4 slots
constexpr uint32_t kTcBatch = 32;    // neighbours per work item
constexpr int kTcWarps = 8;          // warps per block
constexpr int kTcAhead = 4;          // stream items per lane in flight

// multiplicative hashing (Knuth): the top `bits` bits of x * 2^32/phi
__device__ __forceinline__ uint32_t tc_hash(uint32_t x, int bits) {
  return (x * 0x9E3779B1u) >> (32 - bits);
}

// The set: 2^bits buckets of four slots, one 16-byte shared load each.  An
// insert takes the first empty slot of its bucket (slots fill in order, so
// a bucket whose last slot is empty was never passed over), else moves on
// to the next bucket; a lookup stops at a match or at such a bucket.  At
// most half the slots are ever used, so every probe sequence ends.
__device__ __forceinline__ void tc_set_insert(uint4 *tab, uint32_t x, int bits) {
  uint32_t h = tc_hash(x, bits);
  const uint32_t mask = (1u << bits) - 1;
  for (;;) {
    uint32_t *b = reinterpret_cast<uint32_t *>(tab + h);
#pragma unroll
    for (int j = 0; j < 4; j++)
      if (atomicCAS(b + j, kEmpty, x) == kEmpty) return;
    h = (h + 1) & mask;
  }
}

// One lookup per lane, warp-uniform: every lane reads its home bucket; the
// warp loops on only while some lane met a full bucket without its match
// (rare: the set keeps at least two buckets per entry where it can), so the
// probes do not diverge.  Lanes with on = false look nothing up.
__device__ __forceinline__ bool tc_set_has_warp(const uint4 *tab, uint32_t w, int bits,
                                                bool on) {
  const uint32_t mask = (1u << bits) - 1;
  uint32_t h = tc_hash(w, bits);
  uint4 b = on ? tab[h] : make_uint4(0, 0, 0, kEmpty);
  bool hit = on && (b.x == w || b.y == w || b.z == w || b.w == w);
  bool more = on && !hit && b.w != kEmpty;
  while (__any_sync(0xffffffffu, more)) {
    if (more) {
      h = (h + 1) & mask;
      b = tab[h];
      hit = b.x == w || b.y == w || b.z == w || b.w == w;
      more = !hit && b.w != kEmpty;
    }
  }
  return hit;
}

// A vertex's oriented list as one word: (first entry << kTcLenBits) | length.
// |N+(v)| ids have at least v's degree, so |N+(v)|^2 <= m: 24 bits hold it up
// to 2^48 edges, and 40 bits the start.
constexpr int kTcLenBits = 24;
__device__ __forceinline__ uint32_t tc_len(uint64_t d) {
  return (uint32_t)d & ((1u << kTcLenBits) - 1);
}

// Which end of an edge takes the set: the one with the larger (key, id); a
// list that does not fit a set comes last.
__device__ __forceinline__ uint32_t tc_key(uint32_t len) {
  return len <= kTcSlots / 2 ? len : 0u;
}

// Work items over the leaves of a graph's leaf directory: an item is a leaf.
struct TcLeaves {
  static constexpr bool kOriented = false;
  const uint32_t *slots, *owner, *cnt;
  const uint64_t *slot;
  uint64_t n;
  struct Item {
    uint32_t x, cnt;
    uint64_t at;
  };
  __device__ __forceinline__ uint64_t count() const { return n; }
  __device__ __forceinline__ Item item(uint64_t k) const {
    return Item{owner[k], cnt[k], slot[k]};
  }
  __device__ __forceinline__ uint32_t id(uint64_t at) const { return slots[at]; }
};

// Work items over the rows of a CSR: an item is a batch of a row, listed as
// (batch << 32) | row; rows without an oriented list have none.
struct TcRows {
  static constexpr bool kOriented = false;
  const uint64_t *off;
  const uint32_t *cols;
  const uint64_t *items;
  const uint32_t *nitems;
  struct Item {
    uint32_t x, cnt;
    uint64_t at;
  };
  __device__ __forceinline__ uint64_t count() const { return *nitems; }
  __device__ __forceinline__ Item item(uint64_t k) const {
    const uint64_t it = items[k];
    const uint32_t x = (uint32_t)it;
    const uint64_t at = off[x] + (it >> 32) * kTcBatch, left = off[x + 1] - at;
    return Item{x, left < kTcBatch ? (uint32_t)left : kTcBatch, at};
  }
  __device__ __forceinline__ uint32_t id(uint64_t at) const { return cols[at]; }
};

// Work items over the oriented lists: an item is a batch of one, listed likewise;
// lists of one entry have none (no triangle has its lowest vertex there).
struct TcLists {
  static constexpr bool kOriented = true;
  const uint64_t *desc;
  const uint32_t *adj;
  const uint64_t *items;
  const uint32_t *nitems;
  struct Item {
    uint32_t x, cnt;
    uint64_t at;
  };
  __device__ __forceinline__ uint64_t count() const { return *nitems; }
  __device__ __forceinline__ Item item(uint64_t k) const {
    const uint64_t it = items[k];
    const uint32_t x = (uint32_t)it, b = (uint32_t)(it >> 32) * kTcBatch;
    const uint64_t d = desc[x];
    const uint32_t left = tc_len(d) - b;
    return Item{x, left < kTcBatch ? left : kTcBatch, (d >> kTcLenBits) + b};
  }
  __device__ __forceinline__ uint32_t id(uint64_t at) const { return adj[at]; }
};

// per row: its number of work items, of its own entries or (off null) of its
// oriented list's
__global__ void k_tc_items_count(const uint64_t *__restrict__ off,
                                 const uint64_t *__restrict__ desc, uint32_t n,
                                 uint32_t *__restrict__ cnt) {
  const uint64_t u = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (u >= n) return;
  const uint32_t len = tc_len(desc[u]);
  const uint64_t entries = off ? off[u + 1] - off[u] : len;
  cnt[u] = len >= (off ? 1u : 2u) ? (uint32_t)((entries + kTcBatch - 1) / kTcBatch) : 0u;
}

// per row: its items at its exclusive prefix ioff[u]
__global__ void k_tc_items_fill(const uint32_t *__restrict__ cnt,
                                const uint32_t *__restrict__ ioff, uint32_t n,
                                uint64_t *__restrict__ items) {
  const uint64_t u = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (u >= n) return;
  const uint32_t c = cnt[u], o = ioff[u];
  for (uint32_t j = 0; j < c; j++) items[(uint64_t)o + j] = ((uint64_t)j << 32) | u;
}

// The two forms of the count.  By lists, the items are the oriented lists N+(u) and
// the streams N+(v) of their entries v: every edge once, from its lower end.  By
// rows, the items are whole rows, every edge is met from both ends, and the end with
// the longer list takes the set: the streams are shorter, but the items are more than
// twice as many.  Which is less work depends on whether the two lists differ: on
// uniform graphs the upper end's is the shorter already.  So a sample of the kept
// edges adds up what either would stream.  Times by rows / by lists (us), and the
// rows' share of the lists' streams:
//   RMAT a = .57, 2^18 vertices    494   773   .48     a = .40, 2^20    2265  2129   .72
//   a = .45, 2^18                  336   354   .63     a = .35, 2^18     286   271   .83
//   uniform 1e5, 6.4e6 stored      461   414   .99     2^22, 6.7e7      3412  3144   .97
//   path of 2e6 (no stream)        501   325    -      complete, 1500   5566 12231  1.68
// A probe of a list too long for the set is a binary search, some 20 times a hashed
// one's time (the complete graph's share, weighed so, is .52); with counts by
// vertex the atomics hide most of that (47.5 / 37.0 ms).
constexpr uint32_t kTcSortedCost = 16, kTcSortedCostPv = 4;

// the kept edges (x, y), x the lower end, of a graph's leaves and of oriented lists
struct TcKeptLeaves {
  const uint32_t *slots, *owner;
  const uint64_t *slot;
  const uint32_t *kmask;
  uint64_t n;
  template <class F>
  __device__ __forceinline__ void each(uint64_t k, int lane, F f) const {
    if ((kmask[k] >> lane) & 1u) f(owner[k], slots[slot[k] + lane]);
  }
};
struct TcKeptLists {
  const uint64_t *desc;
  const uint32_t *adj;
  uint64_t n;
  template <class F>
  __device__ __forceinline__ void each(uint64_t k, int lane, F f) const {
    const uint64_t d = desc[k];
    for (uint32_t i = lane; i < tc_len(d); i += 32) f((uint32_t)k, adj[(d >> kTcLenBits) + i]);
  }
};

// Block b: est[2b] = the cost of the rows' form over the edges of its items, est[2b + 1]
// = the lists' form's; est[2 * kTcSampleBlocks] = *also, a word the host reads with them.
// A warp an item, every step-th one; sums a block, as atomics on one address queue.
constexpr int kTcSampleBlocks = 28, kTcSampleThreads = 1024;
constexpr uint64_t kTcSamples = kTcSampleBlocks * (kTcSampleThreads / 32);
constexpr int kTcSampleWords = 2 * kTcSampleBlocks + 1;
template <class Kept>
__global__ void __launch_bounds__(kTcSampleThreads)
k_tc_sample(Kept src, const uint64_t *__restrict__ desc, uint64_t step, uint32_t sorted_cost,
            const uint64_t *__restrict__ also, unsigned long long *__restrict__ est) {
  __shared__ unsigned long long s_est[2];
  if (threadIdx.x < 2) s_est[threadIdx.x] = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const uint64_t k = (((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * step;
  unsigned long long rows = 0, lists = 0;
  if (k < src.n)
    src.each(k, lane, [&](uint32_t x, uint32_t y) {
      const uint32_t lx = tc_len(desc[x]), ly = tc_len(desc[y]);
      auto cost = [&](uint32_t set, uint32_t stream) {
        return (unsigned long long)stream * (tc_key(set) ? 1u : sorted_cost);
      };
      if (lx < 2) return;
      lists += cost(lx, ly);
      const uint32_t kx = tc_key(lx), ky = tc_key(ly);
      const bool by_x = kx > ky || (kx == ky && x > y);
      if (ly) rows += by_x ? cost(lx, ly) : cost(ly, lx);
    });
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) {
    rows += __shfl_xor_sync(0xffffffffu, rows, d);
    lists += __shfl_xor_sync(0xffffffffu, lists, d);
  }
  if (lane == 0 && lists) {
    atomicAdd(&s_est[0], rows);
    atomicAdd(&s_est[1], lists);
  }
  __syncthreads();
  if (threadIdx.x < 2) est[2 * blockIdx.x + threadIdx.x] = s_est[threadIdx.x];
  if (blockIdx.x == 0 && threadIdx.x == 2 && also) est[2 * kTcSampleBlocks] = *also;
}
template <class Kept>
inline void tc_sample_launch(const Kept &src, const uint64_t *desc, bool pv, const uint64_t *also,
                             unsigned long long *est, cudaStream_t s) {
  SST_LAUNCH(k_tc_sample<Kept>, kTcSampleBlocks, kTcSampleThreads, 0, s, src, desc,
             (src.n + kTcSamples - 1) / kTcSamples, pv ? kTcSortedCostPv : kTcSortedCost, also, est);
}
// Whether a count of so many items by rows (leaves, or rows and started batches) takes
// the rows' form unseen: it is done in about the time of the sample and of the launches
// that list the oriented lists' items (uniform graphs of 22,000, 40,000 and 60,000
// vertices with 6 edges each: 71, 75 and 84 us by rows and 78, 91 and 93 by lists;
// of 90,000, 97 and 110, but by vertex 127 and 134 and from there on lists come nearer).
// Where rows are long the sample sees work that hides in the rows' form (1500 vertices
// with 350 edges each: 282 us by rows, 416 by the lists that the sample takes); by
// vertex the lists' fewer atomics count there (698 us, rows 775; 1000 vertices with
// 550 edges each 2663 and 2992).
inline bool tc_few_items(uint64_t items) { return items <= 1u << 16; }
// Whether the rows' form is the one to take, by the sample's sums (host memory).
template <class Word>
inline bool tc_by_rows(const Word *est) {
  uint64_t rows = 0, lists = 0;
  for (int b = 0; b < kTcSampleBlocks; b++) rows += est[2 * b], lists += est[2 * b + 1];
  return rows < lists / 100 * 68;
}

// items a warp takes per visit to the cursor; their descriptors load in
// parallel, one per lane
constexpr int kTcGrab = 8;

// position of the set bit of m with i set bits below it (32 if there is none)
__device__ __forceinline__ int tc_nth_bit(uint32_t m, int i) {
  int p = 0;
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) {
    const int c = __popc(m & (((1u << d) - 1u) << p));
    if (i >= c) {
      i -= c;
      p += d;
    }
  }
  return (m >> p) & 1u && i == 0 ? p : 32;
}

// PV: also count, per vertex, the triangles it is in
template <bool PV, class Items>
__global__ void __launch_bounds__(kTcWarps * 32, 3)
k_tc_count(Items src, const uint64_t *__restrict__ desc, const uint32_t *__restrict__ adj,
           unsigned long long *__restrict__ total, unsigned long long *__restrict__ pv) {
  extern __shared__ uint4 tc_sh[];
  const int lane = threadIdx.x & 31;
  const uint32_t full = 0xffffffffu;
  uint4 *tab = tc_sh + (threadIdx.x >> 5) * (kTcSlots / 4);
  const uint64_t Q = src.count();
  unsigned long long local = 0;
  uint32_t set_u = kEmpty;  // the x whose N+ the set holds
  for (;;) {
    unsigned long long q0 = 0;
    if (lane == 0) q0 = atomicAdd(total + 1, (unsigned long long)kTcGrab);
    q0 = __shfl_sync(full, q0, 0);
    if (q0 >= Q) break;
    // lane g < kTcGrab: item q0 + g and its x's list
    typename Items::Item my{0, 0, 0};
    uint64_t my_d = 0;
    if (lane < kTcGrab && q0 + lane < Q) {
      my = src.item(q0 + lane);
      my_d = desc[my.x];
    }
    const int ng = (int)((Q - q0) < (unsigned long long)kTcGrab ? (Q - q0) : kTcGrab);
    // The item's y (stage 1) and their lists (stage 2) load ahead: y two items
    // before the item's turn, the lists one item before (they need y), so a
    // small item's three dependent loads overlap earlier items.  An x without
    // a list (of two entries, if it is the lower end) has nothing to load.
    auto load_y = [&](int g, bool &ok) -> uint32_t {
      const uint64_t at = __shfl_sync(full, my.at, g & 31);
      const uint32_t c = __shfl_sync(full, my.cnt, g & 31);
      const uint64_t d = __shfl_sync(full, my_d, g & 31);
      ok = g < ng && (uint32_t)lane < c && tc_len(d) >= (Items::kOriented ? 2u : 1u);
      return ok ? src.id(at + lane) : 0u;
    };
    bool ok_n1 = false, ok_n2 = false;
    uint32_t v_n1 = load_y(0, ok_n1);  // item gi's y
    uint32_t v_n2 = load_y(1, ok_n2);  // item gi + 1's y
    uint64_t d_n1 = ok_n1 ? desc[v_n1] : 0;
    for (int gi = 0; gi < ng; gi++) {
      const uint32_t u = __shfl_sync(full, my.x, gi);
      const uint64_t ud = __shfl_sync(full, my_d, gi);
      const uint32_t na = tc_len(ud);
      const uint32_t *A = adj + (ud >> kTcLenBits);
      // this lane's y and its list, loaded ahead; of rows, x counts the edge if its
      // own list is the set's
      uint32_t v = v_n1;
      uint64_t b0 = d_n1 >> kTcLenBits;
      uint32_t len = ok_n1 ? tc_len(d_n1) : 0u;
      if (!Items::kOriented) {
        const uint32_t kx = tc_key(na), ky = tc_key(len);
        if (ky > kx || (ky == kx && v >= u)) len = 0;  // v == u: a stored self-loop
        // the lower end's list holds the other end and, in a triangle, one more
        if (na < 2 && len < 2) len = 0;
      }
      // the next items' loads go out before this item's work
      bool ok_n3 = false;
      const uint32_t v_n3 = load_y(gi + 2, ok_n3);
      ok_n1 = ok_n2;
      v_n1 = v_n2;
      d_n1 = ok_n2 ? desc[v_n2] : 0;
      ok_n2 = ok_n3;
      v_n2 = v_n3;
      const uint32_t act = __ballot_sync(full, len != 0);
      if (!act) continue;
      if (!Items::kOriented) {  // the edges that x counts to the front: the stream's
                                // cursor steps over no empty list
        const int from = tc_nth_bit(act, lane);
        v = __shfl_sync(full, v, from & 31);
        b0 = __shfl_sync(full, b0, from & 31);
        len = __shfl_sync(full, len, from & 31);
        if (lane >= __popc(act)) len = 0;
      }
      const bool hashed = na <= kTcSlots / 2;
      int bits = 3;
      while (bits < kTcBucketBits && (1ull << bits) < 2 * na) bits++;
      if (hashed && u != set_u) {
        __syncwarp();  // the last item's lookups are done
        for (uint32_t i = lane; i < (1u << bits); i += 32)
          tab[i] = make_uint4(kEmpty, kEmpty, kEmpty, kEmpty);
        __syncwarp();
        for (uint64_t i = lane; i < na; i += 32) tc_set_insert(tab, A[i], bits);
        __syncwarp();
        set_u = u;
      }
      // inclusive prefix of the lengths: 32 of kTcLenBits bits
      uint32_t P = len;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const uint32_t y = __shfl_up_sync(full, P, d);
        if (lane >= d) P += y;
      }
      const uint32_t T = __shfl_sync(full, P, 31);
      // item k of list i sits at adj[base_i + k], base_i = b0_i - (P_i - len_i)
      const uint64_t base = b0 - (uint64_t)(P - len);
      int cur = 0;  // this lane's list; P_31 = T > k keeps it below 32
      uint32_t cend = __shfl_sync(full, P, 0);
      uint64_t cb = __shfl_sync(full, base, 0);
      uint32_t cvx = PV ? __shfl_sync(full, v, 0) : 0u;
      unsigned long long cu = 0;
      for (uint32_t k0 = 0; k0 < T; k0 += 32 * kTcAhead) {
        uint32_t w[kTcAhead], vv[kTcAhead];
#pragma unroll
        for (int t = 0; t < kTcAhead; t++) {
          w[t] = kEmpty;
          vv[t] = 0;
          if (k0 + 32 * t >= T) continue;  // uniform: the stream ended
          const uint32_t k = k0 + 32 * t + lane;
          bool adv = k < T && k >= cend;
          while (__any_sync(full, adv)) {
            cur += adv ? 1 : 0;
            cend = __shfl_sync(full, P, cur);
            cb = __shfl_sync(full, base, cur);
            if (PV) cvx = __shfl_sync(full, v, cur);
            adv = k < T && k >= cend;
          }
          if (k < T) w[t] = adj[cb + k];  // ids are below n <= 2^32 - 1
          vv[t] = cvx;
        }
#pragma unroll
        for (int t = 0; t < kTcAhead; t++) {
          if (k0 + 32 * t >= T) continue;  // uniform
          const bool on = w[t] != kEmpty;
          bool hit;
          if (hashed) {
            hit = tc_set_has_warp(tab, w[t], bits, on);
          } else {
            hit = on && sorted_has(A, na, w[t]);
          }
          if (hit) {
            cu++;
            if (PV) {
              atomicAdd(&pv[w[t]], 1ull);
              atomicAdd(&pv[vv[t]], 1ull);
            }
          }
        }
      }
      if (PV) {
        unsigned long long c = cu;
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) c += __shfl_xor_sync(full, c, d);
        if (lane == 0 && c) atomicAdd(&pv[u], c);
      }
      local += cu;
    }
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) local += __shfl_down_sync(full, local, d);
  if (lane == 0 && local) atomicAdd(total, local);
}

// an item per started batch of 32 of a list: sum ceil(len / 32) <= madj / 32 + n,
// and, of lists of two entries or more, <= madj / 2
inline uint64_t tc_items_bound(uint32_t n, uint64_t madj) {
  return std::min<uint64_t>(madj / kTcBatch + n, madj / 2) + 1;
}

// The items of the oriented lists (madj entries in all): cnt and ioff hold n + 1
// entries each, items tc_items_bound(n, madj); the arena scan_scratch_bytes(n + 1, 4).
inline cudaError_t tc_list_items(const uint64_t *desc, const uint32_t *adj, uint32_t n,
                                 uint64_t madj, uint32_t *cnt, uint32_t *ioff, uint64_t *items,
                                 Arena &arena, cudaStream_t s, TcLists *out) {
  if (tc_items_bound(n, madj) >= (1ull << 32)) return cudaErrorInvalidValue;
  const unsigned blocks = (unsigned)(((uint64_t)n + 255) / 256);
  SST_LAUNCH(k_tc_items_count, blocks, 256, 0, s, (const uint64_t *)nullptr, desc, n, cnt);
  cudaError_t e = scan<uint32_t, OpAdd>(cnt, ioff, n, 0u, OpAdd{}, true, false, ioff + n, arena, s);
  if (e != cudaSuccess) return e;
  SST_LAUNCH(k_tc_items_fill, blocks, 256, 0, s, cnt, ioff, n, items);
  *out = TcLists{desc, adj, items, ioff + n};
  return cudaSuccess;
}

// Counts the triangles of the oriented lists desc[n] / adj over the items of
// src.  total (device) holds two counters the caller zeroes: total[0] gets the
// count, total[1] is the work cursor.  pv (device, zeroed, may be null) gets
// per-vertex counts.  One persistent grid of as many blocks as fit.
template <class Items>
inline cudaError_t tc_count_launch(const Items &src, const uint64_t *desc, const uint32_t *adj,
                                   unsigned long long *total, unsigned long long *pv,
                                   int sms, cudaStream_t s) {
  const size_t shm = (size_t)kTcWarps * kTcSlots * 4;
  auto kern = pv ? k_tc_count<true, Items> : k_tc_count<false, Items>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shm);
  if (e != cudaSuccess) return e;
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kTcWarps * 32, shm);
  if (e != cudaSuccess) return e;
  const unsigned grid = (unsigned)(std::max(per_sm, 1) * sms);
  if (pv)
    SST_LAUNCH_NB("k_tc_count<true>", 0, (k_tc_count<true, Items>), grid, kTcWarps * 32, shm, s,
                  src, desc, adj, total, pv);
  else
    SST_LAUNCH_NB("k_tc_count<false>", 0, (k_tc_count<false, Items>), grid, kTcWarps * 32, shm, s,
                  src, desc, adj, total, pv);
  return cudaGetLastError();
}

}  // namespace
}  // namespace sst
