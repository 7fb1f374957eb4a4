// Breadth-first search as one cooperative launch: every level of the
// traversal, push or pull, runs in one grid, with a grid barrier where a
// launch per step had a host readback per level.
//
// Why one launch.  A level is a few dependent steps of a few microseconds on
// all but the two or three widest levels, and each step launched by the host
// costs as much again, with a readback to learn the next frontier's size: a
// graph of 2^14 vertices took 190 us for five levels, now 63 us.  Here the sizes
// stay on the device, every block takes the same decision from the same
// counters, and a step costs a barrier (1.5 us).  The widest levels are bound by
// memory: on an RMAT graph of 2^23 vertices and 1.3e8 stored edges (1007 us
// before, 334 us now) the first pull reads its one-leaf rows in 56 us, about
// 270 MB of lists, depths and row sectors.
//
// The grid is one that fits at once (cooperative), and no larger than the
// graph has work for: blocks beyond that only make the barrier wider.  Two
// blocks hold all of an SM's registers, so the largest grid leaves kCoopFree
// block places to the kernels of other streams: a served graph is updated while
// it is searched, and an update's small kernels would otherwise wait for the
// search to end.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "common.cuh"
#include "gridbarrier.h"
#include "primitives.cuh"

namespace sst {
namespace {

constexpr int kCoopThreads = 512;
constexpr int kCoopPerSm = 2;  // blocks of an SM
constexpr int kCoopFree = 16;  // block places left free
constexpr uint32_t kFull = 0xffffffffu;

// ------------------------------------------------------------ grid barrier
// Barrier over a cooperative grid: a counter that every block raises once a
// step.  Thread 0's fences order the block's writes before the step and its
// reads after it (device scope, as the block barrier around them makes the
// order hold for every thread).  The wait is bounded: a block that gives up
// sets *err, which every block reads after each barrier and leaves on, so the
// kernel ends whatever happens.
constexpr unsigned long long kBarrierWaitNs = 20ull * 1000 * 1000 * 1000;

struct GridBarrier {
  BarrierCount *count;  // zero at launch
  unsigned int *err;    // zero at launch
  BarrierCount target;  // arrivals that complete the last barrier (0: none yet)

  // false: some block gave up, leave the kernel
  __device__ __forceinline__ bool wait() {
    __shared__ unsigned int s_err;
    __syncthreads();
    target = barrier_next(target, gridDim.x);
    if (threadIdx.x == 0) {
      __threadfence();
      atomicAdd(count, BarrierCount{1});
      unsigned long long t0 = 0;
      for (uint32_t spin = 0; !barrier_complete(*(volatile BarrierCount *)count, target); spin++) {
        if ((spin & 1023u) != 1023u) continue;
        if (*(volatile unsigned int *)err) break;  // a block may have left already
        unsigned long long t;
        asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
        if (t0 == 0) t0 = t;
        if (t - t0 > kBarrierWaitNs) {
          atomicExch(err, 1u);
          break;
        }
      }
      __threadfence();
      s_err = *(volatile unsigned int *)err;
    }
    __syncthreads();
    return s_err == 0;
  }
};

// a launch of a cooperative grid: all its blocks are resident at once
template <typename... KArgs, typename... Args>
inline cudaError_t launch_coop(const char *name, void (*kernel)(KArgs...), unsigned grid,
                               unsigned block, cudaStream_t s, Args... args) {
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.stream = s;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  cudaEvent_t ev = profiling(name) ? prof_begin(s) : nullptr;
  cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
  note_launch();
  if (ev) prof_end(name, ev, s, 0);
  return e;
}

// ------------------------------------------------------------ the traversal
constexpr uint32_t kBfsLeaves = 4;  // leaves of a push item of a multi-leaf row: one batch of loads

// push items of a multi-leaf row
__device__ __forceinline__ uint32_t bfs_items(uint32_t cap) {
  return ((cap >> kLeafLog) + kBfsLeaves - 1) / kBfsLeaves;
}

// the lane whose inclusive prefix P is the first above k (31 if none is)
__device__ __forceinline__ int warp_owner(uint32_t P, uint32_t k) {
  int r = 0;
#pragma unroll
  for (int d = 16; d > 0; d >>= 1)
    if (__shfl_sync(kFull, P, r + d - 1) <= k) r += d;
  return r;
}

// counters of one level's frontier (three sets, used in turn: one is read,
// one is added to, one is cleared)
struct BfsCount {
  unsigned long long vertices, degrees;
  unsigned int rows, bigs, items;  // its one-leaf and multi-leaf rows, their items
};
// device state of a search, zero at launch; the last block to leave zeroes it
// again (no clearing launch before the next search)
struct BfsCtl {
  BarrierCount bar;
  unsigned int err;
  unsigned int rows, bigs, items;  // tails of the queues
  unsigned int left;               // blocks that have left
  BfsCount cnt[3];
};

struct BfsArgs {
  DGraph g;
  uint64_t m;          // stored edges
  uint32_t src, alpha; // pull once (frontier + its edges) * alpha > m
  const uint32_t *small;             // one-leaf rows, ascending ids
  const unsigned long long *sdesc;   // (first slot << 6) | degree of each
  uint64_t nsmall;
  const uint32_t *cv;                // multi-leaf rows in chunks of leaves:
  const unsigned long long *cdesc;   // (first leaf << 8) | .. | leaves
  uint64_t nchunks;
  int32_t *depth;
  int32_t *parent;                   // may be null
  uint32_t *bits;                    // frontier bitmap of a pull, n / 32 + 1 words
  uint32_t *queue;                   // n entries: one-leaf rows of all levels from
                                     // the front, multi-leaf rows from the back
  unsigned long long *qitems;        // (first leaf << 32) | row, max_items entries
  uint64_t max_items;
  BfsCtl *ctl;
  unsigned long long *result;        // pinned host word: the search's error, 0 = none
};

// entry r of the one-leaf rows, or of the multi-leaf rows.  The queue holds
// each row once, so it cannot overflow; an index beyond it is an error all the
// same, not a write.
__device__ __forceinline__ void bfs_put(const BfsArgs &a, bool big, uint32_t r, uint32_t v) {
  if (r < a.g.n)
    a.queue[big ? a.g.n - 1 - r : r] = v;
  else
    a.ctl->err = 2;
}

// The warp's newly reached rows (a lane's rows v[t] with bit t of mine set) to
// the queue, with one reservation an end for the whole batch.  Every lane
// calls it.
template <int N>
__device__ __forceinline__ void bfs_enqueue(const BfsArgs &a, uint32_t mine,
                                            const uint32_t (&v)[N], const uint32_t (&cap)[N]) {
  const int lane = threadIdx.x & 31;
  uint32_t sm[N], bm[N], nrows = 0, nbigs = 0;
#pragma unroll
  for (int t = 0; t < N; t++) {
    const bool on = (mine >> t) & 1u;
    sm[t] = __ballot_sync(kFull, on && cap[t] <= kLeaf);
    bm[t] = __ballot_sync(kFull, on && cap[t] > kLeaf);
    nrows += __popc(sm[t]);
    nbigs += __popc(bm[t]);
  }
  uint32_t at = 0;  // both tails at once, a lane each
  if (lane == 0 && nrows) at = atomicAdd(&a.ctl->rows, nrows);
  if (lane == 1 && nbigs) at = atomicAdd(&a.ctl->bigs, nbigs);
  uint32_t r = __shfl_sync(kFull, at, 0), b = __shfl_sync(kFull, at, 1);
  const uint32_t lt = (1u << lane) - 1u;
#pragma unroll
  for (int t = 0; t < N; t++) {
    if ((sm[t] >> lane) & 1u) bfs_put(a, false, r + __popc(sm[t] & lt), v[t]);
    if ((bm[t] >> lane) & 1u) bfs_put(a, true, b + __popc(bm[t] & lt), v[t]);
    r += __popc(sm[t]);
    b += __popc(bm[t]);
  }
}

// The items of the queued multi-leaf rows [b, e): a warp takes up to 32 rows
// and writes their items as one flattened list.  Only a level that is pushed
// from needs them (the first levels of a search from a hub find hubs of
// thousands of leaves each and are then pulled: writing their items as they
// were found took 37 us on an RMAT scale-23 graph).
__device__ __forceinline__ void bfs_list_items(const BfsArgs &a, uint32_t b, uint32_t e) {
  const int lane = threadIdx.x & 31;
  const uint32_t nw = (gridDim.x * kCoopThreads) >> 5;
  const uint32_t w0 = (blockIdx.x * kCoopThreads + threadIdx.x) >> 5;
  uint32_t per = (e - b + nw - 1) / nw;
  per = per > 32 ? 32 : per;
  for (uint64_t i0 = b + (uint64_t)w0 * per; i0 < e; i0 += (uint64_t)nw * per) {
    const bool in = (uint32_t)lane < per && i0 + lane < e;
    const uint32_t v = in ? a.queue[a.g.n - 1 - (i0 + lane)] : 0u;
    const uint32_t k = in ? bfs_items(a.g.cap[v]) : 0u;
    const uint32_t P = warp_inclusive(k, OpAdd{});
    const uint32_t T = __shfl_sync(kFull, P, 31);
    uint32_t at = 0;
    if (lane == 0) at = atomicAdd(&a.ctl->items, T);
    at = __shfl_sync(kFull, at, 0);
    for (uint32_t j0 = 0; j0 < T; j0 += 32) {
      const uint32_t j = j0 + lane;
      const int r = warp_owner(P, j);
      const uint32_t row = __shfl_sync(kFull, v, r);
      const uint32_t first = __shfl_sync(kFull, P - k, r);
      if (j >= T) continue;
      if ((uint64_t)at + j < a.max_items)
        a.qitems[at + j] = ((unsigned long long)((j - first) * kBfsLeaves) << 32) | row;
      else
        a.ctl->err = 2;
    }
  }
}

// a thread's part of the next level's counts
struct BfsSum {
  unsigned long long vertices = 0, degrees = 0;
  unsigned int bigs = 0, items = 0;
  __device__ __forceinline__ void add(uint32_t deg, uint32_t cap) {
    vertices++;
    degrees += deg;
    if (cap > kLeaf) {
      bigs++;
      items += bfs_items(cap);
    }
  }
};

constexpr int kBfsAhead = 4;  // edges of a lane in flight in a push

// The ends w[t] (kEmpty: none) of a warp's edges, from rows u[t], claimed for
// level lvl + 1 and queued: each stage's loads and atomics for all of a lane's
// edges go out before any is used.
__device__ __forceinline__ void bfs_reach(const BfsArgs &a, const uint32_t (&w)[kBfsAhead],
                                          const uint32_t (&u)[kBfsAhead], int lvl, BfsSum &sum) {
  int32_t dw[kBfsAhead];
#pragma unroll
  for (int t = 0; t < kBfsAhead; t++) dw[t] = w[t] != kEmpty ? a.depth[w[t]] : 0;
#pragma unroll
  for (int t = 0; t < kBfsAhead; t++)
    if (dw[t] < 0) dw[t] = atomicCAS(&a.depth[w[t]], -1, lvl + 1) == -1 ? -1 : 0;
  uint32_t mine = 0;
#pragma unroll
  for (int t = 0; t < kBfsAhead; t++) mine |= dw[t] < 0 ? 1u << t : 0u;
  if (!__any_sync(kFull, mine)) return;
  uint32_t cap[kBfsAhead], deg[kBfsAhead];
#pragma unroll
  for (int t = 0; t < kBfsAhead; t++) {
    const bool on = (mine >> t) & 1u;
    cap[t] = on ? a.g.cap[w[t]] : 0u;
    deg[t] = on ? a.g.deg[w[t]] : 0u;
    if (on && a.parent) a.parent[w[t]] = (int32_t)u[t];
  }
#pragma unroll
  for (int t = 0; t < kBfsAhead; t++)
    if ((mine >> t) & 1u) sum.add(deg[t], cap[t]);
  bfs_enqueue(a, mine, w, cap);
}

// Push from the queued one-leaf rows [b, e): a warp takes up to 32 rows and
// walks their edges as one flattened stream (edge k belongs to the first row
// whose inclusive degree prefix exceeds k), so rows of a few ids keep every
// lane busy: a warp a row spent 401 us on a level of 1.4e6 rows of an RMAT
// scale-23 graph.  Few rows go to more warps, down to one row each.
__device__ __forceinline__ void bfs_push_rows(const BfsArgs &a, uint32_t b, uint32_t e, int lvl,
                                              BfsSum &sum) {
  const int lane = threadIdx.x & 31;
  const uint32_t nw = (gridDim.x * kCoopThreads) >> 5;
  const uint32_t w0 = (blockIdx.x * kCoopThreads + threadIdx.x) >> 5;
  uint32_t per = (e - b + nw - 1) / nw;
  per = per > 32 ? 32 : per;
  for (uint64_t i0 = b + (uint64_t)w0 * per; i0 < e; i0 += (uint64_t)nw * per) {
    const bool in = (uint32_t)lane < per && i0 + lane < e;
    const uint32_t u = in ? a.queue[i0 + lane] : 0u;
    const uint64_t base = in ? a.g.base[u] : 0ull;
    const uint32_t deg = in ? a.g.deg[u] : 0u;
    const uint32_t P = warp_inclusive(deg, OpAdd{});
    const uint32_t T = __shfl_sync(kFull, P, 31);
    const uint64_t first = base - (P - deg);  // edge k of row i is slot first_i + k
    for (uint32_t k0 = 0; k0 < T; k0 += 32 * kBfsAhead) {
      uint32_t w[kBfsAhead], uu[kBfsAhead];
#pragma unroll
      for (int t = 0; t < kBfsAhead; t++) {
        const uint32_t k = k0 + 32 * t + lane;
        const int r = warp_owner(P, k);
        const uint64_t f = __shfl_sync(kFull, first, r);
        uu[t] = __shfl_sync(kFull, u, r);
        w[t] = k < T ? a.g.slots[f + k] : kEmpty;
      }
      bfs_reach(a, w, uu, lvl, sum);
    }
  }
}

// Push from the queued items [b, e) of multi-leaf rows: a warp an item, lane =
// slot, its leaves at once.  A leaf's slots past its ids hold kEmpty, so no
// counts are read.
__device__ __forceinline__ void bfs_push_items(const BfsArgs &a, uint32_t b, uint32_t e, int lvl,
                                               BfsSum &sum) {
  const int lane = threadIdx.x & 31;
  const uint32_t nw = (gridDim.x * kCoopThreads) >> 5;
  const uint32_t w0 = (blockIdx.x * kCoopThreads + threadIdx.x) >> 5;
  for (uint64_t i = b + (uint64_t)w0; i < e; i += nw) {
    const unsigned long long it = a.qitems[i];
    const uint32_t u = (uint32_t)it, l0 = (uint32_t)(it >> 32);
    const uint64_t base = a.g.base[u];
    const uint32_t l1 = min(l0 + kBfsLeaves, a.g.cap[u] >> kLeafLog);
    static_assert(kBfsAhead == (int)kBfsLeaves, "an item is one batch");
    uint32_t w[kBfsAhead], uu[kBfsAhead];
#pragma unroll
    for (int t = 0; t < kBfsAhead; t++) {
      w[t] = l0 + t < l1 ? a.g.slots[base + ((uint64_t)(l0 + t) << kLeafLog) + lane] : kEmpty;
      uu[t] = u;
    }
    bfs_reach(a, w, uu, lvl, sum);
  }
}

// The frontier bitmap of a pull at level lvl, from the depths: a stream of 4
// bytes a vertex, no queue, no atomics, nothing to clear.
constexpr int kBfsWords = 8;  // words of a warp in flight
__device__ __forceinline__ void bfs_level_bits(const BfsArgs &a, int lvl) {
  const int lane = threadIdx.x & 31;
  const uint32_t nw = (gridDim.x * kCoopThreads) >> 5;
  const uint32_t w0 = (blockIdx.x * kCoopThreads + threadIdx.x) >> 5;
  const uint32_t words = a.g.n / 32 + 1;
  for (uint64_t i = (uint64_t)w0 * kBfsWords; i < words; i += (uint64_t)nw * kBfsWords) {
    int32_t d[kBfsWords];
#pragma unroll
    for (int k = 0; k < kBfsWords; k++) {
      const uint64_t v = (i + k) * 32 + lane;
      d[k] = v < a.g.n ? a.depth[v] : -1;
    }
#pragma unroll
    for (int k = 0; k < kBfsWords; k++) {
      const uint32_t m = __ballot_sync(kFull, d[k] == lvl);
      if (lane == 0 && i + k < words) a.bits[i + k] = m;
    }
  }
}

// The rows of level lvl to the queue, for the push after a pull.  A warp takes
// a contiguous range of the depths and counts its rows first, so a block
// reserves once for all of them: with a reservation a warp and word, the two
// tails' atomics took 182 us for 1.4e6 rows of 8.4e6 vertices.
__device__ __forceinline__ void bfs_queue_level(const BfsArgs &a, int lvl) {
  constexpr int kWarps = kCoopThreads / 32;
  __shared__ uint32_t s_rows[kWarps], s_bigs[kWarps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t words = a.g.n / 32 + 1;
  const uint32_t nw = gridDim.x * kWarps, w = blockIdx.x * kWarps + warp;
  const uint32_t i0 = (uint32_t)((uint64_t)words * w / nw);
  const uint32_t i1 = (uint32_t)((uint64_t)words * (w + 1) / nw);
  uint32_t rows = 0, bigs = 0;
  for (int pass = 0; pass < 2; pass++) {
    for (uint32_t i = i0; i < i1; i += kBfsWords) {
      int32_t d[kBfsWords];
#pragma unroll
      for (int k = 0; k < kBfsWords; k++) {
        const uint64_t v = (uint64_t)(i + k) * 32 + lane;
        d[k] = i + k < i1 && v < a.g.n ? a.depth[v] : -1;
      }
      uint32_t cap[kBfsWords];
#pragma unroll
      for (int k = 0; k < kBfsWords; k++)
        cap[k] = d[k] == lvl ? a.g.cap[(i + k) * 32 + lane] : 0u;
#pragma unroll
      for (int k = 0; k < kBfsWords; k++) {
        const uint32_t sm = __ballot_sync(kFull, d[k] == lvl && cap[k] <= kLeaf);
        const uint32_t bm = __ballot_sync(kFull, cap[k] > kLeaf);
        const uint32_t v = (i + k) * 32 + lane;
        if (pass && (sm >> lane) & 1u)
          bfs_put(a, false, rows + __popc(sm & ((1u << lane) - 1u)), v);
        if (pass && (bm >> lane) & 1u)
          bfs_put(a, true, bigs + __popc(bm & ((1u << lane) - 1u)), v);
        rows += __popc(sm);
        bigs += __popc(bm);
      }
    }
    if (pass) break;
    if (lane == 0) {
      s_rows[warp] = rows;
      s_bigs[warp] = bigs;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      uint32_t r = 0, t = 0;
      for (int k = 0; k < kWarps; k++) {
        const uint32_t x = s_rows[k], y = s_bigs[k];
        s_rows[k] = r;
        s_bigs[k] = t;
        r += x;
        t += y;
      }
      const uint32_t rb = r ? atomicAdd(&a.ctl->rows, r) : 0u;
      const uint32_t tb = t ? atomicAdd(&a.ctl->bigs, t) : 0u;
      for (int k = 0; k < kWarps; k++) {
        s_rows[k] += rb;
        s_bigs[k] += tb;
      }
    }
    __syncthreads();
    rows = s_rows[warp];
    bigs = s_bigs[warp];
  }
}

// Pull into the one-leaf rows: a lane a row, eight ids (one sector) and their
// frontier bits a step, until one is in the frontier.  Ids ascend and an RMAT
// graph's hubs have low ids, so one step settles nearly every row; a warp
// takes 32 rows' chains of loads (row, depth, ids, bits) at once.
__device__ __forceinline__ void bfs_pull_small(const BfsArgs &a, int lvl, BfsSum &sum) {
  const int lane = threadIdx.x & 31;
  const uint32_t nw = (gridDim.x * kCoopThreads) >> 5;
  const uint32_t w0 = (blockIdx.x * kCoopThreads + threadIdx.x) >> 5;
  for (uint64_t i = (uint64_t)w0 * 32 + lane; i - lane < a.nsmall; i += (uint64_t)nw * 32) {
    const bool in = i < a.nsmall;
    const uint32_t v = in ? a.small[i] : 0u;
    const unsigned long long dsc = in ? a.sdesc[i] : 0ull;
    const uint32_t deg = (uint32_t)(dsc & 63);
    bool open = in && a.depth[v] < 0;
    if (!__any_sync(kFull, open)) continue;
    const uint32_t *p = a.g.slots + (dsc >> 6);
    // a segment off the 16-byte boundary holds one or two slots
    const bool wide = ((dsc >> 6) & 3) == 0;
    uint32_t found = kEmpty;
    for (uint32_t j = 0; __any_sync(kFull, open); j += 8) {
      uint32_t x[8];
      if (open && wide) {
        const uint4 q0 = *reinterpret_cast<const uint4 *>(p + j);
        const uint4 q1 = j + 4 < deg ? *reinterpret_cast<const uint4 *>(p + j + 4)
                                     : make_uint4(kEmpty, kEmpty, kEmpty, kEmpty);
        x[0] = q0.x, x[1] = q0.y, x[2] = q0.z, x[3] = q0.w;
        x[4] = q1.x, x[5] = q1.y, x[6] = q1.z, x[7] = q1.w;
      } else {
#pragma unroll
        for (int k = 0; k < 8; k++) x[k] = open && k < 2 && k < deg ? p[k] : kEmpty;
      }
      uint32_t f[8];
#pragma unroll
      for (int k = 0; k < 8; k++) f[k] = open && j + k < deg ? a.bits[x[k] >> 5] : 0u;
#pragma unroll
      for (int k = 7; k >= 0; k--)
        if ((f[k] >> (x[k] & 31)) & 1u) found = x[k];
      if (open && found != kEmpty) {  // its own row: no other lane writes it
        a.depth[v] = lvl + 1;
        if (a.parent) a.parent[v] = (int32_t)found;
        sum.add(deg, kLeaf);
      }
      open = open && found == kEmpty && j + 8 < deg;
    }
  }
}

// Pull into the multi-leaf rows, a chunk of leaves at a time.  A warp takes up
// to 32 chunks: a lane loads one chunk's row, depth and degree, and the warp
// then reads the open chunks' first leaves (lane = slot), kBfsAhead at once.  A
// first leaf holds the row's smallest ids, on an RMAT graph the hubs, and
// settles nearly every row: reading eight leaves at once made 8x the gathers.
// A row it does not settle goes on alone, up to eight leaves in flight, until
// one id is in the frontier or another chunk has claimed the row.
__device__ __forceinline__ void bfs_pull_chunks(const BfsArgs &a, int lvl, BfsSum &sum) {
  const int lane = threadIdx.x & 31;
  const uint32_t nw = (gridDim.x * kCoopThreads) >> 5;
  const uint32_t w0 = (blockIdx.x * kCoopThreads + threadIdx.x) >> 5;
  const uint64_t share = (a.nchunks + nw - 1) / nw;  // few chunks go to more warps
  const uint32_t per = share > 32 ? 32u : (uint32_t)share;
  for (uint64_t c0 = (uint64_t)w0 * per; c0 < a.nchunks; c0 += (uint64_t)nw * per) {
    const bool in = (uint32_t)lane < per && c0 + lane < a.nchunks;
    const uint32_t v = in ? a.cv[c0 + lane] : 0u;
    const unsigned long long dsc = in ? a.cdesc[c0 + lane] : 0ull;
    const bool open = in && __ldcg(a.depth + v) < 0;
    const uint32_t deg = open ? a.g.deg[v] : 0u;
    uint32_t mine = kEmpty;  // the lane's chunk's smallest frontier id
    for (uint32_t om = __ballot_sync(kFull, open); om;) {
      int src[kBfsAhead];
      uint32_t x[kBfsAhead], f[kBfsAhead];
      unsigned long long dq[kBfsAhead];
#pragma unroll
      for (int t = 0; t < kBfsAhead; t++) {
        src[t] = om ? __ffs(om) - 1 : -1;
        om &= om - 1;
        dq[t] = __shfl_sync(kFull, dsc, src[t] & 31);
        x[t] = src[t] >= 0 ? a.g.slots[((dq[t] >> 8) << kLeafLog) + lane] : kEmpty;
      }
#pragma unroll
      for (int t = 0; t < kBfsAhead; t++) f[t] = x[t] != kEmpty ? a.bits[x[t] >> 5] : 0u;
#pragma unroll
      for (int t = 0; t < kBfsAhead; t++) {
        if (src[t] < 0) break;
        uint32_t best = (f[t] >> (x[t] & 31)) & 1u ? x[t] : kEmpty;
        best = __reduce_min_sync(kFull, best);
        const uint32_t l1 = (uint32_t)(dq[t] & 63);
        if (best == kEmpty && l1 > 1) {
          const uint32_t vt = __shfl_sync(kFull, v, src[t]);
          const uint32_t *sl = a.g.slots + ((dq[t] >> 8) << kLeafLog) + lane;
          for (uint32_t l = 1; l < l1; l += 8) {
            // another chunk may claim the row meanwhile: lane 0's look for all
            if (!((dq[t] >> 7) & 1) && __shfl_sync(kFull, __ldcg(a.depth + vt), 0) >= 0) break;
            uint32_t y[8], fy[8];
#pragma unroll
            for (int q = 0; q < 8; q++)
              y[q] = l + q < l1 ? sl[(uint64_t)(l + q) << kLeafLog] : kEmpty;
#pragma unroll
            for (int q = 0; q < 8; q++) fy[q] = y[q] != kEmpty ? a.bits[y[q] >> 5] : 0u;
#pragma unroll
            for (int q = 7; q >= 0; q--)
              if ((fy[q] >> (y[q] & 31)) & 1u) best = y[q];
            best = __reduce_min_sync(kFull, best);
            if (best != kEmpty) break;
          }
        }
        if (lane == src[t]) mine = best;
      }
    }
    // a row of one chunk is this lane's alone
    if (mine != kEmpty &&
        (((dsc >> 7) & 1) || atomicCAS(&a.depth[v], -1, lvl + 1) == -1)) {
      a.depth[v] = lvl + 1;
      if (a.parent) a.parent[v] = (int32_t)mine;
      sum.add(deg, ((dsc >> 7) & 1) ? (uint32_t)(dsc & 63) << kLeafLog : a.g.cap[v]);
    }
  }
}

// the block's counts to the level's counters: one atomic a block and counter
__device__ __forceinline__ void bfs_count(BfsCount *c, const BfsSum &sum) {
  __shared__ BfsCount s_sum;
  if (threadIdx.x == 0) s_sum = BfsCount{};
  __syncthreads();
  unsigned long long v = sum.vertices, dg = sum.degrees;
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) {
    v += __shfl_xor_sync(kFull, v, d);
    dg += __shfl_xor_sync(kFull, dg, d);
  }
  const uint32_t bigs = __reduce_add_sync(kFull, sum.bigs);
  const uint32_t items = __reduce_add_sync(kFull, sum.items);
  if ((threadIdx.x & 31) == 0 && v) {
    atomicAdd(&s_sum.vertices, v);
    atomicAdd(&s_sum.degrees, dg);
    atomicAdd(&s_sum.rows, (uint32_t)v - bigs);
    atomicAdd(&s_sum.bigs, bigs);
    atomicAdd(&s_sum.items, items);
  }
  __syncthreads();
  if (threadIdx.x == 0 && s_sum.vertices) {
    atomicAdd(&c->vertices, s_sum.vertices);
    atomicAdd(&c->degrees, s_sum.degrees);
    atomicAdd(&c->rows, s_sum.rows);
    if (s_sum.bigs) {
      atomicAdd(&c->bigs, s_sum.bigs);
      atomicAdd(&c->items, s_sum.items);
    }
  }
}

// ------------------------------------------------------------ dependencies
// Brandes' single-source dependencies in the same launch: path counts (sigma)
// on the way down, beside the search itself, then the dependencies level by
// level back up.
//
// An edge joins levels that differ by at most one, so a row of level d has
// neighbours at d - 1, d and d + 1 only.  With one array for the even levels'
// values and one for the odd levels', zero until a row is done, the sum over
// all of a row's neighbours in the other parity's array is the sum over the
// wanted level alone (the other one of that parity is still zero, and adding
// zeros changes no bit): one gather an edge, where looking the depth up first
// took one or two.
//
// The order of every row's sum is fixed, the same as the multi-source form's:
// a one-leaf row in neighbour order; a multi-leaf row in chunks of kBcLeaves
// leaves, each lane over its chunk's leaves in order, then the lanes by
// shuffles, then the chunks in order.
constexpr uint32_t kBcLeaves = 32;
constexpr uint32_t kHubCap = kBcLeaves * kLeaf;  // a larger row is a hub: a warp a chunk

// capacity classes of the multi-leaf rows, largest first: hubs, then 32 leaves
// down to 2
constexpr int kBcClasses = 6;
__device__ __forceinline__ int bc_class(uint32_t cap) {
  return cap > kHubCap ? 0 : __clz(cap) - __clz(kHubCap) + 1;
}
struct BcCtl {
  uint32_t items;             // chunks of the hubs
  uint32_t count[kBcClasses]; // rows of a class
  uint32_t at[kBcClasses];    // rows of a class listed so far
};

struct BcArgs {
  double *sigma;      // 2n: of even levels' rows, then of odd levels'
  double *ratio;      // (1 + dependency) / sigma, likewise
  double *dep;        // n, the result
  const uint32_t *big;  // all multi-leaf rows
  uint64_t nbig;
  uint64_t max_hub;     // entries of the four hub arrays
  uint2 *hub;           // hubs: row, first item
  uint2 *hub_item;      // their chunks: hub, chunk
  double *hub_part;     // a chunk's sum
  uint32_t *hub_done;   // chunks summed, of a hub (zero between levels)
  uint32_t *order;      // the other multi-leaf rows by capacity, largest first; nbig entries
  BcCtl *bc;            // zero at launch and after
  bool few;             // few vertices have a row (bc_few)
  uint2 *level;         // per level: queue ends, multi-leaf rows' high bit = not in the queue
};
constexpr uint32_t kNotQueued = 1u << 31;

// Whether the vertices with a row, which are written out of order, cost less to
// clear than all of them, four values each.
inline bool bc_few(uint64_t rows, uint64_t n) { return rows < n / 8; }

constexpr int kBcFlight = 8;  // neighbours (or leaves) in flight

// Row ids are read once a pass and leave L1 to the gathered values; those
// change between levels, so they are not read through the read-only path.  (The
// ids do not change while the kernel runs, and it is no programmatic launch, so
// nothing has to order these loads.)
__device__ __forceinline__ uint32_t ld_id(const uint32_t *p) {
  uint32_t v;
  asm("ld.global.nc.L1::no_allocate.b32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ uint4 ld_id4(const uint32_t *p) {
  uint4 v;
  asm("ld.global.nc.L1::no_allocate.v4.b32 {%0, %1, %2, %3}, [%4];"
      : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
      : "l"(p));
  return v;
}
// the sums of val over the one-leaf rows of a warp, a lane a row (deg = 0: none)
__device__ __forceinline__ double bc_sum_rows(const BfsArgs &a, uint64_t base, uint32_t deg,
                                              const double *val) {
  const uint32_t *p = a.g.slots + base;
  const bool wide = (base & 3) == 0;  // else a segment of one or two slots
  double s = 0.0;
  for (uint32_t j = 0; j < deg; j += kBcFlight) {
    uint32_t x[kBcFlight];
    if (wide) {
      const uint4 q0 = ld_id4(p + j);
      const uint4 q1 = j + 4 < deg ? ld_id4(p + j + 4) : q0;
      x[0] = q0.x, x[1] = q0.y, x[2] = q0.z, x[3] = q0.w;
      x[4] = q1.x, x[5] = q1.y, x[6] = q1.z, x[7] = q1.w;
    } else {
#pragma unroll
      for (int k = 0; k < kBcFlight; k++) x[k] = k < 2 && j + k < deg ? p[k] : 0u;
    }
    double y[kBcFlight];
#pragma unroll
    for (int k = 0; k < kBcFlight; k++) y[k] = j + k < deg ? val[x[k]] : 0.0;
#pragma unroll
    for (int k = 0; k < kBcFlight; k++) s += y[k];
  }
  return s;
}

// the sum of val over leaves [l0, l1) of a multi-leaf row, by a warp (lane 0
// has it); at most kBcLeaves of them
__device__ __forceinline__ double bc_sum_leaves(const BfsArgs &a, uint64_t base, uint32_t l0,
                                                uint32_t l1, const double *val) {
  const uint32_t *p = a.g.slots + base + (threadIdx.x & 31);
  double acc = 0.0;
  for (uint32_t l = l0; l < l1; l += kBcFlight) {
    uint32_t x[kBcFlight];
#pragma unroll
    for (int k = 0; k < kBcFlight; k++)
      x[k] = l + k < l1 ? ld_id(p + ((uint64_t)(l + k) << kLeafLog)) : kEmpty;
    double y[kBcFlight];
#pragma unroll
    for (int k = 0; k < kBcFlight; k++) y[k] = x[k] != kEmpty ? val[x[k]] : 0.0;
#pragma unroll
    for (int k = 0; k < kBcFlight; k++) acc += y[k];
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) acc += __shfl_down_sync(kFull, acc, d);
  return acc;
}

// row v of level lvl has the sum s
__device__ __forceinline__ void bc_finish(const BfsArgs &a, const BcArgs &b, uint32_t v, int lvl,
                                          bool down, double s) {
  const uint64_t i = (lvl & 1 ? (uint64_t)a.g.n : 0) + v;
  if (down) {
    b.sigma[i] = s;
  } else {
    const double sg = b.sigma[i], dv = sg * s;
    b.dep[v] = dv;
    b.ratio[i] = (1.0 + dv) / sg;
  }
}

// Sums over lanes of R accumulators at once: afterwards lanes j * 32/R .. hold
// accumulator j's sum, each the same sum as shuffling it down by 16, 8, 4, 2, 1
// (an addition's two sides may change places).  The first log2(R) steps halve
// the accumulators, so R of them take R - 1 + 5 - log2(R) additions, not 5R: a
// warp's FP64 addition takes about 15 cycles of this device's pipe.  With a reduction
// and a division a row, by one lane, the pipe was busy for 255 of 700 us at RMAT scale
// 20, with this for 36% of 510: the rest is the gathers' latency with half of the SM's
// warps (64 registers a thread) and blocks that wait at the grid barrier for others.
template <int R>
__device__ __forceinline__ double bc_reduce(double (&acc)[R]) {
  const int lane = threadIdx.x & 31;
  int d = 16;
#pragma unroll
  for (int r = R / 2; r > 0; r >>= 1, d >>= 1) {
    const bool up = lane & d;
#pragma unroll
    for (int j = 0; j < r; j++) {
      const double keep = up ? acc[j + r] : acc[j], give = up ? acc[j] : acc[j + r];
      acc[j] = keep + __shfl_xor_sync(kFull, give, d);
    }
  }
#pragma unroll
  for (; d > 0; d >>= 1) acc[0] += __shfl_xor_sync(kFull, acc[0], d);
  return acc[0];
}

// R multi-leaf rows (lane j < R: row v's first slot and leaf count nl, 0: no
// row) summed by the warp, kPair rows and kLeaves leaves in flight, and
// finished together
template <int R, int kPair, int kLeaves>
__device__ __forceinline__ void bc_rows(const BfsArgs &a, const BcArgs &b, uint32_t v,
                                        uint64_t base, uint32_t nl, int lvl, bool down,
                                        const double *val) {
  const int lane = threadIdx.x & 31;
  double acc[R];
#pragma unroll
  for (int r = 0; r < R; r += kPair) {
    const uint32_t *p[kPair];
    uint32_t n[kPair], most = 0;
#pragma unroll
    for (int q = 0; q < kPair; q++) {
      p[q] = a.g.slots + __shfl_sync(kFull, base, r + q) + lane;
      n[q] = __shfl_sync(kFull, nl, r + q);
      most = max(most, n[q]);
      acc[r + q] = 0.0;
    }
    for (uint32_t l = 0; l < most; l += kLeaves) {
      uint32_t x[kPair][kLeaves];
#pragma unroll
      for (int q = 0; q < kPair; q++)
#pragma unroll
        for (int k = 0; k < kLeaves; k++)
          x[q][k] = l + k < n[q] ? ld_id(p[q] + ((uint64_t)(l + k) << kLeafLog)) : kEmpty;
      double y[kPair][kLeaves];
#pragma unroll
      for (int q = 0; q < kPair; q++)
#pragma unroll
        for (int k = 0; k < kLeaves; k++) y[q][k] = x[q][k] != kEmpty ? val[x[q][k]] : 0.0;
#pragma unroll
      for (int q = 0; q < kPair; q++)
#pragma unroll
        for (int k = 0; k < kLeaves; k++)
          if (l + k < n[q]) acc[r + q] += y[q][k];  // the same for the warp
    }
  }
  const double sum = bc_reduce<R>(acc);
  const int j = lane / (32 / R);
  const uint32_t vj = __shfl_sync(kFull, v, j), nj = __shfl_sync(kFull, nl, j);
  if (lane % (32 / R) == 0 && nj) bc_finish(a, b, vj, lvl, down, sum);
}

// The rows of level lvl: sigma from the level above (down), or dependencies
// from the level below.  The level is in the queue ([r0, r1) and [b0, b1)), or
// else, a level that a pull left, every list is searched for it: such levels
// hold a fair share of the graph, so there are few of them.
__device__ __forceinline__ void bc_level(const BfsArgs &a, const BcArgs &b, int lvl, bool down,
                                         bool queued, uint32_t r0, uint32_t r1, uint32_t b0,
                                         uint32_t b1) {
  const int lane = threadIdx.x & 31;
  const uint32_t nw = (gridDim.x * kCoopThreads) >> 5;
  const uint32_t w0 = (blockIdx.x * kCoopThreads + threadIdx.x) >> 5;
  const double *val = (down ? b.sigma : b.ratio) + (lvl & 1 ? 0 : (uint64_t)a.g.n);
  // hubs: a warp a chunk, over all the hubs' chunks; the warp that sums a hub's
  // last chunk adds the chunks up, in their order
  const uint32_t nitems = __ldcg(&b.bc->items);
  for (uint32_t i = w0; i < nitems; i += nw) {
    const uint2 it = b.hub_item[i], hb = b.hub[it.x];
    const uint32_t v = hb.x;
    if (__shfl_sync(kFull, __ldcg(a.depth + v), 0) != lvl) continue;
    const uint32_t nl = a.g.cap[v] >> kLeafLog, l0 = it.y * kBcLeaves;
    const uint32_t nc = (nl + kBcLeaves - 1) / kBcLeaves;
    const double s = bc_sum_leaves(a, a.g.base[v], l0, min(l0 + kBcLeaves, nl), val);
    uint32_t done = 0;
    if (lane == 0) {
      __stcg(b.hub_part + i, s);
      __threadfence();
      done = atomicAdd(b.hub_done + it.x, 1u) + 1;
      __threadfence();
    }
    if (__shfl_sync(kFull, done, 0) != nc) continue;
    double t = 0.0;
    for (uint32_t c0 = 0; c0 < nc; c0 += 32) {
      const double part = c0 + lane < nc ? __ldcg(b.hub_part + hb.y + c0 + lane) : 0.0;
      for (uint32_t c = c0; c < min(c0 + 32, nc); c++) t += __shfl_sync(kFull, part, c - c0);
    }
    if (lane == 0) {
      b.hub_done[it.x] = 0;
      bc_finish(a, b, v, lvl, down, t);
    }
  }
  // The other multi-leaf rows.  The list has the long ones first, and a warp
  // takes the fewer the longer they are, so that the warps end together (in id
  // order an RMAT graph's long rows sit side by side, and a warp with eight of
  // them held the level up for 75 us); a queue is in no order.
  const uint64_t nbig = queued ? b1 - b0 : b.nbig - __ldcg(&b.bc->count[0]);
  uint64_t end[3] = {0, 0, nbig};  // rows of over 16 leaves, of 8 and 16, all
  if (!queued) {
    end[0] = __ldcg(&b.bc->count[1]);
    end[1] = end[0] + __ldcg(&b.bc->count[2]) + __ldcg(&b.bc->count[3]);
  }
  for (int part = 0; part < 3; part++) {
    const uint64_t first = part ? end[part - 1] : 0, n = end[part] - first;
    const uint64_t share = (n + nw - 1) / nw;
    const uint64_t most = part == 0 ? 2 : part == 1 ? 4 : 8;
    const uint32_t per = (uint32_t)(share > most ? most : share);
    for (uint64_t i0 = (uint64_t)w0 * per; i0 < n; i0 += (uint64_t)nw * per) {
      const uint64_t i = first + i0 + lane;
      const bool in = (uint32_t)lane < per && i0 + lane < n;
      const uint32_t v = !in ? 0u : queued ? a.queue[a.g.n - 1 - (b0 + i)] : b.order[i];
      const uint32_t cap = in ? a.g.cap[v] : 0u;
      const uint64_t base = in ? a.g.base[v] : 0ull;
      const bool on = in && cap <= kHubCap && (queued || a.depth[v] == lvl);
      if (!__any_sync(kFull, on)) continue;
      const uint32_t nl = on ? cap >> kLeafLog : 0u;
      if (part == 0)
        bc_rows<2, 1, 8>(a, b, v, base, nl, lvl, down, val);
      else if (part == 1)
        bc_rows<4, 1, 8>(a, b, v, base, nl, lvl, down, val);
      else
        bc_rows<8, 2, 4>(a, b, v, base, nl, lvl, down, val);
    }
  }
  const uint64_t nrow = queued ? r1 - r0 : a.nsmall;
  {  // one-leaf rows: a lane a row
    const uint64_t share = (nrow + nw - 1) / nw;
    const uint32_t per = share > 32 ? 32u : (uint32_t)share;
    for (uint64_t i = (uint64_t)w0 * per + lane; i - lane < nrow; i += (uint64_t)nw * per) {
      const bool in = (uint32_t)lane < per && i < nrow;
      const uint32_t v = !in ? 0u : queued ? a.queue[r0 + i] : a.small[i];
      const unsigned long long dsc = in && !queued ? a.sdesc[i] : 0ull;
      const bool on = in && (queued || a.depth[v] == lvl);
      if (!__any_sync(kFull, on)) continue;
      const uint64_t base = !on ? 0ull : queued ? a.g.base[v] : dsc >> 6;
      const uint32_t deg = !on ? 0u : queued ? a.g.deg[v] : (uint32_t)(dsc & 63);
      const double s = bc_sum_rows(a, base, deg, val);
      if (on) bc_finish(a, b, v, lvl, down, s);
    }
  }
}

// The multi-leaf rows by capacity class, in two passes with a barrier between
// them: the classes' sizes, then their rows (in any order within a class) and
// the hubs' chunks.  A block counts in shared memory and reserves once a class.
__device__ __forceinline__ void bc_count_classes(const BfsArgs &a, const BcArgs &b) {
  __shared__ uint32_t s_cnt[kBcClasses];
  if (threadIdx.x < kBcClasses) s_cnt[threadIdx.x] = 0;
  __syncthreads();
  const uint64_t nt = (uint64_t)gridDim.x * kCoopThreads;
  for (uint64_t i = (uint64_t)blockIdx.x * kCoopThreads + threadIdx.x; i < b.nbig; i += nt)
    atomicAdd(&s_cnt[bc_class(a.g.cap[b.big[i]])], 1u);
  __syncthreads();
  if (threadIdx.x < kBcClasses && s_cnt[threadIdx.x])
    atomicAdd(&b.bc->count[threadIdx.x], s_cnt[threadIdx.x]);
}

__device__ __forceinline__ void bc_list_classes(const BfsArgs &a, const BcArgs &b) {
  __shared__ uint32_t s_cnt[kBcClasses], s_at[kBcClasses];
  const uint64_t nt = (uint64_t)gridDim.x * kCoopThreads;
  const uint64_t t0 = (uint64_t)blockIdx.x * kCoopThreads + threadIdx.x;
  for (uint64_t i0 = t0 - threadIdx.x; i0 < b.nbig; i0 += nt) {  // the same for the block
    if (threadIdx.x < kBcClasses) s_cnt[threadIdx.x] = 0;
    __syncthreads();
    const uint64_t i = i0 + threadIdx.x;
    const uint32_t v = i < b.nbig ? b.big[i] : 0u;
    const uint32_t cap = i < b.nbig ? a.g.cap[v] : 0u;
    const int cls = i < b.nbig ? bc_class(cap) : 0;
    uint32_t r = 0;
    if (i < b.nbig) r = atomicAdd(&s_cnt[cls], 1u);
    __syncthreads();
    if (threadIdx.x < kBcClasses) {
      uint32_t at = 0;  // hubs have a list of their own
      for (int c = 1; c < (int)threadIdx.x; c++) at += __ldcg(&b.bc->count[c]);
      if (s_cnt[threadIdx.x]) at += atomicAdd(&b.bc->at[threadIdx.x], s_cnt[threadIdx.x]);
      s_at[threadIdx.x] = at;
    }
    __syncthreads();
    if (i < b.nbig) {
      r += s_at[cls];
      if (cls) {
        if (r < b.nbig) b.order[r] = v;
      } else {
        const uint32_t k = ((cap >> kLeafLog) + kBcLeaves - 1) / kBcLeaves;
        const uint32_t at = atomicAdd(&b.bc->items, k);
        if ((uint64_t)at + k > b.max_hub || r >= b.max_hub) {
          a.ctl->err = 2;
        } else {
          b.hub[r] = make_uint2(v, at);
          b.hub_done[r] = 0;
          for (uint32_t j = 0; j < k; j++) b.hub_item[at + j] = make_uint2(r, j);
        }
      }
    }
    __syncthreads();
  }
}

// Nothing but the source has a path count yet.  Only vertices with a row are
// anyone's neighbours, so where they are few (see bc_few) only theirs are cleared:
// of 2^27 vertices with 2,000 in use, all four values of each took 1.41 ms with the
// search, these 0.75; of 2^24, 0.32 and 0.24.
__device__ __forceinline__ void bc_clear(const BfsArgs &a, const BcArgs &b, uint32_t t0,
                                         uint32_t nt) {
  const uint64_t n = a.g.n;
  if (b.few) {
    for (uint64_t i = t0; i < a.nsmall + b.nbig; i += nt) {
      const uint64_t v = i < a.nsmall ? a.small[i] : b.big[i - a.nsmall];
      if (v != a.src) b.sigma[v] = 0.0;
      b.sigma[n + v] = b.ratio[v] = b.ratio[n + v] = 0.0;
    }
    for (uint64_t v = t0; v < n; v += nt) b.dep[v] = 0.0;
    if (t0 == 0) b.sigma[a.src] = 1.0;
    return;
  }
  for (uint64_t v = t0; v < n; v += nt) {
    const uint64_t w = v + n;
    b.sigma[v] = v == a.src ? 1.0 : 0.0;
    b.sigma[w] = b.ratio[v] = b.ratio[w] = b.dep[v] = 0.0;
  }
}

// Every level of the search; with kBc also the rows' sigma, each level's beside
// the search for the next one.  Returns the number of levels, -1 on an error.
template <bool kBc>
__device__ __forceinline__ int bfs_levels(const BfsArgs &a, const BcArgs &b, GridBarrier &bar) {
  BfsCtl *ctl = a.ctl;
  const uint32_t t0 = blockIdx.x * kCoopThreads + threadIdx.x;
  const uint32_t nt = gridDim.x * kCoopThreads;
  for (uint64_t v = t0; v < a.g.n; v += nt) {
    a.depth[v] = v == a.src ? 0 : -1;
    if (a.parent) a.parent[v] = v == a.src ? (int32_t)a.src : -1;
  }
  if (kBc) {
    bc_clear(a, b, t0, nt);
    bc_count_classes(a, b);
  }
  if (t0 < 32) {  // the source's row is level 0
    const uint32_t cap = a.g.cap[a.src];
    const uint32_t v1[1] = {a.src}, c1[1] = {cap};
    bfs_enqueue(a, t0 == 0 ? 1u : 0u, v1, c1);
    if (t0 == 0) {
      BfsSum sum;
      sum.add(a.g.deg[a.src], cap);
      ctl->cnt[0] = BfsCount{1, sum.degrees, 1u - sum.bigs, sum.bigs, sum.items};
    }
  }
  if (!bar.wait()) return -1;
  uint32_t rows = 0, bigs = 0, items = 0;  // queue entries of the levels before
  bool queued = true;                      // this level is in the queue
  for (int lvl = 0; (uint32_t)lvl <= a.g.n; lvl++) {
    // the level's counts, the same for every block: complete since the last
    // barrier, and cleared two levels on
    const BfsCount *c = &ctl->cnt[lvl % 3];
    const unsigned long long fv = __ldcg(&c->vertices), fd = __ldcg(&c->degrees);
    if (fv == 0) return lvl;
    const uint32_t r1 = rows + __ldcg(&c->rows), b1 = bigs + __ldcg(&c->bigs);
    const uint32_t ni = __ldcg(&c->items);
    if (t0 == 0) ctl->cnt[(lvl + 2) % 3] = BfsCount{};
    BfsSum sum;
    const bool pull = (fv + fd) * a.alpha > a.m;
    if (pull) {
      bfs_level_bits(a, lvl);
      if (!bar.wait()) return -1;
      bfs_pull_chunks(a, lvl, sum);
      bfs_pull_small(a, lvl, sum);
    } else {
      if (!queued) {  // the level was reached by a pull
        bfs_queue_level(a, lvl);
        if (!bar.wait()) return -1;
      }
      if (b1 > bigs) {
        bfs_list_items(a, bigs, b1);
        if (!bar.wait()) return -1;
        bfs_push_items(a, items, items + ni, lvl, sum);
        items += ni;
      }
      bfs_push_rows(a, rows, r1, lvl, sum);
    }
    if (kBc) {
      const bool listed = queued || !pull;
      if (lvl)
        bc_level(a, b, lvl, true, listed, rows, r1, bigs, b1);
      else
        bc_list_classes(a, b);  // from level 1 on
      if (t0 == 0)
        b.level[lvl] = listed ? make_uint2(r1, b1) : make_uint2(rows, bigs | kNotQueued);
    }
    if (queued || !pull) {
      rows = r1;
      bigs = b1;
    }
    queued = !pull;  // what a push reaches is queued
    bfs_count(&ctl->cnt[(lvl + 1) % 3], sum);
    if (!bar.wait()) return -1;
  }
  if (t0 == 0) ctl->err = 3;  // more than n levels
  return -1;
}

// the last block to leave reports the error and leaves the state zero again
__device__ __forceinline__ void bfs_leave(const BfsArgs &a, BcCtl *bc) {
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(&a.ctl->left, 1u) == gridDim.x - 1) {
      __threadfence();
      *a.result = *(volatile unsigned int *)&a.ctl->err;
      *a.ctl = BfsCtl{};
      if (bc) *bc = BcCtl{};
    }
  }
}

__global__ void __launch_bounds__(kCoopThreads, kCoopPerSm) k_bfs_levels(BfsArgs a) {
  GridBarrier bar{&a.ctl->bar, &a.ctl->err, 0};
  bfs_levels<false>(a, BcArgs{}, bar);
  bfs_leave(a, nullptr);
}

__global__ void __launch_bounds__(kCoopThreads, kCoopPerSm) k_bc_levels(BfsArgs a, BcArgs b) {
  GridBarrier bar{&a.ctl->bar, &a.ctl->err, 0};
  const int levels = bfs_levels<true>(a, b, bar);
  for (int lvl = levels - 1; lvl >= 0; lvl--) {
    const uint2 e = b.level[lvl], e0 = lvl ? b.level[lvl - 1] : make_uint2(0u, 0u);
    bc_level(a, b, lvl, false, !(e.y & kNotQueued), e0.x, e.x, e0.y & ~kNotQueued,
             e.y & ~kNotQueued);
    if (lvl && !bar.wait()) break;
  }
  bfs_leave(a, b.bc);
}

}  // namespace
}  // namespace sst
