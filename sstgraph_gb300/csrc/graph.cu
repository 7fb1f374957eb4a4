// Graph lifetime, slab allocation and the batch update pipeline.
//
// A batch (insert or remove) runs as:
//   1. keys      (row << dbits | col) per pair; self-loops (insert) and ids
//                out of range take a key that no other pair has
//   2. sort      stable LSD radix sort of the keys (primitives.cu)
//   3. locate    per unique key: the leaf of its row's PMA where it belongs
//                (binary search over leaf heads) and whether it is present
//   4. pack      keys that change the graph, as (row, leaf) + col, in order
//   5. group     one group per (row, leaf)
//   6. classify  insert: a group fits its leaf (leaf merge) or climbs to the
//                smallest aligned window of 2^t leaves whose count stays
//                under the upper density bound, or the whole segment is
//                resized.  remove: deletions are applied leaf-locally first,
//                then leaves under the lower bound climb the same way.
//   7. dominance aligned windows nest, so a forward max-scan and a backward
//                min-scan over the groups find, for each group, the largest
//                window of its row that covers it; covered groups drop out
//   8. plan      window/resize tasks are sized and the summary is read back
//                (the one host synchronisation of a batch): it sizes the
//                staging buffer and the slab allocation
//   9. apply     leaf merges (one warp per leaf, shuffle-ranked), then each
//                task gathers old + new elements at their merged rank into
//                staging (parallel over leaves and items) and scatters them
//                evenly over the destination leaves (one warp per leaf)
// Reference counterparts: SparseMatrix.hpp:556-718 (batch split by row),
// PMA.hpp:1028-1082 (place: window climb + redistribute),
// PMA.hpp:612-702 (redistribute / double_list / half_list),
// PMA.hpp:1185-1222 (take: lower-bound climb).
#include <algorithm>
#include <cooperative_groups.h>
#include <cstddef>
#include <cstdarg>
#include <cstdlib>
#include <cstring>
#include <unistd.h>
#include <vector>

#include "graph.cuh"

namespace sst {

namespace {

enum : uint8_t { kNone = 0, kMerge = 1, kWindow = 2, kResize = 3 };

constexpr int kTB = 256;  // threads per block for element-wise kernels

inline unsigned blocks_for(uint64_t n, int per_block = kTB) {
  uint64_t b = (n + per_block - 1) / per_block;
  return (unsigned)(b == 0 ? 1 : b);
}
inline unsigned warp_blocks(uint64_t nwarps) {
  return blocks_for(nwarps * 32);
}

int bits_for(uint64_t x) {
  int b = 0;
  while (b < 64 && (x >> b) != 0) b++;
  return b;
}

// Lower bound (first index with a[i] >= x) of [lo, hi) in a sorted array,
// by a whole warp (every lane gets the answer): each round the 32 lanes
// probe 32 evenly spaced positions and the range shrinks to the gap between
// the last probe below x and the next one, so a range of 1e6 items takes
// four dependent rounds instead of twenty.
__device__ __forceinline__ uint32_t warp_lb_u64(const uint64_t *a, uint32_t lo,
                                                uint32_t hi, uint64_t x) {
  const uint32_t lane = threadIdx.x & 31;
  while (hi - lo > 32) {
    const uint32_t step = (hi - lo + 31) / 32;
    const uint32_t probe = lo + lane * step;
    const bool less = probe < hi && a[probe] < x;
    const uint32_t k = __popc(__ballot_sync(0xffffffffu, less));
    if (k == 0) return lo;  // a[lo] >= x
    const uint32_t nhi = lo + k * step;  // a[nhi] >= x, or nhi >= hi
    lo += (k - 1) * step + 1;
    if (nhi < hi) hi = nhi;
  }
  const uint32_t probe = lo + lane;
  return lo + __popc(__ballot_sync(0xffffffffu, probe < hi && a[probe] < x));
}

// index of the last element <= x in a sorted array (n >= 1, a[0] <= x)
__device__ __forceinline__ uint64_t last_le_u64(const uint64_t *a, uint64_t n,
                                                uint64_t x) {
  uint64_t lo = 0, hi = n;
  while (hi - lo > 1) {
    uint64_t mid = (lo + hi) >> 1;
    if (a[mid] <= x)
      lo = mid;
    else
      hi = mid;
  }
  return lo;
}

// elements of a[lo, hi) below each of four keys, found at once (the
// branchless lower bound: each step halves the range for all four searches,
// so their loads are in flight together)
__device__ __forceinline__ void count_less4(const uint32_t *a, uint32_t lo, uint32_t hi,
                                            const uint32_t (&x)[4], uint32_t (&out)[4]) {
  uint32_t b[4] = {lo, lo, lo, lo};
  uint32_t n = hi - lo;
  if (n == 0) {
#pragma unroll
    for (int r = 0; r < 4; r++) out[r] = 0;
    return;
  }
  while (n > 1) {
    const uint32_t half = n >> 1;
#pragma unroll
    for (int r = 0; r < 4; r++) b[r] = a[b[r] + half] < x[r] ? b[r] + half : b[r];
    n -= half;
  }
#pragma unroll
  for (int r = 0; r < 4; r++) out[r] = (b[r] - lo) + (a[b[r]] < x[r] ? 1u : 0u);
}

__device__ __forceinline__ uint32_t warp_sum_lcnt(const uint8_t *lc,
                                                  uint64_t lo, uint64_t hi) {
  const int lane = threadIdx.x & 31;
  uint32_t s = 0;
  for (uint64_t i = lo + lane; i < hi; i += 32) s += lc[i];
  return __reduce_add_sync(0xffffffffu, s);
}

// count word of an item's leaf: the leaf's element count (bits 0-7), plus
// this bit when the row is a multi-leaf segment (its leaves keep counts in
// lcnt), else the one-leaf row's capacity (0..32) from bit kCapShift
constexpr uint32_t kMultiLeaf = 1u << 8;
constexpr int kCapShift = 16;
__device__ __forceinline__ uint32_t one_leaf_cap(uint32_t cw) { return cw >> kCapShift; }

// ---------------------------------------------------------------- steps 1-5
// Keys of a batch, in one of two forms.
// k_make_keys: key i of pair i, the sentinel n << dbits for a pair that is
// dropped (an id out of range, or a self-loop the insert skips); the stable
// sort keeps equal keys in input order (weighted graphs: the last value
// given wins).
__global__ void k_make_keys(const uint32_t *__restrict__ pairs, uint64_t b,
                            uint32_t n, uint32_t width, int dbits,
                            bool drop_loops, uint64_t *__restrict__ keys,
                            unsigned long long *__restrict__ invalid,
                            const uint32_t *__restrict__ w,
                            uint32_t *__restrict__ wv) {
  pdl_wait();
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= b) return;
  // weighted graphs: the pair's value (1 when the call gives none) rides
  // with the key through the sort
  if (wv) wv[i] = w ? w[i] : 1u;
  const uint32_t r = pairs[2 * i], c = pairs[2 * i + 1];
  const bool ok = r < n && c < width && c != kEmpty;
  if (!ok) atomicAdd(invalid, 1ull);
  keys[i] = (!ok || (drop_loops && r == c)) ? (uint64_t)n << dbits
                                            : (((uint64_t)r << dbits) | c);
}

// k_make_keys_packed (unweighted graphs, where equal keys need no order): a
// dropped pair takes the key `sent`, on a graph without self-loops that of (0, 0),
// which no kept pair has, so the sort needs no bit for a row n.  (Packing only the
// kept keys to the front cost an atomic on one counter for every 2048 pairs, one
// after another: 39 us for 4.8M pairs, 30 now; 15.4 for 1M, 10.6.)  With V2
// (the pairs 8-byte aligned) a pair comes in with one 8-byte load: the warp's
// load covers 256 contiguous bytes once, where two 4-byte loads a pair read
// each line twice (pinned host pairs are read across the host link).
// With sd.passes > 0 it also counts every radix pass's 8-bit digits of the
// keys into sd.totals (zero on entry) and clears the sort's tile
// status words (SortDigits): the sort then skips its own counting read.
constexpr int kPackItems = 8;
template <bool V2>
__global__ void __launch_bounds__(256)
k_make_keys_packed(const uint32_t *__restrict__ pairs, uint64_t b, uint32_t n,
                   uint32_t width, int dbits, bool drop_loops, uint64_t sent,
                   uint64_t *__restrict__ keys,
                   unsigned long long *__restrict__ invalid,
                   uint32_t *__restrict__ nkeys, SortDigits sd) {
  pdl_wait();
  __shared__ uint32_t s_hist[8][256];
  for (int p = 0; p < sd.passes; p++) s_hist[p][threadIdx.x] = 0;
  __syncthreads();
  const uint64_t t0 = (uint64_t)blockIdx.x * (256 * kPackItems) + threadIdx.x;
  uint32_t r[kPackItems], c[kPackItems], bad = 0;
#pragma unroll
  for (int k = 0; k < kPackItems; k++) {
    const uint64_t i = t0 + k * 256;
    r[k] = c[k] = 0;
    if (i >= b) continue;
    if (V2) {
      const uint2 rc = reinterpret_cast<const uint2 *>(pairs)[i];
      r[k] = rc.x;
      c[k] = rc.y;
    } else {
      r[k] = pairs[2 * i];
      c[k] = pairs[2 * i + 1];
    }
  }
#pragma unroll
  for (int k = 0; k < kPackItems; k++) {
    if (t0 + k * 256 >= b) break;
    const bool ok = r[k] < n && c[k] < width && c[k] != kEmpty;
    bad += !ok;
    const uint64_t key =
        !ok || (drop_loops && r[k] == c[k]) ? sent : ((uint64_t)r[k] << dbits) | c[k];
    keys[t0 + k * 256] = key;
    for (int p = 0; p < sd.passes; p++) atomicAdd(&s_hist[p][(key >> (8 * p)) & 0xff], 1u);
  }
  if (bad) atomicAdd(invalid, (unsigned long long)bad);
  if (t0 == 0) *nkeys = (uint32_t)b;
  if (!sd.passes) return;
  for (uint64_t i = (uint64_t)blockIdx.x * 256 + threadIdx.x; i < sd.status_words;
       i += (uint64_t)gridDim.x * 256)
    sd.status[i] = 0;
  __syncthreads();
  for (int p = 0; p < sd.passes; p++)
    if (s_hist[p][threadIdx.x]) atomicAdd(&sd.totals[p * 256 + threadIdx.x], s_hist[p][threadIdx.x]);
}

// Of a run of equal keys the last (in input order: the sort is stable) is
// the one applied, so on a weighted graph the last value given wins, as
// sequential inserts would leave it (PMA.hpp:1137-1145).  A weighted insert
// of an edge already present overwrites its value here, in place.
__global__ void k_locate(const uint64_t *__restrict__ keys, uint64_t b,
                         int dbits, DGraph g, bool insert,
                         uint32_t *__restrict__ flag,
                         uint32_t *__restrict__ leaf_out,
                         const uint32_t *__restrict__ wv,
                         uint64_t *__restrict__ lS, uint32_t *__restrict__ lc,
                         uint64_t sent, const uint32_t *__restrict__ nkeys) {
  pdl_wait();
  uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= b) return;
  // a replayed sequence is sized by more keys than the batch has
  const uint64_t nk = nkeys ? *nkeys : b;
  uint64_t k = i < nk ? keys[i] : sent;
  if (k == sent || (i + 1 < nk && keys[i + 1] == k)) {
    flag[i] = 0;
    leaf_out[i] = 0;
    return;
  }
  uint64_t S = 0;
  uint32_t cw = 0;
  uint32_t u = (uint32_t)(k >> dbits);
  uint32_t x = (uint32_t)(k & ((1ull << dbits) - 1));
  uint64_t base = g.base[u];
  uint32_t cap = g.cap[u], deg = g.deg[u];
  bool present = false;
  uint32_t l = 0;
  if (cap > 0) {
    l = find_leaf(g.slots, base, cap, x);
    uint32_t c = leaf_count(g, base, cap, deg, l);
    const uint32_t *p = g.slots + base + ((uint64_t)l << kLeafLog);
    uint32_t pos = leaf_lower_bound(p, c, x);
    present = pos < c && p[pos] == x;
    if (present && insert && wv && g.vals)
      g.vals[base + ((uint64_t)l << kLeafLog) + pos] = wv[i];
    S = base + ((uint64_t)l << kLeafLog);
    cw = c | (cap > kLeaf ? kMultiLeaf : cap << kCapShift);
  }
  flag[i] = insert ? !present : present;
  leaf_out[i] = l;
  lS[i] = S;
  lc[i] = cw;
}

// k_locate for small batches, a warp per key (a batch of up to
// kLocateWarpKeys keys fills about one wave of warps): the leaf search
// probes 32 leaf heads at once, so a row of L leaves takes about log32(L)
// dependent steps where a thread takes log2(L), and the leaf's 32 slots come
// in with one coalesced load.  Same outputs as k_locate (the heads of a
// segment's leaves ascend, so the leaves whose head is <= x are a prefix).
constexpr uint64_t kLocateWarpKeys = 16384;

struct Located {
  uint64_t S;        // the leaf's first slot
  uint32_t leaf, cw; // its index in the row, its count word
  uint32_t pos;      // ids of the leaf below x
  bool present;
};
__device__ __forceinline__ Located locate_by_warp(const DGraph &g, uint32_t u, uint32_t x) {
  const int lane = threadIdx.x & 31;
  const uint64_t base = g.base[u];
  const uint32_t cap = g.cap[u], deg = g.deg[u];
  Located r{0, 0, 0, 0, false};
  if (cap == 0) return r;
  if (cap > kLeaf) {
    // the answer lies in leaves [lo, lo + n); lane j probes leaf lo + j*step
    uint32_t lo = 0, n = cap >> kLeafLog;
    for (;;) {
      const uint32_t step = n > 32 ? (n + 31) / 32 : 1u;
      const uint32_t j = (uint32_t)lane * step;
      const bool le = lane > 0 && j < n && g.slots[base + ((uint64_t)(lo + j) << kLeafLog)] <= x;
      const uint32_t m = __ballot_sync(0xffffffffu, le);
      const uint32_t jj = m ? 31u - __clz(m) : 0u;
      lo += jj * step;
      if (step == 1) break;
      n = n - jj * step < step ? n - jj * step : step;
    }
    r.leaf = lo;
  }
  const uint32_t c = leaf_count(g, base, cap, deg, r.leaf);
  r.S = base + ((uint64_t)r.leaf << kLeafLog);
  const uint32_t a = (uint32_t)lane < c ? g.slots[r.S + lane] : kEmpty;
  r.pos = __popc(__ballot_sync(0xffffffffu, a < x));
  const uint32_t at = __shfl_sync(0xffffffffu, a, r.pos & 31);
  r.present = r.pos < c && at == x;
  r.cw = c | (cap > kLeaf ? kMultiLeaf : cap << kCapShift);
  return r;
}

__global__ void k_locate_warp(const uint64_t *__restrict__ keys, uint64_t b,
                              int dbits, DGraph g, bool insert,
                              uint32_t *__restrict__ flag,
                              uint32_t *__restrict__ leaf_out,
                              const uint32_t *__restrict__ wv,
                              uint64_t *__restrict__ lS, uint32_t *__restrict__ lc,
                              uint64_t sent, const uint32_t *__restrict__ nkeys) {
  pdl_wait();
  const uint64_t i = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (i >= b) return;  // whole warps
  const uint64_t nk = nkeys ? *nkeys : b;
  const uint64_t k = i < nk ? keys[i] : sent;
  if (k == sent || (i + 1 < nk && keys[i + 1] == k)) {
    if (lane == 0) {
      flag[i] = 0;
      leaf_out[i] = 0;
    }
    return;
  }
  const Located r = locate_by_warp(g, (uint32_t)(k >> dbits),
                                   (uint32_t)(k & ((1ull << dbits) - 1)));
  if (lane == 0) {
    if (r.present && insert && wv && g.vals) g.vals[r.S + r.pos] = wv[i];
    flag[i] = insert ? !r.present : r.present;
    leaf_out[i] = r.leaf;
    lS[i] = r.S;
    lc[i] = r.cw;
  }
}

__global__ void k_pack(const uint64_t *__restrict__ keys,
                       const uint32_t *__restrict__ flag,
                       const uint32_t *__restrict__ pos,
                       const uint32_t *__restrict__ leaf, uint64_t b, int dbits,
                       uint64_t *__restrict__ p_ul, uint32_t *__restrict__ p_x,
                       const uint32_t *__restrict__ wv, uint32_t *__restrict__ p_w,
                       const uint64_t *__restrict__ lS, const uint32_t *__restrict__ lc,
                       uint64_t *__restrict__ p_S, uint32_t *__restrict__ p_c) {
  pdl_wait();
  uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= b || !flag[i]) return;
  uint64_t k = keys[i];
  uint32_t j = pos[i];
  if (j >= b) return;  // positions come from a scan: never trust them blindly
  p_ul[j] = ((k >> dbits) << 32) | leaf[i];
  p_x[j] = (uint32_t)(k & ((1ull << dbits) - 1));
  if (p_w) p_w[j] = wv[i];
  p_S[j] = lS[i];
  p_c[j] = lc[i];
}

__global__ void k_group_flags(const uint64_t *__restrict__ p_ul,
                              const uint32_t *__restrict__ d_nitems, uint64_t b,
                              uint32_t *__restrict__ gflag) {
  pdl_wait();
  uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= b) return;
  uint32_t n = *d_nitems;
  gflag[j] = (j < n && (j == 0 || p_ul[j] != p_ul[j - 1])) ? 1u : 0u;
}

// Group starts, fused into the scan of the group flags: item j that opens
// a group records itself at its group's index; the last item closes the
// list with g_start[groups] = items (g_start[0] = 0 when there are none).
struct GroupStartEpi {
  const uint32_t *gflag;
  const uint32_t *d_nitems;
  uint64_t b;
  uint32_t *g_start;
  __device__ __forceinline__ void operator()(uint64_t j, uint32_t gp) const {
    const uint32_t f = gflag[j];
    if (f && gp < b) g_start[gp] = (uint32_t)j;
    const uint32_t ni = *d_nitems;
    if (ni == 0 ? j == 0 : j + 1 == ni) {
      const uint32_t ng = gp + f;
      if (ng <= b) g_start[ng] = ni;
    }
  }
};

// ---------------------------------------------------------------- step 6
// Group-level kernels run grid-stride over the device-side group count, so
// their grids do not scale with the batch bound.  Classification is one
// thread per group; the rare groups whose leaf over- or underflows are
// appended to a climb list and climbed by one warp each.
#define GRID_STRIDE(i, n)                                                     \
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < (n); \
       i += (uint64_t)gridDim.x * blockDim.x)

// The count word of the group's first item (its leaf's count and, for a
// one-leaf row, the row's capacity, as k_locate read them; nothing has
// changed either since) decides, so no vertex record or leaf count is read
// again.
__device__ __forceinline__ void classify_insert(uint32_t gid, const uint64_t *__restrict__ p_ul,
                                                const uint32_t *__restrict__ p_c,
                                                const uint32_t *__restrict__ g_start,
                                                uint8_t *__restrict__ gtype,
                                                uint8_t *__restrict__ glev,
                                                uint32_t *__restrict__ gw0,
                                                uint32_t *__restrict__ gw1,
                                                uint32_t *__restrict__ climb,
                                                uint32_t *__restrict__ nclimb) {
  const uint32_t j0 = g_start[gid], k = g_start[gid + 1] - j0;
  const uint32_t leaf = (uint32_t)p_ul[j0];
  const uint32_t cw = p_c[j0], c = cw & 0xff;
  uint8_t type = kMerge;
  uint32_t lev = 0, w0 = leaf, w1 = leaf + 1;
  if (!(cw & kMultiLeaf)) {
    if (c + k > one_leaf_cap(cw)) {  // a one-leaf row's count is its degree
      type = kResize;
      lev = 31;
      w0 = 0;
      w1 = 1;
    }
  } else if (c + k > kLeaf) {
    type = kNone;  // decided by the climb
    climb[atomicAdd(nclimb, 1u)] = gid;
  }
  gtype[gid] = type;
  glev[gid] = (uint8_t)lev;
  gw0[gid] = w0;
  gw1[gid] = w1;
}

__global__ void k_classify_insert(const uint64_t *__restrict__ p_ul,
                                  const uint32_t *__restrict__ p_c,
                                  const uint32_t *__restrict__ g_start,
                                  const uint32_t *__restrict__ d_ngroups,
                                  uint8_t *__restrict__ gtype,
                                  uint8_t *__restrict__ glev,
                                  uint32_t *__restrict__ gw0,
                                  uint32_t *__restrict__ gw1,
                                  uint32_t *__restrict__ climb,
                                  uint32_t *__restrict__ nclimb) {
  pdl_wait();
  const uint32_t ng = *d_ngroups;
  GRID_STRIDE(gid, ng)
    classify_insert((uint32_t)gid, p_ul, p_c, g_start, gtype, glev, gw0, gw1, climb, nclimb);
}

constexpr int kGroupsPerWarp = 4;

// The leaf holding slot S, read as its whole aligned 128-byte line (always
// inside the slab: slabs are whole lines, and a one-leaf segment never
// crosses a line), then each lane's slot of the leaf by a shuffle: the load
// does not wait on the leaf's count.
__device__ __forceinline__ uint32_t leaf_slot(uint32_t linev, uint64_t S,
                                              uint32_t c, int lane) {
  const uint32_t o = (uint32_t)(S & (kLeaf - 1));
  uint32_t a = __shfl_sync(0xffffffffu, linev, (o + lane) & 31);
  return (uint32_t)lane < c ? a : kEmpty;
}

// Groups of one item (nearly all of them: a batch rarely puts two ids in
// one leaf) take eight lanes, four at a time in a warp: lane `sub` of the
// eight holds the leaf's slots 4 sub .. 4 sub + 3 from S (kEmpty from c on),
// and the one id's place is the count of the slots below it.  The lists of
// a warp's one-item groups and of its other groups are built per chunk of
// 32 groups in shared memory (one byte per group).
constexpr int kLeafWarps = kTB / 32;  // warps of the leaf kernels' blocks
__device__ __forceinline__ void load_quarter(const uint32_t *slots, uint64_t S,
                                             uint32_t c, int sub, uint32_t (&a)[4]) {
#pragma unroll
  for (int r = 0; r < 4; r++) {
    const uint32_t p = 4 * sub + r;
    a[r] = p < c ? slots[S + p] : kEmpty;
  }
}
// slots below x in the group's eight lanes (aligned lane octets)
__device__ __forceinline__ uint32_t below_in_octet(const uint32_t (&a)[4], uint32_t x) {
  uint32_t b = (uint32_t)(a[0] < x) + (a[1] < x) + (a[2] < x) + (a[3] < x);
  b += __shfl_xor_sync(0xffffffffu, b, 1);
  b += __shfl_xor_sync(0xffffffffu, b, 2);
  b += __shfl_xor_sync(0xffffffffu, b, 4);
  return b;
}
// list the chunk's groups, one-item groups first: list[0, n1) their lanes
// in order, list[n1, cnt) the others'; returns n1
__device__ __forceinline__ uint32_t list_groups(uint8_t *list, bool ok, bool one, int lane) {
  const uint32_t okm = __ballot_sync(0xffffffffu, ok);
  const uint32_t om = __ballot_sync(0xffffffffu, ok && one);
  const uint32_t lt = (1u << lane) - 1u;
  const uint32_t n1 = __popc(om);
  __syncwarp();  // the previous chunk's lists are read
  if (ok) list[one ? __popc(om & lt) : n1 + __popc(okm & ~om & lt)] = (uint8_t)lane;
  __syncwarp();
  return n1;
}

// remove: delete inside each touched leaf, take the count off the row's
// degree and classify the group: a leaf of a multi-leaf segment under the
// lower bound goes to the climb list; a one-leaf segment that emptied or
// fell to a quarter is resized.  (A one-leaf row has exactly one group, so
// its degree afterwards is its leaf's new count.)  lo_leaf is a one-leaf
// window's lower bound in a multi-leaf segment, window_lower(p, 0, H), the
// same for every H >= 1 (computed once on the host: no per-group FP64).
// A warp takes 32 groups at a time: lane l first loads group l's item
// range, its first item's leaf start, count word and key (two dependent
// loads for all 32 groups at once), then the
// groups' leaves go kGroupsPerWarp at a time with their items and leaf
// lines loaded together, one dependent load per batch; the bookkeeping
// (leaf count, degree, classification) runs once for all 32 groups, lane l
// for group l.
__device__ __forceinline__ void leaf_delete_chunk(
    const DGraph &g, uint64_t w, uint32_t ng, uint8_t *list, uint32_t lo_leaf,
    const uint64_t *__restrict__ p_ul, const uint32_t *__restrict__ p_x,
    const uint64_t *__restrict__ p_S, const uint32_t *__restrict__ p_c,
    const uint32_t *__restrict__ g_start, uint8_t *__restrict__ gtype,
    uint8_t *__restrict__ glev, uint32_t *__restrict__ gw0, uint32_t *__restrict__ gw1,
    uint32_t *__restrict__ climb, uint32_t *__restrict__ nclimb) {
  const int lane = threadIdx.x & 31, sub = lane & 7;
  constexpr int Q = kGroupsPerWarp;
  const uint64_t gl = w * 32 + lane;
  const bool okl = gl < ng;
  const uint32_t j0l = okl ? g_start[gl] : 0;
  const uint32_t kl = okl ? g_start[gl + 1] - j0l : 0;
  const uint64_t Sl = okl ? p_S[j0l] : 0;
  const uint32_t cwl = okl ? p_c[j0l] : 0;
  const uint64_t keyl = okl ? p_ul[j0l] : 0;
  const uint32_t ul = (uint32_t)(keyl >> 32), leafl = (uint32_t)keyl;
  // a one-leaf row's capacity is in its count word; a multi-leaf row
  // only needs to be told apart
  const uint32_t capl = (cwl & kMultiLeaf) ? kLeaf + 1 : one_leaf_cap(cwl);
  const uint32_t cnt = ng - w * 32 < 32 ? (uint32_t)(ng - w * 32) : 32u;
  // one-item groups: the slots from the deleted id's place on take their
  // right neighbour (kEmpty past the count)
  const uint32_t n1 = list_groups(list, okl, kl == 1 && !g.vals, lane);
  for (uint32_t f0 = 0; f0 < n1; f0 += 4) {
    const uint32_t f = f0 + (lane >> 3);
    const bool on = f < n1;
    const int src = list[on ? f : 0];
    const uint32_t j0 = __shfl_sync(0xffffffffu, j0l, src);
    const uint64_t S = __shfl_sync(0xffffffffu, Sl, src);
    const uint32_t cw = __shfl_sync(0xffffffffu, cwl, src);
    const uint32_t c = on ? (cw & 0xff) : 0u;
    const uint32_t d = on ? p_x[j0] : kEmpty;
    uint32_t a[4];
    load_quarter(g.slots, S, c, sub, a);
    const uint32_t pos = below_in_octet(a, d);
    const uint32_t nxt = __shfl_down_sync(0xffffffffu, a[0], 1, 8);
#pragma unroll
    for (int r = 0; r < 4; r++) {
      const uint32_t p = 4 * sub + r;
      if (p >= pos && p < c) g.slots[S + p] = r < 3 ? a[r + 1] : (sub == 7 ? kEmpty : nxt);
    }
  }
  // the other groups: a warp each, kGroupsPerWarp at a time
  const uint32_t nrest = cnt - n1;
  for (uint32_t q0 = 0; q0 < nrest; q0 += Q) {
    uint32_t j0[Q], k[Q], d[Q], linev[Q], cw[Q];
    uint64_t S[Q];
    bool ok[Q];
#pragma unroll
    for (int q = 0; q < Q; q++) {
      ok[q] = q0 + q < nrest;
      const int src = list[n1 + (ok[q] ? q0 + q : 0)];
      j0[q] = __shfl_sync(0xffffffffu, j0l, src);
      k[q] = ok[q] ? __shfl_sync(0xffffffffu, kl, src) : 0;
      S[q] = __shfl_sync(0xffffffffu, Sl, src);
      cw[q] = __shfl_sync(0xffffffffu, cwl, src);
    }
#pragma unroll
    for (int q = 0; q < Q; q++) {
      d[q] = (uint32_t)lane < k[q] ? p_x[j0[q] + lane] : kEmpty;
      linev[q] = ok[q] ? g.slots[(S[q] & ~uint64_t(kLeaf - 1)) + lane] : kEmpty;
    }
#pragma unroll
    for (int q = 0; q < Q; q++) {
      if (!ok[q]) break;
      const uint32_t c = cw[q] & 0xff;
      const uint32_t a = leaf_slot(linev[q], S[q], c, lane);
      bool del = false;
      for (uint32_t j = 0; j < k[q]; j++) del |= (__shfl_sync(0xffffffffu, d[q], j) == a);
      const bool keep = (uint32_t)lane < c && !del;
      const uint32_t mask = __ballot_sync(0xffffffffu, keep);
      const uint32_t pos = __popc(mask & ((1u << lane) - 1u));
      if (g.vals) {
        const uint32_t av = (uint32_t)lane < c ? g.vals[S[q] + lane] : 0u;
        __syncwarp();  // every value read before any is moved
        if (keep) g.vals[S[q] + pos] = av;
      }
      // the ids come from registers: no lane reads the line again
      if (keep) g.slots[S[q] + pos] = a;
      if ((uint32_t)lane >= c - k[q] && (uint32_t)lane < c) g.slots[S[q] + lane] = kEmpty;
    }
  }
  // the chunk's bookkeeping, lane l for group l
  const uint32_t gid = (uint32_t)(w * 32) + lane;
  bool to_climb = false;
  if (okl) {
    const uint32_t nc = (cwl & 0xff) - kl;  // every item of a group is present
    if (cwl & kMultiLeaf) g.lcnt[Sl >> kLeafLog] = (uint8_t)nc;
    atomicSub(&g.deg[ul], kl);
    uint8_t type = kNone;
    uint32_t lev = 0, w0 = leafl, w1 = leafl + 1;
    if (capl <= kLeaf) {
      if (nc == 0 || (capl > 1 && 4 * nc <= capl)) {
        type = kResize;
        lev = 31;
        w0 = 0;
        w1 = 1;
      }
    } else if (nc < lo_leaf) {
      to_climb = true;
    }
    gtype[gid] = type;
    glev[gid] = (uint8_t)lev;
    gw0[gid] = w0;
    gw1[gid] = w1;
  }
  // one reservation in the climb list for the warp's climbing groups
  const uint32_t cm = __ballot_sync(0xffffffffu, to_climb);
  if (cm) {
    uint32_t at = 0;
    if (lane == __ffs(cm) - 1) at = atomicAdd(nclimb, (uint32_t)__popc(cm));
    at = __shfl_sync(0xffffffffu, at, __ffs(cm) - 1);
    if (to_climb) climb[at + __popc(cm & ((1u << lane) - 1u))] = gid;
  }
}

__global__ void __launch_bounds__(256, 4)
k_leaf_delete(DGraph g, uint32_t lo_leaf, const uint64_t *__restrict__ p_ul,
              const uint32_t *__restrict__ p_x,
              const uint64_t *__restrict__ p_S, const uint32_t *__restrict__ p_c,
              const uint32_t *__restrict__ g_start,
              const uint32_t *__restrict__ d_ngroups,
              uint8_t *__restrict__ gtype, uint8_t *__restrict__ glev,
              uint32_t *__restrict__ gw0, uint32_t *__restrict__ gw1,
              uint32_t *__restrict__ climb, uint32_t *__restrict__ nclimb) {
  pdl_wait();
  __shared__ uint8_t glist[kLeafWarps][32];
  const uint32_t ng = *d_ngroups;
  const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  for (uint64_t w = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
       w * 32 < ng; w += nw)
    leaf_delete_chunk(g, w, ng, glist[threadIdx.x >> 5], lo_leaf, p_ul, p_x, p_S, p_c, g_start,
                      gtype, glev, gw0, gw1, climb, nclimb);
}

// window density bounds by segment height H (2^H leaves, H < kBoundsH: a
// segment holds at most 2^33 slots) and window level t <= H: entry
// [H * kBoundsH + t] of the table, window_upper for inserts, window_lower
// (the second table) for removes
constexpr uint32_t kBoundsH = 32;

// warp per climbing group: the smallest aligned window of 2^t leaves that
// meets the density bound (insert: upper bound with the batch's new ids in
// the window counted; remove: lower bound), else a resize of the segment
__device__ __forceinline__ void climb_group(const DGraph &g, const uint64_t *__restrict__ bound,
                                            bool insert, const uint64_t *__restrict__ p_ul,
                                            const uint32_t *__restrict__ g_start,
                                            uint32_t nitems, uint32_t gid,
                                            uint8_t *__restrict__ gtype,
                                            uint8_t *__restrict__ glev,
                                            uint32_t *__restrict__ gw0,
                                            uint32_t *__restrict__ gw1) {
  const int lane = threadIdx.x & 31;
  uint32_t j0 = g_start[gid];
  uint64_t key = p_ul[j0];
  uint32_t u = (uint32_t)(key >> 32), leaf = (uint32_t)key;
  uint32_t cap = g.cap[u];
  uint64_t lbase = g.base[u] >> kLeafLog;
  uint32_t H = log2_floor(cap >> kLeafLog);
  uint64_t cur = g.lcnt[lbase + leaf];
  uint32_t w0 = leaf, size = 1, w1 = leaf + 1, lev = 31;
  uint8_t type = kResize;
  const uint64_t kk = (uint64_t)u << 32;
  // new items of the growing window: bounds inside the row's items, the
  // lower one only moving left and the upper one only right
  uint32_t rb = 0, re = 0, ib = 0, ie = 0;
  if (insert) {
    rb = warp_lb_u64(p_ul, 0, j0 + 1, kk);
    re = warp_lb_u64(p_ul, j0, nitems, kk + (1ull << 32));
    ib = j0;
    ie = j0;
  }
  for (uint32_t t = 1; t <= H; t++) {
    uint32_t nw0 = (leaf >> t) << t;
    if (nw0 == w0)
      cur += warp_sum_lcnt(g.lcnt, lbase + w0 + size, lbase + w0 + 2 * size);
    else
      cur += warp_sum_lcnt(g.lcnt, lbase + nw0, lbase + w0);
    w0 = nw0;
    size <<= 1;
    w1 = w0 + size;
    bool ok;
    if (insert) {
      ib = warp_lb_u64(p_ul, rb, ib + 1 < re ? ib + 1 : re, kk | w0);
      ie = warp_lb_u64(p_ul, ie, re, kk | w1);
      ok = cur + (ie - ib) <= bound[H * kBoundsH + t];
    } else {
      ok = cur >= bound[H * kBoundsH + t];
    }
    if (ok) {
      type = kWindow;
      lev = t;
      break;
    }
  }
  if (type == kResize) {
    w0 = 0;
    w1 = cap >> kLeafLog;
  }
  if (lane == 0) {
    gtype[gid] = type;
    glev[gid] = (uint8_t)lev;
    gw0[gid] = w0;
    gw1[gid] = w1;
  }
  __syncwarp();
}

__global__ void k_climb(DGraph g, const uint64_t *__restrict__ bound, bool insert,
                        const uint64_t *__restrict__ p_ul,
                        const uint32_t *__restrict__ g_start,
                        const uint32_t *__restrict__ d_nitems,
                        const uint32_t *__restrict__ climb,
                        const uint32_t *__restrict__ nclimb,
                        uint8_t *__restrict__ gtype, uint8_t *__restrict__ glev,
                        uint32_t *__restrict__ gw0, uint32_t *__restrict__ gw1) {
  pdl_wait();
  const uint32_t nc = *nclimb, nitems = *d_nitems;
  for (uint64_t ci = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
       ci < nc; ci += ((uint64_t)gridDim.x * blockDim.x) >> 5)
    climb_group(g, bound, insert, p_ul, g_start, nitems, climb[ci], gtype, glev, gw0, gw1);
}

// ---------------------------------------------------------------- step 7
constexpr uint64_t kWinMask = (1ull << 27) - 1;

// a group's window as the two scans' keys (0 and ~0: no window)
__device__ __forceinline__ void dom_keys(uint64_t u, uint8_t type, uint64_t lev, uint64_t w0,
                                         uint64_t w1, uint64_t *f, uint64_t *bk) {
  *f = 0;
  *bk = ~0ull;
  if (type >= kWindow) {
    *f = (u << 32) | (w1 << 5) | lev;
    *bk = (u << 32) | (w0 << 5) | (31 - lev);
  }
}

__global__ void k_dom_keys(const uint64_t *__restrict__ p_ul,
                           const uint32_t *__restrict__ g_start,
                           const uint8_t *__restrict__ gtype,
                           const uint8_t *__restrict__ glev,
                           const uint32_t *__restrict__ gw0,
                           const uint32_t *__restrict__ gw1,
                           const uint32_t *__restrict__ d_ngroups, uint64_t gmax,
                           uint64_t *__restrict__ fkey,
                           uint64_t *__restrict__ bkey) {
  pdl_wait();
  uint64_t gid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= gmax) return;
  uint64_t f = 0, bk = ~0ull;
  if (gid < *d_ngroups && gtype[gid] >= kWindow)
    dom_keys(p_ul[g_start[gid]] >> 32, gtype[gid], glev[gid], gw0[gid], gw1[gid], &f, &bk);
  fkey[gid] = f;
  bkey[gid] = bk;
}

// fscan[g] = max of fkey over groups before g, bscan[g] = min of bkey over
// groups after g.  A group is covered when a window of the same row from
// either side contains its leaf and is larger (or equal and earlier).
// The group's flags: merge in the low word, task in the high word (one scan of
// the packed words gives both positions: the counts stay below 2^32).
__device__ __forceinline__ uint64_t dom_flags(uint64_t key, uint8_t type, uint32_t lev, uint64_t L,
                                              uint64_t R) {
  if (type == kNone) return 0;
  const uint64_t u = key >> 32;
  const uint32_t leaf = (uint32_t)key;
  const bool lcov = L != 0 && (L >> 32) == u && ((L >> 5) & kWinMask) > leaf;
  const bool rcov = R != ~0ull && (R >> 32) == u && ((R >> 5) & kWinMask) <= leaf;
  if (type == kMerge) return !(lcov || rcov);
  const uint32_t lt = (uint32_t)(L & 31), rt = 31u - (uint32_t)(R & 31);
  const bool dom = (lcov && lt >= lev) || (rcov && rt > lev);
  return (uint64_t)!dom << 32;
}

__global__ void k_dom_classify(const uint64_t *__restrict__ p_ul,
                               const uint32_t *__restrict__ g_start,
                               const uint8_t *__restrict__ gtype,
                               const uint8_t *__restrict__ glev,
                               const uint64_t *__restrict__ fscan,
                               const uint64_t *__restrict__ bscan,
                               const uint32_t *__restrict__ d_ngroups,
                               uint64_t gmax, uint64_t *__restrict__ mt) {
  pdl_wait();
  uint64_t gid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= gmax) return;
  mt[gid] = gid < *d_ngroups ? dom_flags(p_ul[g_start[gid]], gtype[gid], glev[gid], fscan[gid],
                                         bscan[gid])
                             : 0ull;
}


// ---------------------------------------------------------------- step 8
struct Tasks {
  uint32_t *u;
  uint32_t *w0;      // first source/destination leaf (0 for a resize)
  uint64_t *key;     // (u << 32) | w0, ascending
  uint64_t *nsrc;    // leaves read
  uint64_t *ndst;    // leaves written
  uint32_t *newbeg;  // range of packed items merged in (insert)
  uint32_t *newend;
  uint64_t *total;   // elements after the task
  uint64_t *capn;    // new capacity (resize), else 0
  uint32_t *rank;    // rank within the capacity class (resize)
  uint8_t *type;
  uint64_t *out;     // exclusive prefix of total: staging offset
  uint64_t *soff;    // exclusive prefix of nsrc
  uint64_t *doff;    // exclusive prefix of ndst
  unsigned long long *err;  // count of out-of-range staging ranks
  uint32_t *stage_v;        // weighted graphs: values staged beside the ids
  const uint32_t *p_w;      // weighted graphs: values of the packed items
};

// A task's record (the setup kernels below write it).
__device__ __forceinline__ void task_store(Tasks &t, uint64_t tid, uint32_t u, uint32_t w0,
                                           uint64_t nsrc, uint64_t ndst, uint32_t nb,
                                           uint32_t ne, uint64_t old, uint64_t capn,
                                           uint32_t rank, uint8_t type) {
  t.u[tid] = u;
  t.w0[tid] = w0;
  t.key[tid] = ((uint64_t)u << 32) | w0;
  t.nsrc[tid] = nsrc;
  t.ndst[tid] = ndst;
  t.newbeg[tid] = nb;
  t.newend[tid] = ne;
  t.total[tid] = old + (ne - nb);
  t.capn[tid] = capn;
  t.rank[tid] = rank;
  t.type[tid] = type;
}

// Each group's outputs from the merge/task scan: a merge group's item range
// (and, on an insert, "no task" for its items in itask), a task group's
// slot.  The lane of a task group then sets the task up when it is a
// resize of a one-leaf row -- the common task: the row has one group, so
// its new items are that group's (no search), and the lanes'
// capacity-class ranks come from one atomic per class and warp -- and
// lists every other task (windows, resizes of multi-leaf rows) for
// k_task_setup_hard, which takes them a warp each (a window's leaf counts
// and the row's item range by warp searches).
// k_emit's work for one group (gid with its packed flags f and positions
// p; f = 0 for a lane without a group).  Every lane of the warp calls it
// together: the class ranks and the hard list are reserved per warp.
struct EmitArgs {
  uint64_t gmax;
  const uint32_t *g_start;
  uint64_t *merge_jk;
  uint32_t *task_group;
  uint64_t inv_fill;
  bool insert;
  const uint64_t *p_ul;
  const uint32_t *p_c;  // items' count words (k_locate)
  const uint8_t *gtype;
  Tasks t;
  uint32_t *class_cnt, *hard, *nhard, *itask;
};

__device__ __forceinline__ void emit_group(const EmitArgs &a, uint64_t gid, uint64_t f,
                                           uint64_t p) {
  const uint64_t gmax = a.gmax;
  const uint32_t *__restrict__ g_start = a.g_start;
  const uint64_t *__restrict__ p_ul = a.p_ul;
  const uint8_t *__restrict__ gtype = a.gtype;
  const bool insert = a.insert;
  uint32_t *itask = a.itask;
  const int lane = threadIdx.x & 31;
  const uint32_t full = 0xffffffffu;
  const uint32_t mpos = (uint32_t)p, tpos = (uint32_t)(p >> 32);
  if ((uint32_t)f && mpos < gmax) {
    const uint32_t j0 = g_start[gid], j1 = g_start[gid + 1];
    a.merge_jk[mpos] = ((uint64_t)j0 << 32) | (j1 - j0);
    if (itask)
      for (uint32_t j = j0; j < j1; j++) itask[j] = kEmpty;
  }
  const bool task = (f >> 32) && tpos < gmax;
  bool simple = false;
  uint32_t cls = kEmpty;  // capacity class taking a rank, else none
  uint32_t u = 0, cap = 0, deg = 0, nb = 0, ne = 0;
  uint64_t capn = 0;
  uint8_t type = kNone;
  if (task) {
    a.task_group[tpos] = (uint32_t)gid;
    const uint32_t j0 = g_start[gid];
    type = gtype[gid];
    u = (uint32_t)(p_ul[j0] >> 32);
    // the count word of the group's first item holds a one-leaf row's
    // capacity and count as the batch found them (no vertex record read):
    // an insert has not changed the row yet; a remove's one group of the
    // row has taken its items off (all present)
    const uint32_t cw = a.p_c[j0];
    simple = type != kWindow && !(cw & kMultiLeaf);  // a resize of a one-leaf (or empty) row
    if (simple) {
      cap = one_leaf_cap(cw);
      const uint32_t j1 = g_start[gid + 1];
      deg = insert ? (cw & 0xff) : (cw & 0xff) - (j1 - j0);
      if (insert) {
        nb = j0;
        ne = j1;
      }
      capn = cap_for((uint64_t)deg + (ne - nb), a.inv_fill);
      if (capn > 0) cls = log2_floor(capn);
    }
  }
  // one rank reservation per class among the warp's simple lanes
  const uint32_t peers = __match_any_sync(full, cls);
  const int leader = __ffs(peers) - 1;
  uint32_t rbase = 0;
  if (cls != kEmpty && lane == leader) rbase = atomicAdd(&a.class_cnt[cls], (uint32_t)__popc(peers));
  rbase = __shfl_sync(full, rbase, leader);
  if (simple) {
    const uint32_t rank = cls != kEmpty ? rbase + __popc(peers & ((1u << lane) - 1u)) : 0u;
    const uint64_t ndst = capn == 0 ? 0 : nleaves_of((uint32_t)capn);
    Tasks t = a.t;
    task_store(t, tpos, u, 0, cap == 0 ? 0 : nleaves_of(cap), ndst, nb, ne, deg, capn, rank,
               type);
  }
  // the rest to k_task_setup_hard, one reservation for the warp
  const uint32_t hm = __ballot_sync(full, task && !simple);
  if (hm) {
    uint32_t at = 0;
    if (lane == __ffs(hm) - 1) at = atomicAdd(a.nhard, (uint32_t)__popc(hm));
    at = __shfl_sync(full, at, __ffs(hm) - 1);
    if (task && !simple) a.hard[at + __popc(hm & ((1u << lane) - 1u))] = tpos;
  }
}

__global__ void k_emit(const uint64_t *__restrict__ mt, const uint64_t *__restrict__ mtpos,
                       EmitArgs a) {
  pdl_wait();
  const uint64_t gid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const bool in = gid < a.gmax;  // no early return: the warp votes in emit_group
  emit_group(a, gid, in ? mt[gid] : 0, in ? mtpos[gid] : 0);
}

__device__ __forceinline__ void task_setup_hard(const DGraph &g, uint64_t inv_fill, bool insert,
                                                const uint64_t *__restrict__ p_ul,
                                                const uint32_t *__restrict__ g_start,
                                                const uint8_t *__restrict__ gtype,
                                                const uint32_t *__restrict__ gw0,
                                                const uint32_t *__restrict__ gw1,
                                                const uint32_t *__restrict__ task_group,
                                                uint32_t tid, uint32_t nitems, Tasks &t,
                                                uint32_t *__restrict__ class_cnt) {
  const int lane = threadIdx.x & 31;
  const uint32_t gid = task_group[tid];
  const uint32_t j0 = g_start[gid];
  const uint32_t u = (uint32_t)(p_ul[j0] >> 32);
  const uint8_t type = gtype[gid];
  const uint64_t base = g.base[u];
  const uint32_t cap = g.cap[u];
  const uint64_t kk = (uint64_t)u << 32;
  uint32_t w0, b = 0, e = 0, rank = 0;
  uint64_t nsrc, ndst, old, capn = 0;
  if (type == kWindow) {
    w0 = gw0[gid];
    const uint32_t w1 = gw1[gid];
    nsrc = w1 - w0;
    old = warp_sum_lcnt(g.lcnt, (base >> kLeafLog) + w0, (base >> kLeafLog) + w1);
    if (insert) {  // the group's first item lies between the two bounds
      b = warp_lb_u64(p_ul, 0, j0 + 1, kk | w0);
      e = warp_lb_u64(p_ul, j0, nitems, kk | w1);
    }
    ndst = nsrc;
  } else {
    w0 = 0;
    nsrc = cap == 0 ? 0 : nleaves_of(cap);
    old = g.deg[u];
    if (insert) {
      b = warp_lb_u64(p_ul, 0, j0 + 1, kk);
      e = warp_lb_u64(p_ul, j0, nitems, kk + (1ull << 32));
    }
    capn = cap_for(old + (e - b), inv_fill);
    ndst = capn == 0 ? 0 : nleaves_of((uint32_t)capn);
    if (lane == 0 && capn > 0) rank = atomicAdd(&class_cnt[log2_floor(capn)], 1u);
  }
  if (lane == 0) task_store(t, tid, u, w0, nsrc, ndst, b, e, old, capn, rank, type);
  __syncwarp();
}

__global__ void k_task_setup_hard(DGraph g, uint64_t inv_fill, bool insert,
                                  const uint64_t *__restrict__ p_ul,
                                  const uint32_t *__restrict__ g_start,
                                  const uint8_t *__restrict__ gtype,
                                  const uint32_t *__restrict__ gw0,
                                  const uint32_t *__restrict__ gw1,
                                  const uint32_t *__restrict__ task_group,
                                  const uint32_t *__restrict__ hard,
                                  const uint32_t *__restrict__ nhard,
                                  const uint32_t *__restrict__ d_nitems, Tasks t,
                                  uint32_t *__restrict__ class_cnt) {
  pdl_wait();
  const uint32_t nh = *nhard, nitems = *d_nitems;
  for (uint64_t i = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < nh;
       i += ((uint64_t)gridDim.x * blockDim.x) >> 5)
    task_setup_hard(g, inv_fill, insert, p_ul, g_start, gtype, gw0, gw1, task_group, hard[i],
                    nitems, t, class_cnt);
}

// The plan summary to the host, written by one block straight into the
// pinned host copy (mapped), with the staging-rank error count of the batches
// before it; a kernel follows the planning kernels at once (programmatic
// launch), where a copy-engine transfer would start only after they finish.
static_assert(sizeof(PlanSummary) % 8 == 0 && offsetof(PlanSummary, apply_err) % 8 == 0,
              "the plan summary is copied as 8-byte words");
__device__ __forceinline__ void plan_out(const PlanSummary *P, const unsigned long long *err,
                                         PlanSummary *host) {
  constexpr int kWords = (int)(sizeof(PlanSummary) / 8);
  constexpr int kErrWord = (int)(offsetof(PlanSummary, apply_err) / 8);
  const unsigned long long *src = reinterpret_cast<const unsigned long long *>(P);
  unsigned long long *dst = reinterpret_cast<unsigned long long *>(host);
  for (int i = threadIdx.x; i < kWords; i += blockDim.x) dst[i] = i == kErrWord ? *err : src[i];
}
__global__ void k_plan_out(const PlanSummary *__restrict__ P,
                           const unsigned long long *__restrict__ err,
                           PlanSummary *__restrict__ host) {
  pdl_wait();
  plan_out(P, err, host);
}
// the staging-rank error count alone (the end of a host-pointer call)
__global__ void k_err_out(const unsigned long long *__restrict__ err,
                          unsigned long long *__restrict__ host) {
  pdl_wait();
  if (threadIdx.x == 0) *host = *err;
}

// ---------------------------------------------------------------- step 9
// merge_jk[t] = (first item << 32) | item count of merge group t.  A warp
// takes 32 groups at a time: lane l first loads group l's item range and its
// first item's leaf start and count word (two dependent loads for all 32
// groups at once), then the groups go kGroupsPerWarp at a time with their
// items and leaf lines loaded together, one dependent load per batch.
__device__ __forceinline__ void leaf_merge_chunk(
    const DGraph &g, uint64_t w, uint32_t nmerge, uint8_t *list,
    const uint64_t *__restrict__ p_ul, const uint32_t *__restrict__ p_x,
    const uint64_t *__restrict__ p_S, const uint32_t *__restrict__ p_c,
    const uint64_t *__restrict__ merge_jk, const uint32_t *__restrict__ p_w) {
  const int lane = threadIdx.x & 31, sub = lane & 7;
  constexpr int Q = kGroupsPerWarp;
  const uint64_t gl = w * 32 + lane;
  const bool okl = gl < nmerge;
  const uint64_t jkl = okl ? merge_jk[gl] : 0;
  const uint32_t j0l = (uint32_t)(jkl >> 32), kl = (uint32_t)jkl;
  const uint64_t Sl = okl ? p_S[j0l] : 0;
  const uint32_t cwl = okl ? p_c[j0l] : 0;
  const uint32_t ul = okl ? (uint32_t)(p_ul[j0l] >> 32) : 0u;
  const uint32_t cnt = nmerge - w * 32 < 32 ? (uint32_t)(nmerge - w * 32) : 32u;
  // one-item groups: the new id goes to the count of the slots below it,
  // the slots from there up move one place right
  const uint32_t n1 = list_groups(list, okl, kl == 1 && !g.vals, lane);
  for (uint32_t f0 = 0; f0 < n1; f0 += 4) {
    const uint32_t f = f0 + (lane >> 3);
    const bool on = f < n1;
    const int src = list[on ? f : 0];
    const uint32_t j0 = __shfl_sync(0xffffffffu, j0l, src);
    const uint64_t S = __shfl_sync(0xffffffffu, Sl, src);
    const uint32_t cw = __shfl_sync(0xffffffffu, cwl, src);
    const uint32_t c = on ? (cw & 0xff) : 0u;
    const uint32_t x = on ? p_x[j0] : kEmpty;
    uint32_t a[4];
    load_quarter(g.slots, S, c, sub, a);
    const uint32_t pos = below_in_octet(a, x);
    const uint32_t prev = __shfl_up_sync(0xffffffffu, a[3], 1, 8);
#pragma unroll
    for (int r = 0; r < 4; r++) {
      const uint32_t p = 4 * sub + r;
      if (on && p >= pos && p <= c) g.slots[S + p] = p == pos ? x : (r ? a[r - 1] : prev);
    }
  }
  // the other groups: a warp each, kGroupsPerWarp at a time
  const uint32_t nrest = cnt - n1;
  for (uint32_t q0 = 0; q0 < nrest; q0 += Q) {
    uint32_t j0[Q], k[Q], x[Q], linev[Q], cw[Q];
    uint64_t S[Q];
    bool ok[Q];
#pragma unroll
    for (int q = 0; q < Q; q++) {
      ok[q] = q0 + q < nrest;
      const int src = list[n1 + (ok[q] ? q0 + q : 0)];
      j0[q] = __shfl_sync(0xffffffffu, j0l, src);
      k[q] = ok[q] ? __shfl_sync(0xffffffffu, kl, src) : 0;
      S[q] = __shfl_sync(0xffffffffu, Sl, src);
      cw[q] = __shfl_sync(0xffffffffu, cwl, src);
    }
#pragma unroll
    for (int q = 0; q < Q; q++) {
      x[q] = (uint32_t)lane < k[q] ? p_x[j0[q] + lane] : kEmpty;
      linev[q] = ok[q] ? g.slots[(S[q] & ~uint64_t(kLeaf - 1)) + lane] : kEmpty;
    }
#pragma unroll
    for (int q = 0; q < Q; q++) {
      if (!ok[q]) break;
      const uint32_t c = cw[q] & 0xff;
      const uint32_t a = leaf_slot(linev[q], S[q], c, lane);
      // merged ranks in O(k) steps (k new ids, usually one or two): an old
      // id moves up by the new ids below it; new id j lands at j + the old
      // ids below it (a ballot per new id)
      uint32_t pa = lane, px = lane;
      for (uint32_t j = 0; j < k[q]; j++) {
        uint32_t xj = __shfl_sync(0xffffffffu, x[q], j);
        pa += xj < a;
        uint32_t below = __popc(__ballot_sync(0xffffffffu, (uint32_t)lane < c && a < xj));
        if ((uint32_t)lane == j) px = j + below;
      }
      // values move with their ids (weighted graphs)
      if (g.vals) {
        const uint32_t av = (uint32_t)lane < c ? g.vals[S[q] + lane] : 0u;
        const uint32_t xv = (uint32_t)lane < k[q] ? (p_w ? p_w[j0[q] + lane] : 1u) : 0u;
        __syncwarp();  // every value read before any is moved
        if ((uint32_t)lane < c) g.vals[S[q] + pa] = av;
        if ((uint32_t)lane < k[q]) g.vals[S[q] + px] = xv;
      }
      // the ids come from registers: no lane reads the line again
      if ((uint32_t)lane < c) g.slots[S[q] + pa] = a;
      if ((uint32_t)lane < k[q]) g.slots[S[q] + px] = x[q];
    }
  }
  // the chunk's leaf counts and degrees, lane l for group l.  No task
  // reads these rows' degrees: a one-leaf row is one group (a merge or a
  // resize), and a row with a resize task has no merge group.
  if (okl) {
    if (cwl & kMultiLeaf) g.lcnt[Sl >> kLeafLog] = (uint8_t)((cwl & 0xff) + kl);
    atomicAdd(&g.deg[ul], kl);
  }
}

__global__ void __launch_bounds__(256, 4)
k_leaf_merge(DGraph g, const uint64_t *__restrict__ p_ul, const uint32_t *__restrict__ p_x,
             const uint64_t *__restrict__ p_S, const uint32_t *__restrict__ p_c,
             const uint64_t *__restrict__ merge_jk, const uint32_t *__restrict__ d_nmerge,
             const uint32_t *__restrict__ p_w) {
  pdl_wait();
  __shared__ uint8_t glist[kLeafWarps][32];
  const uint32_t nmerge = *d_nmerge;
  const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  for (uint64_t w = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
       w * 32 < nmerge; w += nw)
    leaf_merge_chunk(g, w, nmerge, glist[threadIdx.x >> 5], p_ul, p_x, p_S, p_c, merge_jk, p_w);
}

// the task of every source and destination leaf of the window / resize
// tasks (a warp per task fills its two ranges), so the apply kernels find a
// leaf's task with one load, not a binary search over the offsets; the
// source leaves' element counts beside (scnt); and, on an insert, the task
// of each new item that a task takes (k_emit marked the merged items)
// (eight lanes a task: most tasks resize a one-leaf row, one leaf each way)
__global__ void k_task_index(DGraph g, Tasks t, uint32_t ntasks, uint32_t *__restrict__ stask,
                             uint32_t *__restrict__ dtask, uint32_t *__restrict__ itask,
                             uint64_t *__restrict__ scnt) {
  pdl_wait();
  const uint64_t w = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 3;
  const uint32_t sub = threadIdx.x & 7;
  if (w >= ntasks) return;
  const uint64_t s0 = t.soff[w], ns = t.nsrc[w], d0 = t.doff[w], nd = t.ndst[w];
  if (ns) {
    const uint32_t u = t.u[w], l0 = t.w0[w];
    const uint64_t base = g.base[u];
    const uint32_t cap = g.cap[u], deg = g.deg[u];
    for (uint64_t j = sub; j < ns; j += 8) {
      stask[s0 + j] = (uint32_t)w;
      scnt[s0 + j] = leaf_count(g, base, cap, deg, l0 + (uint32_t)j);
    }
  }
  for (uint64_t j = sub; j < nd; j += 8) dtask[d0 + j] = (uint32_t)w;
  if (itask)
    for (uint32_t j = t.newbeg[w] + sub; j < t.newend[w]; j += 8) itask[j] = (uint32_t)w;
}


// old elements to their merged rank: eight lanes per source leaf, lane
// `sub` taking slots sub, sub + 8, sub + 16, sub + 24, four leaves a warp
// (the chain of dependent loads -- task, row, count, ids, rank among the
// task's new ids -- is paid once per four leaves, not once per leaf)
__device__ __forceinline__ void gather_old(const uint64_t s, const uint32_t sub, DGraph g, Tasks t, uint32_t ntasks,
                             uint64_t nsrc_total,
                             const uint64_t *spre,
                             const uint32_t *p_x,
                             uint32_t *stage,
                             const uint32_t *stask) {
  if (s >= nsrc_total) return;
  const uint64_t tau = stask[s];
  const uint32_t u = t.u[tau];
  const uint64_t soff = t.soff[tau];
  const uint32_t l = t.w0[tau] + (uint32_t)(s - soff);
  const uint64_t base = g.base[u];
  const uint32_t c = leaf_count(g, base, g.cap[u], g.deg[u], l);
  if (sub >= c) return;
  const uint64_t at = base + ((uint64_t)l << kLeafLog);
  uint32_t a[4], below[4];
#pragma unroll
  for (int r = 0; r < 4; r++) a[r] = sub + 8 * r < c ? g.slots[at + sub + 8 * r] : kEmpty;
  count_less4(p_x, t.newbeg[tau], t.newend[tau], a, below);
  const uint64_t r0 = spre[s] - spre[soff], total = t.total[tau], out = t.out[tau];
#pragma unroll
  for (int r = 0; r < 4; r++) {
    const uint32_t p = sub + 8 * r;
    if (p >= c) break;
    const uint64_t rank = r0 + p + below[r];
    if (rank >= total) {
      atomicAdd(t.err, 1ull);
      continue;
    }
    stage[out + rank] = a[r];
    if (t.stage_v) t.stage_v[out + rank] = g.vals[at + p];
  }
}

__global__ void k_gather_old(DGraph g, Tasks t, uint32_t ntasks,
                             uint64_t nsrc_total,
                             const uint64_t *__restrict__ spre,
                             const uint32_t *__restrict__ p_x,
                             uint32_t *__restrict__ stage,
                             const uint32_t *__restrict__ stask) {
  pdl_wait();
  const uint64_t s = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 3;
  const uint32_t sub = threadIdx.x & 7;
  gather_old(s, sub, g, t, ntasks, nsrc_total, spre, p_x, stage, stask);
}

// thread per packed item owned by a task: new elements to their merged rank
__device__ __forceinline__ void gather_new(const uint64_t j, DGraph g, Tasks t, uint32_t ntasks,
                             const uint64_t *spre,
                             const uint64_t *p_ul,
                             const uint32_t *p_x, uint32_t nitems,
                             uint32_t *stage,
                             const uint32_t *itask) {
  if (j >= nitems || ntasks == 0) return;
  const uint32_t tau = itask[j];
  if (tau >= ntasks) return;  // a leaf merge takes this item (kEmpty)
  const uint32_t u = (uint32_t)(p_ul[j] >> 32);
  uint32_t x = p_x[j];
  uint64_t base = g.base[u];
  uint32_t cap = g.cap[u], deg = g.deg[u];
  uint64_t old_less = 0;
  uint32_t nsrc = (uint32_t)t.nsrc[tau];
  if (nsrc > 0) {
    uint32_t w0 = t.w0[tau];
    uint32_t lo = 0, hi = nsrc;  // last leaf of the window with head <= x
    while (hi - lo > 1) {
      uint32_t mid = (lo + hi) >> 1;
      if (g.slots[base + ((uint64_t)(w0 + mid) << kLeafLog)] <= x)
        lo = mid;
      else
        hi = mid;
    }
    uint32_t l = w0 + lo;
    uint32_t c = leaf_count(g, base, cap, deg, l);
    uint32_t pos = leaf_lower_bound(g.slots + base + ((uint64_t)l << kLeafLog), c, x);
    uint64_t s0 = t.soff[tau];
    old_less = (spre[s0 + lo] - spre[s0]) + pos;
  }
  uint64_t rank = (j - t.newbeg[tau]) + old_less;
  if (rank >= t.total[tau]) {
    atomicAdd(t.err, 1ull);
    return;
  }
  stage[t.out[tau] + rank] = x;
  if (t.stage_v) t.stage_v[t.out[tau] + rank] = t.p_w ? t.p_w[j] : 1u;
}

__global__ void k_gather_new(DGraph g, Tasks t, uint32_t ntasks,
                             const uint64_t *__restrict__ spre,
                             const uint64_t *__restrict__ p_ul,
                             const uint32_t *__restrict__ p_x, uint32_t nitems,
                             uint32_t *__restrict__ stage,
                             const uint32_t *__restrict__ itask) {
  pdl_wait();
  uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  gather_new(j, g, t, ntasks, spre, p_ul, p_x, nitems, stage, itask);
}

// first slab slot of each capacity class's new segments (largest class
// first), passed by value: the apply kernels need no copy of it on the device
struct ClassStarts {
  uint64_t s[kNumClasses];
};

__device__ __forceinline__ uint64_t task_new_base(const Tasks &t, uint64_t tau,
                                                  const ClassStarts &cs) {
  const uint64_t *class_start = cs.s;
  uint64_t capn = t.capn[tau];
  return class_start[log2_floor(capn)] + (uint64_t)t.rank[tau] * capn;
}

// even redistribution of the staged elements: eight lanes per destination
// leaf (slots sub, sub + 8, sub + 16, sub + 24), four leaves a warp.  Each
// lane finds the leaf's task and its share of the task's elements itself
// (the loads are the same address across the eight; 32-bit arithmetic: a
// task holds fewer than 2^32 elements).
__device__ __forceinline__ void task_scatter(const uint64_t d, const uint32_t sub, DGraph g, Tasks t, uint32_t ntasks,
                               uint64_t ndst_total,
                               const ClassStarts class_start,
                               const uint32_t *stage,
                               const uint32_t *dtask) {
  if (d >= ndst_total) return;
  const uint64_t tau = dtask[d];
  const uint32_t i = (uint32_t)(d - t.doff[tau]);
  const uint32_t NL = (uint32_t)t.ndst[tau], T = (uint32_t)t.total[tau];
  const uint32_t per = T / NL, ext = T - per * NL;
  const uint32_t cnt = per + (i < ext);
  const uint64_t src = t.out[tau] + (uint64_t)i * per + (i < ext ? i : ext);
  uint64_t S;
  uint32_t leafsize = kLeaf;
  bool multi = true;
  if (t.type[tau] == kResize) {
    const uint64_t capn = t.capn[tau];
    S = task_new_base(t, tau, class_start) + ((uint64_t)i << kLeafLog);
    if (capn <= kLeaf) {
      leafsize = (uint32_t)capn;
      multi = false;
    }
  } else {
    S = g.base[t.u[tau]] + ((uint64_t)(t.w0[tau] + i) << kLeafLog);
  }
#pragma unroll
  for (int r = 0; r < 4; r++) {
    const uint32_t p = sub + 8 * r;
    if (p < leafsize) g.slots[S + p] = p < cnt ? stage[src + p] : kEmpty;
    if (g.vals && p < cnt) g.vals[S + p] = t.stage_v[src + p];
  }
  if (sub == 0 && multi) g.lcnt[S >> kLeafLog] = (uint8_t)cnt;
}

__global__ void k_task_scatter(DGraph g, Tasks t, uint32_t ntasks,
                               uint64_t ndst_total,
                               const ClassStarts class_start,
                               const uint32_t *__restrict__ stage,
                               const uint32_t *__restrict__ dtask) {
  pdl_wait();
  const uint64_t d = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 3;
  const uint32_t sub = threadIdx.x & 7;
  task_scatter(d, sub, g, t, ntasks, ndst_total, class_start, stage, dtask);
}

// resized rows get their new segment; every task's row gets the new items
// the task took (an insert's items are each taken by one merge group or one
// task, and the merge kernel counts its own)
__device__ __forceinline__ void task_finalize(const uint64_t tau, DGraph g, Tasks t, uint32_t ntasks,
                           const ClassStarts class_start) {
  if (tau >= ntasks) return;
  uint32_t u = t.u[tau];
  const uint32_t added = t.newend[tau] - t.newbeg[tau];
  if (added) atomicAdd(&g.deg[u], added);
  if (t.type[tau] != kResize) return;
  uint64_t capn = t.capn[tau];
  g.base[u] = capn ? task_new_base(t, tau, class_start) : 0;
  g.cap[u] = (uint32_t)capn;
}

__global__ void k_finalize(DGraph g, Tasks t, uint32_t ntasks,
                           const ClassStarts class_start) {
  pdl_wait();
  uint64_t tau = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  task_finalize(tau, g, t, ntasks, class_start);
}

// ------------------------------------------------------ small batches
// A batch of up to kSmallBatch pairs in three launches, where the general
// sequence takes about 26: each of those is one block that runs for 2 to 4 us,
// nearly all of it launch and first loads.  (1) a warp a pair locates it,
// unsorted; (2) one block sorts the pairs that change the graph and plans the
// batch, its steps a block barrier apart; (3) one cluster applies the plan, its
// steps a cluster barrier apart.  An insert and a remove at RMAT scale 20, with
// a degree copy and a lookup: 1 pair 115 -> 54 us, 300 136 -> 74, 1000 150 -> 92.
// The plan's block has 512 threads, half of what an SM holds: one of 1024 would
// wait for an idle SM where other streams' kernels run (a served graph).  Above
// kSmallBatch its shared arrays outgrow the block, and its serial share (20 us
// a batch at 1000 pairs, where the general sequence is flat) the launches.
constexpr uint32_t kSmallBatch = 1024;
constexpr int kSmallThreads = 512;
constexpr int kSmallWarps = kSmallThreads / 32;
constexpr int kSmallPer = kSmallBatch / kSmallThreads;
static_assert(kSmallPer == 2, "two items a thread");

// what the plan makes of a pair
enum : uint32_t { kPairDropped = 0, kPairKept = 1, kPairInvalid = 2 };

__global__ void k_small_locate(const uint32_t *__restrict__ pairs, uint32_t b, DGraph g, int dbits,
                               bool insert, bool drop_loops, uint64_t *__restrict__ keys,
                               uint32_t *__restrict__ state, uint32_t *__restrict__ leaf,
                               uint64_t *__restrict__ lS, uint32_t *__restrict__ lc) {
  pdl_wait();
  const uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (i >= b) return;  // whole warps
  const uint32_t r = pairs[2 * (uint64_t)i], c = pairs[2 * (uint64_t)i + 1];
  const bool ok = r < g.n && c < g.width && c != kEmpty;
  if (!ok || (drop_loops && r == c)) {
    if (lane == 0) state[i] = ok ? kPairDropped : kPairInvalid;
    return;
  }
  const Located p = locate_by_warp(g, r, c);
  if (lane == 0) {
    state[i] = p.present != insert ? kPairKept : kPairDropped;
    keys[i] = ((uint64_t)r << dbits) | c;
    leaf[i] = p.leaf;
    lS[i] = p.S;
    lc[i] = p.cw;
  }
}

// exclusive scan of a value a thread over the plan's block; sm holds one value
// a warp and is free again afterwards
template <int WARPS = kSmallWarps, typename T, typename Op>
__device__ __forceinline__ T small_scan(T v, T identity, Op op, T *total, T *sm) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const T inc = warp_inclusive(v, op);
  if (lane == 31) sm[warp] = inc;
  __syncthreads();
  if (warp == 0) {
    const T w = lane < WARPS ? sm[lane] : identity;
    const T wi = warp_inclusive(w, op);
    if (lane < WARPS) sm[lane] = wi;
  }
  __syncthreads();
  T ex = __shfl_up_sync(0xffffffffu, inc, 1);
  if (lane == 0) ex = identity;
  if (warp) ex = op(sm[warp - 1], ex);
  *total = sm[WARPS - 1];
  __syncthreads();
  return ex;
}

// Sort of n <= kSmallBatch keys in shared memory with their places i: warps
// sort runs of 32 in registers (a bitonic network of shuffles), then each key
// finds its place in its run's neighbour by binary search, run lengths doubling.
// Returns which of the two buffers holds the result.  Equal keys may change
// places.
__device__ __forceinline__ int small_sort(uint64_t (&key)[2][kSmallBatch],
                                          uint16_t (&at)[2][kSmallBatch], uint32_t n) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t N = 32;
  while (N < n) N <<= 1;
  for (uint32_t r = warp; r * 32 < N; r += kSmallWarps) {
    const uint32_t e = r * 32 + lane;
    uint64_t x = e < n ? key[0][e] : ~0ull;
    uint32_t i = e < n ? at[0][e] : 0u;
#pragma unroll
    for (int k = 2; k <= 32; k <<= 1)
#pragma unroll
      for (int j = k >> 1; j > 0; j >>= 1) {
        const uint64_t y = __shfl_xor_sync(0xffffffffu, x, j);
        const uint32_t o = __shfl_xor_sync(0xffffffffu, i, j);
        const bool low = !(lane & j), up = !(lane & k);
        if (x != y && (y < x) == (low == up)) {
          x = y;
          i = o;
        }
      }
    key[0][e] = x;
    at[0][e] = (uint16_t)i;
  }
  __syncthreads();
  int cur = 0;
  for (uint32_t len = 32; len < N; len <<= 1, cur ^= 1) {
    for (uint32_t e = threadIdx.x; e < N; e += kSmallThreads) {
      const bool second = e & len;
      const uint32_t other = (e & ~(2 * len - 1)) + (second ? 0 : len);
      const uint64_t x = key[cur][e];
      uint32_t lo = 0, cnt = len;  // keys of the other run before x
      while (cnt) {
        const uint32_t half = cnt >> 1;
        const uint64_t y = key[cur][other + lo + half];
        if (y < x || (second && y == x)) {
          lo += half + 1;
          cnt -= half + 1;
        } else {
          cnt = half;
        }
      }
      const uint32_t to = (e & ~(2 * len - 1)) + (e & (len - 1)) + lo;
      key[cur ^ 1][to] = x;
      at[cur ^ 1][to] = at[cur][e];
    }
    __syncthreads();
  }
  return cur;
}

struct SmallPlan {
  DGraph g;
  uint32_t b;      // pairs
  int dbits;
  bool insert;
  uint32_t lo_leaf;
  const uint64_t *bounds;
  const uint64_t *keys;  // per pair, from k_small_locate
  const uint32_t *state, *leaf, *lc;
  const uint64_t *lS;
  uint64_t *p_ul, *p_S;  // per item, sorted
  uint32_t *p_x, *p_c;
  uint32_t *g_start, *gw0, *gw1, *climb, *hard;  // per group
  uint8_t *gtype, *glev;
  EmitArgs emit;         // its class counts and hard count are the block's own
  const unsigned long long *err;
  PlanSummary *host;
};

__global__ void __launch_bounds__(kSmallThreads) k_small_plan(SmallPlan a) {
  pdl_wait();
  __shared__ uint64_t s_key[2][kSmallBatch];
  __shared__ uint16_t s_at[2][kSmallBatch];
  __shared__ uint64_t s_w64[kSmallWarps];
  __shared__ uint32_t s_w32[kSmallWarps];
  __shared__ uint64_t s_mirror[kSmallThreads];
  __shared__ uint8_t s_list[kSmallWarps][32];
  __shared__ uint32_t s_class[kNumClasses], s_nclimb, s_nhard;
  const uint32_t t = threadIdx.x;
  const int warp = t >> 5;
  if (t < kNumClasses) s_class[t] = 0;
  if (t == 0) s_nclimb = s_nhard = 0;
  // the pairs that change the graph, to the front
  uint32_t st[kSmallPer], own = 0;
#pragma unroll
  for (int k = 0; k < kSmallPer; k++) {
    const uint32_t i = t + k * kSmallThreads;
    st[k] = i < a.b ? a.state[i] : (uint32_t)kPairDropped;
    own += st[k] == kPairKept ? 1u : st[k] == kPairInvalid ? 1u << 16 : 0u;
  }
  uint32_t tot;
  uint32_t at = small_scan(own, 0u, OpAdd{}, &tot, s_w32) & 0xffff;
  const uint32_t n = tot & 0xffff, invalid = tot >> 16;
#pragma unroll
  for (int k = 0; k < kSmallPer; k++)
    if (st[k] == kPairKept) {
      const uint32_t i = t + k * kSmallThreads;
      s_key[0][at] = a.keys[i];
      s_at[0][at++] = (uint16_t)i;
    }
  __syncthreads();
  const int cur = small_sort(s_key, s_at, n);
  // items (the first of equal pairs) and groups (one leaf of one row each)
  uint64_t *s_ul = s_key[cur ^ 1];
  uint64_t ul[kSmallPer];
  uint32_t src[kSmallPer];
#pragma unroll
  for (int k = 0; k < kSmallPer; k++) {
    const uint32_t j = kSmallPer * t + k;
    src[k] = j < n ? s_at[cur][j] : 0u;
    ul[k] = j < n ? (s_key[cur][j] >> a.dbits) << 32 | a.leaf[src[k]] : ~0ull;
    s_ul[j] = ul[k];
  }
  __syncthreads();
  bool keep[kSmallPer], head[kSmallPer];
  uint32_t cnt = 0;
#pragma unroll
  for (int k = 0; k < kSmallPer; k++) {
    const uint32_t j = kSmallPer * t + k;
    keep[k] = j < n && (j == 0 || s_key[cur][j] != s_key[cur][j - 1]);
    head[k] = keep[k] && (j == 0 || s_ul[j] != s_ul[j - 1]);
    cnt += (keep[k] ? 1u : 0u) + (head[k] ? 1u << 16 : 0u);
  }
  at = small_scan(cnt, 0u, OpAdd{}, &tot, s_w32);
  const uint32_t ni = tot & 0xffff, ng = tot >> 16;
#pragma unroll
  for (int k = 0; k < kSmallPer; k++) {
    const uint32_t j = kSmallPer * t + k, item = at & 0xffff, grp = at >> 16;
    if (head[k]) a.g_start[grp] = item;
    if (keep[k]) {
      a.p_ul[item] = ul[k];
      a.p_x[item] = (uint32_t)(s_key[cur][j] & ((1ull << a.dbits) - 1));
      a.p_S[item] = a.lS[src[k]];
      a.p_c[item] = a.lc[src[k]];
    }
    at += (keep[k] ? 1u : 0u) + (head[k] ? 1u << 16 : 0u);
  }
  if (t == 0) a.g_start[ng] = ni;
  __syncthreads();
  // classify (a remove also deletes), then the climbs
  if (a.insert) {
    for (uint32_t gid = t; gid < ng; gid += kSmallThreads)
      classify_insert(gid, a.p_ul, a.p_c, a.g_start, a.gtype, a.glev, a.gw0, a.gw1, a.climb,
                      &s_nclimb);
  } else {
    for (uint32_t w = warp; w * 32 < ng; w += kSmallWarps)
      leaf_delete_chunk(a.g, w, ng, s_list[warp], a.lo_leaf, a.p_ul, a.p_x, a.p_S, a.p_c,
                        a.g_start, a.gtype, a.glev, a.gw0, a.gw1, a.climb, &s_nclimb);
  }
  __syncthreads();
  for (uint32_t c = warp; c < s_nclimb; c += kSmallWarps)
    climb_group(a.g, a.bounds, a.insert, a.p_ul, a.g_start, ni, a.climb[c], a.gtype, a.glev,
                a.gw0, a.gw1);
  __syncthreads();
  // dominance: the largest window from either side
  uint64_t key[kSmallPer], f[kSmallPer], r[kSmallPer], flags[kSmallPer];
  uint8_t type[kSmallPer], lev[kSmallPer];
#pragma unroll
  for (int k = 0; k < kSmallPer; k++) {
    const uint32_t gid = kSmallPer * t + k;
    const bool in = gid < ng;
    key[k] = in ? a.p_ul[a.g_start[gid]] : 0ull;
    type[k] = in ? a.gtype[gid] : (uint8_t)kNone;
    lev[k] = in ? a.glev[gid] : (uint8_t)0;
    dom_keys(key[k] >> 32, type[k], lev[k], in ? a.gw0[gid] : 0u, in ? a.gw1[gid] : 0u, &f[k],
             &r[k]);
  }
  uint64_t tot64;
  const uint64_t fx = small_scan(f[0] > f[1] ? f[0] : f[1], (uint64_t)0, OpMax{}, &tot64, s_w64);
  s_mirror[kSmallThreads - 1 - t] = r[0] < r[1] ? r[0] : r[1];
  __syncthreads();
  const uint64_t rm = small_scan(s_mirror[t], ~(uint64_t)0, OpMin{}, &tot64, s_w64);
  s_mirror[kSmallThreads - 1 - t] = rm;
  __syncthreads();
  const uint64_t rx = s_mirror[t];
  flags[0] = dom_flags(key[0], type[0], lev[0], fx, r[1] < rx ? r[1] : rx);
  flags[1] = dom_flags(key[1], type[1], lev[1], f[0] > fx ? f[0] : fx, rx);
  const uint64_t px = small_scan(flags[0] + flags[1], (uint64_t)0, OpAdd{}, &tot64, s_w64);
  const uint32_t nmerge = (uint32_t)tot64, ntasks = (uint32_t)(tot64 >> 32);
  EmitArgs e = a.emit;
  e.class_cnt = s_class;
  e.nhard = &s_nhard;
  emit_group(e, kSmallPer * t, flags[0], px);
  emit_group(e, kSmallPer * t + 1, flags[1], px + flags[0]);
  __syncthreads();
  for (uint32_t i = warp; i < s_nhard; i += kSmallWarps)
    task_setup_hard(a.g, e.inv_fill, a.insert, a.p_ul, a.g_start, a.gtype, a.gw0, a.gw1,
                    e.task_group, a.hard[i], ni, e.t, s_class);
  __syncthreads();
  // the tasks' places in the staging and among the leaves read and written
  uint64_t el[kSmallPer], lf[kSmallPer], totl;
#pragma unroll
  for (int k = 0; k < kSmallPer; k++) {
    const uint32_t i = kSmallPer * t + k;
    el[k] = i < ntasks ? e.t.total[i] : 0;
    lf[k] = i < ntasks ? e.t.ndst[i] << 32 | e.t.nsrc[i] : 0;
  }
  const uint64_t ex = small_scan(el[0] + el[1], (uint64_t)0, OpAdd{}, &tot64, s_w64);
  const uint64_t lx = small_scan(lf[0] + lf[1], (uint64_t)0, OpAdd{}, &totl, s_w64);
#pragma unroll
  for (int k = 0; k < kSmallPer; k++) {
    const uint32_t i = kSmallPer * t + k;
    if (i >= ntasks) continue;
    const uint64_t l = lx + (k ? lf[0] : 0);
    e.t.out[i] = ex + (k ? el[0] : 0);
    e.t.soff[i] = l & 0xffffffffu;
    e.t.doff[i] = l >> 32;
  }
  if (t < kNumClasses) a.host->class_cnt[t] = s_class[t];
  if (t == 0) {
    a.host->n_items = ni;
    a.host->n_groups = ng;
    a.host->n_merge = nmerge;
    a.host->n_tasks = ntasks;
    a.host->n_climb = s_nclimb;
    a.host->task_elems = tot64;
    a.host->src_leaves = totl & 0xffffffffu;
    a.host->dst_leaves = totl >> 32;
    a.host->invalid = invalid;
    a.host->apply_err = *a.err;
    a.host->n_keys = n;
    a.host->n_hard = s_nhard;
  }
}

constexpr int kApplyCtas = 8;

// The merges and the tasks of a small batch by one cluster (see k_leaf_merge,
// k_task_index, k_gather_*, k_task_scatter and k_finalize).  A task's source
// leaves are prefixed by its own eight lanes.
__global__ void __cluster_dims__(kApplyCtas, 1, 1) __launch_bounds__(kSmallThreads)
k_small_apply(DGraph g, Tasks t, const ClassStarts class_start, uint32_t nmerge, uint32_t ntasks,
              uint32_t nitems, uint32_t nsrc, uint32_t ndst, const uint64_t *__restrict__ p_ul,
              const uint32_t *__restrict__ p_x, const uint64_t *__restrict__ p_S,
              const uint32_t *__restrict__ p_c, const uint64_t *__restrict__ merge_jk,
              uint32_t *stage, uint64_t *spre, uint32_t *stask, uint32_t *dtask,
              uint32_t *itask) {
  pdl_wait();
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  __shared__ uint8_t s_list[kSmallWarps][32];
  constexpr uint32_t kAll = kApplyCtas * kSmallThreads;
  const uint32_t tid = cl.block_rank() * kSmallThreads + threadIdx.x;
  const uint32_t sub = threadIdx.x & 7;
  for (uint64_t w = tid >> 5; w * 32 < nmerge; w += kAll / 32)
    leaf_merge_chunk(g, w, nmerge, s_list[threadIdx.x >> 5], p_ul, p_x, p_S, p_c, merge_jk,
                     nullptr);
  if (ntasks == 0) return;
  const uint32_t octet = 0xffu << (threadIdx.x & 24);
  for (uint32_t w = tid >> 3; w < ntasks; w += kAll / 8) {
    const uint64_t s0 = t.soff[w], ns = t.nsrc[w], d0 = t.doff[w], nd = t.ndst[w];
    if (ns) {
      const uint32_t u = t.u[w], l0 = t.w0[w];
      const uint64_t base = g.base[u];
      const uint32_t cap = g.cap[u], deg = g.deg[u];
      uint64_t run = 0;
      for (uint64_t j0 = 0; j0 < ns; j0 += 8) {
        const uint64_t j = j0 + sub;
        const uint32_t c = j < ns ? leaf_count(g, base, cap, deg, l0 + (uint32_t)j) : 0u;
        uint32_t inc = c;
#pragma unroll
        for (int d = 1; d < 8; d <<= 1) {
          const uint32_t y = __shfl_up_sync(octet, inc, d, 8);
          if (sub >= (uint32_t)d) inc += y;
        }
        if (j < ns) {
          stask[s0 + j] = w;
          spre[s0 + j] = run + inc - c;
        }
        run += __shfl_sync(octet, inc, 7, 8);
      }
    }
    for (uint64_t j = sub; j < nd; j += 8) dtask[d0 + j] = w;
    if (itask)
      for (uint32_t j = t.newbeg[w] + sub; j < t.newend[w]; j += 8) itask[j] = w;
  }
  cl.sync();
  if (itask)
    for (uint32_t j = tid; j < nitems; j += kAll)
      gather_new(j, g, t, ntasks, spre, p_ul, p_x, nitems, stage, itask);
  for (uint32_t s = tid >> 3; s < nsrc; s += kAll / 8)
    gather_old(s, sub, g, t, ntasks, nsrc, spre, p_x, stage, stask);
  cl.sync();
  for (uint32_t d = tid >> 3; d < ndst; d += kAll / 8)
    task_scatter(d, sub, g, t, ntasks, ndst, class_start, stage, dtask);
  // the scatter reads no row that a resize moves here
  for (uint32_t tau = tid; tau < ntasks; tau += kAll)
    task_finalize(tau, g, t, ntasks, class_start);
}

// ---------------------------------------------------- middling batches
// Up to kMidBatch keys, steps 4 to 8 take one block where the general sequence
// launches a grid a step: of 20 launches of 2 to 4 us, nearly all of it launch
// and first loads, 7 remain.  The steps whose work a key is long (locate, the
// removes' leaf deletes, climbs, the tasks that a warp sets up) keep their grids.
// Bound by the chain of launches.  An insert and a remove at RMAT scale 20, with a
// degree copy and a lookup: 1500 pairs 150 -> 132 us, 4000 170 -> 161; above, a
// block's share grows and a grid's does not.
constexpr uint32_t kMidBatch = 4096;
constexpr int kMidThreads = 1024, kMidWarps = kMidThreads / 32;
constexpr int kMidPer = kMidBatch / kMidThreads;

// k_pack, k_group_flags, the scans of both flags and, for inserts,
// k_classify_insert
__global__ void __launch_bounds__(kMidThreads)
k_mid_items(const uint64_t *__restrict__ keys, const uint32_t *__restrict__ flag,
            const uint32_t *__restrict__ leaf, const uint64_t *__restrict__ lS,
            const uint32_t *__restrict__ lc, uint32_t b, int dbits, bool insert, uint64_t *p_ul,
            uint32_t *__restrict__ p_x, uint64_t *__restrict__ p_S, uint32_t *p_c,
            uint32_t *g_start, uint8_t *gtype, uint8_t *glev, uint32_t *gw0, uint32_t *gw1,
            uint32_t *climb, PlanSummary *__restrict__ P) {
  pdl_wait();
  __shared__ uint64_t s_w64[kMidWarps];
  __shared__ uint32_t s_w32[kMidWarps];
  const uint32_t t = threadIdx.x;
  uint64_t key[kMidPer], ul[kMidPer], last = 0;  // last: the thread's last item's ul, plus one
  bool keep[kMidPer];
#pragma unroll
  for (int k = 0; k < kMidPer; k++) {
    const uint32_t j = kMidPer * t + k;
    keep[k] = j < b && flag[j];
    key[k] = keep[k] ? keys[j] : 0;
    ul[k] = keep[k] ? (key[k] >> dbits) << 32 | leaf[j] : 0;
    if (keep[k]) last = ul[k] + 1;
  }
  // the item before opens another group if it lies in another leaf (ul ascends)
  uint64_t tot64;
  uint64_t prev = small_scan<kMidWarps>(last, (uint64_t)0, OpMax{}, &tot64, s_w64);
  uint32_t cnt = 0;  // items | groups << 16
  bool head[kMidPer];
#pragma unroll
  for (int k = 0; k < kMidPer; k++) {
    head[k] = keep[k] && prev != ul[k] + 1;
    if (keep[k]) prev = ul[k] + 1;
    cnt += (keep[k] ? 1u : 0u) + (head[k] ? 1u << 16 : 0u);
  }
  uint32_t tot;
  uint32_t at = small_scan<kMidWarps>(cnt, 0u, OpAdd{}, &tot, s_w32);
  const uint32_t ni = tot & 0xffff, ng = tot >> 16;
#pragma unroll
  for (int k = 0; k < kMidPer; k++) {
    const uint32_t j = kMidPer * t + k, item = at & 0xffff;
    if (head[k]) g_start[at >> 16] = item;
    if (keep[k]) {
      p_ul[item] = ul[k];
      p_x[item] = (uint32_t)(key[k] & ((1ull << dbits) - 1));
      p_S[item] = lS[j];
      p_c[item] = lc[j];
    }
    at += (keep[k] ? 1u : 0u) + (head[k] ? 1u << 16 : 0u);
  }
  if (t == 0) {
    g_start[ng] = ni;
    P->n_items = ni;
    P->n_groups = ng;
  }
  if (!insert) return;
  __syncthreads();
  for (uint32_t gid = t; gid < ng; gid += kMidThreads)
    classify_insert(gid, p_ul, p_c, g_start, gtype, glev, gw0, gw1, climb, &P->n_climb);
}

// k_dom_keys, the scans from either side, k_dom_classify, the scan of the merge
// and task flags, and k_emit
__global__ void __launch_bounds__(kMidThreads)
k_mid_emit(const uint64_t *__restrict__ p_ul, const uint32_t *__restrict__ g_start,
           const uint8_t *__restrict__ gtype, const uint8_t *__restrict__ glev,
           const uint32_t *__restrict__ gw0, const uint32_t *__restrict__ gw1, EmitArgs e,
           PlanSummary *__restrict__ P) {
  pdl_wait();
  __shared__ uint64_t s_w64[kMidWarps];
  __shared__ uint64_t s_mirror[kMidThreads];
  const uint32_t t = threadIdx.x, ng = P->n_groups;
  uint64_t key[kMidPer], f[kMidPer], r[kMidPer], flags[kMidPer];
  uint8_t type[kMidPer], lev[kMidPer];
  uint64_t fmax = 0, rmin = ~0ull;
#pragma unroll
  for (int k = 0; k < kMidPer; k++) {
    const uint32_t gid = kMidPer * t + k;
    const bool in = gid < ng;
    key[k] = in ? p_ul[g_start[gid]] : 0ull;
    type[k] = in ? gtype[gid] : (uint8_t)kNone;
    lev[k] = in ? glev[gid] : (uint8_t)0;
    dom_keys(key[k] >> 32, type[k], lev[k], in ? gw0[gid] : 0u, in ? gw1[gid] : 0u, &f[k], &r[k]);
    fmax = f[k] > fmax ? f[k] : fmax;
    rmin = r[k] < rmin ? r[k] : rmin;
  }
  uint64_t tot64;
  uint64_t fx = small_scan<kMidWarps>(fmax, (uint64_t)0, OpMax{}, &tot64, s_w64);
  s_mirror[kMidThreads - 1 - t] = rmin;
  __syncthreads();
  const uint64_t rm = small_scan<kMidWarps>(s_mirror[t], ~(uint64_t)0, OpMin{}, &tot64, s_w64);
  s_mirror[kMidThreads - 1 - t] = rm;
  __syncthreads();
  uint64_t rx[kMidPer];
  rx[kMidPer - 1] = s_mirror[t];
#pragma unroll
  for (int k = kMidPer - 1; k > 0; k--) rx[k - 1] = r[k] < rx[k] ? r[k] : rx[k];
  uint64_t sum = 0;
#pragma unroll
  for (int k = 0; k < kMidPer; k++) {
    flags[k] = dom_flags(key[k], type[k], lev[k], fx, rx[k]);
    fx = f[k] > fx ? f[k] : fx;
    sum += flags[k];
  }
  uint64_t px = small_scan<kMidWarps>(sum, (uint64_t)0, OpAdd{}, &tot64, s_w64);
  if (t == 0) {
    P->n_merge = (uint32_t)tot64;
    P->n_tasks = (uint32_t)(tot64 >> 32);
  }
#pragma unroll
  for (int k = 0; k < kMidPer; k++) {
    emit_group(e, kMidPer * t + k, flags[k], px);
    px += flags[k];
  }
}

// the tasks' places in the staging and among the leaves read and written, and
// k_plan_out
__global__ void __launch_bounds__(kMidThreads)
k_mid_out(Tasks t, PlanSummary *P, const unsigned long long *__restrict__ err,
          PlanSummary *__restrict__ host) {
  pdl_wait();
  __shared__ uint64_t s_w64[kMidWarps];
  const uint32_t n = P->n_tasks;
  uint64_t el[kMidPer], src[kMidPer], dst[kMidPer], e = 0, s = 0, d = 0;
#pragma unroll
  for (int k = 0; k < kMidPer; k++) {
    const uint32_t i = kMidPer * threadIdx.x + k;
    e += el[k] = i < n ? t.total[i] : 0;
    s += src[k] = i < n ? t.nsrc[i] : 0;
    d += dst[k] = i < n ? t.ndst[i] : 0;
  }
  uint64_t te, ts, td;
  e = small_scan<kMidWarps>(e, (uint64_t)0, OpAdd{}, &te, s_w64);
  s = small_scan<kMidWarps>(s, (uint64_t)0, OpAdd{}, &ts, s_w64);
  d = small_scan<kMidWarps>(d, (uint64_t)0, OpAdd{}, &td, s_w64);
#pragma unroll
  for (int k = 0; k < kMidPer; k++) {
    const uint32_t i = kMidPer * threadIdx.x + k;
    if (i >= n) break;
    t.out[i] = e;
    t.soff[i] = s;
    t.doff[i] = d;
    e += el[k];
    s += src[k];
    d += dst[k];
  }
  if (threadIdx.x == 0) {
    P->task_elems = te;
    P->src_leaves = ts;
    P->dst_leaves = td;
  }
  __syncthreads();
  plan_out(P, err, host);
}

// ------------------------------------------------------------- first load
// Pairs loaded into a graph that holds no segment: no row has anything to be
// located, merged or moved, so the sorted keys alone give each row's size and
// each id's place: three reads of the keys and two of the rows' ranges, where the
// general sequence makes about twenty passes over them, with 295 B of scratch a pair.
// Bound by the key sort (161 of 272 us; 27 MB of slab and 38 MB of pairs take 10).
// 4.8M pairs of 300,000 rows: kernels 890 -> 272 us, and with the scratch's and the
// graph's allocation and freeing 3.04 -> 0.87 ms.

// Ranks of the kept keys (the first of each run of equal ones) among a tile of
// sorted keys: a warp takes kLoadRows runs of 32 neighbouring keys, a vote gives
// each key its rank in its run, and the block adds up the runs before it.
// Computed twice (k_load_bounds, k_load_place) rather than stored: a key is read
// in 8 bytes, and a stored flag and rank would cost 16 more.
constexpr int kLoadTB = 256, kLoadRows = 4;
constexpr int kLoadTile = kLoadTB * kLoadRows;
struct LoadTile {
  uint64_t key[kLoadRows];
  uint64_t prev[kLoadRows];  // the key before (~0 before the first)
  uint32_t rank[kLoadRows];  // within the tile
  uint32_t kept;             // bit k: key[k] is kept
  uint32_t total;            // kept keys of the tile
  __device__ __forceinline__ static uint64_t index(int k) {
    return (uint64_t)blockIdx.x * kLoadTile + (threadIdx.x >> 5) * (32 * kLoadRows) + 32 * k +
           (threadIdx.x & 31);
  }
  __device__ __forceinline__ void load(const uint64_t *__restrict__ keys, uint64_t nk,
                                       uint64_t sent, uint32_t *s_warp) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < kLoadRows; k++) {
      const uint64_t i = index(k);
      key[k] = i < nk ? keys[i] : ~0ull;
      prev[k] = i && i < nk && lane == 0 ? keys[i - 1] : ~0ull;
    }
    uint32_t run = 0;
    kept = 0;
#pragma unroll
    for (int k = 0; k < kLoadRows; k++) {
      const uint64_t up = __shfl_up_sync(0xffffffffu, key[k], 1);
      if (lane) prev[k] = up;
      const bool f = index(k) < nk && key[k] != sent && prev[k] != key[k];  // no key is ~0
      const uint32_t v = __ballot_sync(0xffffffffu, f);
      rank[k] = run + __popc(v & ((1u << lane) - 1u));
      run += __popc(v);
      kept |= (uint32_t)f << k;
    }
    if (lane == 0) s_warp[warp] = run;
    __syncthreads();
    uint32_t before = 0;
    total = 0;
#pragma unroll
    for (int w = 0; w < kLoadTB / 32; w++) {
      if (w < warp) before += s_warp[w];
      total += s_warp[w];
    }
#pragma unroll
    for (int k = 0; k < kLoadRows; k++) rank[k] += before;
  }
};

__global__ void __launch_bounds__(kLoadTB)
k_load_count(const uint64_t *__restrict__ keys, const uint32_t *__restrict__ nkeys,
             uint64_t sent, uint32_t *__restrict__ tiles) {
  pdl_wait();
  __shared__ uint32_t s_warp[kLoadTB / 32];
  LoadTile t;
  t.load(keys, *nkeys, sent, s_warp);
  if (threadIdx.x == 0) tiles[blockIdx.x] = t.total;
}

// Each row's range of ranks (rows without a key keep the 0 they were cleared to).
__global__ void __launch_bounds__(kLoadTB)
k_load_bounds(const uint64_t *__restrict__ keys, const uint32_t *__restrict__ nkeys, int dbits,
              uint64_t sent, uint32_t n, const uint32_t *__restrict__ tiles, uint32_t *__restrict__ beg,
              uint32_t *__restrict__ end) {
  pdl_wait();
  __shared__ uint32_t s_warp[kLoadTB / 32];
  LoadTile t;
  const uint64_t nk = *nkeys;
  t.load(keys, nk, sent, s_warp);
  const uint32_t at = tiles[blockIdx.x];
#pragma unroll
  for (int k = 0; k < kLoadRows; k++) {
    // a row's first key ends the row before (dropped pairs may form a row n)
    const uint64_t i = LoadTile::index(k), u = t.key[k] >> dbits;
    if (i >= nk) continue;
    if (i == 0 || (t.prev[k] >> dbits) != u) {
      if (u < n) beg[u] = at + t.rank[k];
      if (i) end[t.prev[k] >> dbits] = at + t.rank[k];
    }
    if (i + 1 == nk && u < n) end[u] = at + t.rank[k] + ((t.kept >> k) & 1u);
  }
}

// Each row's rank in its capacity class.  A block takes one range of rows,
// counts its classes in shared memory and reserves each class once: atomics on
// one address take about 25 ns each, so one a warp would be 230 us for 300,000
// rows of one class.
constexpr int kLoadThreads = 1024;
__global__ void __launch_bounds__(kLoadThreads)
k_load_rows(const uint32_t *__restrict__ beg, const uint32_t *__restrict__ end, uint32_t n,
            uint64_t inv_fill, uint32_t *__restrict__ rank, uint32_t *__restrict__ class_cnt) {
  pdl_wait();
  __shared__ uint32_t s_cnt[kNumClasses];
  for (int c = threadIdx.x; c < kNumClasses; c += kLoadThreads) s_cnt[c] = 0;
  __syncthreads();
  const uint64_t r0 = (uint64_t)n * blockIdx.x / gridDim.x;
  const uint64_t r1 = (uint64_t)n * (blockIdx.x + 1) / gridDim.x;
  for (uint64_t u = r0 + threadIdx.x; u < r1; u += kLoadThreads) {
    const uint64_t c = cap_for(end[u] - beg[u], inv_fill);
    if (c) atomicAdd(&s_cnt[log2_floor(c)], 1u);
  }
  __syncthreads();
  for (int c = threadIdx.x; c < kNumClasses; c += kLoadThreads)
    if (s_cnt[c]) s_cnt[c] = atomicAdd(&class_cnt[c], s_cnt[c]);
  __syncthreads();
  for (uint64_t u = r0 + threadIdx.x; u < r1; u += kLoadThreads) {
    const uint64_t c = cap_for(end[u] - beg[u], inv_fill);
    if (c) rank[u] = atomicAdd(&s_cnt[log2_floor(c)], 1u);
  }
}

// Each kept key's id to its slot, rows spread over their leaves as task_scatter
// spreads them (the segments' slots hold kEmpty and their leaf counts 0).  The
// thread of a row's first key writes the row's record, and that of a leaf's
// first key its count.
__global__ void __launch_bounds__(kLoadTB)
k_load_place(const uint64_t *__restrict__ keys, const uint32_t *__restrict__ nkeys, int dbits,
             uint64_t sent, const uint32_t *__restrict__ tiles, const uint32_t *__restrict__ beg,
             const uint32_t *__restrict__ end, const uint32_t *__restrict__ rank,
             uint64_t inv_fill, const ClassStarts cs, DGraph g) {
  pdl_wait();
  __shared__ uint32_t s_warp[kLoadTB / 32];
  LoadTile t;
  t.load(keys, *nkeys, sent, s_warp);
  const uint32_t tile = tiles[blockIdx.x];
#pragma unroll
  for (int k = 0; k < kLoadRows; k++) {
    if (!((t.kept >> k) & 1u)) continue;
    const uint32_t u = (uint32_t)(t.key[k] >> dbits);
    const uint32_t b0 = beg[u], deg = end[u] - b0, r = tile + t.rank[k] - b0;
    const uint64_t cap = cap_for(deg, inv_fill);
    const uint64_t base = cs.s[log2_floor(cap)] + (uint64_t)rank[u] * cap;
    if (r == 0) {
      g.base[u] = base;
      g.cap[u] = (uint32_t)cap;
      g.deg[u] = deg;
    }
    uint64_t at = base + r;
    if (cap > kLeaf) {
      const uint32_t nl = nleaves_of((uint32_t)cap), per = deg / nl, ext = deg - per * nl;
      const uint32_t cut = ext * (per + 1);  // ids of the leaves that take one more
      const uint32_t l = r < cut ? r / (per + 1) : ext + (r - cut) / per;
      const uint32_t o = r < cut ? r - l * (per + 1) : r - cut - (l - ext) * per;
      at = base + ((uint64_t)l << kLeafLog) + o;
      if (o == 0) g.lcnt[at >> kLeafLog] = (uint8_t)(per + (l < ext));
    }
    g.slots[at] = (uint32_t)(t.key[k] & ((1ull << dbits) - 1));
  }
}

// ---------------------------------------------------------------- repack
__global__ void k_class_count(const uint32_t *__restrict__ cap, uint32_t n,
                              uint32_t *__restrict__ cnt) {
  pdl_wait();
  uint32_t v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= n || cap[v] == 0) return;
  atomicAdd(&cnt[log2_floor(cap[v])], 1u);
}

__global__ void k_repack_assign(const uint32_t *__restrict__ cap, uint32_t n,
                                const uint64_t *__restrict__ class_start,
                                uint32_t *__restrict__ ctr,
                                uint64_t *__restrict__ newbase) {
  pdl_wait();
  uint32_t v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= n) return;
  uint32_t c = cap[v];
  if (c == 0) {
    newbase[v] = 0;
    return;
  }
  uint32_t cls = log2_floor(c);
  newbase[v] = class_start[cls] + (uint64_t)atomicAdd(&ctr[cls], 1u) * c;
}

__global__ void k_repack_copy(const uint32_t *__restrict__ cap, uint32_t n,
                              const uint64_t *__restrict__ oldbase,
                              const uint64_t *__restrict__ newbase,
                              const uint32_t *__restrict__ oslots,
                              const uint8_t *__restrict__ olcnt,
                              uint32_t *__restrict__ nslots_,
                              uint8_t *__restrict__ nlcnt,
                              const uint32_t *__restrict__ ovals,
                              uint32_t *__restrict__ nvals) {
  pdl_wait();
  uint64_t v = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (v >= n) return;
  uint32_t c = cap[v];
  if (c == 0) return;
  uint64_t ob = oldbase[v], nb = newbase[v];
  for (uint64_t i = lane; i < c; i += 32) nslots_[nb + i] = oslots[ob + i];
  if (ovals)
    for (uint64_t i = lane; i < c; i += 32) nvals[nb + i] = ovals[ob + i];
  if (c > kLeaf)
    for (uint64_t l = lane; l < (c >> kLeafLog); l += 32)
      nlcnt[(nb >> kLeafLog) + l] = olcnt[(ob >> kLeafLog) + l];
}


}  // namespace

// ====================================================================== host

static thread_local char g_errmsg[512];

void set_error_message(const char *fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_errmsg, sizeof(g_errmsg), fmt, ap);
  va_end(ap);
}
void set_cuda_error(cudaError_t e, const char *what, const char *file,
                    int line) {
  set_error_message("CUDA error %s (%s) at %s:%d: %s", cudaGetErrorName(e),
                    cudaGetErrorString(e), file, line, what);
}
const char *error_message() { return g_errmsg; }

void LeafDir::release() {
  cudaFree(owner);
  cudaFree(slot);
  cudaFree(cnt);
  cudaFree(pre);
  cudaFree(vleaf);
  owner = nullptr;
  slot = nullptr;
  cnt = nullptr;
  pre = nullptr;
  vleaf = nullptr;
  cap = 0;
  nleaves = 0;
  version = ~0ull;
}

void *pinned(sst_graph *g, size_t bytes) {
  if (bytes <= g->h_pinned_cap) return g->h_pinned;
  if (g->h_pinned) cudaFreeHost(g->h_pinned);
  size_t want = bytes + bytes / 4 + 4096;
  if (cudaMallocHost(&g->h_pinned, want) != cudaSuccess) {
    g->h_pinned = nullptr;
    g->h_pinned_cap = 0;
    return nullptr;
  }
  g->h_pinned_cap = want;
  return g->h_pinned;
}

uint64_t graph_device_bytes(const sst_graph *g) {
  return (uint64_t)g->n * 16 + g->nslots * (g->weighted ? 8 : 4) + g->nslots / kLeaf +
         g->arena.cap + g->work.cap + g->io.cap +
         g->dir.cap * (4 + 8 + 4 + 8) + (uint64_t)(g->n + 1) * 8 + trav_device_bytes(g);
}

sst_status release_scratch(sst_graph *g) {
  sst_status st = sync_checked(g);  // reads the last batch's device check
  if (st != SST_OK) return st;
  if (g->side) SST_CUDA_TRY(cudaStreamSynchronize(g->side));
  plan_cache_release(g);  // captured launches point into the arena
  g->arena.release();
  g->work.release();
  g->io.release();
  g->dir.release();
  trav_trim(g);
  return SST_OK;
}

static sst_status budget_check(sst_graph *g, uint64_t extra) {
  if (g->budget && graph_device_bytes(g) + extra > g->budget) {
    set_error_message("HBM budget of %llu bytes exceeded (need %llu more)",
                      (unsigned long long)g->budget,
                      (unsigned long long)extra);
    return SST_EBUDGET;
  }
  return SST_OK;
}

// A slab of nslots slots, a value each on a weighted graph, and the leaf counts,
// in one allocation (its address is *slots): cudaMalloc and cudaFree take 30 us
// each, whatever the size up to some 20 MB.
sst_status alloc_slab(const sst_graph *g, uint64_t nslots, uint32_t **slots, uint8_t **lcnt,
                      uint32_t **vals) {
  const uint64_t words = nslots * (g->weighted ? 2 : 1);
  if (cudaMalloc(slots, words * 4 + nslots / kLeaf + 1) != cudaSuccess) {
    cudaGetLastError();
    *slots = nullptr;
    set_error_message("cannot allocate a slab of %llu slots",
                      (unsigned long long)nslots);
    return SST_ENOMEM;
  }
  *vals = g->weighted ? *slots + nslots : nullptr;
  *lcnt = reinterpret_cast<uint8_t *>(*slots + words);
  return SST_OK;
}

// The host copy of the plan, in a page of its own that kernels write: a page
// registered and unregistered takes 7 and 12 us, where a pinned allocation and its
// freeing took 105 and 149.  Kernels write both alike.
static sst_status plan_host_alloc(sst_graph *g) {
  const size_t page = (size_t)sysconf(_SC_PAGESIZE);
  void *p = aligned_alloc(page, page);
  if (p && cudaHostRegister(p, page, cudaHostRegisterMapped) == cudaSuccess) {
    g->h_plan_registered = true;
  } else {
    cudaGetLastError();
    free(p);
    SST_CUDA_TRY(cudaMallocHost(&p, sizeof(PlanSummary)));
  }
  g->h_plan = static_cast<PlanSummary *>(p);
  SST_CUDA_TRY(cudaHostGetDevicePointer(reinterpret_cast<void **>(&g->h_plan_dev), p, 0));
  return SST_OK;
}
static void plan_host_free(sst_graph *g) {
  if (!g->h_plan) return;
  if (g->h_plan_registered) {
    cudaHostUnregister(g->h_plan);
    free(g->h_plan);
  } else {
    cudaFreeHost(g->h_plan);
  }
  g->h_plan = nullptr;
}

sst_status graph_init(sst_graph *g, uint32_t height, uint32_t width,
                      const sst_config *cfg) {
  g->n = height;
  g->width = width;
  g->rbits = bits_for(height);
  g->dbits = std::max(1, bits_for(width ? width - 1 : 0));
  if (cfg) {
    g->device = cfg->device;
    g->budget = cfg->hbm_budget_bytes;
    if (cfg->upper_root > 0) g->params.upper_root = cfg->upper_root;
    if (cfg->lower_root > 0) g->params.lower_root = cfg->lower_root;
    if (cfg->grow_fill > 0) g->params.grow_fill = cfg->grow_fill;
    g->keep_loops = cfg->keep_self_loops != 0;
    g->weighted = cfg->weighted != 0;
  }
  SST_CUDA_TRY(cudaSetDevice(g->device));
  SST_CUDA_TRY(cudaDeviceGetAttribute(&g->sms, cudaDevAttrMultiProcessorCount, g->device));
  SST_CUDA_TRY(cudaStreamCreateWithFlags(&g->own_stream, cudaStreamNonBlocking));
  g->stream = g->own_stream;
  uint64_t n = std::max<uint64_t>(height, 1);
  // The vertex records and the small per-graph words in one allocation, or in two
  // where that keeps each within 1 MB: beside other graphs such allocations cost next to
  // nothing, larger ones 30 us each way (65,536 rows made and freed beside
  // another graph: 268 us with one, 201 with two or more).
  constexpr uint64_t kBoundsBytes = 2 * kBoundsH * kBoundsH * 8, kSmallBlock = 1 << 20;
  auto line = [](uint64_t bytes) { return (bytes + 255) & ~uint64_t(255); };
  const uint64_t base = line(n * 8), deg = line(n * 4), bounds = deg + line(n * 4);
  const uint64_t plan = bounds + kBoundsBytes, words = plan + sizeof(PlanSummary) + 16;
  const bool two = base + words > kSmallBlock && base <= kSmallBlock && words <= kSmallBlock;
  char *blk = nullptr;
  SST_CUDA_TRY(cudaMalloc(&blk, two ? base : base + words));
  g->d_base = reinterpret_cast<uint64_t *>(blk);
  if (two) {
    SST_CUDA_TRY(cudaMemsetAsync(blk, 0, base, g->stream));
    SST_CUDA_TRY(cudaMalloc(&g->d_words, words));
    blk = static_cast<char *>(g->d_words);
  } else {
    blk += base;
  }
  g->d_cap = reinterpret_cast<uint32_t *>(blk);
  g->d_deg = reinterpret_cast<uint32_t *>(blk + deg);
  g->d_bounds = reinterpret_cast<uint64_t *>(blk + bounds);
  g->d_plan = reinterpret_cast<PlanSummary *>(blk + plan);
  g->d_err = reinterpret_cast<unsigned long long *>(blk + plan + sizeof(PlanSummary));
  g->d_scan_epoch = g->d_err + 1;
  SST_CUDA_TRY(cudaMemsetAsync(two ? blk : blk - base, 0, two ? words : base + words, g->stream));
  uint64_t slots = cfg && cfg->initial_slots ? cfg->initial_slots : (1ull << 20);
  slots = (slots + kLeaf - 1) & ~uint64_t(kLeaf - 1);
  sst_status st = budget_check(g, slots * 4 + slots / kLeaf);
  if (st != SST_OK) return st;
  st = alloc_slab(g, slots, &g->d_slots, &g->d_lcnt, &g->d_vals);
  if (st != SST_OK) return st;
  g->nslots = slots;
  g->bump = 0;
  sst_status hst = plan_host_alloc(g);
  if (hst != SST_OK) return hst;
  // the climb's density bounds per (segment height, window level), computed
  // once here with the graph's parameters: no FP64 on the device
  std::vector<uint64_t> wb(2 * kBoundsH * kBoundsH, 0);
  for (uint32_t H = 0; H < kBoundsH; H++)
    for (uint32_t t = 0; t <= H; t++) {
      wb[H * kBoundsH + t] = window_upper(g->params, t, H);
      wb[kBoundsH * kBoundsH + H * kBoundsH + t] = window_lower(g->params, t, H);
    }
  SST_CUDA_TRY(cudaMemcpyAsync(g->d_bounds, wb.data(), kBoundsBytes, cudaMemcpyHostToDevice,
                               g->stream));
  SST_CUDA_TRY(cudaStreamSynchronize(g->stream));
  return SST_OK;
}

void graph_release(sst_graph *g) {
  cudaSetDevice(g->device);
  if (g->stream) cudaStreamSynchronize(g->stream);
  cudaFree(g->d_base);   // with the other vertex records and words, or
  cudaFree(g->d_words);  // those apart, see graph_init
  cudaFree(g->d_slots);  // and the slab's values and counts
  plan_host_free(g);
  if (g->h_pinned) cudaFreeHost(g->h_pinned);
  g->arena.release();
  g->work.release();
  g->dir.release();
  trav_release(g);
  if (g->own_stream) cudaStreamDestroy(g->own_stream);
  g->own_stream = nullptr;
  if (g->plan_ready) cudaEventDestroy(g->plan_ready);
  g->plan_ready = nullptr;
  plan_cache_release(g);
  if (g->side) cudaStreamDestroy(g->side);
  if (g->fork_ev) cudaEventDestroy(g->fork_ev);
  if (g->merge_done) cudaEventDestroy(g->merge_done);
  g->side = nullptr;
  g->fork_ev = g->merge_done = nullptr;
  for (int k = 0; k < 2; k++) {
    if (g->aux[k]) cudaStreamDestroy(g->aux[k]);
    if (g->aux_join[k]) cudaEventDestroy(g->aux_join[k]);
    g->aux[k] = nullptr;
    g->aux_join[k] = nullptr;
  }
  if (g->aux_fork) cudaEventDestroy(g->aux_fork);
  g->aux_fork = nullptr;
  g->stream = nullptr;
}

sst_status graph_clone(const sst_graph *src, sst_graph *dst) {
  sst_config cfg{};
  cfg.device = src->device;
  cfg.hbm_budget_bytes = src->budget;
  cfg.initial_slots = std::max<uint64_t>(src->nslots, kLeaf);
  cfg.upper_root = src->params.upper_root;
  cfg.lower_root = src->params.lower_root;
  cfg.grow_fill = src->params.grow_fill;
  cfg.keep_self_loops = src->keep_loops ? 1u : 0u;
  cfg.weighted = src->weighted ? 1u : 0u;
  sst_status st = graph_init(dst, src->n, src->width, &cfg);
  if (st != SST_OK) return st;
  SST_CUDA_TRY(cudaStreamSynchronize(src->stream));
  uint64_t n = std::max<uint64_t>(src->n, 1);
  SST_CUDA_TRY(cudaMemcpyAsync(dst->d_base, src->d_base, n * 8, cudaMemcpyDeviceToDevice, dst->stream));
  SST_CUDA_TRY(cudaMemcpyAsync(dst->d_cap, src->d_cap, n * 4, cudaMemcpyDeviceToDevice, dst->stream));
  SST_CUDA_TRY(cudaMemcpyAsync(dst->d_deg, src->d_deg, n * 4, cudaMemcpyDeviceToDevice, dst->stream));
  SST_CUDA_TRY(cudaMemcpyAsync(dst->d_slots, src->d_slots, src->bump * 4, cudaMemcpyDeviceToDevice, dst->stream));
  if (src->d_vals)
    SST_CUDA_TRY(cudaMemcpyAsync(dst->d_vals, src->d_vals, src->bump * 4, cudaMemcpyDeviceToDevice, dst->stream));
  SST_CUDA_TRY(cudaMemcpyAsync(dst->d_lcnt, src->d_lcnt, src->bump / kLeaf + 1, cudaMemcpyDeviceToDevice, dst->stream));
  SST_CUDA_TRY(cudaStreamSynchronize(dst->stream));
  dst->bump = src->bump;
  dst->m = src->m;
  dst->version = 1;
  return SST_OK;
}

// Move every live segment into a fresh slab, packed by capacity class, with
// room for `extra` more slots.  Freed segments are reclaimed here.
sst_status repack(sst_graph *g, uint64_t extra) {
  cudaStream_t s = g->stream;
  uint32_t n = g->n;
  // own temporaries: the arena may hold a batch in flight
  char *tmp = nullptr;
  uint64_t tbytes = 512 + (uint64_t)std::max<uint32_t>(n, 1) * 8;
  SST_CUDA_TRY(cudaMalloc(&tmp, tbytes));
  uint32_t *cnt = reinterpret_cast<uint32_t *>(tmp);
  uint64_t *cstart = reinterpret_cast<uint64_t *>(tmp + 256);
  uint64_t *newbase = reinterpret_cast<uint64_t *>(tmp + 512);
  SST_CUDA_TRY(cudaMemsetAsync(cnt, 0, kNumClasses * 8, s));
  if (n) SST_LAUNCH_PDL(k_class_count, blocks_for(n), kTB, 0, s, g->d_cap, n, cnt);
  uint32_t hcnt[kNumClasses];
  SST_CUDA_TRY(cudaMemcpyAsync(hcnt, cnt, sizeof(hcnt), cudaMemcpyDeviceToHost, s));
  SST_CUDA_TRY(cudaStreamSynchronize(s));
  uint64_t hstart[kNumClasses];
  uint64_t off = 0;
  for (int c = kNumClasses - 1; c >= 0; c--) {
    hstart[c] = off;
    off += (uint64_t)hcnt[c] << c;
  }
  uint64_t live = off;
  uint64_t need = live + extra + kLeaf;
  uint64_t nsl = g->nslots;
  if (need > nsl / 2 + nsl / 4) nsl = std::max<uint64_t>(2 * need, 1ull << 20);
  nsl = (nsl + kLeaf - 1) & ~uint64_t(kLeaf - 1);
  // the new slab coexists with the old one while segments move
  sst_status st = budget_check(g, nsl * 4 + nsl / kLeaf);
  if (st != SST_OK) {
    cudaFree(tmp);
    return st;
  }
  uint32_t *nslots_, *nvals;
  uint8_t *nlcnt;
  st = alloc_slab(g, nsl, &nslots_, &nlcnt, &nvals);
  if (st != SST_OK) {
    cudaFree(tmp);
    return st;
  }
  SST_CUDA_TRY(cudaMemcpyAsync(cstart, hstart, sizeof(hstart), cudaMemcpyHostToDevice, s));
  if (n) {
    SST_LAUNCH_PDL(k_repack_assign, blocks_for(n), kTB, 0, s, g->d_cap, n, cstart,
               cnt + kNumClasses, newbase);
    SST_LAUNCH_PDL(k_repack_copy, warp_blocks(n), kTB, 0, s, g->d_cap, n, g->d_base,
               newbase, g->d_slots, g->d_lcnt, nslots_, nlcnt, g->d_vals, nvals);
    SST_CUDA_TRY(cudaMemcpyAsync(g->d_base, newbase, (uint64_t)n * 8, cudaMemcpyDeviceToDevice, s));
  }
  SST_CUDA_TRY(cudaStreamSynchronize(s));
  SST_CUDA_TRY(cudaGetLastError());
  cudaFree(g->d_slots);
  g->d_slots = nslots_;
  g->d_lcnt = nlcnt;
  g->d_vals = nvals;
  g->nslots = nsl;
  g->bump = live;
  cudaFree(tmp);
  return SST_OK;
}

// The graph's stream waits for an update's leaf merges on the side stream:
// at wait(), or when the pipeline returns early.
struct MergeJoin {
  cudaStream_t s;
  cudaEvent_t ev;
  void wait() {
    if (ev) cudaStreamWaitEvent(s, ev, 0);
    ev = nullptr;
  }
  ~MergeJoin() { wait(); }
};

// ------------------------------------------------ captured planning
// An update's planning launches (sort to plan readback) replayed as one CUDA
// graph.  They depend on the batch size, the operation and where the graph
// and the scratch live; an entry is used only when all of these match.
constexpr uint64_t kPlanGraphMaxBatch = 1u << 20;
constexpr size_t kPlanGraphs = 56;

// Launch size of a replayed batch of b pairs: b rounded up to m * 2^k with
// m in 4..7 (at least 64), so batches of nearby sizes share one captured
// sequence; at most a third more launch size than b, about 12% on average.
inline uint64_t plan_size_class(uint64_t b) {
  if (b <= 64) return 64;
  const int k = 63 - __builtin_clzll(b) - 2;  // b >> k is 4..7
  const uint64_t m = (b + (1ull << k) - 1) >> k;
  return m << k;  // m may reach 8: the next power of two
}

struct PlanKey {
  uint64_t b;
  bool insert;
  DGraph dg;
  PmaParams params;
  const char *arena;
  bool operator==(const PlanKey &o) const {
    return b == o.b && insert == o.insert && arena == o.arena &&
           memcmp(&dg, &o.dg, sizeof(DGraph)) == 0 &&
           memcmp(&params, &o.params, sizeof(PmaParams)) == 0;
  }
};
struct PlanCache {
  struct Entry {
    PlanKey key;
    cudaGraphExec_t exec;
    int64_t kernels;  // kernel launches in the captured sequence
    uint64_t used;
  };
  std::vector<Entry> entries;
  uint64_t tick = 0;
};

void plan_cache_release(sst_graph *g) {
  if (!g->plans) return;
  for (auto &e : g->plans->entries) cudaGraphExecDestroy(e.exec);
  delete g->plans;
  g->plans = nullptr;
}

// Launch the planning sequence `body` (a function of the stream it issues
// on) for this key on stream s: replayed when captured before, else captured
// on the graph's side stream first.  A capture that fails turns replay off
// for the graph; the sequence then runs directly.
template <typename Body>
static sst_status plan_graph_launch(sst_graph *g, uint64_t b, bool insert,
                                    const DGraph &dg, cudaStream_t s, Body body) {
  if (!g->plans) g->plans = new PlanCache;
  PlanCache &C = *g->plans;
  PlanKey key{b, insert, dg, g->params, g->arena.base};
  PlanCache::Entry *hit = nullptr;
  for (auto &e : C.entries)
    if (e.key == key) hit = &e;
  if (!hit) {
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    const uint64_t l0 = launches();
    const size_t mark = g->arena.used;
    cudaError_t e = cudaStreamBeginCapture(g->side, cudaStreamCaptureModeThreadLocal);
    sst_status st = SST_OK;
    if (e == cudaSuccess) {
      ProfPause quiet;
      st = body(g->side);
      e = cudaStreamEndCapture(g->side, &graph);
    }
    const int64_t kernels = (int64_t)(launches() - l0);
    note_launches(-kernels);  // captured, not launched
    if (e == cudaSuccess && st == SST_OK) e = cudaGraphInstantiate(&exec, graph, 0);
    if (graph) cudaGraphDestroy(graph);
    if (e != cudaSuccess || st != SST_OK) {
      cudaGetLastError();
      g->plan_graphs = false;
      g->arena.used = mark;
      return body(s);
    }
    if (C.entries.size() >= kPlanGraphs) {
      auto lru = std::min_element(C.entries.begin(), C.entries.end(),
                                  [](const PlanCache::Entry &x, const PlanCache::Entry &y) {
                                    return x.used < y.used;
                                  });
      cudaGraphExecDestroy(lru->exec);
      C.entries.erase(lru);
    }
    C.entries.push_back({key, exec, kernels, 0});
    hit = &C.entries.back();
  }
  hit->used = ++C.tick;
  cudaEvent_t ev = profiling("update_plan_graph") ? prof_begin(s) : nullptr;
  SST_CUDA_TRY(cudaGraphLaunch(hit->exec, s));
  if (ev) prof_end("update_plan_graph", ev, s, 0);
  note_launches(hit->kernels);
  return SST_OK;
}

// bytes of arena scratch an update batch of b pairs takes
static size_t update_scratch_bytes(uint64_t b) {
  size_t per = 8 * 2 + 4 * 5 + 8 + 4 + 4 * 3 + 1 * 2 + 4 * 2 + 8 * 4 + 4 * 6 +
               8 * 8 + 4 * 4 + 1 + 48 + 4 * 3 /* values */ +
               8 + 4 + 8 + 4 + 4 /* leaf starts and counts, merge ranges */;
  return b * per + radix_sort_scratch_bytes(b) + 8 * scan_scratch_bytes(b, 8) +
         (1 << 16);
}

// One pass of the update pipeline.  Either d_pairs (raw pairs: steps 1-2
// make and sort the keys) or presorted (keys already (row << dbits | col),
// ascending and duplicate-free, in memory outside the arena) is given.
static sst_status run_pipeline(sst_graph *g, const uint32_t *d_pairs,
                               const uint64_t *presorted, uint64_t b,
                               bool insert, uint64_t *n_invalid,
                               const uint32_t *d_w);

sst_status update_batch(sst_graph *g, const uint32_t *d_pairs, uint64_t b,
                        bool insert, uint64_t *n_invalid, const uint32_t *d_w) {
  return run_pipeline(g, d_pairs, nullptr, b, insert, n_invalid, d_w);
}

static Tasks take_tasks(const sst_graph *g, Arena &A, uint64_t b) {
  Tasks T;
  T.u = A.take<uint32_t>(b);
  T.w0 = A.take<uint32_t>(b);
  T.key = A.take<uint64_t>(b);
  T.nsrc = A.take<uint64_t>(b);
  T.ndst = A.take<uint64_t>(b);
  T.newbeg = A.take<uint32_t>(b);
  T.newend = A.take<uint32_t>(b);
  T.total = A.take<uint64_t>(b);
  T.capn = A.take<uint64_t>(b);
  T.rank = A.take<uint32_t>(b);
  T.type = A.take<uint8_t>(b);
  T.out = A.take<uint64_t>(b);
  T.soff = A.take<uint64_t>(b);
  T.doff = A.take<uint64_t>(b);
  T.err = g->d_err;
  T.stage_v = nullptr;  // weighted graphs set these
  T.p_w = nullptr;
  return T;
}

// slab slots of a plan's resized segments, and each capacity class's first one
// (largest class first, so each segment is aligned to min(cap, 32))
static uint64_t plan_growth(const PlanSummary &ps) {
  uint64_t grow = 0;
  for (int c = 0; c < kNumClasses; c++) grow += (uint64_t)ps.class_cnt[c] << c;
  return grow;
}
static ClassStarts plan_class_starts(sst_graph *g, const PlanSummary &ps) {
  ClassStarts cs;
  uint64_t off = (g->bump + kLeaf - 1) & ~uint64_t(kLeaf - 1);
  for (int c = kNumClasses - 1; c >= 0; c--) {
    cs.s[c] = off;
    off += (uint64_t)ps.class_cnt[c] << c;
  }
  if (plan_growth(ps)) g->bump = off;
  return cs;
}

// The key of a dropped pair, one that no kept pair has: on a graph that keeps no
// self-loops that of (0, 0), else of the highest column if that is out of range,
// else of a row n (a bit more if the rows too are a power of two).
static uint64_t free_column(const sst_graph *g) {
  const uint64_t c = (1ull << g->dbits) - 1;
  return c == kEmpty || g->width <= c ? c : 0;
}
static uint64_t dropped_key(const sst_graph *g) {
  if (!g->keep_loops) return 0;
  const uint64_t c = free_column(g);
  return c ? c : (uint64_t)g->n << g->dbits;
}
static int key_bits(const sst_graph *g) {
  const bool row = g->keep_loops && !free_column(g);
  return (row ? g->rbits : bits_for(g->n ? g->n - 1 : 0)) + g->dbits;
}

static void launch_packed_keys(const sst_graph *g, const uint32_t *d_pairs, uint64_t npairs,
                               bool insert, uint64_t *keys, const SortDigits &sdig,
                               cudaStream_t s) {
  PlanSummary *P = g->d_plan;
  auto launch = [&](auto *kernel) {
    SST_LAUNCH_PDL_NB("k_make_keys_packed", 16 * npairs, kernel,
                      blocks_for(npairs, kTB * kPackItems), kTB, 0, s, d_pairs, npairs, g->n,
                      g->width, g->dbits, insert && !g->keep_loops, dropped_key(g), keys,
                      reinterpret_cast<unsigned long long *>(&P->invalid), &P->n_keys, sdig);
  };
  if ((reinterpret_cast<uintptr_t>(d_pairs) & 7) == 0)
    launch(k_make_keys_packed<true>);
  else
    launch(k_make_keys_packed<false>);
}

// the plan that the kernels before it left in the mapped host copy
static sst_status read_plan(sst_graph *g, PlanSummary *ps) {
  if (!g->plan_ready)
    SST_CUDA_TRY(cudaEventCreateWithFlags(&g->plan_ready, cudaEventDisableTiming));
  SST_CUDA_TRY(cudaEventRecord(g->plan_ready, g->stream));
  SST_CUDA_TRY(cudaEventSynchronize(g->plan_ready));
  SST_CUDA_TRY(cudaGetLastError());
  *ps = *g->h_plan;
  if (ps->apply_err) {
    set_error_message("internal error: %llu failed device checks (staging rank out of range)",
                      (unsigned long long)ps->apply_err);
    return SST_EDEVICE;
  }
  return SST_OK;
}

// the streams and events of an update's parallel branches
static sst_status update_streams(sst_graph *g) {
  if (!g->side) {
    SST_CUDA_TRY(cudaStreamCreateWithFlags(&g->side, cudaStreamNonBlocking));
    SST_CUDA_TRY(cudaEventCreateWithFlags(&g->fork_ev, cudaEventDisableTiming));
    SST_CUDA_TRY(cudaEventCreateWithFlags(&g->merge_done, cudaEventDisableTiming));
  }
  if (!g->aux_fork) {
    for (int k = 0; k < 2; k++) {
      SST_CUDA_TRY(cudaStreamCreateWithFlags(&g->aux[k], cudaStreamNonBlocking));
      SST_CUDA_TRY(cudaEventCreateWithFlags(&g->aux_join[k], cudaEventDisableTiming));
    }
    SST_CUDA_TRY(cudaEventCreateWithFlags(&g->aux_fork, cudaEventDisableTiming));
  }
  return SST_OK;
}

// run k independent pieces of work on aux[0..k-1] beside the stream
static cudaError_t aux_fork(sst_graph *g, cudaStream_t from, int k) {
  cudaError_t e = cudaEventRecord(g->aux_fork, from);
  for (int i = 0; i < k && e == cudaSuccess; i++)
    e = cudaStreamWaitEvent(g->aux[i], g->aux_fork, 0);
  return e;
}
static cudaError_t aux_join(sst_graph *g, cudaStream_t to, int k) {
  cudaError_t e = cudaSuccess;
  for (int i = 0; i < k && e == cudaSuccess; i++) {
    e = cudaEventRecord(g->aux_join[i], g->aux[i]);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(to, g->aux_join[i], 0);
  }
  return e;
}

// 9b: a plan's window / resize tasks, with their staging
static sst_status apply_tasks(sst_graph *g, Tasks T, const PlanSummary &ps, bool insert,
                              const uint64_t *p_ul, const uint32_t *p_x, uint32_t *itask,
                              const ClassStarts &cstart) {
  cudaStream_t s = g->stream;
  const DGraph dg = g->view();
  // staging for window / resize tasks
  size_t wneed = ps.task_elems * (g->weighted ? 8 : 4) + ps.src_leaves * 20 +
                 ps.dst_leaves * 4 + scan_scratch_bytes(ps.src_leaves, 8) + 4096;
  if (wneed > g->work.cap) {
    sst_status st = budget_check(g, wneed - g->work.cap);
    if (st != SST_OK) return st;
  }
  SST_CUDA_TRY(g->work.reserve(wneed));
  g->work.reset();
  uint32_t *stage = g->work.take<uint32_t>(ps.task_elems);
  if (g->weighted) T.stage_v = g->work.take<uint32_t>(ps.task_elems);
  uint64_t *scnt = g->work.take<uint64_t>(ps.src_leaves);
  uint64_t *spre = g->work.take<uint64_t>(ps.src_leaves);
  uint32_t *stask = g->work.take<uint32_t>(ps.src_leaves);
  uint32_t *dtask = g->work.take<uint32_t>(ps.dst_leaves);
  uint32_t *const titem = insert && ps.n_tasks && ps.n_items ? itask : nullptr;
  if (!ps.n_tasks) return SST_OK;
  // eight lanes a task (k_task_index) and a leaf (k_gather_old,
  // k_task_scatter); the new ids' gather writes other staging slots than
  // the old ids', so it runs beside it on an aux stream
  SST_LAUNCH_PDL(k_task_index, blocks_for(8 * (uint64_t)ps.n_tasks), kTB, 0, s, dg, T,
             ps.n_tasks, stask, dtask, titem, scnt);
  if (ps.src_leaves)
    SST_CUDA_TRY((scan<uint64_t, OpAdd>(scnt, spre, ps.src_leaves, 0ull,
                                        OpAdd{}, true, false, nullptr,
                                        g->work, s)));
  const bool gnew = insert && ps.n_items;
  if (gnew && ps.src_leaves) {
    SST_CUDA_TRY(aux_fork(g, s, 1));
    SST_LAUNCH_PDL(k_gather_new, blocks_for(ps.n_items), kTB, 0, g->aux[0], dg, T,
               ps.n_tasks, spre, p_ul, p_x, ps.n_items, stage, titem);
  } else if (gnew) {
    SST_LAUNCH_PDL(k_gather_new, blocks_for(ps.n_items), kTB, 0, s, dg, T,
               ps.n_tasks, spre, p_ul, p_x, ps.n_items, stage, titem);
  }
  if (ps.src_leaves)
    SST_LAUNCH_PDL(k_gather_old, blocks_for(8 * ps.src_leaves), kTB, 0, s, dg, T,
               ps.n_tasks, ps.src_leaves, spre, p_x, stage, stask);
  if (gnew && ps.src_leaves) SST_CUDA_TRY(aux_join(g, s, 1));
  if (ps.dst_leaves)
    SST_LAUNCH_PDL(k_task_scatter, blocks_for(8 * ps.dst_leaves), kTB, 0, s, dg, T,
               ps.n_tasks, ps.dst_leaves, cstart, stage, dtask);
  SST_LAUNCH_PDL(k_finalize, blocks_for(ps.n_tasks), kTB, 0, s, dg, T, ps.n_tasks,
             cstart);
  return SST_OK;
}

// Leaves that a small batch's tasks may read and write in the cluster that applies
// it: beyond, a task's eight lanes, which add up its leaves one after another, and
// eight blocks take longer than the general sequence's six launches.  One batch that
// resizes a row of 16,384 leaves: by the cluster 489 us, by grids 224 (the general
// sequence 263); of 4,096 leaves 163 and 101; of 512 leaves 100 either way.
constexpr uint64_t kSmallLeaves = 1024;

// One pass of up to kSmallBatch raw pairs on an unweighted graph, in three
// launches (see k_small_locate); same result as run_pipeline.
static sst_status run_small(sst_graph *g, const uint32_t *d_pairs, uint32_t b, bool insert,
                            uint64_t *n_invalid) {
  cudaStream_t s = g->stream;
  // as the general sequence's (see run_pipeline), which some batches also take
  const size_t need = update_scratch_bytes(g->plan_graphs ? plan_size_class(b) : b);
  if (need > g->arena.cap) {
    sst_status st = budget_check(g, need - g->arena.cap);
    if (st != SST_OK) return st;
  }
  SST_CUDA_TRY(g->arena.reserve(need));
  Arena &A = g->arena;
  A.reset();
  const uint32_t B = b;
  uint64_t *keys = A.take<uint64_t>(B), *lS = A.take<uint64_t>(B);
  uint32_t *state = A.take<uint32_t>(B), *leaf = A.take<uint32_t>(B), *lc = A.take<uint32_t>(B);
  uint64_t *p_ul = A.take<uint64_t>(B), *p_S = A.take<uint64_t>(B);
  uint32_t *p_x = A.take<uint32_t>(B), *p_c = A.take<uint32_t>(B);
  uint32_t *g_start = A.take<uint32_t>(B + 1);
  uint32_t *gw0 = A.take<uint32_t>(B), *gw1 = A.take<uint32_t>(B);
  uint8_t *gtype = A.take<uint8_t>(B), *glev = A.take<uint8_t>(B);
  uint32_t *climb = A.take<uint32_t>(B), *hard = A.take<uint32_t>(B);
  uint64_t *merge_jk = A.take<uint64_t>(B);
  uint32_t *task_group = A.take<uint32_t>(B), *itask = A.take<uint32_t>(B);
  Tasks T = take_tasks(g, A, B);
  if (!T.doff) {
    set_error_message("update scratch sizing error");
    return SST_ENOMEM;
  }
  const DGraph dg = g->view();
  SST_LAUNCH_PDL(k_small_locate, warp_blocks(b), kTB, 0, s, d_pairs, b, dg, g->dbits, insert,
                 insert && !g->keep_loops, keys, state, leaf, lS, lc);
  const EmitArgs ea{b,    g_start, merge_jk, task_group, fill_inv_q24(g->params.grow_fill),
                    insert, p_ul,  p_c,      gtype,      T,
                    nullptr, hard, nullptr,  insert ? itask : nullptr};
  const SmallPlan sp{dg,    b,     g->dbits, insert, (uint32_t)window_lower(g->params, 0, 1),
                     g->d_bounds + (insert ? 0 : kBoundsH * kBoundsH),
                     keys,  state, leaf,     lc,     lS,
                     p_ul,  p_S,   p_x,      p_c,    g_start,
                     gw0,   gw1,   climb,    hard,   gtype,
                     glev,  ea,    g->d_err, g->h_plan_dev};
  SST_LAUNCH_PDL(k_small_plan, 1, kSmallThreads, 0, s, sp);
  PlanSummary ps;
  sst_status rst = read_plan(g, &ps);
  if (rst != SST_OK) return rst;
  if (n_invalid) *n_invalid = ps.invalid;
  // long rows: the tasks take the general sequence's grids (see kSmallLeaves)
  const bool grids = ps.src_leaves + ps.dst_leaves > kSmallLeaves;
  uint32_t *stage = nullptr, *stask = nullptr, *dtask = nullptr;
  uint64_t *spre = nullptr;
  if (!grids) {
    const size_t wneed = ps.task_elems * 4 + ps.src_leaves * 12 + ps.dst_leaves * 4 + 4096;
    if (wneed > g->work.cap) {
      sst_status st = budget_check(g, wneed - g->work.cap);
      if (st != SST_OK) return st;
    }
    SST_CUDA_TRY(g->work.reserve(wneed));
    g->work.reset();
    stage = g->work.take<uint32_t>(ps.task_elems);
    spre = g->work.take<uint64_t>(ps.src_leaves);
    stask = g->work.take<uint32_t>(ps.src_leaves);
    dtask = g->work.take<uint32_t>(ps.dst_leaves);
  }
  auto apply = [&](uint32_t nmerge, uint32_t ntasks, const ClassStarts &cs) {
    SST_LAUNCH_PDL(k_small_apply, kApplyCtas, kSmallThreads, 0, s, g->view(), T, cs, nmerge,
                   ntasks, ps.n_items, (uint32_t)ps.src_leaves, (uint32_t)ps.dst_leaves, p_ul,
                   p_x, p_S, p_c, merge_jk, stage, spre, stask, dtask, insert ? itask : nullptr);
  };
  uint32_t nmerge = insert ? ps.n_merge : 0;
  const uint64_t grow = plan_growth(ps);
  if (grow && ((g->bump + kLeaf - 1) & ~uint64_t(kLeaf - 1)) + grow > g->nslots) {
    // the merges' leaf starts point into the slab that the repack leaves
    if (nmerge) apply(nmerge, 0, ClassStarts{});
    nmerge = 0;
    sst_status st = repack(g, grow);
    if (st != SST_OK) return st;
  }
  const ClassStarts cs = plan_class_starts(g, ps);
  const uint32_t ntasks = grids ? 0 : ps.n_tasks;
  if (nmerge || ntasks) apply(nmerge, ntasks, cs);
  if (grids) {
    sst_status st = update_streams(g);
    if (st == SST_OK) st = apply_tasks(g, T, ps, insert, p_ul, p_x, itask, cs);
    if (st != SST_OK) return st;
  }
  SST_CUDA_TRY(cudaGetLastError());
  if (insert)
    g->m += ps.n_items;
  else
    g->m -= ps.n_items;
  if (ps.n_items) g->version++;
  return SST_OK;
}

// Loads from here on take run_load.  A graph made, loaded and freed, by the general
// sequence and so: 2,200 pairs of 300 rows 0.93 -> 0.66 ms, 18,000 of 2,000 rows
// 0.96 -> 0.67, 18,000 of 300,000 rows 1.20 -> 0.94, 600,000 (RMAT) of 32,768 rows
// 1.29 -> 0.84.  Smaller loads take the launches that later batches of their size
// replay.
constexpr uint64_t kLoadPairs = 2049;

// Its scratch: 16 bytes a pair, and 12 a row.  It is taken only where that is no
// more than the general sequence's (up to some 23 rows a pair), so that no load
// needs more than it did: 3,000 pairs of 2^26 rows took 805 MB and 2.3 ms, where
// the general sequence takes 1 MB and 1.8 ms.
static size_t load_scratch_bytes(uint64_t b, uint64_t n) {
  const uint64_t ntiles = (b + kLoadTile - 1) / kLoadTile;
  return b * 16 + n * 12 + ntiles * 8 + radix_sort_scratch_bytes(b) +
         scan_scratch_bytes(ntiles, 4) + (1 << 14);
}

// Pairs into a graph without segments (see LoadTile); same result as
// run_pipeline.  The slab holds nothing, so one that is too small is replaced,
// not repacked.
static sst_status run_load(sst_graph *g, const uint32_t *d_pairs, uint64_t b,
                           uint64_t *n_invalid) {
  cudaStream_t s = g->stream;
  const uint64_t n = g->n;
  const uint64_t ntiles = (b + kLoadTile - 1) / kLoadTile;
  // with room for later updates of a twelfth of the load: about what the load
  // itself takes, so that the first of them allocate nothing
  const size_t need = std::max(load_scratch_bytes(b, n), update_scratch_bytes(b / 12));
  if (need > g->arena.cap) {
    sst_status st = budget_check(g, need - g->arena.cap);
    if (st != SST_OK) return st;
  }
  SST_CUDA_TRY(g->arena.reserve(need));
  Arena &A = g->arena;
  A.reset();
  PlanSummary *P = g->d_plan;
  SST_CUDA_TRY(cudaMemsetAsync(P, 0, sizeof(PlanSummary), s));
  uint64_t *keys = A.take<uint64_t>(b), *ktmp = A.take<uint64_t>(b);
  uint32_t *tcnt = A.take<uint32_t>(ntiles), *tiles = A.take<uint32_t>(ntiles);
  uint32_t *beg = A.take<uint32_t>(2 * n), *end = beg + n, *rank = A.take<uint32_t>(n);
  if (!rank) {
    set_error_message("update scratch sizing error");
    return SST_ENOMEM;
  }
  const int dbits = g->dbits, bits = key_bits(g);
  const uint64_t sent = dropped_key(g);
  SortDigits sdig;
  if (radix_sort_digits(b, bits, A, &sdig))
    SST_CUDA_TRY(cudaMemsetAsync(sdig.totals, 0, (size_t)sdig.passes * 256 * 4, s));
  else
    sdig = SortDigits{};
  SST_CUDA_TRY(cudaMemsetAsync(beg, 0, n * 8, s));
  launch_packed_keys(g, d_pairs, b, true, keys, sdig, s);
  uint64_t *sorted = keys;
  SST_CUDA_TRY(radix_sort_u64(keys, ktmp, b, bits, A, s, &sorted, &P->n_keys,
                              sdig.passes ? &sdig : nullptr));
  SST_LAUNCH_PDL_B(8 * b, k_load_count, (unsigned)ntiles, kLoadTB, 0, s, sorted, &P->n_keys, sent,
                   tcnt);
  SST_CUDA_TRY((scan<uint32_t, OpAdd>(tcnt, tiles, ntiles, 0u, OpAdd{}, true, false, &P->n_items,
                                      A, s)));
  SST_LAUNCH_PDL_B(8 * b, k_load_bounds, (unsigned)ntiles, kLoadTB, 0, s, sorted, &P->n_keys,
                   dbits, sent, (uint32_t)n, tiles, beg, end);
  const uint64_t inv_fill = fill_inv_q24(g->params.grow_fill);
  SST_LAUNCH_PDL(k_load_rows, std::min(blocks_for(n, kLoadThreads), 2u * g->sms), kLoadThreads,
                 0, s, beg, end, (uint32_t)n, inv_fill, rank, P->class_cnt);
  SST_LAUNCH_PDL(k_plan_out, 1, 64, 0, s, P, g->d_err, g->h_plan_dev);
  PlanSummary ps;
  sst_status st = read_plan(g, &ps);
  if (st != SST_OK) return st;
  if (n_invalid) *n_invalid = ps.invalid;
  const uint64_t grow = plan_growth(ps);
  if (grow == 0) return SST_OK;
  if (grow > g->nslots) {
    // as large as repack would make it
    uint64_t nsl = std::max<uint64_t>(2 * (grow + kLeaf), 1ull << 20);
    nsl = (nsl + kLeaf - 1) & ~uint64_t(kLeaf - 1);
    st = budget_check(g, nsl * 4 + nsl / kLeaf);
    if (st != SST_OK) return st;
    uint32_t *slots, *vals;
    uint8_t *lcnt;
    st = alloc_slab(g, nsl, &slots, &lcnt, &vals);
    if (st != SST_OK) return st;
    cudaFree(g->d_slots);
    g->d_slots = slots;
    g->d_lcnt = lcnt;
    g->nslots = nsl;
  }
  const ClassStarts cs = plan_class_starts(g, ps);
  SST_CUDA_TRY(cudaMemsetAsync(g->d_slots, 0xFF, g->bump * 4, s));
  SST_CUDA_TRY(cudaMemsetAsync(g->d_lcnt, 0, g->bump / kLeaf, s));
  SST_LAUNCH_PDL_B(12 * b, k_load_place, (unsigned)ntiles, kLoadTB, 0, s, sorted, &P->n_keys,
                   dbits, sent, tiles, beg, end, rank, inv_fill, cs, g->view());
  SST_CUDA_TRY(cudaGetLastError());
  g->m += ps.n_items;
  g->version++;
  return SST_OK;
}

// d_w: the pairs' values on a weighted graph (null: value 1)
static sst_status run_pipeline(sst_graph *g, const uint32_t *d_pairs,
                               const uint64_t *presorted, uint64_t b,
                               bool insert, uint64_t *n_invalid,
                               const uint32_t *d_w) {
  if (n_invalid) *n_invalid = 0;
  if (b == 0) return SST_OK;
  if (b > 0xFFFFFFF0ull) {
    set_error_message("batch of %llu pairs exceeds 2^32", (unsigned long long)b);
    return SST_EINVAL;
  }
  if (!presorted && !g->weighted && b <= kSmallBatch)
    return run_small(g, d_pairs, (uint32_t)b, insert, n_invalid);
  if (!presorted && !g->weighted && insert && g->bump == 0 && b >= kLoadPairs && g->n &&
      load_scratch_bytes(b, g->n) <= update_scratch_bytes(b))
    return run_load(g, d_pairs, b, n_invalid);
  // Small batches are bound by the host's launch rate, so their planning
  // sequence (sort to plan readback) is captured once per size class and
  // graph layout and replayed as one graph launch.  Every launch after the
  // keys is sized by the class (b rounded up, see plan_size_class) and does
  // the work of the device-side key count.  Unweighted raw-pair batches only
  // (the keys, which read the caller's pairs, are launched directly).
  const bool wt = g->weighted && insert && !presorted;
  const uint64_t npairs = b;  // pairs the caller gave
  const bool replay = !presorted && !wt && b <= kPlanGraphMaxBatch && g->plan_graphs;
  if (replay) b = plan_size_class(b);
  cudaStream_t s = g->stream;
  size_t need = update_scratch_bytes(b);
  if (need > g->arena.cap) {
    sst_status st = budget_check(g, need - g->arena.cap);
    if (st != SST_OK) return st;
  }
  SST_CUDA_TRY(g->arena.reserve(need));
  Arena &A = g->arena;
  A.reset();
  PlanSummary *P = g->d_plan;
  SST_CUDA_TRY(cudaMemsetAsync(P, 0, sizeof(PlanSummary), s));

  const int dbits = g->dbits;
  DGraph dg = g->view();
  uint64_t *keys = A.take<uint64_t>(b), *ktmp = A.take<uint64_t>(b);
  uint32_t *flag = A.take<uint32_t>(b), *pos = A.take<uint32_t>(b + 1);
  uint32_t *leaf = A.take<uint32_t>(b);
  uint64_t *p_ul = A.take<uint64_t>(b);
  uint32_t *p_x = A.take<uint32_t>(b);
  uint32_t *gflag = A.take<uint32_t>(b);
  uint32_t *g_start = A.take<uint32_t>(b + 1);
  uint8_t *gtype = A.take<uint8_t>(b), *glev = A.take<uint8_t>(b);
  uint32_t *gw0 = A.take<uint32_t>(b), *gw1 = A.take<uint32_t>(b);
  uint64_t *fkey = A.take<uint64_t>(b), *bkey = A.take<uint64_t>(b);
  uint64_t *mt = A.take<uint64_t>(b), *mtpos = A.take<uint64_t>(b);
  uint64_t *merge_jk = A.take<uint64_t>(b);
  uint32_t *task_group = A.take<uint32_t>(b);
  // per key, then per packed item: the leaf's start slot and count word
  uint64_t *lS = A.take<uint64_t>(b), *p_S = A.take<uint64_t>(b);
  uint32_t *lc = A.take<uint32_t>(b), *p_c = A.take<uint32_t>(b);
  uint32_t *climb = A.take<uint32_t>(b);
  uint32_t *itask = A.take<uint32_t>(b);  // inserts: each item's task, or none
  Tasks T = take_tasks(g, A, b);
  // weighted graphs: values beside the keys (sorted with them) and the packed
  // items
  uint32_t *wv = wt ? A.take<uint32_t>(b) : nullptr;
  uint32_t *wtmp = wt ? A.take<uint32_t>(b) : nullptr;
  uint32_t *p_w = wt ? A.take<uint32_t>(b) : nullptr;
  T.stage_v = nullptr;  // set with the staging below
  T.p_w = p_w;

  // 1: keys
  const uint64_t *sorted = presorted;
  uint32_t *nkeys = nullptr;
  const int sort_bits = key_bits(g);  // unweighted keys
  // the key of a dropped pair (none among presorted ones)
  const uint64_t sent = presorted ? ~0ull : wt ? (uint64_t)g->n << dbits : dropped_key(g);
  SortDigits sdig;
  if (!presorted) {
    // pair in (8 B), key out (8 B)
    nkeys = wt ? nullptr : &P->n_keys;
    if (wt)
      SST_LAUNCH_PDL_B(16 * b, k_make_keys, blocks_for(b), kTB, 0, s, d_pairs, b, g->n,
                   g->width, dbits, insert && !g->keep_loops, keys,
                   reinterpret_cast<unsigned long long *>(&P->invalid), d_w, wv);
    else {
      // the sort's digit counts come from the key build when the sort takes
      // the one-sweep form (its tables taken here, before the sort's scratch)
      if (radix_sort_digits(b, sort_bits, A, &sdig)) {
        SST_CUDA_TRY(cudaMemsetAsync(sdig.totals, 0, (size_t)sdig.passes * 256 * 4, s));
      } else {
        sdig = SortDigits{};
      }
      launch_packed_keys(g, d_pairs, npairs, insert, keys, sdig, s);
    }
  }
  MergeJoin join{s, nullptr};
  // 9a (inserts): the leaf merges need only k_emit's output and their count
  // (on the device), so they run on a second stream from there, beside the
  // task planning, the plan readback and the window / resize tasks.  They
  // touch disjoint leaves: a group inside a task's window (or a resized row)
  // is that task's, not a merge, and the merges add their rows' degrees
  // themselves (no task reads those).  Every later step that could meet
  // them -- a repack of the slab, the end of the batch -- waits.
  auto fork_merges = [&](cudaStream_t from) -> sst_status {
    SST_CUDA_TRY(cudaEventRecord(g->fork_ev, from));
    SST_CUDA_TRY(cudaStreamWaitEvent(g->side, g->fork_ev, 0));
    SST_LAUNCH_PDL(k_leaf_merge, std::min(warp_blocks((b + 31) / 32), (unsigned)g->sms * 8),
               kTB, 0, g->side, dg, p_ul, p_x, p_S, p_c, merge_jk, &P->n_merge, p_w);
    SST_CUDA_TRY(cudaEventRecord(g->merge_done, g->side));
    join.ev = g->merge_done;
    return SST_OK;
  };
  sst_status ust = update_streams(g);
  if (ust != SST_OK) return ust;
  auto fork_aux = [&](cudaStream_t from, int k) { return aux_fork(g, from, k); };
  auto join_aux = [&](cudaStream_t to, int k) { return aux_join(g, to, k); };

  // 2-8: sort to plan.  For a given batch size and graph layout this is a
  // fixed sequence of launches over device-resident counts; `fork` starts
  // the merges after k_emit (a captured sequence starts them after its end).
  auto plan = [&](cudaStream_t s, bool fork) -> sst_status {
    // a replayed sequence tags its single-pass scans from the device
    DeviceScanTags tags(replay ? g->d_scan_epoch : nullptr);
    const bool mid = b <= kMidBatch && !wt;  // one-block steps: no scans to tag
    if (replay && !mid) SST_CUDA_TRY(tags.bump(s));
    if (!presorted) {
      uint64_t *out = keys;
      if (wt) {
        uint32_t *wout = wv;
        SST_CUDA_TRY(radix_sort_kv(keys, ktmp, wv, wtmp, b, g->rbits + dbits, A, s,
                                   &out, &wout));
        wv = wout;
      } else {
        SST_CUDA_TRY(radix_sort_u64(keys, ktmp, b, sort_bits, A, s, &out, nkeys,
                                    sdig.passes ? &sdig : nullptr));
      }
      sorted = out;
    }
    // 3-5: locate, pack, group
    // sorted key in (8 B), flag and leaf out (8 B)
    if (b <= kLocateWarpKeys)
      SST_LAUNCH_PDL_B(16 * b, k_locate_warp, warp_blocks(b), kTB, 0, s, sorted, b, dbits, dg,
                   insert, flag, leaf, wt ? wv : nullptr, lS, lc, sent, nkeys);
    else
      SST_LAUNCH_PDL_B(16 * b, k_locate, blocks_for(b), kTB, 0, s, sorted, b, dbits, dg,
                   insert, flag, leaf, wt ? wv : nullptr, lS, lc, sent, nkeys);
    if (mid) {
      SST_LAUNCH_PDL(k_mid_items, 1, kMidThreads, 0, s, sorted, flag, leaf, lS, lc, (uint32_t)b,
                     dbits, insert, p_ul, p_x, p_S, p_c, g_start, gtype, glev, gw0, gw1, climb, P);
    } else {
      SST_CUDA_TRY((scan<uint32_t, OpAdd>(flag, pos, b, 0u, OpAdd{}, true, false,
                                          &P->n_items, A, s)));
      SST_LAUNCH_PDL(k_pack, blocks_for(b), kTB, 0, s, sorted, flag, pos, leaf, b, dbits,
                     p_ul, p_x, wv, p_w, lS, lc, p_S, p_c);
      SST_LAUNCH_PDL(k_group_flags, blocks_for(b), kTB, 0, s, p_ul, &P->n_items, b, gflag);
      SST_CUDA_TRY((scan_epi<uint32_t, OpAdd, GroupStartEpi>(
          gflag, b, 0u, OpAdd{}, true, false, &P->n_groups, A, s, nullptr,
          GroupStartEpi{gflag, &P->n_items, b, g_start}, false)));
    }
    // 6: classify (grids capped: the kernels stride over the device count)
    const unsigned cap_blocks = (unsigned)g->sms * 8;
    const unsigned tgrid = std::min(blocks_for(b), cap_blocks);
    const unsigned wgrid = std::min(warp_blocks(b), cap_blocks);
    if (insert && mid) {
      // classified by k_mid_items
    } else if (insert) {
      SST_LAUNCH_PDL(k_classify_insert, tgrid, kTB, 0, s, p_ul, p_c, g_start,
                 &P->n_groups, gtype, glev, gw0, gw1, climb, &P->n_climb);
    } else {
      // multi-leaf segments have H >= 1 (at least two leaves)
      SST_LAUNCH_PDL(k_leaf_delete, wgrid, kTB, 0, s, dg,
                 (uint32_t)window_lower(g->params, 0, 1), p_ul, p_x, p_S, p_c,
                 g_start, &P->n_groups, gtype, glev, gw0, gw1, climb, &P->n_climb);
    }
    SST_LAUNCH_PDL(k_climb, wgrid, kTB, 0, s, dg,
               g->d_bounds + (insert ? 0 : kBoundsH * kBoundsH), insert, p_ul, g_start,
               &P->n_items, climb, &P->n_climb, gtype, glev, gw0, gw1);
    // 7-8: dominance, classification and emit.  The climb list is free
    // again: it holds the tasks that k_task_setup_hard sets up
    const EmitArgs ea{b, g_start, merge_jk, task_group,
                      fill_inv_q24(g->params.grow_fill), insert, p_ul, p_c, gtype, T,
                      P->class_cnt, climb, &P->n_hard, insert ? itask : nullptr};
    // totals land as one word on (n_merge, n_tasks), adjacent in the plan
    static_assert(offsetof(PlanSummary, n_tasks) == offsetof(PlanSummary, n_merge) + 4 &&
                      offsetof(PlanSummary, n_merge) % 8 == 0,
                  "n_merge and n_tasks share one aligned 64-bit word");
    if (mid) {
      SST_LAUNCH_PDL(k_mid_emit, 1, kMidThreads, 0, s, p_ul, g_start, gtype, glev, gw0, gw1, ea,
                     P);
      if (fork && insert) {
        sst_status st = fork_merges(s);
        if (st != SST_OK) return st;
      }
      SST_LAUNCH_PDL(k_task_setup_hard, wgrid, kTB, 0, s, dg, ea.inv_fill, insert, p_ul, g_start,
                     gtype, gw0, gw1, task_group, climb, &P->n_hard, &P->n_items, T,
                     P->class_cnt);
      SST_LAUNCH_PDL(k_mid_out, 1, kMidThreads, 0, s, T, P, g->d_err, g->h_plan_dev);
      return SST_OK;
    }
    SST_LAUNCH_PDL(k_dom_keys, blocks_for(b), kTB, 0, s, p_ul, g_start, gtype, glev,
                   gw0, gw1, &P->n_groups, b, fkey, bkey);
    // the scans run out of place into merge_jk and mtpos, which hold
    // nothing until the merge/task scan and k_emit below overwrite them
    uint64_t *fscan = merge_jk, *bscan = mtpos;
    // the two are independent: the backward one runs beside the forward one
    SST_CUDA_TRY(fork_aux(s, 1));
    SST_CUDA_TRY((scan<uint64_t, OpMax>(fkey, fscan, b, 0ull, OpMax{}, true, false,
                                        nullptr, A, s)));
    SST_CUDA_TRY((scan<uint64_t, OpMin>(bkey, bscan, b, ~0ull, OpMin{}, true, true,
                                        nullptr, A, g->aux[0])));
    SST_CUDA_TRY(join_aux(s, 1));
    SST_LAUNCH_PDL(k_dom_classify, blocks_for(b), kTB, 0, s, p_ul, g_start, gtype, glev,
                   fscan, bscan, &P->n_groups, b, mt);
    SST_CUDA_TRY((scan<uint64_t, OpAdd>(mt, mtpos, b, 0ull, OpAdd{}, true, false,
                                        reinterpret_cast<uint64_t *>(&P->n_merge), A, s)));
    SST_LAUNCH_PDL(k_emit, blocks_for(b), kTB, 0, s, mt, mtpos, ea);
    if (fork && insert) {
      sst_status st = fork_merges(s);
      if (st != SST_OK) return st;
    }
    SST_LAUNCH_PDL(k_task_setup_hard, wgrid, kTB, 0, s, dg, fill_inv_q24(g->params.grow_fill),
               insert, p_ul, g_start, gtype, gw0, gw1, task_group, climb, &P->n_hard,
               &P->n_items, T, P->class_cnt);
    // three independent scans, two of them beside the stream
    SST_CUDA_TRY(fork_aux(s, 2));
    SST_CUDA_TRY((scan<uint64_t, OpAdd>(T.total, T.out, b, 0ull, OpAdd{}, true,
                                        false, &P->task_elems, A, s, &P->n_tasks)));
    SST_CUDA_TRY((scan<uint64_t, OpAdd>(T.nsrc, T.soff, b, 0ull, OpAdd{}, true,
                                        false, &P->src_leaves, A, g->aux[0], &P->n_tasks)));
    SST_CUDA_TRY((scan<uint64_t, OpAdd>(T.ndst, T.doff, b, 0ull, OpAdd{}, true,
                                        false, &P->dst_leaves, A, g->aux[1], &P->n_tasks)));
    SST_CUDA_TRY(join_aux(s, 2));
    SST_LAUNCH_PDL(k_plan_out, 1, 64, 0, s, P, g->d_err, g->h_plan_dev);
    return SST_OK;
  };

  // replayed for small batches (the kernel profiler times a replay as one
  // entry, update_plan_graph)
  if (replay) {
    sst_status st;
    if (g->plan_direct) {
      CaptureForms forms;
      st = plan(s, false);
    } else {
      st = plan_graph_launch(g, b, insert, dg, s, [&](cudaStream_t cs) {
        return plan(cs, false);
      });
    }
    if (st != SST_OK) return st;
    if (insert) {
      st = fork_merges(s);
      if (st != SST_OK) return st;
    }
  } else {
    sst_status st = plan(s, true);
    if (st != SST_OK) return st;
  }
  PlanSummary ps;
  sst_status rst = read_plan(g, &ps);
  if (rst != SST_OK) return rst;
  if (n_invalid) *n_invalid = ps.invalid;

  const uint64_t grow = plan_growth(ps);
  if (grow > 0 && ((g->bump + kLeaf - 1) & ~uint64_t(kLeaf - 1)) + grow > g->nslots) {
    join.wait();  // the merges write the slab the repack copies and frees
    sst_status st = repack(g, grow);
    if (st != SST_OK) return st;
    dg = g->view();
    // the items' leaf starts (p_S) point into the old slab now, but the leaf
    // merges and deletes that read them have run already
  }
  const ClassStarts cstart = plan_class_starts(g, ps);

  // 9b: apply the window / resize tasks
  ust = apply_tasks(g, T, ps, insert, p_ul, p_x, itask, cstart);
  if (ust != SST_OK) return ust;
  join.wait();
  // the staging-rank check of this batch is read back with the next plan
  // (or by sst_sync), so a batch ends without a second host synchronisation
  SST_CUDA_TRY(cudaGetLastError());
  if (insert)
    g->m += ps.n_items;
  else
    g->m -= ps.n_items;
  if (ps.n_items) g->version++;
  return SST_OK;
}

// ------------------------------------------------------------ batched form
// A sequence of update batches applied as one pipeline pass.  With set
// semantics only the last operation on an edge decides whether it is present
// afterwards, so a stable sort of all pairs by edge (payload: the batch's
// operation) and a last-one-wins selection give the net removals and net
// insertions, which touch disjoint edges and run as one remove pass and one
// insert pass over already sorted keys.  Self-loops are dropped from both
// (an inserted self-loop is skipped, a removed one is absent).
namespace {
// The keys of a sequence of batches, edge ids with the batch's operation.  The
// operation is the key's low bit, below the bits that the sort looks at, so that
// no value is moved beside the key (16 bytes a pass and key, not 24); where an id
// takes all 64 bits (lo = 0) it is a value.  Digits are counted as in
// k_make_keys_packed.
__global__ void __launch_bounds__(256)
k_make_keys_batched(const uint32_t *__restrict__ pairs, uint64_t N,
                    const uint64_t *__restrict__ boff, uint32_t nb,
                    const uint8_t *__restrict__ ops, uint32_t n, uint32_t width, int dbits,
                    int lo, bool drop_loops, uint64_t sent, uint64_t *__restrict__ keys,
                    uint32_t *__restrict__ vals, unsigned long long *__restrict__ invalid,
                    SortDigits sd) {
  pdl_wait();
  __shared__ uint32_t s_hist[8][256];
  for (int p = 0; p < sd.passes; p++) s_hist[p][threadIdx.x] = 0;
  __syncthreads();
  uint32_t bad = 0;
#pragma unroll
  for (int k = 0; k < kPackItems; k++) {
    const uint64_t i = (uint64_t)blockIdx.x * (256 * kPackItems) + k * 256 + threadIdx.x;
    if (i >= N) break;
    uint32_t first = 0, last = nb;  // batch: last with boff[b] <= i
    while (last - first > 1) {
      const uint32_t mid = (first + last) >> 1;
      if (boff[mid] <= i)
        first = mid;
      else
        last = mid;
    }
    const uint32_t r = pairs[2 * i], c = pairs[2 * i + 1];
    const bool ok = r < n && c < width && c != kEmpty;
    bad += !ok;
    const uint64_t id = !ok || (drop_loops && r == c) ? sent : ((uint64_t)r << dbits) | c;
    const uint32_t op = ops[first] ? 1u : 0u;
    if (lo)
      keys[i] = id << 1 | op;
    else {
      keys[i] = id;
      vals[i] = op;
    }
    for (int p = 0; p < sd.passes; p++) atomicAdd(&s_hist[p][(id >> (8 * p)) & 0xff], 1u);
  }
  if (bad) atomicAdd(invalid, (unsigned long long)bad);
  if (!sd.passes) return;
  for (uint64_t i = (uint64_t)blockIdx.x * 256 + threadIdx.x; i < sd.status_words;
       i += (uint64_t)gridDim.x * 256)
    sd.status[i] = 0;
  __syncthreads();
  for (int p = 0; p < sd.passes; p++)
    if (s_hist[p][threadIdx.x])
      atomicAdd(&sd.totals[p * 256 + threadIdx.x], s_hist[p][threadIdx.x]);
}

// The net operations (the last of each run of equal ids) of a tile of sorted
// keys, with their ranks among the tile's insertions and removals; as LoadTile,
// computed twice rather than stored (two flags, two positions and their scans
// took 56 us for 1.8M keys, this and the scan of the tiles' counts 23).
struct NetTile {
  uint64_t id[kLoadRows];
  uint32_t rank[kLoadRows];  // in the tile, among the key's own operation
  uint32_t ins, del;         // bit k: key k is a net insertion / removal
  uint32_t nins, ndel;       // of the tile
  __device__ __forceinline__ void load(const uint64_t *__restrict__ keys,
                                       const uint32_t *__restrict__ vals, uint64_t N, int lo,
                                       uint64_t sent, uint32_t *s_warp) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t below = (1u << lane) - 1u;
    uint64_t key[kLoadRows], after[kLoadRows];
#pragma unroll
    for (int k = 0; k < kLoadRows; k++) {
      const uint64_t i = LoadTile::index(k);
      key[k] = i < N ? keys[i] : 0;
      after[k] = lane == 31 && i + 1 < N ? keys[i + 1] : 0;
    }
    uint32_t run = 0;  // insertions | removals << 16
    ins = del = 0;
#pragma unroll
    for (int k = 0; k < kLoadRows; k++) {
      const uint64_t i = LoadTile::index(k);
      const uint64_t down = __shfl_down_sync(0xffffffffu, key[k], 1);
      if (lane < 31) after[k] = down;
      id[k] = key[k] >> lo;
      const bool net = i < N && id[k] != sent && (i + 1 >= N || after[k] >> lo != id[k]);
      const bool op = lo ? key[k] & 1 : net && vals[i];
      const uint32_t vi = __ballot_sync(0xffffffffu, net && op);
      const uint32_t vd = __ballot_sync(0xffffffffu, net && !op);
      rank[k] = op ? (run & 0xffff) + __popc(vi & below) : (run >> 16) + __popc(vd & below);
      run += __popc(vi) | __popc(vd) << 16;
      ins |= (uint32_t)(net && op) << k;
      del |= (uint32_t)(net && !op) << k;
    }
    if (lane == 0) s_warp[warp] = run;
    __syncthreads();
    uint32_t before = 0, total = 0;
#pragma unroll
    for (int w = 0; w < kLoadTB / 32; w++) {
      if (w < warp) before += s_warp[w];
      total += s_warp[w];
    }
#pragma unroll
    for (int k = 0; k < kLoadRows; k++)
      rank[k] += (ins >> k) & 1u ? before & 0xffff : before >> 16;
    nins = total & 0xffff;
    ndel = total >> 16;
  }
};
static_assert(kLoadTile < 1 << 16, "a tile's counts share a word");

// tiles: (removals << 32) | insertions of each tile
__global__ void __launch_bounds__(kLoadTB)
k_net_count(const uint64_t *__restrict__ keys, const uint32_t *__restrict__ vals, uint64_t N,
            int lo, uint64_t sent, uint64_t *__restrict__ tiles) {
  pdl_wait();
  __shared__ uint32_t s_warp[kLoadTB / 32];
  NetTile t;
  t.load(keys, vals, N, lo, sent, s_warp);
  if (threadIdx.x == 0) tiles[blockIdx.x] = (uint64_t)t.ndel << 32 | t.nins;
}

__global__ void __launch_bounds__(kLoadTB)
k_net_place(const uint64_t *__restrict__ keys, const uint32_t *__restrict__ vals, uint64_t N,
            int lo, uint64_t sent, const uint64_t *__restrict__ tiles,
            uint64_t *__restrict__ ins, uint64_t *__restrict__ del) {
  pdl_wait();
  __shared__ uint32_t s_warp[kLoadTB / 32];
  NetTile t;
  t.load(keys, vals, N, lo, sent, s_warp);
  const uint64_t at = tiles[blockIdx.x];
#pragma unroll
  for (int k = 0; k < kLoadRows; k++) {
    if ((t.ins >> k) & 1u) ins[(uint32_t)at + t.rank[k]] = t.id[k];
    if ((t.del >> k) & 1u) del[(uint32_t)(at >> 32) + t.rank[k]] = t.id[k];
  }
}
}  // namespace

sst_status update_batches(sst_graph *g, const uint32_t *d_pairs,
                          const uint64_t *d_boff, const uint8_t *d_ops,
                          uint32_t nb, uint64_t N, uint64_t *n_invalid) {
  if (n_invalid) *n_invalid = 0;
  if (N == 0 || nb == 0) return SST_OK;
  if (N > 0xFFFFFFF0ull) {
    set_error_message("batched update of %llu pairs exceeds 2^32", (unsigned long long)N);
    return SST_EINVAL;
  }
  cudaStream_t s = g->stream;
  const int dbits = g->dbits;
  const uint64_t sent = dropped_key(g);
  const int bits = key_bits(g);
  const int lo = bits < 64 ? 1 : 0;  // the operation in the key, see k_make_keys_batched
  const uint64_t ntiles = (N + kLoadTile - 1) / kLoadTile;
  const size_t need = N * (lo ? 16 : 24) + ntiles * 16 + radix_sort_scratch_bytes(N) +
                      scan_scratch_bytes(ntiles, 8) + (1 << 14);
  if (need > g->arena.cap) {
    sst_status st = budget_check(g, need - g->arena.cap);
    if (st != SST_OK) return st;
  }
  SST_CUDA_TRY(g->arena.reserve(need));
  Arena &A = g->arena;
  A.reset();
  PlanSummary *P = g->d_plan;
  SST_CUDA_TRY(cudaMemsetAsync(P, 0, sizeof(PlanSummary), s));
  uint64_t *keys = A.take<uint64_t>(N), *ktmp = A.take<uint64_t>(N);
  uint32_t *vals = lo ? nullptr : A.take<uint32_t>(N), *vtmp = lo ? nullptr : A.take<uint32_t>(N);
  uint64_t *tcnt = A.take<uint64_t>(ntiles), *tiles = A.take<uint64_t>(ntiles);
  if (!tiles) {
    set_error_message("batched update scratch sizing error");
    return SST_ENOMEM;
  }
  SortDigits sdig;
  if (lo && radix_sort_digits(N, bits, A, &sdig))
    SST_CUDA_TRY(cudaMemsetAsync(sdig.totals, 0, (size_t)sdig.passes * 256 * 4, s));
  else
    sdig = SortDigits{};
  SST_LAUNCH_PDL(k_make_keys_batched, blocks_for(N, kTB * kPackItems), kTB, 0, s, d_pairs, N,
             d_boff, nb, d_ops, g->n, g->width, dbits, lo, !g->keep_loops, sent, keys, vals,
             reinterpret_cast<unsigned long long *>(&P->invalid), sdig);
  uint64_t *sk = keys;
  uint32_t *sv = vals;
  if (lo)
    SST_CUDA_TRY(radix_sort_u64(keys, ktmp, N, bits, A, s, &sk, nullptr,
                                sdig.passes ? &sdig : nullptr, lo));
  else
    SST_CUDA_TRY(radix_sort_kv(keys, ktmp, vals, vtmp, N, bits, A, s, &sk, &sv));
  SST_LAUNCH_PDL_B(8 * N, k_net_count, (unsigned)ntiles, kLoadTB, 0, s, sk, sv, N, lo, sent, tcnt);
  static_assert(offsetof(PlanSummary, n_items) % 8 == 0 &&
                    offsetof(PlanSummary, n_groups) == offsetof(PlanSummary, n_items) + 4,
                "the net insertions and removals share one aligned 64-bit word");
  SST_CUDA_TRY((scan<uint64_t, OpAdd>(tcnt, tiles, ntiles, 0ull, OpAdd{}, true, false,
                                      reinterpret_cast<uint64_t *>(&P->n_items), A, s)));
  SST_LAUNCH_PDL(k_plan_out, 1, 64, 0, s, P, g->d_err, g->h_plan_dev);
  PlanSummary ps;
  sst_status st = read_plan(g, &ps);
  if (st != SST_OK) return st;
  const uint64_t n_ins = ps.n_items, n_del = ps.n_groups;
  if (n_invalid) *n_invalid = ps.invalid;
  if (n_ins + n_del == 0) return SST_OK;
  uint64_t *net = nullptr;
  SST_CUDA_TRY(cudaMallocAsync(&net, (n_ins + n_del) * 8, s));
  SST_LAUNCH_PDL_B(16 * N, k_net_place, (unsigned)ntiles, kLoadTB, 0, s, sk, sv, N, lo, sent,
                   tiles, net, net + n_ins);
  st = run_pipeline(g, nullptr, net + n_ins, n_del, false, nullptr, nullptr);
  if (st == SST_OK) st = run_pipeline(g, nullptr, net, n_ins, true, nullptr, nullptr);
  cudaFreeAsync(net, s);
  return st;
}

// ------------------------------------------------------------ relabelling
// degree_order_map / rewrite_graph of SparseMatrix.hpp:737-766: vertices
// ranked by (degree, id) descending (std::greater on the pair, so among equal
// degrees the larger id comes first); the rewrite inserts every edge with
// both ends relabelled.
namespace {
__global__ void k_degkey(const uint32_t *__restrict__ deg, uint32_t n,
                         uint64_t *__restrict__ keys) {
  pdl_wait();
  uint32_t v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v < n) keys[v] = ((uint64_t)(0xFFFFFFFFu - deg[v]) << 32) | (0xFFFFFFFFu - v);
}
__global__ void k_rank_to_map(const uint64_t *__restrict__ sorted, uint32_t n,
                              uint32_t *__restrict__ map) {
  pdl_wait();
  uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r < n) map[0xFFFFFFFFu - (uint32_t)sorted[r]] = r;
}
__global__ void k_csr_to_pairs(const uint64_t *__restrict__ off,
                               const uint32_t *__restrict__ cols, uint32_t n,
                               uint32_t *__restrict__ pairs);
__global__ void k_relabel_pairs(uint32_t *__restrict__ pairs, uint64_t m,
                                const uint32_t *__restrict__ map) {
  pdl_wait();
  uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= m) return;
  pairs[2 * i] = map[pairs[2 * i]];
  pairs[2 * i + 1] = map[pairs[2 * i + 1]];
}
}  // namespace

sst_status degree_order_map(sst_graph *g, uint32_t *d_map) {
  cudaStream_t s = g->stream;
  uint32_t n = g->n;
  if (n == 0) return SST_OK;
  g->arena.reset();
  SST_CUDA_TRY(g->arena.reserve((uint64_t)n * 16 + radix_sort_scratch_bytes(n) + 8192));
  uint64_t *keys = g->arena.take<uint64_t>(n), *tmp = g->arena.take<uint64_t>(n);
  SST_LAUNCH_PDL(k_degkey, blocks_for(n), kTB, 0, s, g->d_deg, n, keys);
  uint64_t *sorted = keys;
  SST_CUDA_TRY(radix_sort_u64(keys, tmp, n, 64, g->arena, s, &sorted));
  SST_LAUNCH_PDL(k_rank_to_map, blocks_for(n), kTB, 0, s, sorted, n, d_map);
  SST_CUDA_TRY(cudaGetLastError());
  return SST_OK;
}

sst_status rewrite_graph(sst_graph *g, const uint32_t *d_map, sst_graph *out) {
  cudaStream_t s = g->stream;
  uint32_t n = g->n;
  uint64_t m = g->m;
  if (m == 0) return SST_OK;
  uint64_t *off = nullptr;
  uint32_t *cols = nullptr, *pairs = nullptr;
  SST_CUDA_TRY(cudaMallocAsync(&off, ((uint64_t)n + 1) * 8, s));
  SST_CUDA_TRY(cudaMallocAsync(&cols, m * 4, s));
  SST_CUDA_TRY(cudaMallocAsync(&pairs, m * 8, s));
  sst_status st = to_csr(g, off, cols);
  if (st == SST_OK) {
    SST_LAUNCH_PDL(k_csr_to_pairs, warp_blocks(n), kTB, 0, s, off, cols, n, pairs);
    SST_LAUNCH_PDL(k_relabel_pairs, blocks_for(m), kTB, 0, s, pairs, m, d_map);
    SST_CUDA_TRY(cudaStreamSynchronize(s));
    const uint64_t chunk = 1ull << 25;
    for (uint64_t first = 0; first < m && st == SST_OK; first += chunk)
      st = update_batch(out, pairs + 2 * first, std::min(chunk, m - first), true, nullptr);
    cudaStreamSynchronize(out->stream);
  }
  cudaFreeAsync(pairs, s);
  cudaFreeAsync(cols, s);
  cudaFreeAsync(off, s);
  SST_CUDA_TRY(cudaStreamSynchronize(s));
  return st;
}

// Complete the graph's stream and report a staging-rank error left by an
// earlier batch (device-pointer updates do not wait for it).
sst_status sync_checked(sst_graph *g) {
  SST_LAUNCH_PDL(k_err_out, 1, 32, 0, g->stream, g->d_err, &g->h_plan_dev->apply_err);
  SST_CUDA_TRY(cudaStreamSynchronize(g->stream));
  if (g->h_plan->apply_err) {
    set_error_message("internal error: %llu failed device checks (staging rank out of range)",
                      (unsigned long long)g->h_plan->apply_err);
    return SST_EDEVICE;
  }
  return SST_OK;
}

// ------------------------------------------------------------ other paths
namespace {
__global__ void k_csr_to_pairs(const uint64_t *__restrict__ off,
                               const uint32_t *__restrict__ cols, uint32_t n,
                               uint32_t *__restrict__ pairs) {
  pdl_wait();
  uint64_t v = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (v >= n) return;
  for (uint64_t i = off[v] + lane; i < off[v + 1]; i += 32) {
    pairs[2 * i] = (uint32_t)v;
    pairs[2 * i + 1] = cols[i];
  }
}

// membership of each pair; with vals (weighted graphs) also the edge's
// value (0 where absent)
__global__ void k_has(DGraph g, const uint32_t *__restrict__ pairs, uint64_t n,
                      uint8_t *__restrict__ out, uint32_t *__restrict__ vals) {
  pdl_wait();
  uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint32_t u = pairs[2 * i], x = pairs[2 * i + 1];
  uint8_t r = 0;
  uint32_t v = 0;
  if (u < g.n) {
    uint64_t base = g.base[u];
    uint32_t cap = g.cap[u];
    if (cap) {
      uint32_t l = find_leaf(g.slots, base, cap, x);
      uint32_t c = leaf_count(g, base, cap, g.deg[u], l);
      const uint64_t S = base + ((uint64_t)l << kLeafLog);
      uint32_t pos = leaf_lower_bound(g.slots + S, c, x);
      r = pos < c && g.slots[S + pos] == x;
      if (r && vals) v = g.vals[S + pos];
    }
  }
  if (out) out[i] = r;
  if (vals) vals[i] = v;
}

__global__ void k_vertex_leaves(const uint32_t *__restrict__ cap, uint32_t n,
                                uint64_t *__restrict__ nl) {
  pdl_wait();
  uint32_t v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= n) return;
  nl[v] = cap[v] ? nleaves_of(cap[v]) : 0;
}

// warp per vertex: its leaves into the directory
__global__ void k_dir_fill(DGraph g, const uint64_t *__restrict__ vleaf,
                           uint32_t *__restrict__ owner,
                           uint64_t *__restrict__ slot,
                           uint32_t *__restrict__ cnt) {
  pdl_wait();
  uint64_t v = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (v >= g.n) return;
  uint64_t k0 = vleaf[v], k1 = vleaf[v + 1];
  uint64_t base = g.base[v];
  uint32_t cap = g.cap[v], deg = g.deg[v];
  for (uint64_t k = k0 + lane; k < k1; k += 32) {
    uint32_t l = (uint32_t)(k - k0);
    owner[k] = (uint32_t)v;
    slot[k] = base + ((uint64_t)l << kLeafLog);
    cnt[k] = leaf_count(g, base, cap, deg, l);
  }
}

// warp per leaf: copy into CSR position
__global__ void k_dir_copy(const uint32_t *__restrict__ slots,
                           const uint64_t *__restrict__ slot,
                           const uint32_t *__restrict__ cnt,
                           const uint64_t *__restrict__ pre, uint64_t nleaves,
                           uint32_t *__restrict__ cols) {
  pdl_wait();
  uint64_t k = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (k >= nleaves) return;
  if ((uint32_t)lane < cnt[k]) cols[pre[k] + lane] = slots[slot[k] + lane];
}

__global__ void k_widen(const uint32_t *__restrict__ in, uint64_t n,
                        uint64_t *__restrict__ out) {
  pdl_wait();
  uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = in[i];
}

__global__ void k_sample(const uint32_t *__restrict__ slots,
                         const uint32_t *__restrict__ owner,
                         const uint64_t *__restrict__ slot,
                         const uint64_t *__restrict__ pre, uint64_t nleaves,
                         uint64_t m, uint64_t seed, uint64_t first,
                         uint64_t count, uint32_t *__restrict__ pairs) {
  pdl_wait();
  uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  if (m == 0) {
    pairs[2 * i] = pairs[2 * i + 1] = 0;
    return;
  }
  uint64_t rank = __umul64hi(draw(seed, first + i, 0), m);
  uint64_t k = last_le_u64(pre, nleaves, rank);
  pairs[2 * i] = owner[k];
  pairs[2 * i + 1] = slots[slot[k] + (rank - pre[k])];
}

// warp per leaf; 64-bit sum of its elements added to *out
__global__ void k_sum_leaves(const uint32_t *__restrict__ slots,
                             const uint64_t *__restrict__ slot,
                             const uint32_t *__restrict__ cnt, uint64_t nleaves,
                             unsigned long long *__restrict__ out) {
  pdl_wait();
  uint64_t k = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (k >= nleaves) return;
  uint64_t v = (uint32_t)lane < cnt[k] ? slots[slot[k] + lane] : 0;
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) v += __shfl_down_sync(0xffffffffu, v, d);
  if (lane == 0 && v) atomicAdd(out, (unsigned long long)v);
}
}  // namespace

sst_status build_from_csr(sst_graph *g, const uint64_t *d_off,
                          const uint32_t *d_cols) {
  cudaStream_t s = g->stream;
  uint64_t m = 0;
  SST_CUDA_TRY(cudaMemcpyAsync(&m, d_off + g->n, 8, cudaMemcpyDeviceToHost, s));
  SST_CUDA_TRY(cudaStreamSynchronize(s));
  uint64_t n = std::max<uint64_t>(g->n, 1);
  SST_CUDA_TRY(cudaMemsetAsync(g->d_cap, 0, n * 4, s));
  SST_CUDA_TRY(cudaMemsetAsync(g->d_deg, 0, n * 4, s));
  SST_CUDA_TRY(cudaMemsetAsync(g->d_base, 0, n * 8, s));
  g->bump = 0;
  g->m = 0;
  g->version++;
  if (m == 0) return SST_OK;
  uint32_t *pairs = nullptr;
  SST_CUDA_TRY(cudaMallocAsync(&pairs, m * 8, s));
  SST_LAUNCH_PDL(k_csr_to_pairs, warp_blocks(g->n), kTB, 0, s, d_off, d_cols, g->n, pairs);
  sst_status st = update_batch(g, pairs, m, true, nullptr);
  cudaFreeAsync(pairs, s);
  return st;
}

sst_status has_batch(sst_graph *g, const uint32_t *d_pairs, uint64_t n,
                     uint8_t *d_out, uint32_t *d_vals) {
  if (n == 0) return SST_OK;
  SST_LAUNCH_PDL(k_has, blocks_for(n), kTB, 0, g->stream, g->view(), d_pairs, n, d_out,
             d_vals);
  SST_CUDA_TRY(cudaGetLastError());
  return SST_OK;
}

sst_status ensure_leaf_dir(sst_graph *g) {
  LeafDir &D = g->dir;
  if (D.version == g->version && D.vleaf) return SST_OK;
  cudaStream_t s = g->stream;
  uint32_t n = g->n;
  if (!D.vleaf) SST_CUDA_TRY(cudaMalloc(&D.vleaf, ((uint64_t)n + 1) * 8));
  g->arena.reset();
  SST_CUDA_TRY(g->arena.reserve(scan_scratch_bytes((uint64_t)n + 1, 8) + 4096));
  uint64_t *total = g->arena.take<uint64_t>(1);
  if (n) SST_LAUNCH_PDL(k_vertex_leaves, blocks_for(n), kTB, 0, s, g->d_cap, n, D.vleaf);
  SST_CUDA_TRY((scan<uint64_t, OpAdd>(D.vleaf, D.vleaf, n, 0ull, OpAdd{}, true,
                                      false, total, g->arena, s)));
  uint64_t nl = 0;
  SST_CUDA_TRY(cudaMemcpyAsync(&nl, total, 8, cudaMemcpyDeviceToHost, s));
  SST_CUDA_TRY(cudaStreamSynchronize(s));
  SST_CUDA_TRY(cudaMemcpyAsync(D.vleaf + n, &nl, 8, cudaMemcpyHostToDevice, s));
  if (nl > D.cap) {
    uint64_t want = nl + nl / 4 + 1024;
    sst_status st = budget_check(g, (want - D.cap) * 24);
    if (st != SST_OK) return st;
    SST_CUDA_TRY(cudaStreamSynchronize(s));
    cudaFree(D.owner);
    cudaFree(D.slot);
    cudaFree(D.cnt);
    cudaFree(D.pre);
    D.owner = nullptr;
    D.slot = nullptr;
    D.cnt = nullptr;
    D.pre = nullptr;
    D.cap = 0;
    SST_CUDA_TRY(cudaMalloc(&D.owner, want * 4));
    SST_CUDA_TRY(cudaMalloc(&D.slot, want * 8));
    SST_CUDA_TRY(cudaMalloc(&D.cnt, want * 4));
    SST_CUDA_TRY(cudaMalloc(&D.pre, (want + 1) * 8));
    D.cap = want;
  }
  D.nleaves = nl;
  if (n) SST_LAUNCH_PDL(k_dir_fill, warp_blocks(n), kTB, 0, s, g->view(), D.vleaf,
                    D.owner, D.slot, D.cnt);
  g->arena.reset();
  SST_CUDA_TRY(g->arena.reserve(scan_scratch_bytes(nl + 1, 8) + (nl + 1) * 8 + 4096));
  uint64_t *wide = g->arena.take<uint64_t>(nl + 1);
  if (nl) SST_LAUNCH_PDL(k_widen, blocks_for(nl), kTB, 0, s, D.cnt, nl, wide);
  SST_CUDA_TRY((scan<uint64_t, OpAdd>(wide, D.pre, nl, 0ull, OpAdd{}, true,
                                      false, D.pre + nl, g->arena, s)));
  SST_CUDA_TRY(cudaGetLastError());
  D.version = g->version;
  return SST_OK;
}

sst_status to_csr(sst_graph *g, uint64_t *d_off, uint32_t *d_cols,
                  uint32_t *d_vals) {
  sst_status st = ensure_leaf_dir(g);
  if (st != SST_OK) return st;
  cudaStream_t s = g->stream;
  uint32_t n = g->n;
  LeafDir &D = g->dir;
  // row offsets: CSR position of each vertex's first leaf
  g->arena.reset();
  SST_CUDA_TRY(g->arena.reserve(scan_scratch_bytes((uint64_t)n + 1, 8) + ((uint64_t)n + 1) * 8 + 4096));
  uint64_t *wide = g->arena.take<uint64_t>((uint64_t)n + 1);
  if (n) SST_LAUNCH_PDL(k_widen, blocks_for(n), kTB, 0, s, g->d_deg, n, wide);
  SST_CUDA_TRY((scan<uint64_t, OpAdd>(wide, d_off, n, 0ull, OpAdd{}, true, false,
                                      d_off + n, g->arena, s)));
  if (D.nleaves)
    SST_LAUNCH_PDL(k_dir_copy, warp_blocks(D.nleaves), kTB, 0, s, g->d_slots, D.slot,
               D.cnt, D.pre, D.nleaves, d_cols);
  if (D.nleaves && d_vals && g->d_vals)  // values in the same CSR order
    SST_LAUNCH_PDL(k_dir_copy, warp_blocks(D.nleaves), kTB, 0, s, g->d_vals, D.slot,
               D.cnt, D.pre, D.nleaves, d_vals);
  SST_CUDA_TRY(cudaGetLastError());
  return SST_OK;
}

sst_status neighbors(sst_graph *g, uint32_t v, uint32_t *d_out, uint64_t cap,
                     uint64_t *deg) {
  sst_status st = ensure_leaf_dir(g);
  if (st != SST_OK) return st;
  cudaStream_t s = g->stream;
  LeafDir &D = g->dir;
  uint64_t k[2];
  SST_CUDA_TRY(cudaMemcpyAsync(k, D.vleaf + v, 16, cudaMemcpyDeviceToHost, s));
  uint32_t d = 0;
  SST_CUDA_TRY(cudaMemcpyAsync(&d, g->d_deg + v, 4, cudaMemcpyDeviceToHost, s));
  SST_CUDA_TRY(cudaStreamSynchronize(s));
  *deg = d;
  if (k[1] == k[0] || cap == 0) return SST_OK;
  uint64_t p0 = 0;
  SST_CUDA_TRY(cudaMemcpyAsync(&p0, D.pre + k[0], 8, cudaMemcpyDeviceToHost, s));
  SST_CUDA_TRY(cudaStreamSynchronize(s));
  if (cap >= d) {
    // copy leaves with positions rebased to the vertex's first element
    SST_LAUNCH_PDL(k_dir_copy, warp_blocks(k[1] - k[0]), kTB, 0, s, g->d_slots,
               D.slot + k[0], D.cnt + k[0], D.pre + k[0], k[1] - k[0],
               d_out - p0);
  } else {
    uint32_t *tmp = nullptr;
    SST_CUDA_TRY(cudaMallocAsync(&tmp, (uint64_t)d * 4, s));
    SST_LAUNCH_PDL(k_dir_copy, warp_blocks(k[1] - k[0]), kTB, 0, s, g->d_slots,
               D.slot + k[0], D.cnt + k[0], D.pre + k[0], k[1] - k[0], tmp - p0);
    SST_CUDA_TRY(cudaMemcpyAsync(d_out, tmp, cap * 4, cudaMemcpyDeviceToDevice, s));
    cudaFreeAsync(tmp, s);
  }
  SST_CUDA_TRY(cudaGetLastError());
  return SST_OK;
}

sst_status sample_edges(sst_graph *g, uint64_t seed, uint64_t first,
                        uint64_t count, uint32_t *d_pairs) {
  if (count == 0) return SST_OK;
  sst_status st = ensure_leaf_dir(g);
  if (st != SST_OK) return st;
  LeafDir &D = g->dir;
  SST_LAUNCH_PDL(k_sample, blocks_for(count), kTB, 0, g->stream, g->d_slots, D.owner,
             D.slot, D.pre, D.nleaves, g->m, seed, first, count, d_pairs);
  SST_CUDA_TRY(cudaGetLastError());
  return SST_OK;
}

sst_status touch_all_sum(sst_graph *g, uint64_t *out) {
  sst_status st = ensure_leaf_dir(g);
  if (st != SST_OK) return st;
  cudaStream_t s = g->stream;
  LeafDir &D = g->dir;
  g->arena.reset();
  SST_CUDA_TRY(g->arena.reserve(4096));
  unsigned long long *acc = g->arena.take<unsigned long long>(1);
  SST_CUDA_TRY(cudaMemsetAsync(acc, 0, 8, s));
  if (D.nleaves)
    SST_LAUNCH_PDL(k_sum_leaves, warp_blocks(D.nleaves), kTB, 0, s, g->d_slots,
               D.slot, D.cnt, D.nleaves, acc);
  SST_CUDA_TRY(cudaMemcpyAsync(out, acc, 8, cudaMemcpyDeviceToHost, s));
  SST_CUDA_TRY(cudaStreamSynchronize(s));
  return SST_OK;
}

}  // namespace sst
