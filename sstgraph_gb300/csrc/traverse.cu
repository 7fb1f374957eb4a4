// Traversal kernels over the device PMA (the EdgeMap/VertexMap algorithms the
// reference drivers call at internal/test.hpp:476-618; the algorithm
// library itself, EdgeMapVertexMap, is absent from the reference tree).
//
// Work decomposition, rebuilt when the graph version changes:
//  - a vertex whose segment is one leaf (cap <= 32) is handled by one thread
//    that walks its packed leaf;
//  - a vertex with a multi-leaf segment is cut into chunks of kChunkLeaves
//    leaves; one warp walks a chunk leaf by leaf (lane = slot, one 128-byte
//    line per leaf, only the occupied prefix is read); chunks of one vertex
//    are combined in chunk order, so sums are deterministic.
#include <algorithm>
#include <cooperative_groups.h>
#include <new>
#include <vector>

#include "bfslevels.cuh"
#include "ccshared.cuh"
#include "prfixed.cuh"
#include "tcshared.cuh"
#include "traverse.cuh"
#include "travwords.h"

namespace sst {

namespace {
constexpr int kTB = 256;
constexpr uint32_t kChunkLeaves = 32;
// leaves per work item of the push-style kernels (frontier expansion):
// smaller than kChunkLeaves so a hub's chunks spread over more warps
constexpr uint32_t kPushLeaves = 8;

inline unsigned blocks_for(uint64_t n, int per = kTB) {
  uint64_t b = (n + per - 1) / per;
  return (unsigned)(b == 0 ? 1 : b);
}
inline unsigned warp_blocks(uint64_t nwarps) { return blocks_for(nwarps * 32); }

__device__ __forceinline__ double warp_sum_d(double v) {
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) v += __shfl_down_sync(0xffffffffu, v, d);
  return v;
}
}  // namespace

template <typename T> struct DevBuf {
  T *p = nullptr;
  uint64_t cap = 0;
  cudaError_t ensure(uint64_t n) {
    if (n <= cap) return cudaSuccess;
    return exact(n + n / 8 + 64);
  }
  // without room to grow: for sizes that only the number of vertices sets
  cudaError_t exact(uint64_t n) {
    if (n <= cap) return cudaSuccess;
    release();
    cudaError_t e = cudaMalloc(&p, n * sizeof(T));
    if (e == cudaSuccess) cap = n;
    return e;
  }
  void release() {
    if (p) cudaFree(p);
    p = nullptr;
    cap = 0;
  }
};

struct TravState : TravWords {
  uint64_t version = ~0ull;
  // tuning (sst_autotune): leaves per work-list chunk (<= 32), lanes per
  // one-leaf vertex in PageRank, and the BFS switch to pull once
  // (frontier + its edges) * bfs_alpha > m
  uint32_t chunk_leaves = 32, pr_lanes = 8, bfs_alpha = 20;
  uint32_t pr_hot = 0;        // contributions staged in shared memory
  uint32_t pr_hot_used = ~0u; // pr_hot of the captured graph
  uint32_t lists_cl = 0;      // chunk size the lists were built with
  uint64_t lists_stamp = 0;   // bumped on every rebuild of the lists
  // chunk list of multi-leaf vertices
  uint64_t nchunks = 0, nmulti = 0, nbig = 0, nsmall = 0;
  uint64_t inv_version = ~0ull;
  DevBuf<uint32_t> cv;      // per chunk: vertex
  DevBuf<unsigned long long> cdesc, sdesc;  // packed chunk / one-leaf items
  DevBuf<uint2> multi;      // vertices with more than one chunk: vertex, first chunk
  DevBuf<uint32_t> big;     // vertices with a multi-leaf segment
  DevBuf<uint32_t> small;   // vertices with a one-leaf segment (deg >= 1)
  DevBuf<uint32_t> lsum;    // per block of the list build: its list entries
  // pagerank
  DevBuf<double> inv_deg, ca, cb, partial;
  // bfs
  DevBuf<uint32_t> qa, qb, fbits, icnt, ioff, iv, il0;
  DevBuf<unsigned long long> qitems;
  DevBuf<int32_t> depth_tmp;
  // bc
  DevBuf<double> sigma, ratio;
  DevBuf<uint2> levels, hub;
  DevBuf<uint32_t> hub_done;
  // cc
  DevBuf<uint32_t> par;
  // tc
  DevBuf<uint64_t> toff, tlpre, tlcnt, titems;
  DevBuf<uint32_t> tadj, tmask;
  // multi-source bfs: per-vertex source masks (visited, frontier, next)
  DevBuf<unsigned long long> mvis, mfr, mfr2, mnx, msrc;
  DevBuf<int32_t> mdepth;
  // multi-source bc: per (source, vertex) values and per-source level tables
  DevBuf<double> msig, mrat, mpart;
  DevBuf<uint32_t> mlist, micnt, mioff, miv, mil0, mtab;
  // PageRank iterations captured as one CUDA graph, replayed while the
  // graph version and the call's arguments stay the same
  cudaGraphExec_t pr_exec = nullptr;
  uint64_t pr_version = ~0ull;  // lists_stamp the graph was captured with
  uint32_t pr_lanes_used = 0;
  uint32_t pr_iters = 0;
  double pr_damping = 0.0;
  const void *pr_key[6] = {};  // output, stream and the buffers it reads
  int64_t pr_kernels = 0;      // kernels in the captured graph
};

// frees every buffer and the captured PageRank graph; the tuning stays, and
// the work lists are rebuilt by the next traversal
static void trav_buffers_release(TravState *t) {
  t->cv.release();
  t->cdesc.release();
  t->sdesc.release();
  t->multi.release();
  t->big.release();
  t->small.release();
  t->lsum.release();
  t->inv_deg.release();
  t->ca.release();
  t->cb.release();
  t->partial.release();
  t->qa.release();
  t->qb.release();
  t->fbits.release();
  t->icnt.release();
  t->qitems.release();
  t->ioff.release();
  t->iv.release();
  t->il0.release();
  t->depth_tmp.release();
  t->sigma.release();
  t->ratio.release();
  t->levels.release();
  t->hub.release();
  t->hub_done.release();
  t->par.release();
  t->toff.release();
  t->tlpre.release();
  t->tlcnt.release();
  t->titems.release();
  t->tadj.release();
  t->tmask.release();
  t->mvis.release();
  t->mfr.release();
  t->mfr2.release();
  t->mnx.release();
  t->msrc.release();
  t->mdepth.release();
  t->msig.release();
  t->mrat.release();
  t->mpart.release();
  t->mlist.release();
  t->micnt.release();
  t->mioff.release();
  t->miv.release();
  t->mil0.release();
  t->mtab.release();
  if (t->pr_exec) cudaGraphExecDestroy(t->pr_exec);
  t->pr_exec = nullptr;
  t->version = ~0ull;
  t->inv_version = ~0ull;
  t->lists_stamp++;
}

void trav_trim(sst_graph *g) {
  if (g->trav) trav_buffers_release(g->trav);
}

// the CUDA side of TravWords
struct TravWordsRt {
  cudaStream_t s;
  bool pinned(void **p, size_t bytes) { return cudaMallocHost(p, bytes) == cudaSuccess; }
  bool device(void **p, size_t bytes) { return cudaMalloc(p, bytes) == cudaSuccess; }
  bool zero(void *p, size_t bytes) { return cudaMemsetAsync(p, 0, bytes, s) == cudaSuccess; }
  void free_pinned(void *p) { cudaFreeHost(p); }
  void free_device(void *p) { cudaFree(p); }
};

void trav_release(sst_graph *g) {
  TravState *t = g->trav;
  if (!t) return;
  trav_buffers_release(t);
  trav_words_free(t, TravWordsRt{g->stream});
  delete t;
  g->trav = nullptr;
}

uint64_t trav_device_bytes(const sst_graph *g) {
  const TravState *t = g->trav;
  if (!t) return 0;
  uint64_t b = 0;
  auto add = [&](uint64_t cap, size_t elem) { b += cap * elem; };
  add(t->cv.cap, 4); add(t->cdesc.cap, 8);
  add(t->sdesc.cap, 8); add(t->multi.cap, 8); add(t->big.cap, 4); add(t->small.cap, 4);
  add(t->lsum.cap, 4); add(t->inv_deg.cap, 8); add(t->ca.cap, 8);
  add(t->cb.cap, 8); add(t->partial.cap, 8); add(t->qa.cap, 4); add(t->qb.cap, 4);
  add(t->fbits.cap, 4); add(t->qitems.cap, 8); add(t->icnt.cap, 4); add(t->ioff.cap, 4); add(t->iv.cap, 4);
  add(t->il0.cap, 4); add(t->depth_tmp.cap, 4);
  add(t->sigma.cap, 8); add(t->ratio.cap, 8); add(t->levels.cap, 8);
  add(t->hub.cap, 8); add(t->hub_done.cap, 4); add(t->par.cap, 4); add(t->toff.cap, 8); add(t->tlpre.cap, 8);
  add(t->tlcnt.cap, 8); add(t->titems.cap, 8); add(t->tadj.cap, 4); add(t->tmask.cap, 4);
  add(t->mvis.cap, 8); add(t->mfr.cap, 8);
  add(t->mfr2.cap, 8); add(t->mnx.cap, 8); add(t->msrc.cap, 8); add(t->mdepth.cap, 4);
  add(t->msig.cap, 8); add(t->mrat.cap, 8); add(t->mpart.cap, 8); add(t->mlist.cap, 4);
  add(t->micnt.cap, 4); add(t->mioff.cap, 4); add(t->miv.cap, 4); add(t->mil0.cap, 4);
  add(t->mtab.cap, 4);
  return b;
}

namespace {

// ------------------------------------------------------------- work lists
// The four lists (one-leaf vertices, multi-leaf vertices, those of several
// chunks, all chunks) in three launches: entries a block of vertices, their
// prefix over the blocks, and the entries.  A thread takes kListPer
// consecutive vertices.  Scanning a flag a vertex and list took eleven launches
// and 24 bytes a vertex of scratch, and two readbacks.
constexpr int kListPer = 8;
constexpr uint32_t kListBlock = kScanThreads * kListPer;

__device__ __forceinline__ uint32_t chunks_of(uint32_t cap, uint32_t cl) {
  return cap > kLeaf ? ((cap >> kLeafLog) + cl - 1) / cl : 0u;
}

// list entries of a thread's vertices: one-leaf, multi-leaf and multi-chunk
// vertices (21 bits each, a block has 2048), and chunks
struct ListCount {
  unsigned long long rows = 0;
  uint32_t chunks = 0;
  __device__ __forceinline__ void add(uint32_t cap, uint32_t cl) {
    const uint32_t k = chunks_of(cap, cl);
    rows += (unsigned long long)(cap > 0 && cap <= kLeaf) |
            (unsigned long long)(k > 0) << 21 | (unsigned long long)(k > 1) << 42;
    chunks += k;
  }
};
__device__ __forceinline__ void load_caps(const uint32_t *cap, uint64_t v0, uint32_t n,
                                          uint32_t (&c)[kListPer]) {
  if (v0 + kListPer <= n) {  // the table is a whole allocation: 16-byte aligned
    const uint4 a = *reinterpret_cast<const uint4 *>(cap + v0);
    const uint4 b = *reinterpret_cast<const uint4 *>(cap + v0 + 4);
    c[0] = a.x, c[1] = a.y, c[2] = a.z, c[3] = a.w;
    c[4] = b.x, c[5] = b.y, c[6] = b.z, c[7] = b.w;
  } else {
#pragma unroll
    for (int k = 0; k < kListPer; k++) c[k] = v0 + k < n ? cap[v0 + k] : 0u;
  }
}

__global__ void __launch_bounds__(kScanThreads)
k_list_count(const uint32_t *__restrict__ cap, uint32_t n, uint32_t cl,
             uint4 *__restrict__ sums) {
  pdl_wait();
  const uint64_t v0 = ((uint64_t)blockIdx.x * kScanThreads + threadIdx.x) * kListPer;
  uint32_t c[kListPer];
  load_caps(cap, v0, n, c);
  ListCount e;
#pragma unroll
  for (int k = 0; k < kListPer; k++) e.add(c[k], cl);
  unsigned long long rows;
  uint32_t chunks;
  block_exclusive(e.rows, 0ull, OpAdd{}, &rows);
  block_exclusive(e.chunks, 0u, OpAdd{}, &chunks);
  if (threadIdx.x == 0)
    sums[blockIdx.x] = make_uint4((uint32_t)rows & 0x1FFFFF, (uint32_t)(rows >> 21) & 0x1FFFFF,
                                  (uint32_t)(rows >> 42), chunks);
}

// one block: exclusive prefixes in place, the totals to the host's pinned word
__global__ void __launch_bounds__(kScanThreads)
k_list_prefix(uint4 *__restrict__ sums, uint32_t nb, uint4 *__restrict__ totals) {
  pdl_wait();
  uint4 run = make_uint4(0, 0, 0, 0);
  for (uint32_t i0 = 0; i0 < nb; i0 += kScanThreads) {
    const uint32_t i = i0 + threadIdx.x;
    const uint4 x = i < nb ? sums[i] : make_uint4(0, 0, 0, 0);
    // two counters a word: each total is below 2^32
    unsigned long long t0, t1;
    const unsigned long long p0 =
        block_exclusive((unsigned long long)x.y << 32 | x.x, 0ull, OpAdd{}, &t0);
    const unsigned long long p1 =
        block_exclusive((unsigned long long)x.w << 32 | x.z, 0ull, OpAdd{}, &t1);
    if (i < nb)
      sums[i] = make_uint4(run.x + (uint32_t)p0, run.y + (uint32_t)(p0 >> 32),
                           run.z + (uint32_t)p1, run.w + (uint32_t)(p1 >> 32));
    run.x += (uint32_t)t0;
    run.y += (uint32_t)(t0 >> 32);
    run.z += (uint32_t)t1;
    run.w += (uint32_t)(t1 >> 32);
  }
  if (threadIdx.x == 0) *totals = run;
}

__global__ void __launch_bounds__(kScanThreads)
k_list_fill(DGraph g, uint32_t cl, const uint4 *__restrict__ sums, uint32_t *__restrict__ small,
            unsigned long long *__restrict__ sdesc, uint32_t *__restrict__ big,
            uint2 *__restrict__ multi, uint32_t *__restrict__ cv,
            unsigned long long *__restrict__ cdesc) {
  pdl_wait();
  const uint64_t v0 = ((uint64_t)blockIdx.x * kScanThreads + threadIdx.x) * kListPer;
  uint32_t c[kListPer];
  load_caps(g.cap, v0, g.n, c);
  ListCount e;
#pragma unroll
  for (int k = 0; k < kListPer; k++) e.add(c[k], cl);
  unsigned long long rows;
  uint32_t chunks;
  const unsigned long long r = block_exclusive(e.rows, 0ull, OpAdd{}, &rows);
  const uint32_t h = block_exclusive(e.chunks, 0u, OpAdd{}, &chunks);
  const uint4 at = sums[blockIdx.x];
  uint32_t is = at.x + ((uint32_t)r & 0x1FFFFF), ib = at.y + ((uint32_t)(r >> 21) & 0x1FFFFF);
  uint32_t im = at.z + (uint32_t)(r >> 42), ic = at.w + h;
#pragma unroll
  for (int k = 0; k < kListPer; k++) {
    if (!c[k]) continue;
    const uint32_t v = (uint32_t)(v0 + k);
    const uint64_t base = g.base[v];
    if (c[k] <= kLeaf) {
      small[is] = v;
      sdesc[is++] = ((unsigned long long)base << 6) | g.deg[v];
      continue;
    }
    big[ib++] = v;
    const uint32_t nl = c[k] >> kLeafLog, nc = chunks_of(c[k], cl);
    if (nc > 1) multi[im++] = make_uint2(v, ic);
    const unsigned long long single = nc == 1 ? 128ull : 0ull;
    for (uint32_t j = 0; j < nc; j++, ic++) {
      cv[ic] = v;
      cdesc[ic] = (((base >> kLeafLog) + (uint64_t)j * cl) << 8) | single |
                  (unsigned long long)min(cl, nl - j * cl);
    }
  }
}

// ------------------------------------------------------------- pagerank
// The fixed-point arithmetic (units of 2^-63, exact integer sums) is in
// prfixed.cuh, shared with the byte-width snapshot's PageRank.

// a vertex with an empty row is in no work list, so no iteration writes its
// contribution: zero it in both buffers (a directed graph's rows may still
// name it).  With fresh, the degrees' reciprocals are computed here too.
__global__ void k_pr_start(const uint32_t *__restrict__ deg, uint32_t n,
                           unsigned long long r0, bool fresh,
                           unsigned long long *__restrict__ rdeg,
                           unsigned long long *__restrict__ contrib,
                           unsigned long long *__restrict__ contrib2,
                           double *__restrict__ rank, double base) {
  pdl_wait();
  uint32_t v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= n) return;
  const uint32_t d = deg[v];
  if (d) {
    const unsigned long long rd = fresh ? pr_rdeg_of(d) : rdeg[v];
    if (fresh) rdeg[v] = rd;
    contrib[v] = contrib_of(r0, d, rd);
  } else {  // (its reciprocal is not read either)
    contrib[v] = contrib2[v] = 0ull;
    rank[v] = base;  // no in-edges: constant term only
  }
}


// One-leaf segments (cap <= 32): a group of G lanes per vertex (G = 8: one
// 32-byte sector of the leaf per lane step), four vertices per group in
// flight.  sdesc[i] = (segment base << 6) | degree.
constexpr int kSmallPer = 4;

template <int G>
__device__ __forceinline__ void pr_small(uint64_t block, const DGraph &g,
                                         const unsigned long long *__restrict__ sdesc,
                                         const uint32_t *__restrict__ small, uint64_t nsmall,
                                         const unsigned long long *__restrict__ cin,
                                         unsigned long long *__restrict__ cout,
                                         double *__restrict__ rank,
                                         const unsigned long long *__restrict__ rdeg,
                                         const PrConst &k, bool last) {
  static_assert(G >= kSmallPer && G <= 32 && (G & (G - 1)) == 0, "lanes per vertex");
  constexpr int Q = 32 / G;  // slots per lane
  uint64_t grp = (block * blockDim.x + threadIdx.x) / G;
  const uint32_t sub = threadIdx.x & (G - 1);
  const unsigned long long pol = l2_evict_first();
  const uint64_t i0 = grp * kSmallPer;
  uint32_t x[kSmallPer][Q];
  uint32_t dg[kSmallPer];
#pragma unroll
  for (int u = 0; u < kSmallPer; u++) {
    uint64_t i = i0 + u;
    unsigned long long dsc = i < nsmall ? sdesc[i] : 0ull;
    dg[u] = (uint32_t)(dsc & 63);
    const uint32_t *p = g.slots + (dsc >> 6);
#pragma unroll
    for (int q = 0; q < Q; q++) {
      uint32_t j = sub + G * q;
      x[u][q] = j < dg[u] ? ld_stream(p + j, pol) : kEmpty;
    }
  }
  unsigned long long acc[kSmallPer];
#pragma unroll
  for (int u = 0; u < kSmallPer; u++) {
    acc[u] = 0;
#pragma unroll
    for (int q = 0; q < Q; q++)
      if (x[u][q] != kEmpty) acc[u] += ld_keep(cin + x[u][q]);
  }
  unsigned long long mine = 0;
  uint32_t mydeg = 0;
#pragma unroll
  for (int u = 0; u < kSmallPer; u++) {
    unsigned long long a = acc[u];
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    if (sub == (uint32_t)u) {
      mine = a;
      mydeg = dg[u];
    }
  }
  if (sub < (uint32_t)kSmallPer && i0 + sub < nsmall)
    pr_finish(small[i0 + sub], mine, k, mydeg, rdeg, cout, rank, last);
}

// warp per chunk of <= 32 leaves of a multi-leaf segment (lane = slot);
// the chunk's leaf counts come in with one coalesced load, and eight leaves'
// ids, then their eight gathers, are in flight per step.
// cdesc[c] = (first leaf << 8) | (single chunk << 7) | leaves in the chunk.
__device__ __forceinline__ void pr_chunk(uint64_t c, const DGraph &g,
                                         const unsigned long long *__restrict__ cdesc,
                                         const uint32_t *__restrict__ cv, uint64_t nchunks,
                                         const unsigned long long *__restrict__ cin,
                                         unsigned long long *__restrict__ cout,
                                         double *__restrict__ rank,
                                         const unsigned long long *__restrict__ rdeg,
                                         unsigned long long *__restrict__ partial,
                                         const PrConst &k, bool last) {
  const int lane = threadIdx.x & 31;
  if (c >= nchunks) return;
  const unsigned long long pol = l2_evict_first();
  unsigned long long dsc = cdesc[c];
  const uint64_t leaf0 = dsc >> 8;
  const uint32_t l1 = (uint32_t)(dsc & 63);
  const bool single = (dsc >> 7) & 1;
  const uint32_t mycnt = (uint32_t)lane < l1 ? g.lcnt[leaf0 + lane] : 0u;
  const uint32_t *sl = g.slots + (leaf0 << kLeafLog) + lane;
  unsigned long long acc = 0;
  for (uint32_t l = 0; l < l1; l += 8) {
    uint32_t x[8];
#pragma unroll
    for (int q = 0; q < 8; q++) {
      uint32_t cq = __shfl_sync(0xffffffffu, mycnt, (l + q) & 31);
      if (l + q >= l1) cq = 0;
      x[q] = (uint32_t)lane < cq ? ld_stream(sl + ((uint64_t)(l + q) << kLeafLog), pol)
                                 : kEmpty;
    }
#pragma unroll
    for (int q = 0; q < 8; q++)
      if (x[q] != kEmpty) acc += ld_keep(cin + x[q]);
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, d);
  if (lane == 0) {
    if (single) {
      uint32_t v = cv[c];
      pr_finish(v, acc, k, g.deg[v], rdeg, cout, rank, last);
    } else {
      partial[c] = acc;  // one of several: k_pr_fix
    }
  }
}

// An iteration's gathers: blocks [0, cblocks) take the chunks, a warp each, the
// rest the one-leaf vertices, so the two parts' last and first blocks overlap.
// The chunks of one vertex meet in a launch of their own (k_pr_fix): meeting
// here takes a fence a chunk, and a fence empties the SM's L1, which the
// gathers live on (RMAT scale 22: 5.57 against 4.97 ms for 20 iterations).  32
// registers a thread keep the SM's 64 warps, which the gathers need.
template <int G>
__global__ void __launch_bounds__(kTB, G == 4 ? 5 : 8)
k_pr_iter(DGraph g, const unsigned long long *__restrict__ cdesc, const uint32_t *__restrict__ cv,
          uint64_t nchunks, unsigned cblocks, const unsigned long long *__restrict__ sdesc,
          const uint32_t *__restrict__ small, uint64_t nsmall,
          const unsigned long long *__restrict__ cin, unsigned long long *__restrict__ cout,
          double *__restrict__ rank, const unsigned long long *__restrict__ rdeg,
          unsigned long long *__restrict__ partial, PrConst k, bool last) {
  pdl_wait();
  if (blockIdx.x < cblocks)
    pr_chunk(((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5, g, cdesc, cv, nchunks, cin,
             cout, rank, rdeg, partial, k, last);
  else
    pr_small<G>(blockIdx.x - cblocks, g, sdesc, small, nsmall, cin, cout, rank, rdeg, k, last);
}

// ---- PageRank with the contributions of ids below `hot` staged in shared
// memory once per block: on a degree-ordered graph (highest degree first,
// sst_degree_order_map) those are the vertices most edges point to, so
// their gathers leave L2 alone.  Blocks are persistent and stride over the
// work; the loops stay warp-uniform for the shuffles.
__device__ __forceinline__ void stage_hot(unsigned long long *sh,
                                          const unsigned long long *cin,
                                          uint32_t hot) {
  for (uint32_t i = threadIdx.x; i < hot; i += blockDim.x) sh[i] = cin[i];
  __syncthreads();
}
__device__ __forceinline__ unsigned long long gather(const unsigned long long *sh,
                                                     const unsigned long long *cin,
                                                     uint32_t x, uint32_t hot) {
  return x < hot ? sh[x] : ld_keep(cin + x);
}

constexpr int kHotThreads = 512;  // 4 blocks of 16 warps per SM
// a cache above kHotBig entries leaves room for one block per SM: that block
// takes 1024 threads
constexpr uint32_t kHotBig = 8192;

// launch bounds: 512-thread blocks at least two to an SM (64 registers a
// thread), 1024-thread blocks (large caches) one to an SM
template <int G, int T = kHotThreads>
__global__ void __launch_bounds__(T, T == 1024 ? 1 : 2) k_pr_small_hot(DGraph g, const unsigned long long *__restrict__ sdesc,
                               const uint32_t *__restrict__ small, uint64_t nsmall,
                               const unsigned long long *__restrict__ cin,
                               unsigned long long *__restrict__ cout,
                               double *__restrict__ rank,
                               const unsigned long long *__restrict__ rdeg,
                               PrConst k, bool last, uint32_t hot) {
  extern __shared__ unsigned long long sh[];
  constexpr int Q = 32 / G;
  stage_hot(sh, cin, hot);
  const unsigned long long pol = l2_evict_first();
  const uint32_t sub = threadIdx.x & (G - 1);
  const uint64_t per_warp = (32 / G) * kSmallPer;  // vertices per warp round
  const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  const uint64_t rounds = (nsmall + per_warp - 1) / per_warp;
  for (uint64_t w = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
       w < rounds; w += nwarps) {
    const uint64_t i0 = (w * (32 / G) + ((threadIdx.x & 31) / G)) * kSmallPer;
    uint32_t x[kSmallPer][Q];
    uint32_t dg[kSmallPer];
#pragma unroll
    for (int u = 0; u < kSmallPer; u++) {
      uint64_t i = i0 + u;
      unsigned long long dsc = i < nsmall ? sdesc[i] : 0ull;
      dg[u] = (uint32_t)(dsc & 63);
      const uint32_t *p = g.slots + (dsc >> 6);
#pragma unroll
      for (int q = 0; q < Q; q++) {
        uint32_t j = sub + G * q;
        x[u][q] = j < dg[u] ? ld_stream(p + j, pol) : kEmpty;
      }
    }
    unsigned long long mine = 0;
    uint32_t mydeg = 0;
#pragma unroll
    for (int u = 0; u < kSmallPer; u++) {
      unsigned long long a = 0;
#pragma unroll
      for (int q = 0; q < Q; q++)
        if (x[u][q] != kEmpty) a += gather(sh, cin, x[u][q], hot);
#pragma unroll
      for (int o = G / 2; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
      if (sub == (uint32_t)u) {
        mine = a;
        mydeg = dg[u];
      }
    }
    if (sub < (uint32_t)kSmallPer && i0 + sub < nsmall)
      pr_finish(small[i0 + sub], mine, k, mydeg, rdeg, cout, rank, last);
  }
}

template <int T = kHotThreads>
__global__ void __launch_bounds__(T, T == 1024 ? 1 : 2) k_pr_chunks_hot(DGraph g, const unsigned long long *__restrict__ cdesc,
                                const uint32_t *__restrict__ cv, uint64_t nchunks,
                                const unsigned long long *__restrict__ cin,
                                unsigned long long *__restrict__ cout,
                                double *__restrict__ rank,
                                const unsigned long long *__restrict__ rdeg,
                                unsigned long long *__restrict__ partial, PrConst k,
                                bool last, uint32_t hot) {
  extern __shared__ unsigned long long sh[];
  stage_hot(sh, cin, hot);
  const int lane = threadIdx.x & 31;
  const unsigned long long pol = l2_evict_first();
  const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  for (uint64_t c = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
       c < nchunks; c += nwarps) {
    unsigned long long dsc = cdesc[c];
    const uint64_t leaf0 = dsc >> 8;
    const uint32_t l1 = (uint32_t)(dsc & 63);
    const bool single = (dsc >> 7) & 1;
    const uint32_t mycnt = (uint32_t)lane < l1 ? g.lcnt[leaf0 + lane] : 0u;
    const uint32_t *sl = g.slots + (leaf0 << kLeafLog) + lane;
    unsigned long long acc = 0;
    for (uint32_t l = 0; l < l1; l += 8) {
      uint32_t x[8];
#pragma unroll
      for (int q = 0; q < 8; q++) {
        uint32_t cq = __shfl_sync(0xffffffffu, mycnt, (l + q) & 31);
        if (l + q >= l1) cq = 0;
        x[q] = (uint32_t)lane < cq ? ld_stream(sl + ((uint64_t)(l + q) << kLeafLog), pol)
                                   : kEmpty;
      }
#pragma unroll
      for (int q = 0; q < 8; q++)
        if (x[q] != kEmpty) acc += gather(sh, cin, x[q], hot);
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, d);
    if (lane == 0) {
      if (single) {
        uint32_t v = cv[c];
        pr_finish(v, acc, k, g.deg[v], rdeg, cout, rank, last);
      } else {
        partial[c] = acc;
      }
    }
  }
}

// the vertices of several chunks, a warp each (a thread that walked a hub's
// hundreds of partial sums alone took 7 us)
__global__ void k_pr_fix(DGraph g, const uint2 *__restrict__ multi, uint64_t nmulti,
                         uint32_t cl, const unsigned long long *__restrict__ partial,
                         unsigned long long *__restrict__ cout, double *__restrict__ rank,
                         const unsigned long long *__restrict__ rdeg, PrConst k, bool last) {
  pdl_wait();
  const uint64_t i = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (i >= nmulti) return;
  const uint2 e = multi[i];
  const uint32_t nc = chunks_of(g.cap[e.x], cl);
  unsigned long long s = 0;
  for (uint32_t c = lane; c < nc; c += 32) s += partial[e.y + c];
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
  if (lane == 0) pr_finish(e.x, s, k, g.deg[e.x], rdeg, cout, rank, last);
}

__global__ void k_fill_d(double *__restrict__ p, uint32_t n, double x) {
  uint32_t v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v < n) p[v] = x;
}

// ------------------------------------------------------- frontier queues
// Append of `mine` to the next queue, for kernels in which every thread of the
// block calls it once: one atomic per counter per block (the three queue
// counters are single addresses, so per-warp atomics from a whole grid
// serialise on them).  Counters: [0] queue length, [1] degree sum, [2] work
// items of the queue.
__device__ __forceinline__ void enqueue_block(bool mine, uint32_t w, uint32_t wdeg,
                                              uint32_t witems, uint32_t *q,
                                              unsigned long long *qlen_deg) {
  __shared__ uint32_t s_cnt[kTB / 32];
  __shared__ unsigned long long s_base, s_deg, s_items;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t m = __ballot_sync(0xffffffffu, mine);
  const uint32_t dsum = __reduce_add_sync(0xffffffffu, mine ? wdeg : 0u);
  const uint32_t isum = __reduce_add_sync(0xffffffffu, mine ? witems : 0u);
  if (threadIdx.x == 0) {
    s_deg = 0;
    s_items = 0;
  }
  if (lane == 0) s_cnt[warp] = __popc(m);
  __syncthreads();
  if (lane == 0 && m) {
    atomicAdd(&s_deg, (unsigned long long)dsum);
    atomicAdd(&s_items, (unsigned long long)isum);
  }
  if (threadIdx.x == 0) {
    uint32_t tot = 0;
#pragma unroll
    for (int k = 0; k < kTB / 32; k++) {
      uint32_t c = s_cnt[k];
      s_cnt[k] = tot;
      tot += c;
    }
    s_base = tot ? atomicAdd(&qlen_deg[0], (unsigned long long)tot) : 0ull;
  }
  __syncthreads();
  if (threadIdx.x == 0 && (s_deg || s_items)) {
    atomicAdd(&qlen_deg[1], s_deg);
    atomicAdd(&qlen_deg[2], s_items);
  }
  if (mine) q[s_base + s_cnt[warp] + __popc(m & ((1u << lane) - 1u))] = w;
}

// push work items of one vertex: 1 for a one-leaf segment, else one per
// chunk of kPushLeaves leaves
__device__ __forceinline__ uint32_t items_of(uint32_t cap) {
  return cap > kLeaf ? ((cap >> kLeafLog) + kPushLeaves - 1) / kPushLeaves : 1u;
}

__global__ void k_front_items(const uint32_t *__restrict__ q, uint32_t qn,
                              const uint32_t *__restrict__ cap,
                              uint32_t *__restrict__ cnt) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < qn) cnt[i] = items_of(cap[q[i]]);
}

__global__ void k_front_expand(const uint32_t *__restrict__ q, uint32_t qn,
                               const uint32_t *__restrict__ cap,
                               const uint32_t *__restrict__ off,
                               uint32_t *__restrict__ iv,
                               uint32_t *__restrict__ il0) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= qn) return;
  uint32_t v = q[i], k = items_of(cap[v]), o = off[i];
  for (uint32_t j = 0; j < k; j++) {
    iv[o + j] = v;
    il0[o + j] = j * kPushLeaves;
  }
}

// ------------------------------------------------------------- cc
// Afforest, with the helpers in ccshared.cuh, but the sampled links are hooks
// without a loop.  Linking every vertex to its first two neighbours by find
// and compare-and-swap (the form before) had 2e6 threads chase and extend
// chains of fresh roots: 385 us a neighbour on a uniform graph of 2e6 vertices
// and 14e6 stored edges, where a whole call takes 172 us now.  The rounds
// are bound by scattered 32-byte sectors: a row's first ids (read once, here),
// and two parents a vertex and round.
// The passes go over all vertices, or, where fewer than half of them have a row,
// over the work lists' entries (a vertex without a row is its own root from the
// start; where edges are stored one way it may be linked from another's row, so the
// compressions before the largest tree is sampled and at the end take all vertices).
// Of 2^24 vertices 2,000 with a row: 474 us over all, 158 over those (the sampled links
// by find before took 309); of 2^22 one in 16 with a row 167 and 133, one in 4 200 and
// 171, one in 2 247 and 238.
struct CcVerts {
  const uint32_t *small, *big;  // null: every vertex
  uint32_t nsmall, count;
  __device__ __forceinline__ uint32_t operator[](uint32_t i) const {
    return !small ? i : i < nsmall ? small[i] : big[i - nsmall];
  }
};
__global__ void k_cc_compress_some(CcVerts vs, uint32_t *par,
                                   const unsigned long long *__restrict__ hooks) {
  pdl_wait();
  if (hooks && *hooks == 0) return;
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < vs.count) cc_compress(par, vs[i]);
}

// The start: every vertex below its smallest neighbour (rows ascend), if that
// is smaller.  A parent is smaller than its child, so the links are a forest.
// nb1 and nb2 keep what is left of its first two neighbours' edges for the rounds
// (kEmpty: none): the second, and the smallest if it is larger than u.
__global__ void k_cc_hook_first(DGraph g, CcVerts vs, uint32_t *__restrict__ par,
                                uint32_t *__restrict__ nb1, uint32_t *__restrict__ nb2) {
  pdl_wait();
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= vs.count) return;
  const uint32_t u = vs[i];
  const uint32_t cap = g.cap[u];
  uint4 x = make_uint4(kEmpty, kEmpty, kEmpty, kEmpty);
  if (cap >= 4) {  // starts on a 16-byte boundary; slots past the ids hold kEmpty
    x = *reinterpret_cast<const uint4 *>(g.slots + g.base[u]);
  } else if (cap) {
    const uint32_t *p = g.slots + g.base[u];
    x.x = p[0];
    if (cap > 1) x.y = p[1];
  }
  par[u] = min(u, x.x);
  nb1[i] = x.y;
  nb2[i] = x.x > u ? x.x : kEmpty;
}

// A round, after a compression: of the roots of u and its two kept neighbours
// the larger ones go below the smallest.  A root keeps the smallest that any
// vertex offers it, and a parent that is read while it changes is an ancestor:
// either way a tree only moves below a vertex of its own component with a
// smaller id.  A hook that another one replaces is linked later, by
// k_cc_link_kept.
// Only what was a root at the launch may be offered to: of any other vertex the
// parent may stand for a first edge, which is not kept.  A neighbour without a row
// is not in the lists, so after the first round the compressions have left it where
// that put it, and its root is looked up (`walk`).
// The first round, of every vertex, leaves 5e3 trees on that uniform graph.
// Their roots would get hundreds of offers each, and atomics on one address
// wait for each other (25 ns apiece: a second round of every vertex takes 240
// us, of every 8th 74 us).  So on a large graph the second round takes every
// 32nd vertex and the third every 512th, which joins the two or three trees that
// then hold most vertices and leaves few edges to k_cc_link_kept.  When the second
// round finds nothing to hook the third returns at once.  Below kCcThirdN vertices
// the second takes every 8th and is the last, and what follows looks roots up
// instead of a compression: launches count there.
// Without later rounds k_cc_link_kept's compare-and-swaps wait for each other at the
// same roots: uniform graphs of 20,000, 65,536, 131,000 and 300,000 vertices with
// 4 edges each take 141, 306, 574 and 900 us, and with them 68, 70, 82 and 118; grids,
// stars and skewed graphs, which the first round all but finishes, pay 2-3 us for the
// launch (R-MAT, 65,536 vertices, 54 -> 57).  (A second and third round and their
// compressions below kCcThirdN: 72, 85, 130 and R-MAT 62.)  Below kCcSampledN rows
// there is too little to wait for (10,000: 70 and 63 us with 10 edges each, 55 and 63
// with 40).  Below kCcSampledM[0] / kCcSampledM[1] edges a row the first two edges
// are most of what there is and leave many small trees, to which few wait: of 300,000
// vertices with 2.7 edges each 350 us without and 600 with them, with 3.16 each 520
// and 950, with 3.25 each 490 and 340.
// The parents come through L1: nearly all are one hot root, whose loads would
// queue at one L2 slice, and a stale one is an ancestor too.
constexpr uint32_t kCcFew = 2;  // fewer rows than one vertex in 2: over the lists
constexpr uint32_t kCcSampledN = 1u << 14;
constexpr uint64_t kCcSampledM[2] = {16, 5};
constexpr uint32_t kCcThirdN = 1u << 17;
constexpr int kCcMaxRounds = 3;
constexpr uint32_t kCcStride[kCcMaxRounds][kCcMaxRounds] = {{1}, {1, 8}, {1, 32, 512}};

// the root of x as far as it is known here: nothing is changed on the way
__device__ __forceinline__ uint32_t cc_root(const uint32_t *par, uint32_t x) {
  for (uint32_t p; (p = par[x]) != x;) x = p;
  return x;
}

__global__ void k_cc_hook(CcVerts vs, const uint32_t *__restrict__ nb1,
                          const uint32_t *__restrict__ nb2, uint32_t stride, bool walk,
                          uint32_t *par, const unsigned long long *__restrict__ before,
                          unsigned long long *__restrict__ hooks) {
  pdl_wait();
  if (before && *before == 0) return;
  const uint64_t i = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) * stride;
  bool hooked = false;
  if (i < vs.count) {
    const uint32_t x = nb1[i], y = nb2[i];
    uint32_t a = par[vs[(uint32_t)i]];
    uint32_t b = x != kEmpty ? par[x] : a;
    uint32_t c = y != kEmpty ? par[y] : a;
    if (walk) {
      a = cc_root(par, a);
      b = cc_root(par, b);
      c = cc_root(par, c);
    }
    const uint32_t m = min(a, min(b, c));
    // a look (past L1) before an atomic: an offer that is no better costs less
    if (a > m && ld_par(par, a) > m) hooked |= atomicMin(&par[a], m) > m;
    if (b > m && ld_par(par, b) > m) hooked |= atomicMin(&par[b], m) > m;
    if (c > m && ld_par(par, c) > m) hooked |= atomicMin(&par[c], m) > m;
  }
  if (__syncthreads_or(hooked) && threadIdx.x == 0) *(volatile unsigned long long *)hooks = 1;
}

// The kept edges that the rounds have not joined, by find and compare-and-swap:
// afterwards the trees are the components of every vertex's first two edges, in
// whatever order the hooks went.  After a round that no compression followed the
// roots are looked up (`walk`) before they are compared.
__global__ void k_cc_link_kept(CcVerts vs, const uint32_t *__restrict__ nb1,
                               const uint32_t *__restrict__ nb2, bool walk, uint32_t *par,
                               unsigned long long *__restrict__ hooks,
                               unsigned long long *__restrict__ err) {
  pdl_wait();
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  bool linked = false;
  if (i < vs.count) {
    const uint32_t u = vs[i], x = nb1[i], y = nb2[i];
    uint32_t a = par[u], b = x != kEmpty ? par[x] : a, c = y != kEmpty ? par[y] : a;
    if (walk) {
      a = cc_root(par, a);
      b = cc_root(par, b);
      c = cc_root(par, c);
    }
    // (no neighbour: two walks from one vertex may end apart while others link)
    const bool join_x = x != kEmpty && b != a, join_y = y != kEmpty && c != a;
    if (join_x) cc_link(par, u, x, err);
    if (join_y) cc_link(par, u, y, err);
    linked = join_x || join_y;
  }
  if (__syncthreads_or(linked) && threadIdx.x == 0) *(volatile unsigned long long *)hooks = 1;
}

// phase 3, one-leaf vertices: thread per vertex
__global__ void k_cc_rest_small(DGraph g, const unsigned long long *__restrict__ sdesc,
                                const uint32_t *__restrict__ small, uint64_t nsmall,
                                const unsigned long long *__restrict__ giant,
                                uint32_t *__restrict__ par,
                                unsigned long long *__restrict__ err) {
  pdl_wait();
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nsmall) return;
  const uint32_t u = small[i];
  if (ld_par(par, u) == (uint32_t)*giant) return;
  const unsigned long long d = sdesc[i];
  const uint32_t *p = g.slots + (d >> 6);
  const uint32_t deg = (uint32_t)(d & 63);
  for (uint32_t j = 0; j < deg; j++) cc_link(par, u, p[j], err);
}

// phase 3, multi-leaf vertices: warp per chunk of leaves, lane = slot
__global__ void k_cc_rest_chunks(DGraph g, const unsigned long long *__restrict__ cdesc,
                                 const uint32_t *__restrict__ cv, uint64_t nchunks,
                                 const unsigned long long *__restrict__ giant,
                                 uint32_t *__restrict__ par,
                                 unsigned long long *__restrict__ err) {
  pdl_wait();
  const uint64_t c = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (c >= nchunks) return;
  const uint32_t u = cv[c];
  if (ld_par(par, u) == (uint32_t)*giant) return;
  const unsigned long long dsc = cdesc[c];
  const uint64_t leaf0 = dsc >> 8;
  const uint32_t nl = (uint32_t)(dsc & 63);
  for (uint32_t l = 0; l < nl; l++) {
    const uint32_t cnt = g.lcnt[leaf0 + l];
    if ((uint32_t)lane < cnt) cc_link(par, u, g.slots[((leaf0 + l) << kLeafLog) + lane], err);
  }
}

// ------------------------------------------------------------- bc
// Level bookkeeping: the per-level counters are a handful of addresses hit
// by every vertex, so lanes of a warp that share a level add once (match),
// and the maximum depth is taken per block before its one atomic.
__device__ __forceinline__ uint32_t level_add(uint32_t *ctr, int32_t d, bool on) {
  const uint32_t key = on ? (uint32_t)d : 0xffffffffu;
  const uint32_t peers = __match_any_sync(0xffffffffu, key);
  const int lane = threadIdx.x & 31;
  const int leader = __ffs(peers) - 1;
  uint32_t base = 0;
  if (on && lane == leader) base = atomicAdd(ctr, (uint32_t)__popc(peers));
  base = __shfl_sync(0xffffffffu, base, leader);
  return base + __popc(peers & ((1u << lane) - 1u));
}

__device__ __forceinline__ void block_max_to(int32_t d, unsigned long long *out) {
  __shared__ int32_t s_max;
  if (threadIdx.x == 0) s_max = -1;
  __syncthreads();
  for (int o = 16; o > 0; o >>= 1) d = max(d, __shfl_down_sync(0xffffffffu, d, o));
  if ((threadIdx.x & 31) == 0 && d >= 0) atomicMax(&s_max, d);
  __syncthreads();
  if (threadIdx.x == 0 && s_max >= 0) atomicMax(out, (unsigned long long)s_max);
}

// neighbours (or leaves) whose loads the BC kernels keep in flight together
constexpr int kBcAhead = 8;

// items (big vertices of the level list, one per leaf chunk)
__global__ void k_bc_item_counts(const uint32_t *__restrict__ list, uint32_t nl,
                                 const uint32_t *__restrict__ cap,
                                 uint32_t *__restrict__ cnt) {
  uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= nl) return;
  uint32_t c = cap[list[p]];
  cnt[p] = c > kLeaf ? ((c >> kLeafLog) + kChunkLeaves - 1) / kChunkLeaves : 0;
}

__global__ void k_bc_expand(const uint32_t *__restrict__ list, uint32_t nl,
                            const uint32_t *__restrict__ cnt,
                            const uint32_t *__restrict__ off,
                            uint32_t *__restrict__ iv, uint32_t *__restrict__ il0) {
  uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= nl) return;
  for (uint32_t j = 0; j < cnt[p]; j++) {
    iv[off[p] + j] = list[p];
    il0[off[p] + j] = j * kChunkLeaves;
  }
}

__global__ void k_gather_bounds(const uint32_t *__restrict__ off,
                                const uint32_t *__restrict__ pos, uint32_t k,
                                uint32_t *__restrict__ out) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < k) out[i] = off[pos[i]];
}

// ------------------------------------------------------------- tc
// orientation and counting in tcshared.cuh

// The orientation passes take kTcLeaves leaves a warp, all their loads
// issued before any is used (a leaf alone is three dependent round trips:
// its directory entry, its line, its ids' degrees).  The count pass also
// records each leaf's keep mask, so the fill pass needs no degree lookups.
constexpr int kTcLeaves = 4;

__global__ void k_tc_leafcount(const uint32_t *__restrict__ slots,
                               const uint32_t *__restrict__ owner,
                               const uint64_t *__restrict__ slot,
                               const uint32_t *__restrict__ cnt,
                               uint64_t nleaves, const uint32_t *__restrict__ deg,
                               uint64_t *__restrict__ out, uint32_t *__restrict__ kmask) {
  const uint64_t k0 = (((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * kTcLeaves;
  const int lane = threadIdx.x & 31;
  if (k0 >= nleaves) return;
  uint32_t u[kTcLeaves], c[kTcLeaves], x[kTcLeaves];
  uint64_t sl[kTcLeaves];
#pragma unroll
  for (int j = 0; j < kTcLeaves; j++) {
    const uint64_t k = k0 + j;
    u[j] = 0;
    c[j] = 0;
    sl[j] = 0;
    if (k < nleaves) {
      u[j] = owner[k];
      sl[j] = slot[k];
      c[j] = cnt[k];
    }
  }
#pragma unroll
  for (int j = 0; j < kTcLeaves; j++) x[j] = (uint32_t)lane < c[j] ? slots[sl[j] + lane] : 0u;
#pragma unroll
  for (int j = 0; j < kTcLeaves; j++) {
    const bool keep = (uint32_t)lane < c[j] && ranks_above(deg, x[j], u[j]);
    const uint32_t m = __ballot_sync(0xffffffffu, keep);
    if (lane == 0 && k0 + j < nleaves) {
      out[k0 + j] = __popc(m);
      kmask[k0 + j] = m;
    }
  }
}

__global__ void k_tc_fill(const uint32_t *__restrict__ slots,
                          const uint64_t *__restrict__ slot, uint64_t nleaves,
                          const uint32_t *__restrict__ kmask,
                          const uint64_t *__restrict__ lpre,
                          uint32_t *__restrict__ adj) {
  const uint64_t k0 = (((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * kTcLeaves;
  const int lane = threadIdx.x & 31;
  if (k0 >= nleaves) return;
  uint32_t m[kTcLeaves], x[kTcLeaves];
  uint64_t sl[kTcLeaves], at[kTcLeaves];
#pragma unroll
  for (int j = 0; j < kTcLeaves; j++) {
    const uint64_t k = k0 + j;
    m[j] = 0;
    sl[j] = 0;
    at[j] = 0;
    if (k < nleaves) {
      m[j] = kmask[k];
      sl[j] = slot[k];
      at[j] = lpre[k];
    }
  }
#pragma unroll
  for (int j = 0; j < kTcLeaves; j++) x[j] = (m[j] >> lane) & 1u ? slots[sl[j] + lane] : 0u;
#pragma unroll
  for (int j = 0; j < kTcLeaves; j++)
    if ((m[j] >> lane) & 1u) adj[at[j] + __popc(m[j] & ((1u << lane) - 1u))] = x[j];
}

// per vertex: its oriented list as one word (tcshared.cuh)
__global__ void k_tc_lists(const uint64_t *__restrict__ vleaf,
                           const uint64_t *__restrict__ lpre, uint32_t n,
                           uint64_t *__restrict__ desc) {
  const uint32_t v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= n) return;
  const uint64_t b = lpre[vleaf[v]], e = lpre[vleaf[v + 1]];
  desc[v] = (b << kTcLenBits) | (e - b);
}

// ------------------------------------------------------------- pairs
// Common neighbours of pairs: every id of the shorter row is looked up in the
// longer one.  On a skewed graph one pair of hubs holds more leaves than all
// the rest (a thread per pair, the form before this, spent its time in the one
// thread that walked the longest row: 14.5 ms for 20,000 edges of an RMAT
// scale-18 graph, 0.18 ms this way).  So a
// cluster of kCommonCtas blocks takes its pairs together: each block lists its
// share with the leaf counts of the shorter rows in its shared memory, and the
// cluster's warps split the cluster's leaves evenly, reading the pair
// descriptors of the other blocks through distributed shared memory.  Two rows of one
// leaf each and few ids in all (kCommonMerged) are merged by the thread that lists
// the pair: a warp a leaf would leave most lanes idle (100,000 pairs of rows of four
// ids 64 us, so 36, by a thread a pair 30; of eight ids 62, 42 and 39).  The
// split needs no scratch and no readback, so the call stays one launch that
// neither allocates nor synchronises.  Bound by the chain of dependent loads
// of a lookup and the L1 rate of its scattered sectors.
constexpr int kCommonCtas = 8;       // blocks of a cluster (the portable size)
constexpr int kCommonThreads = 512;  // 128 warps to a cluster
constexpr uint32_t kCommonPairs = kCommonThreads;  // pairs of a block, at most
// ids of both rows that a thread merges: while the blocks all run at once a merge is
// the longer chain (20,000 pairs of an RMAT scale-18 graph 55.6 us with 16, 58.2 with
// 32; of rows of four ids 29 and 27), and later rounds wait for threads (100,000 pairs
// of rows of eight ids 54 and 42)
constexpr uint32_t kCommonMerged = 16, kCommonMergedOfMany = 32;

struct CommonPair {
  uint64_t sbase, obase;  // the shorter and the longer row
  uint32_t scap, sdeg, ocap;
  uint32_t lim;  // ids from here on do not count (early end)
};

// common ids below lim of two rows of one leaf each, na and nb ids: one merge, after
// a load of every sector of both (a merge alone would wait for them one by one)
__device__ __forceinline__ uint32_t common_merged(const uint32_t *pa, uint32_t na,
                                                  const uint32_t *pb, uint32_t nb, uint32_t lim) {
  if (!na || !nb) return 0;
  uint32_t i = 0, j = 0, count = 0, x = pa[0], y = pb[0], t = 0;
#pragma unroll
  for (uint32_t k = 8; k < kLeaf; k += 8) {
    if (k < na) t |= pa[k];
    if (k < nb) t |= pb[k];
  }
  asm volatile("" ::"r"(t));
  while (x < lim && y < lim) {
    const bool ax = x <= y, by = y <= x;
    count += ax && by;
    if (ax) x = ++i < na ? pa[i] : kEmpty;
    if (by) y = ++j < nb ? pb[j] : kEmpty;
  }
  return count;
}

__global__ void __cluster_dims__(kCommonCtas, 1, 1) __launch_bounds__(kCommonThreads, 2)
k_common(DGraph g, const uint32_t *__restrict__ pairs, uint64_t n, uint32_t per_cta,
         uint32_t merged, bool early, unsigned long long *__restrict__ out) {
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  __shared__ CommonPair s_pair[kCommonPairs];
  __shared__ uint64_t s_pre[kCommonPairs + 1];  // leaves of the shorter rows before pair j
  __shared__ uint64_t s_warp[kCommonThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t full = 0xffffffffu;
  const uint64_t cta0 = (uint64_t)blockIdx.x - cl.block_rank();  // the cluster's first block
  {
    const uint32_t j = threadIdx.x;
    const uint64_t i = (uint64_t)blockIdx.x * per_cta + j;
    uint64_t leaves = 0;
    if (j < per_cta && i < n) {
      const uint32_t a = pairs[2 * i], b = pairs[2 * i + 1];
      unsigned long long count = 0;
      if (a < g.n && b < g.n) {
        const uint32_t da = g.deg[a], db = g.deg[b];
        const uint32_t s = da <= db ? a : b, o = s == a ? b : a;
        const uint32_t scap = g.cap[s], ocap = g.cap[o], sdeg = min(da, db);
        const uint32_t lim = early ? min(a, b) : kEmpty;
        const uint64_t sbase = g.base[s], obase = g.base[o];
        if (scap <= kLeaf && ocap <= kLeaf && da + db <= merged) {
          count = common_merged(g.slots + sbase, sdeg, g.slots + obase, max(da, db), lim);
        } else if (scap) {
          s_pair[j] = CommonPair{sbase, obase, scap, sdeg, ocap, lim};
          leaves = nleaves_of(scap);
        }
      }
      out[i] = count;
    }
    // inclusive prefix over the block
    uint64_t inc = leaves;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint64_t y = __shfl_up_sync(full, inc, d);
      if (lane >= d) inc += y;
    }
    if (lane == 31) s_warp[warp] = inc;
    __syncthreads();
    for (int w = 0; w < warp; w++) inc += s_warp[w];
    if (j < kCommonPairs) s_pre[j + 1] = inc;
    if (j == 0) s_pre[0] = 0;
  }
  cl.sync();  // every block's pairs are listed, and their outputs set
  // lane c < kCommonCtas: the leaves of block c, then their inclusive prefix
  uint64_t ctot = lane < kCommonCtas ? cl.map_shared_rank(s_pre, lane)[kCommonPairs] : 0;
  uint64_t cinc = ctot;
#pragma unroll
  for (int d = 1; d < kCommonCtas; d <<= 1) {
    const uint64_t y = __shfl_up_sync(full, cinc, d);
    if (lane >= d) cinc += y;
  }
  const uint64_t total = __shfl_sync(full, cinc, kCommonCtas - 1);
  constexpr uint32_t kWarps = kCommonCtas * (kCommonThreads / 32);
  const uint32_t w = cl.block_rank() * (kCommonThreads / 32) + warp;
  const uint64_t hi = total * (w + 1) / kWarps;
  for (uint64_t at = total * w / kWarps; at < hi;) {
    // block c and pair j of leaf `at` (empty rows own no leaf): the pairs before it
    // by runs of 32, then within the run
    const int c = __popc(__ballot_sync(full, lane < kCommonCtas && cinc <= at));
    const uint64_t rem = at - __shfl_sync(full, cinc - ctot, c);
    const uint64_t *pre = cl.map_shared_rank(s_pre, c);
    const uint32_t j0 = 32 * __popc(__ballot_sync(
        full, lane < (int)kCommonPairs / 32 && pre[min(32u * (lane + 1), kCommonPairs)] <= rem));
    const uint32_t j = j0 + __popc(__ballot_sync(full, pre[j0 + lane + 1] <= rem));
    const CommonPair q = cl.map_shared_rank(s_pair, c)[j];
    const uint32_t l0 = (uint32_t)(rem - pre[j]);
    const uint64_t left = min(pre[j + 1] - rem, hi - at);
    const uint32_t l1 = l0 + (uint32_t)left;
    uint32_t hits = 0;
    for (uint32_t l = l0; l < l1; l++) {
      const uint32_t k = leaf_count(g, q.sbase, q.scap, q.sdeg, l);
      const uint32_t x = (uint32_t)lane < k
                             ? g.slots[q.sbase + ((uint64_t)l << kLeafLog) + lane]
                             : kEmpty;
      if (__shfl_sync(full, x, 0) >= q.lim) break;  // this leaf and the rest
      if (x < q.lim) hits += seg_has(g.slots, q.obase, q.ocap, x);
    }
    hits = __reduce_add_sync(full, hits);
    if (lane == 0 && hits)
      atomicAdd(&out[(cta0 + c) * per_cta + j], (unsigned long long)hits);
    at += left;
  }
  cl.sync();  // no block leaves while another reads its pairs
}

}  // namespace

// ================================================================== host
// the graph's traversal state, made by the first traversal
static sst_status state(sst_graph *g, TravState **out) {
  if (!g->trav) {
    TravState *t = new (std::nothrow) TravState();
    if (!t || !trav_words_init(t, sizeof(BfsCtl) + sizeof(BcCtl), TravWordsRt{g->stream})) {
      cudaGetLastError();
      delete t;
      set_error_message("cannot allocate the traversal state");
      return SST_ENOMEM;
    }
    g->trav = t;
  }
  *out = g->trav;
  return SST_OK;
}

static sst_status ensure_lists(sst_graph *g) {
  TravState *t = nullptr;
  sst_status st = state(g, &t);
  if (st != SST_OK) return st;
  if (t->version == g->version && t->lists_cl == t->chunk_leaves) return SST_OK;
  cudaStream_t s = g->stream;
  const uint32_t n = g->n, cl = t->chunk_leaves;
  // sized by what the slab can hold, so nothing waits for the counts and an
  // update that moves no slab grows no list
  const uint64_t most_big = std::min<uint64_t>(n, g->nslots / (2 * kLeaf));
  // (several chunks: more than cl leaves)
  const uint64_t most_multi = std::min<uint64_t>(n, g->nslots / ((uint64_t)kLeaf * (cl + 1)));
  const uint64_t most_chunks = most_big + g->nslots / ((uint64_t)kLeaf * cl);
  const unsigned nb = blocks_for(n, kListBlock);
  SST_CUDA_TRY(t->lsum.ensure(4 * (uint64_t)nb));
  SST_CUDA_TRY(t->small.exact((uint64_t)n + 1));
  SST_CUDA_TRY(t->sdesc.exact((uint64_t)n + 1));
  SST_CUDA_TRY(t->big.ensure(most_big + 1));
  SST_CUDA_TRY(t->multi.ensure(most_multi + 1));
  SST_CUDA_TRY(t->cv.ensure(most_chunks + 1));
  SST_CUDA_TRY(t->cdesc.ensure(most_chunks + 1));
  uint4 *sums = reinterpret_cast<uint4 *>(t->lsum.p);
  uint4 *totals = reinterpret_cast<uint4 *>(t->h_small + 8);
  SST_LAUNCH_PDL(k_list_count, nb, kScanThreads, 0, s, g->d_cap, n, cl, sums);
  SST_LAUNCH_PDL(k_list_prefix, 1, kScanThreads, 0, s, sums, nb, totals);
  SST_LAUNCH_PDL(k_list_fill, nb, kScanThreads, 0, s, g->view(), cl, sums, t->small.p, t->sdesc.p,
                 t->big.p, t->multi.p, t->cv.p, t->cdesc.p);
  SST_CUDA_TRY(cudaStreamSynchronize(s));
  SST_CUDA_TRY(cudaGetLastError());
  t->nsmall = totals->x;
  t->nbig = totals->y;
  t->nmulti = totals->z;
  t->nchunks = totals->w;
  t->version = g->version;
  t->lists_cl = cl;
  t->lists_stamp++;
  return SST_OK;
}

sst_status pagerank(sst_graph *g, uint32_t iters, double damping, double *d_rank) {
  sst_status st = ensure_lists(g);
  if (st != SST_OK) return st;
  TravState *t = g->trav;
  cudaStream_t s = g->stream;
  uint32_t n = g->n;
  if (n == 0) return SST_OK;
  SST_CUDA_TRY(t->ca.exact(n));
  SST_CUDA_TRY(t->cb.exact(n));
  SST_CUDA_TRY(t->partial.ensure(t->nchunks + 1));
  SST_CUDA_TRY(t->inv_deg.exact(n));
  unsigned long long *rdeg = reinterpret_cast<unsigned long long *>(t->inv_deg.p);
  static bool carveout = false;
  if (!carveout) {
    // these kernels use no shared memory: give the SM's storage to L1
    cudaFuncSetAttribute(k_pr_iter<4>, cudaFuncAttributePreferredSharedMemoryCarveout, 0);
    cudaFuncSetAttribute(k_pr_iter<8>, cudaFuncAttributePreferredSharedMemoryCarveout, 0);
    cudaFuncSetAttribute(k_pr_iter<16>, cudaFuncAttributePreferredSharedMemoryCarveout, 0);
    carveout = true;
  }
  double r0 = 1.0 / (double)n;
  double base = (1.0 - damping) / (double)n;
  if (iters == 0) {
    SST_LAUNCH(k_fill_d, blocks_for(n), kTB, 0, s, d_rank, n, r0);
    SST_CUDA_TRY(cudaGetLastError());
    return SST_OK;
  }
  unsigned long long r0f = 0;
  const PrConst K = pr_const(n, damping, &r0f);
  unsigned long long *cin = reinterpret_cast<unsigned long long *>(t->ca.p);
  unsigned long long *cout = reinterpret_cast<unsigned long long *>(t->cb.p);
  unsigned long long *part = reinterpret_cast<unsigned long long *>(t->partial.p);
  // the shared-memory cache: at most the rows, at most 24,576 entries
  // (192 KiB), one copy per block; persistent grids sized by occupancy at
  // that footprint (more than 8,192 entries leaves under three blocks/SM)
  const uint32_t hot = std::min<uint32_t>(t->pr_hot, std::min<uint32_t>(n, 24576));
  const size_t hot_bytes = (size_t)hot * 8;
  const bool big = hot > kHotBig;  // 1024-thread blocks
  const int hot_threads = big ? 1024 : kHotThreads;
  unsigned hot_grid[4] = {1, 1, 1, 1};
  if (hot) {
    const void *fns[4] = {
        big ? (const void *)k_pr_small_hot<4, 1024> : (const void *)k_pr_small_hot<4>,
        big ? (const void *)k_pr_small_hot<8, 1024> : (const void *)k_pr_small_hot<8>,
        big ? (const void *)k_pr_small_hot<16, 1024> : (const void *)k_pr_small_hot<16>,
        big ? (const void *)k_pr_chunks_hot<1024> : (const void *)k_pr_chunks_hot<>};
    for (int i = 0; i < 4; i++) {
      SST_CUDA_TRY(cudaFuncSetAttribute(fns[i], cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)hot_bytes));
      int per_sm = 0;
      SST_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fns[i], hot_threads,
                                                                 hot_bytes));
      hot_grid[i] = (unsigned)std::max(1, per_sm) * (unsigned)g->sms;
    }
  }
  auto launch_all = [&](bool fresh) {
    unsigned long long *ci = cin, *co = cout;
    SST_LAUNCH_PDL(k_pr_start, blocks_for(n), kTB, 0, s, g->d_deg, n, r0f, fresh, rdeg, ci, co,
               d_rank, base);
    DGraph dg = g->view();
    for (uint32_t it = 0; it < iters; it++) {
      bool last = it + 1 == iters;
      if (hot && t->nsmall) {
#define SST_PR_SMALL_HOT(G, I)                                                        \
  do {                                                                              \
    if (big)                                                                        \
      SST_LAUNCH((k_pr_small_hot<G, 1024>), hot_grid[I], 1024, hot_bytes, s, dg,    \
                 t->sdesc.p, t->small.p, t->nsmall, ci, co, d_rank, rdeg, K, last, hot); \
    else                                                                            \
      SST_LAUNCH((k_pr_small_hot<G>), hot_grid[I], kHotThreads, hot_bytes, s, dg,   \
                 t->sdesc.p, t->small.p, t->nsmall, ci, co, d_rank, rdeg, K, last, hot); \
  } while (0)
        if (t->pr_lanes == 4)
          SST_PR_SMALL_HOT(4, 0);
        else if (t->pr_lanes == 16)
          SST_PR_SMALL_HOT(16, 2);
        else
          SST_PR_SMALL_HOT(8, 1);
#undef SST_PR_SMALL_HOT
      } else if (!hot) {
        const uint32_t lanes = t->pr_lanes == 4 || t->pr_lanes == 16 ? t->pr_lanes : 8;
        const uint64_t groups = (t->nsmall + kSmallPer - 1) / kSmallPer;
        const unsigned cblocks = (unsigned)((32 * t->nchunks + kTB - 1) / kTB);
        const unsigned sblocks = (unsigned)((groups * lanes + kTB - 1) / kTB);
#define SST_PR_ITER(G)                                                                  \
  SST_LAUNCH_PDL(k_pr_iter<G>, cblocks + sblocks, kTB, 0, s, dg, t->cdesc.p, t->cv.p,   \
                 t->nchunks, cblocks, t->sdesc.p, t->small.p, t->nsmall, ci, co, d_rank, rdeg, \
                 part, K, last)
        if (cblocks + sblocks == 0)
          ;  // no edges
        else if (lanes == 4)
          SST_PR_ITER(4);
        else if (lanes == 16)
          SST_PR_ITER(16);
        else
          SST_PR_ITER(8);
#undef SST_PR_ITER
      }
      if (hot && t->nchunks && big)
        SST_LAUNCH(k_pr_chunks_hot<1024>, hot_grid[3], 1024, hot_bytes, s, dg, t->cdesc.p,
                   t->cv.p, t->nchunks, ci, co, d_rank, rdeg, part, K, last, hot);
      else if (hot && t->nchunks)
        SST_LAUNCH(k_pr_chunks_hot<>, hot_grid[3], kHotThreads, hot_bytes, s, dg, t->cdesc.p,
                   t->cv.p, t->nchunks, ci, co, d_rank, rdeg, part, K, last, hot);
      if (t->nmulti)
        SST_LAUNCH_PDL(k_pr_fix, warp_blocks(t->nmulti), kTB, 0, s, dg, t->multi.p, t->nmulti,
                   t->lists_cl, part, co, d_rank, rdeg, K, last);
      std::swap(ci, co);
    }
  };
  // Replay the captured iterations when nothing they depend on changed.  The
  // first call on changed work lists launches them one by one -- a served graph
  // is updated between its queries, and a capture costs more than it saves
  // once -- and the second one captures.  With the kernel profiler on they are
  // launched one by one so each is timed.
  const bool fresh = t->inv_version != g->version;
  t->inv_version = g->version;
  const void *key[6] = {d_rank, s, cin, cout, part, rdeg};
  bool same = t->pr_exec && t->pr_version == t->lists_stamp &&
              t->pr_lanes_used == t->pr_lanes && t->pr_hot_used == t->pr_hot &&
              t->pr_iters == iters && t->pr_damping == damping;
  for (int i = 0; i < 6 && same; i++) same = t->pr_key[i] == key[i];
  if (fresh || profiling("k_pr_iter") || profiling("k_pr_chunks_hot")) {
    launch_all(fresh);
    SST_CUDA_TRY(cudaGetLastError());
    return SST_OK;
  }
  if (!same) {
    if (t->pr_exec) cudaGraphExecDestroy(t->pr_exec);
    t->pr_exec = nullptr;
    cudaGraph_t graph = nullptr;
    const uint64_t l0 = launches();
    SST_CUDA_TRY(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
    launch_all(false);
    cudaError_t e = cudaStreamEndCapture(s, &graph);
    t->pr_kernels = (int64_t)(launches() - l0);
    note_launches(-t->pr_kernels);  // captured, not launched
    if (e == cudaSuccess) e = cudaGraphInstantiate(&t->pr_exec, graph, 0);
    if (graph) cudaGraphDestroy(graph);
    if (e != cudaSuccess) {
      t->pr_exec = nullptr;
      SST_CUDA_TRY(e);
    }
    t->pr_version = t->lists_stamp;
    t->pr_lanes_used = t->pr_lanes;
    t->pr_hot_used = t->pr_hot;
    t->pr_iters = iters;
    t->pr_damping = damping;
    for (int i = 0; i < 6; i++) t->pr_key[i] = key[i];
  }
  SST_CUDA_TRY(cudaGraphLaunch(t->pr_exec, s));
  note_launches(t->pr_kernels);
  return SST_OK;
}

// blocks of a cooperative grid for `threads` threads of work: no more than the
// work fills (see bfslevels.cuh), no more than fit at once
static sst_status coop_grid(const sst_graph *g, const void *kernel, uint64_t threads,
                            unsigned *grid) {
  int per_sm = 0;
  SST_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kCoopThreads, 0));
  if (per_sm < 1) {
    set_error_message("a traversal kernel does not fit the device");
    return SST_EDEVICE;
  }
  const uint64_t most = (uint64_t)std::max(std::min(per_sm, kCoopPerSm) * g->sms - kCoopFree, 1);
  *grid = (unsigned)std::min<uint64_t>(most, (threads + kCoopThreads - 1) / kCoopThreads + 1);
  return SST_OK;
}

constexpr uint32_t kVertsPerThread = 8;

// A search's arguments over the graph's work lists, and its grid (see
// bfslevels.cuh).  d_depths may be null (a temporary), d_parents too (none).
static sst_status bfs_setup(sst_graph *g, uint32_t src, int32_t *d_parents, int32_t *d_depths,
                            const void *kernel, BfsArgs *a, unsigned *grid) {
  sst_status st = ensure_lists(g);
  if (st != SST_OK) return st;
  TravState *t = g->trav;
  const uint32_t n = g->n;
  // a row's push items are at most 32 / kBfsLeaves for each of its chunks in
  // the lists (chunks of up to 32 leaves)
  const uint64_t max_items = t->nchunks * (32 / kBfsLeaves) + 1;
  SST_CUDA_TRY(t->qa.exact((uint64_t)n + 1));
  SST_CUDA_TRY(t->qitems.ensure(max_items));
  SST_CUDA_TRY(t->fbits.ensure(n / 32 + 2));
  if (!d_depths) {
    SST_CUDA_TRY(t->depth_tmp.exact(n));
    d_depths = t->depth_tmp.p;
  }
  *a = BfsArgs{g->view(),   g->m,       src,         t->bfs_alpha, t->small.p,
               t->sdesc.p,  t->nsmall,  t->cv.p,     t->cdesc.p,   t->nchunks,
               d_depths,    d_parents,  t->fbits.p,  t->qa.p,      t->qitems.p,
               max_items,   reinterpret_cast<BfsCtl *>(t->d_bfs),
               reinterpret_cast<unsigned long long *>(t->h_small)};
  // and a thread for eight vertices: the search clears and scans arrays of all
  // vertices, whatever the rows hold (2,000 rows in use of 2^24: BFS 1.3 ms by the
  // five blocks that the rows alone ask for, 0.12 by these; 4 to 32 vertices a thread
  // alike)
  const uint64_t work = std::max<uint64_t>({t->nsmall, 32 * t->nchunks, n / kVertsPerThread});
  return coop_grid(g, kernel, work, grid);
}

// waits for a search and reports its error
static sst_status bfs_finish(sst_graph *g, const char *what) {
  SST_CUDA_TRY(cudaStreamSynchronize(g->stream));
  const uint64_t err = *(volatile uint64_t *)g->trav->h_small;
  if (!err) return SST_OK;
  set_error_message(err == 1   ? "%s: a grid barrier timed out"
                    : err == 2 ? "%s: a level queue overflowed"
                               : "%s exceeded n levels",
                    what);
  return err == 2 ? SST_EDEVICE : SST_ETIMEDOUT;
}

sst_status bfs(sst_graph *g, uint32_t src, int32_t *d_parents, int32_t *d_depths) {
  BfsArgs a;
  unsigned grid = 1;
  sst_status st = bfs_setup(g, src, d_parents, d_depths,
                            reinterpret_cast<const void *>(k_bfs_levels), &a, &grid);
  if (st != SST_OK) return st;
  SST_CUDA_TRY(launch_coop("k_bfs_levels", k_bfs_levels, grid, kCoopThreads, g->stream, a));
  return bfs_finish(g, "BFS");
}

sst_status cc(sst_graph *g, uint32_t *d_labels) {
  sst_status st = ensure_lists(g);
  if (st != SST_OK) return st;
  TravState *t = g->trav;
  cudaStream_t s = g->stream;
  const uint32_t n = g->n;
  if (n == 0) return SST_OK;
  uint32_t *par = d_labels;
  unsigned long long *giant = t->d_small, *err = t->d_small + 1, *hooks = t->d_small + 2;
  SST_CUDA_TRY(t->qa.exact((uint64_t)n + 1));
  SST_CUDA_TRY(t->qb.exact((uint64_t)n + 1));
  SST_CUDA_TRY(cudaMemsetAsync(t->d_small, 0, (3 + kCcMaxRounds) * 8, s));
  const DGraph dg = g->view();
  const uint64_t rows = t->nsmall + t->nbig;
  const bool few = rows < n / kCcFew;
  const CcVerts vs = few ? CcVerts{t->small.p, t->big.p, (uint32_t)t->nsmall, (uint32_t)rows}
                         : CcVerts{nullptr, nullptr, 0, n};
  auto compress = [&](const unsigned long long *if_set) {
    if (few)
      SST_LAUNCH_PDL(k_cc_compress_some, blocks_for(vs.count), kTB, 0, s, vs, par, if_set);
    else
      SST_LAUNCH_PDL(k_cc_compress, blocks_for(n), kTB, 0, s, par, n, if_set);
  };
  const unsigned long long *const none = nullptr;
  if (few) SST_LAUNCH(k_iota, blocks_for(n), kTB, 0, s, par, n);
  SST_LAUNCH_PDL(k_cc_hook_first, blocks_for(vs.count), kTB, 0, s, dg, vs, par, t->qa.p, t->qb.p);
  compress(nullptr);
  const bool later = rows >= kCcSampledN && g->m * kCcSampledM[1] >= rows * kCcSampledM[0];
  const int rounds = !later ? 1 : vs.count < kCcThirdN ? 2 : 3;
  for (int r = 0; r < rounds; r++) {
    const uint32_t stride = kCcStride[rounds - 1][r];
    const bool packed = r == 0 || rounds == 3;  // a compression follows
    SST_LAUNCH_PDL(k_cc_hook, blocks_for((vs.count + stride - 1) / stride), kTB, 0, s, vs, t->qa.p,
                   t->qb.p, stride, few && r, par, r ? hooks + r - 1 : nullptr,
                   hooks + (packed ? r : kCcMaxRounds));
    if (packed) compress(hooks + r);
  }
  SST_LAUNCH_PDL(k_cc_link_kept, blocks_for(vs.count), kTB, 0, s, vs, t->qa.p, t->qb.p, rounds == 2,
                 par, hooks + kCcMaxRounds, err);
  if (few)
    SST_LAUNCH_PDL(k_cc_compress, blocks_for(n), kTB, 0, s, par, n, none);
  else
    compress(hooks + kCcMaxRounds);
  SST_LAUNCH_PDL(k_cc_giant, 1, 1024, 0, s, par, n, giant);
  if (t->nsmall)
    SST_LAUNCH_PDL(k_cc_rest_small, blocks_for(t->nsmall), kTB, 0, s, dg, t->sdesc.p,
               t->small.p, t->nsmall, giant, par, err);
  if (t->nchunks)
    SST_LAUNCH_PDL(k_cc_rest_chunks, warp_blocks(t->nchunks), kTB, 0, s, dg, t->cdesc.p,
               t->cv.p, t->nchunks, giant, par, err);
  SST_LAUNCH_PDL(k_cc_compress, blocks_for(n), kTB, 0, s, par, n, none);
  SST_CUDA_TRY(cudaMemcpyAsync(t->h_small, t->d_small, 16, cudaMemcpyDeviceToHost, s));
  SST_CUDA_TRY(cudaStreamSynchronize(s));
  SST_CUDA_TRY(cudaGetLastError());
  if (t->h_small[1]) {
    set_error_message("connected components: %llu links gave up",
                      (unsigned long long)t->h_small[1]);
    return SST_ETIMEDOUT;
  }
  return SST_OK;
}

sst_status bc(sst_graph *g, uint32_t src, double *d_dep) {
  BfsArgs a;
  unsigned grid = 1;
  sst_status st = bfs_setup(g, src, nullptr, nullptr,
                            reinterpret_cast<const void *>(k_bc_levels), &a, &grid);
  if (st != SST_OK) return st;
  TravState *t = g->trav;
  const uint64_t n = g->n;
  for (DevBuf<double> *buf : {&t->sigma, &t->ratio}) {
    if (buf->cap >= 2 * n) continue;
    SST_CUDA_TRY(buf->exact(2 * n));
    SST_CUDA_TRY(cudaMemsetAsync(buf->p, 0, 16 * n, g->stream));
  }
  SST_CUDA_TRY(t->levels.exact(n + 1));
  SST_CUDA_TRY(t->qb.ensure(t->nbig + 1));
  // a hub's chunks of kBcLeaves leaves are at most its chunks in the lists
  const uint64_t hubs = t->nchunks + 1;
  SST_CUDA_TRY(t->hub.ensure(2 * hubs));
  SST_CUDA_TRY(t->hub_done.ensure(hubs));
  SST_CUDA_TRY(t->partial.ensure(hubs));
  const BcArgs b{t->sigma.p,    t->ratio.p,        d_dep,        t->big.p,
                 t->nbig,       hubs,              t->hub.p,     t->hub.p + hubs,
                 t->partial.p,  t->hub_done.p,     t->qb.p,
                 reinterpret_cast<BcCtl *>(a.ctl + 1),
                 bc_few(t->nsmall + t->nbig, n),   t->levels.p};
  SST_CUDA_TRY(launch_coop("k_bc_levels", k_bc_levels, grid, kCoopThreads, g->stream, a, b));
  return bfs_finish(g, "BC");
}

sst_status tc(sst_graph *g, uint64_t *total, uint64_t *d_pv) {
  sst_status st = ensure_leaf_dir(g);
  if (st != SST_OK) return st;
  TravState *t = nullptr;
  st = state(g, &t);
  if (st != SST_OK) return st;
  cudaStream_t s = g->stream;
  uint32_t n = g->n;
  LeafDir &D = g->dir;
  uint64_t nl = D.nleaves;
  SST_CUDA_TRY(t->tlcnt.ensure(nl + 1));
  SST_CUDA_TRY(t->tlpre.ensure(nl + 1));
  SST_CUDA_TRY(t->tmask.ensure(nl + 1));
  SST_CUDA_TRY(t->toff.exact((uint64_t)n + 1));
  g->arena.reset();
  SST_CUDA_TRY(g->arena.reserve(scan_scratch_bytes(nl + 1, 8) + 4096));
  const uint64_t tc_warps = (nl + kTcLeaves - 1) / kTcLeaves;
  if (nl)
    SST_LAUNCH(k_tc_leafcount, warp_blocks(tc_warps), kTB, 0, s, g->d_slots, D.owner,
               D.slot, D.cnt, nl, g->d_deg, t->tlcnt.p, t->tmask.p);
  SST_CUDA_TRY((scan<uint64_t, OpAdd>(t->tlcnt.p, t->tlpre.p, nl, 0ull, OpAdd{},
                                      true, false, t->tlpre.p + nl, g->arena, s)));
  const TcLeaves leaves{g->d_slots, D.owner, D.cnt, D.slot, nl};
  // few items: by rows; rows of four ids on average: by lists; else by a sample
  const bool few = tc_few_items(nl), sample = !few && g->m > 4 * nl;
  SST_CUDA_TRY(cudaMemsetAsync(t->d_small, 0, 16, s));  // count, work cursor
  if (n) SST_LAUNCH(k_tc_lists, blocks_for(n), kTB, 0, s, D.vleaf, t->tlpre.p, n, t->toff.p);
  uint64_t madj = 0;
  if (!sample) {
    SST_CUDA_TRY(cudaMemcpyAsync(&madj, t->tlpre.p + nl, 8, cudaMemcpyDeviceToHost, s));
  } else {
    static_assert(2 + kTcSampleWords <= (int)kTravWords, "the estimates fit the traversal words");
    tc_sample_launch(TcKeptLeaves{g->d_slots, D.owner, D.slot, t->tmask.p, nl}, t->toff.p,
                     d_pv != nullptr, t->tlpre.p + nl, t->d_small + 2, s);
    SST_CUDA_TRY(cudaMemcpyAsync(t->h_small, t->d_small + 2, kTcSampleWords * 8,
                                 cudaMemcpyDeviceToHost, s));
  }
  SST_CUDA_TRY(cudaStreamSynchronize(s));
  if (sample) madj = t->h_small[kTcSampleWords - 1];
  SST_CUDA_TRY(t->tadj.ensure(madj + 1));
  if (nl)
    SST_LAUNCH(k_tc_fill, warp_blocks(tc_warps), kTB, 0, s, g->d_slots, D.slot, nl,
               t->tmask.p, t->tlpre.p, t->tadj.p);
  if (d_pv) SST_CUDA_TRY(cudaMemsetAsync(d_pv, 0, (uint64_t)n * 8, s));
  unsigned long long *const pv = reinterpret_cast<unsigned long long *>(d_pv);
  // (more batches of the lists than 32 bits count: by rows)
  const bool by_rows = few || tc_items_bound(n, madj) >> 32 || (sample && tc_by_rows(t->h_small));
  if (nl && by_rows) {
    SST_CUDA_TRY(tc_count_launch(leaves, t->toff.p, t->tadj.p, t->d_small, pv, g->sms, s));
  } else if (nl) {
    SST_CUDA_TRY(t->icnt.exact((uint64_t)n + 1));
    SST_CUDA_TRY(t->ioff.exact((uint64_t)n + 1));
    SST_CUDA_TRY(t->titems.ensure(tc_items_bound(n, madj)));
    g->arena.reset();
    SST_CUDA_TRY(g->arena.reserve(scan_scratch_bytes((uint64_t)n + 1, 4) + 4096));
    TcLists lists;
    SST_CUDA_TRY(tc_list_items(t->toff.p, t->tadj.p, n, madj, t->icnt.p, t->ioff.p, t->titems.p,
                               g->arena, s, &lists));
    SST_CUDA_TRY(tc_count_launch(lists, t->toff.p, t->tadj.p, t->d_small, pv, g->sms, s));
  }
  SST_CUDA_TRY(cudaMemcpyAsync(t->h_small, t->d_small, 8, cudaMemcpyDeviceToHost, s));
  SST_CUDA_TRY(cudaStreamSynchronize(s));
  SST_CUDA_TRY(cudaGetLastError());
  *total = t->h_small[0];
  return SST_OK;
}

sst_status common_neighbors_batch(sst_graph *g, const uint32_t *d_pairs,
                                  uint64_t n, bool early_end, uint64_t *d_out) {
  if (n == 0) return SST_OK;
  // pairs of a block: few, so that a small call spreads over every cluster that fits
  // at once (two blocks to an SM); beyond 80, 64 of them, so that a block has few long
  // rows, or as many as make two and a half rounds of blocks (100,000 edges at RMAT
  // scale 18 by 64, 132, 256 and 512: 553, 577, 686 and 763 us; pairs of short rows
  // 50, 36, 33 and 34); at most kCommonPairs
  const uint64_t slots = std::max(1, 2 * g->sms / kCommonCtas) * (uint64_t)kCommonCtas;
  const uint64_t one = (n + slots - 1) / slots, rounds = (2 * n + 5 * slots - 1) / (5 * slots);
  const uint64_t want = one <= 80 ? one : std::max<uint64_t>(64, rounds);
  const uint32_t per = (uint32_t)std::min<uint64_t>(want, kCommonPairs);
  const uint64_t per_cluster = (uint64_t)per * kCommonCtas;
  SST_LAUNCH(k_common, (unsigned)((n + per_cluster - 1) / per_cluster) * kCommonCtas,
             kCommonThreads, 0, g->stream, g->view(), d_pairs, n, per,
             one <= 160 ? kCommonMerged : kCommonMergedOfMany, early_end,
             reinterpret_cast<unsigned long long *>(d_out));
  SST_CUDA_TRY(cudaGetLastError());
  return SST_OK;
}


// ================================================ multi-source BFS and BC
// Multi-source BFS: k <= 64 sources traverse together.  Each vertex holds a
// mask of the sources that have reached it (vis) and of those for which it
// is on the current level (fr); one level is one pass for all sources -- a
// push from the frontier queue while the frontier's edges are few, else a
// pull over all unfinished vertices -- followed by one update pass that
// turns the collected masks into new depths and the next queue.
namespace {

__global__ void k_msbfs_seed(const uint32_t *__restrict__ sv,
                             const unsigned long long *__restrict__ sm,
                             uint32_t cnt, uint32_t n,
                             unsigned long long *__restrict__ vis,
                             unsigned long long *__restrict__ fr,
                             int32_t *__restrict__ depth,
                             const uint32_t *__restrict__ deg,
                             const uint32_t *__restrict__ cap,
                             uint32_t *__restrict__ q,
                             unsigned long long *__restrict__ qc) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= cnt) return;
  uint32_t v = sv[i];
  unsigned long long m = sm[i];
  vis[v] = m;
  fr[v] = m;
  for (unsigned long long b = m; b; b &= b - 1)
    depth[(uint64_t)(__ffsll((long long)b) - 1) * n + v] = 0;
  q[i] = v;
  atomicAdd(&qc[1], (unsigned long long)deg[v]);
  atomicAdd(&qc[2], (unsigned long long)items_of(cap[v]));
}

// push: warp per work item (a frontier vertex's leaf chunk), lane = slot
__global__ void __launch_bounds__(kTB, 8)
k_msbfs_push(DGraph g, const uint32_t *__restrict__ iv,
             const uint32_t *__restrict__ il0, uint32_t nitems,
             const unsigned long long *__restrict__ fr,
             const unsigned long long *__restrict__ vis,
             unsigned long long *__restrict__ nx) {
  uint64_t i = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (i >= nitems) return;
  uint32_t u = iv[i];
  const unsigned long long f = fr[u];
  uint64_t base = g.base[u];
  uint32_t cap = g.cap[u], deg = g.deg[u];
  uint32_t nl = cap ? nleaves_of(cap) : 0;
  uint32_t l0 = il0[i], l1 = min(l0 + kPushLeaves, nl);
  // four leaves' slots and visited masks in flight at once; leaves keep
  // their ids packed left with EMPTY after them
  constexpr int kBatch = 4;
  const uint32_t lim = cap <= kLeaf ? deg : kLeaf;
  for (uint32_t l = l0; l < l1; l += kBatch) {
    uint32_t w[kBatch];
#pragma unroll
    for (int k = 0; k < kBatch; k++)
      w[k] = (l + k < l1 && (uint32_t)lane < lim)
                 ? g.slots[base + ((uint64_t)(l + k) << kLeafLog) + lane]
                 : kEmpty;
    unsigned long long add[kBatch];
#pragma unroll
    for (int k = 0; k < kBatch; k++) add[k] = w[k] != kEmpty ? f & ~vis[w[k]] : 0ull;
#pragma unroll
    for (int k = 0; k < kBatch; k++)
      if (add[k]) atomicOr(&nx[w[k]], add[k]);
  }
}

// pull, one-leaf vertices: thread per vertex, stops once every source that
// has not reached v is seen in the frontier
__global__ void k_msbfs_pull_small(DGraph g, const uint32_t *__restrict__ small,
                                   uint64_t nsmall,
                                   const unsigned long long *__restrict__ fr,
                                   const unsigned long long *__restrict__ vis,
                                   unsigned long long *__restrict__ nx,
                                   unsigned long long full) {
  uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nsmall) return;
  uint32_t v = small[i];
  const unsigned long long need = full & ~vis[v];
  if (!need) return;
  const uint32_t *p = g.slots + g.base[v];
  uint32_t d = g.deg[v];
  unsigned long long acc = 0;
  // four neighbours' ids, then their four masks, in flight per step
  for (uint32_t k = 0; k < d; k += 4) {
    uint32_t w[4];
#pragma unroll
    for (int q = 0; q < 4; q++) w[q] = k + q < d ? p[k + q] : kEmpty;
#pragma unroll
    for (int q = 0; q < 4; q++)
      if (w[q] != kEmpty) acc |= fr[w[q]];
    if ((acc & need) == need) break;
  }
  acc &= need;
  if (acc) nx[v] = acc;
}

__device__ __forceinline__ unsigned long long warp_or64(unsigned long long x) {
  unsigned lo = __reduce_or_sync(0xffffffffu, (unsigned)x);
  unsigned hi = __reduce_or_sync(0xffffffffu, (unsigned)(x >> 32));
  return ((unsigned long long)hi << 32) | lo;
}

// pull, multi-leaf vertices: warp per chunk (lane = slot), early exit
__global__ void k_msbfs_pull_chunks(DGraph g,
                                    const unsigned long long *__restrict__ cdesc,
                                    const uint32_t *__restrict__ cv,
                                    uint64_t nchunks,
                                    const unsigned long long *__restrict__ fr,
                                    const unsigned long long *__restrict__ vis,
                                    unsigned long long *__restrict__ nx,
                                    unsigned long long full) {
  uint64_t c = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (c >= nchunks) return;
  const uint32_t v = cv[c];
  const unsigned long long need = full & ~vis[v];
  if (!need) return;
  const unsigned long long dsc = cdesc[c];
  const uint64_t leaf0 = dsc >> 8;
  const uint32_t l1 = (uint32_t)(dsc & 63);
  const bool single = (dsc >> 7) & 1;
  const uint32_t mycnt = (uint32_t)lane < l1 ? g.lcnt[leaf0 + lane] : 0u;
  const uint32_t *sl = g.slots + (leaf0 << kLeafLog) + lane;
  unsigned long long acc = 0;
  for (uint32_t l = 0; l < l1; l += 4) {
#pragma unroll
    for (int q = 0; q < 4; q++) {
      uint32_t cq = __shfl_sync(0xffffffffu, mycnt, (l + q) & 31);
      if (l + q >= l1) cq = 0;
      if ((uint32_t)lane < cq) acc |= fr[sl[(uint64_t)(l + q) << kLeafLog]];
    }
    if ((warp_or64(acc) & need) == need) break;
  }
  acc = warp_or64(acc) & need;
  if (lane == 0 && acc) {
    if (single)
      nx[v] = acc;
    else
      atomicOr(&nx[v], acc);
  }
}

// new sources per vertex -> depths, next frontier masks and queue
__global__ void k_msbfs_update(uint32_t n, unsigned long long *__restrict__ vis,
                               unsigned long long *__restrict__ nx,
                               unsigned long long *__restrict__ fr_next,
                               int32_t *__restrict__ depth, int32_t lvl,
                               const uint32_t *__restrict__ deg,
                               const uint32_t *__restrict__ cap,
                               uint32_t *__restrict__ q,
                               unsigned long long *__restrict__ qc) {
  uint32_t v = blockIdx.x * blockDim.x + threadIdx.x;
  unsigned long long nw = 0;
  if (v < n) {
    unsigned long long x = nx[v];
    if (x) {
      nx[v] = 0;
      unsigned long long old = vis[v];
      nw = x & ~old;
      if (nw) {
        vis[v] = old | nw;
        for (unsigned long long b = nw; b; b &= b - 1)
          depth[(uint64_t)(__ffsll((long long)b) - 1) * n + v] = lvl;
      }
    }
    fr_next[v] = nw;
  }
  enqueue_block(nw != 0, v, nw ? deg[v] : 0u, nw ? items_of(cap[v]) : 0u, q, qc);
}

// ---- multi-source BC: the single-source passes with the source on
// blockIdx.y; per (source, level) the list start, list count, item start and
// item count come from tab[(s * L + d) * 4 + 0..3]
__global__ void k_msbc_maxdepth(const int32_t *__restrict__ depth, uint32_t n,
                                unsigned long long *__restrict__ out) {
  uint32_t v = blockIdx.x * blockDim.x + threadIdx.x;
  block_max_to(v < n ? depth[(uint64_t)blockIdx.y * n + v] : -1, out);
}

__global__ void k_msbc_level_count(const int32_t *__restrict__ depth, uint32_t n,
                                   uint32_t L, uint32_t *__restrict__ cnt) {
  uint32_t v = blockIdx.x * blockDim.x + threadIdx.x;
  const int32_t d = v < n ? depth[(uint64_t)blockIdx.y * n + v] : -1;
  level_add(cnt + blockIdx.y * L + (d >= 0 ? d : 0), d, d >= 0);
}

__global__ void k_msbc_level_scatter(const int32_t *__restrict__ depth,
                                     uint32_t n, uint32_t L,
                                     const uint32_t *__restrict__ start,
                                     uint32_t *__restrict__ ctr,
                                     uint32_t *__restrict__ list) {
  uint32_t v = blockIdx.x * blockDim.x + threadIdx.x;
  const int32_t d = v < n ? depth[(uint64_t)blockIdx.y * n + v] : -1;
  const uint32_t a = blockIdx.y * L + (d >= 0 ? d : 0);
  const uint32_t at = level_add(ctr + a, d, d >= 0);
  if (d >= 0) list[start[a] + at] = v;
}

__global__ void k_msbc_init(const uint32_t *__restrict__ srcs, uint32_t n,
                            double *__restrict__ sigma, double *__restrict__ ratio,
                            double *__restrict__ dep) {
  uint32_t v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= n) return;
  uint64_t at = (uint64_t)blockIdx.y * n + v;
  sigma[at] = v == srcs[blockIdx.y] ? 1.0 : 0.0;
  ratio[at] = 0.0;
  dep[at] = 0.0;
}

__global__ void k_msbc_sigma_small(DGraph g, const uint32_t *__restrict__ list,
                                   const uint32_t *__restrict__ tab, uint32_t L,
                                   int32_t d, const int32_t *__restrict__ depth,
                                   double *__restrict__ sigma) {
  const uint32_t *e = tab + ((uint64_t)blockIdx.y * L + d) * 4;
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= e[1]) return;
  uint32_t v = list[e[0] + i];
  if (g.cap[v] > kLeaf) return;
  const uint64_t so = (uint64_t)blockIdx.y * g.n;
  const uint32_t *p = g.slots + g.base[v];
  uint32_t dg = g.deg[v];
  double acc = 0.0;
  // neighbours in order, kBcAhead in flight
  for (uint32_t k0 = 0; k0 < dg; k0 += kBcAhead) {
    uint32_t u[kBcAhead];
    bool on[kBcAhead];
#pragma unroll
    for (int q = 0; q < kBcAhead; q++) u[q] = k0 + q < dg ? p[k0 + q] : 0u;
#pragma unroll
    for (int q = 0; q < kBcAhead; q++) on[q] = k0 + q < dg && depth[so + u[q]] == d - 1;
    double x[kBcAhead];
#pragma unroll
    for (int q = 0; q < kBcAhead; q++) x[q] = on[q] ? sigma[so + u[q]] : 0.0;
#pragma unroll
    for (int q = 0; q < kBcAhead; q++)
      if (on[q]) acc += x[q];
  }
  sigma[so + v] = acc;
}

__global__ void k_msbc_chunks(DGraph g, const uint32_t *__restrict__ iv,
                              const uint32_t *__restrict__ il0,
                              const uint32_t *__restrict__ tab, uint32_t L,
                              int32_t d, const int32_t *__restrict__ depth,
                              const double *__restrict__ val, int32_t want,
                              double *__restrict__ partial) {
  const uint32_t *e = tab + ((uint64_t)blockIdx.y * L + d) * 4;
  uint64_t i = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (i >= e[3]) return;
  i += e[2];
  const uint64_t so = (uint64_t)blockIdx.y * g.n;
  uint32_t v = iv[i];
  uint32_t nl = g.cap[v] >> kLeafLog;
  uint32_t l0 = il0[i], l1 = min(l0 + kChunkLeaves, nl);
  uint64_t base = g.base[v];
  // eight leaves' slots, depths and values in flight at once (the leaves of
  // a multi-leaf segment keep their ids packed left with EMPTY after them);
  // each lane still adds in leaf order
  constexpr int kBatch = 8;
  double acc = 0.0;
  for (uint32_t l = l0; l < l1; l += kBatch) {
    uint32_t u[kBatch];
#pragma unroll
    for (int k = 0; k < kBatch; k++)
      u[k] = l + k < l1 ? g.slots[base + ((uint64_t)(l + k) << kLeafLog) + lane] : kEmpty;
    bool on[kBatch];
#pragma unroll
    for (int k = 0; k < kBatch; k++) on[k] = u[k] != kEmpty && depth[so + u[k]] == want;
    double x[kBatch];
#pragma unroll
    for (int k = 0; k < kBatch; k++) x[k] = on[k] ? val[so + u[k]] : 0.0;
#pragma unroll
    for (int k = 0; k < kBatch; k++)
      if (on[k]) acc += x[k];
  }
  double sum = warp_sum_d(acc);
  if (lane == 0) partial[i] = sum;
}

__global__ void k_msbc_fix(DGraph g, const uint32_t *__restrict__ list,
                           const uint32_t *__restrict__ tab, uint32_t L,
                           int32_t d, const uint32_t *__restrict__ cnt,
                           const uint32_t *__restrict__ off,
                           const double *__restrict__ partial, bool sigma_pass,
                           double *__restrict__ sigma, double *__restrict__ ratio,
                           double *__restrict__ dep) {
  const uint32_t *e = tab + ((uint64_t)blockIdx.y * L + d) * 4;
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= e[1]) return;
  uint32_t p = e[0] + i;
  uint32_t k = cnt[p];
  if (k == 0) return;
  double acc = 0.0;
  for (uint32_t j = 0; j < k; j++) acc += partial[off[p] + j];
  const uint64_t at = (uint64_t)blockIdx.y * g.n + list[p];
  if (sigma_pass) {
    sigma[at] = acc;
  } else {
    double dv = sigma[at] * acc;
    dep[at] = dv;
    ratio[at] = (1.0 + dv) / sigma[at];
  }
}

__global__ void k_msbc_delta_small(DGraph g, const uint32_t *__restrict__ list,
                                   const uint32_t *__restrict__ tab, uint32_t L,
                                   int32_t d, const int32_t *__restrict__ depth,
                                   const double *__restrict__ sigma,
                                   double *__restrict__ ratio,
                                   double *__restrict__ dep) {
  const uint32_t *e = tab + ((uint64_t)blockIdx.y * L + d) * 4;
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= e[1]) return;
  uint32_t v = list[e[0] + i];
  if (g.cap[v] > kLeaf) return;
  const uint64_t so = (uint64_t)blockIdx.y * g.n;
  const uint32_t *p = g.slots + g.base[v];
  uint32_t dg = g.deg[v];
  double acc = 0.0;
  // neighbours in order, kBcAhead in flight
  for (uint32_t k0 = 0; k0 < dg; k0 += kBcAhead) {
    uint32_t w[kBcAhead];
    bool on[kBcAhead];
#pragma unroll
    for (int q = 0; q < kBcAhead; q++) w[q] = k0 + q < dg ? p[k0 + q] : 0u;
#pragma unroll
    for (int q = 0; q < kBcAhead; q++) on[q] = k0 + q < dg && depth[so + w[q]] == d + 1;
    double x[kBcAhead];
#pragma unroll
    for (int q = 0; q < kBcAhead; q++) x[q] = on[q] ? ratio[so + w[q]] : 0.0;
#pragma unroll
    for (int q = 0; q < kBcAhead; q++)
      if (on[q]) acc += x[q];
  }
  double dv = sigma[so + v] * acc;
  dep[so + v] = dv;
  ratio[so + v] = (1.0 + dv) / sigma[so + v];
}

}  // namespace

sst_status bfs_multi(sst_graph *g, const uint32_t *h_srcs, uint32_t k,
                     int32_t *d_depth) {
  if (k == 0) return SST_OK;
  if (k > 64) {
    set_error_message("at most 64 sources per multi-source BFS");
    return SST_EINVAL;
  }
  sst_status st = ensure_lists(g);
  if (st != SST_OK) return st;
  TravState *t = g->trav;
  cudaStream_t s = g->stream;
  const uint32_t n = g->n;
  // distinct sources with their source masks
  std::vector<uint32_t> sv;
  std::vector<unsigned long long> sm;
  for (uint32_t i = 0; i < k; i++) {
    if (h_srcs[i] >= n) {
      set_error_message("source %u out of range", h_srcs[i]);
      return SST_EINVAL;
    }
    auto it = std::find(sv.begin(), sv.end(), h_srcs[i]);
    if (it == sv.end()) {
      sv.push_back(h_srcs[i]);
      sm.push_back(1ull << i);
    } else {
      sm[it - sv.begin()] |= 1ull << i;
    }
  }
  const unsigned long long full = k == 64 ? ~0ull : (1ull << k) - 1;
  SST_CUDA_TRY(t->mvis.exact(n));
  SST_CUDA_TRY(t->mfr.exact(n));
  SST_CUDA_TRY(t->mfr2.exact(n));
  SST_CUDA_TRY(t->mnx.exact(n));
  SST_CUDA_TRY(t->qa.exact((uint64_t)n + 1));
  SST_CUDA_TRY(t->qb.exact((uint64_t)n + 1));
  SST_CUDA_TRY(t->icnt.exact((uint64_t)n + 1));
  SST_CUDA_TRY(t->ioff.exact((uint64_t)n + 1));
  SST_CUDA_TRY(t->msrc.ensure(2 * (uint64_t)sv.size()));
  SST_CUDA_TRY(cudaMemsetAsync(t->mvis.p, 0, (uint64_t)n * 8, s));
  SST_CUDA_TRY(cudaMemsetAsync(t->mfr.p, 0, (uint64_t)n * 8, s));
  SST_CUDA_TRY(cudaMemsetAsync(t->mnx.p, 0, (uint64_t)n * 8, s));
  SST_CUDA_TRY(cudaMemsetAsync(d_depth, 0xFF, (uint64_t)k * n * 4, s));
  unsigned long long *d_sm = t->msrc.p;
  uint32_t *d_sv = reinterpret_cast<uint32_t *>(t->msrc.p + sv.size());
  SST_CUDA_TRY(cudaMemcpyAsync(d_sv, sv.data(), sv.size() * 4, cudaMemcpyHostToDevice, s));
  SST_CUDA_TRY(cudaMemcpyAsync(d_sm, sm.data(), sm.size() * 8, cudaMemcpyHostToDevice, s));
  unsigned long long *qc = t->d_small;
  SST_CUDA_TRY(cudaMemsetAsync(qc, 0, 24, s));
  uint32_t *q = t->qa.p, *nq = t->qb.p;
  unsigned long long *fr = t->mfr.p, *fr2 = t->mfr2.p;
  SST_LAUNCH(k_msbfs_seed, blocks_for(sv.size()), kTB, 0, s, d_sv, d_sm,
             (uint32_t)sv.size(), n, t->mvis.p, fr, d_depth, g->d_deg, g->d_cap,
             q, qc);
  SST_CUDA_TRY(cudaMemcpyAsync(t->h_small, qc, 24, cudaMemcpyDeviceToHost, s));
  SST_CUDA_TRY(cudaStreamSynchronize(s));
  uint64_t qn = sv.size(), qdeg = t->h_small[1], qitems = t->h_small[2];
  const uint64_t m = g->m;
  DGraph dg = g->view();
  g->arena.reset();
  SST_CUDA_TRY(g->arena.reserve(scan_scratch_bytes((uint64_t)n + 1, 4) + 4096));
  for (int32_t lvl = 0; qn > 0; lvl++) {
    if ((uint64_t)lvl > n) {
      set_error_message("multi-source BFS exceeded n levels");
      return SST_ETIMEDOUT;
    }
    if ((qn + qdeg) * t->bfs_alpha > m) {
      if (t->nsmall)
        SST_LAUNCH(k_msbfs_pull_small, blocks_for(t->nsmall), kTB, 0, s, dg,
                   t->small.p, t->nsmall, fr, t->mvis.p, t->mnx.p, full);
      if (t->nchunks)
        SST_LAUNCH(k_msbfs_pull_chunks, warp_blocks(t->nchunks), kTB, 0, s, dg,
                   t->cdesc.p, t->cv.p, t->nchunks, fr, t->mvis.p, t->mnx.p, full);
    } else {
      SST_CUDA_TRY(t->iv.ensure(qitems + 1));
      SST_CUDA_TRY(t->il0.ensure(qitems + 1));
      SST_LAUNCH(k_front_items, blocks_for(qn), kTB, 0, s, q, (uint32_t)qn,
                 g->d_cap, t->icnt.p);
      g->arena.reset();
      SST_CUDA_TRY((scan<uint32_t, OpAdd>(t->icnt.p, t->ioff.p, qn, 0u, OpAdd{},
                                          true, false, nullptr, g->arena, s)));
      SST_LAUNCH(k_front_expand, blocks_for(qn), kTB, 0, s, q, (uint32_t)qn,
                 g->d_cap, t->ioff.p, t->iv.p, t->il0.p);
      SST_LAUNCH(k_msbfs_push, warp_blocks(qitems), kTB, 0, s, dg, t->iv.p,
                 t->il0.p, (uint32_t)qitems, fr, t->mvis.p, t->mnx.p);
    }
    SST_CUDA_TRY(cudaMemsetAsync(qc, 0, 24, s));
    SST_LAUNCH(k_msbfs_update, blocks_for(n), kTB, 0, s, n, t->mvis.p, t->mnx.p,
               fr2, d_depth, lvl + 1, g->d_deg, g->d_cap, nq, qc);
    SST_CUDA_TRY(cudaMemcpyAsync(t->h_small, qc, 24, cudaMemcpyDeviceToHost, s));
    SST_CUDA_TRY(cudaStreamSynchronize(s));
    qn = t->h_small[0];
    qdeg = t->h_small[1];
    qitems = t->h_small[2];
    std::swap(q, nq);
    std::swap(fr, fr2);
  }
  SST_CUDA_TRY(cudaGetLastError());
  return SST_OK;
}

sst_status bc_multi(sst_graph *g, const uint32_t *h_srcs, uint32_t k,
                    double *d_dep) {
  if (k == 0) return SST_OK;
  TravState *t = nullptr;
  sst_status st = state(g, &t);
  if (st != SST_OK) return st;
  const uint32_t n = g->n;
  SST_CUDA_TRY(t->mdepth.ensure((uint64_t)k * n));
  st = bfs_multi(g, h_srcs, k, t->mdepth.p);
  if (st != SST_OK) return st;
  cudaStream_t s = g->stream;
  const int32_t *depth = t->mdepth.p;
  const dim3 vgrid(blocks_for(n), k);
  SST_CUDA_TRY(cudaMemsetAsync(t->d_small, 0, 8, s));
  SST_LAUNCH(k_msbc_maxdepth, vgrid, kTB, 0, s, depth, n, t->d_small);
  SST_CUDA_TRY(cudaMemcpyAsync(t->h_small, t->d_small, 8, cudaMemcpyDeviceToHost, s));
  SST_CUDA_TRY(cudaStreamSynchronize(s));
  const uint32_t D = (uint32_t)t->h_small[0];
  const uint32_t L = D + 2;  // levels 0..D plus an end marker
  // per (source, level): vertex counts -> list starts
  SST_CUDA_TRY(t->mtab.ensure((uint64_t)k * L * 7));
  uint32_t *cnt = t->mtab.p, *start = cnt + (uint64_t)k * L, *ctr = start + (uint64_t)k * L;
  uint32_t *tab = ctr + (uint64_t)k * L;  // k * L * 4 words
  SST_CUDA_TRY(cudaMemsetAsync(cnt, 0, (uint64_t)k * L * 4, s));
  SST_CUDA_TRY(cudaMemsetAsync(ctr, 0, (uint64_t)k * L * 4, s));
  SST_LAUNCH(k_msbc_level_count, vgrid, kTB, 0, s, depth, n, L, cnt);
  std::vector<uint32_t> hc((uint64_t)k * L), hs((uint64_t)k * L);
  SST_CUDA_TRY(cudaMemcpyAsync(hc.data(), cnt, hc.size() * 4, cudaMemcpyDeviceToHost, s));
  SST_CUDA_TRY(cudaStreamSynchronize(s));
  uint64_t acc = 0;
  for (uint64_t i = 0; i < hc.size(); i++) {
    hs[i] = (uint32_t)acc;
    acc += hc[i];
  }
  if (acc >= 0xFFFFFFFFull) {
    set_error_message("too many (source, vertex) pairs for one multi-source BC");
    return SST_EINVAL;
  }
  const uint32_t RR = (uint32_t)acc;
  SST_CUDA_TRY(cudaMemcpyAsync(start, hs.data(), hs.size() * 4, cudaMemcpyHostToDevice, s));
  SST_CUDA_TRY(t->mlist.ensure((uint64_t)RR + 1));
  SST_LAUNCH(k_msbc_level_scatter, vgrid, kTB, 0, s, depth, n, L, start, ctr,
             t->mlist.p);
  // leaf-chunk items of the multi-leaf vertices, in list order
  SST_CUDA_TRY(t->micnt.ensure((uint64_t)RR + 1));
  SST_CUDA_TRY(t->mioff.ensure((uint64_t)RR + 1));
  const uint32_t *list = t->mlist.p;
  if (RR) SST_LAUNCH(k_bc_item_counts, blocks_for(RR), kTB, 0, s, list, RR, g->d_cap, t->micnt.p);
  g->arena.reset();
  SST_CUDA_TRY(g->arena.reserve(scan_scratch_bytes((uint64_t)RR + 1, 4) + 4096));
  SST_CUDA_TRY((scan<uint32_t, OpAdd>(t->micnt.p, t->mioff.p, RR, 0u, OpAdd{},
                                      true, false, t->mioff.p + RR, g->arena, s)));
  // item starts at each (source, level) list start, and the total
  std::vector<uint32_t> hpos(hs.size() + 1);
  for (uint64_t i = 0; i < hs.size(); i++) hpos[i] = hs[i];
  hpos[hs.size()] = RR;
  SST_CUDA_TRY(cudaMemcpyAsync(ctr, hpos.data(), (uint64_t)k * L * 4, cudaMemcpyHostToDevice, s));
  std::vector<uint32_t> hib((uint64_t)k * L + 1);
  SST_CUDA_TRY(t->mpart.ensure((uint64_t)k * L + 2));
  uint32_t *d_ib = reinterpret_cast<uint32_t *>(t->mpart.p);
  SST_LAUNCH(k_gather_bounds, blocks_for((uint64_t)k * L), kTB, 0, s, t->mioff.p,
             ctr, (uint32_t)(k * L), d_ib);
  SST_CUDA_TRY(cudaMemcpyAsync(hib.data(), d_ib, (uint64_t)k * L * 4, cudaMemcpyDeviceToHost, s));
  uint32_t items = 0;
  SST_CUDA_TRY(cudaMemcpyAsync(&items, t->mioff.p + RR, 4, cudaMemcpyDeviceToHost, s));
  SST_CUDA_TRY(cudaStreamSynchronize(s));
  hib[(uint64_t)k * L] = items;
  // the table: list start, count, item start, item count per (source, level)
  std::vector<uint32_t> ht((uint64_t)k * L * 4);
  std::vector<uint32_t> maxc(L, 0), maxi(L, 0);
  for (uint32_t sidx = 0; sidx < k; sidx++)
    for (uint32_t d = 0; d < L; d++) {
      uint64_t at = (uint64_t)sidx * L + d;
      uint32_t i0 = hib[at], i1 = hib[at + 1];
      ht[at * 4 + 0] = hs[at];
      ht[at * 4 + 1] = hc[at];
      ht[at * 4 + 2] = i0;
      ht[at * 4 + 3] = i1 - i0;
      maxc[d] = std::max(maxc[d], hc[at]);
      maxi[d] = std::max(maxi[d], i1 - i0);
    }
  SST_CUDA_TRY(cudaMemcpyAsync(tab, ht.data(), ht.size() * 4, cudaMemcpyHostToDevice, s));
  SST_CUDA_TRY(t->miv.ensure((uint64_t)items + 1));
  SST_CUDA_TRY(t->mil0.ensure((uint64_t)items + 1));
  SST_CUDA_TRY(t->mpart.ensure((uint64_t)items + 1));
  if (items && RR)
    SST_LAUNCH(k_bc_expand, blocks_for(RR), kTB, 0, s, list, RR, t->micnt.p,
               t->mioff.p, t->miv.p, t->mil0.p);
  SST_CUDA_TRY(t->msig.ensure((uint64_t)k * n));
  SST_CUDA_TRY(t->mrat.ensure((uint64_t)k * n));
  // the sources, staged in the (now free) scatter counters
  SST_CUDA_TRY(cudaMemcpyAsync(ctr, h_srcs, (uint64_t)k * 4, cudaMemcpyHostToDevice, s));
  SST_LAUNCH(k_msbc_init, vgrid, kTB, 0, s, ctr, n, t->msig.p, t->mrat.p, d_dep);
  DGraph dg = g->view();
  double *part = t->mpart.p;
  for (uint32_t d = 1; d <= D; d++) {
    if (maxc[d])
      SST_LAUNCH(k_msbc_sigma_small, dim3(blocks_for(maxc[d]), k), kTB, 0, s, dg,
                 list, tab, L, (int32_t)d, depth, t->msig.p);
    if (maxi[d]) {
      SST_LAUNCH(k_msbc_chunks, dim3(warp_blocks(maxi[d]), k), kTB, 0, s, dg,
                 t->miv.p, t->mil0.p, tab, L, (int32_t)d, depth, t->msig.p,
                 (int32_t)d - 1, part);
      SST_LAUNCH(k_msbc_fix, dim3(blocks_for(maxc[d]), k), kTB, 0, s, dg, list,
                 tab, L, (int32_t)d, t->micnt.p, t->mioff.p, part, true,
                 t->msig.p, t->mrat.p, d_dep);
    }
  }
  for (int32_t d = (int32_t)D; d >= 0; d--) {
    if (maxc[d])
      SST_LAUNCH(k_msbc_delta_small, dim3(blocks_for(maxc[d]), k), kTB, 0, s, dg,
                 list, tab, L, d, depth, t->msig.p, t->mrat.p, d_dep);
    if (maxi[d]) {
      SST_LAUNCH(k_msbc_chunks, dim3(warp_blocks(maxi[d]), k), kTB, 0, s, dg,
                 t->miv.p, t->mil0.p, tab, L, d, depth, t->mrat.p, d + 1, part);
      SST_LAUNCH(k_msbc_fix, dim3(blocks_for(maxc[d]), k), kTB, 0, s, dg, list,
                 tab, L, d, t->micnt.p, t->mioff.p, part, false, t->msig.p,
                 t->mrat.p, d_dep);
    }
  }
  SST_CUDA_TRY(cudaGetLastError());
  return SST_OK;
}


// ------------------------------------------------------------- autotuner
// Times the traversal knobs on this graph and keeps the fastest: PageRank
// (3 iterations) over chunk sizes {8, 16, 32} x lanes {4, 8, 16}, then its
// shared-memory cache {0, 2048, 4096, 8192}, then BFS from three sources
// over push/pull thresholds {5, 10, 20, 40, 80}.
sst_status get_tuning(sst_graph *g, sst_tuning *out) {
  TravState *t = nullptr;
  sst_status st = state(g, &t);
  if (st != SST_OK) return st;
  out->chunk_leaves = t->chunk_leaves;
  out->pr_lanes = t->pr_lanes;
  out->bfs_alpha = t->bfs_alpha;
  out->pr_hot = t->pr_hot;
  out->pr_ms = 0.f;
  out->bfs_ms = 0.f;
  return SST_OK;
}

sst_status set_tuning(sst_graph *g, const sst_tuning *in) {
  if (in->chunk_leaves < 1 || in->chunk_leaves > 32 ||
      (in->pr_lanes != 4 && in->pr_lanes != 8 && in->pr_lanes != 16) ||
      in->bfs_alpha < 1 || in->pr_hot > 24576) {
    set_error_message("tuning out of range (chunk_leaves 1..32, pr_lanes 4/8/16, "
                      "bfs_alpha >= 1, pr_hot <= 24576)");
    return SST_EINVAL;
  }
  TravState *t = nullptr;
  sst_status st = state(g, &t);
  if (st != SST_OK) return st;
  t->chunk_leaves = in->chunk_leaves;
  t->pr_lanes = in->pr_lanes;
  t->bfs_alpha = in->bfs_alpha;
  t->pr_hot = in->pr_hot;
  return SST_OK;
}

sst_status autotune(sst_graph *g, sst_tuning *out) {
  TravState *t = nullptr;
  sst_status st = state(g, &t);
  if (st != SST_OK) return st;
  const uint32_t n = g->n;
  st = get_tuning(g, out);
  if (st != SST_OK || n == 0 || g->m == 0) return st;
  cudaStream_t s = g->stream;
  double *rank = nullptr;
  int32_t *dep = nullptr;
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  SST_CUDA_TRY(cudaMalloc(&rank, (uint64_t)n * 8));
  SST_CUDA_TRY(cudaMalloc(&dep, (uint64_t)n * 4));
  SST_CUDA_TRY(cudaEventCreate(&e0));
  SST_CUDA_TRY(cudaEventCreate(&e1));
  float best_pr = 1e30f, best_bfs = 1e30f;
  uint32_t bcl = t->chunk_leaves, blanes = t->pr_lanes, balpha = t->bfs_alpha;
  auto timed = [&](auto fn, float *ms) -> sst_status {
    sst_status r = fn();  // warm (lists, captured graph)
    if (r != SST_OK) return r;
    SST_CUDA_TRY(cudaEventRecord(e0, s));
    r = fn();
    if (r != SST_OK) return r;
    SST_CUDA_TRY(cudaEventRecord(e1, s));
    SST_CUDA_TRY(cudaEventSynchronize(e1));
    SST_CUDA_TRY(cudaEventElapsedTime(ms, e0, e1));
    return SST_OK;
  };
  const uint32_t cls[3] = {8, 16, 32}, lanes[3] = {4, 8, 16};
  for (uint32_t a = 0; a < 3 && st == SST_OK; a++)
    for (uint32_t b = 0; b < 3 && st == SST_OK; b++) {
      t->chunk_leaves = cls[a];
      t->pr_lanes = lanes[b];
      float ms = 0.f;
      st = timed([&] { return pagerank(g, 3, 0.85, rank); }, &ms);
      if (st == SST_OK && ms < best_pr) {
        best_pr = ms;
        bcl = cls[a];
        blanes = lanes[b];
      }
    }
  t->chunk_leaves = bcl;
  t->pr_lanes = blanes;
  // then the shared-memory cache of the lowest ids (pays on degree-ordered
  // graphs)
  uint32_t bhot = 0;
  const uint32_t hots[5] = {2048, 4096, 8192, 16384, 24576};
  for (uint32_t a = 0; a < 5 && st == SST_OK; a++) {
    t->pr_hot = hots[a];
    float ms = 0.f;
    st = timed([&] { return pagerank(g, 3, 0.85, rank); }, &ms);
    if (st == SST_OK && ms < best_pr) {
      best_pr = ms;
      bhot = hots[a];
    }
  }
  t->pr_hot = bhot;
  // BFS sources: the first three vertices with edges along a fixed stride
  std::vector<uint32_t> deg(n), src;
  if (st == SST_OK) {
    SST_CUDA_TRY(cudaMemcpy(deg.data(), g->d_deg, (uint64_t)n * 4, cudaMemcpyDeviceToHost));
    for (uint64_t i = 0; i < n && src.size() < 3; i++) {
      uint32_t v = (uint32_t)((i * 2654435761ull) % n);
      if (deg[v]) src.push_back(v);
    }
  }
  const uint32_t alphas[5] = {5, 10, 20, 40, 80};
  for (uint32_t a = 0; a < 5 && st == SST_OK && !src.empty(); a++) {
    t->bfs_alpha = alphas[a];
    float tot = 0.f;
    for (uint32_t v : src) {
      float ms = 0.f;
      st = timed([&] { return bfs(g, v, nullptr, dep); }, &ms);
      if (st != SST_OK) break;
      tot += ms;
    }
    if (st == SST_OK && tot < best_bfs) {
      best_bfs = tot;
      balpha = alphas[a];
    }
  }
  t->bfs_alpha = balpha;
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaFree(rank);
  cudaFree(dep);
  if (st != SST_OK) return st;
  get_tuning(g, out);
  out->pr_ms = best_pr;
  out->bfs_ms = src.empty() ? 0.f : best_bfs / (float)src.size();
  return SST_OK;
}


// ------------------------------------------------------------- bellman-ford
// Single-source shortest paths over a weighted graph (edge values as
// lengths): the reference drivers' BF(g, src) (internal/test.hpp:611-634;
// the algorithm library itself is absent).  Rounds of push relaxation from
// the vertices whose distance dropped in the previous round: a warp per
// frontier chunk (lane = slot) lowers dist[v] to dist[u] + w(u, v) by
// atomicMin on 64-bit distances, and the first thread to stamp v with the
// round enqueues it.  Lengths are unsigned, so no round count exceeds n.
namespace {
constexpr unsigned long long kInfDist = ~0ull;

__global__ void k_bf_init(unsigned long long *__restrict__ dist,
                          uint32_t *__restrict__ stamp, uint32_t n, uint32_t src) {
  uint32_t v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= n) return;
  dist[v] = v == src ? 0ull : kInfDist;
  stamp[v] = 0;
}

__global__ void __launch_bounds__(kTB, 5)
k_bf_push(DGraph g, const uint32_t *__restrict__ iv,
          const uint32_t *__restrict__ il0, uint32_t nitems,
          unsigned long long *__restrict__ dist,
          uint32_t *__restrict__ stamp, uint32_t round,
          uint32_t *__restrict__ nq,
          unsigned long long *__restrict__ cnt) {
  // next-round vertices staged in shared memory, one queue reservation per
  // block (as in the BFS push)
  __shared__ uint32_t stage[(kTB / 32) * kPushLeaves * 32];
  __shared__ uint32_t s_n;
  __shared__ unsigned long long s_deg, s_items, s_base;
  if (threadIdx.x == 0) {
    s_n = 0;
    s_deg = 0;
    s_items = 0;
  }
  __syncthreads();
  const uint64_t i = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (i < nitems) {
    const uint32_t u = iv[i];
    const unsigned long long du = __ldcg(dist + u);
    const uint64_t base = g.base[u];
    const uint32_t cap = g.cap[u], deg = g.deg[u];
    const uint32_t nl = cap ? nleaves_of(cap) : 0;
    const uint32_t l0 = il0[i], l1 = min(l0 + kPushLeaves, nl);
    unsigned long long dsum = 0, isum = 0;
    // four leaves' slots, lengths and distances in flight at once; leaves
    // keep their ids packed left with EMPTY after them
    constexpr int kBatch = 4;
    const uint32_t lim = cap <= kLeaf ? deg : kLeaf;
    const uint32_t below = (1u << lane) - 1u;
    for (uint32_t l = l0; l < l1; l += kBatch) {
      uint32_t v[kBatch], len[kBatch];
#pragma unroll
      for (int k = 0; k < kBatch; k++) {
        const uint64_t at = base + ((uint64_t)(l + k) << kLeafLog) + lane;
        const bool in = l + k < l1 && (uint32_t)lane < lim;
        v[k] = in ? g.slots[at] : kEmpty;
        len[k] = in ? g.vals[at] : 0u;
      }
      unsigned long long dv[kBatch];
#pragma unroll
      for (int k = 0; k < kBatch; k++) dv[k] = v[k] != kEmpty ? __ldcg(dist + v[k]) : 0ull;
      uint32_t mine = 0;  // bit k: this lane enqueues v[k]
#pragma unroll
      for (int k = 0; k < kBatch; k++) {
        const unsigned long long nd = du + len[k];
        if (v[k] != kEmpty && nd < dv[k] && atomicMin(dist + v[k], nd) > nd &&
            atomicExch(stamp + v[k], round) != round)
          mine |= 1u << k;
      }
      uint32_t mm[kBatch], total = 0;
#pragma unroll
      for (int k = 0; k < kBatch; k++) {
        mm[k] = l + k < l1 ? __ballot_sync(0xffffffffu, (mine >> k) & 1u) : 0u;
        total += __popc(mm[k]);
      }
      if (total == 0) continue;
      uint32_t at = 0;
      if (lane == 0) at = atomicAdd(&s_n, total);
      at = __shfl_sync(0xffffffffu, at, 0);
#pragma unroll
      for (int k = 0; k < kBatch; k++) {
        if ((mine >> k) & 1u) {
          stage[at + __popc(mm[k] & below)] = v[k];
          dsum += g.deg[v[k]];
          isum += items_of(g.cap[v[k]]);
        }
        at += __popc(mm[k]);
      }
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
      dsum += __shfl_xor_sync(0xffffffffu, dsum, d);
      isum += __shfl_xor_sync(0xffffffffu, isum, d);
    }
    if (lane == 0 && (dsum || isum)) {
      atomicAdd(&s_deg, dsum);
      atomicAdd(&s_items, isum);
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    s_base = s_n ? atomicAdd(&cnt[0], (unsigned long long)s_n) : 0ull;
    if (s_deg || s_items) {
      atomicAdd(&cnt[1], s_deg);
      atomicAdd(&cnt[2], s_items);
    }
  }
  __syncthreads();
  for (uint32_t k = threadIdx.x; k < s_n; k += blockDim.x) nq[s_base + k] = stage[k];
}

__global__ void k_bf_out(const unsigned long long *__restrict__ dist, uint32_t n,
                         int32_t *__restrict__ out) {
  uint32_t v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= n) return;
  const unsigned long long d = dist[v];
  out[v] = d >= 0x7FFFFFFFull ? 0x7FFFFFFF : (int32_t)d;
}
}  // namespace

static uint64_t items_of_host(uint32_t cap) {
  return cap > kLeaf ? ((cap >> kLeafLog) + kPushLeaves - 1) / kPushLeaves : 1;
}

sst_status bellman_ford(sst_graph *g, uint32_t src, int32_t *d_out) {
  if (!g->weighted || !g->d_vals) {
    set_error_message("Bellman-Ford needs a weighted graph (sst_config.weighted)");
    return SST_ESTATE;
  }
  TravState *t = nullptr;
  sst_status st = state(g, &t);
  if (st != SST_OK) return st;
  cudaStream_t s = g->stream;
  const uint32_t n = g->n;
  if (n == 0) return SST_OK;
  SST_CUDA_TRY(t->msrc.ensure(n));  // 64-bit distances
  SST_CUDA_TRY(t->qa.exact((uint64_t)n + 1));
  SST_CUDA_TRY(t->qb.exact((uint64_t)n + 1));
  SST_CUDA_TRY(t->fbits.ensure((uint64_t)n + 1));  // round stamps
  SST_CUDA_TRY(t->icnt.exact((uint64_t)n + 1));
  SST_CUDA_TRY(t->ioff.exact((uint64_t)n + 1));
  unsigned long long *dist = t->msrc.p;
  uint32_t *stamp = t->fbits.p;
  SST_LAUNCH(k_bf_init, blocks_for(n), kTB, 0, s, dist, stamp, n, src);
  SST_CUDA_TRY(cudaMemcpyAsync(t->qa.p, &src, 4, cudaMemcpyHostToDevice, s));
  uint32_t scap = 0;
  SST_CUDA_TRY(cudaMemcpyAsync(&scap, g->d_cap + src, 4, cudaMemcpyDeviceToHost, s));
  SST_CUDA_TRY(cudaStreamSynchronize(s));
  uint64_t qn = 1, qitems = items_of_host(scap);
  uint32_t *q = t->qa.p, *nq = t->qb.p;
  unsigned long long *cnt = t->d_small;
  DGraph dg = g->view();
  for (uint32_t round = 1; qn > 0; round++) {
    if (round > n + 1) {
      set_error_message("Bellman-Ford did not settle in n rounds");
      return SST_ETIMEDOUT;
    }
    SST_CUDA_TRY(t->iv.ensure(qitems + 1));
    SST_CUDA_TRY(t->il0.ensure(qitems + 1));
    SST_CUDA_TRY(cudaMemsetAsync(cnt, 0, 24, s));
    SST_LAUNCH(k_front_items, blocks_for(qn), kTB, 0, s, q, (uint32_t)qn,
               g->d_cap, t->icnt.p);
    g->arena.reset();
    SST_CUDA_TRY(g->arena.reserve(scan_scratch_bytes(qn, 4) + 4096));
    SST_CUDA_TRY((scan<uint32_t, OpAdd>(t->icnt.p, t->ioff.p, qn, 0u, OpAdd{},
                                        true, false, nullptr, g->arena, s)));
    SST_LAUNCH(k_front_expand, blocks_for(qn), kTB, 0, s, q, (uint32_t)qn,
               g->d_cap, t->ioff.p, t->iv.p, t->il0.p);
    SST_LAUNCH(k_bf_push, warp_blocks(qitems), kTB, 0, s, dg, t->iv.p, t->il0.p,
               (uint32_t)qitems, dist, stamp, round, nq, cnt);
    SST_CUDA_TRY(cudaMemcpyAsync(t->h_small, cnt, 24, cudaMemcpyDeviceToHost, s));
    SST_CUDA_TRY(cudaStreamSynchronize(s));
    qn = t->h_small[0];
    qitems = t->h_small[2];
    std::swap(q, nq);
  }
  SST_LAUNCH(k_bf_out, blocks_for(n), kTB, 0, s, dist, n, d_out);
  SST_CUDA_TRY(cudaGetLastError());
  return SST_OK;
}

}  // namespace sst
