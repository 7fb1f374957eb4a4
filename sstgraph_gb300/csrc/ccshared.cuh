// Connected-components building blocks shared by the PMA graph
// (traverse.cu) and the byte-width snapshot (compact.cu): the
// layout-independent parts of Afforest (Sutton, Ben-Nun, Barak 2018).
//  1. link every vertex to its first neighbours (the snapshot: two rounds of
//     cc_link, each followed by compression; the graph: hooks, traverse.cu);
//  2. sample 1024 vertices' roots and take the most frequent one, c: the
//     largest component so far;
//  3. link every edge of every vertex whose root is not c (on a symmetric
//     graph an edge with one end in c is linked from its other end), then
//     compress.
// A root is only ever linked below a smaller root (compare-and-swap on the
// larger one), so every component's final root -- its label -- is its
// smallest vertex id, independent of the order the links happen in.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "common.cuh"
#include "primitives.cuh"

namespace sst {
namespace {

__global__ void k_iota(uint32_t *__restrict__ p, uint32_t n) {
  uint32_t v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v < n) p[v] = v;
}

__device__ __forceinline__ uint32_t ld_par(const uint32_t *par, uint32_t x) {
  return __ldcg(par + x);
}

// the root of x, halving the path on the way: a visited vertex is pointed
// at its grandparent.  Only roots are ever linked (compare-and-swap on a
// root's own entry), so a non-root's entry changes only here, and always to
// one of its ancestors: still its tree, and a smaller id.  Every step moves
// to a smaller id, so the walk ends.
__device__ __forceinline__ uint32_t cc_find(uint32_t *par, uint32_t x) {
  for (;;) {
    const uint32_t p = ld_par(par, x);
    if (p == x) return x;
    const uint32_t gp = ld_par(par, p);
    if (gp == p) return p;
    par[x] = gp;
    x = gp;
  }
}

// link the trees of u and v: find both roots, link the larger below the
// smaller; a failed compare-and-swap means that root was linked meanwhile,
// so the roots are looked up again.  err counts links that gave up (every
// failed attempt is another link's progress; the bound only keeps every
// loop finite).  Without halving, concurrent links build long chains of
// roots that later links walk again and again.
__device__ __forceinline__ void cc_link(uint32_t *par, uint32_t u, uint32_t v,
                                        unsigned long long *err) {
  // the finds start at the parents (usually the roots themselves)
  uint32_t p1 = ld_par(par, u), p2 = ld_par(par, v);
  if (p1 == p2) return;
  for (int it = 0;; it++) {
    if (it == (1 << 20)) {
      atomicAdd(err, 1ull);
      return;
    }
    const uint32_t r1 = cc_find(par, p1), r2 = cc_find(par, p2);
    if (r1 == r2) return;
    const uint32_t hi = max(r1, r2), lo = min(r1, r2);
    if (atomicCAS(&par[hi], hi, lo) == hi) return;
    p1 = hi;
    p2 = lo;
  }
}

// The most frequent root among 1024 sampled vertices (ties: the smaller).
// One block: the roots meet in a shared hash table of counters (open
// addressing, at most half full), so the kernel is two rounds of loads and a
// reduction; sorting the 1024 roots took 55 block barriers.
constexpr uint32_t kGiantSlots = 2048;
__global__ void __launch_bounds__(1024) k_cc_giant(const uint32_t *__restrict__ par,
                                                   uint32_t n,
                                                   unsigned long long *__restrict__ out) {
  __shared__ uint32_t key[kGiantSlots], cnt[kGiantSlots];
  __shared__ unsigned long long best;
  const uint32_t t = threadIdx.x;
  pdl_wait();
  const uint32_t root = par[(uint32_t)(mix64(0x5EEDull + t) % n)];
  for (uint32_t i = t; i < kGiantSlots; i += 1024) {
    key[i] = kEmpty;  // no vertex has this id
    cnt[i] = 0;
  }
  if (t == 0) best = 0;
  __syncthreads();
  uint32_t h = (root * 0x9E3779B1u) >> 21;  // top 11 bits
  for (;;) {
    const uint32_t k = atomicCAS(&key[h], kEmpty, root);
    if (k == kEmpty || k == root) break;
    h = (h + 1) & (kGiantSlots - 1);
  }
  // lanes of one warp that hold the same root add once
  const uint32_t peers = __match_any_sync(0xffffffffu, root);
  if ((t & 31) == (uint32_t)__ffs(peers) - 1) atomicAdd(&cnt[h], (uint32_t)__popc(peers));
  __syncthreads();
  // larger count first, then the smaller label
  unsigned long long b = 0;
  for (uint32_t i = t; i < kGiantSlots; i += 1024)
    if (cnt[i]) b = max(b, ((unsigned long long)cnt[i] << 32) | (0xFFFFFFFFu - key[i]));
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) b = max(b, __shfl_xor_sync(0xffffffffu, b, d));
  if ((t & 31) == 0 && b) atomicMax(&best, b);
  __syncthreads();
  if (t == 0) out[0] = 0xFFFFFFFFu - (uint32_t)(best & 0xFFFFFFFFu);
}

// Every vertex to its root; with `hooks`, only if it is not zero.  Nothing is
// linked meanwhile, so the parents may come through L1 (an old one is an
// ancestor): most chains end at one hot root, and loads of it past L1 queue at
// its L2 slice (2e6 vertices already compressed: 16 us that way, 8 us
// this way).
__device__ __forceinline__ void cc_compress(uint32_t *par, uint32_t v) {
  const uint32_t p = par[v];
  uint32_t x = p, q;
  while ((q = par[x]) != x) x = q;
  if (x != p) par[v] = x;
}
__global__ void k_cc_compress(uint32_t *par, uint32_t n,
                              const unsigned long long *__restrict__ hooks) {
  pdl_wait();
  if (hooks && *hooks == 0) return;
  const uint32_t v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v < n) cc_compress(par, v);
}

}  // namespace
}  // namespace sst
