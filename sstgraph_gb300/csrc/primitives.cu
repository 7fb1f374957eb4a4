// Stable LSD radix sort of 64-bit keys (8-bit digits) and the launch
// counter.  A pass ranks a tile's keys -- every warp its own contiguous slice,
// by a match word and a counter a digit in shared memory -- reorders the tile in
// shared memory and writes it in runs of one digit.  Up to 4096 keys sort in one
// block; up to 2^30 a pass is one launch, whose tiles add up the counts of the
// tiles before them; longer sorts count and scan in launches of their own.
#include <algorithm>
#include <atomic>
#include <cstdio>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <type_traits>
#include <vector>

#include "primitives.cuh"

namespace sst {

static std::atomic<uint64_t> g_launches{0};
void note_launch() { g_launches.fetch_add(1, std::memory_order_relaxed); }
void note_launches(int64_t k) {
  g_launches.fetch_add((uint64_t)k, std::memory_order_relaxed);
}
uint64_t launches() { return g_launches.load(std::memory_order_relaxed); }

static std::atomic<unsigned long long> g_scan_epoch{0};
unsigned long long next_scan_tag() {
  const unsigned long long e =
      (g_scan_epoch.fetch_add(1, std::memory_order_relaxed) + 1) & kScanEpochMask;
  return kScanTag | (e << 2);
}

thread_local bool t_capture_forms = false;
thread_local DeviceScanTags *t_scan_tags = nullptr;

namespace {
__global__ void k_scan_epoch_bump(unsigned long long *epoch) {
  pdl_wait(); *epoch += 1; }
}  // namespace

DeviceScanTags::DeviceScanTags(unsigned long long *e) : epoch(e), prev(t_scan_tags) {
  t_scan_tags = this;  // with a null epoch: host tags, as without one
}
DeviceScanTags::~DeviceScanTags() { t_scan_tags = prev; }
cudaError_t DeviceScanTags::bump(cudaStream_t s) {
  next = 0;
  SST_LAUNCH_PDL(k_scan_epoch_bump, 1, 1, 0, s, epoch);
  return cudaGetLastError();
}

static std::atomic<int> g_lookback_polls{kLookbackPolls};
int lookback_polls() { return g_lookback_polls.load(std::memory_order_relaxed); }
void set_lookback_polls(int polls) {
  g_lookback_polls.store(polls < 0 ? 0 : polls, std::memory_order_relaxed);
}

// ------------------------------------------------------------- profiler
namespace {
struct Pending {
  const char *name;
  cudaEvent_t a, b;
  uint64_t bytes;
};
struct Totals {
  uint64_t launches = 0;
  double ms = 0;
  uint64_t bytes = 0;  // declared algorithmic bytes (0 where undeclared)
};
std::mutex g_prof_mu;
bool g_prof_on = false;
std::vector<cudaEvent_t> g_pool;
std::vector<Pending> g_pending;
std::map<std::string, Totals> g_totals;

cudaEvent_t take_event() {
  if (!g_pool.empty()) {
    cudaEvent_t e = g_pool.back();
    g_pool.pop_back();
    return e;
  }
  cudaEvent_t e = nullptr;
  cudaEventCreate(&e);
  return e;
}

// fold finished pairs into the totals (caller holds the lock)
void drain(bool wait) {
  size_t keep = 0;
  for (size_t i = 0; i < g_pending.size(); i++) {
    Pending &p = g_pending[i];
    if (wait) cudaEventSynchronize(p.b);
    float ms = 0;
    if (cudaEventElapsedTime(&ms, p.a, p.b) == cudaSuccess) {
      Totals &t = g_totals[p.name];
      t.launches++;
      t.ms += ms;
      t.bytes += p.bytes;
      g_pool.push_back(p.a);
      g_pool.push_back(p.b);
    } else {
      cudaGetLastError();
      g_pending[keep++] = p;
    }
  }
  g_pending.resize(keep);
}
}  // namespace

std::string g_prof_filter;  // profile only kernels whose name contains it

static thread_local bool t_prof_paused = false;
ProfPause::ProfPause() : prev(t_prof_paused) { t_prof_paused = true; }
ProfPause::~ProfPause() { t_prof_paused = prev; }

bool profiling(const char *name) {
  if (!g_prof_on || t_prof_paused) return false;
  return g_prof_filter.empty() || strstr(name, g_prof_filter.c_str()) != nullptr;
}

cudaEvent_t prof_begin(cudaStream_t s) {
  std::lock_guard<std::mutex> lk(g_prof_mu);
  cudaEvent_t e = take_event();
  cudaEventRecord(e, s);
  return e;
}

void prof_end(const char *name, cudaEvent_t start, cudaStream_t s,
              uint64_t bytes) {
  std::lock_guard<std::mutex> lk(g_prof_mu);
  cudaEvent_t e = take_event();
  cudaEventRecord(e, s);
  g_pending.push_back({name, start, e, bytes});
  if (g_pending.size() > 4096) drain(false);
}

void profile_start(const char *filter) {
  std::lock_guard<std::mutex> lk(g_prof_mu);
  drain(true);
  g_totals.clear();
  g_prof_filter = filter ? filter : "";
  g_prof_on = true;
}

// JSON object {"kernel": {"launches": L, "ms": T}, ...}; stops profiling
std::string profile_collect() {
  std::lock_guard<std::mutex> lk(g_prof_mu);
  g_prof_on = false;
  drain(true);
  std::string out = "{";
  bool first = true;
  for (auto &kv : g_totals) {
    char buf[256];
    snprintf(buf, sizeof(buf),
             "%s\"%s\": {\"launches\": %llu, \"ms\": %.6f, \"bytes\": %llu}",
             first ? "" : ", ", kv.first.c_str(),
             (unsigned long long)kv.second.launches, kv.second.ms,
             (unsigned long long)kv.second.bytes);
    out += buf;
    first = false;
  }
  out += "}";
  g_totals.clear();
  return out;
}

namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kItems = 16;
constexpr int kTile = kThreads * kItems;  // 4096
// Shorter sorts use smaller tiles: more blocks, each ranking fewer keys, so a
// pass's dependent chain is shorter, until the blocks no longer fit the GPU at
// once.  Five passes, by items a thread (us; keys alone, then with values):
//   keys        4             8             16
//   60,000     26.7    -     36.1  36.3     35.0  48.8
//   260,000    33.5    -     35.1  38.4     45     50
//   800,000    81      -     50.3  56.7     57.6  65.6
//   1,200,000   -      -     69.6  77.2     59.3  67.4
//   4,800,000   -      -      195   240      169   224
constexpr int kSmallItems = 4;
constexpr uint64_t kSmallTileKeys = 256ull * kThreads * kSmallItems;  // 2^18, no values
constexpr int kMidItems = 8;
constexpr uint64_t kMidTileKeys = 448ull * kThreads * kMidItems;  // 7 * 2^17
constexpr int kRadix = 256;
constexpr uint64_t kOneSweepKeys = 1ull << 30;  // longer sorts count and scan in launches
constexpr uint32_t kNoDigit = 0xffffffffu;  // an item past the end
// Offset of this thread's item `it` in a warp-contiguous tile of ITEMS items
// per thread: warp w owns [w * ITEMS * 32, (w + 1) * ITEMS * 32), item it of
// lane l sits at w * ITEMS * 32 + it * 32 + l.  Loads stay coalesced, and a
// warp's items in (it, lane) order are in index order, so a warp ranks its
// own items without the rest of the block.
template <int ITEMS>
__device__ __forceinline__ uint32_t tile_offset(int it) {
  return (threadIdx.x >> 5) * (ITEMS * 32) + it * 32 + (threadIdx.x & 31);
}

// Stable rank of each of the warp's items among the warp's earlier items of
// the same digit.  The lanes holding one digit find each other through a
// warp-private word per digit in shared memory: each sets its bit with an
// atomic OR and reads the word back (far fewer instructions than eight
// ballots, one per digit bit, or __match_any_sync); the lowest of them then
// advances the digit's counter and clears the word.  wc (the warp's 256
// counters) and wm (its 256 match words) are zero and visible to the warp
// on entry; wc ends as the warp's count of each digit, wm zero again.  Items
// past the end carry kNoDigit.
template <int ITEMS>
__device__ __forceinline__ void warp_rank(const uint32_t (&dg)[ITEMS],
                                          uint32_t (&lr)[ITEMS], uint32_t *wc,
                                          uint32_t *wm) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t below = (1u << lane) - 1u;
#pragma unroll
  for (int it = 0; it < ITEMS; it++) {
    const uint32_t d = dg[it];
    const bool valid = d != kNoDigit;
    if (valid) atomicOr(&wm[d], 1u << lane);
    __syncwarp();
    const uint32_t peers = valid ? wm[d] : 0u;
    lr[it] = (valid ? wc[d] : 0u) + __popc(peers & below);
    __syncwarp();
    if (valid && (peers & below) == 0) {  // the lowest: its rank is the counter
      wc[d] = lr[it] + __popc(peers);
      wm[d] = 0;
    }
    __syncwarp();
  }
}
// a warp clears its 256 match words (then visible to the warp)
__device__ __forceinline__ void clear_match_words(uint32_t *wm) {
  const uint32_t lane = threadIdx.x & 31;
#pragma unroll
  for (int k = 0; k < kRadix / 32; k++) wm[lane + 32 * k] = 0;
  __syncwarp();
}

// Exclusive scan of one value per thread over the block, in thread order
// (one __syncthreads inside).
__device__ __forceinline__ uint32_t block_excl_scan(uint32_t v, uint32_t *wsum) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t inc = v;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    uint32_t o = __shfl_up_sync(0xffffffffu, inc, d);
    if (lane >= d) inc += o;
  }
  if (lane == 31) wsum[warp] = inc;
  __syncthreads();
  uint32_t off = 0;
#pragma unroll
  for (int w = 0; w < kWarps; w++) off += w < warp ? wsum[w] : 0u;
  return off + inc - v;
}

// Per-tile digit counts, digit-major: hist[digit * tiles + tile].
__global__ void __launch_bounds__(kThreads)
k_hist(const uint64_t *__restrict__ keys, uint64_t n, int shift,
       uint32_t *__restrict__ hist, const uint32_t *__restrict__ d_n) {
  pdl_wait();
  if (d_n && *d_n < n) n = *d_n;
  __shared__ uint32_t h[kRadix];
  h[threadIdx.x] = 0;
  __syncthreads();
  const uint64_t t0 = (uint64_t)blockIdx.x * kTile;
#pragma unroll 4
  for (int it = 0; it < kItems; it++) {
    uint64_t i = t0 + (uint64_t)it * kThreads + threadIdx.x;
    if (i < n) atomicAdd(&h[(keys[i] >> shift) & 0xff], 1u);
  }
  __syncthreads();
  hist[(uint64_t)threadIdx.x * gridDim.x + blockIdx.x] = h[threadIdx.x];
}

// One pass's stable scatter of a tile, for sorts too long for the one-sweep form.
// The warps rank their slices, the tile is laid out in shared memory in (digit,
// index) order, and the block writes it out in that order, so the keys of one digit
// leave as one run of consecutive addresses (whole sectors, not one 8-byte write per
// lane).  hist holds the scanned digit-major counts.
// Dynamic shared memory: scatter_smem_bytes<KV, IT>(), IT items per thread; the
// staging area (keys and values of the tile) also holds the match words of the ranking.
template <bool KV, int IT>
constexpr size_t scatter_stage_bytes() {
  static_assert(kThreads * IT * 8 >= kWarps * kRadix * 4, "the match words fit");
  return (size_t)kThreads * IT * (KV ? 12 : 8);
}
template <bool KV, int IT>
constexpr size_t scatter_smem_bytes() {
  return scatter_stage_bytes<KV, IT>() + (size_t)kWarps * kRadix * 4 + kRadix * 4 +
         kWarps * 4;
}

template <bool KV>
__global__ void __launch_bounds__(kThreads, 2)
k_scatter(const uint64_t *__restrict__ in, uint64_t *__restrict__ out,
          uint64_t n, int shift, const uint32_t *__restrict__ hist,
          const uint32_t *__restrict__ vin, uint32_t *__restrict__ vout,
          const uint32_t *__restrict__ d_n) {
  pdl_wait();
  constexpr int IT = kItems, TILE = kTile;
  if (d_n && *d_n < n) n = *d_n;
  extern __shared__ __align__(16) unsigned char smem[];
  uint64_t *skeys = reinterpret_cast<uint64_t *>(smem);
  uint32_t *svals = reinterpret_cast<uint32_t *>(smem + (size_t)TILE * 8);
  uint32_t(*wcnt)[kRadix] = reinterpret_cast<uint32_t(*)[kRadix]>(
      smem + scatter_stage_bytes<KV, IT>());
  uint32_t *adj = &wcnt[kWarps - 1][kRadix - 1] + 1;  // [kRadix]
  uint32_t *wsum = adj + kRadix;                        // [kWarps]
  const int warp = threadIdx.x >> 5;
#pragma unroll
  for (int w = 0; w < kWarps; w++) wcnt[w][threadIdx.x] = 0;
  // the tile's keys (and values) come in at once, ahead of the ranking
  const uint64_t t0 = (uint64_t)blockIdx.x * TILE;
  uint64_t kk[IT];
  uint32_t vv[KV ? IT : 1];
  uint32_t dg[IT];
#pragma unroll
  for (int it = 0; it < IT; it++) {
    const uint64_t i = t0 + tile_offset<IT>(it);
    kk[it] = i < n ? in[i] : 0;
    if (KV) vv[it] = i < n ? vin[i] : 0u;
    dg[it] = i < n ? (uint32_t)(kk[it] >> shift) & 0xff : kNoDigit;
  }
  // output position of this tile's first key of digit threadIdx.x
  const uint32_t gbase = hist[(uint64_t)threadIdx.x * gridDim.x + blockIdx.x];
  __syncthreads();
  // the match words sit in the staging area, free until the reorder
  uint32_t *wm = reinterpret_cast<uint32_t *>(smem) + warp * kRadix;
  clear_match_words(wm);
  uint32_t lr[IT];
  warp_rank<IT>(dg, lr, wcnt[warp], wm);
  __syncthreads();
  // tile-local start of each digit, then of each warp's share of it
  uint32_t tcount = 0;
#pragma unroll
  for (int w = 0; w < kWarps; w++) tcount += wcnt[w][threadIdx.x];
  const uint32_t tstart = block_excl_scan(tcount, wsum);
  uint32_t s = tstart;
#pragma unroll
  for (int w = 0; w < kWarps; w++) {
    const uint32_t c = wcnt[w][threadIdx.x];
    wcnt[w][threadIdx.x] = s;
    s += c;
  }
  adj[threadIdx.x] = gbase - tstart;  // output position = adj[d] + local
  __syncthreads();
#pragma unroll
  for (int it = 0; it < IT; it++) {
    if (dg[it] == kNoDigit) continue;
    const uint32_t lp = wcnt[warp][dg[it]] + lr[it];
    skeys[lp] = kk[it];
    if (KV) svals[lp] = vv[it];
  }
  __syncthreads();
  const uint32_t tn = t0 >= n ? 0u : (uint32_t)(n - t0 < (uint64_t)TILE ? n - t0 : TILE);
  for (uint32_t j = threadIdx.x; j < tn; j += kThreads) {
    const uint64_t key = skeys[j];
    const uint32_t pos = adj[(key >> shift) & 0xff] + j;
    out[pos] = key;
    if (KV) vout[pos] = svals[j];
  }
}

// ---- one-sweep passes (after Adinets and Merrill, "Onesweep", 2022).
// k_hist_all reads the keys once and counts every pass's digits (global
// totals, no per-tile tables) and clears the passes' tile status words.
// Each pass is then one launch: a block ranks its tile as k_scatter does and
// publishes its per-digit counts, and thread d finds the count of digit d in
// all tiles before its own.  Those are not walked tile by tile to the nearest
// inclusive prefix, which moves on by some 32 tiles a step of 0.7 us: every tile
// also adds its counts to the sums of its group of 8 tiles, of 64, and so on, and
// reads the words of the up to 7 tiles, 7 groups of 8, ... that make up the tiles
// before it.  They are read together, and depend on no other tile's look-back.
// A tile's word is kOsAgg | count (0 = not yet published); a group's is (tiles
// published << 32) | count, complete when it holds all its tiles.  Every wait is
// bounded: a word that is not complete in time is made up from its tiles' words
// or keys instead.
constexpr uint32_t kOsAgg = 1u << 30, kOsMask = kOsAgg - 1;
constexpr int kOsPolls = 1 << 14;
constexpr int kOsLog = 3, kOsGroup = 1 << kOsLog;
// levels of groups above nt tiles (at most 2^18): the last has at most
// kOsGroup words
__host__ __device__ inline int os_levels(uint32_t nt) {
  int l = 0;
  while (nt > kOsGroup) {
    nt = (nt + kOsGroup - 1) >> kOsLog;
    l++;
  }
  return l;
}
// status words (32-bit) of a pass over nt tiles: the tiles', then each level's
inline uint64_t os_status_words(uint32_t nt) {
  uint64_t w = (uint64_t)nt * kRadix;
  while (nt > kOsGroup) {
    nt = (nt + kOsGroup - 1) >> kOsLog;
    w += 2 * (uint64_t)nt * kRadix;
  }
  return w;
}

template <int IT>
__global__ void __launch_bounds__(kThreads)
k_hist_all(const uint64_t *__restrict__ keys, uint64_t n, int lo, int passes,
           uint32_t *__restrict__ totals, uint32_t *__restrict__ status,
           uint64_t status_words, const uint32_t *__restrict__ d_n) {
  pdl_wait();
  if (d_n && *d_n < n) n = *d_n;
  __shared__ uint32_t h[8][kRadix];
  for (int p = 0; p < passes; p++) h[p][threadIdx.x] = 0;
  __syncthreads();
  const uint64_t t0 = (uint64_t)blockIdx.x * (kThreads * IT);
#pragma unroll 4
  for (int it = 0; it < IT; it++) {
    const uint64_t i = t0 + (uint64_t)it * kThreads + threadIdx.x;
    if (i < n) {
      const uint64_t k = keys[i];
      for (int p = 0; p < passes; p++) atomicAdd(&h[p][(k >> (lo + 8 * p)) & 0xff], 1u);
    }
  }
  __syncthreads();
  for (int p = 0; p < passes; p++)
    if (h[p][threadIdx.x]) atomicAdd(&totals[p * kRadix + threadIdx.x], h[p][threadIdx.x]);
  for (uint64_t i = (uint64_t)blockIdx.x * kThreads + threadIdx.x; i < status_words;
       i += (uint64_t)gridDim.x * kThreads)
    status[i] = 0;
}

// count of digit d among the keys of tile t (the bounded wait's fallback)
__device__ __forceinline__ uint32_t os_count_tile(const uint64_t *in, uint64_t n,
                                                  uint64_t t, int tile, int shift,
                                                  uint32_t d) {
  uint32_t c = 0;
  const uint64_t a = t * (uint64_t)tile;
  const uint64_t e = a + tile < n ? a + tile : n;
  for (uint64_t i = a; i < e; i++) c += ((uint32_t)(in[i] >> shift) & 0xff) == d;
  return c;
}

// resident blocks an SM that the registers are held to: as many as fit without
// spilling what the ranking holds (4.8M keys in 16 items a thread, 2 / 3 / 4 / 5
// blocks: 207, 174, 169, 220 us; with values 3 / 4: 224, 280)
template <bool KV, int IT>
constexpr int os_blocks() {
  return IT == kSmallItems ? 6 : IT == kMidItems ? (KV ? 4 : 5) : (KV ? 3 : 4);
}
template <bool KV, int IT>
__global__ void __launch_bounds__(kThreads, os_blocks<KV, IT>())
k_scatter_os(const uint64_t *__restrict__ in, uint64_t *__restrict__ out,
             uint64_t n, int shift, const uint32_t *__restrict__ totals,
             uint32_t *__restrict__ status, const uint32_t *__restrict__ vin,
             uint32_t *__restrict__ vout, const uint32_t *__restrict__ d_n) {
  pdl_wait();
  constexpr int TILE = kThreads * IT;
  if (d_n && *d_n < n) n = *d_n;
  extern __shared__ __align__(16) unsigned char smem[];
  uint64_t *skeys = reinterpret_cast<uint64_t *>(smem);
  uint32_t *svals = reinterpret_cast<uint32_t *>(smem + (size_t)TILE * 8);
  uint32_t(*wcnt)[kRadix] = reinterpret_cast<uint32_t(*)[kRadix]>(
      smem + scatter_stage_bytes<KV, IT>());
  uint32_t *adj = &wcnt[kWarps - 1][kRadix - 1] + 1;  // [kRadix]
  uint32_t *wsum = adj + kRadix;                        // [kWarps]
  const int warp = threadIdx.x >> 5;
  const uint32_t d = threadIdx.x;  // this thread's digit in the bookkeeping
#pragma unroll
  for (int w = 0; w < kWarps; w++) wcnt[w][d] = 0;
  const uint32_t tile = blockIdx.x;
  const uint64_t t0 = (uint64_t)tile * TILE;
  uint64_t kk[IT];
  uint32_t vv[KV ? IT : 1];
  uint32_t dg[IT];
#pragma unroll
  for (int it = 0; it < IT; it++) {
    const uint64_t i = t0 + tile_offset<IT>(it);
    kk[it] = i < n ? in[i] : 0;
    if (KV) vv[it] = i < n ? vin[i] : 0u;
    dg[it] = i < n ? (uint32_t)(kk[it] >> shift) & 0xff : kNoDigit;
  }
  // the match words sit in the staging area, free until the reorder
  uint32_t *wm = reinterpret_cast<uint32_t *>(smem) + warp * kRadix;
  clear_match_words(wm);
  // all keys of smaller digits (while the keys are on their way)
  const uint32_t smaller = block_excl_scan(totals[d], wsum);
  uint32_t lr[IT];
  warp_rank<IT>(dg, lr, wcnt[warp], wm);
  __syncthreads();
  uint32_t tcount = 0;
#pragma unroll
  for (int w = 0; w < kWarps; w++) tcount += wcnt[w][d];
  // publish this tile's count of digit d
  const int levels = os_levels(gridDim.x);
  atomicExch(status + (uint64_t)tile * kRadix + d, kOsAgg | tcount);
  unsigned long long *const group =
      reinterpret_cast<unsigned long long *>(status + (uint64_t)gridDim.x * kRadix) + d;
  {
    unsigned long long *at = group;
    uint32_t nt = gridDim.x, i = tile;
    for (int l = 0; l < levels; l++) {
      nt = (nt + kOsGroup - 1) >> kOsLog;
      i >>= kOsLog;
      atomicAdd(at + (uint64_t)i * kRadix, (1ull << 32) | tcount);
      at += (uint64_t)nt * kRadix;
    }
  }
  // the tile in order, while the earlier tiles publish theirs
  const uint32_t tstart = block_excl_scan(tcount, wsum);
  uint32_t sacc = tstart;
#pragma unroll
  for (int w = 0; w < kWarps; w++) {
    const uint32_t c = wcnt[w][d];
    wcnt[w][d] = sacc;
    sacc += c;
  }
  __syncthreads();
#pragma unroll
  for (int it = 0; it < IT; it++) {
    if (t0 + tile_offset<IT>(it) >= n) continue;
    const uint32_t lp = wcnt[warp][(kk[it] >> shift) & 0xff] + lr[it];
    skeys[lp] = kk[it];
    if (KV) svals[lp] = vv[it];
  }
  // the earlier tiles' keys of digit d
  uint32_t before = 0;
  bool whole = true;
  {
    const uint32_t n0 = tile & (kOsGroup - 1);
    const volatile uint32_t *p = status + (uint64_t)(tile - n0) * kRadix + d;
    uint32_t w[kOsGroup - 1];
#pragma unroll
    for (int q = 0; q < kOsGroup - 1; q++) w[q] = q < n0 ? p[q * kRadix] : kOsAgg;
    const unsigned long long *at = group;
    uint32_t nt = gridDim.x, i = tile;
    for (int l = 0; l < levels; l++) {
      nt = (nt + kOsGroup - 1) >> kOsLog;
      i >>= kOsLog;
      const uint32_t nl = i & (kOsGroup - 1);
      const unsigned long long full = 1ull << (kOsLog * (l + 1));
      const volatile unsigned long long *gp = at + (uint64_t)(i - nl) * kRadix;
      unsigned long long v[kOsGroup - 1];
#pragma unroll
      for (int q = 0; q < kOsGroup - 1; q++) v[q] = q < nl ? gp[q * kRadix] : full << 32;
#pragma unroll
      for (int q = 0; q < kOsGroup - 1; q++) {
        for (int t = 0; (v[q] >> 32) != full && t < kOsPolls; t++) {
          __nanosleep(t < 32 ? 20 : 200);
          v[q] = gp[q * kRadix];
        }
        whole &= (v[q] >> 32) == full;
        before += (uint32_t)v[q];
      }
      at += (uint64_t)nt * kRadix;
    }
#pragma unroll
    for (int q = 0; q < kOsGroup - 1; q++) {
      for (int t = 0; w[q] == 0 && t < kOsPolls; t++) {
        __nanosleep(t < 32 ? 20 : 200);
        w[q] = p[q * kRadix];
      }
      whole &= w[q] != 0;
      before += w[q] & kOsMask;
    }
  }
  if (!whole) {  // a tile never published: the words that are there, else the keys
    before = 0;
    for (uint32_t t = 0; t < tile; t++) {
      const uint32_t v = *(const volatile uint32_t *)(status + (uint64_t)t * kRadix + d);
      before += v ? v & kOsMask : os_count_tile(in, n, t, TILE, shift, d);
    }
  }
  adj[d] = smaller + before - tstart;
  __syncthreads();
  const uint32_t tn = t0 >= n ? 0u : (uint32_t)(n - t0 < (uint64_t)TILE ? n - t0 : TILE);
  for (uint32_t j = threadIdx.x; j < tn; j += kThreads) {
    const uint64_t key = skeys[j];
    const uint32_t pos = adj[(key >> shift) & 0xff] + j;
    out[pos] = key;
    if (KV) vout[pos] = svals[j];
  }
}

// The key-value scatter's shared memory is above the 48 KB default: raise
// its limit once per device (before the first launch there).
cudaError_t scatter_smem_optin() {
  static std::atomic<uint64_t> done{0};  // one bit per device below 64
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 64 && ((done.load(std::memory_order_relaxed) >> dev) & 1)) return cudaSuccess;
  e = cudaFuncSetAttribute(k_scatter<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)scatter_smem_bytes<true, kItems>());
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_scatter_os<true, kItems>,
                             cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)scatter_smem_bytes<true, kItems>());
  if (e == cudaSuccess && dev < 64) done.fetch_or(1ull << dev, std::memory_order_relaxed);
  return e;
}

// Whole sort of keys with values in one CTA for n <= TILE, both staged in shared
// memory; each pass ranks warp-contiguous items as k_scatter does, the digit
// offsets coming from a block scan of the warps' counts.
template <int TILE>
__global__ void __launch_bounds__(kThreads)
k_sort_small(uint64_t *__restrict__ keys, uint32_t *__restrict__ vals,
             uint64_t n, int bits, const uint32_t *__restrict__ d_n) {
  pdl_wait();
  if (d_n && *d_n < n) n = *d_n;
  constexpr int IT = TILE / kThreads;
  __shared__ uint64_t buf[2][TILE];
  __shared__ uint32_t vbuf[2][TILE];
  __shared__ uint32_t wcnt[kWarps][kRadix];
  __shared__ uint32_t wmatch[kWarps][kRadix];
  __shared__ uint32_t wsum[kWarps];
  const int warp = threadIdx.x >> 5;
  clear_match_words(wmatch[warp]);  // warp_rank leaves them clear again
  for (uint64_t i = threadIdx.x; i < n; i += kThreads) {
    buf[0][i] = keys[i];
    vbuf[0][i] = vals[i];
  }
  int cur = 0;
  for (int shift = 0; shift < bits; shift += 8) {
#pragma unroll
    for (int w = 0; w < kWarps; w++) wcnt[w][threadIdx.x] = 0;
    __syncthreads();  // counters clear; the previous pass's keys in place
    uint64_t kk[IT];
    uint32_t dg[IT], lr[IT];
#pragma unroll
    for (int it = 0; it < IT; it++) {
      const uint32_t o = tile_offset<IT>(it);
      kk[it] = o < n ? buf[cur][o] : 0;
      dg[it] = o < n ? (uint32_t)(kk[it] >> shift) & 0xff : kNoDigit;
    }
    warp_rank<IT>(dg, lr, wcnt[warp], wmatch[warp]);
    __syncthreads();
    uint32_t tot = 0;
#pragma unroll
    for (int w = 0; w < kWarps; w++) tot += wcnt[w][threadIdx.x];
    uint32_t s = block_excl_scan(tot, wsum);
#pragma unroll
    for (int w = 0; w < kWarps; w++) {
      const uint32_t c = wcnt[w][threadIdx.x];
      wcnt[w][threadIdx.x] = s;
      s += c;
    }
    __syncthreads();
#pragma unroll
    for (int it = 0; it < IT; it++) {
      if (dg[it] == kNoDigit) continue;
      const uint32_t pos = wcnt[warp][dg[it]] + lr[it];
      buf[cur ^ 1][pos] = kk[it];
      vbuf[cur ^ 1][pos] = vbuf[cur][tile_offset<IT>(it)];
    }
    __syncthreads();  // all reads of the counters done before the next pass
    cur ^= 1;
  }
  for (uint64_t i = threadIdx.x; i < n; i += kThreads) {
    keys[i] = buf[cur][i];
    vals[i] = vbuf[cur][i];
  }
}

constexpr int kSmallSortKV = 1024;

// Keys alone, up to kSmallSort, in one CTA of kBlockThreads holding IT keys a
// thread in registers: radix passes whose counts, offsets and exchange stay in
// shared memory, where a pass over several CTAs is a launch of its own (about
// 5 us).  A pass is bound by its warps' chains of match-word rankings, IT of
// them, and seven block barriers.  Five passes against the forms before (one CTA
// of 256 threads, a bitonic network, tiles of 1024; us with the launch): 1000
// keys 10.1 and 10.5, 2048 14.0 and 20.7, 3000 16.5 and 24.0, 4096 18.2 and 24.0;
// with 1024 threads 12.9, 15.1, 18.7, 20.5, and 8192 keys 30.7 where tiles take
// 23.9.
constexpr int kBlockThreads = 512;
constexpr int kBlockWarps = kBlockThreads / 32;
template <int IT>
constexpr size_t block_sort_smem() {
  return (size_t)kBlockThreads * IT * 8 + 2 * (size_t)kBlockWarps * kRadix * 4 +
         (size_t)kBlockThreads * 4 + kBlockWarps * 4;
}
template <int IT>
__global__ void __launch_bounds__(kBlockThreads)
k_sort_block(uint64_t *__restrict__ keys, uint64_t n, int lo, int bits,
             const uint32_t *__restrict__ d_n) {
  pdl_wait();
  if (d_n && *d_n < n) n = *d_n;
  extern __shared__ __align__(16) unsigned char smem[];
  uint64_t *buf = reinterpret_cast<uint64_t *>(smem);
  uint32_t *wcnt = reinterpret_cast<uint32_t *>(buf + kBlockThreads * IT);  // [warp][digit]
  uint32_t *wmatch = wcnt + kBlockWarps * kRadix;
  uint32_t *part = wmatch + kBlockWarps * kRadix;  // [quarter of the warps][digit]
  uint32_t *wsum = part + kBlockThreads;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t t = threadIdx.x, d = t & (kRadix - 1), q = t / kRadix;
  constexpr int kQuarters = kBlockThreads / kRadix, kShare = kBlockWarps / kQuarters;
  uint32_t *wc = wcnt + warp * kRadix, *wm = wmatch + warp * kRadix;
  clear_match_words(wm);  // warp_rank leaves them clear again
  uint64_t kk[IT];
#pragma unroll
  for (int it = 0; it < IT; it++) {
    const uint32_t o = tile_offset<IT>(it);
    kk[it] = o < n ? keys[o] : 0;
  }
  for (int shift = lo; shift < lo + bits; shift += 8) {
    clear_match_words(wc);
    uint32_t dg[IT], lr[IT];
#pragma unroll
    for (int it = 0; it < IT; it++)
      dg[it] = tile_offset<IT>(it) < n ? (uint32_t)(kk[it] >> shift) & 0xff : kNoDigit;
    warp_rank<IT>(dg, lr, wc, wm);
    __syncthreads();
    uint32_t sum = 0;
#pragma unroll
    for (int w = 0; w < kShare; w++) sum += wcnt[(q * kShare + w) * kRadix + d];
    part[t] = sum;
    __syncthreads();
    uint32_t tot = 0, inc = 0;
    if (t < kRadix) {
#pragma unroll
      for (int r = 0; r < kQuarters; r++) tot += part[r * kRadix + t];
      inc = tot;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t x = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += x;
      }
      if (lane == 31) wsum[warp] = inc;
    }
    __syncthreads();
    if (t < kRadix) {
      uint32_t run = inc - tot;
      for (int w = 0; w < warp; w++) run += wsum[w];
#pragma unroll
      for (int r = 0; r < kQuarters; r++) {
        const uint32_t c = part[r * kRadix + t];
        part[r * kRadix + t] = run;
        run += c;
      }
    }
    __syncthreads();
    uint32_t run = part[t];
#pragma unroll
    for (int w = 0; w < kShare; w++) {
      uint32_t *c = wcnt + (q * kShare + w) * kRadix + d;
      const uint32_t x = *c;
      *c = run;
      run += x;
    }
    __syncthreads();
    const bool last = shift + 8 >= lo + bits;
#pragma unroll
    for (int it = 0; it < IT; it++) {
      if (dg[it] == kNoDigit) continue;
      (last ? keys : buf)[wc[dg[it]] + lr[it]] = kk[it];
    }
    if (last) break;
    __syncthreads();
#pragma unroll
    for (int it = 0; it < IT; it++) {
      const uint32_t o = tile_offset<IT>(it);
      if (o < n) kk[it] = buf[o];
    }
  }
}

template <int IT>
cudaError_t sort_block(uint64_t *keys, uint64_t n, int lo, int bits, const uint32_t *d_n,
                       cudaStream_t s) {
  static std::atomic<uint64_t> done{0};  // one bit per device below 64
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev >= 64 || !((done.load(std::memory_order_relaxed) >> dev) & 1)) {
    e = cudaFuncSetAttribute(k_sort_block<IT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)block_sort_smem<IT>());
    if (e != cudaSuccess) return e;
    if (dev < 64) done.fetch_or(1ull << dev, std::memory_order_relaxed);
  }
  SST_LAUNCH_PDL_NB("k_sort_block", 16 * n, k_sort_block<IT>, 1, kBlockThreads,
                    (block_sort_smem<IT>()), s, keys, n, lo, bits, d_n);
  return cudaGetLastError();
}

}  // namespace

size_t radix_sort_scratch_bytes(uint64_t n) {
  const uint64_t tile = n <= kSmallTileKeys ? (uint64_t)kThreads * kSmallItems
                        : n <= kMidTileKeys ? (uint64_t)kThreads * kMidItems
                                            : kTile;
  uint64_t nblocks = (n + tile - 1) / tile;
  uint64_t hn = nblocks * kRadix;
  // the one-sweep form: digit totals and up to eight passes' tile status;
  // the longer sorts' counts and their scan
  const size_t os = 8 * kRadix * 4 + 8 * os_status_words((uint32_t)nblocks) * 4 + 512;
  const size_t cnt = 2 * ((hn * 4 + 255) & ~size_t(255)) + scan_scratch_bytes(hn, 4) + 512;
  return os > cnt ? os : cnt;
}

// profiler name of a one-sweep pass, by its tile size
template <bool KV, int IT>
constexpr const char *scatter_os_name() {
  if constexpr (IT == kSmallItems)
    return KV ? "(k_scatter_os<true, 4>)" : "(k_scatter_os<false, 4>)";
  else if constexpr (IT == kMidItems)
    return KV ? "(k_scatter_os<true, 8>)" : "(k_scatter_os<false, 8>)";
  else
    return KV ? "(k_scatter_os<true, 16>)" : "(k_scatter_os<false, 16>)";
}

// The multi-tile sort with tiles of IT items per thread (see radix_sort_impl).
template <int IT>
static cudaError_t radix_sort_tiles(uint64_t *keys, uint64_t *tmp, uint32_t *vals,
                                    uint32_t *vtmp, uint64_t n, int lo, int bits, Arena &arena,
                                    cudaStream_t s, uint64_t **result,
                                    uint32_t **vresult, const uint32_t *d_n,
                                    const SortDigits *pre) {
  constexpr int TILE = kThreads * IT;
  const uint32_t nblocks = (uint32_t)((n + TILE - 1) / TILE);
  if (vals) {
    cudaError_t e = scatter_smem_optin();
    if (e != cudaSuccess) return e;
  }
  uint64_t *src = keys, *dst = tmp;
  uint32_t *vsrc = vals, *vdst = vtmp;
  const int passes = (bits + 7) / 8;
  if (n < kOneSweepKeys) {
    // one sweep: all passes' digit totals in one read, then one launch a
    // pass whose tiles find their offsets by looking back
    uint32_t *totals, *status;
    const uint64_t sw = os_status_words(nblocks);
    if (pre) {  // counted by the caller, status words cleared
      if (pre->passes != passes || pre->status_words != (uint64_t)passes * sw)
        return cudaErrorInvalidValue;
      totals = pre->totals;
      status = pre->status;
    } else {
      totals = arena.take<uint32_t>(8 * kRadix);
      status = arena.take<uint32_t>((uint64_t)passes * sw);
      if (!totals || !status) return cudaErrorMemoryAllocation;
      cudaError_t e = cudaMemsetAsync(totals, 0, (size_t)passes * kRadix * 4, s);
      if (e != cudaSuccess) return e;
      SST_LAUNCH_PDL_NB("(k_hist_all)", 8 * n, k_hist_all<IT>, nblocks, kThreads, 0, s, src, n,
                    lo, passes, totals, status, (uint64_t)passes * sw, d_n);
    }
    for (int p = 0; p < passes; p++) {
      const uint64_t sb = (vals ? 24 : 16) * n + 8 * (uint64_t)kRadix * nblocks;
      if (vals)
        SST_LAUNCH_PDL_NB((scatter_os_name<true, IT>()), sb, (k_scatter_os<true, IT>), nblocks,
                      kThreads, (scatter_smem_bytes<true, IT>()), s, src, dst, n, lo + 8 * p,
                      totals + p * kRadix, status + (uint64_t)p * sw, vsrc, vdst, d_n);
      else
        SST_LAUNCH_PDL_NB((scatter_os_name<false, IT>()), sb, (k_scatter_os<false, IT>), nblocks,
                      kThreads, (scatter_smem_bytes<false, IT>()), s, src, dst, n, lo + 8 * p,
                      totals + p * kRadix, status + (uint64_t)p * sw, vsrc, vdst, d_n);
      std::swap(src, dst);
      std::swap(vsrc, vdst);
    }
  } else if constexpr (IT == kItems) {
    // counts and their scan in separate tables (the single-pass scan runs
    // out of place)
    const uint64_t hn = (uint64_t)nblocks * kRadix;
    // every scatter reads and writes keys (and values) and reads the counts
    const uint64_t hist_bytes = 8 * n + 4 * hn;
    const uint64_t scatter_bytes = (vals ? 24 : 16) * n + 8 * hn;
    uint32_t *cnts = arena.take<uint32_t>(hn);
    uint32_t *hist = arena.take<uint32_t>(hn);
    if (!cnts || !hist) return cudaErrorMemoryAllocation;
    for (int shift = lo; shift < lo + bits; shift += 8) {
      SST_LAUNCH_PDL_B(hist_bytes, k_hist, nblocks, kThreads, 0, s, src, n, shift, cnts, d_n);
      size_t mark = arena.used;
      cudaError_t e = scan<uint32_t, OpAdd>(cnts, hist, hn, 0u, OpAdd{}, true,
                                            false, nullptr, arena, s);
      arena.used = mark;
      if (e != cudaSuccess) return e;
      if (vals)
        SST_LAUNCH_PDL_B(scatter_bytes, k_scatter<true>, nblocks, kThreads,
                         (scatter_smem_bytes<true, kItems>()), s, src, dst, n, shift, hist, vsrc,
                         vdst, d_n);
      else
        SST_LAUNCH_PDL_B(scatter_bytes, k_scatter<false>, nblocks, kThreads,
                         (scatter_smem_bytes<false, kItems>()), s, src, dst, n, shift, hist, vsrc,
                         vdst, d_n);
      std::swap(src, dst);
      std::swap(vsrc, vdst);
    }
  } else {
    return cudaErrorInvalidValue;  // shorter sorts take the one-sweep form
  }
  *result = src;
  if (vresult) *vresult = vsrc;
  return cudaGetLastError();
}

// items a thread of the multi-tile form
static int sort_items(uint64_t n, bool vals) {
  if (!vals && n <= kSmallTileKeys) return kSmallItems;
  return n <= kMidTileKeys ? kMidItems : kItems;
}
// the form radix_sort_impl takes: 0 none (n < 2), 1 one CTA, 2 tiles
static int sort_form(uint64_t n, int bits, bool vals) {
  if (n < 2 || bits <= 0) return 0;
  if (!vals && n <= (uint64_t)kSmallSort) return 1;
  if (vals && n <= (uint64_t)kSmallSortKV) return 1;
  return 2;
}

bool radix_sort_digits(uint64_t n, int bits, Arena &arena, SortDigits *d) {
  const int form = sort_form(n, bits, false);
  const int passes = (bits + 7) / 8;
  if (form < 2 || n >= kOneSweepKeys) return false;
  const uint64_t tile = (uint64_t)kThreads * sort_items(n, false);
  const uint64_t sw = os_status_words((uint32_t)((n + tile - 1) / tile));
  d->totals = arena.take<uint32_t>(8 * kRadix);
  d->status = arena.take<uint32_t>((uint64_t)passes * sw);
  d->status_words = (uint64_t)passes * sw;
  d->passes = passes;
  return d->totals && d->status;
}

static cudaError_t radix_sort_impl(uint64_t *keys, uint64_t *tmp,
                                   uint32_t *vals, uint32_t *vtmp, uint64_t n,
                                   int lo, int bits, Arena &arena, cudaStream_t s,
                                   uint64_t **result, uint32_t **vresult,
                                   const uint32_t *d_n, const SortDigits *pre = nullptr) {
  *result = keys;
  if (vresult) *vresult = vals;
  if (n < 2 || bits <= 0) return cudaSuccess;
  if (pre && (vals || sort_form(n, bits, false) < 2)) return cudaErrorInvalidValue;
  if (!vals && n <= (uint64_t)kSmallSort) {
    if (n <= kBlockThreads) return sort_block<1>(keys, n, lo, bits, d_n, s);
    if (n <= 2 * kBlockThreads) return sort_block<2>(keys, n, lo, bits, d_n, s);
    if (n <= 4 * kBlockThreads) return sort_block<4>(keys, n, lo, bits, d_n, s);
    return sort_block<8>(keys, n, lo, bits, d_n, s);
  }
  if (vals && n <= (uint64_t)kSmallSortKV) {
    SST_LAUNCH_PDL_B(24 * n, k_sort_small<kSmallSortKV>, 1, kThreads, 0, s, keys, vals,
               n, bits, d_n);
    return cudaGetLastError();
  }
  auto tiles = [&](auto items) {
    return radix_sort_tiles<decltype(items)::value>(keys, tmp, vals, vtmp, n, lo, bits, arena, s,
                                                    result, vresult, d_n, pre);
  };
  switch (sort_items(n, vals != nullptr)) {
    case kSmallItems: return tiles(std::integral_constant<int, kSmallItems>{});
    case kMidItems: return tiles(std::integral_constant<int, kMidItems>{});
    default: return tiles(std::integral_constant<int, kItems>{});
  }
}

cudaError_t radix_sort_u64(uint64_t *keys, uint64_t *tmp, uint64_t n, int bits,
                           Arena &arena, cudaStream_t s, uint64_t **result,
                           const uint32_t *d_n, const SortDigits *pre, int lo) {
  return radix_sort_impl(keys, tmp, nullptr, nullptr, n, lo, bits, arena, s, result,
                         nullptr, d_n, pre);
}

cudaError_t radix_sort_kv(uint64_t *keys, uint64_t *tmp, uint32_t *vals,
                          uint32_t *vtmp, uint64_t n, int bits, Arena &arena,
                          cudaStream_t s, uint64_t **result, uint32_t **vresult) {
  return radix_sort_impl(keys, tmp, vals, vtmp, n, 0, bits, arena, s, result,
                         vresult, nullptr);
}

}  // namespace sst
