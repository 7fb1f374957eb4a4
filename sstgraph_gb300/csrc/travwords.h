// The few words every traversal of a graph uses, allocated all together or not
// at all.  Apart from CUDA, so that the host can check it with allocations that
// fail.
#pragma once
#include <cstddef>
#include <cstdint>

namespace sst {

struct TravWords {
  uint64_t *h_small = nullptr;            // pinned readback slots
  unsigned long long *d_small = nullptr;  // device counters
  void *d_bfs = nullptr;                  // a search's control block, zero between searches
};
constexpr size_t kTravWords = 64;  // of h_small and of d_small

// rt: pinned(void **, bytes), device(void **, bytes) and zero(void *, bytes),
// each false on failure, and free_pinned(void *), free_device(void *)
template <class Rt>
inline void trav_words_free(TravWords *w, Rt &&rt) {
  if (w->h_small) rt.free_pinned(w->h_small);
  if (w->d_small) rt.free_device(w->d_small);
  if (w->d_bfs) rt.free_device(w->d_bfs);
  *w = TravWords{};
}
template <class Rt>
inline bool trav_words_init(TravWords *w, size_t search_bytes, Rt &&rt) {
  void *h = nullptr, *d = nullptr, *b = nullptr;
  bool ok = rt.pinned(&h, kTravWords * sizeof(uint64_t));
  w->h_small = ok ? static_cast<uint64_t *>(h) : nullptr;
  ok = ok && rt.device(&d, kTravWords * sizeof(unsigned long long));
  w->d_small = ok ? static_cast<unsigned long long *>(d) : nullptr;
  ok = ok && rt.device(&b, search_bytes);
  w->d_bfs = ok ? b : nullptr;
  ok = ok && rt.zero(b, search_bytes);
  if (!ok) trav_words_free(w, rt);
  return ok;
}

}  // namespace sst
