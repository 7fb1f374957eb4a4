// A graph's traversal words when an allocation fails: none stays allocated, no
// pointer stays set and nothing is written through one.
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "../../sstgraph_gb300/csrc/travwords.h"

struct Rt {
  int fail, step = 0, live = 0;
  bool take(void **p, size_t bytes) {
    if (step++ == fail) return false;  // *p stays as it was, as with cudaMalloc
    *p = malloc(bytes);
    memset(*p, 0xAB, bytes);
    live++;
    return true;
  }
  bool pinned(void **p, size_t bytes) { return take(p, bytes); }
  bool device(void **p, size_t bytes) { return take(p, bytes); }
  bool zero(void *p, size_t bytes) {
    if (!p) abort();
    if (step++ == fail) return false;
    memset(p, 0, bytes);
    return true;
  }
  void free_pinned(void *p) { live--, free(p); }
  void free_device(void *p) { live--, free(p); }
};

int main() {
  for (int fail = 0; fail <= 4; fail++) {
    Rt rt{fail};
    sst::TravWords w;
    const bool ok = sst::trav_words_init(&w, 200, rt);
    if (ok != (fail == 4)) return 1;
    if (!ok && (w.h_small || w.d_small || w.d_bfs || rt.live)) return 2;
    if (ok) {
      for (int i = 0; i < 200; i++)
        if (static_cast<char *>(w.d_bfs)[i]) return 3;
      sst::trav_words_free(&w, rt);
      if (rt.live || w.d_bfs) return 4;
    }
  }
  printf("words ok\n");
  return 0;
}
