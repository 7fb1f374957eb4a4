// The chunks of triangles at listed vertices are added up without wrapping,
// whatever the lists' lengths (2^28 leaves is the longest row).
#include <cstdio>

#include "../../sstgraph_gb300/csrc/tcvrule.h"

int main() {
  uint32_t last = 1;
  for (uint64_t slots = 32; slots <= 1ull << 26; slots += 32 + slots / 64 * 32) {
    const uint32_t c = sst::tcv_chunk_leaves(slots);
    if (c < last) return 1;
    last = c;
    for (uint64_t leaves = 1; leaves <= 1ull << 28; leaves *= 2) {
      const unsigned __int128 sum = (unsigned __int128)slots * ((leaves + c - 1) / c);
      if (!sst::tcv_wide(slots) && c < 32) return 2;
      if (sst::tcv_wide(slots) && sum >> 64) return 3;
    }
  }
  printf("rule ok\n");
  return 0;
}
