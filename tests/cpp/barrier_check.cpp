// Every barrier of a search's grid holds its blocks until the last has arrived,
// over more barriers than 32 bits of arrivals count.
#include <cstdio>
#include <initializer_list>

#include "../../sstgraph_gb300/csrc/gridbarrier.h"

int main() {
  for (unsigned int blocks : {1u, 7u, 288u, 304u}) {
    sst::BarrierCount target = 0;
    const unsigned long long steps = (1ull << 32) / blocks + 2000;
    unsigned long long k = 0;
    if (blocks < 288) {  // from just before the 32-bit end
      k = (1ull << 32) / blocks - 1000;
      target = k * blocks;
    }
    for (; k < steps; k++) {
      target = sst::barrier_next(target, blocks);
      const unsigned long long before = k * blocks;
      if (sst::barrier_complete(before, target) ||
          sst::barrier_complete(before + blocks - 1, target) ||
          !sst::barrier_complete(before + blocks, target) ||
          !sst::barrier_complete(before + 2ull * blocks - 1, target)) {
        printf("barrier %llu of %u blocks\n", k, blocks);
        return 1;
      }
    }
  }
  printf("barrier ok\n");
  return 0;
}
