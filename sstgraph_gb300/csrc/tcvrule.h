// How triangles at listed vertices cut their work, apart from CUDA so that the
// host can check it.
#pragma once
#include <cstdint>

namespace sst {

// Leaves a chunk, by the pair slots of the call.  A few queries, whose chunks are
// all in flight at once, end when the longest chunk does (2 to 3 us a leaf of
// dependent probes); many have chunks to spare and pay for each one's search among
// the pairs.  Pass 3 at RMAT scale 18 (us, by leaves a chunk; last, a warp a chunk
// of 32):
//   vertices    1     2     4     8    32    warp
//   100        17    23    34    51    81     42
//   1,000      62    56    57    72   141     91
//   10,000    650   526   483   508   668    699
//   100,000  5255  4184  3722  3724  4653   5366
inline uint32_t tcv_chunk_leaves(uint64_t nslots) {
  return nslots <= 1 << 17 ? 2 : nslots <= 1 << 20 ? 4 : nslots <= 1 << 22 ? 8 : 32;
}

// Whether the chunks of all slots are added up in 64 bits.  Short chunks are many:
// 2^22 slots, a vertex of 92,000 neighbours listed 46 times, hold 2^32 chunks of 8
// leaves if all those neighbours have as many.  Above 2^22 slots 8 bytes more a slot
// would be felt, and chunks of 32 leaves in 32 bits are what that many have always had.
inline bool tcv_wide(uint64_t nslots) { return nslots <= 1 << 22; }

}  // namespace sst
