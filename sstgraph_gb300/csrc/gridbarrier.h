// The arithmetic of a grid barrier (bfslevels.cuh), apart from CUDA so that the
// host can check it.
#pragma once

#ifdef __CUDACC__
#define SST_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define SST_HOST_DEVICE inline
#endif

namespace sst {

// Arrivals, counted over a kernel's whole run.  A search takes a barrier or
// more a level and its grid has up to some 290 blocks, so 32 bits pass their
// end after 15 million levels (a path of as many vertices) and a block would
// leave a barrier before the others arrive; 64 bits do not end.
using BarrierCount = unsigned long long;

// arrivals that complete the barrier after the one that `target` completed
SST_HOST_DEVICE BarrierCount barrier_next(BarrierCount target, unsigned int blocks) {
  return target + blocks;
}
// whether every block has arrived
SST_HOST_DEVICE bool barrier_complete(BarrierCount count, BarrierCount target) {
  return count >= target;
}

}  // namespace sst
