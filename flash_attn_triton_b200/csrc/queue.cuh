// Work queue of the persistent kernels with a queue entry per CTA at the start: a CTA's first candidate is its own index;
// `counter[0]` hands out the others, `counter[1]` counts the CTAs that have finished.  The last one to finish puts both back to
// zero, so a launch always finds them at zero.  A launch without others (ncand <= gridDim.x) does not touch them.  Which pair a launch
// has: queue_slots.h.
#pragma once

namespace fa {

__device__ __forceinline__ unsigned int queue_draw(unsigned int* counter, int ncand) {
  return ncand <= (int)gridDim.x ? (unsigned int)ncand : gridDim.x + atomicAdd(&counter[0], 1u);
}

// The candidate behind c, the one that this CTA looked at last whatever became of it, for a whole warp; ncand or more: there is none.
// counter null: no queue, CTA i takes i, i + gridDim.x, i + 2 gridDim.x, ...
__device__ __forceinline__ int queue_next(unsigned int* counter, int ncand, int c, int lane) {
  if (counter == nullptr) return c + gridDim.x;
  return (int)__shfl_sync(0xffffffffu, lane == 0 ? queue_draw(counter, ncand) : 0u, 0);
}
// One thread of a CTA that has drawn its last candidate (or has given up on a wait and draws no more).
__device__ __forceinline__ void queue_finish(unsigned int* counter, int ncand) {
  if (ncand <= (int)gridDim.x) return;
  __threadfence();
  const unsigned int done = atomicAdd(&counter[1], 1u);
  if (done == gridDim.x - 1) {
    counter[0] = 0u;
    counter[1] = 0u;
    __threadfence();
  }
}

}  // namespace fa
