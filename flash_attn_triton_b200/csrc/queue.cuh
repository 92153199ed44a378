// Work queue of the persistent kernels with a queue entry per CTA at the start: a CTA's first candidate is its own index;
// `counter[0]` hands out the others, `counter[1]` counts the CTAs that have finished.  The last one to finish puts both back to
// zero, so a launch always finds them at zero.  A launch without others (ncand <= gridDim.x) does not touch them.  Which pair a launch
// has: queue_slots.h.
#pragma once

namespace fa {

__device__ __forceinline__ unsigned int queue_draw(unsigned int* counter, int ncand) {
  return ncand <= (int)gridDim.x ? (unsigned int)ncand : gridDim.x + atomicAdd(&counter[0], 1u);
}

// The CTA's next item, for a whole warp: candidates are drawn until `decode` takes one; false behind the last.  c is the candidate looked at
// last, at first the CTA's index: it stays with the caller between items, whatever became of the candidate.
// counter null: no queue, CTA i takes i, i + gridDim.x, i + 2 gridDim.x, ...
template <typename F>
__device__ __forceinline__ bool queue_item(unsigned int* counter, int ncand, bool first, int& c, int lane, F decode) {
  for (bool drawn = !first;; drawn = true) {
    if (drawn) {
      unsigned int u = 0;
      if (lane == 0) u = counter == nullptr ? gridDim.x + c : queue_draw(counter, ncand);
      c = (int)min(__shfl_sync(0xffffffffu, u, 0), (unsigned int)ncand);
    }
    if (c >= ncand) return false;
    if (decode(c)) return true;
  }
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
