// Delays in chosen warps, to show that results do not depend on which warps of a CTA are late.  Compiled in only
// with -DFA_SKEW (a tagged side build, never the shipped library), where fa_debug_skew(mode) chooses the warps:
//   0 none   1 the first half of the warps   2 the second half   3 one warp, another one for each tile   4 a quarter, scattered
// of those that a kernel names (backward: the element-wise warps; forward with two CTAs per SM: all, softmax warps first).  A delay is longer than a
// tile takes, and ends by itself.  A translation unit defines SKEW_TAG before including this header; fa::skew_mode_<tag>() sets its mode.
#pragma once

#ifdef FA_SKEW
#define SKEW_CAT2(a, b) a##b
#define SKEW_CAT(a, b) SKEW_CAT2(a, b)
namespace fa {
static __device__ int g_skew_mode;
static __device__ __forceinline__ void skew(int warp, int warps, int step, int point) {
  const int mode = *reinterpret_cast<volatile int*>(&g_skew_mode);
  const bool late = mode == 1   ? warp < warps / 2
                    : mode == 2 ? warp >= warps / 2
                    : mode == 3 ? (step + point) % warps == warp
                                : mode == 4 && ((step * warps + warp * 5 + point) * 0x9E3779B1u >> 30) == 0;
  if (!late) return;
  const long long t0 = clock64();
  while (clock64() - t0 < 6000) __nanosleep(100);
}
int SKEW_CAT(skew_mode_, SKEW_TAG)(int mode) { return (int)cudaMemcpyToSymbol(g_skew_mode, &mode, sizeof(mode)); }
}  // namespace fa
#define SKEW(warp, warps, step, point) fa::skew(warp, warps, step, point)
#else
#define SKEW(warp, warps, step, point) do {} while (0)
#endif
