// Delays in chosen element-wise warps, to show that results do not depend on which warps of a CTA are late.  Compiled in only
// with -DFA_SKEW (a tagged side build, never the shipped library), where fa_debug_skew(mode) chooses the warps:
//   0 none   1 group A (warps 0-3)   2 group B (warps 4-7)   3 one warp, another one for each tile   4 a quarter, scattered
// A delay is longer than a tile takes, and ends by itself.
#pragma once

#ifdef FA_SKEW
namespace fa {
__device__ int g_skew_mode;
__device__ __forceinline__ void skew(int warp, int step, int point) {
  const int mode = *reinterpret_cast<volatile int*>(&g_skew_mode);
  const bool late = mode == 1   ? warp < 4
                    : mode == 2 ? warp >= 4
                    : mode == 3 ? (step + point) % 8 == warp
                                : mode == 4 && ((step * 8 + warp * 5 + point) * 0x9E3779B1u >> 30) == 0;
  if (!late) return;
  const long long t0 = clock64();
  while (clock64() - t0 < 6000) __nanosleep(100);
}
}  // namespace fa
extern "C" int fa_debug_skew(int mode) { return (int)cudaMemcpyToSymbol(fa::g_skew_mode, &mode, sizeof(mode)); }
#define SKEW(warp, step, point) fa::skew(warp, step, point)
#else
#define SKEW(warp, step, point) do {} while (0)
#endif
