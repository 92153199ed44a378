// Row statistics of the dK/dV kernels as GEMM operands.
//
// A thread of those kernels owns a key, and -lse2 and -delta belong to the query rows, which are the columns of its
// tiles: added in the element-wise warps they would cost 128 shared-memory loads per thread and tile.  One more MMA
// step of 16 columns adds them in the tensor pipe instead, from a 128 x 16 operand per query tile.  Its elements have
// 16 bits, so each statistic is the sum of three of them: 24 significant bits, as in fp32.  In fp16 the first piece
// counts 2^14 times, which carries values up to 2^28 (one piece ends at 65504; with loss scaling, or values far from
// zero, |delta| passes that) and gives NaN above.  bf16 has the range of fp32.
//
//   query side, scores:  [t0 t0 t0 t1 t1 t1 t2 t2]   t = -lse2 2^e
//   key side, scores:    [kTop (v0 v1 v2) v0 v1 v2 v0 v1]   v = 2^-e / scale_log2, 1 <= v < 2
//   query side, dP:      [d0 d1 d2 0 0 0 0 0]        d = -delta
//   key side, dP:        [kTop 1 1 0 0 0 0 0]
//
// (the products left out are below 2^-44 of the whole), so the score GEMM yields S - lse2 / scale_log2 and the dP GEMM
// dP - delta.  The two halves of a query tile's operand are read by different GEMMs, with a half of zeros as the other
// eight columns: a delta that is not finite reaches dP alone.
//
// Against fp32 statistics (the mma.sync kernels) gradients at 64 to 255 tokens differ from float64 by the same
// 3.1e-4 (fp16) and 2.5e-3 (bf16) to the third digit.
#pragma once
#include "common.cuh"
#include "sm100.cuh"

namespace fa {

template <typename T> struct StatTop { static constexpr float value = 1.f; };
template <> struct StatTop<__half> { static constexpr float value = 16384.f; };

// Half of an operand: 8 columns of 128 rows, 16 bytes per row (core matrices of 8 rows follow each other).  An operand
// block is two halves; a query tile's block holds the scores' half and the dP half, a key-side block its half and zeros.
constexpr int kStatHalf = 128 * 16;
constexpr int kStatBlock = 2 * kStatHalf;

// Key-side blocks at keys (scores, then dP), by all threads of the CTA.
template <typename T> __device__ __forceinline__ void stat_write_keys(unsigned char* keys, float scale_log2, int tid, int nt) {
  constexpr float top = StatTop<T>::value;
  const float w = 1.f / scale_log2;
  const float v = __int_as_float((__float_as_int(w) & 0x007fffff) | 0x3f800000);       // 1 <= v < 2
  const float v0 = Elem<T>::to_f(Elem<T>::from_f(v)), v1 = Elem<T>::to_f(Elem<T>::from_f(v - v0)), v2 = v - v0 - v1;
  const uint4 score = make_uint4(Elem<T>::pack(top * v0, top * v1), Elem<T>::pack(top * v2, v0), Elem<T>::pack(v1, v2),
                                 Elem<T>::pack(v0, v1));
  const uint4 dp = make_uint4(Elem<T>::pack(top, 1.f), Elem<T>::pack(1.f, 0.f), 0u, 0u);
  uint4* k4 = reinterpret_cast<uint4*>(keys);
  for (int i = tid; i < 2 * kStatBlock / 16; i += nt)
    k4[i] = i < 128 ? score : (i >= kStatBlock / 16 && i < kStatBlock / 16 + 128) ? dp : make_uint4(0u, 0u, 0u, 0u);
}
// 2^e of the scores' statistics.
__device__ __forceinline__ float stat_score_unit(float scale_log2) {
  return __int_as_float(__float_as_int(1.f / scale_log2) & 0x7f800000);
}

// t of a row that sees no key, or does not exist: P = 0.  Not infinite: the pieces of an infinity add up to NaN.
constexpr float kStatNoKey = -1e8f;

// One row of a query tile's block.  Both statistics are split as a pair.
template <typename T, bool kScores>
__device__ __forceinline__ void stat_write_row(unsigned char* block, int row, float neg_lse2, float neg_delta, float unit) {
  constexpr float top = StatTop<T>::value;
  const float t = !kScores ? 0.f : isinf(neg_lse2) ? kStatNoKey : neg_lse2 * unit;
  const uint32_t p0 = Elem<T>::pack(t * (1.f / top), neg_delta * (1.f / top));
  const float2 f0 = Elem<T>::unpack(p0);
  const float2 r0 = make_float2(fmaf(-top, f0.x, t), fmaf(-top, f0.y, neg_delta));
  const uint32_t p1 = Elem<T>::pack(r0.x, r0.y);
  const float2 f1 = Elem<T>::unpack(p1);
  const uint32_t p2 = Elem<T>::pack(r0.x - f1.x, r0.y - f1.y);
  if (kScores)
    reinterpret_cast<uint4*>(block)[row] = make_uint4(__byte_perm(p0, p0, 0x1010), __byte_perm(p0, p1, 0x5410),
                                                      __byte_perm(p1, p1, 0x1010), __byte_perm(p2, p2, 0x1010));
  reinterpret_cast<uint4*>(block + kStatHalf)[row] = make_uint4(__byte_perm(p0, p1, 0x7632), p2 >> 16, 0u, 0u);
}

// Descriptors; keys = address of the key-side blocks, whose second half is zero, block = of a query tile's, below keys.
__device__ __forceinline__ uint64_t stat_desc_key(uint32_t keys, bool dp) {
  return sm100::make_smem_desc_noswizzle(keys + (dp ? kStatBlock : 0), kStatHalf, 128);
}
__device__ __forceinline__ uint64_t stat_desc_query(uint32_t keys, uint32_t block, bool dp) {
  const uint32_t half = block + (dp ? kStatHalf : 0);
  return sm100::make_smem_desc_noswizzle(half, keys + kStatHalf - half, 128);
}

}  // namespace fa
