// KV-cache decode: attention over a paged (or contiguous) cache with the in-place append and the rotary
// embedding fused in.  HBM-bound: the job of the kernel is to stream every cached K/V byte exactly once at
// full bandwidth.
//
//   Work.  A unit is (sequence, kv head, group of 8 or 16 query rows): one K/V byte serves the whole
//   GQA group.  The products are taken transposed, S^T = K Q^T and O^T = V^T P^T, with the keys (the head
//   dimension) as the M=16 side of mma.sync m16n8k16 and the query rows as its N=8 side: with 4 or 8
//   query rows per kv head, as in grouped-query decoding, that is half the products, exponentials
//   and registers of query rows padded to 16.  A sequence has one work tile per 64 keys and is cut into
//   pieces of equal size; a CTA takes a piece of one unit.  The piece size follows from the lengths, which are on the
//   device, so every warp works it out (see the kernel): a grid of (split, head, sequence) sized for the capacity of the cache has long
//   pieces, a last wave that is nearly empty, and CTAs without work.  The U heads and row groups
//   of a piece are neighbouring CTAs, which walk the same cache pages at the same time.
//   Pipeline.  4 warps take 16 keys of a tile each.  Every warp has a 3-stage cp.async ring of its own
//   (16-byte row gathers), so that the warps never wait for one another before they merge at the end.
//   With 16-row products, a barrier per tile and the score options tested per element the compute of
//   two CTAs per SM, not the memory, set the pace: 702 to 850 us for a 64-sequence step over
//   4.3 GB of cache against 660 us now, 0.99 of the measured copy rate (calls in a row, value checks on or off: 670).
//   Append.  The new tokens (k_new rotated, v_new) never come from the cache: the CTA whose tile holds
//   their positions puts them into the staged tile itself, and the one of row group 0 also writes
//   them to their cache slots -- one writer per (sequence, kv head, token), no separate launch.
//   Merge.  A unit of one piece is written straight to the output.  Otherwise its pieces go to
//   the workspace with their base-2 LSEs and the CTA that finishes last merges them, always in the
//   same order.
//   Latency.  A small step is one chain: lengths, piece, tiles and Q, the append, the merge of the warps, the merge of the
//   pieces.  So Q and the new tokens are read and rotated 16 bytes at a time (they came element by element), what the
//   append reads is fetched to L1 under the first tiles, and the warps write their outputs side by side and add them up after
//   one barrier (not in four turns).  Kernel time, before -> after (us): 1 x 1900 tokens, 32 heads over 8 of 128: 15.1 -> 11.9;
//   28 x 66 to 2112, 8 over 2: 20.0 -> 15.0; 47 x 192, 2 new tokens, 32 over 8 of 64: 22.5 -> 16.8; 4 x 600 to 2400, 4 new
//   tokens, 16 over 4 of 128: 34.7 -> 20.7; 17 x 18450, 8 over 2: 69.0 -> 63.1.
//   Value checks of the public call run at the start of the same kernel while the tables are small (one
//   decode step of a few sequences is bounded by launches: 17 small kernels, a copy and a
//   synchronisation took 150 us around a 16 us kernel), in decode_check_kernel otherwise.
#include <sched.h>

#include <atomic>
#include <cmath>
#include <mutex>
#include <type_traits>

#include "cache_geo.cuh"
#include "check_slots.h"
#include "common.cuh"

namespace fa {

constexpr int kTile = 64;             // keys per work tile
constexpr int kMaxBalanced = 512;     // sequences up to which every warp sums the lengths itself
constexpr int kOneWave = 64;          // largest piece, in tiles, that is still run in one wave of CTAs
constexpr int kWaves = 4;             // waves of CTAs beyond that

struct DecodeGeom {
  int shares;      // pieces the grid has room for
  int splits;      // 0: pieces sized on the device; else that many pieces of every sequence
  int resident;    // CTAs the GPU runs at a time
  int max_tiles;   // tiles of a full cache
  int row_groups;  // ceil(seqlen_q * group / rows of a unit)
  int page_shift;  // log2(page_size) or -1
};

// The value checks of one call: their result goes to a word in mapped host memory (bit 31 = done, low
// bits = fa_decode_check of the checks that failed), and to a word of the call's own workspace for the kernels
// behind them.  The host word is handed to the next call once the host has read it; the kernels read theirs until the
// last CTA has started, long after the call has returned, so no other call may write to it.
constexpr uint32_t kCheckDone = 0x80000000u;
constexpr int kInlineCheck = 1024;   // table entries up to which every attention CTA makes the checks itself
struct DecodeCheck {
  uint32_t* host;       // null = no checks in this kernel
  const uint32_t* dev;  // null, or the result of decode_check_kernel
};

// All checks, by the threads of one CTA; every thread gets the mask of those that failed.
__device__ __forceinline__ uint32_t decode_checks(const fa_decode_args& p, int tid, int nt) {
  uint32_t bad = 0;
  if (p.block_table) {
    const int n = p.batch * p.block_table_stride;
    for (int i = tid; i < n; i += nt)
      if ((unsigned)p.block_table[i] >= (unsigned)p.num_pages) bad |= FA_CHECK_PAGES;
  }
  const long long cap = p.block_table ? (long long)p.block_table_stride * p.page_size : p.page_size;
  for (int b = tid; b < p.batch; b += nt) {
    if (p.cache_batch_idx && (unsigned)p.cache_batch_idx[b] >= (unsigned)p.num_pages) bad |= FA_CHECK_ROWS;
    const int pad = p.cache_leftpad ? p.cache_leftpad[b] : 0;
    if (pad < 0) bad |= FA_CHECK_LEFTPAD;
    const int old = p.cache_seqlens[b];
    const long long last = (long long)old + (p.k_new ? p.seqlen_new : 0) + pad;
    if (old < 0 || last > cap) bad |= FA_CHECK_LENGTHS;
    if (p.rotary_cos && last > p.rotary_seqlen) bad |= FA_CHECK_ROTARY;
  }
  if (!__syncthreads_or(bad)) return 0u;
  return (__syncthreads_or(bad & FA_CHECK_PAGES) ? FA_CHECK_PAGES : 0u) |
         (__syncthreads_or(bad & FA_CHECK_ROWS) ? FA_CHECK_ROWS : 0u) |
         (__syncthreads_or(bad & FA_CHECK_LEFTPAD) ? FA_CHECK_LEFTPAD : 0u) |
         (__syncthreads_or(bad & FA_CHECK_LENGTHS) ? FA_CHECK_LENGTHS : 0u) |
         (__syncthreads_or(bad & FA_CHECK_ROTARY) ? FA_CHECK_ROTARY : 0u);
}

int cache_attention_sm100(const fa_decode_args& d, const void* q, const int64_t* q_stride, const CacheGeo& geo,
                          const ScoreCfg& cfg, cudaStream_t st);

__global__ void __launch_bounds__(1024) decode_check_kernel(const fa_decode_args p, uint32_t* host, uint32_t* dev) {
  const uint32_t bad = decode_checks(p, threadIdx.x, blockDim.x);
  if (threadIdx.x == 0) {
    if (dev) *dev = bad;
    *reinterpret_cast<volatile uint32_t*>(host) = bad | kCheckDone;
    __threadfence_system();
  }
}

template <typename T> __device__ __forceinline__ T hmul_rn(T a, T b);
template <> __device__ __forceinline__ __half hmul_rn(__half a, __half b) { return __hmul_rn(a, b); }
template <> __device__ __forceinline__ __nv_bfloat16 hmul_rn(__nv_bfloat16 a, __nv_bfloat16 b) { return __hmul_rn(a, b); }
template <typename T> __device__ __forceinline__ T hadd_rn(T a, T b);
template <> __device__ __forceinline__ __half hadd_rn(__half a, __half b) { return __hadd_rn(a, b); }
template <> __device__ __forceinline__ __nv_bfloat16 hadd_rn(__nv_bfloat16 a, __nv_bfloat16 b) { return __hadd_rn(a, b); }
template <typename T> __device__ __forceinline__ T hsub_rn(T a, T b);
template <> __device__ __forceinline__ __half hsub_rn(__half a, __half b) { return __hsub_rn(a, b); }
template <> __device__ __forceinline__ __nv_bfloat16 hsub_rn(__nv_bfloat16 a, __nv_bfloat16 b) { return __hsub_rn(a, b); }

// Rotary on element d of a head vector x (read through `get`), every product and sum
// rounded to T like the reference's eager arithmetic (flash_attn_interface.py:57-66).
// A position outside the table [0, rotary_seqlen) leaves the element unrotated (the host checks
// the lengths when validation is on; this keeps the read in bounds when it is off).
template <typename T, typename F>
__device__ __forceinline__ T rotary_elem(F get, int d, const T* cos, const T* sin, int pos,
                                         int rotary_dim, int interleaved, int rotary_seqlen) {
  if (d >= rotary_dim || pos < 0 || pos >= rotary_seqlen) return get(d);
  const int half = rotary_dim >> 1;
  int i, partner;
  bool first;
  if (interleaved) {
    i = d >> 1;
    first = (d & 1) == 0;
    partner = d ^ 1;
  } else {
    first = d < half;
    i = first ? d : d - half;
    partner = first ? d + half : d - half;
  }
  const T c = cos[(int64_t)pos * half + i], s = sin[(int64_t)pos * half + i];
  const T x = get(d), y = get(partner);
  // first: x*c - y*s ; second: y*s + x*c  (y = first element of the pair)
  return first ? hsub_rn(hmul_rn(x, c), hmul_rn(y, s)) : hadd_rn(hmul_rn(y, s), hmul_rn(x, c));
}

// Whether rotary_chunk() can read 16 (pairs side by side: 8) bytes of the tables at a time.
template <typename T>
__device__ __forceinline__ bool rotary_in_chunks(const T* cos, const T* sin, int rotary_dim, int interleaved) {
  return (rotary_dim & (interleaved ? 7 : 15)) == 0 &&
         ((reinterpret_cast<uintptr_t>(cos) | reinterpret_cast<uintptr_t>(sin)) & (interleaved ? 7 : 15)) == 0;
}

// The others: halves that are multiples of 4 by 8 bytes, the rest element by element.
template <typename T>
__device__ __forceinline__ uint4 rotary_chunk_any(const T* x, int d, const T* cos, const T* sin, int pos, int rotary_dim,
                                                  int interleaved, int rotary_seqlen) {
  union { uint4 v; uint2 h[2]; T e[8]; } out;
  const int half = rotary_dim >> 1;
  if (!interleaved && half % 4 == 0 && ((reinterpret_cast<uintptr_t>(cos) | reinterpret_cast<uintptr_t>(sin)) & 7) == 0) {
    union Four { uint2 v; T e[4]; };
    out.v = *reinterpret_cast<const uint4*>(x + d);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int at = d + 4 * h;
      if (at >= rotary_dim) break;
      const bool first = at < half;
      const int64_t i = (int64_t)pos * half + (first ? at : at - half);
      Four self, other, c, s;
      self.v = out.h[h];
      other.v = *reinterpret_cast<const uint2*>(x + (first ? at + half : at - half));
      c.v = *reinterpret_cast<const uint2*>(cos + i);
      s.v = *reinterpret_cast<const uint2*>(sin + i);
#pragma unroll
      for (int k = 0; k < 4; ++k)
        self.e[k] = first ? hsub_rn(hmul_rn(self.e[k], c.e[k]), hmul_rn(other.e[k], s.e[k]))
                          : hadd_rn(hmul_rn(other.e[k], s.e[k]), hmul_rn(self.e[k], c.e[k]));
      out.h[h] = self.v;
    }
    return out.v;
  }
#pragma unroll
  for (int k = 0; k < 8; ++k)
    out.e[k] = rotary_elem<T>([&](int j) { return x[j]; }, d + k, cos, sin, pos, rotary_dim, interleaved, rotary_seqlen);
  return out.v;
}
template <typename T>
__device__ __noinline__ uint4 rotary_chunk_call(const T* x, int d, const T* cos, const T* sin, int pos, int rotary_dim,
                                                int interleaved, int rotary_seqlen) {
  return rotary_chunk_any(x, d, cos, sin, pos, rotary_dim, interleaved, rotary_seqlen);
}

// 8 elements of a head row, rotated like rotary_elem.  kCall: the general case out of line.  In the main loop of decode_kernel
// it cost registers and the order of the loads (head_dim 256, 32 x 8000 tokens, 16 heads over 4: 268 us, 233 as a call); a
// kernel that only rotates and copies is better off without the call (4 x 256 tokens behind 300, 32 heads over 8 of 128, with
// their attention: 42 us, 46).  Pairs side by side need no row beside the one at hand and half as much of the tables: 8 x 900
// tokens, 4 new, 16 heads over 4 of 128: a thread per element 30.4 us, eight elements of a thread one by one 20.6, now 16.6.
template <typename T, bool kCall>
__device__ __forceinline__ uint4 rotary_chunk(const T* x, int d, const T* cos, const T* sin, int pos, int rotary_dim,
                                              int interleaved, int rotary_seqlen) {
  union { uint4 v; T e[8]; } out, self, other, c, s;
  self.v = *reinterpret_cast<const uint4*>(x + d);
  if (cos == nullptr || d >= rotary_dim || pos < 0 || pos >= rotary_seqlen) return self.v;
  if (!rotary_in_chunks(cos, sin, rotary_dim, interleaved)) {
    if (kCall) return rotary_chunk_call(x, d, cos, sin, pos, rotary_dim, interleaved, rotary_seqlen);
    return rotary_chunk_any(x, d, cos, sin, pos, rotary_dim, interleaved, rotary_seqlen);
  }
  const int half = rotary_dim >> 1;
  if (interleaved) {
    *reinterpret_cast<uint2*>(c.e) = *reinterpret_cast<const uint2*>(cos + (int64_t)pos * half + (d >> 1));
    *reinterpret_cast<uint2*>(s.e) = *reinterpret_cast<const uint2*>(sin + (int64_t)pos * half + (d >> 1));
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const T x0 = self.e[2 * k], x1 = self.e[2 * k + 1];
      out.e[2 * k] = hsub_rn(hmul_rn(x0, c.e[k]), hmul_rn(x1, s.e[k]));
      out.e[2 * k + 1] = hadd_rn(hmul_rn(x0, s.e[k]), hmul_rn(x1, c.e[k]));
    }
    return out.v;
  }
  const bool first = d < half;
  const int i = first ? d : d - half;
  other.v = *reinterpret_cast<const uint4*>(x + (first ? d + half : d - half));
  c.v = *reinterpret_cast<const uint4*>(cos + (int64_t)pos * half + i);
  s.v = *reinterpret_cast<const uint4*>(sin + (int64_t)pos * half + i);
#pragma unroll
  for (int k = 0; k < 8; ++k)
    out.e[k] = first ? hsub_rn(hmul_rn(self.e[k], c.e[k]), hmul_rn(other.e[k], s.e[k]))
                     : hadd_rn(hmul_rn(other.e[k], s.e[k]), hmul_rn(self.e[k], c.e[k]));
  return out.v;
}

__device__ __forceinline__ int64_t cache_row_offset(const fa_decode_args& p, int b, int pos,
                                                    int page_shift, const int64_t* stride) {
  int page, row;
  if (p.block_table) {
    int pi;
    if (page_shift >= 0) {
      pi = pos >> page_shift;
      row = pos & (p.page_size - 1);
    } else {
      pi = pos / p.page_size;
      row = pos - pi * p.page_size;
    }
    page = p.block_table[(int64_t)b * p.block_table_stride + pi];
  } else {
    page = p.cache_batch_idx ? p.cache_batch_idx[b] : b;
    row = pos;
  }
  return (int64_t)page * stride[0] + (int64_t)row * stride[1];
}

// ---------------------------------------------------------------------------------------
// attention
// ---------------------------------------------------------------------------------------
// Tiles of a sequence: nt work tiles from tile lo on.  Keys that no query row sees (left of the window)
// are skipped, new tokens never are: somebody has to append them.  An empty sequence has one
// (empty) tile, which writes its zeros.
struct SeqTiles {
  int len_old, len, lo, nt;
};
// Rows a sequence can hold behind its left padding: lengths are taken up to here and new tokens stored up to here, so
// that a call whose values are not checked stays inside its rows of the cache and of the table.
__host__ __device__ __forceinline__ int cache_capacity(const fa_decode_args& p) {
  const int64_t cap = p.block_table ? (int64_t)p.block_table_stride * p.page_size : p.page_size;
  return (int)(cap < (1 << 30) ? cap : (1 << 30));
}
__device__ __forceinline__ int seq_capacity(const fa_decode_args& p, int b) {
  return cache_capacity(p) - (p.cache_leftpad ? max(0, p.cache_leftpad[b]) : 0);
}
__device__ __forceinline__ SeqTiles seq_tiles(const fa_decode_args& p, const ScoreCfg& cfg, int max_tiles, int b) {
  SeqTiles s;
  s.len_old = max(0, min(p.cache_seqlens[b], seq_capacity(p, b)));
  s.len = s.len_old + (p.k_new ? p.seqlen_new : 0);
  const int first = cfg.wl >= 0 ? min(max(0, s.len - p.seqlen_q - cfg.wl), s.len_old) : 0;
  s.lo = first / kTile;
  s.nt = min(max(1, (s.len + kTile - 1) / kTile - s.lo), max_tiles);
  return s;
}

// Elements [d, d + 4) of one output row, merged from the `parts` workspace rows r0, r0 + step, ...  Eight
// pieces are loaded at a time, their common maximum taken first.  (Sixteen: longer code in front of few rows, -1 to
// +7 % of a step's time at every head size -- 2 x 411 tokens, one head of 64: 9.7 -> 10.6 us.)
constexpr int kMergeBatch = 8;
template <typename T, int D>
__device__ __forceinline__ void merge_pieces(const float* ws_o, const float* ws_l, int64_t r0, int64_t step, int parts, int d,
                                             T* og) {
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  float wsum = 0.f, m = -INFINITY;
  for (int i0 = 0; i0 < parts; i0 += kMergeBatch) {
    float l[kMergeBatch];
    float4 x[kMergeBatch];
#pragma unroll
    for (int j = 0; j < kMergeBatch; ++j) {
      const int i = i0 + j;
      const int64_t r = r0 + i * step;
      l[j] = i < parts ? ws_l[r] : -INFINITY;
      x[j] = i < parts ? *reinterpret_cast<const float4*>(ws_o + r * D + d) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    float mn = m;
#pragma unroll
    for (int j = 0; j < kMergeBatch; ++j) mn = fmaxf(mn, l[j]);
    // pieces without a finite score weigh 0, which a NaN in them survives
    const float mf = mn == -INFINITY ? 0.f : mn;
    const float sc = exp2f(m - mf);
    acc.x *= sc; acc.y *= sc; acc.z *= sc; acc.w *= sc;
    wsum *= sc;
    m = mn;
#pragma unroll
    for (int j = 0; j < kMergeBatch; ++j) {
      const float w = exp2f(l[j] - mf);
      wsum += w;
      acc.x += w * x[j].x; acc.y += w * x[j].y; acc.z += w * x[j].z; acc.w += w * x[j].w;
    }
  }
  const float inv = wsum > 0.f ? 1.f / wsum : 0.f;
  uint2 pk;
  pk.x = Elem<T>::pack(acc.x * inv, acc.y * inv);
  pk.y = Elem<T>::pack(acc.z * inv, acc.w * inv);
  *reinterpret_cast<uint2*>(og + d) = pk;
}

__device__ __forceinline__ uint32_t transpose_8x8(uint32_t x) {
  uint32_t y;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(y) : "r"(x));
  return y;
}

// kRows: query rows of a unit (8 or 16)
template <int D, int kRows> struct DecodeSmem {
  static constexpr int P = TilePitch<D>::value, NS = 3, OP = D + 4;
  static constexpr size_t ring = (size_t)2 * NS * kTile * P * 2;
  static constexpr size_t q_bytes = kRows * P * 2;
  static constexpr size_t fixed = ring + q_bytes + 4 * kRows * 2 * 4;     // Q rows; each warp's row maxima and sums
  static_assert((size_t)4 * kRows * OP * 4 <= ring, "the warps' outputs, over the ring");
};

template <typename T, int D, int kRows>
__global__ void __launch_bounds__(128, D <= 128 ? 2 : 1)
    decode_kernel(const fa_decode_args p, const ScoreCfg cfg, const DecodeGeom geo, const DecodeCheck chk) {
  using SM = DecodeSmem<D, kRows>;
  constexpr int P = SM::P, NT = 128, NS = SM::NS, OP = SM::OP, NB = kRows / 8;
  constexpr int CPR = D / 8, RPW = 32 / CPR, PASSES = 16 / RPW;     // a warp's loads: 16 rows of CPR 16-byte chunks
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* ring = reinterpret_cast<T*>(smem_raw);      // [stage][warp][K, V][16][P]
  float* sO = reinterpret_cast<float*>(smem_raw); // over the ring, when it is done with: 4 x kRows x OP
  T* sQ = reinterpret_cast<T*>(smem_raw + SM::ring);                       // kRows x P
  float* sM = reinterpret_cast<float*>(smem_raw + SM::ring + SM::q_bytes); // 4 x kRows
  float* sL = sM + 4 * kRows;                    // 4 x kRows

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  if (chk.host) {
    const uint32_t bad = decode_checks(p, tid, NT);
    if (tid == 0 && blockIdx.x == 0) {
      *reinterpret_cast<volatile uint32_t*>(chk.host) = bad | kCheckDone;
      __threadfence_system();
    }
    if (bad) return;
  } else if (chk.dev) {
    // launched while the check kernel may still run (programmatic dependent launch)
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (*chk.dev) return;
  }
  const int G = p.heads_q / p.heads_kv;
  const int R = p.seqlen_q * G;                  // query rows of a kv head: r = sq * G + gi
  const int U = p.heads_kv * geo.row_groups;     // units of a sequence
  const int u = blockIdx.x % U, share = blockIdx.x / U;
  const int hk = u / geo.row_groups, rg = u % geo.row_groups;

  // ---- this CTA's piece: tiles [tile0, tile0 + count) of sequence b ------------------------
  int b, tile0, count, parts, base;              // base: first of the `parts` pieces of the sequence
  SeqTiles w;
  if (geo.splits == 0) {
    // Every warp does this on its own, without shared memory or barriers (which cost a small step 2 to 4
    // us); lane i looks after the sequences [i per, (i + 1) per).
    const int per = (p.batch + 31) / 32, b0 = min(lane * per, p.batch), b1 = min(b0 + per, p.batch);
    int sum = 0, longest = 0;
    for (int i = b0; i < b1; ++i) {
      const int nt = seq_tiles(p, cfg, geo.max_tiles, i).nt;
      sum += nt;
      longest = max(longest, nt);
    }
    sum = __reduce_add_sync(0xffffffffu, sum);
    longest = __reduce_max_sync(0xffffffffu, longest);
    const int64_t work = (int64_t)sum * U;
    int size = (int)((work + geo.resident - 1) / geo.resident), mine = 0;
    auto count_pieces = [&]() {
      mine = 0;
      for (int i = b0; i < b1; ++i) mine += (seq_tiles(p, cfg, geo.max_tiles, i).nt + size - 1) / size;
    };
    if (size > kOneWave) {
      size = max(kOneWave / 2, (int)((work + kWaves * geo.resident - 1) / (kWaves * geo.resident)));
      count_pieces();
    } else {
      size = max(size, (int)ceilf((float)longest / ceilf(sqrtf(7.f * longest))));
      for (; size < longest; size += max(1, size >> 3)) {
        count_pieces();
        if (__reduce_add_sync(0xffffffffu, mine) * U <= geo.resident) break;
      }
    }
    if (size >= longest) {                       // every sequence in one piece
      if (share >= p.batch) return;
      b = base = share;
      parts = 1;
    } else {
      int inc = mine;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int x = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += x;
      }
      const bool owner = share >= inc - mine && share < inc;
      const unsigned who = __ballot_sync(0xffffffffu, owner);
      if (who == 0u) return;                       // the grid is sized for a full cache
      base = inc - mine;
      b = b0;
      parts = 0;
      if (owner) {
        for (;; ++b) {
          parts = (seq_tiles(p, cfg, geo.max_tiles, b).nt + size - 1) / size;
          if (share < base + parts) break;
          base += parts;
        }
      }
      const int src = __ffs(who) - 1;
      b = __shfl_sync(0xffffffffu, b, src);
      base = __shfl_sync(0xffffffffu, base, src);
      parts = __shfl_sync(0xffffffffu, parts, src);
    }
    w = seq_tiles(p, cfg, geo.max_tiles, b);
  } else {
    b = share / geo.splits;
    base = b * geo.splits;
    w = seq_tiles(p, cfg, geo.max_tiles, b);
    parts = min(geo.splits, w.nt);
    if (share - base >= parts) return;
  }
  const int len_old = w.len_old, len = w.len;
  tile0 = (int)((int64_t)(share - base) * w.nt / parts);
  count = (int)((int64_t)(share - base + 1) * w.nt / parts) - tile0;
  tile0 += w.lo;

  // ---- loading --------------------------------------------------------------------------
  const int lc = (lane % CPR) * 8, lr = lane / CPR;         // this lane's 16-byte column and first row
  const bool one_page = p.block_table == nullptr || geo.page_shift >= 4;   // a warp's 16 keys lie inside one page
  const int pad = p.cache_leftpad ? max(0, p.cache_leftpad[b]) : 0;
  const int* table = p.block_table ? p.block_table + (int64_t)b * p.block_table_stride : nullptr;
  int page = table ? 0 : (p.cache_batch_idx ? p.cache_batch_idx[b] : b);
  int ld = tile0;                                           // next tile to load
  auto ld_page = [&]() {                                    // read one tile ahead of its use
    if (table && one_page) {
      const int key = ld * kTile + warp * 16;
      if (key < len_old) page = table[key >> geo.page_shift];
    }
  };
  ld_page();
  auto load_tile = [&](int st) {
    if (ld == tile0 + count) return;
    T* dK = ring + ((st * 4 + warp) * 2 * 16 + lr) * P + lc;
    T* dV = dK + 16 * P;
    const T* kb = reinterpret_cast<const T*>(p.k_cache) + (int64_t)hk * p.kc_stride[2] + lc;
    const T* vb = reinterpret_cast<const T*>(p.v_cache) + (int64_t)hk * p.vc_stride[2] + lc;
    const int key0 = ld * kTile + warp * 16 + lr;
    if (one_page) {
      const int row0 = table ? key0 & (p.page_size - 1) : key0 + pad;
      const T* ks = kb + (int64_t)page * p.kc_stride[0] + (int64_t)row0 * p.kc_stride[1];
      const T* vs = vb + (int64_t)page * p.vc_stride[0] + (int64_t)row0 * p.vc_stride[1];
      const int64_t kstep = RPW * p.kc_stride[1], vstep = RPW * p.vc_stride[1];
#pragma unroll
      for (int i = 0; i < PASSES; ++i) {
        // rows past the cached tokens are zero-filled (new tokens are staged from k_new / v_new later)
        const int bytes = key0 + i * RPW < len_old ? 16 : 0;
        cp_async16(smem_u32(dK + i * RPW * P), bytes ? ks + i * kstep : kb, bytes);
        cp_async16(smem_u32(dV + i * RPW * P), bytes ? vs + i * vstep : vb, bytes);
      }
    } else {
#pragma unroll
      for (int i = 0; i < PASSES; ++i) {
        const int key = key0 + i * RPW;
        const int bytes = key < len_old ? 16 : 0;
        int pi = 0, row = 0;
        if (bytes) {
          if (geo.page_shift >= 0) {
            pi = key >> geo.page_shift;
            row = key & (p.page_size - 1);
          } else {
            pi = key / p.page_size;
            row = key - pi * p.page_size;
          }
          pi = table[pi];
        }
        cp_async16(smem_u32(dK + i * RPW * P), kb + (int64_t)pi * p.kc_stride[0] + (int64_t)row * p.kc_stride[1], bytes);
        cp_async16(smem_u32(dV + i * RPW * P), vb + (int64_t)pi * p.vc_stride[0] + (int64_t)row * p.vc_stride[1], bytes);
      }
    }
    ++ld;
    ld_page();
  };

#pragma unroll
  for (int i = 0; i < NS - 1; ++i) {
    load_tile(i);
    cp_async_commit();
  }

  float* ws_o = reinterpret_cast<float*>(p.workspace);
  float* ws_l = ws_o + (int64_t)(gridDim.x / U) * p.heads_kv * R * D;
  const T* cos = reinterpret_cast<const T*>(p.rotary_cos);
  const T* sin = reinterpret_cast<const T*>(p.rotary_sin);
  int stage = 0;

  // What the append of this piece's new tokens will read, on its way to L1 meanwhile: it is the last thing that the piece
  // with the end of the sequence does, and a small step waits for that piece.
  if (p.k_new && (tile0 + count) * kTile > len_old) {
    const int from = max(len_old, tile0 * kTile), n = min(min(len, (tile0 + count) * kTile) - from, 8);
    for (int i = tid; i < n * 4; i += NT) {
      const int key = from + (i >> 2), tok = key - len_old, what = i & 3;
      const char* a = nullptr;
      int bytes = D * 2;
      if (what == 0) a = reinterpret_cast<const char*>(reinterpret_cast<const T*>(p.k_new) + b * p.kn_stride[0] + tok * p.kn_stride[1] + hk * p.kn_stride[2]);
      if (what == 1) a = reinterpret_cast<const char*>(reinterpret_cast<const T*>(p.v_new) + b * p.vn_stride[0] + tok * p.vn_stride[1] + hk * p.vn_stride[2]);
      if (what >= 2 && cos && key + pad < p.rotary_seqlen) {
        bytes = p.rotary_dim;
        a = reinterpret_cast<const char*>((what == 2 ? cos : sin) + (int64_t)(key + pad) * (p.rotary_dim >> 1));
      }
      if (a != nullptr)
        for (int o = 0; o < bytes; o += 128) asm volatile("prefetch.global.L1 [%0];" ::"l"(a + o));
    }
  }

  // Q rows (rotary fused) -> shared memory -> B fragments held in registers
#pragma unroll
  for (int i0 = 0; i0 < kRows * CPR; i0 += NT) {
    const int i = i0 + tid;
    if (kRows * CPR % NT != 0 && i >= kRows * CPR) break;
    const int r = i / CPR, d = i % CPR * 8;
    const int gr = rg * kRows + r;
    uint4 val = make_uint4(0u, 0u, 0u, 0u);
    if (gr < R) {
      const int sq = gr / G, gi = gr % G;
      const T* qrow = reinterpret_cast<const T*>(p.q) + b * p.q_stride[0] + sq * p.q_stride[1] +
                      (int64_t)(hk * G + gi) * p.q_stride[2];
      val = rotary_chunk<T, true>(qrow, d, cos, sin, len - p.seqlen_q + sq + pad, p.rotary_dim, p.rotary_interleaved, p.rotary_seqlen);
    }
    *reinterpret_cast<uint4*>(sQ + r * P + d) = val;
  }
  __syncthreads();
  uint32_t bq[NB][D / 16][2];
#pragma unroll
  for (int n = 0; n < NB; ++n) {
    if constexpr (D >= 32) {
#pragma unroll
      for (int kk = 0; kk < D / 32; ++kk)
        ldsm_x4(smem_u32(sQ + (n * 8 + (lane & 7)) * P + kk * 32 + (lane >> 3) * 8), bq[n][2 * kk][0], bq[n][2 * kk][1],
                bq[n][2 * kk + 1][0], bq[n][2 * kk + 1][1]);
    } else {
      const uint32_t* row = reinterpret_cast<const uint32_t*>(sQ + (n * 8 + g) * P);
      bq[n][0][0] = row[t];
      bq[n][0][1] = row[t + 4];
    }
  }
  // this thread's score columns: query rows 8 n + 2 t and 8 n + 2 t + 1
  int qpos[NB][2];
  float slope[NB][2];
#pragma unroll
  for (int n = 0; n < NB; ++n) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int gr = min(rg * kRows + n * 8 + 2 * t + i, R - 1);
      const int sq = gr / G, gi = gr % G;
      qpos[n][i] = len - p.seqlen_q + sq;
      slope[n][i] = cfg.has_alibi ? p.alibi_slopes[b * p.heads_q + hk * G + gi] : 0.f;
    }
  }
  const int qmin = len - p.seqlen_q + rg * kRows / G, qmax = len - p.seqlen_q + min(rg * kRows + kRows - 1, R - 1) / G;
  float o[NB][D / 16][4];
#pragma unroll
  for (int n = 0; n < NB; ++n) {
#pragma unroll
    for (int i = 0; i < D / 16; ++i) o[n][i][0] = o[n][i][1] = o[n][i][2] = o[n][i][3] = 0.f;
  }
  float mrow[NB][2], lrow[NB][2];                // the maximum all scores are taken relative to; sums of this lane's keys
#pragma unroll
  for (int n = 0; n < NB; ++n) {
    mrow[n][0] = mrow[n][1] = -INFINITY;
    lrow[n][0] = lrow[n][1] = 0.f;
  }

  for (int ti = 0; ti < count; ++ti) {
    const int keyw = (tile0 + ti) * kTile + warp * 16;   // this warp's first key
    cp_async_wait<NS - 2>();
    __syncwarp();
    load_tile(stage == 0 ? NS - 1 : stage - 1);
    cp_async_commit();
    T* tK = ring + (stage * 4 + warp) * 2 * 16 * P;
    T* tV = tK + 16 * P;
    if (++stage == NS) stage = 0;
    if (keyw >= len) continue;
    // ---- append: new tokens among these keys, rotated, into the staged rows and the cache ----
    const int nfirst = max(keyw, len_old), nlast = min(keyw + 16, len);   // new keys [nfirst, nlast)
    if (nlast > nfirst) {
      for (int i = lane; i < (nlast - nfirst) * CPR; i += 32) {
        const int key = nfirst + i / CPR, d = i % CPR * 8;
        const int tok = key - len_old, pos = key + pad;
        const T* kn = reinterpret_cast<const T*>(p.k_new) + b * p.kn_stride[0] + tok * p.kn_stride[1] + hk * p.kn_stride[2];
        const T* vn = reinterpret_cast<const T*>(p.v_new) + b * p.vn_stride[0] + tok * p.vn_stride[1] + hk * p.vn_stride[2];
        const uint4 vv = *reinterpret_cast<const uint4*>(vn + d);
        const uint4 kv = rotary_chunk<T, true>(kn, d, cos, sin, pos, p.rotary_dim, p.rotary_interleaved, p.rotary_seqlen);
        *reinterpret_cast<uint4*>(tK + (key - keyw) * P + d) = kv;
        *reinterpret_cast<uint4*>(tV + (key - keyw) * P + d) = vv;
        if (rg == 0 && pos < cache_capacity(p)) {
          *reinterpret_cast<uint4*>(reinterpret_cast<T*>(p.k_cache) + cache_row_offset(p, b, pos, geo.page_shift, p.kc_stride) +
                                    (int64_t)hk * p.kc_stride[2] + d) = kv;
          *reinterpret_cast<uint4*>(reinterpret_cast<T*>(p.v_cache) + cache_row_offset(p, b, pos, geo.page_shift, p.vc_stride) +
                                    (int64_t)hk * p.vc_stride[2] + d) = vv;
        }
      }
      __syncwarp();
    }

    // ---- S^T = K Q^T: keys keyw + g and keyw + g + 8 ------------------------------------
    float s[NB][4];
#pragma unroll
    for (int n = 0; n < NB; ++n) s[n][0] = s[n][1] = s[n][2] = s[n][3] = 0.f;
#pragma unroll
    for (int kk = 0; kk < D / 16; ++kk) {
      uint32_t a[4];
      ldsm_x4(smem_u32(tK + (lane & 15) * P + kk * 16 + (lane >> 4) * 8), a[0], a[1], a[2], a[3]);
#pragma unroll
      for (int n = 0; n < NB; ++n) mma16816<T>(s[n], a, bq[n][kk][0], bq[n][kk][1]);
    }
    // ---- softmax.  Plain scores that every row sees need no test per element; their scale goes
    // into the exponent's FMA --------------------------------------------------------------
    const bool full = !cfg.has_alibi && keyw + 16 <= len && (!cfg.causal || keyw + 15 <= qmin) &&
                      (cfg.wl < 0 || keyw >= qmax - cfg.wl) && (cfg.wr < 0 || keyw + 15 <= qmin + cfg.wr);
    float mul = cfg.scale_log2;
    if (!full) {
      mul = 1.f;
#pragma unroll
      for (int n = 0; n < NB; ++n) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int i = e & 1, key = keyw + g + (e >> 1) * 8;
          float th;
          const float v = score_log2(cfg, slope[n][i], s[n][e], qpos[n][i], key, th);
          s[n][e] = visible(cfg, qpos[n][i], key, len) ? v : -INFINITY;
        }
      }
    }
    float mx[NB][2];
    bool grow = false;
#pragma unroll
    for (int n = 0; n < NB; ++n) {
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        // the scale may be negative: scale before the maximum
        float m = fmaxf(s[n][i] * mul, s[n][2 + i] * mul);
        m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 4));
        m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 8));
        mx[n][i] = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 16));
        // raised whenever it grows: the largest probability is then exactly 1 (ScoreCfg::rescale_at)
        grow |= mx[n][i] > mrow[n][i];
      }
    }
    if (__any_sync(0xffffffffu, grow)) {
#pragma unroll
      for (int n = 0; n < NB; ++n) {
        float alpha[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const bool up = mx[n][i] > mrow[n][i];
          alpha[i] = up ? exp2f(mrow[n][i] - mx[n][i]) : 1.f;    // from -inf: 0
          if (up) mrow[n][i] = mx[n][i];
          lrow[n][i] *= alpha[i];
        }
#pragma unroll
        for (int db = 0; db < D / 16; ++db) {
          o[n][db][0] *= alpha[0]; o[n][db][1] *= alpha[1];
          o[n][db][2] *= alpha[0]; o[n][db][3] *= alpha[1];
        }
      }
    }
    uint32_t pb[NB][2];
#pragma unroll
    for (int n = 0; n < NB; ++n) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        // no finite score yet: exponents relative to 0, so that -inf gives 0 and NaN stays NaN
        const float m = mrow[n][e & 1] == -INFINITY ? 0.f : mrow[n][e & 1];
        s[n][e] = ex2(fmaf(s[n][e], mul, -m));
        lrow[n][e & 1] += s[n][e];
      }
      // P^T[key][row] as the accumulator holds it -> B fragment [keys] x [rows]
      pb[n][0] = transpose_8x8(Elem<T>::pack(s[n][0], s[n][1]));
      pb[n][1] = transpose_8x8(Elem<T>::pack(s[n][2], s[n][3]));
    }
    // ---- O^T += V^T P^T -----------------------------------------------------------------
#pragma unroll
    for (int db = 0; db < D / 16; ++db) {
      uint32_t a[4];
      ldsm_x4_t(smem_u32(tV + ((lane & 7) + ((lane >> 4) << 3)) * P + db * 16 + ((lane >> 3) & 1) * 8), a[0], a[1], a[2], a[3]);
#pragma unroll
      for (int n = 0; n < NB; ++n) mma16816<T>(o[n][db], a, pb[n][0], pb[n][1]);
    }
  }

  // ---- merge the 4 warps (each saw a quarter of every tile) -----------------------------------
#pragma unroll
  for (int n = 0; n < NB; ++n) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      float l = lrow[n][i];
      l += __shfl_xor_sync(0xffffffffu, l, 4);
      l += __shfl_xor_sync(0xffffffffu, l, 8);
      l += __shfl_xor_sync(0xffffffffu, l, 16);
      if (g == 0) {
        sM[warp * kRows + n * 8 + 2 * t + i] = mrow[n][i];
        sL[warp * kRows + n * 8 + 2 * t + i] = l;
      }
    }
  }
  __syncthreads();
  float wgt[NB][2];
#pragma unroll
  for (int n = 0; n < NB; ++n) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int r = n * 8 + 2 * t + i;
      const float mstar = fmaxf(fmaxf(sM[r], sM[kRows + r]), fmaxf(sM[2 * kRows + r], sM[3 * kRows + r]));
      wgt[n][i] = (mstar == -INFINITY) ? 0.f : exp2f(mrow[n][i] - mstar);
    }
  }
#pragma unroll
  for (int n = 0; n < NB; ++n) {
#pragma unroll
    for (int db = 0; db < D / 16; ++db) {
#pragma unroll
      for (int e = 0; e < 4; ++e)
        sO[(warp * kRows + n * 8 + 2 * t + (e & 1)) * OP + db * 16 + g + (e >> 1) * 8] = wgt[n][e & 1] * o[n][db][e];
    }
  }
  __syncthreads();

  // ---- output, or a piece of it -----------------------------------------------------------
  // workspace: the R query rows of every (piece, kv head), not padded to units
  const int64_t ws_row = ((int64_t)share * p.heads_kv + hk) * R + rg * kRows;
  for (int i = tid; i < kRows * (D / 4); i += NT) {
    const int r = i / (D / 4), c4 = (i % (D / 4)) * 4;
    const int gr = rg * kRows + r;
    if (gr >= R) continue;
    const float mstar = fmaxf(fmaxf(sM[r], sM[kRows + r]), fmaxf(sM[2 * kRows + r], sM[3 * kRows + r]));
    float lsum = 0.f;
    if (mstar != -INFINITY) {
#pragma unroll
      for (int wv = 0; wv < 4; ++wv) lsum += exp2f(sM[wv * kRows + r] - mstar) * sL[wv * kRows + r];
    }
    float4 acc = *reinterpret_cast<const float4*>(sO + r * OP + c4);
#pragma unroll
    for (int wv = 1; wv < 4; ++wv) {
      const float4 x = *reinterpret_cast<const float4*>(sO + (wv * kRows + r) * OP + c4);
      acc.x += x.x; acc.y += x.y; acc.z += x.z; acc.w += x.w;
    }
    const float inv = lsum > 0.f ? 1.f / lsum : 0.f;
    acc.x *= inv; acc.y *= inv; acc.z *= inv; acc.w *= inv;
    const int sq = gr / G, h = hk * G + gr % G;
    if (parts == 1) {
      T* og = reinterpret_cast<T*>(p.o) + b * p.o_stride[0] + sq * p.o_stride[1] + (int64_t)h * p.o_stride[2] + c4;
      uint2 pk;
      pk.x = Elem<T>::pack(acc.x, acc.y);
      pk.y = Elem<T>::pack(acc.z, acc.w);
      *reinterpret_cast<uint2*>(og) = pk;
    } else {
      *reinterpret_cast<float4*>(ws_o + (ws_row + r) * D + c4) = acc;
      if (c4 == 0) ws_l[ws_row + r] = lsum > 0.f ? mstar + log2f(lsum) : -INFINITY;
    }
  }
  if (parts > 1) {
    // the CTA that comes last merges; the pieces are ordered before the count by each writer's fence
    __shared__ int last;
    __threadfence();
    __syncthreads();
    if (tid == 0) {
      uint32_t* ctr = p.counters + ((int64_t)b * U + u);
      last = atomicAdd(ctr, 1u) == (uint32_t)(parts - 1);
      if (last) *ctr = 0u;
    }
    __syncthreads();
    if (last) {
      __threadfence();
      const int rows = min(kRows, R - rg * kRows);
      for (int i = tid; i < rows * (D / 4); i += NT) {
        const int r = i / (D / 4), gr = rg * kRows + r;
        const int sq = gr / G, h = hk * G + gr % G;
        merge_pieces<T, D>(ws_o, ws_l, ((int64_t)base * p.heads_kv + hk) * R + gr, (int64_t)p.heads_kv * R, parts, (i % (D / 4)) * 4,
                           reinterpret_cast<T*>(p.o) + b * p.o_stride[0] + sq * p.o_stride[1] + (int64_t)h * p.o_stride[2]);
      }
    }
  }
}

// ---------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------
static int page_shift_of(const fa_decode_args& a) {
  if (a.page_size <= 0 || (a.page_size & (a.page_size - 1)) != 0) return -1;
  int s = 0;
  while ((1 << s) < a.page_size) ++s;
  return s;
}
static int decode_unit_rows(const fa_decode_args& a) { return a.seqlen_q * (a.heads_q / a.heads_kv) <= 8 ? 8 : 16; }
static int decode_row_groups(const fa_decode_args& a) {
  const int n = decode_unit_rows(a);
  return (a.seqlen_q * (a.heads_q / a.heads_kv) + n - 1) / n;
}

// ---------------------------------------------------------------------------------------
// Chunks of tokens: more than 16 query rows per KV head.  The kernel above would read the cache once per 16
// rows; these calls append and rotate in a kernel of their own and attend on the tensor cores
// (fwd_alt_sm100.cu), which takes about as long for 128 rows as the kernel above for 16.
// ---------------------------------------------------------------------------------------
constexpr int kAppendPerSm = 5;    // CTAs of 256 threads with 48 registers each
// New keys (rotated) and values into the cache, rotated queries into q_out (batch, tokens, heads, D); a
// 16-byte chunk per thread and step, HBM-bound.  host / dev: value checks made by every CTA, see decode_kernel.
// Index: of a chunk.  With 64-bit indices the five divisions of a thread were most of the kernel; and as every CTA makes the
// checks, there are no more CTAs than run at a time (4 x 256 tokens of 32 heads over 8 of 128: 15.5 -> 10.9 us).
template <typename T, typename Index>
__global__ void __launch_bounds__(256, kAppendPerSm) cache_append_kernel(const fa_decode_args p, T* q_out, int page_shift, uint32_t* host,
                                                           uint32_t* dev, bool check_here) {
  if (check_here) {
    const uint32_t bad = decode_checks(p, threadIdx.x, 256);
    if (threadIdx.x == 0 && blockIdx.x == 0) {
      *dev = bad;
      *reinterpret_cast<volatile uint32_t*>(host) = bad | kCheckDone;
      __threadfence_system();
    }
    if (bad) return;
  } else if (dev && *dev) {
    return;
  }
  const int D = p.head_dim, cpr_log2 = 31 - __clz(D / 8);      // (a power of two)
  const int n_new = p.k_new ? p.seqlen_new : 0;
  const Index nq = q_out ? ((Index)p.batch * p.seqlen_q * p.heads_q) << cpr_log2 : 0;
  const Index nk = ((Index)p.batch * n_new * p.heads_kv) << cpr_log2;
  const T* cos = reinterpret_cast<const T*>(p.rotary_cos);
  const T* sin = reinterpret_cast<const T*>(p.rotary_sin);
  for (Index at = (Index)blockIdx.x * 256 + threadIdx.x; at < nq + 2 * nk; at += (Index)gridDim.x * 256) {
    Index i = at;
    const int d = (int)(i & ((1 << cpr_log2) - 1)) * 8;
    if (i < nq) {
      const Index row = i >> cpr_log2, bt = row / (Index)p.heads_q;
      const int h = (int)(row - bt * p.heads_q), b = (int)(bt / (Index)p.seqlen_q), tok = (int)(bt - (Index)b * p.seqlen_q);
      const int pos = p.cache_seqlens[b] + n_new - p.seqlen_q + tok + (p.cache_leftpad ? p.cache_leftpad[b] : 0);
      const T* x = reinterpret_cast<const T*>(p.q) + b * p.q_stride[0] + tok * p.q_stride[1] + h * p.q_stride[2];
      *reinterpret_cast<uint4*>(q_out + (int64_t)i * 8) =
          rotary_chunk<T, false>(x, d, cos, sin, pos, p.rotary_dim, p.rotary_interleaved, p.rotary_seqlen);
      continue;
    }
    i -= nq;
    const bool val = i >= nk;
    if (val) i -= nk;
    const Index row = i >> cpr_log2, bt = row / (Index)p.heads_kv;
    const int h = (int)(row - bt * p.heads_kv), b = (int)(bt / (Index)n_new), tok = (int)(bt - (Index)b * n_new);
    const int pos = max(0, min(p.cache_seqlens[b], seq_capacity(p, b))) + tok + (p.cache_leftpad ? max(0, p.cache_leftpad[b]) : 0);
    if (pos >= cache_capacity(p)) continue;
    if (val) {
      const T* x = reinterpret_cast<const T*>(p.v_new) + b * p.vn_stride[0] + tok * p.vn_stride[1] + h * p.vn_stride[2];
      T* dst = reinterpret_cast<T*>(p.v_cache) + cache_row_offset(p, b, pos, page_shift, p.vc_stride) + h * p.vc_stride[2];
      *reinterpret_cast<uint4*>(dst + d) = *reinterpret_cast<const uint4*>(x + d);
    } else {
      const T* x = reinterpret_cast<const T*>(p.k_new) + b * p.kn_stride[0] + tok * p.kn_stride[1] + h * p.kn_stride[2];
      T* dst = reinterpret_cast<T*>(p.k_cache) + cache_row_offset(p, b, pos, page_shift, p.kc_stride) + h * p.kc_stride[2];
      *reinterpret_cast<uint4*>(dst + d) = rotary_chunk<T, false>(x, d, cos, sin, pos, p.rotary_dim, p.rotary_interleaved, p.rotary_seqlen);
    }
  }
}

struct ChunkPlan {
  int pack_log2, units, parts, capacity;
  size_t q_bytes, piece_bytes;   // workspace: rotated queries, pieces, then the counters if the caller brings none
};
// Whether a call is a chunk, and how it is cut.
static bool chunk_plan(const fa_decode_args& a, ChunkPlan& c) {
  const int G = a.heads_q / a.heads_kv;
  if (a.num_splits != 0 || a.seqlen_q * G <= 16 || a.softmax_scale < 0.f) return false;
  if (a.head_dim != 64 && a.head_dim != 128 && a.head_dim != 256) return false;
  if (a.block_table) {       // a tile of 128 keys is whole pages, or lies inside one
    const bool pow2 = (a.page_size & (a.page_size - 1)) == 0;
    if (!(pow2 && a.page_size >= 16 && a.page_size < 128) && a.page_size % 128 != 0) return false;
  }
  c.pack_log2 = 0;
  if ((G & (G - 1)) == 0 && G <= 64)
    while ((1 << c.pack_log2) < G) ++c.pack_log2;
  const int64_t cap = a.block_table ? (int64_t)a.block_table_stride * a.page_size : a.page_size;
  const int mtiles = (int)((((int64_t)a.seqlen_q << c.pack_log2) + 127) / 128);
  const int64_t units = (int64_t)a.batch * (a.heads_q >> c.pack_log2) * mtiles;
  if (units > (1 << 28) || cap > (1 << 30)) return false;
  c.units = (int)units;
  c.capacity = (int)cap;
  // pieces of at least four key tiles, only while the units leave SMs idle
  const int64_t fill = sm_count(a.device) / units, most = (cap + 511) / 512;
  c.parts = (int)(fill < most ? fill : most);
  if (c.parts < 1) c.parts = 1;
  c.q_bytes = a.rotary_cos ? (size_t)a.batch * a.seqlen_q * a.heads_q * a.head_dim * 2 : 0;
  c.piece_bytes = c.parts > 1 ? (size_t)c.units * c.parts * 128 * (a.head_dim + 1) * sizeof(float) : 0;
  return true;
}

int decode_num_counters(const fa_decode_args& a) {
  ChunkPlan c;
  if (chunk_plan(a, c)) return c.parts > 1 ? c.units : 0;
  return a.batch * a.heads_kv * decode_row_groups(a);
}

// Room for the pieces the kernel may make.  It picks their size so that
//   * one wave of CTAs (two per SM, one at head_dim 256) takes all of them, while that needs no more
//     than kOneWave tiles each: every CTA costs about 3.5 us beside its tiles (16 sequences of 4000 keys,
//     8 heads: one wave of 32-tile pieces 55 us, two of 16 61 us, 68 us without pieces);
//   * a sequence has no more than sqrt(7 nt) pieces of its nt tiles: a tile costs about 0.7 us and a piece
//     0.1 us in the merge (one sequence of 8000 keys, two heads: 126 pieces 20 us, 32 pieces 16.4 us);
//   * more work than that runs as kWaves waves, which the hardware balances over SMs of unequal speed
//     (64 sequences of 16000 keys: one wave of equal shares 688 us, 3.5 waves 656 us = 0.98 of the copy
//     bandwidth).
// An explicit num_splits, and batches too large to sum in every warp, cut every sequence into the
// same number of pieces.
static DecodeGeom decode_geometry(const fa_decode_args& a) {
  DecodeGeom g;
  g.row_groups = decode_row_groups(a);
  const int64_t cap = a.block_table ? (int64_t)a.block_table_stride * a.page_size : a.page_size;
  const int64_t nt = cap > 0 ? (cap + kTile - 1) / kTile : 1;
  const int64_t U = (int64_t)a.heads_kv * g.row_groups;
  g.max_tiles = (int)nt;
  g.splits = 0;
  g.resident = sm_count(a.device) * (a.head_dim == 256 ? 1 : 2);
  if (a.num_splits > 0 || a.batch > kMaxBalanced || a.batch * nt > (1 << 30)) {
    g.splits = a.num_splits > 0 ? (int)(a.num_splits < nt ? a.num_splits : nt) : 1;
    g.shares = a.batch * g.splits;
  } else {
    const int64_t most = a.batch * nt, whole = a.batch;
    int64_t n = most * U <= (int64_t)kOneWave * g.resident ? g.resident / U : kWaves * g.resident / U + 1;
    n += whole;                                // rounding up adds less than a piece per sequence
    g.shares = (int)(n < most ? n : most);
  }
  g.page_shift = page_shift_of(a);
  return g;
}

// pieces (their query rows in fp32, then the LSEs of those), then the counters if the caller brings none
static size_t decode_piece_bytes(const fa_decode_args& a, const DecodeGeom& g) {
  if (g.splits == 1) return 0;
  return (size_t)g.shares * a.seqlen_q * a.heads_q * (a.head_dim + 1) * sizeof(float);
}
size_t decode_workspace_bytes(const fa_decode_args& a) {
  if (a.heads_kv <= 0 || a.heads_q <= 0 || a.batch <= 0 || a.seqlen_q <= 0) return 0;
  ChunkPlan c;
  if (chunk_plan(a, c)) {
    if (c.q_bytes + c.piece_bytes == 0) return 0;
    return c.q_bytes + c.piece_bytes + (c.parts > 1 && !a.counters ? (size_t)c.units * sizeof(uint32_t) : 0);
  }
  const size_t pieces = decode_piece_bytes(a, decode_geometry(a));
  return pieces == 0 ? 0 : pieces + (a.counters ? 0 : (size_t)decode_num_counters(a) * sizeof(uint32_t));
}

template <typename T, int D, int kRows>
static int launch_rows(const fa_decode_args& a, const ScoreCfg& cfg, const DecodeGeom& g, const DecodeCheck& chk,
                         cudaStream_t st) {
  const size_t smem = DecodeSmem<D, kRows>::fixed;
  auto kern = decode_kernel<T, D, kRows>;
  // once per kernel and device: a step of one conversation is bounded by the host's part
  static std::atomic<uint64_t> prepared{0};
  const uint64_t bit = a.device < 64 ? 1ull << a.device : 0;
  if ((prepared.load(std::memory_order_relaxed) & bit) == 0) {
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) {
      set_error("decode: cudaFuncSetAttribute: %s", cudaGetErrorString(e));
      return FA_ERR_LAUNCH;
    }
    prepared.fetch_or(bit, std::memory_order_relaxed);
  }
  cudaLaunchConfig_t lc = {};
  cudaLaunchAttribute attr;
  lc.gridDim = dim3((unsigned)g.shares * a.heads_kv * g.row_groups);
  lc.blockDim = dim3(128);
  lc.dynamicSmemBytes = smem;
  lc.stream = st;
  if (chk.dev) {
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    lc.attrs = &attr;
    lc.numAttrs = 1;
  }
  cudaLaunchKernelEx(&lc, kern, a, cfg, g, chk);
  return check_launch("decode");
}

template <typename T, int D>
static int launch_decode(const fa_decode_args& a, const ScoreCfg& cfg, const DecodeGeom& g, const DecodeCheck& chk,
                         cudaStream_t st) {
  return decode_unit_rows(a) == 8 ? launch_rows<T, D, 8>(a, cfg, g, chk, st) : launch_rows<T, D, 16>(a, cfg, g, chk, st);
}

template <typename T>
static int decode_t(const fa_decode_args& a, const ScoreCfg& cfg, const DecodeGeom& g, const DecodeCheck& chk,
                    cudaStream_t st) {
  switch (a.head_dim) {
    case 16: return launch_decode<T, 16>(a, cfg, g, chk, st);
    case 32: return launch_decode<T, 32>(a, cfg, g, chk, st);
    case 64: return launch_decode<T, 64>(a, cfg, g, chk, st);
    case 128: return launch_decode<T, 128>(a, cfg, g, chk, st);
    case 256: return launch_decode<T, 256>(a, cfg, g, chk, st);
  }
  set_error("head_dim %d not in {16,32,64,128,256}", a.head_dim);
  return FA_ERR_UNSUPPORTED;
}

// What a call is refused for, before any of its kernels is launched.  c: its cut as a chunk, or null.
static int decode_refused(const fa_decode_args& a, const ChunkPlan* c) {
  if (c != nullptr)
    if (const int code = host_wait_status(a.device)) {
      set_error("fa_decode_paged: a bounded device-side wait ran out earlier on device %d (code %d); the tcgen05 kernels "
                "stay off until fa_device_wait_clear()", a.device, code);
      return FA_ERR_DEVICE_WAIT;
    }
  const size_t need = decode_workspace_bytes(a);
  if (need > 0 && (a.workspace == nullptr || a.workspace_bytes < need)) {
    set_error("decode workspace too small: need %zu bytes, got %zu", need, a.workspace_bytes);
    return FA_ERR_WORKSPACE;
  }
  FA_REQUIRE(a.counters == nullptr || a.num_counters >= decode_num_counters(a), "decode: too few counters");
  return FA_OK;
}

static int decode_run(const fa_decode_args& args, const DecodeCheck& chk, cudaStream_t st) {
  fa_decode_args a = args;
  const DecodeGeom g = decode_geometry(a);
  const size_t pieces = decode_piece_bytes(a, g), need = decode_workspace_bytes(a);
  if (need > 0 && a.counters == nullptr) {
    a.counters = reinterpret_cast<uint32_t*>(static_cast<char*>(a.workspace) + pieces);
    const cudaError_t e = cudaMemsetAsync(a.counters, 0, need - pieces, st);
    if (e != cudaSuccess) {
      set_error("decode: cudaMemsetAsync: %s", cudaGetErrorString(e));
      return FA_ERR_LAUNCH;
    }
  }
  // bottom-right alignment: the causal mask and window are relative to the query's
  // position at the end of the cached sequence
  ScoreCfg cfg = make_score_cfg(a.softmax_scale, 0.f, a.causal, a.window_left, a.window_right,
                                a.alibi_slopes != nullptr);
  return a.dtype == FA_BF16 ? decode_t<__nv_bfloat16>(a, cfg, g, chk, st) : decode_t<__half>(a, cfg, g, chk, st);
}

// dev: the call's word with the result of the value checks, or null.  host != null: the append kernel makes the
// checks; *queued is set once it is on the stream and will write the host word.
static int chunk_run(const fa_decode_args& args, const ChunkPlan& c, uint32_t* host, uint32_t* dev, bool* queued, cudaStream_t st) {
  fa_decode_args a = args;
  const bool inside = host != nullptr;
  char* ws = static_cast<char*>(a.workspace);
  CacheGeo geo = {};
  geo.seqlens = a.cache_seqlens;
  geo.table = a.block_table;
  geo.table_stride = a.block_table_stride;
  geo.batch_idx = a.cache_batch_idx;
  geo.leftpad = a.cache_leftpad;
  geo.page_size = a.page_size;
  geo.page_log2 = page_shift_of(a);
  geo.box_rows = a.block_table && a.page_size < 128 ? a.page_size : 128;
  geo.n_new = a.k_new ? a.seqlen_new : 0;
  geo.tokens = a.seqlen_q;
  geo.pack_log2 = c.pack_log2;
  geo.parts = c.parts;
  geo.capacity = c.capacity;
  geo.ws = reinterpret_cast<float*>(ws + c.q_bytes);
  geo.bad = dev;
  if (c.parts > 1) {
    geo.counters = a.counters;
    if (geo.counters == nullptr) {
      geo.counters = reinterpret_cast<uint32_t*>(ws + c.q_bytes + c.piece_bytes);
      const cudaError_t e = cudaMemsetAsync(geo.counters, 0, (size_t)c.units * sizeof(uint32_t), st);
      if (e != cudaSuccess) {
        set_error("decode: cudaMemsetAsync: %s", cudaGetErrorString(e));
        return FA_ERR_LAUNCH;
      }
    }
  }
  void* q_out = c.q_bytes ? ws : nullptr;
  const int64_t chunks = ((q_out ? (int64_t)a.batch * a.seqlen_q * a.heads_q : 0) + 2ll * a.batch * geo.n_new * a.heads_kv) *
                         (a.head_dim / 8);
  if (chunks > 0 || inside) {
    const int64_t need = chunks > 0 ? (chunks + 255) / 256 : 1, fit = (int64_t)sm_count(a.device) * kAppendPerSm;
    const unsigned grid = (unsigned)(need < fit ? need : fit);
    const int shift = page_shift_of(a);
    const bool small = chunks < (int64_t)1 << 31;
    auto append = [&](auto* q) {
      using T = std::remove_pointer_t<decltype(q)>;
      auto kern = small ? cache_append_kernel<T, uint32_t> : cache_append_kernel<T, int64_t>;
      kern<<<grid, 256, 0, st>>>(a, q, shift, host, dev, inside);
    };
    if (a.dtype == FA_BF16) append(static_cast<__nv_bfloat16*>(q_out));
    else append(static_cast<__half*>(q_out));
    if (int r = check_launch("cache_append")) return r;
    if (inside) *queued = true;
  }
  const int64_t qs[3] = {(int64_t)a.seqlen_q * a.heads_q * a.head_dim, (int64_t)a.heads_q * a.head_dim, a.head_dim};
  const ScoreCfg cfg = make_score_cfg(a.softmax_scale, 0.f, a.causal, a.window_left, a.window_right, a.alibi_slopes != nullptr);
  return cache_attention_sm100(a, q_out ? q_out : a.q, q_out ? qs : a.q_stride, geo, cfg, st);
}

int decode_paged(const fa_decode_args& a, cudaStream_t st) {
  if (a.batch == 0 || a.seqlen_q == 0 || a.heads_q == 0) return FA_OK;
  ChunkPlan c;
  const bool chunk = chunk_plan(a, c);
  if (int r = decode_refused(a, chunk ? &c : nullptr)) return r;
  return chunk ? chunk_run(a, c, nullptr, nullptr, nullptr, st) : decode_run(a, DecodeCheck{nullptr, nullptr}, st);
}

// ---------------------------------------------------------------------------------------
// Value checks.  A call takes a slot -- one word in mapped host memory --, launches, and polls the word: it
// changes as soon as the checks have run, so the host goes on while the attention is still running, without
// a stream synchronisation.
// ---------------------------------------------------------------------------------------
constexpr int kCheckSlots = 256, kTickets = FA_VARLEN_TICKETS;
alignas(4096) static volatile uint32_t g_check_host[kCheckSlots * 16];      // a cache line per slot

namespace {
CheckSlots<kCheckSlots, kTickets> g_slots(g_check_host);
volatile uint32_t* slot_word(int i) { return g_slots.word_of(g_check_host, i); }

// The words as `device`, the current one, sees them; null (error set) without mapped host memory.  Tried again by the next call
// where it fails (another thread may be capturing a graph right now).
uint32_t* check_words(int device) {
  static std::atomic<uint32_t*> words[64];
  const bool kept = device >= 0 && device < 64;
  if (kept)
    if (uint32_t* w = words[device].load(std::memory_order_acquire)) return w;
  static std::mutex mu;
  static bool mapped = false;
  std::lock_guard<std::mutex> lock(mu);
  if (!mapped) {
    const cudaError_t e = cudaHostRegister(const_cast<uint32_t*>(g_check_host), sizeof(g_check_host),
                                           cudaHostRegisterPortable | cudaHostRegisterMapped);
    if (e != cudaSuccess) {
      cudaGetLastError();
      set_error("no mapped host memory for the value checks: %s", cudaGetErrorString(e));
      return nullptr;
    }
    mapped = true;
  }
  void* h = nullptr;
  if (cudaHostGetDevicePointer(&h, const_cast<uint32_t*>(g_check_host), 0) != cudaSuccess) {
    set_error("value checks: cudaHostGetDevicePointer: %s", cudaGetErrorString(cudaGetLastError()));
    return nullptr;
  }
  if (kept) words[device].store(static_cast<uint32_t*>(h), std::memory_order_release);
  return static_cast<uint32_t*>(h);
}

// Index of a slot, its word at *dptr; -1 (error set) without one.  A call waits for another call's, a ticket does not.
int take_slot(bool ticket, int device, uint32_t** dptr) {
  uint32_t* words = check_words(device);
  if (words == nullptr) return -1;
  for (;;) {
    const int i = g_slots.take(ticket, device);
    if (i >= 0) {
      *dptr = words + i * 16;
      return i;
    }
    if (ticket || i == g_slots.kNever) {
      set_error(ticket ? "%d tickets of value checks are out" : "no word for the value checks is left", kTickets);
      return -1;
    }
    sched_yield();                     // as many threads as slots are inside this function
  }
}

// Waits until the kernel that was given the slot has written it.
int await_slot(int i, uint32_t* failed, cudaStream_t st) {
  volatile uint32_t* word = slot_word(i);
  for (uint32_t it = 1; *word == 0u; ++it) {
#if defined(__x86_64__)
    __builtin_ia32_pause();
#endif
    if ((it & 0x3fffu) == 0) {         // every few hundred microseconds: has the stream died?
      const cudaError_t e = cudaStreamQuery(st);
      if (e == cudaErrorNotReady) continue;
      if (e != cudaSuccess || *word == 0u) {
        set_error("value checks did not run: %s", cudaGetErrorString(e));
        return FA_ERR_LAUNCH;
      }
    }
  }
  *failed = *word & ~kCheckDone;
  return FA_OK;
}

// Packed calls: both cu_seqlens arrays, by one CTA.
__global__ void __launch_bounds__(1024) varlen_check_kernel(const int32_t* cu_q, const int32_t* cu_k, int batch, int64_t total_q,
                                                            int64_t total_k, bool k_at_most, int64_t max_q, int64_t max_k,
                                                            uint32_t* host) {
  uint32_t bad = 0;
  for (int i = threadIdx.x; i < batch; i += blockDim.x) {
    const int64_t q = (int64_t)cu_q[i + 1] - cu_q[i], k = (int64_t)cu_k[i + 1] - cu_k[i];
    if (q < 0 || k < 0) bad |= FA_VARLEN_ORDER;
    if (q > max_q || k > max_k) bad |= FA_VARLEN_LONGEST;
  }
  if (threadIdx.x == 0) {
    if (cu_q[0] != 0 || cu_k[0] != 0) bad |= FA_VARLEN_START;
    const int64_t k = cu_k[batch];
    if (cu_q[batch] != total_q || (k_at_most ? k > total_k : k != total_k)) bad |= FA_VARLEN_COVER;
  }
  __shared__ uint32_t all;
  if (threadIdx.x == 0) all = 0u;
  __syncthreads();
  if (bad) atomicOr(&all, bad);
  __syncthreads();
  if (threadIdx.x == 0) *reinterpret_cast<volatile uint32_t*>(host) = all | kCheckDone;
}

// What the checks of a call need: `inside`, its first kernel makes them, in every CTA, because the tables are
// small; `word`, kernels behind that one read the result from device memory.
struct CheckPlan {
  bool chunk, inside, word;
  ChunkPlan c;
};
CheckPlan check_plan(const fa_decode_args& a) {
  CheckPlan k;
  k.chunk = chunk_plan(a, k.c);
  k.inside = (int64_t)a.batch * (a.block_table ? a.block_table_stride : 1) <= kInlineCheck;
  k.word = k.chunk || !k.inside;
  return k;
}
constexpr size_t kWordBytes = 16;
size_t word_offset(const fa_decode_args& a) { return (decode_workspace_bytes(a) + kWordBytes - 1) / kWordBytes * kWordBytes; }
}  // namespace

// A copy of both arrays to the host, looked at in Python, cost a packed call 17 to 33 us.  Whole calls, before -> after (us): forward of
// 2 prompts of 30 and 34 tokens, 2 heads of 64, 40 -> 20; of 7 of 67 to 540, 32 heads of 64, 54 -> 35; of 24 of 17 to 2048, 32 heads
// over 8 of 128, 392 -> 374 (404 -> 389 on another box); forward and backward of 14 of 64, 32 heads of 64, 127 -> 93; of 23 of 261
// to 522, 16 heads of 128, 257 -> 225.
int varlen_check(const int32_t* cu_q, const int32_t* cu_k, int batch, int64_t total_q, int64_t total_k, bool k_at_most, int64_t max_q,
                 int64_t max_k, int device, int32_t* ticket, cudaStream_t st) {
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(st, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone) {
    cudaGetLastError();
    set_error("value checks cannot run while the stream is being captured; turn them off with set_validation(False)");
    return FA_ERR_LAUNCH;
  }
  uint32_t* host = nullptr;
  const int slot = take_slot(true, device, &host);
  if (slot < 0) return FA_ERR_UNSUPPORTED;
  varlen_check_kernel<<<1, batch > 128 ? 1024 : 128, 0, st>>>(cu_q, cu_k, batch, total_q, total_k, k_at_most, max_q, max_k, host);
  if (int r = check_launch("varlen_check")) {
    g_slots.give(slot, false);
    return r;
  }
  *ticket = slot;
  return FA_OK;
}
// The caller's current device may be another by now, and a stream of that device (0 is one of each) would be asked about
// a kernel that it never had.
int check_result(int32_t ticket, uint32_t* failed, cudaStream_t st) {
  int device = -1, current = -1;
  FA_REQUIRE(g_slots.hand_in(ticket, &device), "ticket %d is not out", ticket);
  int r = cudaGetDevice(&current) == cudaSuccess ? ensure_device(device) : FA_ERR_LAUNCH;
  if (r == FA_OK) r = await_slot(ticket, failed, st);
  g_slots.give(ticket, true);
  if (current >= 0 && current != device) cudaSetDevice(current);
  return r;
}

size_t decode_checked_workspace_bytes(const fa_decode_args& a) {
  if (a.heads_kv <= 0 || a.heads_q <= 0 || a.batch <= 0 || a.seqlen_q <= 0) return 0;
  return check_plan(a).word ? word_offset(a) + kWordBytes : decode_workspace_bytes(a);
}

int decode_paged_checked(const fa_decode_args& a, uint32_t* failed, cudaStream_t st) {
  *failed = 0;
  if (a.batch == 0 || a.seqlen_q == 0 || a.heads_q == 0) return FA_OK;
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(st, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone) {
    cudaGetLastError();
    set_error("value checks cannot run while the stream is being captured; turn them off with set_validation(False)");
    return FA_ERR_LAUNCH;
  }
  CheckPlan k = check_plan(a);
  if (int r = decode_refused(a, k.chunk ? &k.c : nullptr)) return r;
  uint32_t* word = nullptr;
  if (k.word && a.workspace != nullptr && a.workspace_bytes >= word_offset(a) + kWordBytes)
    word = reinterpret_cast<uint32_t*>(static_cast<char*>(a.workspace) + word_offset(a));
  const bool host_order = k.word && word == nullptr;   // no room for the word: launch nothing before the result is here
  if (host_order) k.inside = false;
  uint32_t* host = nullptr;
  const int slot = take_slot(false, a.device, &host);
  if (slot < 0) return FA_ERR_LAUNCH;
  int r = FA_OK;
  bool queued = false;                                 // a kernel that writes the host word is on the stream
  if (!k.inside) {
    decode_check_kernel<<<1, 1024, 0, st>>>(a, host, word);
    r = check_launch("decode_check");
    queued = r == FA_OK;
  }
  if (r == FA_OK && !host_order) {
    if (k.chunk) {
      r = chunk_run(a, k.c, k.inside ? host : nullptr, word, &queued, st);
    } else {
      r = decode_run(a, k.inside ? DecodeCheck{host, nullptr} : DecodeCheck{nullptr, word}, st);
      queued = queued || r == FA_OK;
    }
  }
  if (queued) {
    const int w = await_slot(slot, failed, st);
    if (r == FA_OK) r = w;
  }
  g_slots.give(slot, queued);
  if (r != FA_OK || *failed || !host_order) return r;
  return k.chunk ? chunk_run(a, k.c, nullptr, nullptr, nullptr, st) : decode_run(a, DecodeCheck{nullptr, nullptr}, st);
}

// ---------------------------------------------------------------------------------------
// Decode without any allocation by anyone: the split-KV partials live in a fixed array
// that is part of the library image.
// ---------------------------------------------------------------------------------------
constexpr size_t kStaticScratchBytes = 16u << 20;  // 16 MiB, held by every GPU that loads the library
static __device__ __align__(256) unsigned char g_decode_static_scratch[kStaticScratchBytes];

// In host code the array's name is only a handle: the device address has to be asked for,
// once per device, while that device is current.
static void* static_scratch_ptr(int device) {
  constexpr int kMaxDevices = 64;
  static void* ptrs[kMaxDevices] = {nullptr};
  static std::mutex mu;
  if (device < 0 || device >= kMaxDevices) {
    set_error("device ordinal %d out of range for the static decode scratch", device);
    return nullptr;
  }
  std::lock_guard<std::mutex> lock(mu);
  if (ptrs[device] == nullptr) {
    void* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_decode_static_scratch);
    if (e != cudaSuccess || p == nullptr) {
      set_error("cudaGetSymbolAddress(static decode scratch) on device %d: %s", device,
                cudaGetErrorString(e));
      return nullptr;
    }
    ptrs[device] = p;
  }
  return ptrs[device];
}

size_t decode_static_scratch_bytes() { return kStaticScratchBytes; }

// Pieces of a full cache when each is a multiple of 64 keys, from 256 keys on of 256.
static int whole_splits(const fa_decode_args& a) {
  const int64_t cap = a.block_table ? (int64_t)a.block_table_stride * a.page_size : a.page_size;
  int64_t keys = (cap + a.num_splits - 1) / a.num_splits;
  keys = (keys + 63) / 64 * 64;
  if (keys >= 256) keys = (keys + 255) / 256 * 256;
  const int64_t n = keys > 0 ? (cap + keys - 1) / keys : 1;
  return n < 1 ? 1 : (int)n;
}

int decode_paged_static(const fa_decode_args& a, cudaStream_t st) {
  if (a.batch == 0 || a.seqlen_q == 0 || a.heads_q == 0) return FA_OK;
  fa_decode_args b = a;
  // Fewer pieces rather than a refusal: they cost time where a sequence is long and the batch small, and such
  // calls fit.  A number of pieces that the caller asked for stands for pieces of whole 64 or 256 keys.
  if (decode_workspace_bytes(b) > kStaticScratchBytes) {
    if (a.num_splits > 0) {
      b.num_splits = whole_splits(a);
    } else {
      for (b.num_splits = 8; b.num_splits > 1 && decode_workspace_bytes(b) > kStaticScratchBytes;) b.num_splits /= 2;
    }
  }
  const size_t need = decode_workspace_bytes(b);
  if (need > kStaticScratchBytes) {
    set_error("fa_decode_paged_static: this problem needs %zu bytes of split-KV scratch but the "
              "built-in array holds %zu; pass a smaller num_splits or use fa_decode_paged with "
              "your own workspace", need, kStaticScratchBytes);
    return FA_ERR_WORKSPACE;
  }
  void* p = static_scratch_ptr(a.device);
  if (p == nullptr) return FA_ERR_LAUNCH;
  b.workspace = p;
  b.workspace_bytes = kStaticScratchBytes;
  return decode_paged(b, st);
}

}  // namespace fa
