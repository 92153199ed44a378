// Forward attention on the 5th-generation tensor cores with ONE tile of 128 query rows per CTA and two
// softmax warpgroups that take its key tiles in turn.  Used where the two-tile kernels (fwd_sm100.cu,
// fwd_persist_sm100.cu) do not fit:
//
//   head_dim 256   two output accumulators and two score buffers would need 768 tensor-memory columns;
//   few tiles      dense problems of head_dim 64 and 128 with few tiles per SM, or very long ones: see
//                  one_tile_is_faster() in fwd_sm100.cu;
//   KV cache       a chunk of new tokens against a paged or contiguous cache.  The query heads of a KV head
//                  are packed into the rows of a tile (row = token * group + head), so a K/V tile is
//                  read once per group and a short chunk still fills its tile.
//
//   warps 0-3   softmax group 0 : key tiles 0, 2, 4, ...
//   warps 4-7   softmax group 1 : key tiles 1, 3, 5, ...
//   warp  8     TMA producer    : the Q tile once, then K/V through a ring of 128-key x 128-column units
//   warp  9     MMA issuer      : S[j] = Q K_j^T (SS);  O += P_j V_j (A = P_j from tensor memory)
//   warps 10-11 idle (they complete the warpgroup that gives its registers to the softmax groups)
//
// For a KV cache P is held in two 16-bit parts, the second in the other 64 columns of its score buffer, and P V is two
// products per 16 keys.  The kernel these calls came from had a maximum per warp and 16 keys, and every new maximum is a
// probability without rounding; with one per 128 keys the outputs were 4 to 8 % further from float64 over chunks of 4 to
// 600 tokens, with two parts they are 16 to 23 % closer.  Rounding no longer depends on the maximum then, so the
// accumulator is rescaled past 2^8 only.  Four chunks of 256 tokens against 1024 to 8192: 194 -> 207 us.
//
// Tensor memory (512 columns): two score buffers and a 256-column accumulator at head_dim 256, else
// three score buffers.  P_j overwrites the first 64 columns of its score buffer; Q K^T of the tile that
// takes the buffer next is issued right after P_j V_j, which reads them, in the in-order pipe.  Neither
// group waits for the other's exponentials: what a tile needs from the tile before it is only the
// row maximum that all exponents are taken relative to.  It sits in shared memory (mref), is read and
// raised in tile order -- only when a row's maximum grows by more than cfg.rescale_at, and the accumulator is then
// rescaled by the group that raised it.  The row sum travels with it, one tile late: a group adds the sum of its tile
// j when it settles tile j + 2, so that nothing waits for it and the sums are added in tile order all the same.  The results
// are therefore those of the two-tile kernels bit for bit, and which kernel a call takes may depend on its batch:
// an entry has the same result in any batch.
//
// Bound: the tensor pipe needs 2 * head_dim * 8 cycles per tile (128 x 128 scores), the exponentials
// 1024, and two groups have the load-max-exp-store chain of about 2200 cycles per tile half each.
// Every mbarrier wait is bounded; on timeout the CTA raises a status word, frees its tensor memory and
// returns.
#include <cmath>
#include <type_traits>

#include "common.cuh"
#include "cache_geo.cuh"
#include "sm100.cuh"

namespace fa {

using namespace sm100;

__device__ int g_fwd_alt_status = 0;

namespace {

constexpr int kBM = 128;          // query rows of the tile
constexpr int kBN = 128;          // keys per tile
constexpr int kThreads = 384;
constexpr int kMaxStages = 8;

template <int D> struct ACfg {
  static constexpr int kUnitCols = D < 128 ? D : 128;
  static constexpr int kUnits = D / kUnitCols;                      // ring units of a K (or V) tile
  static constexpr int kUnitBytes = kBN * kUnitCols * 2;
  static constexpr int kBoxes = kUnitCols / 64;                     // TMA boxes of a unit
  static constexpr int kStages = D == 256 ? 5 : D == 128 ? 5 : 8;
  static constexpr int kSBuf = D == 256 ? 2 : 3;                    // score buffers
  static constexpr int kOCol = kSBuf * 128;                         // first column of the accumulator
  static constexpr int kQBytes = kBM * D * 2;
  static constexpr int kSmemTiles = kQBytes + kStages * kUnitBytes;
  static constexpr int kSmemBytes = kSmemTiles + 1024 /*align slack*/ + 2048 /*AShared*/;
  static_assert(kSmemBytes <= 227 * 1024, "shared memory budget");
};

struct AShared {
  uint64_t q_full;
  uint64_t kv_full[kMaxStages];
  uint64_t kv_empty[kMaxStages];
  uint64_t s_full[3];      // [buffer]: scores computed
  // (Barriers that count threads: none may arrive for a phase before the one ahead of it is complete.  For P: the next scores
  // of the same buffer are issued behind its p_ready.  For `decided`: a group settles tile j + 2 after the other group's
  // tile j + 1, which each of that group's threads settled after tile j was settled by all.)
  uint64_t p_half[3];      // [buffer]: the first 64 keys of P written back (128 arrivals)
  uint64_t p_ready[3];     // [buffer]: P written back (128 arrivals)
  uint64_t o_done[3];      // [buffer]: its P V finished
  uint64_t decided[2];     // [group]: mref settled for the group's tile (128 arrivals)
  uint32_t tmem_base;
  volatile int abort_flag;
  int last;                // split keys: this CTA merges the pieces
  alignas(16) float mref[kBM];
  float lrun[kBM];         // row sums, up to the tile before the last one each group has settled
};
static_assert(sizeof(AShared) <= 2048, "AShared must fit its reserve");

__device__ __forceinline__ bool wait_bar(uint64_t* bar, uint32_t parity, AShared* sh, int code) {
  return bounded_wait(bar, parity, &sh->abort_flag, &g_fwd_alt_status, code);
}

// Barrier 1 of the 256 softmax threads: is the predicate set in any of them?
__device__ __forceinline__ bool any_of_256(bool x) {
  int r;
  asm volatile(
      "{\n"
      ".reg .pred p, q;\n"
      "setp.ne.s32 p, %1, 0;\n"
      "barrier.cta.red.or.pred q, 1, 256, p;\n"
      "selp.s32 %0, 1, 0, q;\n"
      "}\n"
      : "=r"(r) : "r"((int)x) : "memory");
  return r != 0;
}

// First of two parts: rounded from a little less, so that the rest is never negative (an infinite value times two parts
// of one sign stays infinite).
template <typename T> __device__ __forceinline__ float2 first_part(float2 p);
template <> __device__ __forceinline__ float2 first_part<__half>(float2 p) {
  return f2mul(p, make_float2(1.f - 0x1p-11f, 1.f - 0x1p-11f));
}
template <> __device__ __forceinline__ float2 first_part<__nv_bfloat16>(float2 p) {
  return f2mul(p, make_float2(1.f - 0x1p-8f, 1.f - 0x1p-8f));
}

template <typename T> struct AFmt;
template <> struct AFmt<__half> { static constexpr int code = 0; };
template <> struct AFmt<__nv_bfloat16> { static constexpr int code = 1; };

// What a CTA works on.
struct Tile {
  int b, h;                // sequence; first query head of the rows
  int hk, batch_row;       // KV head; batch coordinate of a contiguous K/V
  int m0, rows;            // first row of the tile, rows of the problem (tokens * packed heads)
  int pack_log2;           // log2 of the query heads packed into a tile's rows
  int pos0;                // position of row r: pos0 + (r >> pack_log2)
  int k_len;
  int key_off;             // added to a key to give its row (packed batches, left padding)
  int n_hi, nt;            // key tiles [n_hi - nt, n_hi); tile j of the CTA is n_hi - 1 - j
  int q_row0, q_boff;      // dense: coordinates of the query rows
  int part, parts;         // piece of the keys
};

}  // namespace

// kPoly > 0: every kPoly-th pair of exponentials of unmasked tiles on the FMA pipe, as in fwd_persist_sm100.cu.
// kCache: K/V through the page table of a cache, query heads packed into rows, optional key pieces.
// kGrid: the CTA's tile is its grid index (dense calls whose order does not matter, packed ones without a list); as one of
// several ways in one kernel it took a CTA 0.2 us longer to start: 4096 packed sequences of 16 to 128, 8 heads of 256,
// 2063 -> 2001 us.
template <typename T, int D, bool kExtras, bool kCache, int kPoly, bool kGrid = false>
__global__ void __launch_bounds__(kThreads, 1)
fwd_alt_sm100_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                     const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmO,
                     const fa_attn_args p, const ScoreCfg cfg, const CacheGeo geo, int* const host_status) {
  constexpr bool kPvSplit = !kExtras, kTwoParts = kCache;
  // Head_dim 256 rescales on nearly every tile (rescale_at = 0), and with the rescale ahead of the exponentials the product
  // of the tile before, the rescale and the exponentials came one after the other.  Behind them, they run under that
  // product: 2 x 1999 tokens of 16 heads, causal, 115 -> 107 us.  Where rescales are rare (all others) it only costs
  // registers: a chunk of 4 x 256 tokens 182 -> 185 us.
  constexpr bool kLate = D == 256;
  using C = ACfg<D>;
  constexpr int S = C::kStages, NB = C::kSBuf, NU = C::kUnits;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* tiles = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  AShared* sh = reinterpret_cast<AShared*>(tiles + C::kSmemTiles);
  const uint32_t sQ = smem_u32(tiles);
  const uint32_t sKV = sQ + C::kQBytes;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  // ---- what this CTA works on --------------------------------------------------------------
  Tile w;
  bool packed = false;                           // rows of several sequences in one tensor (cu_seqlens)
  if constexpr (kCache) {
    if (geo.bad && *geo.bad) return;
    const int heads = p.heads_q >> geo.pack_log2;        // units of heads per sequence
    w.pack_log2 = geo.pack_log2;
    w.rows = geo.tokens << geo.pack_log2;
    const int mtiles = (w.rows + kBM - 1) / kBM;
    int i = blockIdx.x;
    w.part = i % geo.parts;
    i /= geo.parts;
    const int mt = mtiles - 1 - i % mtiles;
    i /= mtiles;
    const int hu = i % heads, rank = i / heads;
    // long sequences first (their CTAs set the time of the launch)
    w.b = rank;
    if (p.batch > 1 && p.batch <= 32) {
      const int mine = lane < p.batch ? geo.seqlens[lane] : -1;
      int before = 0;
      for (int o = 0; o < p.batch; ++o) {
        const int other = __shfl_sync(0xffffffffu, mine, o);
        before += other > mine || (other == mine && o < lane);
      }
      w.b = __ffs(__ballot_sync(0xffffffffu, lane < p.batch && before == rank)) - 1;
    }
    w.h = hu << geo.pack_log2;
    w.hk = w.h / (p.heads_q / p.heads_kv);
    w.m0 = mt * kBM;
    w.k_len = min(max(geo.seqlens[w.b], 0) + geo.n_new, geo.capacity);
    w.pos0 = w.k_len - geo.tokens;
    w.key_off = geo.leftpad ? geo.leftpad[w.b] : 0;
    w.batch_row = geo.batch_idx ? geo.batch_idx[w.b] : w.b;
    w.q_row0 = 0;
    w.q_boff = w.b;
  } else {
    packed = p.cu_seqlens_q != nullptr;
    int mt;
    SeqInfo si;
    if constexpr (kGrid) {
      mt = cfg.causal ? gridDim.x - 1 - blockIdx.x : blockIdx.x;   // heavy tiles first
      w.h = blockIdx.y;
      w.b = blockIdx.z;
      si = seq_info(p, w.b);
    } else if (packed) {
      if (!packed_tile<kBM>(p, cfg, lane, w.h, w.b, si, mt)) return;
    } else {
      const int mtiles = (p.seqlen_q + kBM - 1) / kBM;
      dense_block(p, cfg, mtiles, w.b, w.h, mt);
      if (cfg.causal) mt = mtiles - 1 - mt;        // heavy tiles first
      si = seq_info(p, w.b);
    }
    w.hk = w.h / (p.heads_q / p.heads_kv);
    w.m0 = mt * kBM;
    w.rows = si.q_len;
    w.pack_log2 = 0;
    if (w.m0 >= w.rows) return;
    w.k_len = si.k_len;
    w.pos0 = p.q_pos_offset;
    w.key_off = (int)si.k_row0;
    w.batch_row = (int)si.k_boff;
    w.q_row0 = (int)si.q_row0;
    w.q_boff = (int)si.q_boff;
    w.part = 0;
  }
  const int tq_min = w.pos0 + (w.m0 >> w.pack_log2);
  const int tq_max = w.pos0 + ((min(w.m0 + kBM, w.rows) - 1) >> w.pack_log2);
  const int tq_end = w.pos0 + ((w.m0 + kBM - 1) >> w.pack_log2);     // of the tile's last row, existing or not
  {
    int klo, khi;
    visible_key_range(cfg, tq_min, tq_max, w.k_len, klo, khi);
    const int lo = klo / kBN, hi = (khi + kBN - 1) / kBN;
    const int all = khi > klo ? hi - lo : 0;
    w.parts = 1;
    if (kCache) {
      w.parts = max(1, min(geo.parts, all));
      if (w.part >= w.parts) return;
    }
    const int first = (int)((int64_t)w.part * all / w.parts), last = (int)((int64_t)(w.part + 1) * all / w.parts);
    w.n_hi = lo + last;
    w.nt = last - first;
  }
  const int nt = w.nt;

  if (tid == 0) {
    mbar_init(smem_u32(&sh->q_full), 1);
    for (int i = 0; i < NB; ++i) {
      mbar_init(smem_u32(&sh->s_full[i]), 1);
      mbar_init(smem_u32(&sh->o_done[i]), 1);
      mbar_init(smem_u32(&sh->p_half[i]), 128);
      mbar_init(smem_u32(&sh->p_ready[i]), 128);
    }
    for (int i = 0; i < S; ++i) {
      mbar_init(smem_u32(&sh->kv_full[i]), 1);
      mbar_init(smem_u32(&sh->kv_empty[i]), 1);
    }
    mbar_init(smem_u32(&sh->decided[0]), 128);
    mbar_init(smem_u32(&sh->decided[1]), 128);
    sh->abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 8) {
    tmem_alloc(smem_u32(&sh->tmem_base), 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sh->tmem_base;

  if (warp >= 10) {
    reg_dealloc<72>();
  } else if (warp == 8) {
    // ------------------------------- TMA producer ---------------------------------------
    reg_dealloc<72>();
    if (nt > 0 && (lane == 0 || (kCache && geo.box_rows < kBN))) {
      if (lane == 0) {
        prefetch_tmap(&tmQ);
        prefetch_tmap(&tmK);
        prefetch_tmap(&tmV);
        prefetch_tmap(&tmO);
        const uint32_t bar = smem_u32(&sh->q_full);
        mbar_expect_tx(bar, C::kQBytes);
        for (int bx = 0; bx < D / 64; ++bx)
          tma_load_4d(sQ + bx * (kBM * 128), &tmQ, bar, bx * 64, w.h, w.q_row0 + (w.m0 >> w.pack_log2), w.q_boff);
      }
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      // Page of box `lane` of a key tile (boxes of one page each; a contiguous cache is one page); read one
      // tile ahead of its use.  No divisions here and no lock-step of the warp unless a tile has several
      // boxes: with both, a load took this warp 900 cycles, and two of them per tile were what bounded
      // the kernel.
      const bool many = kCache && geo.box_rows < kBN;
      const int box_log2 = many ? 31 - __clz(geo.box_rows) : 7;
      auto page_of = [&](int tile) {
        int pg = w.batch_row;
        if (kCache && geo.table) {
          const int key = tile * kBN + (many ? lane << box_log2 : 0);
          pg = (lane < (kBN >> box_log2) && key < w.k_len)
                   ? geo.table[(int64_t)w.b * geo.table_stride + (geo.page_log2 >= 0 ? key >> geo.page_log2 : key / geo.page_size)]
                   : 0;
        }
        return pg;
      };
      auto load_tile = [&](const CUtensorMap* tm, int tile, int pages) {
#pragma unroll
        for (int un = 0; un < NU; ++un) {
          const uint32_t bar = smem_u32(&sh->kv_full[stage]);
          const uint32_t dst = sKV + stage * C::kUnitBytes;
          if (many) {
            // boxes that start past the last key are not loaded (their rows are masked, and zeroed in V)
            if (lane == 0) ok = ok && wait_bar(&sh->kv_empty[stage], phase ^ 1, sh, 11);
            ok = __shfl_sync(0xffffffffu, (int)ok, 0) != 0;
            if (!ok) return;
            const int n = min(kBN >> box_log2, ((w.k_len - tile * kBN - 1) >> box_log2) + 1);
            if (lane == 0) mbar_expect_tx(bar, n * (C::kUnitCols * 2 << box_log2));
            __syncwarp();
            if (lane < n) {
              for (int bx = 0; bx < C::kBoxes; ++bx)
                tma_load_4d(dst + bx * (kBN * 128) + (lane << box_log2) * 128, tm, bar, un * C::kUnitCols + bx * 64, w.hk, 0, pages);
            }
          } else if (lane == 0) {
            ok = ok && wait_bar(&sh->kv_empty[stage], phase ^ 1, sh, 11);
            if (!ok) return;
            const int row = !kCache || geo.table == nullptr ? tile * kBN + w.key_off
                            : geo.page_log2 >= 0            ? (tile * kBN) & (geo.page_size - 1)
                                                            : (tile * kBN) % geo.page_size;
            mbar_expect_tx(bar, C::kUnitBytes);
            for (int bx = 0; bx < C::kBoxes; ++bx)
              tma_load_4d(dst + bx * (kBN * 128), tm, bar, un * C::kUnitCols + bx * 64, w.hk, row, pages);
          }
          if (++stage == S) { stage = 0; phase ^= 1; }
        }
      };
      // order of use: K_0 .. K_(NB-1), then V_j, K_(j+NB)
      int pg[NB + 1];
#pragma unroll
      for (int i = 0; i < NB; ++i) pg[i] = i < nt ? page_of(w.n_hi - 1 - i) : 0;
#pragma unroll
      for (int i = 0; i < NB; ++i)
        if (i < nt) load_tile(&tmK, w.n_hi - 1 - i, pg[i]);
      pg[NB] = NB < nt ? page_of(w.n_hi - 1 - NB) : 0;
      for (int j = 0; j < nt && ok; ++j) {
        const int nxt = j + NB + 1 < nt ? page_of(w.n_hi - 2 - j - NB) : 0;
        load_tile(&tmV, w.n_hi - 1 - j, pg[0]);
        if (j + NB < nt) load_tile(&tmK, w.n_hi - 1 - j - NB, pg[NB]);
#pragma unroll
        for (int i = 0; i < NB; ++i) pg[i] = pg[i + 1];
        pg[NB] = nxt;
      }
    }
  } else if (warp == 9) {
    // ------------------------------- MMA issuer -----------------------------------------
    // The whole warp runs the control flow in lock step and every lane polls the barriers;
    // the lane chosen once by elect_one issues the MMAs and commits.
    reg_dealloc<72>();
    if (nt > 0) {
      constexpr uint32_t idesc_qk = make_idesc(1, AFmt<T>::code, 0, 0, kBM, kBN);
      constexpr uint32_t idesc_pv = make_idesc(1, AFmt<T>::code, 0, 1, kBM, C::kUnitCols);
      const uint32_t leader = elect_one() ? 1u : 0u;
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      auto wwait = [&](uint64_t* bar, uint32_t parity, int code) {
        if (ok) ok = wait_bar(bar, parity, sh, code);
        tc_fence_after();
      };
      auto advance = [&]() { if (++stage == S) { stage = 0; phase ^= 1; } };
      auto issue_qk = [&](int buf) {                       // S[buf] = Q K^T with the next K tile of the ring
#pragma unroll
        for (int un = 0; un < NU; ++un) {
          wwait(&sh->kv_full[stage], phase, 22);
          if (!ok) return;
          const uint64_t dq = make_smem_desc(sQ + un * (C::kUnitCols / 64) * (kBM * 128), 16, 1024);
          const uint64_t dk = make_smem_desc(sKV + stage * C::kUnitBytes, 16, 1024);
#pragma unroll
          for (int kk = 0; kk < C::kUnitCols / 16; ++kk) {
            const uint32_t o = ((kk / 4) * (kBM * 128) + (kk % 4) * 32) >> 4;
            mma_f16_ss_lp(tmem + buf * kBN, dq + o, dk + o, idesc_qk, (un > 0 || kk > 0) ? 1u : 0u, leader);
          }
          mma_commit_lp(smem_u32(&sh->kv_empty[stage]), leader);
          advance();
        }
        mma_commit_lp(smem_u32(&sh->s_full[buf]), leader);
      };
      wwait(&sh->q_full, 0, 21);
      for (int i = 0; i < NB && i < nt && ok; ++i) issue_qk(i);
      int buf = 0;
      uint32_t par = 0;                                    // (j / NB) & 1
      for (int j = 0; j < nt && ok; ++j) {
        const uint32_t a = tmem + buf * kBN;
        // the V units of tile j are in the next NU stages
        int st[NU];
#pragma unroll
        for (int un = 0; un < NU; ++un) {
          wwait(&sh->kv_full[stage], phase, 24);
          st[un] = stage;
          advance();
        }
        if (!ok) break;
        if (kPvSplit) {
          wwait(&sh->p_half[buf], par, 25);
          if (!ok) break;
#pragma unroll
          for (int un = 0; un < NU; ++un) {
            const uint64_t dv = make_smem_desc(sKV + st[un] * C::kUnitBytes, kBN * 128, 1024);
#pragma unroll
            for (int kk = 0; kk < kBN / 32; ++kk) {
              mma_f16_ts_lp(tmem + C::kOCol + un * C::kUnitCols, a + kk * 8, dv + ((kk * 2048) >> 4), idesc_pv,
                            (j > 0 || kk > 0) ? 1u : 0u, leader);
              if (kTwoParts)
                mma_f16_ts_lp(tmem + C::kOCol + un * C::kUnitCols, a + 64 + kk * 8, dv + ((kk * 2048) >> 4), idesc_pv, 1u, leader);
            }
          }
        }
        wwait(&sh->p_ready[buf], par, 26);
        if (!ok) break;
#pragma unroll
        for (int un = 0; un < NU; ++un) {
          const uint64_t dv = make_smem_desc(sKV + st[un] * C::kUnitBytes, kBN * 128, 1024);
#pragma unroll
          for (int kk = kPvSplit ? kBN / 32 : 0; kk < kBN / 16; ++kk) {
            mma_f16_ts_lp(tmem + C::kOCol + un * C::kUnitCols, a + kk * 8, dv + ((kk * 2048) >> 4), idesc_pv,
                          (j > 0 || kk > 0) ? 1u : 0u, leader);
            if (kTwoParts)
              mma_f16_ts_lp(tmem + C::kOCol + un * C::kUnitCols, a + 64 + kk * 8, dv + ((kk * 2048) >> 4), idesc_pv, 1u, leader);
          }
          mma_commit_lp(smem_u32(&sh->kv_empty[st[un]]), leader);
        }
        mma_commit_lp(smem_u32(&sh->o_done[buf]), leader);
        if (j + NB < nt) issue_qk(buf);
        if (++buf == NB) { buf = 0; par ^= 1; }
      }
    }
  } else {
    // ------------------------------- softmax groups -------------------------------------
    reg_alloc<216>();
    const int x = warp >> 2;                         // group
    const int row_in_tile = (warp & 3) * 32 + lane;  // TMEM lane
    const int row = w.m0 + row_in_tile;
    const int qpos = w.pos0 + (row >> w.pack_log2);
    const uint32_t lane_addr = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t tO = tmem + lane_addr + C::kOCol;
    float slope = 0.f;
    if (kExtras && cfg.has_alibi)
      slope = p.alibi_slopes[w.b * p.heads_q + w.h + (row & ((1 << w.pack_log2) - 1))];
    // of this group's latest tile: the factor its maximum asked of what came before, and its row sum
    float alpha = 1.f, sum = 0.f;
    bool ok = true;
    const bool zero_tail = kCache || packed;         // rows past k_len of the last V tile are not ours

    for (int j = x; j < nt && ok; j += 2) {
      const int buf = j % NB;
      const uint32_t par = (j / NB) & 1;
      const uint32_t tS = tmem + lane_addr + buf * kBN;
      const int k0 = (w.n_hi - 1 - j) * kBN;
      bool masked = (k0 + kBN > w.k_len);
      if (cfg.causal) masked |= (k0 + kBN - 1 > tq_min);
      if (cfg.wl >= 0) masked |= (k0 < tq_end - cfg.wl);
      if (cfg.wr >= 0) masked |= (k0 + kBN - 1 > tq_min + cfg.wr);

      ok = wait_bar(&sh->s_full[buf], par, sh, 31 + x);
      if (!ok) break;
      tc_fence_after();

      // ---- the 128 scores of this row into registers -------------------------------------
      uint32_t r[4][32];
#pragma unroll
      for (int cc = 0; cc < 4; ++cc) tmem_ld32(tS + cc * 32, r[cc]);
      tmem_wait_ld();

      const bool prescaled = kExtras || masked;
      ColMask cm;
      if (masked) {
        int vk_lo, vk_hi;
        visible_k_interval(cfg, qpos, w.k_len, vk_lo, vk_hi);
        cm = make_col_mask(vk_lo - k0, vk_hi - k0);
      }
      if (prescaled) {
        // score pipeline and mask applied once, in place; values end up in the log2 domain.
        // One body, compiled per (masked tile, soft cap): no branch inside the unrolled loops.
        const float dist0 = (float)(qpos - k0);
        auto score_tile = [&](auto mask_tag, auto cap_tag, auto abs_tag) {
          constexpr bool kMask = decltype(mask_tag)::value;
          constexpr bool kCap = decltype(cap_tag)::value;
          constexpr bool kAbs = decltype(abs_tag)::value;
          if (kExtras) {
            const FeatK fk = feat_k<kCap>(cfg, slope);
            const float2 step2 = make_float2(-2.f, -2.f);
            float2 d2 = make_float2(dist0, dist0 - 1.f);
#pragma unroll
            for (int cc = 0; cc < 4; ++cc) {
#pragma unroll
              for (int i = 0; i < 32; i += 2) {
                float2 v = score_unit_feat2<kCap, kAbs, true>(
                    fk, make_float2(__uint_as_float(r[cc][i]), __uint_as_float(r[cc][i + 1])), d2);
                if (kMask) {
                  v.x = col_visible(cm, cc * 32 + i) ? v.x : -INFINITY;
                  v.y = col_visible(cm, cc * 32 + i + 1) ? v.y : -INFINITY;
                }
                r[cc][i] = __float_as_uint(v.x);
                r[cc][i + 1] = __float_as_uint(v.y);
                d2 = f2add(d2, step2);
              }
            }
          } else {
#pragma unroll
            for (int cc = 0; cc < 4; ++cc) {
#pragma unroll
              for (int i = 0; i < 32; ++i) {
                float v = __uint_as_float(r[cc][i]) * cfg.scale_log2;
                if (kMask) v = col_visible(cm, cc * 32 + i) ? v : -INFINITY;
                r[cc][i] = __float_as_uint(v);
              }
            }
          }
        };
        const bool cap = kExtras && cfg.softcap > 0.f;
        const bool need_abs = kExtras && !cfg.causal;    // under the causal mask visible keys lie at distance >= 0
        auto run_score = [&](auto mask_tag) {
          if (cap) {
            if (need_abs) score_tile(mask_tag, std::true_type{}, std::true_type{});
            else score_tile(mask_tag, std::true_type{}, std::false_type{});
          } else {
            if (need_abs) score_tile(mask_tag, std::false_type{}, std::true_type{});
            else score_tile(mask_tag, std::false_type{}, std::false_type{});
          }
        };
        if (masked) run_score(std::true_type{});
        else run_score(std::false_type{});
      }

      // ---- rows past the last key hold other values, or none: out of P V ------------------
      // Their probabilities are exactly 0, but 0 * inf or 0 * NaN is NaN.  Only the first tile of a CTA can
      // reach past k_len, so the ring position of its V is a constant.  One thread per row.
      if (zero_tail && k0 + kBN > w.k_len) {
#pragma unroll
        for (int un = 0; un < NU; ++un) {
          const int pos = min(NB, nt) * NU + un;
          ok = ok && wait_bar(&sh->kv_full[pos % S], (pos / S) & 1, sh, 39);
          if (ok && k0 + row_in_tile >= w.k_len) {
            unsigned char* vrow = tiles + C::kQBytes + (pos % S) * C::kUnitBytes + row_in_tile * 128;
#pragma unroll
            for (int bx = 0; bx < C::kBoxes; ++bx) {
#pragma unroll
              for (int c = 0; c < 8; ++c)
                reinterpret_cast<uint4*>(vrow + bx * (kBN * 128))[c] = make_uint4(0u, 0u, 0u, 0u);
            }
          }
        }
        if (!ok) break;
        fence_proxy_async();
      }

      // ---- row maximum: eight chains of three-input maxima --------------------------------
      float mx;
      {
        float mt[8];
#pragma unroll
        for (int i = 0; i < 8; ++i)
          mt[i] = fmax3(__uint_as_float(r[0][i]), __uint_as_float(r[0][8 + i]), __uint_as_float(r[0][16 + i]));
#pragma unroll
        for (int i = 0; i < 8; ++i) mt[i] = fmaxf(mt[i], __uint_as_float(r[0][24 + i]));
#pragma unroll
        for (int cc = 1; cc < 4; ++cc) {
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            mt[i] = fmax3(mt[i], __uint_as_float(r[cc][i]), __uint_as_float(r[cc][8 + i]));
            mt[i] = fmax3(mt[i], __uint_as_float(r[cc][16 + i]), __uint_as_float(r[cc][24 + i]));
          }
        }
        mx = fmaxf(fmax3(mt[0], mt[1], mt[2]), fmaxf(fmax3(mt[3], mt[4], mt[5]), fmaxf(mt[6], mt[7])));
      }
      const float mul = !prescaled ? cfg.scale_log2 : ((kExtras && cfg.softcap > 0.f) ? cfg.softcap * FA_LOG2E : 1.f);
      mx *= mul;

      // ---- the maximum the exponents are relative to, settled in tile order ---------------
      float m_use;
      [[maybe_unused]] bool grown = false;             // kLate: a row of this warp wants the accumulator rescaled
      if (j == 0) {
        m_use = mx;
        sh->mref[row_in_tile] = mx;
        sh->lrun[row_in_tile] = 0.f;
      } else {
        ok = wait_bar(&sh->decided[x ^ 1], ((j - 1) >> 1) & 1, sh, 33 + x);
        if (!ok) break;
        const float m_old = sh->mref[row_in_tile];
        if (j >= 2) sh->lrun[row_in_tile] = __fadd_rn(__fmul_rn(sh->lrun[row_in_tile], alpha), sum);
        const bool need = mx > m_old + cfg.rescale_at;
        m_use = need ? mx : m_old;
        alpha = 1.f;
        if constexpr (kLate) {
          grown = __any_sync(0xffffffffu, need);
          if (need) alpha = exp2f(m_old - mx);                    // m_old = -inf -> 0
          if (need) sh->mref[row_in_tile] = mx;
        } else if (__any_sync(0xffffffffu, need)) {
          // The accumulator may be touched once P V of the tile before is finished: the one of this
          // tile cannot start before P is written below.  (Score buffers come round in order, so the
          // barrier's earlier phase is complete: the parity is not ambiguous.)
          const int pb = (j - 1) % NB;
          ok = wait_bar(&sh->o_done[pb], ((j - 1) / NB) & 1, sh, 35 + x);
          if (!ok) break;
          tc_fence_after();
          if (need) alpha = exp2f(m_old - mx);
          if (need) sh->mref[row_in_tile] = mx;
#pragma unroll
          for (int cc = 0; cc < D / 32; ++cc) {
            uint32_t ro[32];
            tmem_ld32(tO + cc * 32, ro);
            tmem_wait_ld();
#pragma unroll
            for (int i = 0; i < 32; ++i) ro[i] = __float_as_uint(__uint_as_float(ro[i]) * alpha);
            tmem_st32(tO + cc * 32, ro);
          }
          tmem_wait_st();
          tc_fence_before();
        }
      }
      mbar_arrive(smem_u32(&sh->decided[x]));
      const float m_safe = (m_use == -INFINITY) ? 0.f : m_use;

      // ---- P = exp2(s - m), row sum, P -> TMEM in place over S ----------------------------
      if (kPoly > 0 && !prescaled) {
        // the scores once more from tensor memory, a quarter at a time: the polynomial wants the registers
        const float2 mul2 = make_float2(mul, mul), nm2 = make_float2(-m_safe, -m_safe);
        float2 acc2[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
        uint32_t ra[32], rb[32];
        tmem_ld32(tS, ra);
#pragma unroll
        for (int cc = 0; cc < 4; ++cc) {
          uint32_t (&cur)[32] = (cc & 1) ? rb : ra;
          uint32_t (&nxt)[32] = (cc & 1) ? ra : rb;
          tmem_wait_ld();
          if (cc < 3) tmem_ld32(tS + (cc + 1) * 32, nxt);
          uint32_t pk[16];
#pragma unroll
          for (int i = 0; i < 32; i += 2) {
            const float2 a = f2fma(make_float2(__uint_as_float(cur[i]), __uint_as_float(cur[i + 1])), mul2, nm2);
            const float2 pe = ex2_pair<kPoly>(a, i >> 1);
            pk[i >> 1] = Elem<T>::pack(pe.x, pe.y);
            acc2[(i >> 1) & 1] = f2add(acc2[(i >> 1) & 1], pe);
          }
          tmem_st16(tS + cc * 16, pk);
          if (kPvSplit && cc == 1 && !(kLate && grown)) {
            tmem_wait_st();
            tc_fence_before();
            mbar_arrive(smem_u32(&sh->p_half[buf]));
          }
        }
        sum = (acc2[0].x + acc2[0].y) + (acc2[1].x + acc2[1].y);
      } else {
        const float2 mul2 = make_float2(mul, mul), nm2 = make_float2(-m_safe, -m_safe);
        float2 acc2[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
        for (int cc = 0; cc < 4; ++cc) {
          uint32_t pk[16], rest[16];
#pragma unroll
          for (int i = 0; i < 32; i += 2) {
            const float2 a = f2fma(make_float2(__uint_as_float(r[cc][i]), __uint_as_float(r[cc][i + 1])), mul2, nm2);
            const float2 pe = make_float2(ex2(a.x), ex2(a.y));
            acc2[(i >> 1) & 1] = f2add(acc2[(i >> 1) & 1], pe);
            if (kTwoParts) {
              const float2 first = first_part<T>(pe);
              pk[i >> 1] = Elem<T>::pack(first.x, first.y);
              const float2 left = f2fma(Elem<T>::unpack(pk[i >> 1]), make_float2(-1.f, -1.f), pe);
              rest[i >> 1] = Elem<T>::pack(left.x, left.y);
            } else {
              pk[i >> 1] = Elem<T>::pack(pe.x, pe.y);
            }
          }
          tmem_st16(tS + cc * 16, pk);
          if (kTwoParts) tmem_st16(tS + 64 + cc * 16, rest);
          if (kPvSplit && cc == 1 && !(kLate && grown)) {
            tmem_wait_st();
            tc_fence_before();
            mbar_arrive(smem_u32(&sh->p_half[buf]));
          }
        }
        sum = (acc2[0].x + acc2[0].y) + (acc2[1].x + acc2[1].y);
      }

      if constexpr (kLate) {
        if (grown) {                                   // (waits as above)
          const int pb = (j - 1) % NB;
          ok = wait_bar(&sh->o_done[pb], ((j - 1) / NB) & 1, sh, 35 + x);
          if (!ok) break;
          tc_fence_after();
#pragma unroll
          for (int c0 = 0; c0 < D / 32; c0 += 4) {     // 128 columns in flight
            uint32_t ro[4][32];
#pragma unroll
            for (int c = 0; c < 4; ++c) tmem_ld32(tO + (c0 + c) * 32, ro[c]);
            tmem_wait_ld();
#pragma unroll
            for (int c = 0; c < 4; ++c) {
#pragma unroll
              for (int i = 0; i < 32; ++i) ro[c][i] = __float_as_uint(__uint_as_float(ro[c][i]) * alpha);
              tmem_st32(tO + (c0 + c) * 32, ro[c]);
            }
          }
        }
      }
      tmem_wait_st();
      tc_fence_before();
      if (kLate && kPvSplit && grown) mbar_arrive(smem_u32(&sh->p_half[buf]));
      mbar_arrive(smem_u32(&sh->p_ready[buf]));
    }

    // ---- epilogue: both groups, half of the columns each ----------------------------------
    asm volatile("bar.sync 1, 256;\n" ::: "memory");     // every decision is made
    const float m_fin = nt > 0 ? sh->mref[row_in_tile] : -INFINITY;
    // the row sum: the tile before the last, then the last
    const bool last_group = ((nt - 1) & 1) == x;
    if (nt > 0 && !last_group) sh->lrun[row_in_tile] = __fadd_rn(__fmul_rn(sh->lrun[row_in_tile], alpha), sum);
    if (ok && nt > 0) ok = wait_bar(&sh->o_done[(nt - 1) % NB], ((nt - 1) / NB) & 1, sh, 37 + x);
    const bool failed = any_of_256(!ok || sh->abort_flag != 0);
    tc_fence_after();
    float l_all = 0.f;
    if (nt > 0) {
      if (last_group) sh->lrun[row_in_tile] = __fadd_rn(__fmul_rn(sh->lrun[row_in_tile], alpha), sum);
      asm volatile("bar.sync 1, 256;\n" ::: "memory");
      l_all = sh->lrun[row_in_tile];
    }
    if (!failed) {
      const float inv = l_all > 0.f ? 1.f / l_all : 0.f;
      const float lse = l_all > 0.f ? m_fin + log2f(l_all) : -INFINITY;
      const bool row_ok = row < w.rows;
      const bool piece = kCache && w.parts > 1;
      const bool via_tma = !piece && (!packed || w.m0 + kBM <= w.rows);
      const int64_t slot = blockIdx.x;
      T* og = reinterpret_cast<T*>(p.o) + (int64_t)w.q_boff * p.o_stride[0] +
              ((int64_t)w.q_row0 + (row >> w.pack_log2)) * p.o_stride[1] +
              (int64_t)(w.h + (row & ((1 << w.pack_log2) - 1))) * p.o_stride[2];
#pragma unroll
      for (int c2 = 0; c2 < D / 64; ++c2) {
        const int cc = x * (D / 64) + c2;                // 32 columns
        uint32_t ra[32];
        if (nt > 0) {
          tmem_ld32(tO + cc * 32, ra);
          tmem_wait_ld();
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) ra[i] = 0u;
        }
        if (piece) {
          float* dst = geo.ws + (slot * kBM + row_in_tile) * D + cc * 32;
#pragma unroll
          for (int i = 0; i < 32; i += 4) {
            if (row_ok)
              *reinterpret_cast<float4*>(dst + i) = make_float4(__uint_as_float(ra[i]) * inv, __uint_as_float(ra[i + 1]) * inv,
                                                                __uint_as_float(ra[i + 2]) * inv, __uint_as_float(ra[i + 3]) * inv);
          }
        } else {
#pragma unroll
          for (int i = 0; i < 32; i += 8) {
            uint4 v;
            v.x = Elem<T>::pack(__uint_as_float(ra[i]) * inv, __uint_as_float(ra[i + 1]) * inv);
            v.y = Elem<T>::pack(__uint_as_float(ra[i + 2]) * inv, __uint_as_float(ra[i + 3]) * inv);
            v.z = Elem<T>::pack(__uint_as_float(ra[i + 4]) * inv, __uint_as_float(ra[i + 5]) * inv);
            v.w = Elem<T>::pack(__uint_as_float(ra[i + 6]) * inv, __uint_as_float(ra[i + 7]) * inv);
            if (via_tma) {
              const int col = cc * 32 + i;
              st_shared_v4(sw128_addr(sQ + (col / 64) * (kBM * 128), row_in_tile, (col % 64) / 8), v);
            } else if (row_ok) {
              *reinterpret_cast<uint4*>(og + cc * 32 + i) = v;
            }
          }
        }
      }
      if (via_tma) {
        // staged over the Q tile, which no MMA reads any more
        fence_proxy_async();
        asm volatile("bar.sync 1, 256;\n" ::: "memory");
        if (tid == 0) {
#pragma unroll
          for (int bx = 0; bx < D / 64; ++bx)
            tma_store_4d(&tmO, sQ + bx * (kBM * 128), bx * 64, w.h, w.q_row0 + (w.m0 >> w.pack_log2), w.q_boff);
          tma_store_commit();
          tma_store_wait_read();
        }
      }
      if (!kCache && x == 0 && row_ok && p.lse2 != nullptr)
        p.lse2[(int64_t)w.q_boff * p.lse_stride[0] + ((int64_t)w.q_row0 + row) * p.lse_stride[1] +
               (int64_t)w.h * p.lse_stride[2]] = lse;
      if (piece) {
        // the CTA that finishes last merges; pieces are ordered before the count by the fence of each writer
        float* ws_l = geo.ws + (int64_t)gridDim.x * kBM * D;
        if (x == 0 && row_ok) ws_l[slot * kBM + row_in_tile] = lse;
        __threadfence();
        asm volatile("bar.sync 1, 256;\n" ::: "memory");
        if (tid == 0) {
          uint32_t* ctr = geo.counters + blockIdx.x / geo.parts;
          sh->last = atomicAdd(ctr, 1u) == (uint32_t)(w.parts - 1);
          if (sh->last) *ctr = 0u;
        }
        asm volatile("bar.sync 1, 256;\n" ::: "memory");
        if (sh->last) {
          __threadfence();
          const int64_t s0 = (int64_t)(blockIdx.x / geo.parts) * geo.parts;
          const int rows = min(kBM, w.rows - w.m0);
          // weights of the pieces per row, over the ring (every K/V tile has been read)
          float* wt = reinterpret_cast<float*>(tiles + C::kQBytes);
          if (tid < rows) {
            float m = -INFINITY, sum = 0.f;
            for (int s = 0; s < w.parts; ++s) m = fmaxf(m, ws_l[(s0 + s) * kBM + tid]);
            for (int s = 0; s < w.parts; ++s) {
              const float v = m == -INFINITY ? 0.f : exp2f(ws_l[(s0 + s) * kBM + tid] - m);
              wt[s * kBM + tid] = v;
              sum += v;
            }
            const float f = sum > 0.f ? 1.f / sum : 0.f;
            for (int s = 0; s < w.parts; ++s) wt[s * kBM + tid] *= f;
          }
          asm volatile("bar.sync 1, 256;\n" ::: "memory");
          // four elements of four rows per thread at a time, two pieces in flight each
          constexpr int kStep = 256 / (D / 4);             // rows between a thread's items
          const int d = (tid % (D / 4)) * 4;
          for (int r0 = tid / (D / 4); r0 < rows; r0 += 4 * kStep) {
            float4 acc[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) acc[k] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 2
            for (int s = 0; s < w.parts; ++s) {
#pragma unroll
              for (int k = 0; k < 4; ++k) {
                const int r = min(r0 + k * kStep, rows - 1);
                const float4 v = *reinterpret_cast<const float4*>(geo.ws + ((s0 + s) * kBM + r) * D + d);
                const float f = wt[s * kBM + r];
                acc[k].x += f * v.x; acc[k].y += f * v.y; acc[k].z += f * v.z; acc[k].w += f * v.w;
              }
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const int r = r0 + k * kStep, gr = w.m0 + r;
              if (r >= rows) break;
              uint2 pk;
              pk.x = Elem<T>::pack(acc[k].x, acc[k].y);
              pk.y = Elem<T>::pack(acc[k].z, acc[k].w);
              *reinterpret_cast<uint2*>(reinterpret_cast<T*>(p.o) + (int64_t)w.q_boff * p.o_stride[0] +
                                        (int64_t)(gr >> w.pack_log2) * p.o_stride[1] +
                                        (int64_t)(w.h + (gr & ((1 << w.pack_log2) - 1))) * p.o_stride[2] + d) = pk;
            }
          }
        }
      }
    } else if (kCache && w.parts > 1 && tid == 0) {
      // A piece whose wait ran out counts too: the counters outlive the call and have to be zero again once the
      // status has been cleared.  (If another CTA is the last, it merges what there is: the call has failed.)
      uint32_t* ctr = geo.counters + blockIdx.x / geo.parts;
      if (atomicAdd(ctr, 1u) == (uint32_t)(w.parts - 1)) *ctr = 0u;
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 8) tmem_dealloc(tmem, 512);
  if (tid == 0) report_abort(sh->abort_flag, host_status);
}

// ---------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------
static bool encode_rows(CUtensorMap* m, const void* base, int D, int heads, int64_t rows, int64_t batch, const int64_t* stride,
                        int box_heads, int box_rows) {
  // dims (innermost first): head_dim, heads, rows, batch (or page)
  const uint64_t dims[4] = {(uint64_t)D, (uint64_t)heads, (uint64_t)rows, (uint64_t)batch};
  const uint64_t strides[3] = {(uint64_t)stride[2] * 2, (uint64_t)stride[1] * 2, (uint64_t)stride[0] * 2};
  const uint32_t box[4] = {64, (uint32_t)box_heads, (uint32_t)box_rows, 1};
  return encode_tmap(m, base, 2, 4, dims, strides, box);
}

template <typename K>
static int launch_alt(K kern, int smem, dim3 grid, cudaStream_t st, const CUtensorMap (&tm)[4], const fa_attn_args& a,
                      const ScoreCfg& cfg, const CacheGeo& geo) {
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) {
    set_error("fwd_alt_sm100: cudaFuncSetAttribute(%d): %s", smem, cudaGetErrorString(e));
    return FA_ERR_LAUNCH;
  }
  kern<<<grid, kThreads, smem, st>>>(tm[0], tm[1], tm[2], tm[3], a, cfg, geo, host_wait_word(a.device));
  return check_launch("fwd_alt_sm100");
}

// Dense or packed forward; poly: exponentials as the persistent kernel would take them.  With ALiBi or a soft cap only head_dim 256 comes here (one_tile_is_faster()).
template <typename T, int D>
static int launch_rows(const fa_attn_args& a, const ScoreCfg& plain, bool poly, cudaStream_t st) {
  const bool packed = a.cu_seqlens_q != nullptr;
  const int64_t q_rows = packed ? a.total_q : a.seqlen_q, k_rows = packed ? a.total_k : a.seqlen_k;
  const int64_t batch = packed ? 1 : a.batch;
  auto map = [&](CUtensorMap* m, const void* base, const int64_t* stride, int heads, int64_t rows) {
    const int64_t s[3] = {packed ? rows * stride[1] : stride[0], stride[1], stride[2]};
    return encode_rows(m, base, D, heads, rows, batch, s, 1, 128);
  };
  CUtensorMap tm[4];
  if (!map(&tm[0], a.q, a.q_stride, a.heads_q, q_rows) || !map(&tm[1], a.k, a.k_stride, a.heads_kv, k_rows) ||
      !map(&tm[2], a.v, a.v_stride, a.heads_kv, k_rows) || !map(&tm[3], a.o, a.o_stride, a.heads_q, q_rows)) {
    set_error("fwd_alt_sm100: cuTensorMapEncodeTiled failed");
    return FA_ERR_LAUNCH;
  }
  ScoreCfg cfg = plain;
  const dim3 grid = packed ? packed_grid<kBM>(a, cfg) : dense_grid(a, (a.seqlen_q + kBM - 1) / kBM, cfg);
  const CacheGeo geo = {};
  auto go = [&](auto kern) { return launch_alt(kern, ACfg<D>::kSmemBytes, grid, st, tm, a, cfg, geo); };
  if constexpr (D == 256) {
    const bool extras = cfg.has_alibi || cfg.softcap > 0.f;
    if (packed ? !cfg.packed_list : cfg.unit_group == 0)
      return extras ? go(fwd_alt_sm100_kernel<T, D, true, false, 0, true>) : go(fwd_alt_sm100_kernel<T, D, false, false, 0, true>);
    if (extras) return go(fwd_alt_sm100_kernel<T, D, true, false, 0>);
  } else if (poly) {
    return go(fwd_alt_sm100_kernel<T, D, false, false, 4>);
  }
  return go(fwd_alt_sm100_kernel<T, D, false, false, 0>);
}

int fwd_alt_sm100(const fa_attn_args& a, const ScoreCfg& cfg, bool poly, cudaStream_t st) {
  const bool bf = a.dtype == FA_BF16;
  if (a.head_dim == 64) return bf ? launch_rows<__nv_bfloat16, 64>(a, cfg, poly, st) : launch_rows<__half, 64>(a, cfg, poly, st);
  if (a.head_dim == 128) return bf ? launch_rows<__nv_bfloat16, 128>(a, cfg, poly, st) : launch_rows<__half, 128>(a, cfg, poly, st);
  return bf ? launch_rows<__nv_bfloat16, 256>(a, cfg, poly, st) : launch_rows<__half, 256>(a, cfg, poly, st);
}

template <typename T, int D>
static int launch_cache(const fa_decode_args& d, const void* q, const int64_t* q_stride, const CacheGeo& geo,
                        const ScoreCfg& cfg, cudaStream_t st) {
  fa_attn_args a = {};
  a.dtype = d.dtype;
  a.device = d.device;
  a.batch = d.batch;
  a.seqlen_q = d.seqlen_q;
  a.heads_q = d.heads_q;
  a.heads_kv = d.heads_kv;
  a.head_dim = D;
  a.o = d.o;
  for (int i = 0; i < 3; ++i) a.o_stride[i] = d.o_stride[i];
  a.alibi_slopes = d.alibi_slopes;
  const int pack = 1 << geo.pack_log2;
  CUtensorMap tm[4];
  if (!encode_rows(&tm[0], q, D, d.heads_q, d.seqlen_q, d.batch, q_stride, pack, kBM / pack) ||
      !encode_rows(&tm[1], d.k_cache, D, d.heads_kv, d.page_size, d.num_pages, d.kc_stride, 1, geo.box_rows) ||
      !encode_rows(&tm[2], d.v_cache, D, d.heads_kv, d.page_size, d.num_pages, d.vc_stride, 1, geo.box_rows) ||
      !encode_rows(&tm[3], d.o, D, d.heads_q, d.seqlen_q, d.batch, d.o_stride, pack, kBM / pack)) {
    set_error("cache_sm100: cuTensorMapEncodeTiled failed");
    return FA_ERR_LAUNCH;
  }
  const int mtiles = (d.seqlen_q * pack + kBM - 1) / kBM;
  const dim3 grid((unsigned)d.batch * (d.heads_q / pack) * mtiles * geo.parts);
  if (cfg.has_alibi)
    return launch_alt(fwd_alt_sm100_kernel<T, D, true, true, 0>, ACfg<D>::kSmemBytes, grid, st, tm, a, cfg, geo);
  return launch_alt(fwd_alt_sm100_kernel<T, D, false, true, 0>, ACfg<D>::kSmemBytes, grid, st, tm, a, cfg, geo);
}

int cache_attention_sm100(const fa_decode_args& d, const void* q, const int64_t* q_stride, const CacheGeo& geo,
                          const ScoreCfg& cfg, cudaStream_t st) {
  const bool bf = d.dtype == FA_BF16;
  switch (d.head_dim) {
    case 64: return bf ? launch_cache<__nv_bfloat16, 64>(d, q, q_stride, geo, cfg, st) : launch_cache<__half, 64>(d, q, q_stride, geo, cfg, st);
    case 128: return bf ? launch_cache<__nv_bfloat16, 128>(d, q, q_stride, geo, cfg, st) : launch_cache<__half, 128>(d, q, q_stride, geo, cfg, st);
    case 256: return bf ? launch_cache<__nv_bfloat16, 256>(d, q, q_stride, geo, cfg, st) : launch_cache<__half, 256>(d, q, q_stride, geo, cfg, st);
  }
  set_error("cache_sm100: head_dim %d", d.head_dim);
  return FA_ERR_UNSUPPORTED;
}

int fwd_alt_sm100_status() {
  int v = 0;
  if (cudaMemcpyFromSymbol(&v, g_fwd_alt_status, sizeof(int)) != cudaSuccess) return -1;
  return v;
}
int fwd_alt_sm100_clear_status() {
  const int z = 0;
  return cudaMemcpyToSymbol(g_fwd_alt_status, &z, sizeof(int)) == cudaSuccess ? 0 : -1;
}

}  // namespace fa
