// Forward attention on the 5th-generation tensor cores, one tile of 128 query rows per work item and TWO PERSISTENT CTAs per SM.
//
// A CTA has a softmax warpgroup, a TMA producer, an MMA issuer and a store agent, one score buffer and one accumulator: half of an
// SM's tensor memory, shared memory and registers.  The two CTAs of an SM run out of phase by themselves, so that while
// one is in its exponentials the tensor pipe runs the other's P V and Q K^T, and the end of an item (the last P V and the output)
// lies under the other's work.
//
// Items come from a queue (queue.cuh).  The producer warp decodes the next one under the current one's last tile, and its Q and K_0 follow
// as soon as the last K tile has been read, so that its first scores are there when the softmax warps have staged the output;
// barriers, tensor memory and tensor maps are set up once.  With a CTA per tile instead, set-up, first loads, first scores, output and the
// change of CTAs took 12 k cycles per tile of rows, of 33 k where those had five key tiles.  Before -> after (us): 64 x 16 heads x
// 256 x 256 of 64 52.1 -> 39.7; 16 x 16 x 700, causal, head_dim 128 73.6 -> 60.8; 24 packed prompts of 17 to 2048, 32 heads over 8
// of 128 332 -> 280; 32 packed of 256 to 4096 with window, ALiBi and soft cap 1580 -> 1403; long rows of 64 (4 x 16 x 4096, causal) 219 -> 214; a
// launch of less than two items per CTA unchanged.
//
//   warps 0-3   softmax: one thread per query row (TMEM lane = row), all 128 scores of a tile in registers
//   warp  4     TMA producer and work queue: the Q tile once, then K/V tiles through a ring, in order of use K0 V0 K1 V1 ...
//   warp  5     MMA issuer: S = Q K_j^T (SS);  O += P V_j (A = P from tensor memory)
//   warp  6     store agent: hands the output, staged over the item's last V tile, to the TMA unit
//   warp  7     idle (completes the warpgroup that gives its registers to the softmax warps)
//
// At head_dim 128 P (fp16/bf16) overwrites the first 64 columns of S; Q K_{j+1}^T may overwrite it because P V_j precedes it
// in the in-order tensor pipe.  At head_dim 64 the accumulator leaves 64 columns, which P has to itself: Q K_{j+1}^T follows
// as soon as the scores of tile j are in registers and runs under their exponentials, where it came behind P V_j, with
// nothing of this CTA to do meanwhile (with a CTA per tile of rows, us, before -> after: 4 x 32 heads x 1024 x 1531 92.1 -> 88.0, 4 x 16 x 4096 causal
// 225 -> 219, 8 x 16 x 512 with dropout 25.3 -> 24.3, 24 packed of 64 to 2048 211 -> 206); rows that are too short for that keep P over S
// (p_over_s_is_faster).  Arithmetic, order of the tiles and of the sums are those of the two-tile kernels
// (fwd_sm100.cu, fwd_persist_sm100.cu): results are equal bit for bit.
//
// What bounds it: at head_dim 64 the exponentials, which the two CTAs contend for (1.8 k of 3.5 k cycles per tile and CTA, 1.02 k alone);
// at head_dim 128 the chain P V, Q K, load, maximum, exponentials (1.1 k of 4.5 k are spent waiting for the scores).
// Spills of the plain variants and those with options 72 to 96 bytes of stores a thread, of INT8 192 (what the compiler prints; it allots 128 registers).
// Tried: two threads per row (256 softmax threads of 104 registers, maxima and sums exchanged through shared memory), +2 to +15 %.
//
// TMEM (256 columns): S (128) | O (head_dim) | P of its own (64).  Every mbarrier wait is bounded.
#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "queue.cuh"
#define SKEW_TAG duo
#include "skew.cuh"
#include "sm100.cuh"

namespace fa {

using namespace sm100;

__device__ int g_fwd_duo_status = 0;

namespace {

constexpr int kBM = 128;          // query rows of the tile
constexpr int kBN = 128;          // keys per K/V tile
constexpr int kThreads = 256;
// 128 registers per thread at launch; the softmax warps take 216, the others keep 40
constexpr int kRegsSoftmax = 216, kRegsService = 40;
static_assert(128 * (kRegsSoftmax + kRegsService) <= 128 * kThreads, "register split");
constexpr int kSched = 4;         // depth of the in-CTA ring of work-queue entries
constexpr int kConsumers = 6;     // warps that read it: softmax, issuer, store agent (INT8: and the one that loads the scales)
constexpr int kSkSlots = 4;       // INT8: key tiles whose scales are staged ahead

template <int D> struct DCfg {
  static constexpr int kTileBytes = kBN * D * 2;
  static constexpr int kStages = (D == 128) ? 2 : 4;
  static constexpr int kBoxes = D / 64;
  static constexpr int kSmemTiles = (1 + kStages) * kTileBytes;
  static constexpr int kSmemBytes = kSmemTiles + 1024 /*align slack*/ + 1024 /*DShared*/;
  static constexpr int kSmemBytesInt8 = kSmemBytes + kSkSlots * kBN * 4;
  static_assert(2 * (kSmemBytesInt8 + 1024) <= 228 * 1024, "two CTAs per SM");
};

// A work item: one tile of query rows.  Decoded once, by the producer warp.
struct Item {
  int q_len, k_len, q_row0, k_row0, boff;  // geometry of its sequence
  int b, h, hk, m0;
  int n_hi, nt;            // step j works on key tile n_hi - 1 - j: masked tiles first; nt = -1: no more items
  int pad;
};
static_assert(sizeof(Item) == 48, "an item travels as three 16-byte words");

struct DShared {
  uint64_t q_full, q_empty;
  uint64_t kv_full[4];
  uint64_t kv_empty[4];
  uint64_t s_full;         // scores computed
  uint64_t s_free;         // P in columns of its own: scores in registers (128 arrivals)
  // (Barriers that count threads: none may arrive for a phase before the one ahead of it is complete.  For P: the next
  // scores, which a thread needs first, are issued behind p_ready -- with kOwnP behind s_free, but a thread writes
  // P only when the P V before, which was issued behind p_ready, has finished.)
  uint64_t p_half;         // the first 64 keys of P written back (128 arrivals)
  uint64_t p_ready;        // P written back (128 arrivals)
  uint64_t o_ready;        // the latest P V finished
  uint64_t stg_ready;      // output of an item staged for the store agent (128 arrivals)
  uint64_t stg_taken;      // ... and seen by it
  uint64_t sk_full[kSkSlots];    // INT8: scales of the tile's keys written (slot: tile % kSkSlots)
  uint64_t sk_empty[kSkSlots];   // ... read (128 arrivals: a slot is written again behind them)
  uint64_t sched_full[kSched];   // queue entry published by the producer warp
  uint64_t sched_empty[kSched];  // ... read by every consuming warp
  int4 sched_item[kSched][3];
  uint32_t tmem_base;
  volatile int abort_flag;
};

__device__ __forceinline__ bool wait_bar(uint64_t* bar, uint32_t parity, DShared* sh, int code) {
  return bounded_wait(bar, parity, &sh->abort_flag, &g_fwd_duo_status, code);
}

// Entry number idx of this CTA's queue ring, as seen by a consuming warp (all lanes together).
__device__ __forceinline__ Item sched_get(DShared* sh, int idx, bool& ok) {
  Item w;
  const int slot = idx % kSched;
  if (!wait_bar(&sh->sched_full[slot], (idx / kSched) & 1, sh, 61)) {
    ok = false;
    w.nt = -1;
    return w;
  }
  int4* dst = reinterpret_cast<int4*>(&w);
#pragma unroll
  for (int i = 0; i < 3; ++i) dst[i] = sh->sched_item[slot][i];
  __syncwarp();
  if ((threadIdx.x & 31) == 0) mbar_arrive(smem_u32(&sh->sched_empty[slot]));
  return w;
}

// Item of candidate c (whole warp); false where there is none.
__device__ __forceinline__ bool item_of(const fa_attn_args& p, const ScoreCfg& cfg, int by_weight, int c, int lane, Item& w) {
  SeqInfo si;
  int mt;
  if (!item_tile<kBM>(p, cfg, by_weight, c, lane, w.h, w.b, si, mt)) return false;
  w.m0 = mt * kBM;
  w.q_len = si.q_len;
  w.k_len = si.k_len;
  w.q_row0 = (int)si.q_row0;
  w.k_row0 = (int)si.k_row0;
  w.boff = (int)si.q_boff;
  w.hk = w.h / (p.heads_q / p.heads_kv);
  w.pad = 0;
  int klo, khi;
  visible_key_range(cfg, w.m0 + p.q_pos_offset, min(w.m0 + kBM, w.q_len) - 1 + p.q_pos_offset, w.k_len, klo, khi);
  w.n_hi = (khi + kBN - 1) / kBN;
  w.nt = khi > klo ? w.n_hi - klo / kBN : 0;
  return true;
}

static_assert(sizeof(DShared) <= 1024, "DShared must fit its reserve");

template <typename T> struct DFmt;
template <> struct DFmt<__half> { static constexpr int code = 0; };
template <> struct DFmt<__nv_bfloat16> { static constexpr int code = 1; };

}  // namespace

// kDrop: probabilities whose bit in cfg.keep is 0 do not enter P V (they stay in the row sum); the scale of
// the kept ones goes into the normalisation of the output.  kOwnP: P in columns of its own (head_dim 64).
// kInt8: INT8 scores on codes held as 16-bit floats (exact sums), sq and sk the scales of the query rows and of the keys, as in fwd_sm100.cu
// and equal to it bit for bit.  (The form with int32 accumulators, head_dim 128, spilled 290 bytes and was 13 to 22 % slower than there.)
template <typename T, int D, Feat kFeat, bool kDrop, bool kOwnP, bool kInt8 = false>
__global__ void __launch_bounds__(kThreads, 2)
fwd_duo_sm100_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                     const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmO,
                     const fa_attn_args p, const ScoreCfg cfg, const int ncand, const int by_weight, unsigned int* const queue,
                     int* const host_status, const float* const sq, const float* const sk) {
  constexpr bool kExtras = kFeat != Feat::kNone, kCap = kFeat == Feat::kCap;
  constexpr bool kPvSplit = !kExtras;     // P V in two key halves (measured: helps the plain variants only)
  static_assert(!kInt8 || (kFeat == Feat::kNone && !kDrop), "INT8 is plain");
  static_assert(!kOwnP || D == 64, "at head_dim 128 S and O fill the columns");
  constexpr int kPCol = kOwnP ? kBN + D : 0;
  using C = DCfg<D>;
  constexpr int S = C::kStages;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* tiles = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  DShared* sh = reinterpret_cast<DShared*>(tiles + C::kSmemTiles);
  const uint32_t sQ = smem_u32(tiles), sKV = sQ + C::kTileBytes;
  float* const skt = reinterpret_cast<float*>(tiles + C::kSmemTiles + 1024);     // INT8: [slot][key]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  const int off = p.q_pos_offset;

  // Side by side: barriers, tensor memory, tensor maps, and the producer's first item (the producer joins the others behind it).
  if (warp == 5) {
    tmem_alloc(smem_u32(&sh->tmem_base), 256);
    tmem_relinquish();
  } else if (warp == 6) {
    if (lane == 0) {
      mbar_init(smem_u32(&sh->q_full), 1);
      mbar_init(smem_u32(&sh->q_empty), 1);
      mbar_init(smem_u32(&sh->s_full), 1);
      mbar_init(smem_u32(&sh->s_free), 128);
      mbar_init(smem_u32(&sh->o_ready), 1);
      mbar_init(smem_u32(&sh->p_half), 128);
      mbar_init(smem_u32(&sh->stg_ready), 128);
      mbar_init(smem_u32(&sh->stg_taken), 1);
      for (int i = 0; kInt8 && i < kSkSlots; ++i) {
        mbar_init(smem_u32(&sh->sk_full[i]), 1);
        mbar_init(smem_u32(&sh->sk_empty[i]), 128);
      }
      for (int i = 0; i < kSched; ++i) {
        mbar_init(smem_u32(&sh->sched_full[i]), 1);
        mbar_init(smem_u32(&sh->sched_empty[i]), kConsumers + (kInt8 ? 1 : 0));
      }
      mbar_init(smem_u32(&sh->p_ready), 128);
      for (int i = 0; i < S; ++i) {
        mbar_init(smem_u32(&sh->kv_full[i]), 1);
        mbar_init(smem_u32(&sh->kv_empty[i]), 1);
      }
      sh->abort_flag = 0;
      fence_barrier_init();
    }
  } else if (warp == 7 && lane == 0) {
    prefetch_tmap(&tmQ);
    prefetch_tmap(&tmK);
    prefetch_tmap(&tmV);
    prefetch_tmap(&tmO);
  }
  if (warp != 4) {
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
  }
  const uint32_t tmem = sh->tmem_base;             // (not for the producer)

  // Ring bookkeeping: an item with nt key tiles takes the ring positions K_0 V_0 K_1 V_1 ... (2 nt entries); every role advances
  // one position counter, position `pos` lives in slot pos % S and completes phase (pos / S) & 1 of that slot's barriers.
  // The last V entry of an item is released by the store agent (the output is staged over it), the others by the commits of
  // the issuer.  Barriers of tiles follow a running count of tiles, those of items one of the items with tiles.

  if (warp == 7) {
    reg_dealloc<kRegsService>();
    if constexpr (kInt8) {
      // Scales of the keys, times softmax_scale log2(e) (what the softmax warps need with them), a few tiles ahead.
      int sidx = 0, tc = 0;
      bool ok = true;
      for (;;) {
        const Item w = sched_get(sh, sidx++, ok);
        if (!ok || w.nt < 0) break;
        const float* const row = sk + ((int64_t)w.b * p.heads_q + w.h) * p.total_k;
        for (int j = 0; j < w.nt && ok; ++j, ++tc) {
          const int slot = tc % kSkSlots;
          float v[kBN / 32];
#pragma unroll
          for (int i = 0; i < kBN / 32; ++i) {
            const int col = (w.n_hi - 1 - j) * kBN + lane + 32 * i;
            v[i] = col < w.k_len ? row[col] : 1.f;
          }
          SKEW(warp, 8, tc, 0);
          ok = wait_bar(&sh->sk_empty[slot], ((tc / kSkSlots) & 1) ^ 1, sh, 12);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
#pragma unroll
          for (int i = 0; i < kBN / 32; ++i) skt[slot * kBN + lane + 32 * i] = v[i] * (cfg.scale * 1.44269504f);
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(&sh->sk_full[slot]));
        }
        if (!ok) break;
      }
    }
  } else if (warp == 4) {
    // ------------------------------- TMA producer and work queue ------------------------
    // The warp draws and decodes the next item before it waits for the slot of the current one's last V tile: publishing it
    // costs nobody time, and Q and K_0 follow as soon as the issuer has read the last K tile.
    // (One copy of each part: what a CTA executes first it waits for, and where other kernels have run in between 40 KB more of
    // code were 5 k cycles at the start of a launch.)
    int fidx = 0, pos = 0, qi = 0;
    int c = blockIdx.x;                                // the candidate looked at last, an item or not
    bool ok = true;
    auto wwait = [&](uint64_t* bar, uint32_t parity, int code) {
      if (ok) ok = wait_bar(bar, parity, sh, code);
    };
    // the item under way: entry i of its 2 nt ring entries comes next
    int nt = 0, n_hi = 0, k_row0 = 0, boff = 0, hk = 0, i = 0;
    while (ok) {
      if (i + 1 >= 2 * nt) {
        Item w;
        for (bool drawn = fidx > 0;; drawn = true) {
          if (drawn) c = queue_next(queue, ncand, c, lane);
          if ((unsigned int)c >= (unsigned int)ncand) {
            w.nt = -1;
            break;
          }
          if (item_of(p, cfg, by_weight, c, lane, w)) break;
        }
        if (fidx == 0) {
          __syncthreads();                             // barriers are set up
          reg_dealloc<kRegsService>();
        }
        wwait(&sh->sched_empty[fidx % kSched], ((fidx / kSched) & 1) ^ 1, 60);
        if (ok && lane == 0) {
          const int4* src = reinterpret_cast<const int4*>(&w);
#pragma unroll
          for (int k = 0; k < 3; ++k) sh->sched_item[fidx % kSched][k] = src[k];
          mbar_arrive(smem_u32(&sh->sched_full[fidx % kSched]));
        }
        __syncwarp();
        ++fidx;
      }
      if (i < 2 * nt) {                                // K_0 V_0 K_1 V_1 ...
        const int slot = pos % S;
        SKEW(warp, 8, pos, 0);
        wwait(&sh->kv_empty[slot], ((pos / S) & 1) ^ 1, 11);
        if (ok && lane == 0) {
          const uint32_t bar = smem_u32(&sh->kv_full[slot]);
          mbar_expect_tx(bar, C::kTileBytes);
          for (int bx = 0; bx < C::kBoxes; ++bx)
            tma_load_4d(sKV + slot * C::kTileBytes + bx * (kBN * 128), (i & 1) ? &tmV : &tmK, bar, bx * 64, hk,
                        k_row0 + (n_hi - 1 - (i >> 1)) * kBN, boff);
        }
        ++pos;
        ++i;
      }
      if (i >= 2 * nt) {
        // on to the item published last (read back from the ring: its entry is written again four items later)
        const Item& entry = *reinterpret_cast<const Item*>(&sh->sched_item[(fidx - 1) % kSched][0]);
        nt = entry.nt;
        n_hi = entry.n_hi;
        k_row0 = entry.k_row0;
        boff = entry.boff;
        hk = entry.hk;
        i = 0;
        if (nt < 0) break;
        if (nt > 0) {
          wwait(&sh->q_empty, (qi & 1) ^ 1, 12);
          if (ok && lane == 0) {
            const int row = entry.q_row0 + entry.m0, h = entry.h;
            const uint32_t bar = smem_u32(&sh->q_full);
            mbar_expect_tx(bar, C::kTileBytes);
            for (int bx = 0; bx < C::kBoxes; ++bx) tma_load_4d(sQ + bx * (kBM * 128), &tmQ, bar, bx * 64, h, row, boff);
          }
          ++qi;
        }
      }
    }
  } else if (warp == 5) {
    // ------------------------------- MMA issuer -----------------------------------------
    // The whole warp runs the control flow in lock step and every lane polls the barriers;
    // the lane chosen once by elect_one issues the MMAs and commits.
    reg_dealloc<kRegsService>();
    constexpr uint32_t idesc_qk = make_idesc(1, DFmt<T>::code, 0, 0, kBM, kBN);
    constexpr uint32_t idesc_pv = make_idesc(1, DFmt<T>::code, 0, 1, kBM, D);
    const uint32_t leader = elect_one() ? 1u : 0u;
    int pos = 0, qi = 0, sidx = 0, tc = 0;             // tc: tiles so far
    bool ok = true;
    auto wwait = [&](uint64_t* bar, uint32_t parity, int code) {
      if (ok) ok = wait_bar(bar, parity, sh, code);
      tc_fence_after();
    };
    auto issue_qk = [&](int ps, bool last) {           // S = Q K^T with the K tile at ring position ps
      wwait(&sh->kv_full[ps % S], (ps / S) & 1, 22);
      if (!ok) return;
      const uint64_t dq = make_smem_desc(sQ, 16, 1024), dk = make_smem_desc(sKV + (ps % S) * C::kTileBytes, 16, 1024);
#pragma unroll
      for (int kk = 0; kk < D / 16; ++kk) {
        const uint32_t o = ((kk / 4) * (kBM * 128) + (kk % 4) * 32) >> 4;
        mma_f16_ss_lp(tmem, dq + o, dk + o, idesc_qk, kk > 0, leader);
      }
      mma_commit_lp(smem_u32(&sh->s_full), leader);
      mma_commit_lp(smem_u32(&sh->kv_empty[ps % S]), leader);
      if (last) mma_commit_lp(smem_u32(&sh->q_empty), leader);
    };
    auto issue_pv = [&](int ps, int t, bool first, bool last) {   // O += P V with the V tile at ring position ps
      wwait(&sh->kv_full[ps % S], (ps / S) & 1, 24);
      const uint64_t dv = make_smem_desc(sKV + (ps % S) * C::kTileBytes, kBN * 128, 1024);
      if (kPvSplit) {
        wwait(&sh->p_half, t & 1, 25);
        if (!ok) return;
#pragma unroll
        for (int kk = 0; kk < kBN / 32; ++kk)
          mma_f16_ts_lp(tmem + kBN, tmem + kPCol + kk * 8, dv + ((kk * 2048) >> 4), idesc_pv, (!first || kk > 0) ? 1u : 0u, leader);
      }
      wwait(&sh->p_ready, t & 1, 25);
      if (!ok) return;
#pragma unroll
      for (int kk = kPvSplit ? kBN / 32 : 0; kk < kBN / 16; ++kk)
        mma_f16_ts_lp(tmem + kBN, tmem + kPCol + kk * 8, dv + ((kk * 2048) >> 4), idesc_pv, (!first || kk > 0) ? 1u : 0u, leader);
      mma_commit_lp(smem_u32(&sh->o_ready), leader);
      if (!last) mma_commit_lp(smem_u32(&sh->kv_empty[ps % S]), leader);
    };
    for (;;) {
      const int nt = sched_get(sh, sidx++, ok).nt;
      if (!ok || nt < 0) break;
      if (nt == 0) continue;
      wwait(&sh->q_full, qi & 1, 21);
      ++qi;
      // (the scores of the item's first tile overwrite those, or P, of the last item's last: read before the
      // epilogue that is now in the softmax warps, and by the P V ahead in the in-order pipe)
      for (int j = 0; j <= nt && ok; ++j) {
        SKEW(warp, 8, tc + j, 0);
        // P in columns of its own: S(j) goes before P V_{j-1}, while the softmax warps have S(j - 1) in registers
        if (kOwnP && j > 0) wwait(&sh->s_free, (tc + j - 1) & 1, 26);
        if (!kOwnP && j > 0) issue_pv(pos + 2 * j - 1, tc + j - 1, j == 1, j == nt);
        if (ok && j < nt) issue_qk(pos + 2 * j, j + 1 == nt);
        if (kOwnP && j > 0 && ok) issue_pv(pos + 2 * j - 1, tc + j - 1, j == 1, j == nt);
      }
      pos += 2 * nt;
      tc += nt;
    }
    __syncwarp();
  } else if (warp == 6) {
    // ------------------------------- store agent ----------------------------------------
    // Hands the staged outputs to the TMA unit and releases their ring entries once the unit has read them.
    reg_dealloc<kRegsService>();
    const uint32_t leader = elect_one() ? 1u : 0u;
    int pos = 0, sidx = 0, wi = 0;
    bool ok = true;
    for (;;) {
      const Item w = sched_get(sh, sidx++, ok);
      if (!ok || w.nt < 0) break;
      if (w.nt == 0) continue;
      pos += 2 * w.nt;
      const int slot = (pos - 1) % S;
      ok = wait_bar(&sh->stg_ready, wi & 1, sh, 62);
      if (!ok) break;
      ++wi;
      SKEW(warp, 8, wi, 2);
      if (leader) {
        mbar_arrive(smem_u32(&sh->stg_taken));
        if (p.cu_seqlens_q == nullptr || w.m0 + kBM <= w.q_len) {
#pragma unroll
          for (int bx = 0; bx < D / 64; ++bx)
            tma_store_4d(&tmO, sKV + slot * C::kTileBytes + bx * (kBM * 128), bx * 64, w.h, w.q_row0 + w.m0, w.boff);
          tma_store_commit();
          tma_store_wait_read();
        }
        mbar_arrive(smem_u32(&sh->kv_empty[slot]));
      }
      __syncwarp();
    }
    __syncwarp();
  } else {
    // ------------------------------- softmax --------------------------------------------
    reg_alloc<kRegsSoftmax>();
    const int row_in_tile = tid;                     // TMEM lane
    const uint32_t lane_addr = (uint32_t)(warp * 32) << 16;
    const uint32_t tSx = tmem + lane_addr, tOx = tSx + kBN;
    bool ok = true;
    int pos = 0, sidx = 0, wi = 0, tc = 0;             // tc: tiles before this item

    for (;;) {
      // (what only the epilogue needs is read there, and the entry released behind it: the registers are short)
      const Item& entry = *reinterpret_cast<const Item*>(&sh->sched_item[sidx % kSched][0]);
      if (!wait_bar(&sh->sched_full[sidx % kSched], (sidx / kSched) & 1, sh, 61)) break;
      const int nt = entry.nt, n_hi = entry.n_hi, k_len = entry.k_len, m0 = entry.m0;
      if (nt < 0) break;
      const int qpos = m0 + row_in_tile + off;
      const float slope = (kExtras && cfg.has_alibi) ? p.alibi_slopes[entry.b * p.heads_q + entry.h] : 0.f;
      const float sq_row = kInt8 && m0 + row_in_tile < entry.q_len
                               ? sq[((int64_t)entry.b * p.heads_q + entry.h) * p.total_k + m0 + row_in_tile] : 1.f;
      float m_used = -INFINITY, l = 0.f;
      const int tq_min = m0 + off, tq_max = tq_min + kBM - 1;

      for (int j = 0; j < nt && ok; ++j) {
        const int k0 = (n_hi - 1 - j) * kBN;
        bool masked = (k0 + kBN > k_len);
        if (cfg.causal) masked |= (k0 + kBN - 1 > tq_min);
        if (cfg.wl >= 0) masked |= (k0 < tq_max - cfg.wl);
        if (cfg.wr >= 0) masked |= (k0 + kBN - 1 > tq_min + cfg.wr);

        // The row's 128 bits of the tile, on their way during the wait.  At head_dim 128 only to L1: four registers less across the
        // maxima are worth more there (8 x 16 x 512 36.3 -> 32.4 us; at 64 25.6 -> 26.3).
        uint4 keep4;
        const uint4* const keep_at = reinterpret_cast<const uint4*>(cfg.keep + (m0 + row_in_tile) * cfg.keep_words + (k0 >> 5));
        if (kDrop && D == 64) keep4 = __ldg(keep_at);
        if (kDrop && D == 128) asm volatile("prefetch.global.L1 [%0];\n" ::"l"(keep_at));

        ok = wait_bar(&sh->s_full, (tc + j) & 1, sh, 31);
        if (!ok) break;
        SKEW(warp, 8, tc + j, 0);
        tc_fence_after();

        // ---- the 128 scores of this row into registers -------------------------------------
        uint32_t r[4][32];
#pragma unroll
        for (int cc = 0; cc < 4; ++cc) tmem_ld32(tSx + cc * 32, r[cc]);
        tmem_wait_ld();
        if (kOwnP) {                                   // (behind the last tile too: a branch here undoes the gain)
          tc_fence_before();
          mbar_arrive(smem_u32(&sh->s_free));
        }

        const bool prescaled = kExtras || masked || kInt8;
        // columns (keys) of this tile that this thread's query row sees (used by masked tiles only)
        ColMask cm;
        if (masked) {
          int vk_lo, vk_hi;
          visible_k_interval(cfg, qpos, k_len, vk_lo, vk_hi);
          cm = make_col_mask(vk_lo - k0, vk_hi - k0);
        }
        if constexpr (kInt8) {
          // score = acc * s_q * (s_k * softmax_scale * log2 e), s_q in the FMA that forms the exponent
          const int slot = (tc + j) % kSkSlots;
          ok = wait_bar(&sh->sk_full[slot], ((tc + j) / kSkSlots) & 1, sh, 37);
          if (!ok) break;
          const float4* S4 = reinterpret_cast<const float4*>(skt + slot * kBN);
          auto scale_tile = [&](auto mask_tag) {
            constexpr bool kMask = decltype(mask_tag)::value;
#pragma unroll
            for (int cc = 0; cc < 4; ++cc) {
#pragma unroll
              for (int i = 0; i < 32; i += 4) {
                const float4 s4 = S4[cc * 8 + i / 4];
                const float2 v01 = f2mul(make_float2(__uint_as_float(r[cc][i]), __uint_as_float(r[cc][i + 1])), make_float2(s4.x, s4.y));
                const float2 v23 = f2mul(make_float2(__uint_as_float(r[cc][i + 2]), __uint_as_float(r[cc][i + 3])), make_float2(s4.z, s4.w));
                float v[4] = {v01.x, v01.y, v23.x, v23.y};
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                  if (kMask) v[e] = col_visible(cm, cc * 32 + i + e) ? v[e] : -INFINITY;
                  r[cc][i + e] = __float_as_uint(v[e]);
                }
              }
            }
          };
          if (masked) scale_tile(std::true_type{});
          else scale_tile(std::false_type{});
          mbar_arrive(smem_u32(&sh->sk_empty[slot]));
        } else if (prescaled) {
          // score pipeline and mask applied once, in place; values end up in the log2 domain.
          // One body, compiled per masked tile: no branch inside the unrolled loops.
          const float dist0 = (float)(qpos - k0);
          auto score_tile = [&](auto mask_tag, auto abs_tag) {
            constexpr bool kMask = decltype(mask_tag)::value;
            constexpr bool kAbs = decltype(abs_tag)::value;
            if (kExtras) {
              // packed pairs; the distance of a pair's columns goes down by (2, 2)
              const FeatK fk = feat_k<kCap>(cfg, slope);
              const float2 step2 = make_float2(-2.f, -2.f);
              float2 d2 = make_float2(dist0, dist0 - 1.f);
#pragma unroll
              for (int cc = 0; cc < 4; ++cc) {
#pragma unroll
                for (int i = 0; i < 32; i += 2) {
                  float2 v = score_unit_feat2<kCap, kAbs>(
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
          const bool need_abs = kExtras && !cfg.causal;    // under the causal mask visible keys lie at distance >= 0
          auto run_score = [&](auto mask_tag) {
            if (need_abs) score_tile(mask_tag, std::true_type{});
            else score_tile(mask_tag, std::false_type{});
          };
          if (masked) run_score(std::true_type{});
          else run_score(std::false_type{});
        }

        // ---- packed batches: keep the next sequence's values out of P V ---------------------
        // The last key tile of a packed sequence also holds rows of the NEXT sequence.  Their probabilities are
        // exactly 0, but 0 * inf or 0 * NaN is NaN: zero those rows of the V tile before P is handed
        // to the issuer.  One thread per row; the swizzle does not matter.
        if (p.cu_seqlens_k != nullptr && k0 + kBN > k_len) {
          const int vpos = pos + 2 * j + 1;
          ok = wait_bar(&sh->kv_full[vpos % S], (vpos / S) & 1, sh, 39);
          if (!ok) break;
          if (k0 + row_in_tile >= k_len) {
            unsigned char* vrow = tiles + C::kTileBytes * (1 + vpos % S) + row_in_tile * 128;
#pragma unroll
            for (int bx = 0; bx < C::kBoxes; ++bx) {
#pragma unroll
              for (int c = 0; c < 8; ++c)
                reinterpret_cast<uint4*>(vrow + bx * (kBN * 128))[c] = make_uint4(0u, 0u, 0u, 0u);
            }
          }
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
        // what the stored values are multiplied by to give log2-domain scores: softmax_scale log2e
        // on the plain path, cap log2e for capped scores (stored as tanh), else 1; all >= 0
        const float mul = !prescaled ? cfg.scale_log2 : (kCap ? cfg.softcap * FA_LOG2E : 1.f);
        mx *= mul;
        if (kInt8) mx *= sq_row;                       // s_q > 0

        // ---- lazy rescale ----------------------------------------------------------------
        if (j == 0) {
          m_used = mx;
        } else {
          const bool need = mx > m_used + cfg.rescale_at;
          if (__any_sync(0xffffffffu, need)) {
            // The previous P V of this stream is its (j-1)-th; the one of this tile cannot
            // complete before P is written below, so the barrier is at most one phase ahead
            // of the parity waited for here.
            ok = wait_bar(&sh->o_ready, (tc + j - 1) & 1, sh, 33);
            if (!ok) break;
            tc_fence_after();
            const float alpha = need ? exp2f(m_used - mx) : 1.f;  // m_used = -inf -> 0
            if (need) {
              m_used = mx;
              l *= alpha;
            }
#pragma unroll
            for (int cc = 0; cc < D / 32; ++cc) {
              uint32_t ro[32];
              tmem_ld32(tOx + cc * 32, ro);
              tmem_wait_ld();
#pragma unroll
              for (int i = 0; i < 32; ++i) ro[i] = __float_as_uint(__uint_as_float(ro[i]) * alpha);
              tmem_st32(tOx + cc * 32, ro);
            }
            tmem_wait_st();
          }
        }
        const float m_safe = (m_used == -INFINITY) ? 0.f : m_used;
        SKEW(warp, 8, tc + j, 1);

        // ---- P = exp2(s - m), row sum, P -> TMEM, over S or in columns of its own -------------
        // packed pairs: one FMA, two exponentials, one conversion and one add per two scores
        if (kOwnP && j > 0) {                          // the P V before has read its P (as good as always)
          ok = wait_bar(&sh->o_ready, (tc + j - 1) & 1, sh, 33);
          if (!ok) break;
          tc_fence_after();
        }
        if (kDrop && D == 128) keep4 = __ldg(keep_at);
        const float mul_x = kInt8 ? sq_row : mul;
        const float2 mul2 = make_float2(mul_x, mul_x), nm2 = make_float2(-m_safe, -m_safe);
        float2 acc2[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
        auto half_done = [&]() {
          // the first 64 keys of P are complete: the issuer starts P V on them while the
          // second half of the exponentials runs
          tmem_wait_st();
          tc_fence_before();
          mbar_arrive(smem_u32(&sh->p_half));
        };
#pragma unroll
        for (int cc = 0; cc < 4; ++cc) {
          uint32_t pk[16];
#pragma unroll
          for (int i = 0; i < 32; i += 2) {
            const float2 a = f2fma(make_float2(__uint_as_float(r[cc][i]), __uint_as_float(r[cc][i + 1])), mul2, nm2);
            float2 pe = make_float2(ex2(a.x), ex2(a.y));
            if constexpr (kInt8) {
              // l sums the ROUNDED values that enter P V: with outlier keys a row's dominant probability is 2^x relative to a stale
              // maximum, and its rounding has to cancel in O / l
              pk[i >> 1] = Elem<T>::pack(pe.x, pe.y);
              acc2[(i >> 1) & 1] = f2add(acc2[(i >> 1) & 1], Elem<T>::unpack(pk[i >> 1]));
              continue;
            }
            acc2[(i >> 1) & 1] = f2add(acc2[(i >> 1) & 1], pe);
            if (kDrop) {
              const uint32_t kw = cc == 0 ? keep4.x : cc == 1 ? keep4.y : cc == 2 ? keep4.z : keep4.w;
              pe.x = (kw >> i) & 1u ? pe.x : 0.f;
              pe.y = (kw >> (i + 1)) & 1u ? pe.y : 0.f;
            }
            pk[i >> 1] = Elem<T>::pack(pe.x, pe.y);
          }
          tmem_st16(tSx + kPCol + cc * 16, pk);
          if (kPvSplit && cc == 1) half_done();
        }
        l += (acc2[0].x + acc2[0].y) + (acc2[1].x + acc2[1].y);
        tmem_wait_st();
        tc_fence_before();
        mbar_arrive(smem_u32(&sh->p_ready));
      }

      // ---- epilogue: O / l -> global, base-2 LSE ------------------------------------------
      // The tile is staged over the item's last V tile, which no MMA reads any more, in the swizzled box layout, for the store
      // agent, which lets the TMA unit write full rows; a packed tile that reaches past the end of its sequence is stored
      // row by row instead (the unit would write the neighbour's rows).
      tc += nt;
      pos += 2 * nt;
      SKEW(warp, 8, wi, 2);
      if (ok && nt > 0) ok = wait_bar(&sh->o_ready, (tc - 1) & 1, sh, 35);
      if (!ok) break;
      tc_fence_after();
      const float inv = l > 0.f ? (kDrop ? cfg.dropout_scale : 1.f) / l : 0.f;
      const Item w = entry;
      const int row = m0 + row_in_tile;                // query row inside the sequence
      const bool row_ok = row < w.q_len;
      const bool via_tma = nt > 0 && (p.cu_seqlens_q == nullptr || w.m0 + kBM <= w.q_len);
      const uint32_t stg = sKV + ((pos - 1) & (S - 1)) * C::kTileBytes;
      T* og = reinterpret_cast<T*>(p.o) + (int64_t)w.boff * p.o_stride[0] + (int64_t)(w.q_row0 + row) * p.o_stride[1] +
              (int64_t)w.h * p.o_stride[2];
#pragma unroll 1                                       // (a CTA's first epilogue waits for its instructions)
      for (int cc = 0; cc < D / 32; ++cc) {
        uint32_t ra[32];
        if (nt > 0) {
          tmem_ld32(tOx + cc * 32, ra);
          tmem_wait_ld();
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) ra[i] = 0u;
        }
#pragma unroll
        for (int i = 0; i < 32; i += 8) {
          uint4 v;
          v.x = Elem<T>::pack(__uint_as_float(ra[i]) * inv, __uint_as_float(ra[i + 1]) * inv);
          v.y = Elem<T>::pack(__uint_as_float(ra[i + 2]) * inv, __uint_as_float(ra[i + 3]) * inv);
          v.z = Elem<T>::pack(__uint_as_float(ra[i + 4]) * inv, __uint_as_float(ra[i + 5]) * inv);
          v.w = Elem<T>::pack(__uint_as_float(ra[i + 6]) * inv, __uint_as_float(ra[i + 7]) * inv);
          if (via_tma) {
            const int col = cc * 32 + i;                   // first of 8 columns = one 16-byte chunk
            st_shared_v4(sw128_addr(stg + (col / 64) * (kBM * 128), row_in_tile, (col % 64) / 8), v);
          } else if (row_ok) {
            *reinterpret_cast<uint4*>(og + cc * 32 + i) = v;
          }
        }
      }
      if (nt > 0) {
        tc_fence_before();
        if (via_tma) fence_proxy_async();
        // (the agent has seen the previous item's tile: its barrier is never a whole phase behind)
        SKEW(warp, 8, wi, 3);
        if (wi > 0 && !(ok = wait_bar(&sh->stg_taken, (wi - 1) & 1, sh, 63))) break;
        mbar_arrive(smem_u32(&sh->stg_ready));
        ++wi;
      }
      if (row_ok && p.lse2 != nullptr)
        p.lse2[(int64_t)w.boff * p.lse_stride[0] + (int64_t)(w.q_row0 + row) * p.lse_stride[1] + (int64_t)w.h * p.lse_stride[2]] =
            l > 0.f ? m_used + log2f(l) : -INFINITY;
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&sh->sched_empty[sidx % kSched]));
      ++sidx;
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 5) tmem_dealloc(tmem, 256);
  if (tid == 0) {
    if (queue != nullptr) queue_finish(queue, ncand);
    report_abort(sh->abort_flag, host_status);
  }
}

// ---------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------
// head_dim 64: P in columns of its own, or over S as at head_dim 128?  Rows of one key tile have no next scores to compute
// early, and rows of two gain what rows of one lose.  Own columns against P over S, 16 heads, two orders of launches:
//   dense      one tile +2 % (64 x 128: 20.8 -> 21.3 us), causal two tiles 0 to +1 % (64 x 200: 55.5 -> 56.0), causal three 0, no
//              mask two -2 % (64 x 256: 54.0 -> 52.9), more -1 to -3 %
//   packed, causal    17 to 256 tokens +1.3 %, 100 to 200 +1.9 %, 17 to 400 +0.3 %, 17 to 640 -0.6 %, 550 to 1100 -2 %
//   packed, no mask   100 to 200 +1.1 %, 128 to 256 -0.3 %, 250 to 500 -1.4 %
//   windows    below two key tiles +0.3 to +2 % (16 x 1024, 50 on either side: 81.1 -> 82.6), 300 -1.7 %, 150 on either side 0
// Of a packed batch only the sum and the longest length are known here.
static bool p_over_s_is_faster(const fa_attn_args& a, const ScoreCfg& cfg) {
  const bool packed = a.cu_seqlens_q != nullptr;
  const int64_t keys = packed ? (a.total_k / a.batch + a.seqlen_k) / 2 : a.seqlen_k, nk = (keys + kBN - 1) / kBN;
  if ((cfg.causal ? nk + 1 : 2 * nk) <= (packed ? 4 : 3)) return true;    // twice the key tiles of a row tile
  const int right = cfg.causal ? 0 : cfg.wr;
  return cfg.wl >= 0 && right >= 0 && (int64_t)cfg.wl + right < 2 * kBN;
}

template <typename K>
static int launch_items(K kern, int smem, const CUtensorMap (&tm)[4], const fa_attn_args& a, const ScoreCfg& plain, cudaStream_t st,
                        const float* sq = nullptr, const float* sk = nullptr) {
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) {
    set_error("fwd_duo_sm100: cudaFuncSetAttribute(%d): %s", smem, cudaGetErrorString(e));
    return FA_ERR_LAUNCH;
  }
  ScoreCfg cfg = plain;
  int by_weight;
  const int64_t ncand = item_candidates<kBM>(a, cfg, by_weight);
  if (ncand > 0x7fffffff - 4096) {
    set_error("fwd_duo_sm100: too many work items");
    return FA_ERR_UNSUPPORTED;
  }
  const int ctas = 2 * sm_count(a.device);
  // Up to two items per CTA, no mask that makes their sizes differ: no queue, CTA i takes items i and grid + i, so that second items go to CTAs on SMs of their own.
  // Drawn from the queue, both CTAs of an SM may get one while another SM gets none (us, queue -> so: 8 x 16 x 512 of 64 with dropout 25.6 -> 24.7,
  // 7 x 16 x 640 of 128 33.1 -> 31.9, 6 packed of 252, 32 heads over 8 of 128 23.0 -> 21.5); with items of different sizes under a mask the queue
  // is as good or better (7 x 16 x 640 of 128, causal 27.4 for 30.4).  Packed sequences without a mask, on average over 300 random calls: lengths within
  // 40 % of one another, 2.5 to 3 CTAs per SM, queue 5 % slower; otherwise 0 +- 2 %.
  const int right = cfg.causal ? 0 : cfg.wr;
  const bool even = (!cfg.causal && cfg.wl < 0 && cfg.wr < 0) || (cfg.wl >= 0 && right >= 0 && (int64_t)cfg.wl + right < 2 * kBN);
  unsigned int* queue = nullptr;
  const int grid = even && ncand <= 2 * (int64_t)ctas ? std::min((int)ncand, ctas) : queue_grid(a.device, st, (int)ncand, ctas, &queue);
  kern<<<grid, kThreads, smem, st>>>(tm[0], tm[1], tm[2], tm[3], a, cfg, (int)ncand, by_weight, queue, host_wait_word(a.device), sq, sk);
  return check_launch("fwd_duo_sm100");
}

template <typename T, int D>
static int launch_duo(const fa_attn_args& a, const ScoreCfg& plain, cudaStream_t st) {
  using C = DCfg<D>;
  const bool packed = a.cu_seqlens_q != nullptr;
  const int64_t q_rows = packed ? a.total_q : a.seqlen_q, k_rows = packed ? a.total_k : a.seqlen_k;
  auto map = [&](CUtensorMap* m, const void* base, const int64_t* stride, int heads, int64_t rows) {
    // dims (innermost first): head_dim, heads, rows, batch
    const uint64_t dims[4] = {(uint64_t)D, (uint64_t)heads, (uint64_t)rows, (uint64_t)(packed ? 1 : a.batch)};
    const uint64_t strides[3] = {(uint64_t)stride[2] * 2, (uint64_t)stride[1] * 2,
                                 (uint64_t)(packed ? rows * stride[1] : stride[0]) * 2};
    const uint32_t box[4] = {64, 1, 128, 1};
    return encode_tmap(m, base, 2, 4, dims, strides, box);
  };
  CUtensorMap tm[4];
  if (!map(&tm[0], a.q, a.q_stride, a.heads_q, q_rows) || !map(&tm[1], a.k, a.k_stride, a.heads_kv, k_rows) ||
      !map(&tm[2], a.v, a.v_stride, a.heads_kv, k_rows) || !map(&tm[3], a.o, a.o_stride, a.heads_q, q_rows)) {
    set_error("fwd_duo_sm100: cuTensorMapEncodeTiled failed");
    return FA_ERR_LAUNCH;
  }
  auto pick = [&](auto own) {
    constexpr bool kOwn = decltype(own)::value;
    return plain.keep != nullptr  ? fwd_duo_sm100_kernel<T, D, Feat::kNone, true, kOwn>
           : plain.softcap > 0.f ? fwd_duo_sm100_kernel<T, D, Feat::kCap, false, kOwn>
           : plain.has_alibi     ? fwd_duo_sm100_kernel<T, D, Feat::kAlibi, false, kOwn>
                                 : fwd_duo_sm100_kernel<T, D, Feat::kNone, false, kOwn>;
  };
  auto kern = pick(std::false_type{});
  if constexpr (D == 64) {
    if (!p_over_s_is_faster(a, plain)) kern = pick(std::true_type{});
  }
  return launch_items(kern, C::kSmemBytes, tm, a, plain, st);
}

int fwd_duo_sm100(const fa_attn_args& a, const ScoreCfg& cfg, cudaStream_t st) {
  const bool bf = a.dtype == FA_BF16;
  if (a.head_dim == 64) return bf ? launch_duo<__nv_bfloat16, 64>(a, cfg, st) : launch_duo<__half, 64>(a, cfg, st);
  return bf ? launch_duo<__nv_bfloat16, 128>(a, cfg, st) : launch_duo<__half, 128>(a, cfg, st);
}

// INT8 forward of head_dim 64 on the maps of its caller (fwd_sm100.cu).
int fwd_duo_int8(const CUtensorMap (&tm)[4], const fa_attn_args& a, const ScoreCfg& cfg, const float* sq, const float* sk, cudaStream_t st) {
  return launch_items(fwd_duo_sm100_kernel<__half, 64, Feat::kNone, false, true, true>, DCfg<64>::kSmemBytesInt8, tm, a, cfg, st, sq, sk);
}

int fwd_duo_sm100_status() {
  int v = 0;
  if (cudaMemcpyFromSymbol(&v, g_fwd_duo_status, sizeof(int)) != cudaSuccess) return -1;
  return v;
}
int fwd_duo_sm100_clear_status() {
  const int z = 0;
  return cudaMemcpyToSymbol(g_fwd_duo_status, &z, sizeof(int)) == cudaSuccess ? 0 : -1;
}

}  // namespace fa
