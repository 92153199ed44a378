// Backward attention on the 5th-generation tensor cores (tcgen05 + TMEM + TMA), as two
// PERSISTENT kernels with one writer per output element (no atomics, deterministic):
//
//   bwd_dkdv_sm100_kernel  work item = 128 keys of one (batch, kv head); loops over the query
//                          tiles (and the query heads of the GQA group) that can see them.
//                          Works on the TRANSPOSED tiles  S^T = K Q^T,  dP^T = V dO^T  so
//                          that a TMEM lane is a key: P^T and dS^T are written back to TMEM
//                          and feed  dV += P^T dO,  dK += dS^T Q  as the A operand.
//   bwd_dq_sm100_kernel    work item = 128 query rows of one (batch, head); loops over key
//                          tiles: S = Q K^T, dP = dO V^T, dS in place over dP, dQ += dS K.
//
// One CTA per SM takes work items from a queue: a counter in global memory hands out candidates
// in an order in which the CTAs that run together work on the same heads (the tiles they stream
// stay in L2) and in which the heavy items of a causal mask come first.  The producer thread
// draws from the counter, one item ahead, and publishes what it drew to the other roles through
// a small ring in shared memory.  Barriers, tensor memory and tensor maps are set up once per CTA.  Every role runs ahead into the next item on
// its own: the producer fetches the next item's tiles as ring slots free up, the MMA warps issue
// its first products while the element-wise warps still store the previous item's result.  The
// result tiles are staged over the LAST streamed tiles of the item, whose ring slots are released
// by the store instead of by the MMAs that read them: the next item's first tiles are already in
// the other slots by then.
//
// Both kernels are software-pipelined through the ORDER in which the MMA warps feed the (in-
// order) tensor pipe, so that the element-wise warps always work while independent MMAs run:
//
//   dK/dV, per query tile i:   dV += P(i)^T dO(i) | S(i + buffers)   then   dK += dS(i)^T Q(i) | dP(i+1)
//       P and dS (16-bit) overwrite the fp32 regions of S and dP; S has a second buffer at head_dim 64.
//   dQ, per key tile k:        S(k+1) -> other S buffer | dQ += dS(k) K(k) | dP(k+1)
//
// Roles (384 threads; 640 with score options: see Roles):
//   element-wise     two groups of four warps, with score options four groups: 64 (32) columns of the
//                    128 x 128 tiles each, one TMEM lane (row) per thread
//   producer         TMA loads
//   issuer           MMAs (uniform control flow, one elected lane issues)
//   statistics       dK/dV kernel: loads the per-row statistics (base-2 LSE, delta) of the
//                    streamed query tile and writes them as a 16-column GEMM operand
//   store            dK/dV kernel: hands the staged dV and dK tiles to the TMA unit
//
// TMEM, dK/dV kernel: S^T, P^T (128 columns) | dP^T, dS^T (128) | dV (128) | dK (128); at head_dim 64
//                     S^T, P^T [0] | S^T, P^T [1] | dP^T, dS^T | dV (64) | dK (64).
// What it measured, against the two kernels it replaced (one with S and dP in turns in one region, one with a CTA per
// key block): 32 packed sequences of 256 to 4096 tokens with window, ALiBi and soft cap 3610 -> 3045 us; 16 x 16 heads
// x 4096 tokens of 128, causal, unchanged within calls (3.3 k cycles per tile instead of 4.2 k; the power limit
// gives it back); 4 x 32 heads x 1024 x 1531 of 64 171 -> 139 us.
// TMEM, dQ kernel:    S[0] | S[1] | dP | dQ    (4 x 128 columns).
// All operand tiles are written by TMA with the 128-byte swizzle; the same tile is read
// K-major (contraction over head_dim) or MN-major (contraction over its rows) through
// different descriptors.  Every mbarrier wait is bounded.
#include <cstddef>
#include <type_traits>

#include <cstdlib>
#include "bwd_stats.cuh"
#include "common.cuh"
#include "queue.cuh"
#define PROF_TAG bwd
#include "prof.cuh"
#define SKEW_TAG bwd
#include "skew.cuh"
#include "sm100.cuh"

namespace fa {

using namespace sm100;

__device__ int g_bwd_sm100_status = 0;

namespace {

constexpr int kT = 128;        // tile edge: rows of Q / keys of K,V per tile
// Roles of the warps with G element-wise warpgroups, each of which takes 128 / G columns of a tile, and the split of the
// registers (setmaxnreg): the CTA starts with kRegsLaunch per thread; the four service warps drop to kRegsService and the
// element-wise warps grow to kRegsEw, out of what the CTA was launched with.
template <int G> struct Roles {
  static constexpr int kCols = kT / G;             // columns of a 128 x 128 tile per element-wise thread
  static constexpr int kEwThreads = 128 * G, kEwWarps = 4 * G;
  static constexpr int kProducer = kEwWarps, kIssuer = kEwWarps + 1, kStats = kEwWarps + 2, kStore = kEwWarps + 3;
  static constexpr int kThreads = kEwThreads + 128;
  static constexpr int kRegsLaunch = G == 2 ? 168 : 96;          // what a CTA of kThreads can have
  static constexpr int kRegsService = G == 2 ? 88 : 64, kRegsEw = G == 2 ? 208 : 104;
  static_assert(kThreads * kRegsLaunch <= 65536, "registers of an SM");
  static_assert((kRegsEw - kRegsLaunch) * kEwThreads <= (kRegsLaunch - kRegsService) * 128, "register split");
};
// Groups of a variant.  With score options a score takes two special-function results and a dozen other instructions, and
// two warps per scheduler leave most of their latencies open: with four the exponential phase of dK/dV takes 2.0 k cycles
// instead of 2.5 k (the special-function unit needs 2.05 k).  dK/dV and dQ, two groups -> four (us), causal: soft cap,
// 4 x 16 x 2048 of 64 156 -> 139, 118 -> 112; 2 x 16 x 4096 of 128 315 -> 302, 219 -> 207; ALiBi, 4 x 16 x 2048 of 128
// 150 -> 144, 105 -> 102.  Without options the phase is close to the unit's 1.02 k with two groups (1.35 k), and
// the larger number of warps delays the MMAs: 4 x 16 x 4096 of 128 864 -> 877, 605 -> 617; 4 x 32 x 1024 x 1531 of 64
// 137 -> 141, 101 -> 100.  (An arrival per warp instead of per thread: 0 to +1 %.  The LSE of the next tile read under this
// one's dS phase: +8 to +13 %, spills.  The LSE read next to its use: +4 to +8 %.)  dK/dV with soft cap spills 60 (head_dim 64) and 84 bytes a
// thread, the other variants up to 12.
__host__ __device__ constexpr int ew_groups(Feat f) { return f == Feat::kNone ? 2 : 4; }
constexpr int kSched = 4;      // depth of the in-CTA ring of work-queue entries
template <int D> struct BCfg {
  static constexpr int kTileBytes = kT * D * 2;
  static constexpr int kBoxes = D / 64;
  // dK/dV kernel: K and V resident, ring A of Q entries (Q(i) lives from S(i) to dK(i); dK is
  // staged over the last Q), ring B of dO entries (dO(i) lives from dP(i) to dV(i); dV is
  // staged over the last dO).
  static constexpr int kStagesQ = (D == 128) ? 2 : 4;
  static constexpr int kStagesO = (D == 128) ? 2 : 4;
  static constexpr int kSmemTiles = (2 + kStagesQ + kStagesO) * kTileBytes;
  // head_dim 64 leaves tensor-memory columns for a second score buffer.  The element-wise warps then find their scores
  // ready (they waited 0.4 k of 2.3 k cycles per tile for them, or, with P and dS in columns of their own instead, spent
  // as much on four more barriers): 4 x 32 heads x 1024 x 1531 153 -> 139 us, 2 x 16 over 4 heads x 1024, causal, 50 -> 46.
  // (Tried with those columns: one group half a tile behind the other, so that their exponentials do not meet, 4 % slower.)
  static constexpr int kSBuf = D == 64 ? 2 : 1;
  // dK/dV kernel: 128 x 16 operand tiles that carry the row statistics into the GEMMs
  // (two constant ones on the key side, one per ring stage on the query side)
  static constexpr int kAugTotal = (2 + kStagesQ) * kStatBlock;
  static constexpr int kSmemBytes = kSmemTiles + kAugTotal + 1024 + 4096;
  static_assert(kSmemBytes <= 227 * 1024, "shared memory budget");
  // dQ kernel: Q and dO resident, ring A of K tiles (dQ is staged over the last one), ring B of V tiles.  The K
  // ring is one stage deeper than the V ring: K(k+1) is needed by S(k+1) at the START of step k
  // while K(k) is still read by dQ(k) at its end.
  static constexpr int kStagesK = (D == 128) ? 3 : 4;
  static constexpr int kStagesV = (D == 128) ? 2 : 4;
  static constexpr int kSmemTilesDq = (2 + kStagesK + kStagesV) * kTileBytes;
  static constexpr int kSmemBytesDq = kSmemTilesDq + 1024 + 1024;
  static_assert(kSmemBytesDq <= 227 * 1024, "shared memory budget (dQ)");
};

struct BShared {
  uint64_t full_a[4];     // ring A entry landed (dK/dV: K, Q + statistics; dQ: K)
  uint64_t full_b[4];     // ring B entry landed (dK/dV: dO; dQ: V)
  uint64_t empty_a[4];    // ring A entry released
  uint64_t empty_b[4];    // ring B entry released
  uint64_t res_full;      // resident tiles of the item landed (dK/dV: V; dQ: Q and dO)
  uint64_t res_free;      // last MMA reading the resident tiles of the item finished
  uint64_t k_full, k_free;  // dK/dV kernel: the same for K
  uint64_t s_full[2];     // [buffer]: S computed
  uint64_t dp_full;       // dP computed
  uint64_t p_ready[2];    // dK/dV kernel, [score buffer]: P written back (every element-wise thread)
  uint64_t ds_ready;      // dS written back (every element-wise thread)
  uint64_t dv_done;       // dK/dV kernel: every dV MMA of the item finished
  uint64_t acc_done;      // every accumulation MMA of the item finished
  uint64_t sched_full[kSched];   // work-queue entry published by the producer thread
  uint64_t sched_empty[kSched];  // ... read by every consuming warp
  int4 sched_item[kSched][3];    // the item, decoded once by the producer thread (KItem / QItem)
  // (dK/dV: every warp has seen the previous item's tiles taken; dQ: see the end of its element-wise groups)
  uint64_t stg_ready[2];  // result tile of an item staged for the store lane (and its message written); dK/dV: dV, dK
  uint64_t stg_taken[2];  // [group] the store lane has read the message; dK/dV: [0], both tiles seen by the agent
  // [group] message to the store lane: shared-memory address of the staged tile (0 = nothing to
  // store, -1 = no more items), tensor-map coordinates head / row / batch, barrier to release
  volatile int stg_msg[2][5];
  uint32_t tmem_base;
  volatile int abort_flag;
  alignas(16) float lse[4][kT];  // [stage][row of the streamed query tile]: MINUS the base-2 LSE (feature variant)
};
static_assert(sizeof(BShared) <= 4096, "BShared must fit its reserve");
static_assert(offsetof(BShared, lse) <= 1024, "the dQ kernel reserves 1024 bytes for the barriers and the work queue");

template <typename T> struct BFmt;
template <> struct BFmt<__half> { static constexpr int code = 0; };
template <> struct BFmt<__nv_bfloat16> { static constexpr int code = 1; };

__device__ __forceinline__ bool bwait(uint64_t* bar, uint32_t parity, BShared* sh, int code) {
  return bounded_wait(bar, parity, &sh->abort_flag, &g_bwd_sm100_status, code);
}

// For roles that are far ahead of the critical path (producer, statistics loader): back off
// between polls so the spin does not take issue slots from the element-wise warps.
__device__ __forceinline__ bool bwait_relaxed(uint64_t* bar, uint32_t parity, BShared* sh, int code) {
  const uint32_t a = smem_u32(bar);
  for (int i = 0; i < 64; ++i) {
    if (mbar_try_wait(a, parity)) return true;
    __nanosleep(100);
  }
  return bwait(bar, parity, sh, code);
}

// Work queue (queue.cuh).
// The producer thread draws a candidate (just before the last loads of the current item, so that the
// round trip to the counter is over when they are issued), decodes it into an item (12 ints: KItem / QItem) and
// publishes the item to the other roles; entry number i of this CTA travels in ring slot
// i % kSched.  Candidates outside their sequence are skipped; an item with total < 0 ends the queue.
template <typename Item, typename F>
__device__ __forceinline__ Item sched_publish(BShared* sh, unsigned int* counter, int ncand, unsigned int u, int& fidx,
                                              bool& ok, F decode) {
  static_assert(sizeof(Item) == 48, "an item travels as three 16-byte words");
  Item w;
  for (;; u = queue_draw(counter, ncand)) {
    if (u >= (unsigned int)ncand) {
      w.total = -1;
      break;
    }
    if (decode((int)u, w)) break;
  }
  const int slot = fidx % kSched;
  if (!bwait_relaxed(&sh->sched_empty[slot], ((fidx / kSched) & 1) ^ 1, sh, 60)) {
    ok = false;
    w.total = -1;
    return w;
  }
  const int4* src = reinterpret_cast<const int4*>(&w);
  sh->sched_item[slot][0] = src[0];
  sh->sched_item[slot][1] = src[1];
  sh->sched_item[slot][2] = src[2];
  mbar_arrive(smem_u32(&sh->sched_full[slot]));
  ++fidx;
  return w;
}
// Entry number idx as seen by a consuming warp (all lanes call this together).  `consume` releases
// the entry; without it the call only looks at an entry that will be consumed later.
template <typename Item>
__device__ __forceinline__ Item sched_get(BShared* sh, int idx, bool consume, bool& ok) {
  Item w;
  const int slot = idx % kSched;
  if (!bwait(&sh->sched_full[slot], (idx / kSched) & 1, sh, 61)) {
    ok = false;
    w.total = -1;
    return w;
  }
  int4* dst = reinterpret_cast<int4*>(&w);
  dst[0] = sh->sched_item[slot][0];
  dst[1] = sh->sched_item[slot][1];
  dst[2] = sh->sched_item[slot][2];
  if (consume) {
    __syncwarp();
    if ((threadIdx.x & 31) == 0) mbar_arrive(smem_u32(&sh->sched_empty[slot]));
  }
  return w;
}
// Releases an entry that this warp has already looked at.
__device__ __forceinline__ void sched_release(BShared* sh, int idx) {
  __syncwarp();
  if ((threadIdx.x & 31) == 0) mbar_arrive(smem_u32(&sh->sched_empty[idx % kSched]));
}

// For an agent that waits for a whole item (tens of microseconds; items differ in length by orders of magnitude):
// sleeps between polls instead of spinning next to the other roles.
__device__ __forceinline__ bool bwait_long(uint64_t* bar, uint32_t parity, BShared* sh, int code) {
  const uint32_t a = smem_u32(bar);
  const long long t0 = clock64();
  while (!mbar_try_wait(a, parity)) {
    __nanosleep(200);
    if (sh->abort_flag || *reinterpret_cast<volatile int*>(&g_bwd_sm100_status) != 0) return false;
    if (clock64() - t0 > 4 * FA_WAIT_CLOCKS) {
      sh->abort_flag = code;
      atomicCAS(&g_bwd_sm100_status, 0, code);
      return false;
    }
  }
  return true;
}

// Store lane: one thread that writes the result tiles the element-wise warps stage, so that none of
// them has to wait for the TMA unit.  Per item it waits for the tile (and the message that
// describes it), issues the store, waits until the unit has read the tile and releases the ring
// entry the tile was staged over (two stand-in arrivals, or one in the dQ kernel).
template <int D>
__device__ __forceinline__ void store_lane(BShared* sh, int x, const CUtensorMap* tm, uint32_t release_count) {
  for (uint32_t n = 0;; ++n) {
    if (!bwait_long(&sh->stg_ready[x], n & 1, sh, 62)) return;
    const int addr = sh->stg_msg[x][0], head = sh->stg_msg[x][1], row = sh->stg_msg[x][2],
              batch = sh->stg_msg[x][3], rel = sh->stg_msg[x][4];
    mbar_arrive(smem_u32(&sh->stg_taken[x]));
    if (addr == -1) return;
    if (addr > 0) {
#pragma unroll
      for (int bx = 0; bx < D / 64; ++bx) tma_store_4d(tm, (uint32_t)addr + bx * (kT * 128), bx * 64, head, row, batch);
      tma_store_commit();
      tma_store_wait_read();
    }
    mbar_arrive_cnt((uint32_t)rel, release_count);
  }
}
// Element-wise side: thread `poster` of the group writes the message for item number n (after the
// store lane has taken the previous one); every thread of the group then arrives on stg_ready
// once its part of the tile is staged.
__device__ __forceinline__ bool post_store(BShared* sh, int x, int n, int addr, int head, int row, int batch,
                                           uint32_t release_bar) {
  if (n > 0 && !bwait(&sh->stg_taken[x], (n - 1) & 1, sh, 63)) return false;
  sh->stg_msg[x][0] = addr;
  sh->stg_msg[x][1] = head;
  sh->stg_msg[x][2] = row;
  sh->stg_msg[x][3] = batch;
  sh->stg_msg[x][4] = (int)release_bar;
  return true;
}

// TMA loads of one 128 x D tile (D/64 boxes) at (row, head, batch)
template <int D>
__device__ __forceinline__ void load_tile(uint32_t dst, const CUtensorMap* tm, uint32_t bar, int row,
                                          int head, int batch) {
#pragma unroll
  for (int x = 0; x < D / 64; ++x) tma_load_4d(dst + x * (kT * 128), tm, bar, x * 64, head, row, batch);
}

// 128 x 128 x D product of two K-major tiles (contraction over head_dim): D/16 MMAs.
// Whole warp, uniform control flow; the lane with leader != 0 issues.
template <int D>
__device__ __forceinline__ void mma_kmajor(uint32_t d_tmem, uint32_t a_smem, uint32_t b_smem,
                                           uint32_t idesc, uint32_t leader) {
  const uint64_t da = make_smem_desc(a_smem, 16, 1024), db = make_smem_desc(b_smem, 16, 1024);
#pragma unroll
  for (int kk = 0; kk < D / 16; ++kk) {
    const uint32_t o = ((kk / 4) * (kT * 128) + (kk % 4) * 32) >> 4;
    mma_f16_ss_lp(d_tmem, da + o, db + o, idesc, kk > 0, leader);
  }
}

// acc(128 x D) += A(128 x 128, fp16 pairs in TMEM) * B(128 rows x D, MN-major smem tile).
// A is stored by the element-wise groups, each over the first half of its kCols columns.
template <int D, int kCols>
__device__ __forceinline__ void mma_from_tmem(uint32_t d_tmem, uint32_t a_tmem, uint32_t b_smem,
                                              uint32_t idesc, bool accumulate, uint32_t leader) {
  const uint64_t db = make_smem_desc(b_smem, kT * 128, 1024);
#pragma unroll
  for (int kk = 0; kk < kT / 16; ++kk) {
    constexpr int kPer = kCols / 16;               // MMAs per group
    const uint32_t a = a_tmem + (kk / kPer) * kCols + (kk % kPer) * 8;
    mma_f16_ts_lp(d_tmem, a, db + ((kk * 2048) >> 4), idesc, (accumulate || kk > 0) ? 1u : 0u, leader);
  }
}

// TMEM accumulator (128 lanes x kCols fp32 columns starting at tsrc, this thread's lane) scaled
// by `mul`, converted to T and either staged in the swizzled box layout at `stg` (column
// `col0 + c` of the tile) or, when `direct` is set, stored to the row pointer `grow` (null = skip).
template <typename T, int kCols>
__device__ __forceinline__ void drain_acc(uint32_t tsrc, float mul, bool staged, uint32_t stg, int lrow,
                                          int col0, T* grow) {
  constexpr int kW = kCols < 32 ? kCols : 32;
  uint32_t r[kCols / kW][kW];
#pragma unroll
  for (int cc = 0; cc < kCols / kW; ++cc) {
    if constexpr (kW == 16) tmem_ld16(tsrc + cc * kW, r[cc]);
    else tmem_ld32(tsrc + cc * kW, r[cc]);
  }
  tmem_wait_ld();
#pragma unroll
  for (int cc = 0; cc < kCols / kW; ++cc) {
#pragma unroll
    for (int i = 0; i < kW; i += 8) {
      uint4 v;
      v.x = Elem<T>::pack(__uint_as_float(r[cc][i]) * mul, __uint_as_float(r[cc][i + 1]) * mul);
      v.y = Elem<T>::pack(__uint_as_float(r[cc][i + 2]) * mul, __uint_as_float(r[cc][i + 3]) * mul);
      v.z = Elem<T>::pack(__uint_as_float(r[cc][i + 4]) * mul, __uint_as_float(r[cc][i + 5]) * mul);
      v.w = Elem<T>::pack(__uint_as_float(r[cc][i + 6]) * mul, __uint_as_float(r[cc][i + 7]) * mul);
      const int col = col0 + cc * kW + i;
      if (staged) st_shared_v4(sw128_addr(stg + (col / 64) * (kT * 128), lrow, (col % 64) / 8), v);
      else if (grow != nullptr) *reinterpret_cast<uint4*>(grow + cc * kW + i) = v;
    }
  }
}

// ---------------------------------------------------------------------------------------
// work items
// ---------------------------------------------------------------------------------------
struct Geo {          // one sequence's geometry, as ints (tensor-map coordinates are 32-bit)
  int q_len, k_len, q_row0, k_row0, q_boff, k_boff;
};
__device__ __forceinline__ Geo geo_of(const fa_attn_args& p, int b) {
  const SeqInfo si = seq_info(p, b);
  Geo g;
  g.q_len = si.q_len; g.k_len = si.k_len;
  g.q_row0 = (int)si.q_row0; g.k_row0 = (int)si.k_row0;
  g.q_boff = (int)si.q_boff; g.k_boff = (int)si.k_boff;
  return g;
}

// dK/dV: candidates in the order of block_of(), units = (batch entry, kv head); key block 0 sees the most
// query tiles under a causal mask.  Returns false when the key block lies outside its sequence.
struct KItem {
  Geo g;
  int n0, hk, b;
  int m_lo, ntiles, total;   // query tiles [m_lo, m_lo + ntiles) per query head; total = ntiles * group
};
__device__ __forceinline__ bool dkdv_item(const fa_attn_args& p, const ScoreCfg& cfg, int cand, int nkb, KItem& w) {
  int nblk, rem;
  block_of(cand, nkb, p.batch * p.heads_kv, cfg.unit_group, rem, nblk);
  w.hk = rem % p.heads_kv;
  w.b = rem / p.heads_kv;
  w.n0 = nblk * kT;
  w.g = geo_of(p, w.b);
  w.m_lo = w.ntiles = w.total = 0;
  if (w.n0 >= w.g.k_len) return false;
  const int off = p.q_pos_offset;
  int qlo, qhi;
  visible_query_range(cfg, w.n0, min(w.n0 + kT, w.g.k_len) - 1, off, w.g.q_len + off, qlo, qhi);
  w.m_lo = max(qlo - off, 0) / kT;
  const int m_hi = (max(qhi - off, 0) + kT - 1) / kT;
  w.ntiles = max(m_hi - w.m_lo, 0);
  w.total = w.ntiles * (p.heads_q / p.heads_kv);
  return true;
}

// dQ: the same with units = (batch entry, head); with a causal mask block i counts
// down from the last (heaviest) query block.  Returns false when the block lies outside its sequence.
struct QItem {
  Geo g;
  int m0, h, b;
  int n_hi, total;           // step j works on key tile n_hi - 1 - j (masked tiles first)
  int pad;
};
__device__ __forceinline__ bool dq_item(const fa_attn_args& p, const ScoreCfg& cfg, int cand, int nmb, QItem& w) {
  int i, rem;
  block_of(cand, nmb, p.batch * p.heads_q, cfg.unit_group, rem, i);
  w.h = rem % p.heads_q;
  w.b = rem / p.heads_q;
  w.m0 = (cfg.causal ? (nmb - 1 - i) : i) * kT;
  w.g = geo_of(p, w.b);
  w.n_hi = w.total = w.pad = 0;
  if (w.m0 >= w.g.q_len) return false;
  const int off = p.q_pos_offset;
  int klo, khi;
  visible_key_range(cfg, w.m0 + off, min(w.m0 + kT, w.g.q_len) - 1 + off, w.g.k_len, klo, khi);
  const int n_lo = klo / kT;
  w.n_hi = (khi + kT - 1) / kT;
  w.total = max(w.n_hi - n_lo, 0);
  return true;
}

}  // namespace

// =======================================================================================
// dK, dV
// =======================================================================================
// kDrop: P^T and dS^T are zero where the bit of (key, query row) in cfg.keep is 0, and scaled by
// dropout_scale, which is folded into the statistics operand (its log2 is added to -lse2).
template <typename T, int D, Feat kFeat, bool kDrop>
__global__ void __launch_bounds__(Roles<ew_groups(kFeat)>::kThreads, 1)
bwd_dkdv_sm100_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                      const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmdO,
                      const __grid_constant__ CUtensorMap tmdK, const __grid_constant__ CUtensorMap tmdV,
                      const fa_attn_args p, const ScoreCfg cfg, const int nkb, const int ncand,
                      unsigned int* const queue, int* const host_status) {
  using C = BCfg<D>;
  constexpr bool kExtras = kFeat != Feat::kNone, kCap = kFeat == Feat::kCap;
  constexpr int SQ = C::kStagesQ, SO = C::kStagesO;
  using R = Roles<ew_groups(kFeat)>;
  constexpr int kEwCols = R::kCols;              // columns per element-wise thread
  constexpr int kConsumers = R::kEwWarps + 3;   // warps that read the work queue: every element-wise one, issuer, statistics, store agent
  extern __shared__ unsigned char smem_raw[];
  unsigned char* tiles = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  BShared* sh = reinterpret_cast<BShared*>(tiles + C::kSmemTiles + C::kAugTotal);
  const uint32_t sK = smem_u32(tiles), sV = sK + C::kTileBytes;
  const uint32_t sRingQ = sV + C::kTileBytes, sRingO = sRingQ + SQ * C::kTileBytes;
  // statistics operands: one block per ring stage, then the two of the key side (bwd_stats.cuh)
  unsigned char* aug = tiles + C::kSmemTiles;
  const uint32_t sAug = sK + C::kSmemTiles, sAugKeys = sAug + SQ * kStatBlock;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int G = p.heads_q / p.heads_kv;
  const int off = p.q_pos_offset;

  auto slotA = [&](int pos) { return sRingQ + (pos % SQ) * C::kTileBytes; };
  auto slotB = [&](int pos) { return sRingO + (pos % SO) * C::kTileBytes; };

  if (tid == 0) {
    mbar_init(smem_u32(&sh->res_full), 1);
    mbar_init(smem_u32(&sh->res_free), 1);
    mbar_init(smem_u32(&sh->k_full), 1);
    mbar_init(smem_u32(&sh->k_free), 1);
    mbar_init(smem_u32(&sh->s_full[0]), 1);
    mbar_init(smem_u32(&sh->s_full[1]), 1);
    mbar_init(smem_u32(&sh->dp_full), 1);
    mbar_init(smem_u32(&sh->p_ready[0]), R::kEwThreads);
    mbar_init(smem_u32(&sh->p_ready[1]), R::kEwThreads);
    mbar_init(smem_u32(&sh->ds_ready), R::kEwThreads);
    mbar_init(smem_u32(&sh->dv_done), 1);
    mbar_init(smem_u32(&sh->acc_done), 1);
    for (int i = 0; i < 4; ++i) {
      mbar_init(smem_u32(&sh->full_a[i]), 2);   // the TMA load and the statistics warp
      mbar_init(smem_u32(&sh->full_b[i]), 1);
      mbar_init(smem_u32(&sh->empty_a[i]), 1);  // commit behind the slot's last reader, or the store agent
      mbar_init(smem_u32(&sh->empty_b[i]), 1);
    }
    for (int i = 0; i < kSched; ++i) {
      mbar_init(smem_u32(&sh->sched_full[i]), 1);
      mbar_init(smem_u32(&sh->sched_empty[i]), kConsumers);
    }
    mbar_init(smem_u32(&sh->stg_ready[0]), R::kEwThreads);
    mbar_init(smem_u32(&sh->stg_ready[1]), R::kEwThreads);
    mbar_init(smem_u32(&sh->stg_taken[0]), 1);
    sh->abort_flag = 0;
    fence_barrier_init();
  }
  stat_write_keys<T>(aug + SQ * kStatBlock, cfg.scale_log2, tid, R::kThreads);
  fence_proxy_async();
  if (warp == R::kProducer) {
    tmem_alloc(smem_u32(&sh->tmem_base), 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sh->tmem_base;
  // TMEM: S^T (128 fp32 columns, two buffers at head_dim 64) | dP^T (128) | dV (D) | dK (D).  P^T overwrites S^T and
  // dS^T overwrites dP^T, each element-wise group over its own columns.
  constexpr int NB = C::kSBuf;
  auto sbuf = [](int pos) { return pos % NB; };
  auto sphase = [](int pos) { return (uint32_t)(pos / NB) & 1u; };
  const uint32_t tS = tmem /* + buffer * 128 */, tdP = tmem + NB * 128;
  const uint32_t tdV = tmem + 512 - 2 * D, tdK = tmem + 512 - D;

  // Ring bookkeeping shared by every role.  An item with `total` query tiles takes ring A entries
  // Q(0) ... Q(total-1) and ring B entries dO(0) ... dO(total-1); every role advances one position
  // counter, entry `pos` lives in slot pos % stages and completes phase (pos / stages) & 1 of that
  // slot's barriers.  The entries of the LAST tile are released by the store agent (the epilogue stages
  // dK and dV over them), the others by the commits of the issuer.

  if (warp == R::kProducer) {
    // ------------------------------- TMA producer ---------------------------------------
    reg_dealloc<R::kRegsService>();
    if (lane == 0) {
      prefetch_tmap(&tmQ);
      prefetch_tmap(&tmK);
      prefetch_tmap(&tmV);
      prefetch_tmap(&tmdO);
      prefetch_tmap(&tmdK);
      prefetch_tmap(&tmdV);
      int pos = 0, wi = 0, fidx = 0;
      unsigned int u = blockIdx.x;
      bool ok = true;
      auto decode = [&](int c, KItem& w) { return dkdv_item(p, cfg, c, nkb, w); };
      // An item is drawn from the queue as late as possible -- before the last loads of the previous one,
      // two tiles or three before it ends -- so that the CTAs share the work evenly.
      for (;;) {
        const KItem w = sched_publish<KItem>(sh, queue, ncand, u, fidx, ok, decode);
        if (!ok || w.total < 0) break;
        if (w.total == 0) {
          u = queue_draw(queue, ncand);
          continue;
        }
        // Loads in order of use: K Q(0) V dO(0), Q(1) dO(1), ...  K's slot is free once the last score GEMM of the previous item has read it,
        // V's after its last dP GEMM.  (One copy, see the issuer.)
        int hq = w.hk * G, m = w.m_lo;
        const int m_end = w.m_lo + w.ntiles;
        for (int it = 0; it < w.total && ok; ++it, ++pos) {
          if (it + 1 == w.total) u = queue_draw(queue, ncand);
#pragma unroll 1
          for (int e = it == 0 ? 0 : 2; e < 4 && ok; ++e) {
            const int what = it == 0 ? e : 2 * e - 3;            // 0 K, 1 Q, 2 V, 3 dO
            const bool q = what == 1, resident = (what & 1) == 0, b = what >= 2;
            uint64_t* const empty = resident ? (b ? &sh->res_free : &sh->k_free) : q ? &sh->empty_a[pos % SQ] : &sh->empty_b[pos % SO];
            uint64_t* const full = resident ? (b ? &sh->res_full : &sh->k_full) : q ? &sh->full_a[pos % SQ] : &sh->full_b[pos % SO];
            const uint32_t parity = resident ? (wi - 1) & 1 : (((q ? pos / SQ : pos / SO) & 1) ^ 1);
            if (!resident || wi > 0) ok = bwait_relaxed(empty, parity, sh, 41);
            if (!ok) break;
            mbar_expect_tx(smem_u32(full), C::kTileBytes);
            load_tile<D>(resident ? (b ? sV : sK) : q ? slotA(pos) : slotB(pos), resident ? (b ? &tmV : &tmK) : q ? &tmQ : &tmdO, smem_u32(full),
                         resident ? w.g.k_row0 + w.n0 : w.g.q_row0 + m * kT, resident ? w.hk : hq, resident ? w.g.k_boff : w.g.q_boff);
          }
          if (++m == m_end) {
            m = w.m_lo;
            ++hq;
          }
        }
        if (!ok) break;
        ++wi;
      }
    }
  } else if (warp == R::kStats) {
    // ------------------------------- statistics loader ----------------------------------
    // The loads of the next tile are ISSUED right after the current one has been written and only consumed
    // after the wait for the next slot, so their latency hides behind that wait (nothing reads
    // the registers in between: a scoreboard stall before the poll would serialise the two; the pieces worked
    // out there too cost 4 x 1024 x 1531 of 32 heads of 64 387 -> 488 us).
    reg_dealloc<R::kRegsService>();
    float rl[kT / 32], rd[kT / 32];                  // statistics of rows lane, lane + 32, ... as loaded
    const float unit = stat_score_unit(cfg.scale_log2);
    auto fetch = [&](const KItem& w, int it) {
      const int hq = w.hk * G + it / w.ntiles, m = w.m_lo + it % w.ntiles;
#pragma unroll
      for (int k = 0; k < kT / 32; ++k) {
        const int row = m * kT + lane + 32 * k;
        rl[k] = INFINITY;
        rd[k] = 0.f;
        if (row < w.g.q_len) {
          const int64_t idx = (int64_t)w.g.q_boff * p.lse_stride[0] + (int64_t)(w.g.q_row0 + row) * p.lse_stride[1] +
                              (int64_t)hq * p.lse_stride[2];
          rl[k] = p.lse2[idx];
          rd[k] = p.delta[idx];
        }
      }
    };
    int pos = 0, sidx = 0;
    bool ok = true, fetched = false;                 // fetched: tile 0 of the item about to run is in rl/rd
    KItem w = sched_get<KItem>(sh, sidx++, true, ok);
    while (ok && w.total >= 0) {
      if (w.total == 0) {
        w = sched_get<KItem>(sh, sidx++, true, ok);
        continue;
      }
      bool haven = false;
      if (!fetched) fetch(w, 0);
      for (int it = 0; it < w.total; ++it, ++pos) {
        const int stage = pos % SQ;
        bool wt = true;
        if (lane == 0) wt = bwait_relaxed(&sh->empty_a[stage], ((pos / SQ) & 1) ^ 1, sh, 42);
        if (!__all_sync(0xffffffffu, wt)) { ok = false; break; }
#pragma unroll
        for (int k = 0; k < kT / 32; ++k) {
          const int i = lane + 32 * k;
          // NEGATED.  The feature variant adds the LSE after the soft cap, in the element-wise warps.
          const float nl2 = kDrop ? cfg.drop_log2 - rl[k] : -rl[k];
          if (kExtras) sh->lse[stage][i] = isinf(nl2) ? -INFINITY : nl2;
          stat_write_row<T, !kExtras>(aug + stage * kStatBlock, i, nl2, -rd[k], unit);
        }
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&sh->full_a[stage]));
        // the item's next tile, or the first one of the entry after this (published once the loads of this item are issued), if
        // that has work
        KItem wf = w;
        if (it + 1 == w.total) {
          wf = sched_get<KItem>(sh, sidx, false, ok);
          if (!ok) break;
          haven = wf.total > 0;
        }
        if (wf.total > 0) fetch(wf, it + 1 < w.total ? it + 1 : 0);
      }
      if (!ok) break;
      fetched = haven;
      w = sched_get<KItem>(sh, sidx++, true, ok);
    }
  } else if (warp == R::kIssuer) {
    // ------------------------------- MMA issuer -----------------------------------------
    // The GEMMs of tile i+1 follow, in the in-order tensor pipe, the accumulation of tile i that
    // reads the region they overwrite:
    //   P(i) stored:   dV += P(i)^T dO(i)   S(i + buffers)   (under the dS phase of tile i)
    //   dS(i) stored:  dK += dS(i)^T Q(i)   dP(i+1)          (under the exp2 phase of tile i+1)
    // so no barrier protects the regions from the GEMMs, and with one score buffer two stages of Q and of dO are
    // enough.  What protects them, and the barriers, from the warps: no warp arrives on a barrier again before its phase
    // is complete, because the scores that it needs first, S(i + buffers) after P(i), are issued behind that phase.  With
    // two score buffers that holds per buffer only: a warp can store P(i+1) while another has not stored P(i), so
    // each buffer has a barrier of its own.  For dS: dP(i+1), which dS(i+1) needs, is issued behind dS(i) of all warps.
    reg_dealloc<R::kRegsService>();
    constexpr uint32_t idesc_s = make_idesc(1, BFmt<T>::code, 0, 0, kT, kT);
    constexpr uint32_t idesc_acc = make_idesc(1, BFmt<T>::code, 0, 1, kT, D);
    const uint32_t leader = elect_one() ? 1u : 0u;
    bool ok = true;
    // every lane polls (uniform control flow, no vote needed: a completed phase is seen by all)
    auto wq = [&](uint64_t* bar, uint32_t parity, int code) {
      if (ok) ok = bwait(bar, parity, sh, code);
      tc_fence_after();
    };
    const uint64_t dstat_s = stat_desc_key(sAugKeys, false), dstat_dp = stat_desc_key(sAugKeys, true);
    auto stat_desc = [&](int ps, bool dp) { return stat_desc_query(sAugKeys, sAug + (ps % SQ) * kStatBlock, dp); };
    // The last query tile of a packed sequence also stages rows of the NEXT sequence.  Their P is
    // 0 (the statistics say so), but 0 * inf is NaN and dS^T Q, P^T dO contract over those rows:
    // this warp, the first reader of every staged Q and dO tile, zeroes them once the tile has
    // landed (scores and dP of those rows then are 0 too).
    // S^T = K Q^T - lse2 / scale_log2 for the tile at ring position ps
    auto issue_s = [&](int ps, int tail) {
      wq(&sh->full_a[ps % SQ], (ps / SQ) & 1, 44);
      if (!ok) return;
      if (tail < kT) zero_tile_tail<C::kBoxes, kT>(slotA(ps), tail, lane);
      const uint32_t d = tS + sbuf(ps) * 128;
      mma_kmajor<D>(d, sK, slotA(ps), idesc_s, leader);
      if (!kExtras) mma_f16_ss_lp(d, dstat_s, stat_desc(ps, false), idesc_s, 1u, leader);
      mma_commit_lp(smem_u32(&sh->s_full[sbuf(ps)]), leader);
    };
    // dP^T = V dO^T - delta
    auto issue_dp = [&](int ps, int tail) {
      wq(&sh->full_b[ps % SO], (ps / SO) & 1, 44);
      if (!ok) return;
      if (tail < kT) zero_tile_tail<C::kBoxes, kT>(slotB(ps), tail, lane);
      mma_kmajor<D>(tdP, sV, slotB(ps), idesc_s, leader);
      mma_f16_ss_lp(tdP, dstat_dp, stat_desc(ps, true), idesc_s, 1u, leader);
      mma_commit_lp(smem_u32(&sh->dp_full), leader);
    };
    int pos = 0, wi = 0, sidx = 0;
    for (;;) {
      const KItem w = sched_get<KItem>(sh, sidx++, true, ok);
      if (!ok || w.total < 0) break;
      if (w.total == 0) continue;
      const int last = w.total - 1;
      // the query tile that crosses the end of its sequence (-1: none) and its first row to zero;
      // the tiles repeat per query head
      const int tail_m = (p.cu_seqlens_q != nullptr && (w.g.q_len % kT) != 0) ? w.g.q_len / kT : -1;
      const int tail_first = w.g.q_len % kT, m_end = w.m_lo + w.ntiles;
      int ms = w.m_lo, mdp = w.m_lo;                   // query tiles of the next score and dP GEMMs
      wq(&sh->k_full, wi & 1, 43);
      // One copy of each part here, in the producer and in the element-wise warps: a launch that follows other kernels waits for what it
      // executes first (kernel of 104 -> 84 KB; within a training step, 8 x 16 x 512 of 128, causal 38.0 -> 34.7 us, 2 x 4 x 128 of 64
      // 8.4 -> 8.0, 60 x 32 x 128 of 64 72.8 -> 67.2).  At head_dim 64, where a tile is half as long, the tests of this form cost longer items 3 to
      // 10 %: first steps of their own there.
      if constexpr (NB == 1) {
        // Step -1 issues the first score and dP GEMMs.
        for (int i = -NB; i < w.total && ok; ++i) {
          const int ps = pos + i;
          if (i >= 0) {
            wq(&sh->p_ready[sbuf(ps)], sphase(ps), 45);
            if (!ok) break;
            mma_from_tmem<D, kEwCols>(tdV, tS + sbuf(ps) * 128, slotB(ps), idesc_acc, i > 0, leader);   // dV += P(i)^T dO(i)
            // (dO(i)'s other reader, dP(i), precedes in the pipe)
            mma_commit_lp(smem_u32(i < last ? &sh->empty_b[ps % SO] : &sh->dv_done), leader);
          }
          if (i + NB <= last) {
            issue_s(ps + NB, ms == tail_m ? tail_first : kT);
            if (ok && i + NB == last) mma_commit_lp(smem_u32(&sh->k_free), leader);      // K's last reader
            ms = (ms + 1 == m_end) ? w.m_lo : ms + 1;
          }
          if (i >= 0) {
            wq(&sh->ds_ready, ps & 1, 46);
            if (!ok) break;
            mma_from_tmem<D, kEwCols>(tdK, tdP, slotA(ps), idesc_acc, i > 0, leader);                   // dK += dS(i)^T Q(i)
            if (i < last) mma_commit_lp(smem_u32(&sh->empty_a[ps % SQ]), leader);
          }
          if (i >= -1 && i < last) {
            if (i < 0) wq(&sh->res_full, wi & 1, 43);
            issue_dp(ps + 1, mdp == tail_m ? tail_first : kT);
            if (ok && i + 1 == last) mma_commit_lp(smem_u32(&sh->res_free), leader);     // V's last reader
            mdp = (mdp + 1 == m_end) ? w.m_lo : mdp + 1;
          }
        }
      } else {
        auto next_s = [&](int i) {                       // S(i) of the item, whose tile 0 is at ring position pos
          if (i > last || !ok) return;
          issue_s(pos + i, ms == tail_m ? tail_first : kT);
          if (ok && i == last) mma_commit_lp(smem_u32(&sh->k_free), leader);     // K's last reader
          ms = (ms + 1 == m_end) ? w.m_lo : ms + 1;
        };
        auto next_dp = [&](int i) {
          if (i > last || !ok) return;
          issue_dp(pos + i, mdp == tail_m ? tail_first : kT);
          if (ok && i == last) mma_commit_lp(smem_u32(&sh->res_free), leader);   // V's last reader
          mdp = (mdp + 1 == m_end) ? w.m_lo : mdp + 1;
        };
        next_s(0);
        wq(&sh->res_full, wi & 1, 43);
        next_dp(0);
        if (NB == 2) next_s(1);
        for (int i = 0; i < w.total && ok; ++i) {
          const int ps = pos + i;
          const bool more = i < last;
          wq(&sh->p_ready[sbuf(ps)], sphase(ps), 45);
          if (!ok) break;
          mma_from_tmem<D, kEwCols>(tdV, tS + sbuf(ps) * 128, slotB(ps), idesc_acc, i > 0, leader);   // dV += P(i)^T dO(i)
          // (dO(i)'s other reader, dP(i), precedes in the pipe)
          mma_commit_lp(smem_u32(more ? &sh->empty_b[ps % SO] : &sh->dv_done), leader);
          next_s(i + NB);
          wq(&sh->ds_ready, ps & 1, 46);
          if (!ok) break;
          mma_from_tmem<D, kEwCols>(tdK, tdP, slotA(ps), idesc_acc, i > 0, leader);                   // dK += dS(i)^T Q(i)
          if (more) mma_commit_lp(smem_u32(&sh->empty_a[ps % SQ]), leader);
          next_dp(i + 1);
        }
      }
      pos += w.total;
      if (ok) mma_commit_lp(smem_u32(&sh->acc_done), leader);
      ++wi;
    }
    __syncwarp();
  } else if (warp == R::kStore) {
    // ------------------------------- store agent ----------------------------------------
    // The element-wise warps stage dV and dK over the item's last dO and Q tiles; this warp hands them
    // to the TMA unit and releases the two ring entries once the unit has read them.
    reg_dealloc<R::kRegsService>();
    const uint32_t leader = elect_one() ? 1u : 0u;
    int pos = 0, sidx = 0, wi = 0;
    bool ok = true;
    for (;;) {
      const KItem w = sched_get<KItem>(sh, sidx++, true, ok);
      if (!ok || w.total < 0) break;
      if (w.total == 0) continue;
      pos += w.total;
      const int stg = pos - 1;
      const bool via_tma = (p.cu_seqlens_k == nullptr) || (w.n0 + kT <= w.g.k_len);
      ok = bwait_long(&sh->stg_ready[0], wi & 1, sh, 62);
      if (ok && via_tma && leader) {
#pragma unroll
        for (int bx = 0; bx < D / 64; ++bx)
          tma_store_4d(&tmdV, slotB(stg) + bx * (kT * 128), bx * 64, w.hk, w.g.k_row0 + w.n0, w.g.k_boff);
        tma_store_commit();
      }
      if (ok) ok = bwait_long(&sh->stg_ready[1], wi & 1, sh, 62);
      if (!ok) break;
      if (leader) {
        mbar_arrive(smem_u32(&sh->stg_taken[0]));
        if (via_tma) {
#pragma unroll
          for (int bx = 0; bx < D / 64; ++bx)
            tma_store_4d(&tmdK, slotA(stg) + bx * (kT * 128), bx * 64, w.hk, w.g.k_row0 + w.n0, w.g.k_boff);
          tma_store_commit();
          tma_store_wait_read();
        }
        // released like tiles whose last reader has finished
        mbar_arrive(smem_u32(&sh->empty_b[stg % SO]));
        mbar_arrive(smem_u32(&sh->empty_a[stg % SQ]));
      }
      __syncwarp();
      ++wi;
    }
    __syncwarp();
  } else {
    // ------------------------------- element-wise groups --------------------------------
    reg_alloc<R::kRegsEw>();
    const int x = warp >> 2;                         // group: columns x * kEwCols and on
    const int lrow = (warp & 3) * 32 + lane;         // TMEM lane = key inside the tile
    const uint32_t lane_addr = (uint32_t)((warp & 3) * 32) << 16;
    // this group's kEwCols columns; the 16-bit pairs of P, of dS take the first half of them
    const uint32_t tSg = tS + lane_addr + x * kEwCols, tdPx = tdP + lane_addr + x * kEwCols;
    bool ok = true;
    int pos = 0, wi = 0, sidx = 0;
    PROF_VARS(16);
#ifdef FA_PROF
    const long long prof_start = clock64();
#endif

    KItem w;
    bool have = false;                               // w was looked at behind the item before it
    for (;;) {
      if (!have) w = sched_get<KItem>(sh, sidx++, true, ok);
      have = false;
      if (!ok || w.total < 0) break;
      const int key = w.n0 + lrow;
      // each group stores its part of the head_dim columns of dV and of dK * softmax_scale
      constexpr int DH = D * kEwCols / kT;
      auto row_of = [&](void* base, const int64_t* stride) -> T* {     // this thread's part of its key's row
        if (key >= w.g.k_len) return nullptr;
        return reinterpret_cast<T*>(base) + (int64_t)w.g.k_boff * stride[0] + (int64_t)(w.g.k_row0 + key) * stride[1] +
               (int64_t)w.hk * stride[2] + x * DH;
      };
      // Worked out here, under the wait for the first scores, or, with score options, where they are used (the registers are short): for
      // items of one query tile 1.5 % (60 x 32 heads x 128 of 64, causal 73.5 -> 72.5 us).
      T *gdv = nullptr, *gdk = nullptr;
      if (!kExtras || w.total == 0) {
        gdv = row_of(p.dv, p.dv_stride);
        gdk = row_of(p.dk, p.dk_stride);
      }
      if (w.total == 0) {
        // no query can see these keys: their gradients are zero
        if (gdv != nullptr) {
#pragma unroll
          for (int c = 0; c < DH / 8; ++c) {
            reinterpret_cast<uint4*>(gdv)[c] = make_uint4(0u, 0u, 0u, 0u);
            reinterpret_cast<uint4*>(gdk)[c] = make_uint4(0u, 0u, 0u, 0u);
          }
        }
        continue;
      }
      int vq_lo, vq_hi;                              // query positions that see this thread's key
      visible_q_interval(cfg, key, vq_lo, vq_hi);
      PROF_COUNT(9, w.total);
      PROF_COUNT(10, 1);

      // (the divisions of the other roles would be 0.2 k cycles at the start of every tile here, where nothing hides them)
      int hq = w.hk * G, m = w.m_lo;
      const int m_end = w.m_lo + w.ntiles;
      float slope = 0.f;
      for (int it = 0; it < w.total && ok; ++it, ++pos) {
        const int stage = pos % SQ;
        const int q0 = m * kT + x * kEwCols;            // first query row of this thread's columns
        if (kExtras && m == w.m_lo && cfg.has_alibi) slope = p.alibi_slopes[w.b * p.heads_q + hq];
        if (++m == m_end) {
          m = w.m_lo;
          ++hq;
        }
        bool masked = false;
        if (cfg.causal) masked |= (w.n0 + kT - 1 > q0 + off);
        if (cfg.wl >= 0) masked |= (w.n0 < q0 + kEwCols - 1 + off - cfg.wl);
        if (cfg.wr >= 0) masked |= (w.n0 + kT - 1 > q0 + off + cfg.wr);

        // Only the feature variant needs the LSE per column (it is added after the soft cap); otherwise the GEMMs deliver
        // S - lse and dP - delta.  It is fetched into registers BEFORE the wait for the scores: shared-memory loads issued
        // while the tensor pipe streams its operands take hundreds of cycles, and here that latency hides behind the wait.
        float st[kEwCols];                             // -lse
        if (kExtras) {
          ok = bwait(&sh->full_a[stage], (pos / SQ) & 1, sh, 47);
          if (!ok) break;
          const float4* L4 = reinterpret_cast<const float4*>(&sh->lse[stage][x * kEwCols]);
#pragma unroll
          for (int i4 = 0; i4 < kEwCols / 4; ++i4) {
            const float4 l4 = L4[i4];
            st[i4 * 4] = l4.x; st[i4 * 4 + 1] = l4.y; st[i4 * 4 + 2] = l4.z; st[i4 * 4 + 3] = l4.w;
          }
        }
        uint32_t keep[kEwCols / 32];                   // this thread's bits of the tile, on their way during the wait
        if (kDrop) {
#pragma unroll
          for (int h = 0; h < kEwCols / 32; ++h) keep[h] = __ldg(cfg.keep + key * cfg.keep_words + (q0 >> 5) + h);
        }
        PROF_T0();
        ok = bwait(&sh->s_full[sbuf(pos)], sphase(pos), sh, 46);
#ifdef FA_PROF
        if (it == 0) PROF_ADD(11); else PROF_ADD(0);
        PROF_T0();
#endif
        if (!ok) break;
        SKEW(warp, R::kEwWarps, pos, 0);
        tc_fence_after();

        // ---- exp phase: P = exp2(score - lse), written back as T pairs ---------------------
        uint32_t r[kEwCols / 32][32];
        const uint32_t tSx = tSg + sbuf(pos) * 128;
#pragma unroll
        for (int h = 0; h < kEwCols / 32; ++h) tmem_ld32(tSx + h * 32, r[h]);
        tmem_wait_ld();
        float pf[kEwCols];                              // P in fp32, kept for the dS phase
        const float dist0 = (float)(q0 + off - key);   // query position - key position of column 0
        // columns (query rows) of this tile that see this thread's key
        const ColMask cm = make_col_mask(vq_lo - (q0 + off), vq_hi - (q0 + off));
        // One body, compiled per masked tile: no branch inside the unrolled loops.
        // Half h of the group's columns: 32 scores to 16 pairs of P.
        auto exp_body = [&](const int h, const uint32_t (&rr)[32], auto mask_tag, auto abs_tag) {
          constexpr bool kMask = decltype(mask_tag)::value;
          [[maybe_unused]] constexpr bool kAbs = decltype(abs_tag)::value;
          uint32_t pk[16];
          if constexpr (kExtras) {
            // Packed pairs throughout (the loop body is what the instruction cache has to hold:
            // as 64 scalar chains this variant stalled more on instruction fetch than on anything
            // else).  The distance of a pair's columns advances by (2, 2); under the causal mask
            // every visible element has distance >= 0 and |.| is not needed.
            const float ka = kCap ? -(slope * cfg.inv_softcap) : -(slope * FA_LOG2E);
            const float kb = kCap ? cfg.scale * cfg.inv_softcap : cfg.scale_log2;
            const float cl = cfg.softcap * FA_LOG2E;
            const float2 ka2 = make_float2(ka, ka), kb2 = make_float2(kb, kb), cl2 = make_float2(cl, cl);
            const float2 one2 = make_float2(1.f, 1.f), none2 = make_float2(-1.f, -1.f), two2 = make_float2(2.f, 2.f);
            const float dh = dist0 + 32.f * h;
            float2 d2 = make_float2(dh, dh + 1.f);
#pragma unroll
            for (int i = 0; i < 32; i += 2) {
              const int c = h * 32 + i;
              const float2 sv2 = make_float2(__uint_as_float(rr[i]), __uint_as_float(rr[i + 1]));
              const float2 da = kAbs ? make_float2(fabsf(d2.x), fabsf(d2.y)) : d2;
              const float2 st2 = make_float2(st[c], st[c + 1]);
              float2 pe;
              if (kCap) {
                const float2 y2 = f2fma(ka2, da, f2mul(sv2, kb2));
                const float2 th2 = make_float2(tanh_approx(y2.x), tanh_approx(y2.y));
                const float2 a2 = f2fma(th2, cl2, st2);
                pe = make_float2(ex2(a2.x), ex2(a2.y));
                if (kMask) {
                  pe.x = col_visible(cm, c) ? pe.x : 0.f;
                  pe.y = col_visible(cm, c + 1) ? pe.y : 0.f;
                }
                pk[i >> 1] = Elem<T>::pack(pe.x, pe.y);
                // the tanh factor of the soft cap goes into the copy kept for dS
                pe = f2mul(pe, f2fma(f2mul(th2, th2), none2, one2));
              } else {
                const float2 a2 = f2fma(ka2, da, f2fma(sv2, kb2, st2));
                pe = make_float2(ex2(a2.x), ex2(a2.y));
                if (kMask) {
                  pe.x = col_visible(cm, c) ? pe.x : 0.f;
                  pe.y = col_visible(cm, c + 1) ? pe.y : 0.f;
                }
                pk[i >> 1] = Elem<T>::pack(pe.x, pe.y);
              }
              pf[c] = pe.x;
              pf[c + 1] = pe.y;
              d2 = f2add(d2, two2);
            }
          } else {
            const float2 c2 = make_float2(cfg.scale_log2, cfg.scale_log2);
#pragma unroll
            for (int i = 0; i < 32; i += 2) {
              const int c = h * 32 + i;
              const float2 a = f2mul(make_float2(__uint_as_float(rr[i]), __uint_as_float(rr[i + 1])), c2);
              float2 pe = make_float2(ex2(a.x), ex2(a.y));
              if (kMask) {
                pe.x = col_visible(cm, c) ? pe.x : 0.f;
                pe.y = col_visible(cm, c + 1) ? pe.y : 0.f;
              }
              if (kDrop) {
                const uint32_t kw = keep[h];
                pe.x = (kw >> i) & 1u ? pe.x : 0.f;
                pe.y = (kw >> (i + 1)) & 1u ? pe.y : 0.f;
              }
              pf[c] = pe.x;
              pf[c + 1] = pe.y;
              pk[i >> 1] = Elem<T>::pack(pe.x, pe.y);
            }
          }
          tmem_st16(tSx + h * 16, pk);
        };
        // |distance| only where a visible element can lie on the other side of the diagonal
        const bool need_abs = kExtras && !cfg.causal;
        auto run_exp = [&](auto mask_tag) {
#pragma unroll
          for (int h = 0; h < kEwCols / 32; ++h) {
            if (need_abs) exp_body(h, r[h], mask_tag, std::true_type{});
            else exp_body(h, r[h], mask_tag, std::false_type{});
          }
        };
        if (masked) run_exp(std::true_type{});
        else run_exp(std::false_type{});
        tmem_wait_st();
        tc_fence_before();
        mbar_arrive(smem_u32(&sh->p_ready[sbuf(pos)]));
#ifdef FA_PROF
        if (masked) { PROF_ADD(13); prof_acc[14] += 1; } else PROF_ADD(12);
#endif

        // ---- dS phase: dS = P (dP - delta) -------------------------------------------------
        PROF_T0();
        ok = bwait(&sh->dp_full, pos & 1, sh, 48);
        PROF_ADD(2);
        if (!ok) break;
        SKEW(warp, R::kEwWarps, pos, 1);
        PROF_T0();
        tc_fence_after();
#pragma unroll
        for (int h = 0; h < kEwCols / 32; ++h) tmem_ld32(tdPx + h * 32, r[h]);
        tmem_wait_ld();
#pragma unroll
        for (int c = 0; c < kEwCols / 32; ++c) {
          uint32_t pk[16];
          const uint32_t (&rr)[32] = r[c];
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const float2 ds = f2mul(make_float2(pf[c * 32 + 2 * i], pf[c * 32 + 2 * i + 1]),
                                    make_float2(__uint_as_float(rr[2 * i]), __uint_as_float(rr[2 * i + 1])));
            pk[i] = Elem<T>::pack(ds.x, ds.y);
          }
          tmem_st16(tdPx + c * 16, pk);
        }
        tmem_wait_st();
        tc_fence_before();
        mbar_arrive(smem_u32(&sh->ds_ready));
        PROF_ADD(15);
      }
      if (!ok) break;

      // Epilogue: dV is staged over the item's last dO tile while the last dK GEMM still runs, then dK over
      // the last Q tile (swizzled box layout), for the store agent, which lets the TMA unit write
      // full rows; a packed tile that reaches past the end of its sequence is stored row by row instead.
      // The first score and dP GEMMs of the next item run meanwhile.
      PROF_T0();
      const KItem wn = sched_get<KItem>(sh, sidx++, true, ok);
      PROF_ADD(7);
      if (!ok) break;
      const bool via_tma = (p.cu_seqlens_k == nullptr) || (w.n0 + kT <= w.g.k_len);
      PROF_T0();
      ok = bwait(&sh->dv_done, wi & 1, sh, 49);
      PROF_ADD(5);
      if (!ok) break;
      SKEW(warp, R::kEwWarps, wi, 2);
      tc_fence_after();
      PROF_T0();
      drain_acc<T, DH>(tdV + lane_addr + x * DH, 1.f, via_tma, slotB(pos - 1), lrow, x * DH, kExtras && !via_tma ? row_of(p.dv, p.dv_stride) : gdv);
      tc_fence_before();
      if (via_tma) fence_proxy_async();
      // (the agent has seen the previous item's tiles: its barrier is never a whole phase behind)
      if (wi > 0 && !(ok = bwait(&sh->stg_taken[0], (wi - 1) & 1, sh, 63))) break;
      mbar_arrive(smem_u32(&sh->stg_ready[0]));
      ok = bwait(&sh->acc_done, wi & 1, sh, 49);
      if (!ok) break;
      SKEW(warp, R::kEwWarps, wi, 3);
      tc_fence_after();
      drain_acc<T, DH>(tdK + lane_addr + x * DH, cfg.scale, via_tma, slotA(pos - 1), lrow, x * DH, kExtras && !via_tma ? row_of(p.dk, p.dk_stride) : gdk);
      tc_fence_before();
      if (via_tma) fence_proxy_async();
      mbar_arrive(smem_u32(&sh->stg_ready[1]));
      w = wn;
      have = true;
      PROF_ADD(6);
      ++wi;
    }
#ifdef FA_PROF
    prof_acc[8] = (unsigned int)(clock64() - prof_start);
#endif
    PROF_FLUSH(tid == 0, 0, 16);
  }

  tc_fence_before();
  __syncthreads();
  if (warp == R::kProducer) tmem_dealloc(tmem, 512);
  if (tid == 0) {
    queue_finish(queue, ncand);
    report_abort(sh->abort_flag, host_status);
  }
}

// =======================================================================================
// dQ
// =======================================================================================
// kDrop: dS is zero where the bit of (query row, key) in cfg.keep is 0; the scale of the kept probabilities
// is folded into the row's LSE.
template <typename T, int D, Feat kFeat, bool kDrop>
__global__ void __launch_bounds__(Roles<ew_groups(kFeat)>::kThreads, 1)
bwd_dq_sm100_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                    const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmdO,
                    const __grid_constant__ CUtensorMap tmdQ, const fa_attn_args p, const ScoreCfg cfg,
                    const int nmb, const int ncand, unsigned int* const queue,
                    int* const host_status) {
  using C = BCfg<D>;
  constexpr bool kExtras = kFeat != Feat::kNone, kCap = kFeat == Feat::kCap;
  constexpr int SK = C::kStagesK, SV = C::kStagesV;
  using R = Roles<ew_groups(kFeat)>;
  constexpr int kEwCols = R::kCols;              // columns per element-wise thread
  constexpr int kConsumers = R::kEwWarps + 1;    // warps that read the work queue: every element-wise one and the issuer
  extern __shared__ unsigned char smem_raw[];
  unsigned char* tiles = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  BShared* sh = reinterpret_cast<BShared*>(tiles + C::kSmemTilesDq);
  const uint32_t sQ = smem_u32(tiles), sdO = sQ + C::kTileBytes;
  const uint32_t sRingK = sdO + C::kTileBytes, sRingV = sRingK + SK * C::kTileBytes;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int off = p.q_pos_offset;

  auto slotK = [&](int pos) { return sRingK + (pos % SK) * C::kTileBytes; };
  auto slotV = [&](int pos) { return sRingV + (pos % SV) * C::kTileBytes; };

  if (tid == 0) {
    mbar_init(smem_u32(&sh->res_full), 1);
    mbar_init(smem_u32(&sh->res_free), 2);    // the last S GEMM and the last dP GEMM of the item
    mbar_init(smem_u32(&sh->s_full[0]), 1);
    mbar_init(smem_u32(&sh->s_full[1]), 1);
    mbar_init(smem_u32(&sh->dp_full), 1);
    mbar_init(smem_u32(&sh->ds_ready), R::kEwThreads);
    mbar_init(smem_u32(&sh->acc_done), 1);
    for (int i = 0; i < 4; ++i) {
      mbar_init(smem_u32(&sh->full_a[i]), 1);
      mbar_init(smem_u32(&sh->full_b[i]), 1);
      mbar_init(smem_u32(&sh->empty_a[i]), 1);
      mbar_init(smem_u32(&sh->empty_b[i]), 1);
    }
    for (int i = 0; i < kSched; ++i) {
      mbar_init(smem_u32(&sh->sched_full[i]), 1);
      mbar_init(smem_u32(&sh->sched_empty[i]), kConsumers);
    }
    mbar_init(smem_u32(&sh->stg_ready[0]), R::kEwThreads);
    mbar_init(smem_u32(&sh->stg_taken[0]), 1);
    sh->abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == R::kProducer) {
    tmem_alloc(smem_u32(&sh->tmem_base), 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sh->tmem_base;
  const uint32_t tS = tmem /* + buffer * 128 */, tdP = tmem + 256, tdQ = tmem + 384;

  // Ring bookkeeping: an item with `total` key tiles takes ring A entries K(0) ... K(total-1) and
  // ring B entries V(0) ... V(total-1); the last K entry is released by the epilogue, which
  // stages dQ over it.

  if (warp >= R::kStats) {
    reg_dealloc<R::kRegsService>();
    if (warp == R::kStats && lane == 0) {
      prefetch_tmap(&tmdQ);
      store_lane<D>(sh, 0, &tmdQ, 1);                 // the store lane of dQ
    }
  } else if (warp == R::kProducer) {
    // ------------------------------- TMA producer ---------------------------------------
    reg_dealloc<R::kRegsService>();
    if (lane == 0) {
      prefetch_tmap(&tmQ);
      prefetch_tmap(&tmK);
      prefetch_tmap(&tmV);
      prefetch_tmap(&tmdO);
      int posA = 0, posB = 0, wi = 0, fidx = 0;
      unsigned int u = blockIdx.x;
      bool ok = true;
      auto decode = [&](int c, QItem& w) { return dq_item(p, cfg, c, nmb, w); };
      for (;;) {
        const QItem w = sched_publish<QItem>(sh, queue, ncand, u, fidx, ok, decode);
        if (!ok || w.total < 0) break;
        if (w.total == 0) {
          u = queue_draw(queue, ncand);
          continue;
        }
        const int hk = w.h / (p.heads_q / p.heads_kv);
        // Q and dO: their slots are free once the last S and dP GEMMs of the previous item are done
        if (wi > 0 && !(ok = bwait_relaxed(&sh->res_free, (wi - 1) & 1, sh, 51))) break;
        {
          const uint32_t bar = smem_u32(&sh->res_full);
          mbar_expect_tx(bar, 2 * C::kTileBytes);
          load_tile<D>(sQ, &tmQ, bar, w.g.q_row0 + w.m0, w.h, w.g.q_boff);
          load_tile<D>(sdO, &tmdO, bar, w.g.q_row0 + w.m0, w.h, w.g.q_boff);
        }
        // K runs one tile ahead of V: K(j+1) is requested before V(j)
        auto load_k = [&](int j) {
          const int pos = posA + j;
          if (!bwait_relaxed(&sh->empty_a[pos % SK], ((pos / SK) & 1) ^ 1, sh, 51)) return false;
          const uint32_t bar = smem_u32(&sh->full_a[pos % SK]);
          mbar_expect_tx(bar, C::kTileBytes);
          load_tile<D>(slotK(pos), &tmK, bar, w.g.k_row0 + (w.n_hi - 1 - j) * kT, hk, w.g.k_boff);
          return true;
        };
        auto load_v = [&](int j) {
          const int pos = posB + j;
          if (!bwait_relaxed(&sh->empty_b[pos % SV], ((pos / SV) & 1) ^ 1, sh, 51)) return false;
          const uint32_t bar = smem_u32(&sh->full_b[pos % SV]);
          mbar_expect_tx(bar, C::kTileBytes);
          load_tile<D>(slotV(pos), &tmV, bar, w.g.k_row0 + (w.n_hi - 1 - j) * kT, hk, w.g.k_boff);
          return true;
        };
        ok = load_k(0);
        for (int j = 0; j < w.total && ok; ++j) {
          if (j + 1 == w.total) u = queue_draw(queue, ncand);
          if (j + 1 < w.total) ok = load_k(j + 1);
          if (ok) ok = load_v(j);
        }
        if (!ok) break;
        posA += w.total;
        posB += w.total;
        ++wi;
      }
    }
  } else if (warp == R::kIssuer) {
    // ------------------------------- MMA issuer -----------------------------------------
    reg_dealloc<R::kRegsService>();
    constexpr uint32_t idesc_s = make_idesc(1, BFmt<T>::code, 0, 0, kT, kT);
    constexpr uint32_t idesc_acc = make_idesc(1, BFmt<T>::code, 0, 1, kT, D);
    const uint32_t leader = elect_one() ? 1u : 0u;
    bool ok = true;
    auto wq = [&](uint64_t* bar, uint32_t parity, int code) {
      if (ok) ok = bwait(bar, parity, sh, code);
      tc_fence_after();
    };
    int posA = 0, posB = 0, wi = 0, tg = 0, sidx = 0; // tg: key tiles issued so far by this CTA
    for (;;) {
      const QItem w = sched_get<QItem>(sh, sidx++, true, ok);
      if (!ok || w.total < 0) break;
      if (w.total == 0) continue;
      const int last = w.total - 1;
      // The last key tile of a packed sequence (the first one visited) also stages rows of the NEXT
      // sequence.  Their P is 0, but 0 * inf is NaN and dS K contracts over those rows: this warp,
      // the first reader of every staged K and V tile, zeroes them once the tile has landed.
      const int tail = p.cu_seqlens_k == nullptr ? kT : max(0, min(kT, w.g.k_len - (w.n_hi - 1) * kT));
      wq(&sh->res_full, wi & 1, 53);
      wq(&sh->full_a[posA % SK], (posA / SK) & 1, 54);
      if (ok && tail < kT) zero_tile_tail<C::kBoxes, kT>(slotK(posA), tail, lane);
      if (ok) {
        mma_kmajor<D>(tS + (tg & 1) * kT, sQ, slotK(posA), idesc_s, leader);      // S(0) = Q K(0)^T
        mma_commit_lp(smem_u32(&sh->s_full[tg & 1]), leader);
        if (last == 0) mma_commit_lp(smem_u32(&sh->res_free), leader);
      }
      wq(&sh->full_b[posB % SV], (posB / SV) & 1, 54);
      if (ok && tail < kT) zero_tile_tail<C::kBoxes, kT>(slotV(posB), tail, lane);
      if (ok) {
        mma_kmajor<D>(tdP, sdO, slotV(posB), idesc_s, leader);                    // dP(0) = dO V(0)^T
        mma_commit_lp(smem_u32(&sh->dp_full), leader);
        mma_commit_lp(smem_u32(&sh->empty_b[posB % SV]), leader);
        if (last == 0) mma_commit_lp(smem_u32(&sh->res_free), leader);
      }
      for (int k = 0; k < w.total && ok; ++k, ++tg) {
        const int kpos = posA + k, k1pos = kpos + 1, v1pos = posB + k + 1;
        const bool more = k < last;
        if (more) {
          wq(&sh->full_a[k1pos % SK], (k1pos / SK) & 1, 54);
          if (!ok) break;
          mma_kmajor<D>(tS + ((tg + 1) & 1) * kT, sQ, slotK(k1pos), idesc_s, leader);   // S(k+1)
          mma_commit_lp(smem_u32(&sh->s_full[(tg + 1) & 1]), leader);
          if (k + 1 == last) mma_commit_lp(smem_u32(&sh->res_free), leader);      // Q's last reader
        }
        wq(&sh->ds_ready, tg & 1, 55);                // (dP(k+1), which dS(k+1) needs, is issued behind this phase)
        if (!ok) break;
        mma_from_tmem<D, kEwCols>(tdQ, tdP, slotK(kpos), idesc_acc, k > 0, leader);        // dQ += dS(k) K(k)
        if (more) mma_commit_lp(smem_u32(&sh->empty_a[kpos % SK]), leader);       // (the epilogue releases the last)
        if (more) {
          wq(&sh->full_b[v1pos % SV], (v1pos / SV) & 1, 54);
          if (!ok) break;
          mma_kmajor<D>(tdP, sdO, slotV(v1pos), idesc_s, leader);                 // dP(k+1)
          mma_commit_lp(smem_u32(&sh->dp_full), leader);
          mma_commit_lp(smem_u32(&sh->empty_b[v1pos % SV]), leader);
          if (k + 1 == last) mma_commit_lp(smem_u32(&sh->res_free), leader);      // dO's last reader
        }
      }
      if (ok) mma_commit_lp(smem_u32(&sh->acc_done), leader);
      posA += w.total;
      posB += w.total;
      ++wi;
    }
    __syncwarp();
  } else {
    // ------------------------------- element-wise groups --------------------------------
    reg_alloc<R::kRegsEw>();
    const int x = warp >> 2;
    const int lrow = (warp & 3) * 32 + lane;  // TMEM lane = query row inside the tile
    const uint32_t lane_addr = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t tdPx = tdP + lane_addr + x * kEwCols;
    constexpr int DH = D * kEwCols / kT;                 // each group stores its part of the head_dim columns
    bool ok = true;
    int posA = 0, wi = 0, tg = 0, sidx = 0;
    // statistics of this thread's row: base-2 LSE (+inf for rows that do not exist or see no
    // key: P = 0) and delta; those of the next item are fetched before the epilogue of this one
    auto row_stats = [&](const QItem& w, float& l2, float& dl) {
      l2 = INFINITY;
      dl = 0.f;
      const int row = w.m0 + lrow;
      if (row < w.g.q_len) {
        const int64_t idx = (int64_t)w.g.q_boff * p.lse_stride[0] + (int64_t)(w.g.q_row0 + row) * p.lse_stride[1] +
                            (int64_t)w.h * p.lse_stride[2];
        l2 = p.lse2[idx];
        dl = p.delta[idx];
        if (l2 == -INFINITY) l2 = INFINITY;
        if (kDrop) l2 -= cfg.drop_log2;
      }
    };
    float l2n = INFINITY, dln = 0.f;
    bool stats_ready = false;

    QItem w, wn;                                     // wn: the entry after the current one, once looked at
    bool peeked = false;
    for (;;) {
      if (peeked) {
        sched_release(sh, sidx++);
        w = wn;
      } else {
        w = sched_get<QItem>(sh, sidx++, true, ok);
      }
      if (!ok || w.total < 0) break;
      peeked = false;
      const int row = w.m0 + lrow;
      const int qpos = row + off;
      T* grow = nullptr;
      if (row < w.g.q_len)
        grow = reinterpret_cast<T*>(p.dq) + (int64_t)w.g.q_boff * p.dq_stride[0] +
               (int64_t)(w.g.q_row0 + row) * p.dq_stride[1] + (int64_t)w.h * p.dq_stride[2] + x * DH;
      if (w.total == 0) {
        // no key is visible from these rows: their gradient is zero
        if (grow != nullptr) {
#pragma unroll
          for (int c = 0; c < DH / 8; ++c) reinterpret_cast<uint4*>(grow)[c] = make_uint4(0u, 0u, 0u, 0u);
        }
        continue;
      }
      float l2, dl;
      if (stats_ready) { l2 = l2n; dl = dln; }
      else row_stats(w, l2, dl);
      const float slope = (kExtras && cfg.has_alibi) ? p.alibi_slopes[w.b * p.heads_q + w.h] : 0.f;
      int vk_lo, vk_hi;                              // key positions this thread's query row sees
      visible_k_interval(cfg, qpos, w.g.k_len, vk_lo, vk_hi);

      for (int j = 0; j < w.total && ok; ++j, ++tg) {
        const int k0 = (w.n_hi - 1 - j) * kT + x * kEwCols;   // first key of this thread's columns
        bool masked = (k0 + kEwCols > w.g.k_len);
        if (cfg.causal) masked |= (k0 + kEwCols - 1 > w.m0 + off);
        if (cfg.wl >= 0) masked |= (k0 < w.m0 + kT - 1 + off - cfg.wl);
        if (cfg.wr >= 0) masked |= (k0 + kEwCols - 1 > w.m0 + off + cfg.wr);

        uint32_t keep[kEwCols / 32];                   // this thread's bits of the tile, on their way during the wait
        if (kDrop) {
#pragma unroll
          for (int h = 0; h < kEwCols / 32; ++h) keep[h] = __ldg(cfg.keep + row * cfg.keep_words + (k0 >> 5) + h);
        }
        ok = bwait(&sh->s_full[tg & 1], (tg >> 1) & 1, sh, 56);
        if (!ok) break;
        SKEW(warp, R::kEwWarps, tg, 0);
        tc_fence_after();
        uint32_t r[kEwCols / 32][32];
        const uint32_t tSx = tS + (tg & 1) * kT + lane_addr + x * kEwCols;
#pragma unroll
        for (int h = 0; h < kEwCols / 32; ++h) tmem_ld32(tSx + h * 32, r[h]);
        tmem_wait_ld();
        // ---- exp phase: P (times the soft cap's tanh factor) in fp32 registers -------------
        const float dist0 = (float)(qpos - k0);        // query position - key position of column 0
        float pf[kEwCols];
        // columns (keys) of this tile that this thread's query row sees
        const ColMask cm = make_col_mask(vk_lo - k0, vk_hi - k0);
        // One body, compiled per masked tile: no branch inside the unrolled loops.
        auto exp_body = [&](auto mask_tag, auto abs_tag) {
          constexpr bool kMask = decltype(mask_tag)::value;
          constexpr bool kAbs = decltype(abs_tag)::value;
          if (kExtras) {
            // packed pairs; the distance of a pair's columns goes down by (2, 2)
            const FeatK fk = feat_k<kCap>(cfg, slope);
            const float cl = cfg.softcap * FA_LOG2E;
            const float2 cl2 = make_float2(cl, cl), nl2 = make_float2(-l2, -l2);
            const float2 one2 = make_float2(1.f, 1.f), none2 = make_float2(-1.f, -1.f), step2 = make_float2(-2.f, -2.f);
            float2 d2 = make_float2(dist0, dist0 - 1.f);
#pragma unroll
            for (int i = 0; i < kEwCols; i += 2) {
              const uint32_t (&rr)[32] = r[i / 32];
              const float2 sv2 = make_float2(__uint_as_float(rr[i & 31]), __uint_as_float(rr[(i & 31) + 1]));
              const float2 u2 = score_unit_feat2<kCap, kAbs>(fk, sv2, d2);
              const float2 a2 = kCap ? f2fma(u2, cl2, nl2) : f2add(u2, nl2);
              float2 pe = make_float2(ex2(a2.x), ex2(a2.y));
              if (kMask) {
                pe.x = col_visible(cm, i) ? pe.x : 0.f;
                pe.y = col_visible(cm, i + 1) ? pe.y : 0.f;
              }
              if (kCap) pe = f2mul(pe, f2fma(f2mul(u2, u2), none2, one2));   // times 1 - tanh^2
              pf[i] = pe.x;
              pf[i + 1] = pe.y;
              d2 = f2add(d2, step2);
            }
          } else {
            const float2 c2 = make_float2(cfg.scale_log2, cfg.scale_log2), nl = make_float2(-l2, -l2);
#pragma unroll
            for (int i = 0; i < kEwCols; i += 2) {
              const uint32_t (&rr)[32] = r[i / 32];
              const float2 a = f2fma(make_float2(__uint_as_float(rr[i & 31]), __uint_as_float(rr[(i & 31) + 1])), c2, nl);
              float2 pe = make_float2(ex2(a.x), ex2(a.y));
              if (kMask) {
                pe.x = col_visible(cm, i) ? pe.x : 0.f;
                pe.y = col_visible(cm, i + 1) ? pe.y : 0.f;
              }
              if (kDrop) {
                const uint32_t kw = keep[i / 32];
                pe.x = (kw >> (i & 31)) & 1u ? pe.x : 0.f;
                pe.y = (kw >> ((i & 31) + 1)) & 1u ? pe.y : 0.f;
              }
              pf[i] = pe.x;
              pf[i + 1] = pe.y;
            }
          }
        };
        const bool need_abs = kExtras && !cfg.causal;    // under the causal mask visible keys lie at distance >= 0
        auto run_exp = [&](auto mask_tag) {
          if (need_abs) exp_body(mask_tag, std::true_type{});
          else exp_body(mask_tag, std::false_type{});
        };
        if (masked) run_exp(std::true_type{});
        else run_exp(std::false_type{});

        // ---- dS phase --------------------------------------------------------------------
        ok = bwait(&sh->dp_full, tg & 1, sh, 57);
        if (!ok) break;
        SKEW(warp, R::kEwWarps, tg, 1);
        tc_fence_after();
#pragma unroll
        for (int h = 0; h < kEwCols / 32; ++h) tmem_ld32(tdPx + h * 32, r[h]);
        tmem_wait_ld();
#pragma unroll
        for (int c = 0; c < kEwCols / 32; ++c) {
          uint32_t pk[16];
          const uint32_t (&rr)[32] = r[c];
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const float2 d = f2add(make_float2(__uint_as_float(rr[2 * i]), __uint_as_float(rr[2 * i + 1])),
                                   make_float2(-dl, -dl));
            const float2 ds = f2mul(make_float2(pf[c * 32 + 2 * i], pf[c * 32 + 2 * i + 1]), d);
            pk[i] = Elem<T>::pack(ds.x, ds.y);
          }
          tmem_st16(tdPx + c * 16, pk);
        }
        tmem_wait_st();
        tc_fence_before();
        mbar_arrive(smem_u32(&sh->ds_ready));
      }
      if (!ok) break;

      // ---- end of the item: fetch the next item's row statistics, then store dQ * softmax_scale --
      {
        wn = sched_get<QItem>(sh, sidx, false, ok);
        if (!ok) break;
        peeked = true;
        stats_ready = wn.total > 0;
        if (stats_ready) row_stats(wn, l2n, dln);
      }
      // The tile is staged over the item's last K tile (every MMA is done) and handed to the store
      // lane, which lets the TMA unit write it; a packed tile that crosses the end of its sequence
      // is stored row by row instead.
      const int spos = posA + w.total - 1;
      ok = bwait(&sh->acc_done, wi & 1, sh, 58);
      if (!ok) break;
      SKEW(warp, R::kEwWarps, wi, 2);
      tc_fence_after();
      const bool via_tma = (p.cu_seqlens_q == nullptr) || (w.m0 + kT <= w.g.q_len);
      const uint32_t stg = slotK(spos);
      if (tid == 0)
        ok = post_store(sh, 0, wi, via_tma ? (int)stg : 0, w.h, w.g.q_row0 + w.m0, w.g.q_boff,
                        smem_u32(&sh->empty_a[spos % SK]));
      drain_acc<T, DH>(tdQ + lane_addr + x * DH, cfg.scale, via_tma, stg, lrow, x * DH, grow);
      tc_fence_before();
      if (via_tma) fence_proxy_async();
      mbar_arrive(smem_u32(&sh->stg_ready[0]));
      posA += w.total;
      ++wi;
    }
    // No more items: the store lane may leave.  Between items the products of the next one wait for every warp, so that none
    // arrives on stg_ready twice in a phase; here the warps wait for one another (all of them get here, whatever `ok` says).
    asm volatile("bar.sync 1, %0;\n" ::"n"(R::kEwThreads) : "memory");
    if (ok) {
      if (tid == 0) ok = post_store(sh, 0, wi, -1, 0, 0, 0, 0);
      mbar_arrive(smem_u32(&sh->stg_ready[0]));
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == R::kProducer) tmem_dealloc(tmem, 512);
  if (tid == 0) {
    queue_finish(queue, ncand);
    report_abort(sh->abort_flag, host_status);
  }
}

// =======================================================================================
// host side
// =======================================================================================
bool bwd_sm100_supported(const fa_attn_args& a) {
  if (a.head_dim != 128 && a.head_dim != 64) return false;
  if (a.softmax_scale < 0.f) return false;
  if (a.batch == 0 || a.seqlen_q == 0 || a.seqlen_k == 0) return false;
  // No lower bound on the lengths: even where one tile is mostly padding these kernels are ahead of the
  // mma.sync ones (GPU time of the three backward launches, causal: 2 x 16 tokens, 4 heads of 64 28 -> 16 us,
  // 2 x 128 42 -> 17, 16 x 64 of 16 heads 32 -> 26, 16 x 200 of 16 heads of 128 295 -> 68 us).  With a soft cap they
  // start where the tanh of these kernels, good to 2^-11 of the capped score, always set the precision.
  if (a.impl == FA_IMPL_AUTO && a.softcap > 0.f && (a.seqlen_k < 256 || a.seqlen_q < 128)) return false;
  return true;
}

namespace {

bool make_map4(CUtensorMap* m, const void* base, const int64_t* stride, int rows, int heads, int batch,
               int D, bool packed) {
  const uint64_t dims[4] = {(uint64_t)D, (uint64_t)heads, (uint64_t)rows, (uint64_t)(packed ? 1 : batch)};
  const uint64_t strides[3] = {(uint64_t)stride[2] * 2, (uint64_t)stride[1] * 2,
                               (uint64_t)(packed ? (int64_t)rows * stride[1] : stride[0]) * 2};
  const uint32_t box[4] = {64, 1, 128, 1};
  return encode_tmap(m, base, 2, 4, dims, strides, box);
}

struct Maps { CUtensorMap q, k, v, dout, dq, dk, dv; };

bool make_maps(Maps& m, const fa_attn_args& a) {
  const bool packed = a.cu_seqlens_q != nullptr;
  const int qr = packed ? a.total_q : a.seqlen_q, kr = packed ? a.total_k : a.seqlen_k;
  const int D = a.head_dim;
  return make_map4(&m.q, a.q, a.q_stride, qr, a.heads_q, a.batch, D, packed) &&
         make_map4(&m.k, a.k, a.k_stride, kr, a.heads_kv, a.batch, D, packed) &&
         make_map4(&m.v, a.v, a.v_stride, kr, a.heads_kv, a.batch, D, packed) &&
         make_map4(&m.dout, a.dout, a.do_stride, qr, a.heads_q, a.batch, D, packed) &&
         (a.dq == nullptr || make_map4(&m.dq, a.dq, a.dq_stride, qr, a.heads_q, a.batch, D, packed)) &&
         (a.dk == nullptr || make_map4(&m.dk, a.dk, a.dk_stride, kr, a.heads_kv, a.batch, D, packed)) &&
         (a.dv == nullptr || make_map4(&m.dv, a.dv, a.dv_stride, kr, a.heads_kv, a.batch, D, packed));
}

template <typename K> int set_smem_attr(K kern, int bytes, const char* what) {
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e != cudaSuccess) {
    set_error("%s: cudaFuncSetAttribute(%d): %s", what, bytes, cudaGetErrorString(e));
    return FA_ERR_LAUNCH;
  }
  return FA_OK;
}

// threads of a CTA of the plain variants, of those with score options
int threads_of(bool options) {
  return options ? Roles<ew_groups(Feat::kCap)>::kThreads : Roles<ew_groups(Feat::kNone)>::kThreads;
}
static_assert(ew_groups(Feat::kAlibi) == ew_groups(Feat::kCap), "one size for all options");

// candidates of a launch: blocks x heads x batch must stay a 32-bit count
bool candidate_count(int64_t blocks, int64_t heads, int64_t batch, int* out) {
  const int64_t n = blocks * heads * batch;
  if (n <= 0 || n > 0x7fffffff) return false;
  *out = (int)n;
  return true;
}

// Q, dO, K and V of a group: 64 MB.  dQ and dK/dV together without groups, in groups of 16, 32, 64 and 96 MB (us), causal:
// 16 x 16 x 4096 of 128 3964, 3973, 3954, 3869, 3854; 16 x 16 x 2048 of 64 836, 740, 725, 717, 717; 64 x 16 x 512 of 64
// 438, 366, 357, 356, 358; 1 x 16 x 8192 of 128 972, 897, 881, 877, 880; window of 200, 16 x 16 x 2048 of 64 446, 388, 382, 377, 377;
// 48 packed sequences of 64 to 4096, 16 heads of 128 4655, 4576, 4488, 4461, 4510.
ScoreCfg with_order(const fa_attn_args& a, const ScoreCfg& cfg, int heads) {
  const bool packed = a.cu_seqlens_q != nullptr;
  const int64_t q = packed ? a.total_q : (int64_t)a.batch * a.seqlen_q, k = packed ? a.total_k : (int64_t)a.batch * a.seqlen_k;
  ScoreCfg c = cfg;
  c.unit_group = unit_group(a, cfg, heads, 4 * a.head_dim * (q * a.heads_q + k * a.heads_kv), (int64_t)64 << 20);
  return c;
}

template <typename T, int D>
int launch_dkdv(const fa_attn_args& a, const ScoreCfg& cfg, cudaStream_t st) {
  Maps m{};
  if (!make_maps(m, a)) {
    set_error("bwd_dkdv_sm100: cuTensorMapEncodeTiled failed");
    return FA_ERR_LAUNCH;
  }
  // The plain variant folds -lse2 / scale_log2 into the score GEMM through 16-bit operands; a
  // scale so small that its reciprocal leaves the fp16 range takes the feature variant, whose
  // element-wise warps add the LSE themselves.
  const bool extras = cfg.has_alibi || cfg.softcap > 0.f || !(cfg.scale_log2 > 2e-5f);
  auto kern = cfg.keep != nullptr  ? bwd_dkdv_sm100_kernel<T, D, Feat::kNone, true>
              : cfg.softcap > 0.f ? bwd_dkdv_sm100_kernel<T, D, Feat::kCap, false>
              : extras            ? bwd_dkdv_sm100_kernel<T, D, Feat::kAlibi, false>
                                  : bwd_dkdv_sm100_kernel<T, D, Feat::kNone, false>;
  if (int r = set_smem_attr(kern, BCfg<D>::kSmemBytes, "bwd_dkdv_sm100")) return r;
  const int nkb = (a.seqlen_k + kT - 1) / kT;
  int ncand = 0;
  if (!candidate_count(nkb, a.heads_kv, a.batch, &ncand)) {
    set_error("bwd_dkdv_sm100: too many work items");
    return FA_ERR_UNSUPPORTED;
  }
  unsigned int* queue;
  const int grid = queue_grid(a.device, st, ncand, sm_count(a.device), &queue);
  kern<<<grid, threads_of(cfg.keep == nullptr && extras), BCfg<D>::kSmemBytes, st>>>(
      m.q, m.k, m.v, m.dout, m.dk, m.dv, a, with_order(a, cfg, a.heads_kv), nkb, ncand, queue, host_wait_word(a.device));
  return check_launch("bwd_dkdv_sm100");
}

template <typename T, int D>
int launch_dq(const fa_attn_args& a, const ScoreCfg& cfg, cudaStream_t st) {
  Maps m{};
  if (!make_maps(m, a)) {
    set_error("bwd_dq_sm100: cuTensorMapEncodeTiled failed");
    return FA_ERR_LAUNCH;
  }
  auto kern = cfg.keep != nullptr  ? bwd_dq_sm100_kernel<T, D, Feat::kNone, true>
              : cfg.softcap > 0.f ? bwd_dq_sm100_kernel<T, D, Feat::kCap, false>
              : cfg.has_alibi     ? bwd_dq_sm100_kernel<T, D, Feat::kAlibi, false>
                                  : bwd_dq_sm100_kernel<T, D, Feat::kNone, false>;
  if (int r = set_smem_attr(kern, BCfg<D>::kSmemBytesDq, "bwd_dq_sm100")) return r;
  const int nmb = (a.seqlen_q + kT - 1) / kT;
  int ncand = 0;
  if (!candidate_count(nmb, a.heads_q, a.batch, &ncand)) {
    set_error("bwd_dq_sm100: too many work items");
    return FA_ERR_UNSUPPORTED;
  }
  unsigned int* queue;
  const int grid = queue_grid(a.device, st, ncand, sm_count(a.device), &queue);
  kern<<<grid, threads_of(cfg.keep == nullptr && (cfg.has_alibi || cfg.softcap > 0.f)), BCfg<D>::kSmemBytesDq, st>>>(
      m.q, m.k, m.v, m.dout, m.dq, a, with_order(a, cfg, a.heads_q), nmb, ncand, queue, host_wait_word(a.device));
  return check_launch("bwd_dq_sm100");
}

}  // namespace

int bwd_dkdv_sm100(const fa_attn_args& a, const ScoreCfg& cfg, cudaStream_t st) {
  if (a.head_dim == 128)
    return a.dtype == FA_BF16 ? launch_dkdv<__nv_bfloat16, 128>(a, cfg, st) : launch_dkdv<__half, 128>(a, cfg, st);
  return a.dtype == FA_BF16 ? launch_dkdv<__nv_bfloat16, 64>(a, cfg, st) : launch_dkdv<__half, 64>(a, cfg, st);
}

int bwd_dq_sm100(const fa_attn_args& a, const ScoreCfg& cfg, cudaStream_t st) {
  if (a.head_dim == 128)
    return a.dtype == FA_BF16 ? launch_dq<__nv_bfloat16, 128>(a, cfg, st) : launch_dq<__half, 128>(a, cfg, st);
  return a.dtype == FA_BF16 ? launch_dq<__nv_bfloat16, 64>(a, cfg, st) : launch_dq<__half, 64>(a, cfg, st);
}

void bwd_sm100_clear_status() {
  const int z = 0;
  cudaMemcpyToSymbol(g_bwd_sm100_status, &z, sizeof(int));
}

int bwd_sm100_status() {
  int v = 0;
  cudaMemcpyFromSymbol(&v, g_bwd_sm100_status, sizeof(int));
  return v;
}

}  // namespace fa
