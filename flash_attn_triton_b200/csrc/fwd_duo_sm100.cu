// Forward attention on the 5th-generation tensor cores, one tile of 128 query rows per CTA and TWO CTAs per SM.
//
// A CTA has a softmax warpgroup, a TMA producer and an MMA issuer, one score buffer and one accumulator: half of an
// SM's tensor memory, shared memory and registers.  The two CTAs of an SM run out of phase by themselves, so that while
// one is in its exponentials the tensor pipe runs the other's P V and Q K^T, and the start and the end of a CTA (barriers,
// tensor memory, the first loads; the last P V and the output) lie under the other's work.
//
//   warps 0-3   softmax: one thread per query row (TMEM lane = row), all 128 scores of a tile in registers
//   warp  4     TMA producer: the Q tile once, then K/V tiles through a ring, in order of use K0 V0 K1 V1 ...
//   warp  5     MMA issuer: S = Q K_j^T (SS);  O += P V_j (A = P from tensor memory)
//   warps 6-7   idle (they complete the warpgroup that gives its registers to the softmax warps)
//
// At head_dim 128 P (fp16/bf16) overwrites the first 64 columns of S; Q K_{j+1}^T may overwrite it because P V_j precedes it
// in the in-order tensor pipe.  At head_dim 64 the accumulator leaves 64 columns, which P has to itself: Q K_{j+1}^T follows
// as soon as the scores of tile j are in registers and runs under their exponentials, where it came behind P V_j, with
// nothing of this CTA to do meanwhile (us, before -> after: 4 x 32 heads x 1024 x 1531 92.1 -> 88.0, 4 x 16 x 4096 causal 225 -> 219,
// 8 x 16 x 512 with dropout 25.3 -> 24.3, 24 packed of 64 to 2048 211 -> 206); rows that are too short for that keep P over S
// (p_over_s_is_faster).  Arithmetic, order of the tiles and of the sums are those of the two-tile kernels
// (fwd_sm100.cu, fwd_persist_sm100.cu): results are equal bit for bit.
//
// TMEM (256 columns): S (128) | O (head_dim) | P of its own (64).  Every mbarrier wait is bounded.
#include <type_traits>

#include "common.cuh"
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

template <int D> struct DCfg {
  static constexpr int kTileBytes = kBN * D * 2;
  static constexpr int kStages = (D == 128) ? 2 : 4;
  static constexpr int kBoxes = D / 64;
  static constexpr int kSmemTiles = (1 + kStages) * kTileBytes;
  static constexpr int kSmemBytes = kSmemTiles + 1024 /*align slack*/ + 1024 /*DShared*/;
  static_assert(2 * (kSmemBytes + 1024) <= 228 * 1024, "two CTAs per SM");
};

struct DShared {
  uint64_t q_full;
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
  uint32_t tmem_base;
  volatile int abort_flag;
};

__device__ __forceinline__ bool wait_bar(uint64_t* bar, uint32_t parity, DShared* sh, int code) {
  return bounded_wait(bar, parity, &sh->abort_flag, &g_fwd_duo_status, code);
}

template <typename T> struct DFmt;
template <> struct DFmt<__half> { static constexpr int code = 0; };
template <> struct DFmt<__nv_bfloat16> { static constexpr int code = 1; };

}  // namespace

// kDrop: probabilities whose bit in cfg.keep is 0 do not enter P V (they stay in the row sum); the scale of
// the kept ones goes into the normalisation of the output.  kOwnP: P in columns of its own (head_dim 64).
template <typename T, int D, Feat kFeat, bool kDrop, bool kOwnP>
__global__ void __launch_bounds__(kThreads, 2)
fwd_duo_sm100_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                     const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmO,
                     const fa_attn_args p, const ScoreCfg cfg, int* const host_status) {
  constexpr bool kExtras = kFeat != Feat::kNone, kCap = kFeat == Feat::kCap;
  constexpr bool kPvSplit = !kExtras;     // P V in two key halves (measured: helps the plain variants only)
  static_assert(!kOwnP || D == 64, "at head_dim 128 S and O fill the columns");
  constexpr int kPCol = kOwnP ? kBN + D : 0;
  using C = DCfg<D>;
  constexpr int S = C::kStages;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* tiles = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  DShared* sh = reinterpret_cast<DShared*>(tiles + C::kSmemTiles);
  const uint32_t sQ = smem_u32(tiles), sKV = sQ + C::kTileBytes;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  int h, b, mt;
  SeqInfo si;
  if (p.cu_seqlens_q != nullptr) {
    if (!packed_tile<kBM>(p, cfg, lane, h, b, si, mt)) return;
  } else {
    const int mtiles = (p.seqlen_q + kBM - 1) / kBM;
    dense_block(p, cfg, mtiles, b, h, mt);
    if (cfg.causal) mt = mtiles - 1 - mt;          // heavy tiles first
    si = seq_info(p, b);
  }
  const int m0 = mt * kBM;
  if (m0 >= si.q_len) return;
  const int hk = h / (p.heads_q / p.heads_kv);
  const int off = p.q_pos_offset;
  int n_hi, nt;                                    // step j works on key tile n_hi - 1 - j: masked tiles first
  {
    int klo, khi;
    visible_key_range(cfg, m0 + off, min(m0 + kBM, si.q_len) - 1 + off, si.k_len, klo, khi);
    n_hi = (khi + kBN - 1) / kBN;
    nt = khi > klo ? n_hi - klo / kBN : 0;
  }

  if (tid == 0) {
    mbar_init(smem_u32(&sh->q_full), 1);
    mbar_init(smem_u32(&sh->s_full), 1);
    mbar_init(smem_u32(&sh->s_free), 128);
    mbar_init(smem_u32(&sh->o_ready), 1);
    mbar_init(smem_u32(&sh->p_half), 128);
    mbar_init(smem_u32(&sh->p_ready), 128);
    for (int i = 0; i < S; ++i) {
      mbar_init(smem_u32(&sh->kv_full[i]), 1);
      mbar_init(smem_u32(&sh->kv_empty[i]), 1);
    }
    sh->abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 4) {
    tmem_alloc(smem_u32(&sh->tmem_base), 256);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sh->tmem_base;

  if (warp >= 6) {
    reg_dealloc<kRegsService>();
  } else if (warp == 4) {
    // ------------------------------- TMA producer ---------------------------------------
    reg_dealloc<kRegsService>();
    if (lane == 0 && nt > 0) {
      const uint32_t qbar = smem_u32(&sh->q_full);
      mbar_expect_tx(qbar, C::kTileBytes);
      for (int bx = 0; bx < C::kBoxes; ++bx)
        tma_load_4d(sQ + bx * (kBM * 128), &tmQ, qbar, bx * 64, h, (int)si.q_row0 + m0, (int)si.q_boff);
      prefetch_tmap(&tmO);
      const int krow0 = (int)si.k_row0, kb = (int)si.k_boff;
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int i = 0; i < 2 * nt && ok; ++i) {       // K_0 V_0 K_1 V_1 ...
        ok = wait_bar(&sh->kv_empty[stage], phase ^ 1, sh, 11);
        if (!ok) break;
        const uint32_t bar = smem_u32(&sh->kv_full[stage]);
        mbar_expect_tx(bar, C::kTileBytes);
        for (int bx = 0; bx < C::kBoxes; ++bx)
          tma_load_4d(sKV + stage * C::kTileBytes + bx * (kBN * 128), (i & 1) ? &tmV : &tmK, bar, bx * 64, hk,
                      krow0 + (n_hi - 1 - (i >> 1)) * kBN, kb);
        if (++stage == S) { stage = 0; phase ^= 1; }
      }
    }
  } else if (warp == 5) {
    // ------------------------------- MMA issuer -----------------------------------------
    // The whole warp runs the control flow in lock step and every lane polls the barriers;
    // the lane chosen once by elect_one issues the MMAs and commits.
    reg_dealloc<kRegsService>();
    if (nt > 0) {
      constexpr uint32_t idesc_qk = make_idesc(1, DFmt<T>::code, 0, 0, kBM, kBN);
      constexpr uint32_t idesc_pv = make_idesc(1, DFmt<T>::code, 0, 1, kBM, D);
      const uint32_t leader = elect_one() ? 1u : 0u;
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      auto wwait = [&](uint64_t* bar, uint32_t parity, int code) {
        if (ok) ok = wait_bar(bar, parity, sh, code);
        tc_fence_after();
      };
      auto issue_qk = [&]() {                        // S = Q K^T with this tile of the ring
        wwait(&sh->kv_full[stage], phase, 22);
        if (!ok) return;
        const uint64_t dq = make_smem_desc(sQ, 16, 1024), dk = make_smem_desc(sKV + stage * C::kTileBytes, 16, 1024);
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
          const uint32_t o = ((kk / 4) * (kBM * 128) + (kk % 4) * 32) >> 4;
          mma_f16_ss_lp(tmem, dq + o, dk + o, idesc_qk, kk > 0, leader);
        }
        mma_commit_lp(smem_u32(&sh->s_full), leader);
        mma_commit_lp(smem_u32(&sh->kv_empty[stage]), leader);
      };
      auto advance = [&]() {
        if (++stage == S) { stage = 0; phase ^= 1; }
      };
      auto issue_pv = [&](int j) {                   // O += P V_j with this tile of the ring
        wwait(&sh->kv_full[stage], phase, 24);
        const uint64_t dv = make_smem_desc(sKV + stage * C::kTileBytes, kBN * 128, 1024);
        if (kPvSplit) {
          wwait(&sh->p_half, j & 1, 25);
          if (!ok) return;
#pragma unroll
          for (int kk = 0; kk < kBN / 32; ++kk)
            mma_f16_ts_lp(tmem + kBN, tmem + kPCol + kk * 8, dv + ((kk * 2048) >> 4), idesc_pv, (j > 0 || kk > 0) ? 1u : 0u, leader);
        }
        wwait(&sh->p_ready, j & 1, 25);
        if (!ok) return;
#pragma unroll
        for (int kk = kPvSplit ? kBN / 32 : 0; kk < kBN / 16; ++kk)
          mma_f16_ts_lp(tmem + kBN, tmem + kPCol + kk * 8, dv + ((kk * 2048) >> 4), idesc_pv, (j > 0 || kk > 0) ? 1u : 0u, leader);
        mma_commit_lp(smem_u32(&sh->o_ready), leader);
        mma_commit_lp(smem_u32(&sh->kv_empty[stage]), leader);
      };
      wwait(&sh->q_full, 0, 21);
      if constexpr (kOwnP) {
        // S(j + 1) goes before P V_j, while the softmax warps have S(j) in registers.  K_j is entry 2 j of the ring, V_j the
        // one behind it.
        static_assert(S == 4, "K tiles take slots 0 and 2, V tiles 1 and 3");
        for (int j = 0; j <= nt && ok; ++j) {
          if (j < nt) {
            if (j > 0) wwait(&sh->s_free, (j - 1) & 1, 26);
            stage = 2 * (j & 1);
            phase = (j >> 1) & 1;
            if (ok) issue_qk();
          }
          if (j > 0 && ok) {
            stage = 2 * ((j - 1) & 1) + 1;
            phase = ((j - 1) >> 1) & 1;
            issue_pv(j - 1);
          }
        }
      } else {
        if (ok) issue_qk();
        advance();
        for (int j = 0; j < nt && ok; ++j) {
          issue_pv(j);
          if (!ok) break;
          advance();
          if (j + 1 < nt) {
            issue_qk();
            advance();
          }
        }
      }
    }
  } else {
    // ------------------------------- softmax --------------------------------------------
    reg_alloc<kRegsSoftmax>();
    const int row_in_tile = tid;                     // TMEM lane
    const int row = m0 + row_in_tile;                // query row inside the sequence
    const int qpos = row + off;
    const uint32_t lane_addr = (uint32_t)(warp * 32) << 16;
    const uint32_t tSx = tmem + lane_addr, tOx = tSx + kBN;
    const float slope = (kExtras && cfg.has_alibi) ? p.alibi_slopes[b * p.heads_q + h] : 0.f;
    float m_used = -INFINITY, l = 0.f;
    bool ok = true;
    const int tq_min = m0 + off, tq_max = tq_min + kBM - 1;

    for (int j = 0; j < nt && ok; ++j) {
      const int k0 = (n_hi - 1 - j) * kBN;
      bool masked = (k0 + kBN > si.k_len);
      if (cfg.causal) masked |= (k0 + kBN - 1 > tq_min);
      if (cfg.wl >= 0) masked |= (k0 < tq_max - cfg.wl);
      if (cfg.wr >= 0) masked |= (k0 + kBN - 1 > tq_min + cfg.wr);

      uint4 keep4;                                   // the row's 128 bits of the tile, on their way during the wait
      if (kDrop) keep4 = __ldg(reinterpret_cast<const uint4*>(cfg.keep + row * cfg.keep_words + (k0 >> 5)));

      ok = wait_bar(&sh->s_full, j & 1, sh, 31);
      if (!ok) break;
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

      const bool prescaled = kExtras || masked;
      // columns (keys) of this tile that this thread's query row sees (used by masked tiles only)
      ColMask cm;
      if (masked) {
        int vk_lo, vk_hi;
        visible_k_interval(cfg, qpos, si.k_len, vk_lo, vk_hi);
        cm = make_col_mask(vk_lo - k0, vk_hi - k0);
      }
      if (prescaled) {
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
      // exactly 0, but 0 * inf or 0 * NaN is NaN: zero those rows of the V tile (ring entry 2 j + 1) before P is handed
      // to the issuer.  One thread per row; the swizzle does not matter.
      if (p.cu_seqlens_k != nullptr && k0 + kBN > si.k_len) {
        const int vpos = 2 * j + 1;
        ok = wait_bar(&sh->kv_full[vpos % S], (vpos / S) & 1, sh, 39);
        if (!ok) break;
        if (k0 + row_in_tile >= si.k_len) {
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

      // ---- lazy rescale ----------------------------------------------------------------
      if (j == 0) {
        m_used = mx;
      } else {
        const bool need = mx > m_used + cfg.rescale_at;
        if (__any_sync(0xffffffffu, need)) {
          // The previous P V of this stream is its (j-1)-th; the one of this tile cannot
          // complete before P is written below, so the barrier is at most one phase ahead
          // of the parity waited for here.
          ok = wait_bar(&sh->o_ready, (j - 1) & 1, sh, 33);
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

      // ---- P = exp2(s - m), row sum, P -> TMEM, over S or in columns of its own -------------
      // packed pairs: one FMA, two exponentials, one conversion and one add per two scores
      if (kOwnP && j > 0) {                          // the P V before has read its P (as good as always)
        ok = wait_bar(&sh->o_ready, (j - 1) & 1, sh, 33);
        if (!ok) break;
        tc_fence_after();
      }
      const float2 mul2 = make_float2(mul, mul), nm2 = make_float2(-m_safe, -m_safe);
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
    if (ok && nt > 0) ok = wait_bar(&sh->o_ready, (nt - 1) & 1, sh, 35);
    tc_fence_after();
    if (ok && sh->abort_flag == 0) {
      const float inv = l > 0.f ? (kDrop ? cfg.dropout_scale : 1.f) / l : 0.f;
      const bool row_ok = row < si.q_len;
      // The tile is staged over the Q tile, which no MMA reads any more, in the swizzled box layout and written by
      // the TMA unit as full rows; a packed tile that reaches past the end of its sequence is stored row by row
      // instead (the unit would write the neighbour's rows).
      const bool via_tma = (p.cu_seqlens_q == nullptr) || (m0 + kBM <= si.q_len);
      T* og = reinterpret_cast<T*>(p.o) + si.q_boff * p.o_stride[0] +
              (si.q_row0 + row) * p.o_stride[1] + (int64_t)h * p.o_stride[2];
#pragma unroll
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
            st_shared_v4(sw128_addr(sQ + (col / 64) * (kBM * 128), row_in_tile, (col % 64) / 8), v);
          } else if (row_ok) {
            *reinterpret_cast<uint4*>(og + cc * 32 + i) = v;
          }
        }
      }
      if (via_tma) {
        fence_proxy_async();
        asm volatile("bar.sync 1, 128;\n" ::: "memory");
        if (tid == 0) {
#pragma unroll
          for (int bx = 0; bx < D / 64; ++bx)
            tma_store_4d(&tmO, sQ + bx * (kBM * 128), bx * 64, h, (int)si.q_row0 + m0, (int)si.q_boff);
          tma_store_commit();
          tma_store_wait_read();
        }
      }
      if (row_ok && p.lse2 != nullptr)
        p.lse2[si.q_boff * p.lse_stride[0] + (si.q_row0 + row) * p.lse_stride[1] +
               (int64_t)h * p.lse_stride[2]] = l > 0.f ? m_used + log2f(l) : -INFINITY;
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 4) tmem_dealloc(tmem, 256);
  if (tid == 0) report_abort(sh->abort_flag, host_status);
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
  CUtensorMap tq, tk, tv, to;
  if (!map(&tq, a.q, a.q_stride, a.heads_q, q_rows) || !map(&tk, a.k, a.k_stride, a.heads_kv, k_rows) ||
      !map(&tv, a.v, a.v_stride, a.heads_kv, k_rows) || !map(&to, a.o, a.o_stride, a.heads_q, q_rows)) {
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
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmemBytes);
  if (e != cudaSuccess) {
    set_error("fwd_duo_sm100: cudaFuncSetAttribute(%d): %s", C::kSmemBytes, cudaGetErrorString(e));
    return FA_ERR_LAUNCH;
  }
  ScoreCfg cfg = plain;
  const dim3 grid = packed ? packed_grid<kBM>(a, cfg) : dense_grid(a, (a.seqlen_q + kBM - 1) / kBM, cfg);
  kern<<<grid, kThreads, C::kSmemBytes, st>>>(tq, tk, tv, to, a, cfg, host_wait_word(a.device));
  return check_launch("fwd_duo_sm100");
}

int fwd_duo_sm100(const fa_attn_args& a, const ScoreCfg& cfg, cudaStream_t st) {
  const bool bf = a.dtype == FA_BF16;
  if (a.head_dim == 64) return bf ? launch_duo<__nv_bfloat16, 64>(a, cfg, st) : launch_duo<__half, 64>(a, cfg, st);
  return bf ? launch_duo<__nv_bfloat16, 128>(a, cfg, st) : launch_duo<__half, 128>(a, cfg, st);
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
