// Sequences of a call, and the order in which the tiles of its rows are worked on: geometry, grids, items of a queue.
// Needs ScoreCfg and sm_count() (common.cuh includes it behind them) and nothing of a GPU but the warp votes, so that the order can be
// run on the CPU.
#pragma once

namespace fa {

struct SeqInfo {
  int q_len, k_len;
  int64_t q_row0, k_row0;  // first row of this sequence in the row dimension
  int64_t q_boff, k_boff;  // 1 for dense (multiply stride[0] by batch), 0 for packed
};

__device__ __forceinline__ SeqInfo seq_info(const fa_attn_args& p, int b) {
  SeqInfo s;
  if (p.cu_seqlens_q) {
    int q0 = p.cu_seqlens_q[b], q1 = p.cu_seqlens_q[b + 1];
    int k0 = p.cu_seqlens_k[b], k1 = p.cu_seqlens_k[b + 1];
    s.q_len = q1 - q0;
    s.k_len = k1 - k0;
    s.q_row0 = q0;
    s.k_row0 = k0;
    s.q_boff = 0;
    s.k_boff = 0;
  } else {
    s.q_len = p.seqlen_q;
    s.k_len = p.seqlen_k;
    s.q_row0 = 0;
    s.k_row0 = 0;
    s.q_boff = b;
    s.k_boff = b;
  }
  if (p.seqused_q) s.q_len = max(0, min(s.q_len, p.seqused_q[b]));
  if (p.seqused_k) s.k_len = max(0, min(s.k_len, p.seqused_k[b]));
  return s;
}

// Order in which the blocks (of rows, or of keys) of all units (batch entries x heads) are worked on: groups of units one
// after the other, within a group the first, heaviest block of every unit, then the second, and so on.  Unit by unit, the last
// units' heavy blocks come last and set the time of a launch; all units at once, what their blocks share does
// not stay in L2.  Measured where everything fits a group (before, after): 1 x 32 heads x 4001 tokens of 128 over 8, causal
// forward 153 -> 145 us, 2 x 16 x 1999 of 256 107 -> 89; 32 packed sequences of 256 to 4096 with a window: dK/dV 2990 -> 2290;
// backward, dK/dV: 6 x 8 x 802 of 128 47 -> 34 us, 1 x 16 x 2048 58 -> 42, dQ 40 -> 30.
__device__ __forceinline__ void block_of(int c, int blocks, int units, int group, int& unit, int& block) {
  const int first = c / (group * blocks) * group;
  const int n = min(group, units - first), r = c - first * blocks;
  block = r / n;
  unit = first + r % n;
}
// Units per group: groups of one size (a last group of one unit brings back its light blocks at the end: 1 x 16 heads x 8192 of
// 128, where 15 fitted, 277 -> 300 us by the order it should have gained from), as few as what their units read again and
// again allows.  Blocks of one size have no order to keep.  In packed batches groups also bring the blocks that lie outside their
// sequences together, where all SMs skip them at once.
inline int unit_group(const fa_attn_args& a, const ScoreCfg& cfg, int heads, int64_t bytes, int64_t limit) {
  const int64_t units = (int64_t)a.batch * heads;
  if (!cfg.causal || units <= 1) return 1;
  const int64_t groups = bytes > limit ? (bytes + limit - 1) / limit : 1;
  return (int)((units + groups - 1) / groups);
}

// Keys and values of a group: 32 MB.  Without groups, 16, 32 and 64 MB (us): 1 x 16 x 8192 of 128 277, 263, 264, 263;
// 8 x 16 x 2048 of 128 209, 194, 197, 190; 64 x 16 x 512 of 128 179, 174, 174, 181; 32 x 16 x 256 of 256 84, 82, 85, 89.
inline int fwd_unit_group(const fa_attn_args& a, const ScoreCfg& cfg) {
  const int64_t keys = a.cu_seqlens_q != nullptr ? a.total_k : (int64_t)a.batch * a.seqlen_k;
  return unit_group(a, cfg, a.heads_q, 4 * keys * a.heads_kv * a.head_dim, (int64_t)32 << 20);
}

// The same for a kernel with one CTA per block of a dense call: where the order does not matter (blocks of one size, or a
// CTA for each at once) the grid has three dimensions and unit_group is 0, which saves the divisions (0.3 us).
inline dim3 dense_grid(const fa_attn_args& a, int blocks, ScoreCfg& cfg) {
  const int64_t all = (int64_t)blocks * a.heads_q * a.batch;
  cfg.unit_group = blocks == 1 ? 1 : fwd_unit_group(a, cfg);
  if ((cfg.unit_group == 1 || all <= sm_count(a.device)) && a.heads_q <= 65535 && a.batch <= 65535) {
    cfg.unit_group = 0;
    return dim3(blocks, a.heads_q, a.batch);
  }
  return dim3((unsigned)all);
}
__device__ __forceinline__ void dense_block(const fa_attn_args& p, const ScoreCfg& cfg, int blocks, int& b, int& h, int& block) {
  if (cfg.unit_group == 0) {
    block = blockIdx.x;
    h = blockIdx.y;
    b = blockIdx.z;
  } else {
    int unit;
    block_of(blockIdx.x, blocks, p.heads_q * p.batch, cfg.unit_group, unit, block);
    h = unit % p.heads_q;
    b = unit / p.heads_q;
  }
}

// Packed forwards have a CTA per tile that their sequences can have together, not per tile of the longest one: they
// differ in length, and a CTA without a tile still waits for an SM to itself.  Sequence b starts at entry cu_seqlens_q[b] / kBM + b
// of the list of tiles, which leaves it at least as many entries as it has tiles; so a CTA finds its sequence by a search in
// cu_seqlens_q, 32 samples at a time.  Where the longest sequence times their number gives no more entries (many short
// sequences) the grid has three dimensions and there is nothing to search, nor to divide (4096 sequences of 16 to 128 tokens, 8
// heads of 256: 2090 -> 2063 us).
// (A scan that counted the tiles of all sequences before, in every CTA: 4096 of 16 to 128, 8 heads of 128, 5700 us for 984;
// 1024 of 17 to 512 1403 for 833; 24 to 64 sequences within 3 %.)
template <int kBM> inline dim3 packed_grid(const fa_attn_args& a, ScoreCfg& cfg) {
  const int per = (a.seqlen_q + kBM - 1) / kBM;
  const int64_t entries = a.total_q / kBM + (int64_t)a.batch;
  cfg.packed_list = !((int64_t)per * a.batch <= entries && a.heads_q <= 65535 && a.batch <= 65535);
  return cfg.packed_list ? dim3((unsigned)(entries * a.heads_q)) : dim3(per, a.heads_q, a.batch);
}
// Head, sequence and tile of entry (t, h) of the list, or of tile t, head h, sequence b without one (with a causal mask the
// last, heaviest tile of a sequence comes first).  Called by whole warps; false when there is no such tile.
template <int kBM>
__device__ __forceinline__ bool packed_entry(const fa_attn_args& p, const ScoreCfg& cfg, int lane, int t, int& b, SeqInfo& si, int& mt) {
  if (cfg.packed_list) {
    auto first = [&](int s) { return p.cu_seqlens_q[s] / kBM + s; };
    b = 0;
    for (int n = p.batch; n > 1;) {                  // the last sequence of [b, b + n) that starts at t or before
      const int step = (n + 31) / 32, at = lane * step;
      const unsigned before = __ballot_sync(0xffffffffu, at < n && first(b + at) <= t);
      const int skip = before != 0u ? (31 - __clz(before)) * step : 0;
      b += skip;
      n = min(step, n - skip);
    }
    t -= first(b);
  }
  si = seq_info(p, b);
  const int tiles = (min(si.q_len, p.seqlen_q) + kBM - 1) / kBM;
  mt = cfg.causal ? tiles - 1 - t : t;
  return t >= 0 && t < tiles;
}
// The tile of a CTA of packed_grid().
template <int kBM>
__device__ __forceinline__ bool packed_tile(const fa_attn_args& p, const ScoreCfg& cfg, int lane, int& h, int& b, SeqInfo& si, int& mt) {
  int t = blockIdx.x;
  if (cfg.packed_list) {
    h = t % p.heads_q;                               // the heads of a tile next to one another
    t /= p.heads_q;
  } else {
    h = blockIdx.y;
    b = blockIdx.z;
  }
  return packed_entry<kBM>(p, cfg, lane, t, b, si, mt);
}
// The c-th of its blocks, for kernels that take them from a queue.  With a mask whose tiles see different numbers of keys the order
// is that of block_of(): the heaviest tiles of 32 sequences (one per lane), then the second, ..., for `by_weight` heads at a time
// (0: not so), so that what the CTAs read together stays in L2.  Sequence by sequence, heavy tiles of the last one set the time of a launch,
// and items of different lengths in turn bring the two CTAs of an SM into each other's exponentials (us, before -> after): 14 sequences of 461, 32
// heads of 64 67 -> 52, 24 prompts of 17 to 2048, 32 heads over 8 of 128 290 -> 276, 111 of 394 with a window of 1024 and 128 273 -> 215.
constexpr int kPackedLevels = 64;      // tiles of the longest sequence; the search looks at one level after the other
inline int packed_by_weight(const fa_attn_args& a, const ScoreCfg& cfg, int bm) {
  if (!(cfg.causal || cfg.wl >= 0 || cfg.wr >= 0) || (a.seqlen_q + bm - 1) / bm > kPackedLevels) return 0;
  int kv = a.heads_kv;                 // keys and values of the heads: 32 MB, see fwd_unit_group()
  while (kv > 1 && (a.heads_kv % kv != 0 || (int64_t)4 * a.total_k * kv * a.head_dim > (int64_t)32 << 20)) --kv;
  return kv * (a.heads_q / a.heads_kv);
}
template <int kBM>
__device__ __forceinline__ bool packed_tile_of(const fa_attn_args& p, const ScoreCfg& cfg, int by_weight, int c, int lane,
                                               int& h, int& b, SeqInfo& si, int& mt) {
  auto first = [&](int s) { return p.cu_seqlens_q[s] / kBM + s; };       // entry of the list, see above
  if (by_weight > 0) {
    h = c % by_weight;
    c /= by_weight;
    const int entries = p.total_q / kBM + p.batch;
    h += c / entries * by_weight;
    c %= entries;
    int b0 = 0;                                      // first of the 32 sequences that entry c belongs to
    for (int n = (p.batch + 31) / 32; n > 1;) {
      const int step = (n + 31) / 32, at = lane * step;
      const unsigned before = __ballot_sync(0xffffffffu, at < n && first(32 * (b0 + at)) <= c);
      const int skip = before != 0u ? (31 - __clz(before)) * step : 0;
      b0 += skip;
      n = min(step, n - skip);
    }
    b0 *= 32;
    c -= first(b0);
    if (c < 0) return false;                         // rows before the first sequence
    int tiles = 0;
    if (b0 + lane < p.batch) {
      si = seq_info(p, b0 + lane);
      tiles = (min(si.q_len, p.seqlen_q) + kBM - 1) / kBM;
    }
    const int most = __reduce_max_sync(0xffffffffu, tiles);
    const bool down = cfg.causal || cfg.wr >= 0;     // the last tiles see most keys
    unsigned have = 0u;                              // sequences with a tile mt
    int i = 0;
    for (; i < most; ++i) {
      mt = down ? most - 1 - i : i;
      have = __ballot_sync(0xffffffffu, tiles > mt);
      if (c < __popc(have)) break;
      c -= __popc(have);
    }
    if (i == most) return false;                     // (the list has up to 32 entries more than these sequences have tiles)
    const unsigned mine = __ballot_sync(0xffffffffu, (have >> lane & 1u) != 0u && __popc(have & ((1u << lane) - 1u)) == c);
    b = b0 + __ffs(mine) - 1;                        // the c-th of them
    si = seq_info(p, b);
    return true;
  }
  int t = c;
  if (cfg.packed_list) {
    h = t % p.heads_q;
    t /= p.heads_q;
  } else {
    const int per = (p.seqlen_q + kBM - 1) / kBM;
    t = c % per;
    c /= per;
    h = c % p.heads_q;
    b = c / p.heads_q;
  }
  return packed_entry<kBM>(p, cfg, lane, t, b, si, mt);
}

// The same for kernels whose CTAs take candidates by number, dense calls included: how many there are, and the c-th (whole warps; false where it is
// no tile).  cfg and by_weight are set for the launch.
template <int kBM> inline int64_t item_candidates(const fa_attn_args& a, ScoreCfg& cfg, int& by_weight) {
  by_weight = 0;
  if (a.cu_seqlens_q != nullptr) {
    const dim3 list = packed_grid<kBM>(a, cfg);
    by_weight = packed_by_weight(a, cfg, kBM);
    if (by_weight > 0) return (a.total_q / kBM + (int64_t)a.batch) * a.heads_q;
    return (int64_t)list.x * list.y * list.z;
  }
  const int blocks = (a.seqlen_q + kBM - 1) / kBM;
  // Windows have the order of a causal mask: tiles that see equally many keys one behind the other.  The two CTAs of an SM then stay
  // out of phase; with items of one to four tiles in turn they run into each other's exponentials (111 x 16 heads x 512 of 64, window of
  // 1024 and 0: 230 -> 172 us).
  ScoreCfg order = cfg;
  order.causal = cfg.causal || cfg.wl >= 0 || cfg.wr >= 0;
  cfg.unit_group = blocks == 1 ? 1 : fwd_unit_group(a, order);
  return (int64_t)blocks * a.heads_q * a.batch;
}
template <int kBM>
__device__ __forceinline__ bool item_tile(const fa_attn_args& p, const ScoreCfg& cfg, int by_weight, int c, int lane,
                                          int& h, int& b, SeqInfo& si, int& mt) {
  if (p.cu_seqlens_q != nullptr) {
    if (!packed_tile_of<kBM>(p, cfg, by_weight, c, lane, h, b, si, mt)) return false;
  } else {
    const int mtiles = (p.seqlen_q + kBM - 1) / kBM;
    int unit;
    block_of(c, mtiles, p.heads_q * p.batch, cfg.unit_group, unit, mt);
    h = unit % p.heads_q;
    b = unit / p.heads_q;
    if (cfg.causal || cfg.wr >= 0) mt = mtiles - 1 - mt;   // heavy tiles first
    si = seq_info(p, b);
  }
  return mt * kBM < si.q_len;
}

}  // namespace fa
