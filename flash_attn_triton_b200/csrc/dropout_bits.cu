// The dropout mask of a dense call as bits, for the tcgen05 kernels.
//
// The random stream depends on (query row, key) alone: every batch entry and head of a call has the same
// mask.  The mma.sync kernels draw it per element of every head, in the forward and in both backward
// kernels (ten Philox rounds, about fifty integer instructions per score, on warps whose scores cost ten);
// here it is drawn once per call and read as one bit per score.
//
// Two copies: bits of a row of keys, for kernels whose threads own a query row (forward, dQ), and bits of a
// column of queries, for the dK/dV kernel, whose threads own a key.  Both are padded to tiles of 128, so a
// kernel reads the 64 or 128 bits of its part of a tile as one aligned load without a bounds test.
// A CTA draws a block of 32 x 32, eight rows per warp: lane = key, and a vote per row gives the row's word while each
// lane collects its own column (a warp for the whole block left the chip idle: 6 us for 512 x 512).
//
// Bound: integer issue, 50 instructions per 1 / (batch * heads) of a score.  Measured on B200, forward + backward
// of 8 x 512 tokens, 16 heads of 64, without a mask: 834 -> 117 us with the three attention kernels on tcgen05
// and the bits drawn twice (once per direction: keeping them would hold memory per layer).
#include "common.cuh"

namespace fa {

namespace {
constexpr int kTile = 128, kBlock = 32, kWarps = 4, kRows = kBlock / kWarps;
}

__global__ void __launch_bounds__(kWarps * 32)
dropout_bits_kernel(const ScoreCfg cfg, uint32_t* __restrict__ rows, uint32_t* __restrict__ cols, const int row_blocks,
                    const int col_blocks, const int off) {
  __shared__ uint32_t part[kWarps][kBlock];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int rb = (int)(blockIdx.x / (unsigned)col_blocks), cb = (int)(blockIdx.x % (unsigned)col_blocks);
  // no row of the block sees a key of it: the kernels mask those scores whatever the bits say
  if (cfg.causal && cb * kBlock > rb * kBlock + kBlock - 1 + off) return;
  const int row0 = rb * kBlock + warp * kRows, col = cb * kBlock + lane;
  uint32_t row_word = 0u, col_bits = 0u;
#pragma unroll
  for (int r = 0; r < kRows; ++r) {
    const bool keep = dropout_keep(cfg, 0u, row0 + r, col);
    const uint32_t w = __ballot_sync(0xffffffffu, keep);
    if (r == lane) row_word = w;
    col_bits |= (keep ? 1u : 0u) << (warp * kRows + r);
  }
  if (lane < kRows) rows[(int64_t)(row0 + lane) * col_blocks + cb] = row_word;
  part[warp][lane] = col_bits;
  __syncthreads();
  if (warp == 0) cols[(int64_t)col * row_blocks + rb] = part[0][lane] | part[1][lane] | part[2][lane] | part[3][lane];
}

// Words of ONE copy of the mask of a rows x keys problem.
int64_t dropout_bits_words(int seqlen_q, int seqlen_k) {
  const int64_t m = (seqlen_q + kTile - 1) / kTile, n = (seqlen_k + kTile - 1) / kTile;
  return m * n * (kTile * kTile / 32);
}

int dropout_bits(const fa_attn_args& a, const ScoreCfg& cfg, uint32_t* bits, cudaStream_t st) {
  const int rb = (a.seqlen_q + kTile - 1) / kTile * (kTile / kBlock), cb = (a.seqlen_k + kTile - 1) / kTile * (kTile / kBlock);
  dropout_bits_kernel<<<(unsigned)rb * (unsigned)cb, kWarps * 32, 0, st>>>(
      cfg, bits, bits + dropout_bits_words(a.seqlen_q, a.seqlen_k), rb, cb, a.q_pos_offset);
  return check_launch("dropout_bits");
}

}  // namespace fa
