// What the cache kernels know about a call beyond the attention itself.
#pragma once
#include <stdint.h>

namespace fa {

struct CacheGeo {
  const int* seqlens;      // tokens in the cache before the call (null: not a cache call)
  const int* table;        // block table, or null
  const int* batch_idx;    // cache row of a sequence, or null
  const int* leftpad;      // or null
  int table_stride;
  int page_size;           // rows of a page (of a sequence when contiguous)
  int page_log2;           // of page_size, or -1
  int box_rows;            // rows of one TMA box: min(page_size, 128)
  int n_new;               // tokens appended by the call
  int tokens;              // query tokens of a sequence
  int pack_log2;           // query heads packed into the rows of a tile
  int parts;               // pieces the keys of a sequence are cut into, at most
  int capacity;            // keys a sequence can hold
  float* ws;               // pieces: fp32 outputs, then their base-2 LSEs
  uint32_t* counters;      // per unit, zero
  const uint32_t* bad;     // set by the value checks: do nothing
};

}  // namespace fa
