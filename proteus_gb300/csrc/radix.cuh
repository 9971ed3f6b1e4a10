// Radix partitioning shared by the partitioned join and group-by.
#pragma once
#include "auto_plan.h"
#include "gbj_internal.cuh"

namespace gbj {

// Partitions n (key, value) tuples on digit = (f(key) >> shift) & (2^bits-1)
// into a contiguous, partition-major output.  vals == nullptr carries the
// row position.  Output either AoS (out_pairs != nullptr, int2 {key, val})
// or SoA (out_keys / out_vals).  offsets gets 2^bits + 1 entries.
// One histogram pass, then one pass per digit group; tuples keep no
// particular order inside a partition.  passes: 0 = one pass up to 12 bits,
// two above (two from 9 bits on where the output columns overlap the input);
// 1 = one pass (bits <= 8); 2 = two passes (bits >= 2).
// hash_out (GBJ_DIGIT_HASH, AoS output only): each tuple leaves with
// fmix32(key) in place of the key, as the partitioned join consumes them.
int partition_tuples(gbj_ctx *ctx, const int32_t *keys, const int32_t *vals,
                     uint64_t n, int digit, int shift, int bits,
                     int2 *out_pairs, int32_t *out_keys, int32_t *out_vals,
                     uint64_t *offsets, cudaStream_t s, int passes = 0,
                     bool hash_out = false);

}  // namespace gbj

namespace gbjd {

// Partition of work item `item`: largest p with item_off[p] <= item, where
// item_off[0] = 0 <= item < item_off[P] = total.  Starts from the
// proportional guess and gallops, so the common case (about one item per
// partition) costs two or three dependent loads.
__device__ __forceinline__ uint32_t item_partition(const uint64_t *__restrict__ off, uint32_t P,
                                                   uint64_t total, uint64_t item) {
  uint32_t lo = (uint32_t)((item * (uint64_t)P) / total);
  if (lo >= P) lo = P - 1;
  uint32_t hi;
  if (off[lo] <= item) {
    uint32_t step = 1;
    hi = lo + 1;
    while (hi < P && off[hi] <= item) {
      lo = hi;
      step <<= 1;
      hi = lo + step < P ? lo + step : P;
    }
  } else {
    uint32_t step = 1;
    hi = lo;
    for (;;) {  // off[hi] > item; off[0] = 0 <= item ends the walk
      lo = hi > step ? hi - step : 0;
      if (off[lo] <= item) break;
      hi = lo;
      step <<= 1;
    }
  }
  while (hi - lo > 1) {  // off[lo] <= item < off[hi]
    const uint32_t mid = (lo + hi) >> 1;
    if (off[mid] <= item) lo = mid; else hi = mid;
  }
  return lo;
}

}  // namespace gbjd
