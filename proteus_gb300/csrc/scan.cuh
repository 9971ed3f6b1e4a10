// Exclusive prefix sums by one CTA: the offsets of a small table, used by the
// partitioner and the partitioned operators.
#pragma once
#include "gbj_internal.cuh"

namespace gbjd {

// Exclusive sum of x over a CTA of 1024 threads; `warps` is 32 words of shared
// memory.  Every thread calls it; it may be called again at once.
__device__ __forceinline__ uint64_t cta_scan(uint64_t x, uint64_t *warps) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint64_t incl = x;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint64_t y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  __syncthreads();
  if (lane == 31) warps[warp] = incl;
  __syncthreads();
  uint64_t w = warps[lane], before = lane < warp ? w : 0;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) before += __shfl_xor_sync(0xffffffffu, before, o);
  return before + incl - x;
}

// off[i] = f(0) + .. + f(i - 1) for i <= n, by one CTA of 1024 threads: a
// table of up to some ten thousand entries takes one launch instead of the
// three to five of a multi-level scan.
template <typename F>
__device__ __forceinline__ void cta_offsets(uint32_t n, F f, uint64_t *__restrict__ off, uint64_t *warps) {
  const uint32_t per = (n + 1023) / 1024, lo = min(n, threadIdx.x * per), hi = min(n, lo + per);
  uint64_t sum = 0;
  for (uint32_t i = lo; i < hi; ++i) sum += f(i);
  uint64_t run = cta_scan(sum, warps);
  for (uint32_t i = lo; i < hi; ++i) {
    const uint64_t x = f(i);
    off[i] = run;
    run += x;
  }
  if (lo < n && hi == n) off[n] = run;
}

}  // namespace gbjd
