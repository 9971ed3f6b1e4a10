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
// three to five of a multi-level scan.  4096 entries a round, the next
// round's read while this one is summed (16,384 entries: 35 us when a thread
// read its sixteen neighbours one after the other, 21 us now).
template <typename F>
__device__ __forceinline__ void cta_offsets(uint32_t n, F f, uint64_t *__restrict__ off, uint64_t *warps) {
  __shared__ uint64_t s_total;
  uint64_t x[4], carry = 0;
  auto read = [&](uint32_t base) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t i = base + 4 * threadIdx.x + j;
      x[j] = i < n ? f(i) : 0;
    }
  };
  read(0);
  for (uint32_t base = 0; base < n; base += 4096) {
    uint64_t v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = x[j];
    if (base + 4096 < n) read(base + 4096);
    const uint64_t sum = v[0] + v[1] + v[2] + v[3];
    uint64_t run = carry + cta_scan(sum, warps);
    if (threadIdx.x == 1023) s_total = run + sum;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t i = base + 4 * threadIdx.x + j;
      if (i < n) off[i] = run;
      run += v[j];
    }
    __syncthreads();
    carry = s_total;
  }
  if (threadIdx.x == 0) off[n] = carry;
}

}  // namespace gbjd
