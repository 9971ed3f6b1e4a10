// Ordered row compaction shared by the range select and the bloom-filter
// probe: the positions of rows that pass a predicate, ascending, in one pass
// over the column.
//
// A CTA tests a tile of 8192 rows (four 16-byte loads per thread) and takes
// its place in the output from the counts that earlier tiles have published
// (tiles are taken by ticket, so all of them have started), 32 of them at a
// time; the last tile writes the total.
//
// What bounds it is HBM: 4 B a row and 4 B a passing row.  Measured on GB300,
// 2^24 rows of which a tenth pass: 47 us (a count, a multi-level scan, a write
// that re-read the column and a total before: 147 us in six launches).
#pragma once
#include "gbj_internal.cuh"

namespace gbj {

constexpr int kCompactThreads = 512;
constexpr int kCompactWarps = kCompactThreads / 32;
constexpr uint32_t kCompactTile = 16 * kCompactThreads;

// Published per tile: {rows that pass, 2 flag bits}.
enum : unsigned long long { kTileOwn = 1, kTileUpTo = 2, kTileGaveUp = 3 };

struct CompactState {
  uint32_t ticket, pad;
  unsigned long long tile[1];  // [tiles]
};

// Pred: `col` (the int32 column) and test(value).  vec: col is 16-byte aligned.
template <typename Pred>
__global__ void __launch_bounds__(kCompactThreads)
    k_compact(Pred pred, uint32_t n, bool vec, CompactState *st, int32_t *__restrict__ out,
              uint64_t *__restrict__ count, uint32_t *dev_status) {
  __shared__ uint32_t s_tile, s_ok, s_off[4 * kCompactWarps];
  __shared__ uint64_t s_before;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) s_tile = atomicAdd(&st->ticket, 1u);
  __syncthreads();
  const uint32_t tile = s_tile, base = tile * kCompactTile + 4 * threadIdx.x;
  // rows base + 4 j * threads .. + 3: bit b of pass[j] is row b of load j
  int4 v[4];
  uint32_t pass[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const uint32_t i = base + 4 * j * kCompactThreads;
    if (vec && i + 4 <= n) {
      v[j] = __ldcs(reinterpret_cast<const int4 *>(pred.col + i));
    } else {
      v[j].x = i < n ? pred.col[i] : 0;
      v[j].y = i + 1 < n ? pred.col[i + 1] : 0;
      v[j].z = i + 2 < n ? pred.col[i + 2] : 0;
      v[j].w = i + 3 < n ? pred.col[i + 3] : 0;
    }
  }
  uint32_t own = 0;  // rows that pass, 8 bits per load (a warp's total is at most 128)
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const uint32_t i = base + 4 * j * kCompactThreads;
    pass[j] = (uint32_t)(i < n && pred.test(v[j].x)) | ((uint32_t)(i + 1 < n && pred.test(v[j].y)) << 1) |
              ((uint32_t)(i + 2 < n && pred.test(v[j].z)) << 2) | ((uint32_t)(i + 3 < n && pred.test(v[j].w)) << 3);
    own |= (uint32_t)__popc(pass[j]) << (8 * j);
  }
  uint32_t incl = own;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) {
#pragma unroll
    for (int j = 0; j < 4; ++j) s_off[j * kCompactWarps + warp] = (incl >> (8 * j)) & 0xffu;
  }
  __syncthreads();
  if (warp == 0) {
    // the 64 (load, warp) counts in row order, two a lane
    const uint32_t a = s_off[2 * lane], b = s_off[2 * lane + 1];
    uint32_t run = a + b;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, run, o);
      if (lane >= o) run += y;
    }
    s_off[2 * lane] = run - a - b;
    s_off[2 * lane + 1] = run - b;
    const uint32_t total = __shfl_sync(0xffffffffu, run, 31);
    volatile unsigned long long *tiles = st->tile;
    if (lane == 0) tiles[tile] = ((unsigned long long)total << 2) | (tile ? kTileOwn : kTileUpTo);
    uint64_t before = 0;
    bool ok = true;
    uint32_t spin = 0;
    for (uint32_t left = tile; left > 0 && ok;) {
      const unsigned long long w = lane < left ? tiles[left - 1 - lane] : kTileUpTo;
      const uint32_t f = (uint32_t)(w & 3);
      const unsigned up = __ballot_sync(0xffffffffu, f == kTileUpTo), none = __ballot_sync(0xffffffffu, f == 0);
      ok = __ballot_sync(0xffffffffu, f == kTileGaveUp) == 0;
      const uint32_t to = up ? __ffs(up) : 32, open = none ? __ffs(none) - 1 : 32;  // usable: the first min(to, open)
      uint64_t x = (uint32_t)lane < min(to, open) ? w >> 2 : 0;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
      before += x;
      if (up && to <= open) break;
      left -= open;
      if (open == 0 && ++spin == kSpinLimit) ok = false;
    }
    if (lane == 0) {
      if (tile) tiles[tile] = ok ? ((before + total) << 2) | kTileUpTo : kTileGaveUp;
      if (!ok) gbjd::latch(dev_status, GBJ_DEV_TIMEOUT);
      s_ok = ok;
      s_before = before;
      if (ok && tile == gridDim.x - 1) *count = before + total;
    }
  }
  __syncthreads();
  if (!s_ok) return;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    uint64_t pos = s_before + s_off[j * kCompactWarps + warp] + (((incl - own) >> (8 * j)) & 0xffu);
    const uint32_t i = base + 4 * j * kCompactThreads;
#pragma unroll
    for (int b = 0; b < 4; ++b)
      if ((pass[j] >> b) & 1u) out[pos++] = (int32_t)(i + b);
  }
}

// Writes the passing row ids of [0, n), n < 2^31, to d_rows_out (ascending)
// and their number to *d_count.
template <typename Pred>
int compact_rows(gbj_ctx *ctx, Pred pred, uint64_t n, int32_t *d_rows_out, uint64_t *d_count,
                 cudaStream_t s) {
  if (n == 0) {
    GBJ_CHECK_CUDA(ctx, cudaMemsetAsync(d_count, 0, sizeof(uint64_t), s));
    return GBJ_OK;
  }
  const uint64_t ntiles = (n + kCompactTile - 1) / kCompactTile;
  const uint64_t bytes = sizeof(CompactState) + ntiles * sizeof(unsigned long long);
  Scratch scratch(ctx, s);
  char *mem;
  GBJ_TRY(scratch.get(bytes, &mem));
  GBJ_CHECK_CUDA(ctx, cudaMemsetAsync(mem, 0, bytes, s));
  const bool vec = reinterpret_cast<uintptr_t>(pred.col) % 16 == 0;
  k_compact<<<(unsigned)ntiles, kCompactThreads, 0, s>>>(pred, (uint32_t)n, vec, reinterpret_cast<CompactState *>(mem),
                                                         d_rows_out, d_count, ctx->d_status);
  return after_launch(ctx, "k_compact", s);
}

}  // namespace gbj
