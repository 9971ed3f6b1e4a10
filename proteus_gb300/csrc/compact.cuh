// Ordered row compaction shared by the range select and the bloom-filter
// probe: the positions of rows that pass a predicate, ascending, in one pass
// over the column.
//
// A CTA tests a tile of 8192 rows (four 16-byte loads per thread) and takes
// its place in the output from what earlier tiles have published (tiles are
// taken by ticket, so all of them have started): the sums of the groups of 32
// tiles before its own, 32 of them at a time back to one whose end is known,
// and the counts of the tiles before it in its group.  The last tile writes
// the total.
//
// What bounds it is the way from a tile's start to its place: ticket, rows and
// two or three reads of others' words, one after the other.  With tiles alone,
// 32 at a time, some 600 of them in flight made that twenty reads, and reading
// 64 or 256 at a time only more of them (2^26 rows: 145 us, 155, 246).
// Measured on GB300, a tenth of the rows passing, the column not in L2: 2^24
// rows 37 us (47 without groups; 147 in six launches, with a count, a
// multi-level scan, a write that re-read the column and a total), 2^26 rows
// 100 us (145).
#pragma once
#include "gbj_internal.cuh"

namespace gbj {

constexpr int kCompactThreads = 512;
constexpr int kCompactWarps = kCompactThreads / 32;
constexpr uint32_t kCompactTile = 16 * kCompactThreads;

// Words that tiles publish: {rows that pass << 2, 2 flag bits}.
enum : unsigned long long { kWordOwn = 1, kWordUpTo = 2, kWordGaveUp = 3 };

constexpr uint32_t kGroup = 32;  // tiles

struct CompactGroup {
  unsigned long long own;   // {rows that pass in its tiles, tiles that have added theirs << 32}
  unsigned long long upto;  // rows that pass up to the group's end, a word of its last tile
};

// A ticket, then the groups, then a word for each tile.
struct CompactState {
  uint32_t ticket, pad;
  CompactGroup group[1];
};

// Pred: `col` (the int32 column) and test(value).  vec: col is 16-byte aligned.
template <typename Pred>
__global__ void __launch_bounds__(kCompactThreads)
    k_compact(Pred pred, uint32_t n, bool vec, CompactState *st, unsigned long long *words, int32_t *__restrict__ out,
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
    const uint32_t g = tile / kGroup, in_group = tile % kGroup;
    volatile unsigned long long *tiles = words;
    volatile CompactGroup *groups = st->group;
    if (lane == 0) {
      tiles[tile] = ((unsigned long long)total << 2) | kWordOwn;
      atomicAdd(&st->group[g].own, (unsigned long long)total | (1ull << 32));
    }
    // all counts together are below 2^31
    uint32_t before = 0, spin = 0;
    bool ok = true;
    // the groups before this one, 32 at a time, back to one whose end is known
    for (uint32_t left = g; left > 0 && ok;) {
      unsigned long long up = kWordUpTo, own = 0;
      if ((uint32_t)lane < left) {
        up = groups[left - 1 - lane].upto;
        own = groups[left - 1 - lane].own;
      }
      const unsigned ends = __ballot_sync(0xffffffffu, (up & 3) == kWordUpTo);
      const unsigned open = __ballot_sync(0xffffffffu, (up & 3) == 0 && (uint32_t)(own >> 32) < kGroup);
      ok = __ballot_sync(0xffffffffu, (up & 3) == kWordGaveUp) == 0;
      const uint32_t to = ends ? __ffs(ends) : 32, usable = min(to, open ? (uint32_t)__ffs(open) - 1 : 32u);
      const uint32_t x = (up & 3) == kWordUpTo ? (uint32_t)(up >> 2) : (uint32_t)own;
      before += __reduce_add_sync(0xffffffffu, (uint32_t)lane < usable ? x : 0u);
      if (ends && usable == to) break;
      left -= usable;
      if (usable == 0 && ++spin == kSpinLimit) ok = false;
    }
    // the tiles before this one in its group
    for (;;) {
      const unsigned long long w = (uint32_t)lane < in_group ? tiles[g * kGroup + lane] : kWordOwn;
      ok &= __ballot_sync(0xffffffffu, (w & 3) == kWordGaveUp) == 0;
      if (!ok) break;
      if (__ballot_sync(0xffffffffu, (w & 3) == 0) == 0) {
        before += __reduce_add_sync(0xffffffffu, (uint32_t)(w >> 2));
        break;
      }
      if (++spin >= kSpinLimit) ok = false;
    }
    if (lane == 0) {
      if (!ok) {
        tiles[tile] = kWordGaveUp;
        gbjd::latch(dev_status, GBJ_DEV_TIMEOUT);
      }
      if (in_group == kGroup - 1)
        groups[g].upto = ok ? ((unsigned long long)(before + total) << 2) | kWordUpTo : kWordGaveUp;
      s_ok = ok;
      s_before = before;
      if (ok && tile == gridDim.x - 1) *count = (uint64_t)before + total;
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
  const uint64_t ngroups = (ntiles + kGroup - 1) / kGroup;
  const uint64_t head = sizeof(CompactState) + ngroups * sizeof(CompactGroup);
  const uint64_t bytes = head + ntiles * sizeof(unsigned long long);
  Scratch scratch(ctx, s);
  char *mem;
  GBJ_TRY(scratch.get(bytes, &mem));
  GBJ_CHECK_CUDA(ctx, cudaMemsetAsync(mem, 0, bytes, s));
  const bool vec = reinterpret_cast<uintptr_t>(pred.col) % 16 == 0;
  k_compact<<<(unsigned)ntiles, kCompactThreads, 0, s>>>(pred, (uint32_t)n, vec, reinterpret_cast<CompactState *>(mem),
                                                         reinterpret_cast<unsigned long long *>(mem + head),
                                                         d_rows_out, d_count, ctx->d_status);
  return after_launch(ctx, "k_compact", s);
}

}  // namespace gbj
