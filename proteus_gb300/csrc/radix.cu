// Radix partitioning and the partitioned (radix) hash join.
//
// Stands in for the GPU radix join of the reference: HashPartitioner +
// build_partitions (core/olap/lib/operators/gpu/
// gpu-partitioned-hash-join-chained.cpp:249-404,
// gpu-partitioned-hash-join-chained-helpers.cpp:243-481) followed by the
// per-partition shared-memory build/probe loop of
// GpuPartitionedHashJoinChained (gpu-partitioned-hash-join-chained.cpp:
// 612-1586), and for the CPU RJStepwise / partitionHT path
// (core/platform/lib/util/radix/joins/radix-join.cpp:253-375).  Like the
// reference's GPU partitioner it uses two passes for wide fan-outs (there
// 7 + 6 bits); each pass here is a tile sort rather than bucket chains.
//
// GB300 layout:
//  * a histogram kernel counts the final partition ids (<= 2^15) once;
//  * each pass (<= 8 digit bits) sorts 4096-tuple tiles by digit in shared
//    memory (one histogram row per warp gives every tuple its rank), takes
//    one output range per digit with a single global atomic, and writes the
//    tile digit-run by digit-run, so stores are coalesced and at most 256
//    output regions are open per pass (the first pass of a 2^14 fan-out
//    writes 128 regions; the second writes inside one 32 MB bucket).  The
//    pass is software-pipelined: a CTA issues the next tile's loads as soon
//    as the current tile sits in shared memory, and the output-range atomic
//    is in flight while the tile is scattered on chip.  Fan-outs of 2^9 to
//    2^12 take one pass with larger tiles (k_wide_pass);
//  * radix bits are chosen so the largest build partition fits an on-chip
//    table of kRMax tuples (a 2^27-row side: 16384 partitions of 8192 +- 90
//    tuples) and every SM gets work;
//  * the join kernel is persistent: CTAs pull work items (partition, build
//    chunk, probe chunk) from an atomic counter, so a skewed probe partition
//    (Zipf keys) is spread over many SMs.  The on-chip table stores keys and
//    values in two arrays; a probe reads four keys per 16-byte shared load
//    and resolves match / empty with bit masks, so nearly every probe is one
//    load.  The partition that INT32_MIN (the empty marker) hashes to uses
//    an index table instead.
#include <algorithm>

#include "auto_plan.h"
#include "gbj_internal.cuh"
#include "radix.cuh"
#include "scan.cuh"
#include "tma.cuh"

using namespace gbj;

namespace {

// Tile shapes of the partition passes: 0 = 2048 tuples x 256 threads (4
// CTAs per SM), for passes of up to 7 digit bits with 8-byte pair output;
// 1 = 4096 x 512 (2 CTAs per SM), for 8-bit passes and 4-byte column
// output, whose digit runs would be too short in a smaller tile.  Measured
// on GB300 (radix join, R 2^27, S 2^29, 14 bits; ms of tile passes per 60
// launches): 2048 x 256 66.0, 3072 x 256 68.1, 4096 x 512 70.1, 4096 x 256
// 80.7, 2048 x 512 85.0, 4096 x 1024 95.6, 1024 x 256 102.4; the group-by's
// 8-bit column passes ran 60 % longer with the small tile.
template <int kSh>
struct TileShape {
  static constexpr int tile = kSh == 0 ? 2048 : 4096;
  static constexpr int threads = kSh == 0 ? 256 : 512;  // >= 256: one thread per digit in the scans
  static constexpr int per = tile / threads;            // tuples per thread
  static constexpr int warps = threads / 32;
  static constexpr int ctas = 1024 / threads;  // CTAs per SM (64 registers per thread)
};
constexpr int kMaxDigits = 256;      // <= 8 digit bits per pass
#ifndef GBJ_TILE_TMA
#define GBJ_TILE_TMA 0
#endif
// Tile passes load through bulk copies when set.  Measured on GB300 (radix
// join, R 2^27, S 2^29, 14 bits): 77.3 ms of tile passes per 60 launches with
// bulk copies against 70.0 ms through registers -- the copies add a shared
// read of every tuple to a kernel bound by its shared-memory pipe, and the
// pair passes have only one 32 KB stage -- so registers are the default.
constexpr bool kTileTma = GBJ_TILE_TMA;
constexpr int32_t kEmpty = INT32_MIN;

// Digit functions: of the key itself (GBJ_DIGIT_KEY), of fmix32(key)
// (GBJ_DIGIT_HASH), or of a tuple word that already holds fmix32(key)
// (kDigitPre: the partitioned join's tuples).
constexpr int kDigitPre = 2;

template <int kDigit>
__device__ __forceinline__ uint32_t digit_of(int32_t key, int shift, uint32_t mask) {
  const uint32_t v = kDigit == GBJ_DIGIT_HASH ? gbjd::fmix32((uint32_t)key) : (uint32_t)key;
  return (v >> shift) & mask;
}

// What the passes need, written by the histogram's last CTA: offsets of the
// P partitions and the output cursors; with two passes also the pass-1
// buckets' (partition >> bits2) offsets, cursors and the prefix of their
// tiles of `tile2` tuples.
struct PartPlan {
  uint64_t *off;       // [P + 1]
  uint32_t *cursor;    // [P]
  uint64_t *boff;      // [B1 + 1], null: one pass
  uint32_t *bcursor;   // [B1]
  uint64_t *btiles;    // [B1 + 1]
  int bits2;
  uint32_t tile2;
};

// Global histogram of partition ids (shared-memory counts, one global
// atomic per non-empty bin and CTA), and the plan of the passes: the last
// CTA to finish works it out, which takes the place of nine launches (a
// multi-level scan, the cursors, the buckets' tiles and their scan).
// ghist[P] counts the CTAs that are done.
template <int kDigit>
__global__ void __launch_bounds__(1024)
    k_pid_hist(const int32_t *__restrict__ keys, uint64_t n, int shift, uint32_t pmask,
               uint32_t *ghist, PartPlan plan) {
  extern __shared__ uint32_t sh[];
  __shared__ uint64_t s_scan[32];
  __shared__ bool s_last;
  const uint32_t P = pmask + 1;
  for (uint32_t p = threadIdx.x; p < P; p += blockDim.x) sh[p] = 0;
  __syncthreads();
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  const uint64_t tid = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  uint64_t done = 0;
  if ((reinterpret_cast<uintptr_t>(keys) & 15) == 0) {
    // 16-byte loads, four in flight per thread (16 keys)
    const int4 *k4 = reinterpret_cast<const int4 *>(keys);
    const uint64_t n4 = n / 4;
    uint64_t i = tid;
    for (; i + 3 * stride < n4; i += 4 * stride) {
      int4 k[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) k[u] = __ldcs(k4 + i + u * stride);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        atomicAdd(&sh[digit_of<kDigit>(k[u].x, shift, pmask)], 1u);
        atomicAdd(&sh[digit_of<kDigit>(k[u].y, shift, pmask)], 1u);
        atomicAdd(&sh[digit_of<kDigit>(k[u].z, shift, pmask)], 1u);
        atomicAdd(&sh[digit_of<kDigit>(k[u].w, shift, pmask)], 1u);
      }
    }
    for (; i < n4; i += stride) {
      const int4 k = __ldcs(k4 + i);
      atomicAdd(&sh[digit_of<kDigit>(k.x, shift, pmask)], 1u);
      atomicAdd(&sh[digit_of<kDigit>(k.y, shift, pmask)], 1u);
      atomicAdd(&sh[digit_of<kDigit>(k.z, shift, pmask)], 1u);
      atomicAdd(&sh[digit_of<kDigit>(k.w, shift, pmask)], 1u);
    }
    done = n4 * 4;
  }
  for (uint64_t i = done + tid; i < n; i += stride)
    atomicAdd(&sh[digit_of<kDigit>(__ldg(keys + i), shift, pmask)], 1u);
  __syncthreads();
  for (uint32_t p = threadIdx.x; p < P; p += blockDim.x)
    if (sh[p]) atomicAdd(&ghist[p], sh[p]);
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(&ghist[P], 1u) + 1 == gridDim.x;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  gbjd::cta_offsets(P, [&](uint32_t p) -> uint64_t { return __ldcg(ghist + p); }, plan.off, s_scan);
  __syncthreads();
  for (uint32_t p = threadIdx.x; p < P; p += 1024) plan.cursor[p] = (uint32_t)plan.off[p];
  if (!plan.boff) return;
  const uint32_t B1 = P >> plan.bits2;
  for (uint32_t b = threadIdx.x; b <= B1; b += 1024) {
    const uint64_t o = plan.off[b << plan.bits2];
    plan.boff[b] = o;
    if (b < B1) plan.bcursor[b] = (uint32_t)o;
  }
  __syncthreads();
  gbjd::cta_offsets(B1, [&](uint32_t b) { return (plan.boff[b + 1] - plan.boff[b] + plan.tile2 - 1) / plan.tile2; },
                    plan.btiles, s_scan);
}

template <int kSh>
struct TileSmem {
  uint32_t whist[TileShape<kSh>::warps][kMaxDigits];  // per-warp digit counts, then each warp's run start
  int2 sorted[TileShape<kSh>::tile];
  uint32_t gdelta[kMaxDigits];  // output position of sorted[i] = gdelta[digit] + i
  uint32_t wsum[8];
};

// One partition pass.  Tiles of kTile tuples: contiguous from the SoA input
// (kPairsIn = false), or, for a second pass, kTile-tuple pieces of each
// parent bucket of the AoS input (tile_off = prefix of tiles per bucket).
// digit = (f(key) >> dshift) & dmask; the output cursor of (bucket b,
// digit d) is cursor[b * (dmask + 1) + d].  kHashLoad: the SoA keys are
// replaced by fmix32(key) as they are loaded (the tuples then carry the
// hash and kDigit is kDigitPre).  Row positions are below 2^31, so tile
// arithmetic is 32-bit.
//
// kTma: the input tiles arrive by bulk copies (cp.async.bulk) into a 32 KB
// shared-memory ring behind TileSmem -- two 16 KB stages (key columns
// without values: two tiles ahead) or one 32 KB stage (pairs, or keys and
// values: one tile ahead) -- instead of through registers.  A copy covers
// the 16-byte aligned middle of the tile; the (at most three) tuples either
// side of it are loaded directly.  Input columns must be 16-byte aligned.
template <int kDigit, bool kPairsIn, bool kAoSOut, bool kHashLoad, bool kTma, int kSh>
__global__ void __launch_bounds__(TileShape<kSh>::threads, TileShape<kSh>::ctas)
    k_tile_pass(const int32_t *__restrict__ keys, const int32_t *__restrict__ vals,
                const int2 *__restrict__ pin, uint32_t n, int dshift, uint32_t dmask,
                const uint64_t *__restrict__ bucket_off, const uint64_t *__restrict__ tile_off,
                uint32_t nb, uint32_t *__restrict__ cursor, int2 *__restrict__ out_pairs,
                int32_t *__restrict__ out_k, int32_t *__restrict__ out_v, uint32_t *status) {
  constexpr int kTile = TileShape<kSh>::tile, kTileThreads = TileShape<kSh>::threads;
  constexpr int kTilePer = TileShape<kSh>::per, kTileWarps = TileShape<kSh>::warps;
  constexpr uint32_t kRingBytes = kTile * 8;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  TileSmem<kSh> &S = *reinterpret_cast<TileSmem<kSh> *>(smem_raw);
  unsigned char *ring = smem_raw + sizeof(TileSmem<kSh>);
  uint64_t *bars = reinterpret_cast<uint64_t *>(ring + kRingBytes);
  const uint32_t stage_bytes = (kPairsIn || vals) ? kRingBytes : kRingBytes / 2;
  const uint32_t nst = kRingBytes / stage_bytes;  // stages: 1 or 2
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t ndig = dmask + 1;
  const uint32_t ntiles = kPairsIn ? (uint32_t)tile_off[nb] : (n + kTile - 1) / kTile;
  // tile t -> its rows [lo, hi) and bucket b
  auto tile_range = [&](uint32_t t, uint32_t &lo, uint32_t &hi, uint32_t &b) {
    b = 0;
    if (kPairsIn) {
      uint32_t a = 0, z = nb;  // tile_off[a] <= t < tile_off[z]
      while (z - a > 1) {
        const uint32_t mid = (a + z) >> 1;
        if (tile_off[mid] <= t) a = mid; else z = mid;
      }
      b = a;
      const uint32_t bend = (uint32_t)bucket_off[b + 1];
      lo = (uint32_t)bucket_off[b] + (t - (uint32_t)tile_off[b]) * kTile;
      hi = lo + kTile < bend ? lo + kTile : bend;
    } else {
      lo = t * kTile;
      hi = lo + kTile < n ? lo + kTile : n;
    }
  };
  int2 tup[kTilePer];
  auto load_tile = [&](uint32_t lo, uint32_t hi) {
#pragma unroll
    for (int j = 0; j < kTilePer; ++j) {
      const uint32_t i = lo + tid + j * kTileThreads;
      if (i < hi) {
        if (kPairsIn) {
          tup[j] = __ldcs(pin + i);
        } else {
          // (kHashLoad: hashed when the tile is consumed, so this prefetch
          // stays in flight through the previous tile's write phase)
          tup[j].x = __ldcs(keys + i);
          tup[j].y = vals ? __ldcs(vals + i) : (int32_t)i;
        }
      }
    }
  };
  // kTma: the bulk-copied range [a, e) of the tile [lo, hi)
  auto tma_range = [&](uint32_t l, uint32_t h, uint32_t &a, uint32_t &e) {
    if (kPairsIn) {  // 8-byte tuples: even positions are 16-byte aligned
      a = (l + 1) & ~1u;
      e = h & ~1u;
    } else {  // 4-byte columns: tiles start at multiples of kTile
      a = l;
      e = l + ((h - l) & ~3u);
    }
    if (e < a) e = a;
  };
  auto issue = [&](uint32_t tt, uint32_t st) {
    uint32_t l, h, bb, a, e;
    tile_range(tt, l, h, bb);
    tma_range(l, h, a, e);
    unsigned char *dst = ring + st * stage_bytes;
    const uint32_t cols = kPairsIn ? 2 : (vals ? 2 : 1);
    gbjd::mbar_arrive_expect_tx(&bars[st], (e - a) * 4 * cols);
    if (e > a) {
      if (kPairsIn) {
        gbjd::bulk_load(dst, pin + a, (e - a) * 8, &bars[st]);
      } else {
        gbjd::bulk_load(dst, keys + a, (e - a) * 4, &bars[st]);
        if (vals) gbjd::bulk_load(dst + kTile * 4, vals + a, (e - a) * 4, &bars[st]);
      }
    }
  };
  auto read_tile = [&](uint32_t l, uint32_t h, uint32_t st) {
    uint32_t a, e;
    tma_range(l, h, a, e);
    const unsigned char *src = ring + st * stage_bytes;
#pragma unroll
    for (int j = 0; j < kTilePer; ++j) {
      const uint32_t i = l + tid + j * kTileThreads;
      if (i < h) {
        if (i >= a && i < e) {
          if (kPairsIn) {
            tup[j] = reinterpret_cast<const int2 *>(src)[i - a];
          } else {
            tup[j].x = reinterpret_cast<const int32_t *>(src)[i - a];
            tup[j].y = vals ? reinterpret_cast<const int32_t *>(src + kTile * 4)[i - a] : (int32_t)i;
          }
        } else if (kPairsIn) {
          tup[j] = __ldcs(pin + i);
        } else {
          tup[j].x = __ldcs(keys + i);
          tup[j].y = vals ? __ldcs(vals + i) : (int32_t)i;
        }
      }
    }
  };
  uint32_t t = blockIdx.x, lo = 0, hi = 0;
  uint32_t b = 0, it = 0;
  if (kTma) {
    if (tid == 0) {
      gbjd::mbar_init(&bars[0], 1);
      gbjd::mbar_init(&bars[1], 1);
      gbjd::mbar_init_fence();
    }
    __syncthreads();
    if (tid == 0)
      for (uint32_t k = 0; k < nst; ++k)
        if (t + k * gridDim.x < ntiles) issue(t + k * gridDim.x, k);
  } else if (t < ntiles) {
    tile_range(t, lo, hi, b);
    load_tile(lo, hi);
  }
  // Software pipeline: the next tile's loads are issued once this tile's
  // tuples sit in shared memory, so their DRAM latency overlaps the write
  // phase; the cursor atomic's L2 round trip overlaps the shared scatter.
  for (; t < ntiles; t += gridDim.x, ++it) {
    if (kTma) {
      tile_range(t, lo, hi, b);
      const uint32_t st = it % nst;
      const bool ok = gbjd::mbar_wait(&bars[st], (it / nst) & 1, kSpinLimit);
      if (__syncthreads_or(!ok)) {
        // a copy did not complete: report, wait (bounded) for the other
        // stage's copy, and stop
        if (tid == 0) {
          gbjd::latch(status, GBJ_DEV_TIMEOUT);
          if (nst == 2 && t + gridDim.x < ntiles)
            gbjd::mbar_wait(&bars[(it + 1) % nst], ((it + 1) / nst) & 1, kSpinLimit);
        }
        return;
      }
      read_tile(lo, hi, st);
    }
    for (uint32_t d = lane; d < ndig; d += 32) S.whist[warp][d] = 0;
    __syncwarp();
    const uint32_t cnt = hi - lo;
    uint32_t dg[kTilePer], rk[kTilePer];
#pragma unroll
    for (int j = 0; j < kTilePer; ++j) {
      if (kHashLoad) tup[j].x = (int32_t)gbjd::fmix32((uint32_t)tup[j].x);
      if (tid + j * kTileThreads < cnt) {
        dg[j] = digit_of<kDigit>(tup[j].x, dshift, dmask);
        rk[j] = atomicAdd(&S.whist[warp][dg[j]], 1u);
      }
    }
    __syncthreads();
    // kTma: every thread has read this stage; refill it two tiles ahead
    if (kTma && tid == 0 && t + nst * gridDim.x < ntiles) issue(t + nst * gridDim.x, it % nst);
    // per digit: the tile total (the per-warp starts follow the digit scan)
    uint32_t tot = 0;
    if ((uint32_t)tid < ndig) {
#pragma unroll
      for (int w = 0; w < kTileWarps; ++w) tot += S.whist[w][tid];
    }
    // this tile's run of each digit in the output (consumed after the scatter)
    uint32_t gpos = 0;
    if ((uint32_t)tid < ndig && tot) gpos = atomicAdd(&cursor[(uint64_t)b * ndig + tid], tot);
    // exclusive scan of the digit totals (ndig <= 256: warps 0..7)
    uint32_t incl = 0;
    if (tid < kMaxDigits) {
      incl = tot;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
      }
      if (lane == 31) S.wsum[warp] = incl;
    }
    __syncthreads();
    uint32_t my_start = 0;
    if ((uint32_t)tid < ndig) {
      uint32_t add = 0;
      for (int w = 0; w < warp; ++w) add += S.wsum[w];
      my_start = add + incl - tot;
      // absolute start of each warp's run of this digit in the tile
      uint32_t run = my_start;
#pragma unroll
      for (int w = 0; w < kTileWarps; ++w) {
        const uint32_t c = S.whist[w][tid];
        S.whist[w][tid] = run;
        run += c;
      }
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kTilePer; ++j) {
      if (tid + j * kTileThreads < cnt) {
        const uint32_t pos = S.whist[warp][dg[j]] + rk[j];
        S.sorted[pos] = tup[j];
      }
    }
    // written after the scatter, so the cursor atomic's round trip overlaps it
    // (modulo 2^32: gdelta + i is the output position)
    if ((uint32_t)tid < ndig) S.gdelta[tid] = gpos - my_start;
    const uint32_t tn = t + gridDim.x;
    if (!kTma && tn < ntiles) {
      tile_range(tn, lo, hi, b);
      load_tile(lo, hi);
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kTilePer; ++j) {
      const uint32_t i = tid + j * kTileThreads;
      if (i < cnt) {
        // the digit again from the key: cheaper than storing it beside the
        // tuple at the scatter (a bank-conflicting shared store) and loading it
        const int2 v = S.sorted[i];
        const uint32_t g = S.gdelta[digit_of<kDigit>(v.x, dshift, dmask)] + i;
        if (kAoSOut) {
          out_pairs[g] = v;
        } else {
          out_k[g] = v.x;
          out_v[g] = v.y;
        }
      }
    }
    __syncthreads();
  }
}

// A pass of 9 to 12 digit bits over the input columns, instead of two passes
// over half of the bits each: one CTA of 1024 threads per SM sorts tiles of
// kPer * 1024 tuples, so that a tile still has three or more tuples of a digit
// and its runs are written in whole sectors.  One shared histogram for the CTA
// (a row per warp would not fit) gives every tuple its rank; more than 4096
// digits would leave runs of one or two tuples.
//
// What bounds it is the shared-memory pipe and the phases of the one CTA that
// follow one another.  Measured on GB300, 2^27 keys with row positions (ms;
// two passes: 0.88): 9 bits 0.44, 10 bits 0.48, 11 bits 0.51, 12 bits 0.61, 13
// bits 0.93, 14 bits 1.46; with a value column 8 tuples a thread are faster
// than 12, which spill (9 to 12 bits 0.47, 0.54, 0.64, 0.78; two passes 0.93).
constexpr int kWideBits = 12;
constexpr int kWideThreads = 1024;

template <int kPer>
struct WideSmem {
  int2 sorted[kWideThreads * kPer];
  uint32_t start[1 << kWideBits];   // counts, then where a digit starts in the tile
  uint32_t gdelta[1 << kWideBits];  // output position of sorted[i] = gdelta[digit] + i
  uint32_t wsum[kWideThreads / 32];
};

template <int kDigit, bool kAoSOut, bool kHashLoad, bool kVals>
__global__ void __launch_bounds__(kWideThreads, 1)
    k_wide_pass(const int32_t *__restrict__ keys, const int32_t *__restrict__ vals, uint32_t n, int dshift,
                uint32_t dmask, uint32_t *__restrict__ cursor, int2 *__restrict__ out_pairs,
                int32_t *__restrict__ out_k, int32_t *__restrict__ out_v) {
  constexpr int kPer = kVals ? 8 : 12;
  constexpr uint32_t kTile = kWideThreads * kPer;
  constexpr int kDigits = (1 << kWideBits) / kWideThreads;  // of a thread, at most
  extern __shared__ __align__(16) unsigned char smem_raw[];
  WideSmem<kPer> &S = *reinterpret_cast<WideSmem<kPer> *>(smem_raw);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t ndig = dmask + 1, ntiles = (n + kTile - 1) / kTile;
  int32_t next[kPer];
  auto load_tile = [&](uint32_t t) {
    const uint32_t lo = t * kTile;
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
      const uint32_t i = lo + tid + j * kWideThreads;
      next[j] = i < n ? __ldcs(keys + i) : 0;
    }
  };
  uint32_t t = blockIdx.x;
  if (t < ntiles) load_tile(t);
  for (uint32_t d = tid; d < ndig; d += kWideThreads) S.start[d] = 0;
  __syncthreads();
  for (; t < ntiles; t += gridDim.x) {
    const uint32_t lo = t * kTile, cnt = n - lo < kTile ? n - lo : kTile;
    int32_t key[kPer], val[kVals ? kPer : 1];
    uint32_t rank[kPer / 2];  // 16 bits each
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
      key[j] = kHashLoad ? (int32_t)gbjd::fmix32((uint32_t)next[j]) : next[j];
      uint32_t r = 0;
      if (tid + j * kWideThreads < cnt) r = atomicAdd(&S.start[digit_of<kDigit>(key[j], dshift, dmask)], 1u);
      if (j & 1) rank[j / 2] |= r << 16;
      else rank[j / 2] = r;
    }
    if (kVals) {  // in flight through the scan
#pragma unroll
      for (int j = 0; j < kPer; ++j) {
        const uint32_t i = tid + j * kWideThreads;
        val[kVals ? j : 0] = i < cnt ? __ldcs(vals + lo + i) : 0;
      }
    }
    __syncthreads();
    // a thread's digits for the scan are neighbours
    uint32_t c[kDigits], sum = 0;
#pragma unroll
    for (int j = 0; j < kDigits; ++j) {
      const uint32_t d = tid * kDigits + j;
      c[j] = d < ndig ? S.start[d] : 0;
      sum += c[j];
    }
    uint32_t incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    if (lane == 31) S.wsum[warp] = incl;
    __syncthreads();
    uint32_t before = lane < warp ? S.wsum[lane] : 0;
    before = __reduce_add_sync(0xffffffffu, before);
    uint32_t run = before + incl - sum;
#pragma unroll
    for (int j = 0; j < kDigits; ++j) {
      const uint32_t d = tid * kDigits + j;
      if (d < ndig) S.start[d] = run;
      run += c[j];
    }
    __syncthreads();
    // and for the cursors neighbouring threads have neighbouring digits
    uint32_t gpos[kDigits], st[kDigits];
#pragma unroll
    for (int j = 0; j < kDigits; ++j) {
      const uint32_t d = j * kWideThreads + tid;
      gpos[j] = st[j] = 0;
      if (d < ndig) {
        st[j] = S.start[d];
        const uint32_t end = d + 1 < ndig ? S.start[d + 1] : cnt;
        if (end > st[j]) gpos[j] = atomicAdd(&cursor[d], end - st[j]);
      }
    }
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
      const uint32_t i = tid + j * kWideThreads;
      if (i < cnt) {
        const uint32_t r = j & 1 ? rank[j / 2] >> 16 : rank[j / 2] & 0xffffu;
        S.sorted[S.start[digit_of<kDigit>(key[j], dshift, dmask)] + r] =
            make_int2(key[j], kVals ? val[kVals ? j : 0] : (int32_t)(lo + i));
      }
    }
#pragma unroll
    for (int j = 0; j < kDigits; ++j) {
      const uint32_t d = j * kWideThreads + tid;
      if (d < ndig) S.gdelta[d] = gpos[j] - st[j];
    }
    if (t + gridDim.x < ntiles) load_tile(t + gridDim.x);
    __syncthreads();
    for (uint32_t d = tid; d < ndig; d += kWideThreads) S.start[d] = 0;
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
      const uint32_t i = tid + j * kWideThreads;
      if (i < cnt) {
        const int2 x = S.sorted[i];
        const uint32_t g = S.gdelta[digit_of<kDigit>(x.x, dshift, dmask)] + i;
        if (kAoSOut) {
          out_pairs[g] = x;
        } else {
          out_k[g] = x.x;
          out_v[g] = x.y;
        }
      }
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------- join

// Work items per partition: ceil(|R_p| / rmax) build chunks times
// ceil(|S_p| / w) probe chunks (zero when either side is empty), as offsets;
// the item counter and the results' start values beside them.
__global__ void __launch_bounds__(1024)
    k_join_plan(const uint64_t *__restrict__ ro, const uint64_t *__restrict__ so, uint32_t P, uint32_t rmax,
                uint64_t w, uint64_t *__restrict__ items, unsigned long long *ctr, gbj::AggSpec spec, int64_t *out) {
  __shared__ uint64_t s_scan[32];
  if (threadIdx.x == 0) *ctr = 0;
  if (threadIdx.x < (uint32_t)spec.n) out[threadIdx.x] = gbjd::agg_identity(spec.op[threadIdx.x]);
  gbjd::cta_offsets(P, [&](uint32_t p) -> uint64_t {
    const uint64_t nr = ro[p + 1] - ro[p], ns = so[p + 1] - so[p];
    return nr && ns ? ((nr + rmax - 1) / rmax) * ((ns + w - 1) / w) : 0;
  }, items, s_scan);
}

// kAggRows: both sides carry row positions; a match first compares the
// minor keys (when given), then reads the payloads by row.
enum : int { kAggList = 0, kAggCountXor = 1, kAggCountProduct = 2, kAggRows = 3 };

// Columns a kAggRows match reads by row position (any may be null; the
// minor-key columns are both set or both null).
struct RowCols {
  const int32_t *bmin, *pmin, *bpay, *ppay;
};

// The join works on hashed tuples: the first word of every partitioned
// tuple is h = fmix32(key), which is a bijection of the 32-bit keys, so
// h equality is key equality and the key itself is fmix32_inv(h) when an
// aggregate reads it.  The partition id is the low `bits` bits of h; the
// on-chip table places h by its high bits (independent of the partition).
//
// Table: 4-slot buckets; bucket b = slots [4b, 4b + 4), filled in order.  A
// tuple takes the next slot of its home bucket, or of a later bucket when
// that is full; a probe reads a whole bucket with one 16-byte shared load and
// stops at a bucket with room (slots only fill during the build, so no key
// was placed past a bucket that still has room).
__device__ __forceinline__ uint32_t home_bucket(uint32_t h, uint32_t nb) { return __umulhi(h, nb); }

// One work item's extent, computed by thread 0 and shared with the block.
struct JoinItem {
  unsigned long long rb, sb;  // first build / probe tuple (global index)
  uint32_t m, ns;             // build chunk size, probe chunk size
  uint32_t part;
  int valid;
};

// A warp's rings: tuples (of the build, then of the probe) that go on past
// their home bucket, and matches on their way to the accumulators.
struct JoinQueue {
  uint32_t h[64];
  int32_t v[64];
  uint32_t b[64];  // the bucket to look at next
};
struct JoinMatches {
  uint32_t h[64];
  int32_t bv[64], pv[64];
};

template <int kRMax, int kThreads, bool kRing>
struct JoinSmem {
  // slots: as many as two CTAs' (or one CTA's) shared memory holds beside the
  // rings; at least 2 kRMax
  static constexpr uint32_t cap = (kRMax / 4608) * (kRing ? 10432 : 11776);
  union {
    struct {
      int32_t key[cap];
      int32_t val[cap];
    } t;
    struct {  // the partition whose tuples may hash to the empty marker
      int2 pair[kRMax];
      unsigned short tab[cap];  // index + 1 of the pair
    } x;
  };
  uint32_t fill[cap / 8];  // tuples that asked for the bucket, 16 bits each
  JoinQueue q[kThreads / 32];
  JoinMatches m[kRing ? kThreads / 32 : 1];
};

// Persistent partition join.  kCtas blocks share an SM, so one block's clear /
// build / barriers overlap another's probes.  kAgg: the two specialised lists
// accumulate a match where it is found; other lists (of at most kMaxA
// aggregates) and kAggRows send it to the warp's ring and apply 32 at once.
//
// What bounds it is issue.  The build takes a slot with one shared addition
// (7.5 a clock and SM, a CAS 4.2) and no loop; the tuples that find their home
// bucket full, in the build and in the probe, wait in a ring until 32 of them
// can go on together.  Measured on GB300, 2^27 build and 2^29 probe tuples,
// 15 bits, COUNT + SUM(rowid xor): 2.45 -> 2.06 ms (the build's share 0.95 -> 0.74);
// 3 M and 24 M, COUNT + SUM + MIN + MAX: 0.556 -> 0.188 ms.
template <int kRMax, int kThreads, int kCtas, int kAgg, int kMaxA>
__global__ void __launch_bounds__(kThreads, kCtas)
    k_radix_join(const int2 *__restrict__ R, const uint64_t *__restrict__ ro,
                 const int2 *__restrict__ S, const uint64_t *__restrict__ so,
                 const uint64_t *__restrict__ item_off, uint32_t P, uint32_t w,
                 uint32_t sentinel_part, gbj::AggSpec spec, RowCols rc, int64_t *out,
                 unsigned long long *item_ctr) {
  constexpr bool kRing = kAgg == kAggList || kAgg == kAggRows;
  using Smem = JoinSmem<kRMax, kThreads, kRing>;
  static_assert(Smem::cap >= 2 * kRMax && Smem::cap % 64 == 0 && kRMax < 65535, "16-bit index entries and counts");
  extern __shared__ __align__(16) unsigned char smem[];
  Smem &sm = *reinterpret_cast<Smem *>(smem);
  __shared__ int64_t red[32 * GBJ_MAX_AGGS];
  __shared__ JoinItem s_it;
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  JoinQueue &q = sm.q[threadIdx.x >> 5];
  JoinMatches &mq = sm.m[kRing ? threadIdx.x >> 5 : 0];
  int64_t a_cnt = 0, a_sum = 0;  // the specialised accumulators
  int64_t v[kRing ? kMaxA : 1];
  if (kRing) {
#pragma unroll
    for (int j = 0; j < kMaxA; ++j) v[j] = j < spec.n ? gbjd::agg_identity(spec.op[j]) : 0;
  }
  const unsigned long long total = item_off[P];
  // thread 0: claims the next item and resolves its extent
  auto fetch = [&]() {
    const unsigned long long item = atomicAdd(item_ctr, 1ull);
    s_it.valid = item < total;
    if (item < total) {
      const uint32_t p = gbjd::item_partition(item_off, P, total, item);
      const uint64_t r0 = ro[p], r1 = ro[p + 1], s0 = so[p], s1 = so[p + 1];
      const uint64_t nrc = (r1 - r0 + kRMax - 1) / kRMax;
      const uint64_t local = item - item_off[p];
      const uint64_t rb = r0 + (local % nrc) * kRMax, sb = s0 + (local / nrc) * w;
      s_it.rb = rb;
      s_it.m = (uint32_t)((rb + kRMax < r1 ? rb + kRMax : r1) - rb);
      s_it.sb = sb;
      s_it.ns = (uint32_t)((sb + w < s1 ? sb + w : s1) - sb);
      s_it.part = p;
    }
  };

  // ---- matches ----
  uint32_t mn = 0, mh = 0;  // the match ring's length and head (warp-uniform)
  auto apply = [&](uint32_t c) {  // the first c (<= 32) matches of the ring
    __syncwarp();
    if ((uint32_t)lane < c) {
      const uint32_t p = (mh + lane) & 63u;
      const int32_t key = (int32_t)gbjd::fmix32_inv(mq.h[p]), bv = mq.bv[p], pv = mq.pv[p];
      // the minor-key check of the reference's partitioned join
      // (gpu-partitioned-hash-join-chained.cpp:1284-1333)
      if (kAgg != kAggRows || !rc.bmin || __ldg(rc.bmin + bv) == __ldg(rc.pmin + pv)) {
        const int64_t b = kAgg != kAggRows ? bv : rc.bpay ? __ldg(rc.bpay + bv) : 0;
        const int64_t x = kAgg != kAggRows ? pv : rc.ppay ? __ldg(rc.ppay + pv) : 0;
#pragma unroll
        for (int j = 0; j < kMaxA; ++j)
          if (j < spec.n) gbjd::agg_step(v[kRing ? j : 0], spec.op[j], spec.operand[j], key, b, x, bv, pv);
      }
    }
    __syncwarp();
    mh = (mh + c) & 63u;
    mn -= c;
  };
  // a match of this lane's tuple (all lanes call it)
  auto emit = [&](bool hit, uint32_t h, int32_t bv, int32_t pv) {
    if (kAgg == kAggCountXor) {
      // row ids are non-negative: their xor is a zero-extended 32-bit value
      a_cnt += hit;
      a_sum += hit ? (uint32_t)(bv ^ pv) : 0u;
    } else if (kAgg == kAggCountProduct) {
      a_cnt += hit;
      a_sum += (int64_t)(hit ? bv : 0) * pv;
    } else {
      const unsigned bal = __ballot_sync(0xffffffffu, hit);
      if (hit) {
        const uint32_t p = (mh + mn + __popc(bal & lt)) & 63u;
        mq.h[p] = h;
        mq.bv[p] = bv;
        mq.pv[p] = pv;
      }
      mn += __popc(bal);
      if (mn >= 32) apply(32);
    }
  };
  auto hits_of = [](const int4 &kk, uint32_t h) -> uint32_t {
    const int32_t k = (int32_t)h;
    return (uint32_t)(kk.x == k) | ((uint32_t)(kk.y == k) << 1) | ((uint32_t)(kk.z == k) << 2) |
           ((uint32_t)(kk.w == k) << 3);
  };

  // ---- the ring of tuples that go on ----
  uint32_t qn = 0, qh = 0;
  auto push = [&](bool yes, uint32_t h, int32_t x, uint32_t b) {
    const unsigned bal = __ballot_sync(0xffffffffu, yes);
    if (yes) {
      const uint32_t p = (qh + qn + __popc(bal & lt)) & 63u;
      q.h[p] = h;
      q.v[p] = x;
      q.b[p] = b;
    }
    qn += __popc(bal);
  };
  auto pop = [&](uint32_t c, uint32_t &h, int32_t &x, uint32_t &b) -> bool {
    __syncwarp();
    const bool mine = (uint32_t)lane < c;
    const uint32_t p = (qh + lane) & 63u;
    h = mine ? q.h[p] : 0;
    x = mine ? q.v[p] : 0;
    b = mine ? q.b[p] : 0;
    __syncwarp();  // read before any of them is written again
    qh = (qh + c) & 63u;
    qn -= c;
    return mine;
  };

  if (threadIdx.x == 0) fetch();
  __syncthreads();
  for (;;) {
    if (!s_it.valid) break;
    const int2 *Rp = R + s_it.rb;
    const int2 *Sp = S + s_it.sb;
    const uint32_t m = s_it.m, ns = s_it.ns;
    const bool fast = s_it.part != sentinel_part;
    // buckets: one a tuple while they fit (few full buckets: a probe of a
    // full bucket goes on), always two slots a tuple
    const uint32_t nb = min((m + 15) & ~15u, Smem::cap / 4);
    const uint32_t cap = 4 * nb;
    const int4 *tk4 = reinterpret_cast<const int4 *>(sm.t.key);
    auto next = [&](uint32_t b) { return b + 1 == nb ? 0 : b + 1; };
    if (fast) {
      for (uint32_t i = threadIdx.x; i < nb; i += kThreads)
        reinterpret_cast<int4 *>(sm.t.key)[i] = make_int4(kEmpty, kEmpty, kEmpty, kEmpty);
      for (uint32_t i = threadIdx.x; i < (nb + 1) / 2; i += kThreads) sm.fill[i] = 0;
      __syncthreads();
      // true when the bucket had a slot left
      auto place = [&](uint32_t h, int32_t x, uint32_t b) -> bool {
        const uint32_t sh = 16 * (b & 1u);
        const uint32_t at = (atomicAdd(&sm.fill[b >> 1], 1u << sh) >> sh) & 0xffffu;  // < 65536: m tuples at most
        if (at >= 4) return false;
        sm.t.key[4 * b + at] = (int32_t)h;
        sm.t.val[4 * b + at] = x;
        return true;
      };
      auto place_on = [&](uint32_t c) {  // the table has 2 m slots: every tuple finds one
        uint32_t h, b;
        int32_t x;
        const bool mine = pop(c, h, x, b);
        const bool again = mine && !place(h, x, b);
        push(again, h, x, next(b));
      };
      // the whole chunk's loads in flight at once (8 per thread per round)
      for (uint32_t i0 = threadIdx.x - lane; i0 < m; i0 += 8 * kThreads) {
        int2 t[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const uint32_t i = i0 + lane + u * kThreads;
          if (i < m) t[u] = __ldcs(Rp + i);
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const bool in = i0 + lane + u * kThreads < m;
          const uint32_t b = home_bucket((uint32_t)t[u].x, nb);
          push(in && !place((uint32_t)t[u].x, t[u].y, b), (uint32_t)t[u].x, t[u].y, next(b));
          while (qn >= 32) place_on(32);
        }
      }
      while (qn) place_on(qn < 32 ? qn : 32);
    } else {
      // ---- pairs + 16-bit index table (any hash value allowed) ----
      uint32_t *tab32 = reinterpret_cast<uint32_t *>(sm.x.tab);
      for (uint32_t i = threadIdx.x; i < cap / 2; i += kThreads) tab32[i] = 0;
      for (uint32_t i = threadIdx.x; i < m; i += kThreads) sm.x.pair[i] = Rp[i];
      __syncthreads();
      for (uint32_t i = threadIdx.x; i < m; i += kThreads) {
        uint32_t hh = __umulhi((uint32_t)sm.x.pair[i].x, cap);
        for (uint32_t step = 0; step < cap; ++step) {
          if (atomicCAS(&sm.x.tab[hh], (unsigned short)0, (unsigned short)(i + 1)) == 0) break;
          if (++hh == cap) hh = 0;
        }
      }
    }
    __syncthreads();
    // next item: fetched now, consumed after the closing barrier (every
    // thread has read this item's extent above)
    if (threadIdx.x == 0) fetch();
    if (fast) {
      // every match of one bucket for one tuple a lane
      auto bucket = [&](uint32_t hits, uint32_t h, int32_t x, uint32_t b) {
        while (__any_sync(0xffffffffu, hits != 0)) {
          const uint32_t i = hits ? __ffs(hits) - 1 : 0;
          emit(hits != 0, h, hits ? sm.t.val[4 * b + i] : 0, x);
          hits &= hits - 1;
        }
      };
      auto probe_on = [&](uint32_t c) {
        uint32_t h, b;
        int32_t x;
        const bool mine = pop(c, h, x, b);
        const int4 kk = tk4[b];
        bucket(mine ? hits_of(kk, h) : 0u, h, x, b);
        push(mine && kk.w != kEmpty, h, x, next(b));
      };
      // Probe rounds of 4 tuples per thread; the next round's tuples are
      // loaded while this round is probed.
      int2 nxt[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const uint32_t j = threadIdx.x + u * kThreads;
        nxt[u] = j < ns ? __ldcs(Sp + j) : make_int2(0, 0);
      }
      for (uint32_t j0 = 0; j0 < ns; j0 += 4 * kThreads) {
        int2 t[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          t[u] = nxt[u];
          const uint32_t j = j0 + 4 * kThreads + threadIdx.x + u * kThreads;
          nxt[u] = j < ns ? __ldcs(Sp + j) : make_int2(0, 0);
        }
        uint32_t more = 0;              // bit u: tuple u goes on past its home bucket
        uint32_t slots = 0, tuples = 0;  // matching slots, tuples that match
        auto tuple = [&](int u) { return u == 0 ? t[0] : u == 1 ? t[1] : u == 2 ? t[2] : t[3]; };
        auto home = [&](int u, const int2 &x) {
          const bool valid = j0 + threadIdx.x + u * kThreads < ns;
          const uint32_t b = home_bucket((uint32_t)x.x, nb);
          const int4 kk = tk4[b];
          const bool e0 = kk.x == x.x, e1 = kk.y == x.x, e2 = kk.z == x.x, e3 = kk.w == x.x;
          const uint32_t i = e0 ? 0 : e1 ? 1 : e2 ? 2 : 3;
          // loaded whether or not it is a match
          emit(valid & (e0 | e1 | e2 | e3), (uint32_t)x.x, sm.t.val[4 * b + i], x.y);
          slots += (uint32_t)(valid & e0) + (uint32_t)(valid & e1) + (uint32_t)(valid & e2) + (uint32_t)(valid & e3);
          tuples += valid & (e0 | e1 | e2 | e3);
          more |= (uint32_t)(valid & (kk.w != kEmpty)) << u;
        };
        if (kRing) {  // rolled: one copy of the code that applies matches
#pragma unroll 1
          for (int u = 0; u < 4; ++u) home(u, tuple(u));
        } else {
#pragma unroll
          for (int u = 0; u < 4; ++u) home(u, t[u]);
        }
        if (__any_sync(0xffffffffu, slots != tuples)) {  // copies of a build key in one bucket
#pragma unroll 1
          for (int u = 0; u < 4; ++u) {
            const int2 x = tuple(u);
            const uint32_t b = home_bucket((uint32_t)x.x, nb);
            const bool valid = j0 + threadIdx.x + u * kThreads < ns;
            const uint32_t hits = valid ? hits_of(tk4[b], (uint32_t)x.x) : 0u;
            bucket(hits & (hits - 1), (uint32_t)x.x, x.y, b);  // all but the first
          }
        }
        if (__any_sync(0xffffffffu, more != 0)) {
          auto on = [&](int u, const int2 &x) {
            push((more >> u) & 1u, (uint32_t)x.x, x.y, next(home_bucket((uint32_t)x.x, nb)));
            while (qn >= 32) probe_on(32);
          };
          if (kRing) {
#pragma unroll 1
            for (int u = 0; u < 4; ++u) on(u, tuple(u));
          } else {
#pragma unroll
            for (int u = 0; u < 4; ++u) on(u, t[u]);
          }
        }
      }
      while (qn) probe_on(qn < 32 ? qn : 32);
    } else {
      // index table: plain linear probing, one slot per step
      for (uint32_t j0 = threadIdx.x - lane; j0 < ns; j0 += kThreads) {
        bool active = j0 + lane < ns;
        const int2 t = active ? __ldcs(Sp + j0 + lane) : make_int2(0, 0);
        uint32_t hh = __umulhi((uint32_t)t.x, cap);
        for (uint32_t step = 0; step < cap; ++step) {
          if (!__any_sync(0xffffffffu, active)) break;
          const unsigned short idx = active ? sm.x.tab[hh] : 0;
          active = idx != 0;
          const int2 bt = active ? sm.x.pair[idx - 1] : make_int2(0, 0);
          emit(active && bt.x == t.x, (uint32_t)t.x, bt.y, t.y);
          if (++hh == cap) hh = 0;
        }
      }
    }
    __syncthreads();
  }
  if (kRing)
    while (mn) apply(mn < 32 ? mn : 32);
  gbjd::Acc acc;
#pragma unroll
  for (int j = 0; j < GBJ_MAX_AGGS; ++j)
    acc.v[j] = kRing ? (j < kMaxA ? v[kRing && j < kMaxA ? j : 0] : 0) : j == 0 ? a_cnt : j == 1 ? a_sum : 0;
  gbjd::block_flush(spec, acc, red, out);
}

template <int kRMax, int kThreads, int kCtas, int kAgg, int kMaxA>
int launch_join(gbj_ctx *ctx, const int2 *R, const uint64_t *ro, const int2 *S,
                const uint64_t *so, const uint64_t *item_off, uint32_t P,
                uint32_t w, uint32_t sentinel_part, const AggSpec &spec, const RowCols &rc,
                int64_t *out, unsigned long long *ctr, cudaStream_t s) {
  constexpr size_t smem = sizeof(JoinSmem<kRMax, kThreads, kAgg == kAggList || kAgg == kAggRows>);
  auto kern = k_radix_join<kRMax, kThreads, kCtas, kAgg, kMaxA>;
  GBJ_CHECK_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)smem));
  int per_sm = 0;
  GBJ_CHECK_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kThreads, smem));
  if (per_sm < 1) return set_error(ctx, GBJ_ERR_CUDA, "k_radix_join: no resident block fits");
  kern<<<ctx->sm_count * per_sm, kThreads, smem, s>>>(R, ro, S, so, item_off, P, w,
                                                     sentinel_part, spec, rc, out, ctr);
  return after_launch(ctx, "k_radix_join", s);
}

template <int kRMax, int kThreads, int kCtas>
int launch_join_agg(gbj_ctx *ctx, bool by_rows, const AggSpec &spec, const int2 *R, const uint64_t *ro,
                    const int2 *S, const uint64_t *so, const uint64_t *items, uint32_t P, uint32_t w,
                    uint32_t sentinel_part, const RowCols &rc, int64_t *d_out, unsigned long long *ctr,
                    cudaStream_t s) {
#define GBJ_JOIN(A, M) \
  launch_join<kRMax, kThreads, kCtas, A, M>(ctx, R, ro, S, so, items, P, w, sentinel_part, spec, rc, d_out, ctr, s)
  if (by_rows) return GBJ_JOIN(kAggRows, GBJ_MAX_AGGS);
  const bool two = spec.n == 2 && spec.op[0] == GBJ_AGG_COUNT && spec.op[1] == GBJ_AGG_SUM;
  if (two && spec.operand[1] == GBJ_VAL_ROWID_XOR) return GBJ_JOIN(kAggCountXor, 2);
  if (two && spec.operand[1] == GBJ_VAL_PRODUCT) return GBJ_JOIN(kAggCountProduct, 2);
  return spec.n <= 4 ? GBJ_JOIN(kAggList, 4) : GBJ_JOIN(kAggList, GBJ_MAX_AGGS);
#undef GBJ_JOIN
}

// The tile shape of a pass with `ndig` digits and pair (AoS) or column output.
int tile_shape_for(uint32_t ndig, bool aos) { return ndig <= 128 && aos ? 0 : 1; }

template <int kDigit, bool kPairsIn, bool kAoSOut, bool kHashLoad, int kSh>
int launch_tile_pass_sh(gbj_ctx *ctx, const int32_t *keys, const int32_t *vals, const int2 *pin,
                        uint64_t n, int dshift, uint32_t dmask, const uint64_t *bucket_off,
                        const uint64_t *tile_off, uint32_t nb, uint32_t *cursor, int2 *op, int32_t *ok,
                        int32_t *ov, cudaStream_t s) {
  using TS = TileShape<kSh>;
  // bulk-copy loads when the input columns are 16-byte aligned
  auto al16 = [](const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
  const bool tma = kTileTma && (kPairsIn ? al16(pin) : (al16(keys) && (!vals || al16(vals))));
  auto kern = tma ? k_tile_pass<kDigit, kPairsIn, kAoSOut, kHashLoad, true, kSh>
                  : k_tile_pass<kDigit, kPairsIn, kAoSOut, kHashLoad, false, kSh>;
  const size_t smem = sizeof(TileSmem<kSh>) + (tma ? (size_t)TS::tile * 8 + 16 : 0);
  GBJ_CHECK_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  int per_sm = 0;
  GBJ_CHECK_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, TS::threads, smem));
  if (per_sm < 1) per_sm = 1;
  const uint64_t tiles_hint = (n + TS::tile - 1) / TS::tile + nb;
  const uint64_t grid = std::max<uint64_t>(1, std::min<uint64_t>((uint64_t)ctx->sm_count * per_sm, tiles_hint));
  kern<<<(unsigned)grid, TS::threads, smem, s>>>(keys, vals, pin, (uint32_t)n, dshift, dmask, bucket_off, tile_off,
                                                 nb, cursor, op, ok, ov, ctx->d_status);
  return after_launch(ctx, "k_tile_pass", s);
}

template <int kDigit, bool kPairsIn, bool kAoSOut, bool kHashLoad>
int launch_tile_pass(gbj_ctx *ctx, const int32_t *keys, const int32_t *vals, const int2 *pin,
                     uint64_t n, int dshift, uint32_t dmask, const uint64_t *bucket_off,
                     const uint64_t *tile_off, uint32_t nb, uint32_t *cursor, int2 *op, int32_t *ok,
                     int32_t *ov, cudaStream_t s) {
  if (tile_shape_for(dmask + 1, kAoSOut) == 0)
    return launch_tile_pass_sh<kDigit, kPairsIn, kAoSOut, kHashLoad, 0>(ctx, keys, vals, pin, n, dshift, dmask,
                                                                       bucket_off, tile_off, nb, cursor, op, ok,
                                                                       ov, s);
  return launch_tile_pass_sh<kDigit, kPairsIn, kAoSOut, kHashLoad, 1>(ctx, keys, vals, pin, n, dshift, dmask,
                                                                     bucket_off, tile_off, nb, cursor, op, ok, ov,
                                                                     s);
}

template <int kDigit, bool kAoSOut, bool kHashLoad, bool kVals>
int launch_wide_pass_v(gbj_ctx *ctx, const int32_t *keys, const int32_t *vals, uint64_t n, int dshift, uint32_t dmask,
                       uint32_t *cursor, int2 *op, int32_t *ok, int32_t *ov, cudaStream_t s) {
  constexpr int kPer = kVals ? 8 : 12;
  auto kern = k_wide_pass<kDigit, kAoSOut, kHashLoad, kVals>;
  constexpr size_t smem = sizeof(WideSmem<kPer>);
  GBJ_CHECK_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const uint64_t tiles = (n + kWideThreads * kPer - 1) / (kWideThreads * kPer);
  kern<<<(unsigned)std::min<uint64_t>(tiles, ctx->sm_count), kWideThreads, smem, s>>>(keys, vals, (uint32_t)n, dshift,
                                                                                      dmask, cursor, op, ok, ov);
  return after_launch(ctx, "k_wide_pass", s);
}

template <int kDigit, bool kAoSOut, bool kHashLoad>
int launch_wide_pass(gbj_ctx *ctx, const int32_t *keys, const int32_t *vals, uint64_t n, int dshift, uint32_t dmask,
                     uint32_t *cursor, int2 *op, int32_t *ok, int32_t *ov, cudaStream_t s) {
  if (vals)
    return launch_wide_pass_v<kDigit, kAoSOut, kHashLoad, true>(ctx, keys, vals, n, dshift, dmask, cursor, op, ok, ov,
                                                                s);
  return launch_wide_pass_v<kDigit, kAoSOut, kHashLoad, false>(ctx, keys, vals, n, dshift, dmask, cursor, op, ok, ov,
                                                               s);
}

// kHashOut: the tuples leave with fmix32(key) in place of the key (the
// partitioned join's layout; AoS output only), and the passes take their
// digits from that word.
template <int kDigit, bool kHashOut>
int partition_impl(gbj_ctx *ctx, const int32_t *keys, const int32_t *vals, uint64_t n, int shift,
                   int bits, int2 *out_pairs, int32_t *out_keys, int32_t *out_vals,
                   uint64_t *offsets, cudaStream_t s, int passes) {
  if ((passes == 1 && bits > 8) || (passes == 2 && bits < 2) || passes < 0 || passes > 2)
    return set_error(ctx, GBJ_ERR_UNSUPPORTED,
                     "partition: one pass takes at most 8 radix bits, two passes at least 2");
  if (n >= (1ull << 31)) return set_error(ctx, GBJ_ERR_INVALID, "partition: n >= 2^31");
  if (kHashOut && !out_pairs) return set_error(ctx, GBJ_ERR_INVALID, "partition: hashed tuples are AoS only");
  // digit function of the tile passes: of the loaded key, or of the hash word
  constexpr int kPass = kHashOut ? kDigitPre : kDigit;
  const uint32_t P = 1u << bits, pmask = P - 1;
  Scratch scratch(ctx, s);
  // one pass writes the output while it still reads the columns, two passes do
  // not: columns that are partitioned in place take two from 9 bits on
  auto apart = [&](const void *in, const void *out) {
    const uintptr_t a = reinterpret_cast<uintptr_t>(in), b = reinterpret_cast<uintptr_t>(out);
    return !in || !out || a + 4 * n <= b || b + 4 * n <= a;
  };
  const bool in_place = !out_pairs && !(apart(keys, out_keys) && apart(keys, out_vals) && apart(vals, out_keys) &&
                                        apart(vals, out_vals));
  const bool wide = passes == 0 && bits > 8 && bits <= kWideBits && !in_place;
  const bool one = wide || passes == 1 || (passes == 0 && bits <= 8);
  const int bits2 = bits / 2, bits1 = bits - bits2;
  const uint32_t B1 = 1u << bits1, m2 = (1u << bits2) - 1;
  uint32_t *hist, *cursors;
  uint64_t *off = offsets;
  GBJ_TRY(scratch.get(P + 1, &hist));
  GBJ_TRY(scratch.get(P + B1, &cursors));
  if (!off) GBJ_TRY(scratch.get(P + 1, &off));
  PartPlan plan{off, cursors, nullptr, nullptr, nullptr, 0, 1};
  int2 *tmp = nullptr;
  if (!one) {
    GBJ_TRY(scratch.get(B1 + 1, &plan.boff));
    GBJ_TRY(scratch.get(B1 + 1, &plan.btiles));
    plan.bcursor = cursors + P;
    plan.bits2 = bits2;
    plan.tile2 = tile_shape_for(m2 + 1, out_pairs != nullptr) == 0 ? TileShape<0>::tile : TileShape<1>::tile;
    GBJ_TRY(scratch.get(n + 1, &tmp));
  }
  GBJ_CHECK_CUDA(ctx, cudaMemsetAsync(hist, 0, sizeof(uint32_t) * (P + 1), s));
  {
    const size_t smem = (size_t)P * sizeof(uint32_t);
    // the most any call takes: the limit is the kernel's, not the call's
    GBJ_CHECK_CUDA(ctx, cudaFuncSetAttribute(k_pid_hist<kDigit>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)(sizeof(uint32_t) << kMaxPartBits)));
    int per_sm = 1;
    GBJ_CHECK_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_pid_hist<kDigit>, 1024, smem));
    const uint64_t grid = std::max<uint64_t>(
        1, std::min<uint64_t>((uint64_t)ctx->sm_count * std::max(per_sm, 1), (n + 16383) / 16384));
    k_pid_hist<kDigit><<<(unsigned)grid, 1024, smem, s>>>(keys, n, shift, pmask, hist, plan);
    GBJ_TRY(after_launch(ctx, "k_pid_hist", s));
  }
  if (wide) {
    if (out_pairs)
      return launch_wide_pass<kPass, true, kHashOut>(ctx, keys, vals, n, shift, pmask, plan.cursor, out_pairs, nullptr,
                                                     nullptr, s);
    return launch_wide_pass<kPass, false, false>(ctx, keys, vals, n, shift, pmask, plan.cursor, nullptr, out_keys,
                                                 out_vals, s);
  }
  if (one) {
    if (out_pairs)
      return launch_tile_pass<kPass, false, true, kHashOut>(ctx, keys, vals, nullptr, n, shift, pmask, nullptr,
                                                            nullptr, 1, plan.cursor, out_pairs, nullptr, nullptr, s);
    return launch_tile_pass<kPass, false, false, false>(ctx, keys, vals, nullptr, n, shift, pmask, nullptr, nullptr,
                                                        1, plan.cursor, nullptr, out_keys, out_vals, s);
  }
  GBJ_TRY((launch_tile_pass<kPass, false, true, kHashOut>(ctx, keys, vals, nullptr, n, shift + bits2, B1 - 1, nullptr,
                                                          nullptr, 1, plan.bcursor, tmp, nullptr, nullptr, s)));
  if (out_pairs)
    return launch_tile_pass<kPass, true, true, false>(ctx, nullptr, nullptr, tmp, n, shift, m2, plan.boff, plan.btiles,
                                                      B1, plan.cursor, out_pairs, nullptr, nullptr, s);
  return launch_tile_pass<kPass, true, false, false>(ctx, nullptr, nullptr, tmp, n, shift, m2, plan.boff, plan.btiles,
                                                     B1, plan.cursor, nullptr, out_keys, out_vals, s);
}

}  // namespace

namespace gbj {

int partition_tuples(gbj_ctx *ctx, const int32_t *keys, const int32_t *vals, uint64_t n,
                     int digit, int shift, int bits, int2 *out_pairs, int32_t *out_keys,
                     int32_t *out_vals, uint64_t *offsets, cudaStream_t s, int passes, bool hash_out) {
  if (hash_out) {
    if (digit != GBJ_DIGIT_HASH) return set_error(ctx, GBJ_ERR_INVALID, "partition: hashed tuples need hash digits");
    return partition_impl<GBJ_DIGIT_HASH, true>(ctx, keys, vals, n, shift, bits, out_pairs, out_keys, out_vals,
                                                offsets, s, passes);
  }
  if (digit == GBJ_DIGIT_HASH)
    return partition_impl<GBJ_DIGIT_HASH, false>(ctx, keys, vals, n, shift, bits, out_pairs, out_keys,
                                                 out_vals, offsets, s, passes);
  return partition_impl<GBJ_DIGIT_KEY, false>(ctx, keys, vals, n, shift, bits, out_pairs, out_keys,
                                              out_vals, offsets, s, passes);
}

}  // namespace gbj

extern "C" {

int gbj_partition(gbj_ctx *ctx, const int32_t *d_keys, const int32_t *d_payload, uint64_t n,
                  int32_t digit, int32_t shift, int32_t bits, int32_t *d_out_keys,
                  int32_t *d_out_payload, uint64_t *d_offsets, void *stream) {
  if (!ctx) return GBJ_ERR_INVALID;
  if (digit != GBJ_DIGIT_KEY && digit != GBJ_DIGIT_HASH)
    return set_error(ctx, GBJ_ERR_INVALID, "partition: bad digit function");
  if (bits < 1 || bits > kMaxPartBits || shift < 0 || shift + bits > 32)
    return set_error(ctx, GBJ_ERR_INVALID, "partition: bits must be in [1, 15], shift+bits <= 32");
  if (n >= (1ULL << 31)) return set_error(ctx, GBJ_ERR_INVALID, "partition: n >= 2^31");
  if (n && (!d_keys || !d_out_keys || !d_out_payload))
    return set_error(ctx, GBJ_ERR_INVALID, "partition: null column");
  cudaStream_t s = pick_stream(ctx, stream);
  prof_mark(ctx, s);
  if (n == 0) {
    if (d_offsets)
      GBJ_CHECK_CUDA(ctx, cudaMemsetAsync(d_offsets, 0, sizeof(uint64_t) * ((1ull << bits) + 1), s));
    return GBJ_OK;
  }
  return partition_tuples(ctx, d_keys, d_payload, n, digit, shift, bits, nullptr, d_out_keys,
                          d_out_payload, d_offsets, s);
}

}  // extern "C"

// Shared body of gbj_radix_join_agg and gbj_radix_join_agg_minor.  `least`: an
// untuned call takes the fewest partitions that fit, whose offsets are the
// fewest words.
static int radix_join_plan(gbj_ctx *ctx, const int32_t *d_build_keys, const int32_t *d_build_minor,
                           const int32_t *d_build_payload, uint64_t n_build,
                           const int32_t *d_probe_keys, const int32_t *d_probe_minor,
                           const int32_t *d_probe_payload, uint64_t n_probe,
                           const gbj_radix_params *params, const gbj_agg *aggs, int32_t n_aggs,
                           int64_t *d_out, void *stream, bool least) {
  if (!ctx || !d_out) return GBJ_ERR_INVALID;
  GBJ_TRY(validate_aggs(ctx, aggs, n_aggs));
  if (n_build >= (1ULL << 31) || n_probe >= (1ULL << 31))
    return set_error(ctx, GBJ_ERR_INVALID, "radix_join: inputs must have < 2^31 rows");
  if ((n_build && !d_build_keys) || (n_probe && !d_probe_keys))
    return set_error(ctx, GBJ_ERR_INVALID, "radix_join: null key column");
  const bool minor = d_build_minor || d_probe_minor;
  if (minor && ((n_build && !d_build_minor) || (n_probe && !d_probe_minor)))
    return set_error(ctx, GBJ_ERR_INVALID,
                     "radix_join: a minor key needs both sides (build_k_minor and probe_k_minor)");
  // Every field of the parameters is honoured or refused.
  if (params) {
    if (params->bits < 0 || params->bits > kMaxPartBits || params->log_parts < 0 ||
        params->log_parts > kMaxPartBits)
      return set_error(ctx, GBJ_ERR_UNSUPPORTED, "radix_join: radix bits must be in [0, 15]");
    if (params->passes < 0 || params->passes > 2)
      return set_error(ctx, GBJ_ERR_UNSUPPORTED, "radix_join: passes must be 0 (auto), 1 or 2");
    if (params->block != 0 && params->block != kJoinWide.threads && params->block != kJoinPair.threads)
      return set_error(ctx, GBJ_ERR_UNSUPPORTED,
                       "radix_join: the join kernel runs 512 or 1024 threads per block (block 0, 512 or 1024)");
  }
  AggSpec spec = make_spec(aggs, n_aggs);
  // Which value each side carries into the partitions.
  bool b_row = false, b_pay = false, p_row = false, p_pay = false;
  for (int j = 0; j < n_aggs; ++j) {
    switch (spec.operand[j]) {
      case GBJ_VAL_BUILD: b_pay = true; break;
      case GBJ_VAL_PROBE: p_pay = true; break;
      case GBJ_VAL_PRODUCT: b_pay = p_pay = true; break;
      case GBJ_VAL_BUILD_ROWID: b_row = true; break;
      case GBJ_VAL_PROBE_ROWID: p_row = true; break;
      case GBJ_VAL_ROWID_XOR: b_row = p_row = true; break;
      default: break;
    }
  }
  if ((b_pay && !d_build_payload && n_build) || (p_pay && !d_probe_payload && n_probe))
    return set_error(ctx, GBJ_ERR_INVALID, "radix_join: aggregate reads a missing payload");
  // Row mode: both sides carry row positions and a match reads the minor
  // keys and payloads by row (a composite key, or one side needing both its
  // payload and its row id).
  const bool by_rows = minor || (b_row && b_pay) || (p_row && p_pay);
  cudaStream_t s = pick_stream(ctx, stream);
  prof_mark(ctx, s);
  if (n_build == 0 || n_probe == 0) return init_agg_out(ctx, spec, d_out, s);

  // ---- plan: the fewest radix bits whose largest expected build partition
  //      fits the on-chip table, but enough partitions to give every CTA a few
  //      work items (auto_plan.h); explicit params override ----
  const int passes = params ? params->passes : 0;
  // Join kernel shape: the caller's block size, else an autotuned one, else by
  // the sizes (auto_plan.h).
  const bool explicit_bits = params && (params->log_parts > 0 || params->bits > 0);
  int block = params ? params->block : 0;
  if (!block) {
    const int32_t tb = tuned_value(ctx, tune_key("radixblock", n_build, n_probe));
    if (tb > 0) {
      block = tb;
    } else if (explicit_bits) {
      const int b = params->bits > 0 ? params->bits : params->log_parts;
      block = radix_fit_bits(n_build, kJoinPair.rmax) <= b ? kJoinPair.threads : kJoinWide.threads;
    } else {
      block = least ? kJoinPair.threads : radix_auto_threads(n_build, n_probe);
    }
  }
  const JoinShape shape = block == kJoinWide.threads ? kJoinWide : kJoinPair;
  const uint32_t kRMax = (uint32_t)shape.rmax;
  int bits = least ? radix_fit_bits(n_build, shape.rmax) : radix_auto_bits(n_build, n_probe, shape.threads);
  if (!explicit_bits) {  // an autotuned choice for this size bucket, if any
    const int32_t tb = tuned_value(ctx, tune_key(shape.threads == kJoinWide.threads ? "radix" : "radix512",
                                                 n_build, n_probe));
    if (tb > 0) bits = std::min<int>(tb, kMaxPartBits);
    // a pinned pass count bounds the automatic choice
    if (passes == 1) bits = std::min(bits, 8);
    if (passes == 2) bits = std::max(bits, 2);
  }
  if (params && params->log_parts > 0) bits = params->log_parts;
  if (params && params->bits > 0) bits = params->bits;
  if ((passes == 1 && bits > 8) || (passes == 2 && bits < 2))
    return set_error(ctx, GBJ_ERR_UNSUPPORTED,
                     "radix_join: one pass takes at most 8 radix bits, two passes at least 2");
  const uint32_t P = 1u << bits;
  const uint64_t w = 1u << 17;  // probe tuples per work item
  // tuples carry fmix32(key); the partition of the hash equal to the empty
  // marker takes the index-table path
  const uint32_t sentinel_part = (uint32_t)kEmpty & (P - 1);

  Scratch scratch(ctx, s);
  int2 *R, *S;
  uint64_t *ro, *so, *items;
  unsigned long long *ctr;
  GBJ_TRY(scratch.get(n_build + 2, &R));
  GBJ_TRY(scratch.get(n_probe + 2, &S));
  GBJ_TRY(scratch.get(P + 1, &ro));
  GBJ_TRY(scratch.get(P + 1, &so));
  GBJ_TRY(scratch.get(P + 1, &items));
  GBJ_TRY(scratch.get(1, &ctr));
  GBJ_TRY(partition_tuples(ctx, d_build_keys, b_pay && !by_rows ? d_build_payload : nullptr, n_build,
                           GBJ_DIGIT_HASH, 0, bits, R, nullptr, nullptr, ro, s, passes, true));
  GBJ_TRY(partition_tuples(ctx, d_probe_keys, p_pay && !by_rows ? d_probe_payload : nullptr, n_probe,
                           GBJ_DIGIT_HASH, 0, bits, S, nullptr, nullptr, so, s, passes, true));
  k_join_plan<<<1, 1024, 0, s>>>(ro, so, P, kRMax, w, items, ctr, spec, d_out);
  GBJ_TRY(after_launch(ctx, "k_join_plan", s));
  const RowCols rc{minor ? d_build_minor : nullptr, minor ? d_probe_minor : nullptr,
                   b_pay ? d_build_payload : nullptr, p_pay ? d_probe_payload : nullptr};
  if (shape.threads == kJoinWide.threads)
    return launch_join_agg<kJoinWide.rmax, kJoinWide.threads, 1>(ctx, by_rows, spec, R, ro, S, so, items, P, w,
                                                                 sentinel_part, rc, d_out, ctr, s);
  return launch_join_agg<kJoinPair.rmax, kJoinPair.threads, 2>(ctx, by_rows, spec, R, ro, S, so, items, P, w,
                                                               sentinel_part, rc, d_out, ctr, s);
}

static int radix_join_impl(gbj_ctx *ctx, const int32_t *d_build_keys, const int32_t *d_build_minor,
                           const int32_t *d_build_payload, uint64_t n_build,
                           const int32_t *d_probe_keys, const int32_t *d_probe_minor,
                           const int32_t *d_probe_payload, uint64_t n_probe,
                           const gbj_radix_params *params, const gbj_agg *aggs, int32_t n_aggs,
                           int64_t *d_out, void *stream) {
  auto plan = [&](bool least) {
    return radix_join_plan(ctx, d_build_keys, d_build_minor, d_build_payload, n_build, d_probe_keys, d_probe_minor,
                           d_probe_payload, n_probe, params, aggs, n_aggs, d_out, stream, least);
  };
  const int rc = plan(false);
  return rc == GBJ_ERR_OOM ? plan(true) : rc;  // a pool without room for as many partitions
}

extern "C" {

int gbj_radix_join_agg(gbj_ctx *ctx, const int32_t *d_build_keys,
                       const int32_t *d_build_payload, uint64_t n_build,
                       const int32_t *d_probe_keys, const int32_t *d_probe_payload,
                       uint64_t n_probe, const gbj_radix_params *params, const gbj_agg *aggs,
                       int32_t n_aggs, int64_t *d_out, void *stream) {
  return radix_join_impl(ctx, d_build_keys, nullptr, d_build_payload, n_build, d_probe_keys, nullptr,
                         d_probe_payload, n_probe, params, aggs, n_aggs, d_out, stream);
}

int gbj_radix_join_agg_minor(gbj_ctx *ctx, const int32_t *d_build_keys,
                             const int32_t *d_build_minor, const int32_t *d_build_payload,
                             uint64_t n_build, const int32_t *d_probe_keys,
                             const int32_t *d_probe_minor, const int32_t *d_probe_payload,
                             uint64_t n_probe, const gbj_radix_params *params,
                             const gbj_agg *aggs, int32_t n_aggs, int64_t *d_out,
                             void *stream) {
  if (ctx && ((n_build && !d_build_minor) || (n_probe && !d_probe_minor)))
    return set_error(ctx, GBJ_ERR_INVALID, "radix_join_minor: both minor-key columns are required");
  return radix_join_impl(ctx, d_build_keys, d_build_minor, d_build_payload, n_build, d_probe_keys,
                         d_probe_minor, d_probe_payload, n_probe, params, aggs, n_aggs, d_out, stream);
}

}  // extern "C"
