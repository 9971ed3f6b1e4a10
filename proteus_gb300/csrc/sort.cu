// Sort rows by an int32 key (ORDER BY), e.g. a group-by's output.
//
// Stands in for the reference's GPU sort (core/olap/lib/operators/gpu/
// gpu-sort.cpp; core/platform/lib/util/sort/gpu/sort-util.cu:191-218 calls
// thrust::sort on packed tuples).  Here: a stable LSD radix sort with 8-bit
// digits of an order-preserving form of the key, so ties keep their input
// order and the result is deterministic.
//
// A key travels with one 32-bit word: the other column when there are two
// columns (then no row is ever gathered), the row position when there are
// more -- the last pass then writes the columns through it.  Digits that all
// keys share are skipped: a column of row ids below 2^24 takes three passes.
//
//  * up to kBlockMax rows: one CTA sorts them in shared memory, one launch;
//  * above: one kernel reads the keys once and counts all four digits, then
//    one kernel per digit (the one-sweep scheme of Adinets and Merrill, 2022:
//    a tile's place in each digit's output range comes from its predecessors'
//    published counts instead of a scan between two kernels), so a pass reads
//    and writes every row once.
//
// What bounds a pass over many rows is HBM (16 B a row) together with issue:
// ranking a row costs eight ballots.  A sort of few rows is launches and
// barriers.  Measured on GB300, two columns (before: per pass a histogram, a
// three-kernel scan and a scatter, then a gather), host
// calls included: 1000 rows 74 -> 20 us, 65,536 rows 139 -> 45 us, 2^20 rows
// 189 -> 85 us, 2^24 rows 1302 -> 505 us, 2^26 rows 7663 -> 1900 us.  At 2^24
// rows a pass takes 115 us: 147 warp instructions per 32 rows, issue 55 %,
// ALU 57 %, DRAM 220 MB; tiles of 256 threads, 10 to 20 rows a thread and
// walks of 8 or 16 predecessors at a time were within 5 % or slower.
#include <algorithm>

#include "gbj_internal.cuh"

using namespace gbj;

namespace {

constexpr int kMaxCols = GBJ_SORT_MAX_COLS;
constexpr int kRadix = 256;

struct Cols {
  const int32_t *in[kMaxCols];
  int32_t *out[kMaxCols];
  int32_t n, key;
  uint32_t flip;  // order-preserving form: key ^ flip, unsigned
};

// The word that travels with row i's key.
__device__ __forceinline__ uint32_t carried(const Cols &c, uint32_t i) {
  return c.n == 2 ? (uint32_t)__ldcs(c.in[1 - c.key] + i) : i;
}
// Row `pos` of the result.
__device__ __forceinline__ void put_row(const Cols &c, uint32_t pos, uint32_t k, uint32_t v) {
  c.out[c.key][pos] = (int32_t)(k ^ c.flip);
  if (c.n == 2) {
    c.out[1 - c.key][pos] = (int32_t)v;
  } else {
#pragma unroll 4
    for (int j = 0; j < c.n; ++j)
      if (j != c.key) c.out[j][pos] = __ldg(c.in[j] + v);
  }
}

// Lanes whose 8-bit value equals this lane's: one ballot per bit
// (__match_any_sync costs far more on this part).
__device__ __forceinline__ unsigned same_digit(uint32_t d) {
  unsigned peers = 0xffffffffu;
#pragma unroll
  for (int bit = 0; bit < 8; ++bit) {
    const uint32_t all = (uint32_t)((int32_t)(d << (31 - bit)) >> 31);  // the bit, in every position
    peers &= ~(__ballot_sync(0xffffffffu, all != 0) ^ all);
  }
  return peers;
}

template <int kWarps>
struct RankSmem {
  uint32_t whist[kWarps][kRadix];  // a warp's digit counts, then where its run of the digit starts in the tile
  uint32_t start[kRadix];          // where the digit starts in the tile
  uint32_t wsum[kRadix / 32];
};

// Stable ranks of a tile held warp by warp (a warp's kItems x 32 rows are
// consecutive, its i-th load covers rows 32 i .. 32 i + 31 of them): on
// return S.whist[warp][digit] + rank[i] is a row's place in the sorted tile.
// Thread d < 256 returns the tile's count of digit d.
template <int kItems, int kWarps>
__device__ __forceinline__ uint32_t rank_tile(RankSmem<kWarps> &S, const uint32_t (&key)[kItems], int shift,
                                              uint16_t (&rank)[kItems]) {
  static_assert(kItems * 32 * kWarps <= 65536, "16-bit ranks");
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned lt = (1u << lane) - 1u;
#pragma unroll
  for (int d = lane; d < kRadix; d += 32) S.whist[warp][d] = 0;
  __syncwarp();
#pragma unroll
  for (int i = 0; i < kItems; ++i) {
    const uint32_t d = (key[i] >> shift) & 0xffu;
    const unsigned peers = same_digit(d);
    const uint32_t before = S.whist[warp][d];
    rank[i] = (uint16_t)(before + __popc(peers & lt));
    __syncwarp();
    if ((peers & lt) == 0) S.whist[warp][d] = before + __popc(peers);
    __syncwarp();
  }
  __syncthreads();
  uint32_t tot = 0, incl = 0;
  if (tid < kRadix) {
#pragma unroll 4
    for (int w = 0; w < kWarps; ++w) {
      const uint32_t c = S.whist[w][tid];
      S.whist[w][tid] = tot;
      tot += c;
    }
    incl = tot;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    if (lane == 31) S.wsum[warp] = incl;
  }
  __syncthreads();
  if (tid < kRadix) {
    uint32_t s = incl - tot;
    for (int w = 0; w < warp; ++w) s += S.wsum[w];
    S.start[tid] = s;
#pragma unroll 4
    for (int w = 0; w < kWarps; ++w) S.whist[w][tid] += s;
  }
  __syncthreads();
  return tot;
}

// ------------------------------------------------------------ one CTA
constexpr int kBlockThreads = 1024;
constexpr int kBlockWarps = kBlockThreads / 32;
constexpr int kBlockItems = 8;
constexpr uint32_t kBlockMax = kBlockThreads * kBlockItems;

template <int kItems>
struct BlockSmem {
  RankSmem<kBlockWarps> r;
  uint32_t k[kBlockThreads * kItems], v[kBlockThreads * kItems];
};

// All of it in one CTA: n <= 1024 * kItems rows.
template <int kItems>
__global__ void __launch_bounds__(kBlockThreads) k_sort_block(Cols c, uint32_t n) {
  extern __shared__ __align__(16) unsigned char smem[];
  BlockSmem<kItems> &S = *reinterpret_cast<BlockSmem<kItems> *>(smem);
  __shared__ uint32_t s_diff;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t first = warp * (32 * kItems) + lane;
  uint32_t key[kItems], val[kItems];
  uint16_t rank[kItems];
  if (tid == 0) s_diff = 0;
  const uint32_t k0 = (uint32_t)c.in[c.key][0] ^ c.flip;
  uint32_t diff = 0;
#pragma unroll
  for (int i = 0; i < kItems; ++i) {
    const uint32_t p = first + 32 * i;
    key[i] = p < n ? (uint32_t)c.in[c.key][p] ^ c.flip : 0xffffffffu;  // behind all rows, stably
    val[i] = p < n ? carried(c, p) : 0;
    if (p < n) diff |= key[i] ^ k0;
  }
  __syncthreads();
  diff = __reduce_or_sync(0xffffffffu, diff);
  if (lane == 0 && diff) atomicOr(&s_diff, diff);
  __syncthreads();
  const uint32_t differ = s_diff;  // bits in which some keys differ
#pragma unroll 1
  for (int shift = 0; shift < 32; shift += 8) {
    if (!((differ >> shift) & 0xffu)) continue;
    rank_tile<kItems, kBlockWarps>(S.r, key, shift, rank);
#pragma unroll
    for (int i = 0; i < kItems; ++i) {
      const uint32_t p = S.r.whist[warp][(key[i] >> shift) & 0xffu] + rank[i];
      S.k[p] = key[i];
      S.v[p] = val[i];
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kItems; ++i) {
      key[i] = S.k[first + 32 * i];
      val[i] = S.v[first + 32 * i];
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < kItems; ++i)
    if (first + 32 * i < n) put_row(c, first + 32 * i, key[i], val[i]);
}

// ------------------------------------------------------------ many CTAs
constexpr int kThreads = 512;
constexpr int kSmallItems = 4, kBigItems = 12;  // rows per thread
constexpr int kWarps = kThreads / 32;

// The digits' counts, and what the passes do, worked out on the device by the
// histogram's last CTA.
struct SortState {
  uint32_t hist[4][kRadix];  // rows with the digit, then rows with a smaller one
  uint32_t done;
  uint32_t ticket[4];      // the passes' next tile
  int32_t src[4], dst[4];  // buffer a pass reads / writes: 0, 1; -1 the columns; src -2: the digit is skipped
  uint32_t pad[3];
};

constexpr int kHistThreads = 512;

__global__ void __launch_bounds__(kHistThreads)
    k_sort_hist(const int32_t *__restrict__ keys, uint32_t n, uint32_t flip, SortState *__restrict__ st) {
  __shared__ uint32_t h[4][kRadix];
  __shared__ uint32_t s_last, s_triv[4], wsum[32];
  const int tid = threadIdx.x, lane = tid & 31;
  for (int i = tid; i < 4 * kRadix; i += kHistThreads) (&h[0][0])[i] = 0;
  if (tid < 4) s_triv[tid] = 0;
  __syncthreads();
  const uint32_t stride = gridDim.x * kHistThreads;
  for (uint32_t b = blockIdx.x * kHistThreads + (tid & ~31); b < n; b += stride) {
    const uint32_t i = b + lane;
    const bool ok = i < n;
    const uint32_t k = (ok ? (uint32_t)__ldg(keys + i) : (uint32_t)__ldg(keys + b)) ^ flip;
    const uint32_t k0 = __shfl_sync(0xffffffffu, k, 0);
    const uint32_t diff = __reduce_or_sync(0xffffffffu, k ^ k0);
    const uint32_t rows = __popc(__ballot_sync(0xffffffffu, ok));
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      // a digit that the warp's rows share (high digits of small keys): one atomic
      if (!((diff >> (8 * p)) & 0xffu)) {
        if (lane == 0) atomicAdd(&h[p][(k0 >> (8 * p)) & 0xffu], rows);
      } else if (ok) {
        atomicAdd(&h[p][(k >> (8 * p)) & 0xffu], 1u);
      }
    }
  }
  __syncthreads();
  for (int i = tid; i < 4 * kRadix; i += kHistThreads) {
    const uint32_t x = (&h[0][0])[i];
    if (x) atomicAdd(&(&st->hist[0][0])[i], x);
  }
  __threadfence();
  __syncthreads();
  if (tid == 0) s_last = atomicAdd(&st->done, 1u) + 1 == gridDim.x;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  // exclusive sums of the four histograms, two digits at a time
  for (int p0 = 0; p0 < 4; p0 += 2) {
    const int p = p0 + (tid >> 8), d = tid & 255;
    const uint32_t x = *(volatile uint32_t *)&st->hist[p][d];
    if (x == n) s_triv[p] = 1;
    uint32_t incl = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    if (lane == 31) wsum[tid >> 5] = incl;
    __syncthreads();
    uint32_t s = incl - x;
    for (int w = (tid >> 8) * 8; w < (tid >> 5); ++w) s += wsum[w];
    st->hist[p][d] = s;  // this thread read it above
    __syncthreads();
  }
  if (tid == 0) {
    // the passes that run, in order; all keys equal: the last one does
    if (s_triv[0] && s_triv[1] && s_triv[2] && s_triv[3]) s_triv[3] = 0;
    int last = 3;
    while (s_triv[last]) --last;
    int at = -1;  // where the rows are
    for (int p = 0; p < 4; ++p) {
      st->src[p] = s_triv[p] ? -2 : at;
      if (s_triv[p]) continue;
      at = p == last ? -1 : at == 0 ? 1 : 0;
      st->dst[p] = at;
    }
  }
}

// One digit pass.  Tiles are taken by ticket, so every tile before this one
// has started; status[tile][digit] is published twice, with the tile's own
// count and then with the count of all rows up to it: {count, 2 flag bits}.
// W is 64 bits wide where a count may need more than 30 bits.
constexpr uint32_t kOwn = 1, kUpTo = 2, kGaveUp = 3;
constexpr int kLook = 4;

template <typename W>
__device__ __forceinline__ W ld_status(const W *p) {
  return *(const volatile W *)p;
}
template <typename W>
__device__ __forceinline__ void st_status(W *p, W v) {
  *(volatile W *)p = v;
}

template <int kItems, typename W>
__global__ void __launch_bounds__(kThreads, 2)
    k_sort_pass(Cols c, uint32_t n, int pass, SortState *__restrict__ st, uint32_t *__restrict__ k0,
                uint32_t *__restrict__ v0, uint32_t *__restrict__ k1, uint32_t *__restrict__ v1,
                W *__restrict__ status, uint32_t *dev_status) {
  constexpr uint32_t kTile = kThreads * kItems;
  extern __shared__ __align__(16) unsigned char smem[];
  RankSmem<kWarps> &S = *reinterpret_cast<RankSmem<kWarps> *>(smem);
  uint32_t *sk = reinterpret_cast<uint32_t *>(smem + sizeof(RankSmem<kWarps>)), *sv = sk + kTile;
  __shared__ uint32_t s_tile, s_out[kRadix];
  const int src = st->src[pass];
  if (src == -2) return;
  const int dst = st->dst[pass];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, shift = 8 * pass;
  if (tid == 0) s_tile = atomicAdd(&st->ticket[pass], 1u);
  __syncthreads();
  const uint32_t tile = s_tile, lo = tile * kTile, cnt = n - lo < kTile ? n - lo : kTile;
  const uint32_t first = warp * (32 * kItems) + lane;
  uint32_t key[kItems];
  uint16_t rank[kItems];
  const uint32_t *ik = src == 0 ? k0 : src == 1 ? k1 : reinterpret_cast<const uint32_t *>(c.in[c.key]);
  const uint32_t flip = src < 0 ? c.flip : 0;
#pragma unroll
  for (int i = 0; i < kItems; ++i) {
    const uint32_t p = first + 32 * i;
    key[i] = p < cnt ? __ldcs(ik + lo + p) ^ flip : 0xffffffffu;  // behind the last tile's rows
  }
  const uint32_t tot = rank_tile<kItems, kWarps>(S, key, shift, rank);
  // thread d < 256 publishes and looks back; the others go on
  W *mine = status + (uint64_t)tile * kRadix;
  if (tid < kRadix) st_status<W>(mine + tid, ((W)tot << 2) | (tile ? kOwn : kUpTo));
  const uint32_t *iv = src == 0 ? v0 : v1;
  uint32_t val[kItems];
#pragma unroll
  for (int i = 0; i < kItems; ++i) {
    const uint32_t p = first + 32 * i;
    val[i] = p < cnt ? (src < 0 ? carried(c, lo + p) : __ldcs(iv + lo + p)) : 0;
  }
#pragma unroll
  for (int i = 0; i < kItems; ++i) {
    const uint32_t p = S.whist[warp][(key[i] >> shift) & 0xffu] + rank[i];
    sk[p] = key[i];
    sv[p] = val[i];
  }
  bool ok = true;
  if (tid < kRadix) {
    // kLook predecessors are read at a time: one after the other, a walk over
    // the tiles in flight would cost an L2 round trip each
    uint32_t before = 0, spin = 0;
    const W *p = mine + tid - kRadix;  // the nearest predecessor not added yet
    for (uint32_t left = tile; left > 0;) {
      W w[kLook];
#pragma unroll
      for (int j = 0; j < kLook; ++j) w[j] = j < (int)left ? ld_status<W>(p - j * kRadix) : 0;
      uint32_t got = 0;
      bool open = true;
#pragma unroll
      for (int j = 0; j < kLook; ++j) {
        const uint32_t f = (uint32_t)(w[j] & 3);
        open = open && f != 0;
        if (open) {
          before += (uint32_t)(w[j] >> 2);
          ++got;
          ok = ok && f != kGaveUp;
          if (f != kOwn) {  // the rest is in it
            left = got;
            open = false;
          }
        }
      }
      if (!got && ++spin == kSpinLimit) {
        ok = false;
        break;
      }
      left -= got;
      p -= got * kRadix;
    }
    if (tile) st_status<W>(mine + tid, ok ? ((W)(before + tot) << 2) | kUpTo : (W)kGaveUp);
    s_out[tid] = st->hist[pass][tid] + before - S.start[tid];
  }
  if (__syncthreads_or(!ok)) {  // a predecessor never published: report and stop
    if (tid == 0) gbjd::latch(dev_status, GBJ_DEV_TIMEOUT);
    return;
  }
  uint32_t *ok_ = dst == 0 ? k0 : k1, *ov = dst == 0 ? v0 : v1;
#pragma unroll
  for (int i = 0; i < kItems; ++i) {
    const uint32_t p = tid + i * kThreads;
    if (p < cnt) {
      const uint32_t k = sk[p], o = s_out[(k >> shift) & 0xffu] + p;
      if (dst < 0) {
        put_row(c, o, k, sv[p]);
      } else {
        ok_[o] = k;
        ov[o] = sv[p];
      }
    }
  }
}

template <int kItems>
int sort_block(gbj_ctx *ctx, const Cols &c, uint32_t n, cudaStream_t s) {
  constexpr size_t smem = sizeof(BlockSmem<kItems>);
  GBJ_CHECK_CUDA(ctx, cudaFuncSetAttribute(k_sort_block<kItems>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)smem));
  k_sort_block<kItems><<<1, kBlockThreads, smem, s>>>(c, n);
  return after_launch(ctx, "k_sort_block", s);
}

template <int kItems, typename W>
int sort_tiles(gbj_ctx *ctx, const Cols &c, uint32_t n, cudaStream_t s) {
  constexpr uint32_t kTile = kThreads * kItems;
  constexpr size_t smem = sizeof(RankSmem<kWarps>) + (size_t)kTile * 8;
  const uint32_t ntiles = (n + kTile - 1) / kTile;
  Scratch scratch(ctx, s);
  uint32_t *buf;
  char *zero;  // counters and the passes' status words, cleared together
  const uint64_t words = (uint64_t)ntiles * kRadix, zbytes = sizeof(SortState) + 4 * words * sizeof(W);
  GBJ_TRY(scratch.get(4 * (uint64_t)n, &buf));
  GBJ_TRY(scratch.get(zbytes, &zero));
  GBJ_CHECK_CUDA(ctx, cudaMemsetAsync(zero, 0, zbytes, s));
  SortState *st = reinterpret_cast<SortState *>(zero);
  W *status = reinterpret_cast<W *>(zero + sizeof(SortState));
  const unsigned hgrid = (unsigned)std::min<uint64_t>((n + 4 * kHistThreads - 1) / (4 * kHistThreads),
                                                      (uint64_t)ctx->sm_count * 4);
  k_sort_hist<<<hgrid, kHistThreads, 0, s>>>(c.in[c.key], n, c.flip, st);
  GBJ_TRY(after_launch(ctx, "k_sort_hist", s));
  auto kern = k_sort_pass<kItems, W>;
  GBJ_CHECK_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  for (int pass = 0; pass < 4; ++pass) {
    kern<<<ntiles, kThreads, smem, s>>>(c, n, pass, st, buf, buf + n, buf + 2 * (uint64_t)n,
                                        buf + 3 * (uint64_t)n, status + pass * words, ctx->d_status);
    GBJ_TRY(after_launch(ctx, "k_sort_pass", s));
  }
  return GBJ_OK;
}

}  // namespace

extern "C" int gbj_sort_by_key(gbj_ctx *ctx, const int32_t *const *d_cols, int32_t n_cols, uint64_t n,
                               int32_t key_col, int32_t descending, int32_t *const *d_out_cols, void *stream) {
  if (!ctx) return GBJ_ERR_INVALID;
  if (n_cols < 1 || n_cols > kMaxCols || key_col < 0 || key_col >= n_cols || !d_cols || !d_out_cols)
    return set_error(ctx, GBJ_ERR_INVALID, "sort: need 1..16 columns and a key column among them");
  if (n >= (1ull << 31)) return set_error(ctx, GBJ_ERR_INVALID, "sort: n >= 2^31");
  for (int j = 0; j < n_cols; ++j)
    if (n && (!d_cols[j] || !d_out_cols[j])) return set_error(ctx, GBJ_ERR_INVALID, "sort: null column");
  cudaStream_t s = pick_stream(ctx, stream);
  prof_mark(ctx, s);
  if (n == 0) return GBJ_OK;
  Cols c{};
  c.n = n_cols;
  c.key = key_col;
  c.flip = descending ? 0x7fffffffu : 0x80000000u;
  for (int j = 0; j < n_cols; ++j) {
    c.in[j] = d_cols[j];
    c.out[j] = d_out_cols[j];
  }
  // one CTA while that is faster than five launches over several (8192 rows:
  // 28 us against 42); tiles of 2048 rows while tiles of 6144 would leave SMs
  // idle (300,000 rows: 53 us against 61; 2^20 rows: 90 against 83; 2^22: 231
  // against 171)
  if (n <= kBlockThreads) return sort_block<1>(ctx, c, (uint32_t)n, s);
  if (n <= 4 * kBlockThreads) return sort_block<4>(ctx, c, (uint32_t)n, s);
  if (n <= kBlockMax) return sort_block<kBlockItems>(ctx, c, (uint32_t)n, s);
  if (n < (1u << 20)) {
    const int rc = sort_tiles<kSmallItems, uint32_t>(ctx, c, (uint32_t)n, s);
    if (rc != GBJ_ERR_OOM) return rc;
    // a pool without room for the small tiles' status words: a third as many
  }
  if (n < (1u << 30)) return sort_tiles<kBigItems, uint32_t>(ctx, c, (uint32_t)n, s);
  return sort_tiles<kBigItems, unsigned long long>(ctx, c, (uint32_t)n, s);
}
