// Non-partitioned hash join: build, probe with fused aggregate, probe with
// pair materialisation; plus the column helpers (reduce, gather, select).
//
// Replaces the JIT'd build / probe loops of HashJoinChained and
// GpuHashJoinChained (core/olap/lib/operators/hash-join-chained.cpp:262-566,
// core/olap/lib/operators/gpu/gpu-hash-join-chained.cpp:31-73).  The
// reference chains entries behind a head array; here the table is an array
// of 32-byte buckets of four slots {key, payload or row + 1} sized
// to a power of two with load factor <= 1/2, so a probe is one L2 sector in
// the common case and the table for a 2^20-row build side (16 MiB) stays
// resident in the 129 MB L2 while the probe side streams from HBM.  The
// allocation-free entry point keeps a plain open-addressing array of 64-bit
// {key, row + 1} slots in a static device array.
// Semantics are the reference's: every build row is inserted (duplicates
// allowed) and a probe row meets every build row with an equal key.
#include <algorithm>

#include "compact.cuh"
#include "gbj_internal.cuh"

using namespace gbj;

namespace {

constexpr int kThreads = 512;

__device__ __forceinline__ uint64_t make_slot(int32_t key, uint64_t row) {
  return ((row + 1) << 32) | (uint32_t)key;
}

// Build of the allocation-free entry point's table: 64-bit slots {key,
// row + 1}, 0 = empty, linear probing; meta[0] = 1 once a duplicate build key
// was seen (probes may then not stop at the first match).  The table has at
// least 2n slots, so every row finds one.
__global__ void __launch_bounds__(kThreads)
    k_join_build(const int32_t *__restrict__ keys, uint64_t n, uint64_t *__restrict__ slots, uint64_t mask,
                 uint32_t *__restrict__ meta) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  bool dup = false;
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += stride) {
    const int32_t k = keys[i];
    const uint64_t entry = make_slot(k, i);
    uint64_t h = gbjd::fmix32((uint32_t)k) & mask;
    for (uint64_t probe = 0; probe <= mask; ++probe) {
      unsigned long long *w = reinterpret_cast<unsigned long long *>(slots) + h;
      uint64_t cur = *(volatile uint64_t *)w;
      if (cur == 0) {
        cur = atomicCAS(w, 0ull, (unsigned long long)entry);
        if (cur == 0) break;
      }
      dup |= ((int32_t)(uint32_t)cur == k);
      h = (h + 1) & mask;
    }
  }
  if (dup) meta[0] = 1;
}

enum : int { kAggGeneric = 0, kAggCountXor = 1, kAggCountProduct = 2 };

// Probe with fused aggregate over the allocation-free entry point's table.
// Eight probe keys per thread walk their slot chains in lockstep: every
// round checks the slot each still-open probe holds and issues the next
// slot loads of all of them together, so a warp waits for the longest chain
// once per round instead of once per probe and keeps up to eight L2
// requests per thread in flight.  kAgg selects a specialised accumulator
// for the two aggregate lists the workloads use.
template <bool kVec, int kAgg>
__global__ void __launch_bounds__(kThreads)
    k_join_probe_agg(const int32_t *__restrict__ keys, const int32_t *__restrict__ pay, uint64_t n,
                     const uint64_t *__restrict__ slots, uint64_t mask, const int32_t *__restrict__ bpay,
                     const uint32_t *__restrict__ meta, gbj::AggSpec spec, int64_t *out) {
  __shared__ int64_t red[32 * GBJ_MAX_AGGS];
  gbjd::Acc acc;
  acc.init(spec);
  int64_t a_cnt = 0, a_sum = 0;
  const bool unique = meta[0] == 0;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  // a slot is {key (low word), row + 1 (high word)}; row + 1 == 0: empty
  auto skey = [](uint64_t e) { return (int32_t)(uint32_t)e; };
  auto srow1 = [](uint64_t e) { return (uint32_t)(e >> 32); };
  auto match = [&](int32_t k, int64_t pv, uint64_t prow, uint64_t e) {
    const uint32_t r = srow1(e) - 1;
    if (kAgg == kAggCountXor) {
      a_cnt += 1;
      a_sum += (int64_t)r ^ (int64_t)prow;
    } else {
      const int64_t bv = bpay ? (int64_t)__ldg(&bpay[r]) : 0;
      if (kAgg == kAggCountProduct) {
        a_cnt += 1;
        a_sum += bv * pv;
      } else {
        acc.update(spec, k, bv, pv, r, prow);
      }
    }
  };
  uint64_t done = 0;
  if (kVec) {
    const uint64_t n8 = n / 8;
    const int4 *k4 = reinterpret_cast<const int4 *>(keys);
    const int4 *p4 = reinterpret_cast<const int4 *>(pay);
    for (uint64_t q = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; q < n8; q += stride) {
      const int4 ka = __ldcs(k4 + 2 * q), kb = __ldcs(k4 + 2 * q + 1);
      int4 pa = make_int4(0, 0, 0, 0), pb = pa;
      if (pay) {
        pa = __ldcs(p4 + 2 * q);
        pb = __ldcs(p4 + 2 * q + 1);
      }
      const int32_t kk[8] = {ka.x, ka.y, ka.z, ka.w, kb.x, kb.y, kb.z, kb.w};
      const int32_t pp[8] = {pa.x, pa.y, pa.z, pa.w, pb.x, pb.y, pb.z, pb.w};
      // slot indices fit 32 bits: the table holds at most 2^21 slots
      const uint32_t m32 = (uint32_t)mask;
      uint32_t h[8];
      uint64_t e[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        h[j] = gbjd::fmix32((uint32_t)kk[j]) & m32;
        e[j] = __ldg(slots + h[j]);
      }
      uint32_t open = 0xffu;  // probes whose chain is not finished
      for (uint64_t step = 0; open && step <= mask; ++step) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          if (open >> j & 1u) {
            if (srow1(e[j]) == 0) {
              open &= ~(1u << j);
            } else if (skey(e[j]) == kk[j]) {
              match(kk[j], pp[j], q * 8 + j, e[j]);
              if (unique) open &= ~(1u << j);
            }
          }
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          if (open >> j & 1u) {
            h[j] = (h[j] + 1) & m32;
            e[j] = __ldg(slots + h[j]);
          }
        }
      }
    }
    done = n8 * 8;
  }
  // rows the vector loop did not cover (all of them without kVec)
  for (uint64_t i = done + blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += stride) {
    const int32_t k = keys[i];
    const int64_t pv = pay ? pay[i] : 0;
    uint64_t h = gbjd::fmix32((uint32_t)k) & mask;
    for (uint64_t step = 0; step <= mask; ++step) {
      const uint64_t e = __ldg(slots + h);
      if (srow1(e) == 0) break;
      if (skey(e) == k) {
        match(k, pv, i, e);
        if (unique) break;
      }
      h = (h + 1) & mask;
    }
  }
  if (kAgg != kAggGeneric) {
    acc.v[0] = a_cnt;
    acc.v[1] = a_sum;
  }
  gbjd::block_flush(spec, acc, red, out);
}

// ------------------------------------------------ bucketed join table
// The table gbj_join_build makes: buckets of four slots, 32 bytes each -- a
// slot is {key, value} (the build payload, or row + 1 when the build side has
// none) and is claimed by one 64-bit CAS -- so a probe reads one L2 sector per
// bucket and finds the key and its payload without a second, dependent load.  Keys are stored
// xor INT32_MIN, so the all-zero word of a cleared table marks an empty
// slot; build rows whose key is INT32_MIN (stored word 0) go to a side list
// instead.  A table with a payload keeps row + 1 of every slot in a
// parallel array of 16-byte bucket rows, read only when an aggregate or the
// pair output needs the build row.  A key sits in its home bucket (fmix32
// bits) or, when that bucket was full at insert time, in a later one; a
// probe stops at the first bucket with an empty slot.
// Probe shape: kJbGroup probes per thread at a time (a multiple of 4), and
// the CTAs per SM the specialised probe kernels are compiled for (512
// threads each).  Measured on GB300 for the plain join (2^20 build rows,
// 2^24 probes): 4 probes x 2 CTAs ahead of 8 x 2 (register spills), 8 x 1
// and 4 x 3.
#ifndef GBJ_JB_MIN_BLOCKS
#define GBJ_JB_MIN_BLOCKS 2
#endif
#ifndef GBJ_JB_GROUP
#define GBJ_JB_GROUP 4
#endif
constexpr int kJbGroup = GBJ_JB_GROUP;
// In memory: {key ^ INT32_MIN (0 = empty), payload or row + 1} four times.
struct __align__(32) JBucket {
  int4 k, x;  // as loaded
};

// One bucket in a single 256-bit load (ld.global.nc.v8, sm_100 and later):
// one L2 request per bucket instead of two.
__device__ __forceinline__ JBucket ld_bucket(const JBucket *p) {
  JBucket r;
  asm("ld.global.nc.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
      : "=r"(r.k.x), "=r"(r.x.x), "=r"(r.k.y), "=r"(r.x.y), "=r"(r.k.z), "=r"(r.x.z), "=r"(r.k.w), "=r"(r.x.w)
      : "l"(p));
  return r;
}
constexpr int32_t kKeyFlip = INT32_MIN;

__device__ __forceinline__ int32_t lane4(const int4 &v, uint32_t i) {
  return i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w;
}
__device__ __forceinline__ uint32_t hits4(const int4 &k, int32_t kf) {
  return (uint32_t)(k.x == kf) | ((uint32_t)(k.y == kf) << 1) | ((uint32_t)(k.z == kf) << 2) |
         ((uint32_t)(k.w == kf) << 3);
}
__device__ __forceinline__ bool room4(const int4 &k) { return (k.x == 0) | (k.y == 0) | (k.z == 0) | (k.w == 0); }

__device__ __forceinline__ unsigned long long jb_word(int32_t kf, int32_t value) {
  return ((unsigned long long)(uint32_t)value << 32) | (uint32_t)kf;
}
// A bucket's empty slots while rows are being placed; dup: one of the others has
// key kf.
__device__ __forceinline__ uint32_t jb_empty(const unsigned long long *bucket, int32_t kf, bool &dup) {
  unsigned long long w[4];
  asm volatile("ld.relaxed.gpu.global.v4.u64 {%0, %1, %2, %3}, [%4];"
               : "=l"(w[0]), "=l"(w[1]), "=l"(w[2]), "=l"(w[3])
               : "l"(bucket)
               : "memory");
  uint32_t m = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    m |= (uint32_t)(w[i] == 0) << i;
    dup |= (int32_t)(uint32_t)w[i] == kf;
  }
  return m;
}

// A row's slot in a table at `bk`: it claims the first free slot of its home
// bucket, starting at a slot chosen by the top hash bits, then of the following
// buckets; a bucket is passed when it is full.  All lanes call it, `todo` with a
// row; rows may be null.  False: full.
//
// The home slot is claimed unseen, which is all there is to do for most rows;
// after that a bucket is read before one slot of it is claimed: copies of a key
// ask for the same slots at the same time, and a claim that fails costs as much
// as one that does not.  Where a warp has kTogether copies of one key and more,
// those go on together, one read for all of them and each at another slot.
// Measured on GB300, build with its clear, us, with a claim for every slot on the
// way / now: 4 M rows, 1, 2, 3 and 16 a key 139 / 138, 238 / 181, 310 / 207, 1046
// / 416; 10,000 rows with 16, 2 and 1 keys 792 / 710, 3115 / 1398, 8836 / 2061.
constexpr int kTogether = 8;

__device__ __forceinline__ bool jb_place(unsigned long long *bk, int32_t *rows, uint32_t bmask, bool todo, uint32_t h,
                                         int32_t kf, int32_t value, int32_t row1, bool &dup) {
  uint32_t b = h & bmask;
  const uint32_t o = h >> 30;  // start slot (high bits, independent of the bucket for 2^30 buckets or fewer)
  const unsigned long long word = jb_word(kf, value);
  auto claim = [&](uint32_t bucket, uint32_t i) {
    const uint64_t sl = 4ull * bucket + i;
    const unsigned long long old = atomicCAS(&bk[sl], 0ull, word);
    if (old == 0) {
      if (rows) rows[sl] = row1;
      todo = false;
    }
    dup |= (int32_t)(uint32_t)old == kf;  // no row's kf is 0
  };
  if (todo) claim(b, o);
  const int lane = threadIdx.x & 31;
  // a bucket is looked at again only when another row took a slot meanwhile
  const uint64_t most = 5ull * (bmask + 1ull);
  for (;;) {
    const unsigned left = __ballot_sync(0xffffffffu, todo);
    if (__popc(left) < kTogether) break;
    const int32_t lk = __shfl_sync(0xffffffffu, kf, __ffs(left) - 1);
    uint32_t lb = __shfl_sync(0xffffffffu, b, __ffs(left) - 1);
    unsigned group = __ballot_sync(0xffffffffu, todo && kf == lk);
    if (__popc(group) < kTogether) break;
    for (uint64_t looks = 0; group; ++looks) {
      if (looks == most) return false;
      const uint32_t m = jb_empty(bk + 4ull * lb, lk, dup);
      dup |= __popc(group) > 1;
      if (todo && kf == lk) {
        const uint32_t i = __fns(m, 0, __popc(group & ((1u << lane) - 1u)) + 1);
        if (i < 4) claim(lb, i);
      }
      if (__popc(group) >= __popc(m)) lb = (lb + 1) & bmask;
      group = __ballot_sync(0xffffffffu, todo && kf == lk);
    }
  }
  for (uint64_t looks = 0; todo; ++looks) {
    if (looks == most) return false;
    const uint32_t m = jb_empty(bk + 4ull * b, kf, dup);
    if (m) claim(b, (o + __ffs((m | m << 4) >> o) - 1) & 3u);
    else b = (b + 1) & bmask;
  }
  return true;
}

// meta[0]: a duplicate build key was seen; meta[1]: side-list length.  One
// row at a time per thread: two or four claims in flight together were slower
// (2^20 rows 48, 50, 77 us; 2^22 rows 178, 205, 323).
__global__ void __launch_bounds__(kThreads)
    k_jb_build(const int32_t *__restrict__ keys, const int32_t *__restrict__ payload, uint64_t n,
               unsigned long long *__restrict__ bk, int32_t *__restrict__ rows, uint32_t bmask,
               uint32_t *__restrict__ meta, int32_t *__restrict__ side, uint32_t *status) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  bool dup = false;
  const int lane = threadIdx.x & 31;
  for (uint64_t base = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x - lane; base < n; base += stride) {
    const uint64_t i = base + lane;
    const bool in = i < n;
    const int32_t key = in ? keys[i] : 0, kf = key ^ kKeyFlip;
    const int32_t val = in && payload ? payload[i] : (int32_t)(i + 1);
    if (in && kf == 0) side[atomicAdd(&meta[1], 1u)] = (int32_t)i;  // INT32_MIN: the side list
    if (!jb_place(bk, rows, bmask, in && kf != 0, gbjd::fmix32((uint32_t)key), kf, val, (int32_t)(i + 1), dup))
      gbjd::latch(status, GBJ_DEV_CAPACITY);
  }
  if (dup) meta[0] = 1;
}

// A small table (at most kSmallSlots slots) in one CTA: built in shared memory
// and written out whole, so that it needs no clearing before it and no chain
// of L2 atomics.  A row takes a slot with one addition to its bucket's count (a
// claim of each slot by a 64-bit CAS on shared memory made copies of a key wait
// for one another: 4000 rows with 1, 2 and 16 keys 4260, 6198, 988 us, now 383,
// 717, 166), and copies are looked for when the table is complete.  Build and
// clear, 100, 1000 and 4000 unique rows with payloads, by events around the call:
// 16, 16, 15 us, cleared and built in L2 22, 25, 27.
constexpr int kSmallThreads = 1024;
constexpr uint32_t kSmallSlots = 8192;

__global__ void __launch_bounds__(kSmallThreads)
    k_jb_build_small(const int32_t *__restrict__ keys, const int32_t *__restrict__ payload, uint32_t n,
                     uint4 *__restrict__ bk, uint4 *__restrict__ rows, uint32_t slots, uint32_t *__restrict__ meta,
                     int32_t *__restrict__ side) {
  extern __shared__ __align__(16) unsigned char smem[];
  unsigned long long *s_bk = reinterpret_cast<unsigned long long *>(smem);
  int32_t *s_rows = rows ? reinterpret_cast<int32_t *>(s_bk + slots) : nullptr;
  __shared__ uint32_t s_meta[2];
  constexpr int kPer = kSmallSlots / 2 / kSmallThreads;  // rows of a thread, at most
  int32_t key[kPer], val[kPer];
#pragma unroll
  for (int u = 0; u < kPer; ++u) {
    const uint32_t i = threadIdx.x + u * kSmallThreads;
    key[u] = i < n ? __ldg(keys + i) : 0;
    val[u] = payload ? (i < n ? __ldg(payload + i) : 0) : (int32_t)(i + 1);
  }
  const uint32_t nbk = slots / 4, words = slots * (rows ? 12 : 8) / 16;
  uint32_t *s_fill = reinterpret_cast<uint32_t *>(smem + words * 16);  // rows that asked for the bucket
  for (uint32_t i = threadIdx.x; i < words + nbk / 4; i += kSmallThreads)
    reinterpret_cast<uint4 *>(smem)[i] = make_uint4(0, 0, 0, 0);
  if (threadIdx.x < 2) s_meta[threadIdx.x] = 0;
  __syncthreads();
  uint32_t at[kPer];  // the row's bucket
#pragma unroll
  for (int u = 0; u < kPer; ++u) {
    const uint32_t i = threadIdx.x + u * kSmallThreads;
    const int32_t kf = key[u] ^ kKeyFlip;
    at[u] = gbjd::fmix32((uint32_t)key[u]) & (nbk - 1);
    if (i >= n) continue;
    if (kf == 0) {
      side[atomicAdd(&s_meta[1], 1u)] = (int32_t)i;
      continue;
    }
    for (;;) {  // ends: the table has 2 n slots
      if (*(volatile uint32_t *)&s_fill[at[u]] < 4) {
        const uint32_t j = atomicAdd(&s_fill[at[u]], 1u);
        if (j < 4) {
          s_bk[4 * at[u] + j] = jb_word(kf, val[u]);
          if (rows) s_rows[4 * at[u] + j] = (int32_t)(i + 1);
          break;
        }
      }
      at[u] = (at[u] + 1) & (nbk - 1);
    }
  }
  __syncthreads();
  // copies of a key: two in one bucket, or one in a bucket that another passed
  bool dup = false;
#pragma unroll
  for (int u = 0; u < kPer; ++u) {
    const int32_t kf = key[u] ^ kKeyFlip;
    for (uint32_t b = gbjd::fmix32((uint32_t)key[u]) & (nbk - 1);
         threadIdx.x + u * kSmallThreads < n && kf != 0 && !dup && b != at[u]; b = (b + 1) & (nbk - 1)) {
#pragma unroll
      for (int j = 0; j < 4; ++j) dup |= (int32_t)(uint32_t)s_bk[4 * b + j] == kf;
    }
  }
  for (uint32_t b = threadIdx.x; b < nbk; b += kSmallThreads) {
    const uint4 x = reinterpret_cast<const uint4 *>(s_bk)[2 * b], y = reinterpret_cast<const uint4 *>(s_bk)[2 * b + 1];
    bk[2 * b] = x;
    bk[2 * b + 1] = y;
    // {key, value} twice each; 0 is no key
    dup |= (x.x == x.z && x.x) || (x.x == y.x && x.x) || (x.x == y.z && x.x) || (x.z == y.x && x.z) ||
           (x.z == y.z && x.z) || (y.x == y.z && y.x);
  }
  if (rows)
    for (uint32_t i = threadIdx.x; i < nbk; i += kSmallThreads) rows[i] = reinterpret_cast<const uint4 *>(s_rows)[i];
  if (__syncthreads_or(dup) && threadIdx.x == 0) s_meta[0] = 1;
  __syncthreads();
  if (threadIdx.x < 2) meta[threadIdx.x] = s_meta[threadIdx.x];
}

// Probe with fused aggregate over the bucketed table.  A probe visits its
// home bucket and folds every slot whose key matches into the aggregate
// without branching (a count of the matches and a select-and-sum of their
// values, for the two specialised aggregate lists); it moves on to the
// next bucket only when the bucket is full and either has no match or the
// build keys are not unique -- the rare case, taken out of line.  Each
// thread handles kJbGroup probes at a time: their bucket loads (one 256-bit
// load each) are issued together, and the next group's probe keys and
// payloads are loaded while they are in flight.  kPay: the values are build
// payloads and build rows come from the row array.
template <bool kVec, int kAgg, bool kPay>
__global__ void __launch_bounds__(kThreads, GBJ_JB_MIN_BLOCKS)
    k_jb_probe_agg(const int32_t *__restrict__ keys, const int32_t *__restrict__ pay, uint64_t n,
                   const JBucket *__restrict__ bk, const int4 *__restrict__ rows, uint32_t bmask,
                   const int32_t *__restrict__ bpay, const uint32_t *__restrict__ meta,
                   const int32_t *__restrict__ side, gbj::AggSpec spec, int64_t *out) {
  __shared__ int64_t red[32 * GBJ_MAX_AGGS];
  static_assert(kAgg != kAggGeneric, "other aggregate lists: k_jb_probe_list");
  int64_t a_cnt = 0, a_sum = 0;
  const bool unique = meta[0] == 0;
  const uint32_t nside = meta[1];
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  // folds the matching slots of bucket b (contents e) into the aggregate;
  // returns the number of matches
  auto visit = [&](int32_t kf, int64_t pv, uint64_t prow, uint32_t b, const JBucket &e) -> uint32_t {
    const bool m0 = e.k.x == kf, m1 = e.k.y == kf, m2 = e.k.z == kf, m3 = e.k.w == kf;
    const uint32_t c = (uint32_t)m0 + (uint32_t)m1 + (uint32_t)m2 + (uint32_t)m3;
    if (kAgg == kAggCountProduct) {
      a_cnt += c;
      if (kPay)
        a_sum += ((int64_t)(m0 ? e.x.x : 0) + (m1 ? e.x.y : 0) + (int64_t)(m2 ? e.x.z : 0) + (m3 ? e.x.w : 0)) * pv;
    } else if (kAgg == kAggCountXor && !kPay) {
      a_cnt += c;
      const int64_t pr = (int64_t)prow;
      a_sum += (m0 ? ((int64_t)(e.x.x - 1) ^ pr) : 0) + (m1 ? ((int64_t)(e.x.y - 1) ^ pr) : 0) +
               (m2 ? ((int64_t)(e.x.z - 1) ^ pr) : 0) + (m3 ? ((int64_t)(e.x.w - 1) ^ pr) : 0);
    } else if (c) {
      const int4 rw = kPay ? __ldg(&rows[b]) : e.x;
      uint32_t hits = (uint32_t)m0 | ((uint32_t)m1 << 1) | ((uint32_t)m2 << 2) | ((uint32_t)m3 << 3);
      while (hits) {
        const uint32_t idx = __ffs(hits) - 1;
        a_cnt += 1;
        a_sum += (int64_t)(lane4(rw, idx) - 1) ^ (int64_t)prow;
        hits &= hits - 1;
      }
    }
    return c;
  };
  // the buckets after a full home bucket (out of line, rare)
  auto walk = [&](int32_t kf, int64_t pv, uint64_t prow, uint32_t b, uint32_t matched) {
    for (uint32_t step = 1; step <= bmask; ++step) {
      b = (b + 1) & bmask;
      const JBucket e = ld_bucket(&bk[b]);
      matched += visit(kf, pv, prow, b, e);
      if (room4(e.k) || (unique && matched)) return;
    }
  };
  // a probe key INT32_MIN meets the side list
  auto side_probe = [&](int64_t pv, uint64_t prow) {
    for (uint32_t s = 0; s < nside; ++s) {
      const int32_t r = side[s];
      a_cnt += 1;
      if (kAgg == kAggCountProduct) a_sum += (kPay ? (int64_t)bpay[r] : 0) * pv;
      else a_sum += (int64_t)r ^ (int64_t)prow;
    }
  };
  auto finish = [&](int32_t k, int64_t pv, uint64_t prow, uint32_t b, const JBucket &e) {
    const int32_t kf = k ^ kKeyFlip;
    if (kf == 0) {
      side_probe(pv, prow);
      return;
    }
    const uint32_t c = visit(kf, pv, prow, b, e);
    if (!room4(e.k) && !(unique && c)) walk(kf, pv, prow, b, c);
  };
  uint64_t done = 0;
  if (kVec) {
    constexpr int G = kJbGroup;  // probes per thread at a time (a multiple of 4)
    const uint64_t ng = n / G;
    const int4 *k4 = reinterpret_cast<const int4 *>(keys);
    const int4 *p4 = reinterpret_cast<const int4 *>(pay);
    int4 nk[G / 4], np[G / 4];
    auto load_group = [&](uint64_t qq) {
#pragma unroll
      for (int v = 0; v < G / 4; ++v) {
        nk[v] = __ldcs(k4 + (G / 4) * qq + v);
        np[v] = pay ? __ldcs(p4 + (G / 4) * qq + v) : make_int4(0, 0, 0, 0);
      }
    };
    uint64_t q = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (q < ng) load_group(q);
    for (; q < ng; q += stride) {
      int32_t kk[G], pp[G];
#pragma unroll
      for (int v = 0; v < G / 4; ++v) {
        kk[4 * v] = nk[v].x, kk[4 * v + 1] = nk[v].y, kk[4 * v + 2] = nk[v].z, kk[4 * v + 3] = nk[v].w;
        pp[4 * v] = np[v].x, pp[4 * v + 1] = np[v].y, pp[4 * v + 2] = np[v].z, pp[4 * v + 3] = np[v].w;
      }
      uint32_t b[G];
      JBucket e[G];
#pragma unroll
      for (int j = 0; j < G; ++j) {
        b[j] = gbjd::fmix32((uint32_t)kk[j]) & bmask;
        e[j] = ld_bucket(&bk[b[j]]);
      }
      if (q + stride < ng) load_group(q + stride);
#pragma unroll
      for (int j = 0; j < G; ++j) finish(kk[j], pp[j], q * G + j, b[j], e[j]);
    }
    done = ng * G;
  }
  for (uint64_t i = done + blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += stride) {
    const int32_t k = keys[i];
    const uint32_t b = gbjd::fmix32((uint32_t)k) & bmask;
    finish(k, pay ? pay[i] : 0, i, b, ld_bucket(&bk[b]));
  }
  gbjd::Acc acc;
  acc.init(spec);
  acc.v[0] = a_cnt;
  acc.v[1] = a_sum;
  gbjd::after_init();
  gbjd::block_flush(spec, acc, red, out);
}

// Probes whose home bucket does not end them: they look at their next bucket
// 32 at a time.
template <typename X>
struct WalkRing {
  int32_t kf[128];
  uint32_t b[128];  // the next bucket to look at
  X x[128];         // the probe's payload (product list) or row (xor list)
};

// The same for a table that is more than a third full, where a tenth of the
// probes and more go on to the next bucket.  Taken where the need is found,
// those walks leave 20 of 32 lanes active; here they wait in the warp's ring
// and 32 of them look at their next bucket together.  Four probes a lane are in
// flight as above, in tiles of 128 a warp.  Bound by the buckets' way from L2
// and by issue.  Measured on GB300, 2^24 probes, walks alone / ring, us: 2^20
// dense keys 102 / 84, 2^20 keys without a pattern and half the probes without a
// match 132 / 93, two rows a key 290 / 166, three and the xor list 459 / 207.
// In a table that is less full its instructions and its shared memory, which
// the first-level cache then lacks, only cost (2^26 probes: 5000 rows,
// load 0.3, 199 / 248; 20,000 rows, 0.31, 270 / 274; 60,000 rows, 0.46, 333 /
// 287).
template <bool kVec, int kAgg, bool kPay>
__global__ void __launch_bounds__(kThreads, GBJ_JB_MIN_BLOCKS)
    k_jb_probe_ring(const int32_t *__restrict__ keys, const int32_t *__restrict__ pay, uint64_t n,
                    const JBucket *__restrict__ bk, const int4 *__restrict__ rows, uint32_t bmask,
                    const int32_t *__restrict__ bpay, const uint32_t *__restrict__ meta,
                    const int32_t *__restrict__ side, gbj::AggSpec spec, int64_t *out) {
  __shared__ int64_t red[32 * GBJ_MAX_AGGS];
  using X = std::conditional_t<kAgg == kAggCountProduct, int32_t, int64_t>;
  __shared__ WalkRing<X> s_ring[kThreads / 32];
  static_assert(kAgg != kAggGeneric, "other aggregate lists: k_jb_probe_list");
  constexpr int G = kJbGroup;  // probes per lane at a time
  static_assert(G == 4, "one 16-byte load a lane");
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  WalkRing<X> &ring = s_ring[threadIdx.x >> 5];
  int64_t a_cnt = 0, a_sum = 0;
  const bool unique = meta[0] == 0;
  const uint32_t nside = meta[1];
  // folds the matching slots of bucket b (contents e) into the aggregate;
  // returns the number of matches
  auto visit = [&](int32_t kf, X x, uint32_t b, const JBucket &e) -> uint32_t {
    const bool m0 = e.k.x == kf, m1 = e.k.y == kf, m2 = e.k.z == kf, m3 = e.k.w == kf;
    const uint32_t c = (uint32_t)m0 + (uint32_t)m1 + (uint32_t)m2 + (uint32_t)m3;
    a_cnt += c;
    if (kAgg == kAggCountProduct) {
      if (kPay)
        a_sum += ((int64_t)(m0 ? e.x.x : 0) + (m1 ? e.x.y : 0) + (int64_t)(m2 ? e.x.z : 0) + (m3 ? e.x.w : 0)) * x;
    } else if (c) {
      const int4 rw = kPay ? __ldg(&rows[b]) : e.x;
      a_sum += (m0 ? ((int64_t)(rw.x - 1) ^ x) : 0) + (m1 ? ((int64_t)(rw.y - 1) ^ x) : 0) +
               (m2 ? ((int64_t)(rw.z - 1) ^ x) : 0) + (m3 ? ((int64_t)(rw.w - 1) ^ x) : 0);
    }
    return c;
  };
  // a probe key INT32_MIN meets the side list
  auto side_probe = [&](X x) {
    for (uint32_t s = 0; s < nside; ++s) {
      const int32_t r = side[s];
      a_cnt += 1;
      if (kAgg == kAggCountProduct) a_sum += (kPay ? (int64_t)bpay[r] : 0) * x;
      else a_sum += (int64_t)r ^ x;
    }
  };
  uint32_t qn = 0, qh = 0;  // the ring's length and head (warp-uniform)
  auto push = [&](bool yes, int32_t kf, X x, auto b) {
    const unsigned bal = __ballot_sync(0xffffffffu, yes);
    if (bal == 0) return;
    if (yes) {
      const uint32_t p = (qh + qn + __popc(bal & lt)) & 127u;
      ring.kf[p] = kf;
      ring.b[p] = b();
      ring.x[p] = x;
    }
    qn += __popc(bal);
  };
  auto home = [&](int32_t kf) { return gbjd::fmix32((uint32_t)(kf ^ kKeyFlip)) & bmask; };
  // the next bucket of the first c (<= 32) probes of the ring.  With unique
  // keys those have no match yet, with others a match does not end them; the
  // table is at most half full, and all of it is the most they look at.
  auto walk = [&](uint32_t c) {
    __syncwarp();
    const bool mine = (uint32_t)lane < c;
    const uint32_t p = (qh + lane) & 127u;
    const int32_t kf = mine ? ring.kf[p] : 0;
    const uint32_t b = mine ? ring.b[p] : 0, next = (b + 1) & bmask;
    const X x = mine ? ring.x[p] : 0;
    __syncwarp();  // read before any of them is written again
    qh = (qh + c) & 127u;
    qn -= c;
    bool on = false;
    if (mine) {
      const JBucket e = ld_bucket(&bk[b]);
      const uint32_t m = visit(kf, x, b, e);
      on = !room4(e.k) && !(unique && m) && next != home(kf);
    }
    __syncwarp();
    push(on, kf, x, [&] { return next; });
  };
  // a probe meets its home bucket (its contents in e): true when it goes on
  auto meet = [&](int32_t k, X x, const JBucket &e) -> bool {
    const int32_t kf = k ^ kKeyFlip;
    if (kf == 0) {
      side_probe(x);
      return false;
    }
    // the home bucket again where it is wanted: kept, it takes four registers
    const uint32_t c = visit(kf, x, kPay && kAgg == kAggCountXor ? home(kf) : 0u, e);
    return !room4(e.k) && !(unique && c);
  };
  auto enqueue = [&](bool on, int32_t k, X x) {
    const int32_t kf = k ^ kKeyFlip;
    push(on, kf, x, [&] { return (home(kf) + 1) & bmask; });
  };
  // tiles of 32 G probes; probe j of a lane is one of four neighbours, or with
  // a column that is not 16-byte aligned one of every 32nd
  constexpr uint32_t kTile = 32 * G;
  constexpr bool kValues = kAgg == kAggCountProduct && kPay;
  const bool values = kValues && pay;
  const uint64_t tiles = n / kTile, stride = (uint64_t)gridDim.x * (kThreads / 32);
  auto load = [&](const int32_t *col, uint64_t t, int32_t *v) {
    if (kVec) {
      const int4 v4 = __ldcs(reinterpret_cast<const int4 *>(col + t * kTile) + lane);
      v[0] = v4.x, v[1] = v4.y, v[2] = v4.z, v[3] = v4.w;
    } else {
#pragma unroll
      for (int j = 0; j < G; ++j) v[j] = __ldcs(col + t * kTile + j * 32 + lane);
    }
  };
  uint64_t t = blockIdx.x * (uint64_t)(kThreads / 32) + (threadIdx.x >> 5);
  int32_t nk[G], np[G] = {0, 0, 0, 0};
  if (t < tiles) {
    load(keys, t, nk);
    if (values) load(pay, t, np);
  }
  for (; t < tiles; t += stride) {
    int32_t kk[G], pp[G];
    JBucket e[G];
#pragma unroll
    for (int j = 0; j < G; ++j) {
      kk[j] = nk[j];
      pp[j] = np[j];
      e[j] = ld_bucket(&bk[gbjd::fmix32((uint32_t)kk[j]) & bmask]);
    }
    if (t + stride < tiles) {
      load(keys, t + stride, nk);
      if (values) load(pay, t + stride, np);
    }
    auto value = [&](int j) {
      return kAgg == kAggCountProduct ? (X)pp[j] : (X)(t * kTile + (kVec ? lane * G + j : j * 32 + lane));
    };
    bool on[G];
#pragma unroll
    for (int j = 0; j < G; ++j) on[j] = meet(kk[j], value(j), e[j]);
    if (!__any_sync(0xffffffffu, on[0] | on[1] | on[2] | on[3])) continue;
#pragma unroll
    for (int j = 0; j < G; ++j) {
      enqueue(on[j], kk[j], value(j));
      if (j & 1)
        while (qn >= 32) walk(32);
    }
  }
  if (t == tiles) {  // the last n mod 32 G probes: this warp's
    for (uint64_t base = tiles * kTile; base < n; base += 32) {
      const uint64_t i = base + lane;
      bool on = false;
      int32_t k = 0;
      X x = 0;
      if (i < n) {
        k = keys[i];
        x = kAgg == kAggCountProduct ? (X)(values ? pay[i] : 0) : (X)i;
        on = meet(k, x, ld_bucket(&bk[gbjd::fmix32((uint32_t)k) & bmask]));
      }
      __syncwarp();
      enqueue(on, k, x);
      while (qn >= 32) walk(32);
    }
  }
  while (qn) walk(qn < 32 ? qn : 32);
  gbjd::Acc acc;
  acc.init(spec);
  acc.v[0] = a_cnt;
  acc.v[1] = a_sum;
  gbjd::after_init();
  gbjd::block_flush(spec, acc, red, out);
}

// ------------------------------------------------ int64-key table
// gbj_join_build_i64's table: 32-byte buckets of two slots -- two keys
// (xor 2^63, so zero marks an empty slot; INT64_MIN goes to the side list),
// their build payloads and their rows + 1 -- read with one 256-bit load.
// Placement is the reference's int64 hash, the murmur3 64-bit finaliser
// (core/olap/lib/expressions/expressions-hasher.cpp:66-84).
struct __align__(32) JBucket64 {
  unsigned long long k[2];
  int2 x[2];  // {build payload (0 without one), row + 1}; x[1].y's top bit: a row went past this bucket
};
constexpr unsigned long long kFlip64 = 0x8000000000000000ull;

__device__ __forceinline__ uint64_t fmix64(uint64_t k) {
  k ^= k >> 33;
  k *= 0xff51afd7ed558ccdull;
  k ^= k >> 33;
  k *= 0xc4ceb9fe1a85ec53ull;
  k ^= k >> 33;
  return k;
}

__device__ __forceinline__ JBucket64 ld_bucket64(const JBucket64 *p) {
  uint32_t w[8];
  asm("ld.global.nc.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
      : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]), "=r"(w[4]), "=r"(w[5]), "=r"(w[6]), "=r"(w[7])
      : "l"(p));
  JBucket64 b;
  b.k[0] = ((unsigned long long)w[1] << 32) | w[0];
  b.k[1] = ((unsigned long long)w[3] << 32) | w[2];
  b.x[0] = make_int2((int32_t)w[4], (int32_t)w[5]);
  b.x[1] = make_int2((int32_t)w[6], (int32_t)w[7]);
  return b;
}

// meta[0]: a duplicate build key was seen; meta[1]: side-list length.  A row
// that finds both slots of a bucket taken marks the bucket: a probe goes on
// from marked buckets only, where a full bucket used to send every probe of a
// key that is not unique to the next one (1.5 M rows, two a key, 20 M probes:
// 541 -> 391 us; unique keys, half of the probes without a match: 224 -> 208;
// the build with its clear, without marks / with them: 4 M rows unique 167 / 173,
// two a key 209 / 218, sixteen 871 / 1033; reading a bucket before its slots are
// claimed or marked is better for sixteen, 670, and worse for two, 260).
__global__ void __launch_bounds__(kThreads)
    k_jb64_build(const int64_t *__restrict__ keys, const int32_t *__restrict__ payload, uint64_t n,
                 JBucket64 *__restrict__ bk, uint64_t bmask, uint32_t *__restrict__ meta,
                 int32_t *__restrict__ side, uint32_t *status) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  bool dup = false;
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += stride) {
    const int64_t key = keys[i];
    const int32_t pv = payload ? payload[i] : 0;
    const unsigned long long kf = (unsigned long long)key ^ kFlip64;
    if (kf == 0) {
      side[atomicAdd(&meta[1], 1u)] = (int32_t)i;
      continue;
    }
    const uint64_t h = fmix64((uint64_t)key);
    uint64_t b = h & bmask;
    const uint32_t o = (uint32_t)(h >> 63);
    bool placed = false;
    for (uint64_t step = 0; step <= bmask && !placed; ++step) {
#pragma unroll
      for (uint32_t j = 0; j < 2; ++j) {
        if (placed) break;
        const uint32_t sl = (o + j) & 1u;
        const unsigned long long old = atomicCAS(&bk[b].k[sl], 0ull, kf);
        if (old == 0) {
          // into zeroes, so an or beside the bit that rows going past set (a
          // plain store for slot 0 only: 1.5 M rows 60 us, this 51)
          atomicOr(reinterpret_cast<unsigned long long *>(&bk[b].x[sl]),
                   ((unsigned long long)(uint32_t)(i + 1) << 32) | (uint32_t)pv);
          placed = true;
        } else {
          dup |= old == kf;
        }
      }
      // 64 bits wide, as the row's own word that may be written meanwhile
      if (!placed) atomicOr(reinterpret_cast<unsigned long long *>(&bk[b].x[1]), 1ull << 63);
      b = (b + 1) & bmask;
    }
    if (!placed) gbjd::latch(status, GBJ_DEV_CAPACITY);
  }
  if (dup) meta[0] = 1;
}

// ------------------------------ probe with any aggregate list, or pair output
// The two table layouts as k_jb_probe_list reads them.
struct JTable {
  const void *bk;
  const int4 *rows;
  uint32_t bmask;  // buckets - 1
  const int32_t *bpay;
  const uint32_t *meta;
  const int32_t *side;
};

template <bool kPay>
struct JLayout32 {
  using Key = int32_t;
  using Word = int32_t;  // the key as stored; 0 is the empty slot
  using Bucket = JBucket;
  static __device__ __forceinline__ Word word(Key k) { return k ^ kKeyFlip; }
  static __device__ __forceinline__ uint32_t home(Key k, uint32_t m) { return gbjd::fmix32((uint32_t)k) & m; }
  static __device__ __forceinline__ Bucket load(const JTable &t, uint32_t b) {
    return ld_bucket(static_cast<const JBucket *>(t.bk) + b);
  }
  static __device__ __forceinline__ uint32_t hits(const Bucket &e, Word w) { return hits4(e.k, w); }
  // a key with this home may be in a later bucket
  static __device__ __forceinline__ bool passed(const Bucket &e) { return !room4(e.k); }
  static __device__ __forceinline__ int32_t value(const Bucket &e, uint32_t i) { return kPay ? lane4(e.x, i) : 0; }
  static __device__ __forceinline__ int32_t row(const JTable &t, const Bucket &e, uint32_t b, uint32_t i) {
    return (kPay ? __ldg(reinterpret_cast<const int32_t *>(t.rows + b) + i) : lane4(e.x, i)) - 1;
  }
};

struct JLayout64 {
  using Key = int64_t;
  using Word = unsigned long long;
  using Bucket = JBucket64;
  static __device__ __forceinline__ Word word(Key k) { return (unsigned long long)k ^ kFlip64; }
  static __device__ __forceinline__ uint32_t home(Key k, uint32_t m) { return (uint32_t)fmix64((uint64_t)k) & m; }
  static __device__ __forceinline__ Bucket load(const JTable &t, uint32_t b) {
    return ld_bucket64(static_cast<const JBucket64 *>(t.bk) + b);
  }
  static __device__ __forceinline__ uint32_t hits(const Bucket &e, Word w) {
    return (uint32_t)(e.k[0] == w) | ((uint32_t)(e.k[1] == w) << 1);
  }
  static __device__ __forceinline__ bool passed(const Bucket &e) { return e.x[1].y < 0; }
  static __device__ __forceinline__ int32_t value(const Bucket &e, uint32_t i) { return i ? e.x[1].x : e.x[0].x; }
  static __device__ __forceinline__ int32_t row(const JTable &, const Bucket &e, uint32_t, uint32_t i) {
    return (i ? e.x[1].y & INT32_MAX : e.x[0].y) - 1;
  }
};

constexpr int kListThreads = 256;
// CTAs per SM of k_jb_probe_list.  Measured on the case below with unique
// keys: 3 (80 registers) 234 us, 4 (64, spills) 268, 5 (48, spills) 452.
constexpr int kListCtas = 3;
constexpr int kListWarps = kListThreads / 32;

// A warp's queues, both rings: matches on their way to the accumulators, and
// probes that go on past their home bucket (the last bucket looked at, and
// how many are left; for the lowest key, which has no bucket, the next side
// entry).
// Pair output: matches wait in a buffer of 256 {build row, probe row}.
constexpr uint32_t kPairBuf = 256;

template <typename Key, bool kPairs>
struct ListQueue {
  union {
    struct {
      Key mkey[64];
      uint64_t mprow[64];
      int32_t mbv[64], mpv[64], mbr[64];
    };
    struct {
      int32_t pb[kPairs ? kPairBuf : 1], pp[kPairs ? kPairBuf : 1];
    };
  };
  Key wkey[64];
  uint64_t wprow[64];
  int32_t wpv[64];
  uint32_t wb[64], wleft[64];
};

// Probe with an aggregate list that has no specialised kernel, and every
// list over int64 keys.  One probe per lane at a time: the next one's bucket
// is loaded while this one's is looked at, and its key one step earlier.
//
// What bounds it is issue.  The accumulator update takes some 20 instructions
// per aggregate, and matches are few lanes of a warp at a time when they are
// applied where they are found; inlined at each of the places where a match
// can turn up it also overran the instruction cache (31 of 38 stalled warps
// per issue waited for instructions, 8.4 active lanes).  So a match goes to
// the warp's ring of 64, and 32 of them are applied at once by all lanes;
// probes whose home bucket is full go to a second ring, from which 32 at a
// time look at their next bucket and go back if that does not end them.
// Measured on GB300, 1.5 M int64 build rows (two per key), 20 M probes, COUNT
// + SUM + MIN + MAX: 8.21 ms before, 0.54 ms now (one row per key: 4.54 -> 0.23
// ms; the same over int32 keys: 0.90 -> 0.22 ms); with marked buckets (see
// k_jb64_build) 0.39 and 0.21 ms.
//
// kMaxA = 0 is the pair output: `pay` holds the probe rows' ids (null: their
// positions), matches wait in the warp's buffer, and one reservation in the
// output takes 225 to 256 of them (one per 32 probes was 75 us of an atomic's
// turn for 1.7 M probes, now 26 us).
struct PairOut {
  int32_t *build, *probe;
  uint64_t cap;
  unsigned long long *count;
  uint32_t *status;
};

template <typename L, int kMaxA>
__global__ void __launch_bounds__(kListThreads, kListCtas)
    k_jb_probe_list(const typename L::Key *__restrict__ keys, const int32_t *__restrict__ pay, uint64_t n,
                    JTable t, gbj::AggSpec spec, int64_t *out, PairOut po) {
  using Key = typename L::Key;
  using Bucket = typename L::Bucket;
  constexpr bool kPairs = kMaxA == 0;
  __shared__ int64_t red[kPairs ? 1 : 32 * GBJ_MAX_AGGS];
  __shared__ ListQueue<Key, kPairs> s_q[kListWarps];
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  ListQueue<Key, kPairs> &q = s_q[threadIdx.x >> 5];
  const bool unique = t.meta[0] == 0;
  const uint32_t nside = t.meta[1];
  bool need_row = kPairs;
#pragma unroll
  for (int j = 0; j < kMaxA; ++j)
    if (j < spec.n)
      need_row |= spec.operand[j] == GBJ_VAL_BUILD_ROWID || spec.operand[j] == GBJ_VAL_ROWID_XOR;
  int64_t v[kPairs ? 1 : kMaxA];
#pragma unroll
  for (int j = 0; j < kMaxA; ++j) v[j] = j < spec.n ? gbjd::agg_identity(spec.op[j]) : 0;

  uint32_t mn = 0, mh = 0;  // the ring's length and head (warp-uniform)
  // writes the buffered pairs
  auto flush = [&]() {
    __syncwarp();
    unsigned long long base = 0;
    if (lane == 0) base = atomicAdd(po.count, (unsigned long long)mn);
    base = __shfl_sync(0xffffffffu, base, 0);
    for (uint32_t i = lane; i < mn; i += 32) {
      if (base + i < po.cap) {
        po.build[base + i] = q.pb[i];
        po.probe[base + i] = q.pp[i];
      }
    }
    if (base + mn > po.cap && lane == 0) gbjd::latch(po.status, GBJ_DEV_CAPACITY);
    __syncwarp();
    mn = 0;
  };
  // applies the first `c` (<= 32) matches of the ring
  auto apply = [&](uint32_t c) {
    __syncwarp();
    if ((uint32_t)lane < c) {
      const uint32_t p = (mh + lane) & 63u;
      const int32_t bv = q.mbv[p], pv = q.mpv[p], br = q.mbr[p];
      const int64_t pr = (int64_t)q.mprow[p];
#pragma unroll
      for (int j = 0; j < kMaxA; ++j) {
        if (j < spec.n)
          gbjd::agg_step(v[j], spec.op[j], spec.operand[j], (int64_t)q.mkey[p], bv, pv, br, pr);
      }
    }
    __syncwarp();
    mh = (mh + c) & 63u;
    mn -= c;
  };
  // every match of a bucket (or side row srow >= 0) into the ring; all lanes call it
  auto push = [&](uint32_t hits, Key k, int32_t pv, uint64_t prow, uint32_t b, const Bucket &e, int32_t srow) {
    for (;;) {
      const unsigned bal = __ballot_sync(0xffffffffu, hits != 0);
      if (!bal) break;
      if (hits) {
        const uint32_t i = __ffs(hits) - 1;
        const int32_t br = srow >= 0 ? srow : need_row ? L::row(t, e, b, i) : 0;
        if (kPairs) {
          const uint32_t p = mn + __popc(bal & lt);
          q.pb[p] = br;
          q.pp[p] = pv;
        } else {
          const uint32_t p = (mh + mn + __popc(bal & lt)) & 63u;
          q.mkey[p] = k;
          q.mprow[p] = prow;
          q.mpv[p] = pv;
          q.mbv[p] = srow < 0 ? L::value(e, i) : t.bpay ? __ldg(t.bpay + srow) : 0;
          q.mbr[p] = br;
        }
        hits = unique ? 0u : hits & (hits - 1);
      }
      mn += __popc(bal);
      if (kPairs) {
        if (mn > kPairBuf - 32) flush();
      } else if (mn >= 32) {
        apply(32);
      }
    }
  };
  uint32_t wn = 0, wh = 0;  // the second ring's length and head
  auto queue_walk = [&](bool go_on, Key k, int32_t pv, uint64_t prow, auto b, uint32_t left) {
    const unsigned bal = __ballot_sync(0xffffffffu, go_on);
    if (go_on) {
      const uint32_t p = (wh + wn + __popc(bal & lt)) & 63u;
      q.wkey[p] = k;
      q.wprow[p] = prow;
      q.wpv[p] = pv;
      q.wb[p] = b;
      q.wleft[p] = left;
    }
    wn += __popc(bal);
  };
  // one bucket (or side entry) further for the first `c` (<= 32) of them
  auto walk = [&](uint32_t c) {
    __syncwarp();
    const bool active = (uint32_t)lane < c;
    const uint32_t p = (wh + lane) & 63u;
    const Key k = active ? q.wkey[p] : 0;
    const uint64_t prow = active ? q.wprow[p] : 0;
    const int32_t pv = active ? q.wpv[p] : 0;
    uint32_t b = active ? q.wb[p] : 0;
    const uint32_t left = active ? q.wleft[p] - 1 : 0;
    __syncwarp();  // read before any of them is written again
    wh = (wh + c) & 63u;
    wn -= c;
    uint32_t hits = 0;
    int32_t srow = -1;
    Bucket e{};
    bool go_on = false;
    if (active) {
      if (L::word(k) == 0) {
        srow = __ldg(t.side + b);
        ++b;
        hits = 1;
        go_on = left != 0;
      } else {
        b = (b + 1) & t.bmask;
        e = L::load(t, b);
        hits = L::hits(e, L::word(k));
        go_on = left != 0 && L::passed(e) && !(unique && hits);
      }
    }
    push(hits, k, pv, prow, b, e, srow);
    queue_walk(go_on, k, pv, prow, b, left);
  };

  const uint64_t wstep = (uint64_t)gridDim.x * kListThreads;
  const uint64_t first = blockIdx.x * (uint64_t)kListThreads + (threadIdx.x & ~31u);  // of the warp
  auto load_key = [&](uint64_t i, Key &k, int32_t &p) {
    k = i < n ? __ldcs(keys + i) : 0;
    p = pay ? (i < n ? __ldcs(pay + i) : 0) : kPairs ? (int32_t)i : 0;
  };
  Key k0, k1;
  int32_t p0, p1;
  load_key(first + lane, k0, p0);
  uint32_t b0 = L::home(k0, t.bmask);
  Bucket e0 = L::load(t, b0);
  load_key(first + wstep + lane, k1, p1);
  for (uint64_t base = first; base < n; base += wstep) {
    const Key k = k0;
    const int32_t pv = p0;
    const uint32_t b = b0;
    const Bucket e = e0;
    k0 = k1;
    p0 = p1;
    b0 = L::home(k0, t.bmask);
    e0 = L::load(t, b0);
    load_key(base + 2 * wstep + lane, k1, p1);
    const uint64_t i = base + lane;
    const bool valid = i < n, to_side = L::word(k) == 0;  // the lowest key is in the side list
    const uint32_t hits = valid && !to_side ? L::hits(e, L::word(k)) : 0u;
    push(hits, k, pv, i, b, e, -1);
    const bool go_on = valid && (to_side ? nside != 0 : t.bmask != 0 && L::passed(e) && !(unique && hits));
    queue_walk(go_on, k, pv, i, to_side ? 0u : b, to_side ? nside : t.bmask);
    while (wn >= 32) walk(32);
  }
  while (wn) walk(wn < 32 ? wn : 32);
  if constexpr (kPairs) {
    if (mn) flush();
  } else {
    while (mn) apply(mn < 32 ? mn : 32);
    gbjd::Acc acc;
#pragma unroll
    for (int j = 0; j < GBJ_MAX_AGGS; ++j) acc.v[j] = j < kMaxA ? v[j < kMaxA ? j : 0] : 0;
    gbjd::after_init();
    gbjd::block_flush(spec, acc, red, out);
  }
}

// Column reduce (Reduce over one column, optional row list): four rows of a
// thread in flight.
template <int kMaxA>
__global__ void __launch_bounds__(kThreads)
    k_reduce(const int32_t *__restrict__ col, const int32_t *__restrict__ rows,
             uint64_t n, gbj::AggSpec spec, int64_t *out) {
  __shared__ int64_t red[32 * GBJ_MAX_AGGS];
  gbjd::Acc acc;
  acc.init(spec);
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += 4 * stride) {
    int64_t r[4];
    int32_t v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const uint64_t k = i + u * stride;
      r[u] = rows ? (k < n ? __ldg(rows + k) : 0) : (int64_t)k;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) v[u] = col && i + u * stride < n ? __ldg(col + r[u]) : 0;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (i + u * stride < n) {
#pragma unroll
        for (int j = 0; j < kMaxA; ++j)
          if (j < spec.n) gbjd::agg_step(acc.v[j], spec.op[j], spec.operand[j], v[u], v[u], v[u], r[u], r[u]);
      }
    }
  }
  gbjd::after_init();
  gbjd::block_flush(spec, acc, red, out);
}

// Four rows of a thread in flight.
__global__ void __launch_bounds__(256)
    k_gather(const int32_t *__restrict__ col, const int32_t *__restrict__ rows, uint64_t n,
             int32_t *__restrict__ out) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += 4 * stride) {
    int32_t r[4], v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) r[u] = i + u * stride < n ? __ldcs(rows + i + u * stride) : 0;
#pragma unroll
    for (int u = 0; u < 4; ++u) v[u] = i + u * stride < n ? __ldg(col + r[u]) : 0;
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (i + u * stride < n) out[i + u * stride] = v[u];
  }
}

// Range predicate of gbj_select_range (inclusive bounds).
struct RangePred {
  const int32_t *col;
  int32_t lo, hi;
  __device__ __forceinline__ bool test(int32_t v) const { return v >= lo && v <= hi; }
};

int grid_for_sms(int sm_count, uint64_t work, int threads, int per_sm = 4) {
  uint64_t blocks = (work + threads - 1) / threads;
  uint64_t cap = (uint64_t)sm_count * per_sm;
  if (blocks > cap) blocks = cap;
  if (blocks == 0) blocks = 1;
  return (int)blocks;
}

int grid_for(gbj_ctx *ctx, uint64_t work, int threads, int per_sm = 4) {
  return grid_for_sms(ctx->sm_count, work, threads, per_sm);
}

// Probe kernel of the allocation-free entry point: 16-byte loads when both
// probe columns are 16-byte aligned, a specialised accumulator for COUNT +
// SUM(product / xor).
void launch_probe(int sm_count, const int32_t *keys, const int32_t *pay, uint64_t n, const uint64_t *slots,
                  uint64_t mask, const int32_t *bpay, const uint32_t *meta, const gbj::AggSpec &spec,
                  int64_t *out, cudaStream_t s) {
  const bool vec = ((uintptr_t)keys % 16 == 0) && (!pay || (uintptr_t)pay % 16 == 0);
  const bool two = spec.n == 2 && spec.op[0] == GBJ_AGG_COUNT && spec.op[1] == GBJ_AGG_SUM;
  const int agg = two && spec.operand[1] == GBJ_VAL_ROWID_XOR ? kAggCountXor
                  : two && spec.operand[1] == GBJ_VAL_PRODUCT ? kAggCountProduct
                                                              : kAggGeneric;
  const int gv = grid_for_sms(sm_count, (n + 7) / 8, kThreads);
  const int gs = grid_for_sms(sm_count, n, kThreads);
#define GBJ_PROBE(V, A) \
  k_join_probe_agg<V, A><<<V ? gv : gs, kThreads, 0, s>>>(keys, pay, n, slots, mask, bpay, meta, spec, out)
  if (vec) {
    if (agg == kAggCountXor) GBJ_PROBE(true, kAggCountXor);
    else if (agg == kAggCountProduct) GBJ_PROBE(true, kAggCountProduct);
    else GBJ_PROBE(true, kAggGeneric);
  } else {
    if (agg == kAggCountXor) GBJ_PROBE(false, kAggCountXor);
    else if (agg == kAggCountProduct) GBJ_PROBE(false, kAggCountProduct);
    else GBJ_PROBE(false, kAggGeneric);
  }
#undef GBJ_PROBE
}

// Any other list, and every list over int64 keys: kernels for up to four and
// up to eight aggregates (the accumulators are registers).
template <typename L>
void launch_jb_list(int sm_count, const gbj_table *t, uint64_t nbk, const typename L::Key *keys, const int32_t *pay,
                    uint64_t n, const gbj::AggSpec &spec, int64_t *out, cudaStream_t s) {
  const JTable jt{t->slots, t->rows, (uint32_t)(nbk - 1), t->payload, t->meta, t->side};
  const int grid = grid_for_sms(sm_count, n, kListThreads, kListCtas);
  launch_behind_init(spec.n <= 4 ? k_jb_probe_list<L, 4> : k_jb_probe_list<L, 8>, grid, kListThreads, s, keys, pay, n,
                     jt, spec, out, PairOut{});
}

template <typename L>
void launch_jb_pairs(int sm_count, const gbj_table *t, uint64_t nbk, const typename L::Key *keys, const int32_t *prows,
                     uint64_t n, const PairOut &po, cudaStream_t s) {
  const JTable jt{t->slots, t->rows, (uint32_t)(nbk - 1), t->payload, t->meta, t->side};
  k_jb_probe_list<L, 0><<<grid_for_sms(sm_count, n, kListThreads, kListCtas), kListThreads, 0, s>>>(
      keys, prows, n, jt, gbj::AggSpec{}, nullptr, po);
}

// Probe kernel over a bucketed table: 16-byte probe loads when both probe
// columns are aligned, the specialised accumulators, the table's layout.
template <bool kPay>
const char *launch_jb_probe_t(int sm_count, const gbj_table *t, const int32_t *keys, const int32_t *pay, uint64_t n,
                       const gbj::AggSpec &spec, int64_t *out, cudaStream_t s) {
  const bool vec = ((uintptr_t)keys % 16 == 0) && (!pay || (uintptr_t)pay % 16 == 0);
  const bool two = spec.n == 2 && spec.op[0] == GBJ_AGG_COUNT && spec.op[1] == GBJ_AGG_SUM;
  const bool is_xor = two && spec.operand[1] == GBJ_VAL_ROWID_XOR;
  const JBucket *bk = static_cast<const JBucket *>(t->slots);
  const uint64_t nbk = (t->mask + 1) / 4;
  const uint32_t bmask = (uint32_t)(nbk - 1);
  if (!is_xor && !(two && spec.operand[1] == GBJ_VAL_PRODUCT)) {
    launch_jb_list<JLayout32<kPay>>(sm_count, t, nbk, keys, pay, n, spec, out, s);
    return "k_jb_probe_list";
  }
  const int gv = grid_for_sms(sm_count, (n + kJbGroup - 1) / kJbGroup, kThreads, 2);
  const int gs = grid_for_sms(sm_count, n, kThreads);
  const bool ring = 3 * t->n > t->mask + 1;  // the table is more than a third full: times at k_jb_probe_ring
#define GBJ_JB_PROBE(V, A)                                                                                   \
  launch_behind_init(ring ? k_jb_probe_ring<V, A, kPay> : k_jb_probe_agg<V, A, kPay>, V || ring ? gv : gs, kThreads, \
                     s, keys, pay, n, bk, t->rows, bmask, t->payload, t->meta, t->side, spec, out)
  if (vec) {
    if (is_xor) GBJ_JB_PROBE(true, kAggCountXor);
    else GBJ_JB_PROBE(true, kAggCountProduct);
  } else {
    if (is_xor) GBJ_JB_PROBE(false, kAggCountXor);
    else GBJ_JB_PROBE(false, kAggCountProduct);
  }
#undef GBJ_JB_PROBE
  return ring ? "k_jb_probe_ring" : "k_jb_probe_agg";
}

// Returns the name of the kernel that it launched.
const char *launch_jb_probe(int sm_count, const gbj_table *t, const int32_t *keys, const int32_t *pay, uint64_t n,
                            const gbj::AggSpec &spec, int64_t *out, cudaStream_t s) {
  if (t->rows) return launch_jb_probe_t<true>(sm_count, t, keys, pay, n, spec, out, s);
  return launch_jb_probe_t<false>(sm_count, t, keys, pay, n, spec, out, s);
}

// ------------------------------------------------ allocation-free variant
// Hash table of gbj_join_agg_noalloc: a fixed array in the module's device
// memory, so that entry point never allocates.  Slots for build sides of up
// to GBJ_NOALLOC_MAX_BUILD rows at load factor 1/2, then 32 words of table
// metadata (the duplicate-key flag).  The table always has at least 2n
// slots, so its build cannot run out of room and needs no status word.
constexpr uint64_t kNoAllocSlots = 2ull * GBJ_NOALLOC_MAX_BUILD;
static __device__ __align__(256) uint64_t g_noalloc_scratch[kNoAllocSlots + 32];

__global__ void k_noalloc_init_out(gbj::AggSpec s, int64_t *out) {
  const int j = threadIdx.x;
  if (j < s.n) out[j] = gbjd::agg_identity(s.op[j]);
}

// Per-device set-up of the allocation-free entry point: the device address
// of g_noalloc_scratch (host code cannot use the symbol itself) and the SM
// count, looked up once per device and CUDA context with that device current.
// The context is part of the key because cudaDeviceReset ends the context
// that address belongs to; the next call then looks it up again.
struct NoAllocDevice {
  uint64_t *scratch = nullptr;
  int sm_count = 0;
};
std::mutex g_noalloc_mu;
std::map<std::pair<int, unsigned long long>, NoAllocDevice> g_noalloc_devices;

// Unique id of the calling thread's current CUDA context (0 when there is
// none yet), through the driver entry points the runtime hands out, so the
// library needs no link against the driver library.
unsigned long long current_context_id() {
  typedef int (*GetCurrent)(void **);
  typedef int (*GetId)(void *, unsigned long long *);
  static GetCurrent get_current = nullptr;
  static GetId get_id = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void *f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &f, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      get_current = reinterpret_cast<GetCurrent>(f);
    f = nullptr;
    if (cudaGetDriverEntryPointByVersion("cuCtxGetId", &f, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      get_id = reinterpret_cast<GetId>(f);
    (void)cudaGetLastError();
  });
  void *c = nullptr;
  unsigned long long id = 0;
  if (!get_current || !get_id || get_current(&c) != 0 || !c || get_id(c, &id) != 0) return 0;
  return id;
}
thread_local std::string g_noalloc_error;

int noalloc_fail(int code, const char *msg) {
  g_noalloc_error = msg;
  return code;
}

}  // namespace

namespace gbj {
const char *noalloc_error_text_impl() { return g_noalloc_error.c_str(); }
}  // namespace gbj

extern "C" {

int gbj_join_build(gbj_ctx *ctx, const int32_t *d_keys,
                   const int32_t *d_payload, uint64_t n, int32_t hash_bits,
                   uint64_t max_build, void *stream, gbj_table **out) {
  if (!ctx || !out) return GBJ_ERR_INVALID;
  *out = nullptr;
  if (n && !d_keys) return set_error(ctx, GBJ_ERR_INVALID, "join_build: null keys");
  if (n >= (1ULL << 31)) return set_error(ctx, GBJ_ERR_INVALID, "join_build: n >= 2^31");
  if (hash_bits < 0 || hash_bits > 31)
    return set_error(ctx, GBJ_ERR_INVALID, "join_build: hash_bits out of range");
  if (max_build && n > max_build)
    return set_error(ctx, GBJ_ERR_CAPACITY,
                     "Build input size exceeded given parameter (maxBuildInputSize)");
  cudaStream_t s = pick_stream(ctx, stream);
  prof_mark(ctx, s);
  uint64_t slots = next_pow2(2 * (n ? n : 1));
  if (!hash_bits) {  // an autotuned table size for build sides of this size, if any
    const int32_t tb = tuned_value(ctx, tune_key("join", n, 0));
    if (tb > 0) hash_bits = tb;
  }
  if (hash_bits && (1ULL << hash_bits) > slots) slots = 1ULL << hash_bits;
  if (slots < 64) slots = 64;
  if (slots > (1ULL << 32)) return set_error(ctx, GBJ_ERR_INVALID, "join_build: table above 2^32 slots");
  const uint64_t nbk = slots / 4;
  const bool with_pay = d_payload != nullptr;
  // buckets | rows (payload tables) | metadata | INT32_MIN side list
  const uint64_t b_bytes = nbk * sizeof(JBucket), r_bytes = with_pay ? nbk * sizeof(int4) : 0;
  const uint64_t clear_bytes = b_bytes + r_bytes + 256;
  gbj_table *t = new gbj_table();
  void *mem = nullptr;
  int rc = pool_alloc(ctx, clear_bytes + (n + 4) * sizeof(int32_t), s, &mem);
  if (rc) {
    delete t;
    return rc;
  }
  char *base = static_cast<char *>(mem);
  t->slots = mem;
  t->rows = with_pay ? reinterpret_cast<int4 *>(base + b_bytes) : nullptr;
  t->meta = reinterpret_cast<uint32_t *>(base + b_bytes + r_bytes);
  t->side = reinterpret_cast<int32_t *>(base + clear_bytes);
  t->mask = slots - 1;
  t->keys = d_keys;
  t->payload = d_payload;
  t->n = n;
  auto fail = [&](int code) {
    pool_release(ctx, mem, s);
    delete t;
    return code;
  };
  if (n && slots <= kSmallSlots) {
    const size_t smem = slots * (with_pay ? 13 : 9);
    cudaError_t e = cudaFuncSetAttribute(k_jb_build_small, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)(kSmallSlots * 13));
    if (e != cudaSuccess) return fail(cuda_error(ctx, e, "k_jb_build_small"));
    k_jb_build_small<<<1, kSmallThreads, smem, s>>>(d_keys, d_payload, (uint32_t)n, static_cast<uint4 *>(mem),
                                                    reinterpret_cast<uint4 *>(t->rows), (uint32_t)slots, t->meta,
                                                    t->side);
    rc = after_launch(ctx, "k_jb_build_small", s);
    if (rc) return fail(rc);
  } else {
    cudaError_t e = cudaMemsetAsync(mem, 0, clear_bytes, s);
    if (e != cudaSuccess) return fail(cuda_error(ctx, e, "cudaMemsetAsync(table)"));
    if (n) {
      k_jb_build<<<grid_for(ctx, n, kThreads), kThreads, 0, s>>>(
          d_keys, d_payload, n, static_cast<unsigned long long *>(mem), reinterpret_cast<int32_t *>(t->rows),
          (uint32_t)(nbk - 1), t->meta, t->side, ctx->d_status);
      rc = after_launch(ctx, "k_jb_build", s);
      if (rc) return fail(rc);
    }
  }
  note_use(ctx, t->uses, s);
  *out = t;
  return GBJ_OK;
}

int gbj_table_destroy(gbj_ctx *ctx, gbj_table *table) {
  if (!ctx || !table) return GBJ_ERR_INVALID;
  const int rc = pool_release_used(ctx, table->slots, table->uses);
  delete table;
  return rc;
}

uint64_t gbj_table_slots(const gbj_table *table) { return table ? table->mask + 1 : 0; }

int gbj_join_probe_agg(gbj_ctx *ctx, const gbj_table *t, const int32_t *d_keys,
                       const int32_t *d_payload, uint64_t n, const gbj_agg *aggs,
                       int32_t n_aggs, int64_t *d_out, void *stream) {
  if (!ctx || !t || !d_out) return GBJ_ERR_INVALID;
  if (t->i64) return set_error(ctx, GBJ_ERR_INVALID, "join_probe: the table has int64 keys (use the _i64 probe)");
  if (n && !d_keys) return set_error(ctx, GBJ_ERR_INVALID, "join_probe: null keys");
  GBJ_TRY(validate_aggs(ctx, aggs, n_aggs));
  AggSpec spec = make_spec(aggs, n_aggs);
  for (int j = 0; j < n_aggs; ++j) {
    int o = spec.operand[j];
    if ((o == GBJ_VAL_BUILD || o == GBJ_VAL_PRODUCT) && !t->payload && t->n)
      return set_error(ctx, GBJ_ERR_INVALID, "aggregate reads the build payload, table has none");
    if ((o == GBJ_VAL_PROBE || o == GBJ_VAL_PRODUCT) && !d_payload && n)
      return set_error(ctx, GBJ_ERR_INVALID, "aggregate reads the probe payload, none given");
  }
  cudaStream_t s = pick_stream(ctx, stream);
  prof_mark(ctx, s);
  GBJ_TRY(init_agg_out(ctx, spec, d_out, s));
  if (n == 0) return GBJ_OK;
  const char *kernel = launch_jb_probe(ctx->sm_count, t, d_keys, d_payload, n, spec, d_out, s);
  const int rc = after_launch(ctx, kernel, s);
  note_use(ctx, t->uses, s);
  return rc;
}

int gbj_join_probe_pairs(gbj_ctx *ctx, const gbj_table *t, const int32_t *d_keys,
                         const int32_t *d_probe_rows, uint64_t n,
                         int32_t *d_build_rows, int32_t *d_out_probe_rows,
                         uint64_t capacity, uint64_t *d_count, void *stream) {
  if (!ctx || !t || !d_count || !d_build_rows || !d_out_probe_rows)
    return GBJ_ERR_INVALID;
  if (t->i64) return set_error(ctx, GBJ_ERR_INVALID, "join_probe: the table has int64 keys (use the _i64 probe)");
  if (n && !d_keys) return set_error(ctx, GBJ_ERR_INVALID, "join_probe: null keys");
  cudaStream_t s = pick_stream(ctx, stream);
  prof_mark(ctx, s);
  GBJ_CHECK_CUDA(ctx, cudaMemsetAsync(d_count, 0, sizeof(uint64_t), s));
  if (n == 0) return GBJ_OK;
  const PairOut po{d_build_rows, d_out_probe_rows, capacity, (unsigned long long *)d_count, ctx->d_status};
  const uint64_t nbk = (t->mask + 1) / 4;
  if (t->rows) launch_jb_pairs<JLayout32<true>>(ctx->sm_count, t, nbk, d_keys, d_probe_rows, n, po, s);
  else launch_jb_pairs<JLayout32<false>>(ctx->sm_count, t, nbk, d_keys, d_probe_rows, n, po, s);
  const int rc = after_launch(ctx, "k_jb_probe_list", s);
  note_use(ctx, t->uses, s);
  return rc;
}

int gbj_join_build_i64(gbj_ctx *ctx, const int64_t *d_keys, const int32_t *d_payload, uint64_t n,
                       int32_t hash_bits, uint64_t max_build, void *stream, gbj_table **out) {
  if (!ctx || !out) return GBJ_ERR_INVALID;
  *out = nullptr;
  if (n && !d_keys) return set_error(ctx, GBJ_ERR_INVALID, "join_build: null keys");
  if (n >= (1ULL << 31)) return set_error(ctx, GBJ_ERR_INVALID, "join_build: n >= 2^31");
  if (hash_bits < 0 || hash_bits > 32)
    return set_error(ctx, GBJ_ERR_INVALID, "join_build: hash_bits out of range");
  if (max_build && n > max_build)
    return set_error(ctx, GBJ_ERR_CAPACITY, "Build input size exceeded given parameter (maxBuildInputSize)");
  cudaStream_t s = pick_stream(ctx, stream);
  prof_mark(ctx, s);
  uint64_t slots = next_pow2(2 * (n ? n : 1));
  if (hash_bits && (1ULL << hash_bits) > slots) slots = 1ULL << hash_bits;
  if (slots < 64) slots = 64;
  const uint64_t nbk = slots / 2;
  const uint64_t clear_bytes = nbk * sizeof(JBucket64) + 256;
  gbj_table *t = new gbj_table();
  void *mem = nullptr;
  int rc = pool_alloc(ctx, clear_bytes + (n + 4) * sizeof(int32_t), s, &mem);
  if (rc) {
    delete t;
    return rc;
  }
  char *base = static_cast<char *>(mem);
  t->slots = mem;
  t->meta = reinterpret_cast<uint32_t *>(base + nbk * sizeof(JBucket64));
  t->side = reinterpret_cast<int32_t *>(base + clear_bytes);
  t->mask = slots - 1;
  t->payload = d_payload;
  t->n = n;
  t->i64 = true;
  cudaError_t e = cudaMemsetAsync(mem, 0, clear_bytes, s);
  if (e != cudaSuccess) {
    pool_release(ctx, mem, s);
    delete t;
    return cuda_error(ctx, e, "cudaMemsetAsync(table)");
  }
  if (n) {
    k_jb64_build<<<grid_for(ctx, n, kThreads), kThreads, 0, s>>>(d_keys, d_payload, n,
                                                                  reinterpret_cast<JBucket64 *>(mem), nbk - 1,
                                                                  t->meta, t->side, ctx->d_status);
    rc = after_launch(ctx, "k_jb64_build", s);
    if (rc) {
      pool_release(ctx, mem, s);
      delete t;
      return rc;
    }
  }
  note_use(ctx, t->uses, s);
  *out = t;
  return GBJ_OK;
}

int gbj_join_probe_agg_i64(gbj_ctx *ctx, const gbj_table *t, const int64_t *d_keys, const int32_t *d_payload,
                           uint64_t n, const gbj_agg *aggs, int32_t n_aggs, int64_t *d_out, void *stream) {
  if (!ctx || !t || !d_out) return GBJ_ERR_INVALID;
  if (!t->i64) return set_error(ctx, GBJ_ERR_INVALID, "join_probe_i64: the table has int32 keys");
  if (n && !d_keys) return set_error(ctx, GBJ_ERR_INVALID, "join_probe: null keys");
  GBJ_TRY(validate_aggs(ctx, aggs, n_aggs));
  AggSpec spec = make_spec(aggs, n_aggs);
  for (int j = 0; j < n_aggs; ++j) {
    int o = spec.operand[j];
    if ((o == GBJ_VAL_BUILD || o == GBJ_VAL_PRODUCT) && !t->payload && t->n)
      return set_error(ctx, GBJ_ERR_INVALID, "aggregate reads the build payload, table has none");
    if ((o == GBJ_VAL_PROBE || o == GBJ_VAL_PRODUCT) && !d_payload && n)
      return set_error(ctx, GBJ_ERR_INVALID, "aggregate reads the probe payload, none given");
  }
  cudaStream_t s = pick_stream(ctx, stream);
  prof_mark(ctx, s);
  GBJ_TRY(init_agg_out(ctx, spec, d_out, s));
  if (n == 0) return GBJ_OK;
  launch_jb_list<JLayout64>(ctx->sm_count, t, (t->mask + 1) / 2, d_keys, d_payload, n, spec, d_out, s);
  const int rc = after_launch(ctx, "k_jb_probe_list", s);
  note_use(ctx, t->uses, s);
  return rc;
}

int gbj_join_probe_pairs_i64(gbj_ctx *ctx, const gbj_table *t, const int64_t *d_keys,
                             const int32_t *d_probe_rows, uint64_t n, int32_t *d_build_rows,
                             int32_t *d_out_probe_rows, uint64_t capacity, uint64_t *d_count, void *stream) {
  if (!ctx || !t || !d_count || !d_build_rows || !d_out_probe_rows) return GBJ_ERR_INVALID;
  if (!t->i64) return set_error(ctx, GBJ_ERR_INVALID, "join_probe_i64: the table has int32 keys");
  if (n && !d_keys) return set_error(ctx, GBJ_ERR_INVALID, "join_probe: null keys");
  cudaStream_t s = pick_stream(ctx, stream);
  prof_mark(ctx, s);
  GBJ_CHECK_CUDA(ctx, cudaMemsetAsync(d_count, 0, sizeof(uint64_t), s));
  if (n == 0) return GBJ_OK;
  const PairOut po{d_build_rows, d_out_probe_rows, capacity, (unsigned long long *)d_count, ctx->d_status};
  launch_jb_pairs<JLayout64>(ctx->sm_count, t, (t->mask + 1) / 2, d_keys, d_probe_rows, n, po, s);
  const int rc = after_launch(ctx, "k_jb_probe_list", s);
  note_use(ctx, t->uses, s);
  return rc;
}

int gbj_reduce(gbj_ctx *ctx, const int32_t *d_col, const int32_t *d_rows,
               uint64_t n, const gbj_agg *aggs, int32_t n_aggs, int64_t *d_out,
               void *stream) {
  if (!ctx || !d_out) return GBJ_ERR_INVALID;
  GBJ_TRY(validate_aggs(ctx, aggs, n_aggs));
  AggSpec spec = make_spec(aggs, n_aggs);
  for (int j = 0; j < n_aggs; ++j)
    if (spec.operand[j] != GBJ_VAL_ONE && !d_col)
      return set_error(ctx, GBJ_ERR_INVALID, "reduce: aggregate reads a null column");
  cudaStream_t s = pick_stream(ctx, stream);
  prof_mark(ctx, s);
  GBJ_TRY(init_agg_out(ctx, spec, d_out, s));
  if (n == 0) return GBJ_OK;
  launch_behind_init(spec.n <= 2 ? k_reduce<2> : k_reduce<GBJ_MAX_AGGS>, grid_for(ctx, n, kThreads), kThreads, s, d_col,
                     d_rows, n, spec, d_out);
  return after_launch(ctx, "k_reduce", s);
}

int gbj_gather(gbj_ctx *ctx, const int32_t *d_col, const int32_t *d_rows,
               uint64_t n, int32_t *d_out, void *stream) {
  if (!ctx || (n && (!d_col || !d_rows || !d_out))) return GBJ_ERR_INVALID;
  if (n == 0) return GBJ_OK;
  cudaStream_t s = pick_stream(ctx, stream);
  prof_mark(ctx, s);
  k_gather<<<grid_for(ctx, n, 256, 8), 256, 0, s>>>(d_col, d_rows, n, d_out);
  return after_launch(ctx, "k_gather", s);
}

int gbj_select_range(gbj_ctx *ctx, const int32_t *d_col, uint64_t n, int32_t lo,
                     int32_t hi, int32_t *d_rows_out, uint64_t *d_count,
                     void *stream) {
  if (!ctx || !d_count || (n && (!d_col || !d_rows_out))) return GBJ_ERR_INVALID;
  if (n >= (1ULL << 31)) return set_error(ctx, GBJ_ERR_INVALID, "select: n >= 2^31");
  cudaStream_t s = pick_stream(ctx, stream);
  prof_mark(ctx, s);
  if (n == 0) {
    GBJ_CHECK_CUDA(ctx, cudaMemsetAsync(d_count, 0, sizeof(uint64_t), s));
    return GBJ_OK;
  }
  return compact_rows(ctx, RangePred{d_col, lo, hi}, n, d_rows_out, d_count, s);
}

int gbj_join_agg_noalloc(const int32_t *d_build_keys, const int32_t *d_build_payload,
                         uint64_t n_build, const int32_t *d_probe_keys,
                         const int32_t *d_probe_payload, uint64_t n_probe, const gbj_agg *aggs,
                         int32_t n_aggs, int64_t *d_out, void *stream) {
  g_noalloc_error.clear();
  if (!d_out || !aggs || n_aggs < 1 || n_aggs > GBJ_MAX_AGGS)
    return noalloc_fail(GBJ_ERR_INVALID, "join_agg_noalloc: null output or bad aggregate count");
  if ((n_build && !d_build_keys) || (n_probe && !d_probe_keys))
    return noalloc_fail(GBJ_ERR_INVALID, "join_agg_noalloc: null key column");
  if (n_build > GBJ_NOALLOC_MAX_BUILD)
    return noalloc_fail(GBJ_ERR_CAPACITY,
                        "join_agg_noalloc: build side larger than GBJ_NOALLOC_MAX_BUILD "
                        "(1048576 rows); use gbj_join_build / gbj_join_probe_agg instead");
  if (n_probe >= (1ULL << 32))
    return noalloc_fail(GBJ_ERR_INVALID, "join_agg_noalloc: probe side must have < 2^32 rows");
  for (int j = 0; j < n_aggs; ++j) {
    if (aggs[j].op < GBJ_AGG_COUNT || aggs[j].op > GBJ_AGG_AND || aggs[j].operand < GBJ_VAL_ONE ||
        aggs[j].operand > GBJ_VAL_BUILD_KEY)
      return noalloc_fail(GBJ_ERR_INVALID, "join_agg_noalloc: bad aggregate");
    const int o = aggs[j].operand;
    if ((o == GBJ_VAL_BUILD || o == GBJ_VAL_PRODUCT) && !d_build_payload && n_build)
      return noalloc_fail(GBJ_ERR_INVALID, "join_agg_noalloc: aggregate reads a null build payload");
    if ((o == GBJ_VAL_PROBE || o == GBJ_VAL_PRODUCT) && !d_probe_payload && n_probe)
      return noalloc_fail(GBJ_ERR_INVALID, "join_agg_noalloc: aggregate reads a null probe payload");
  }
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) {
    (void)cudaGetLastError();
    return noalloc_fail(GBJ_ERR_CUDA, "join_agg_noalloc: no current CUDA device");
  }
  NoAllocDevice d;
  {
    std::lock_guard<std::mutex> g(g_noalloc_mu);
    auto it = g_noalloc_devices.find({dev, current_context_id()});
    if (it == g_noalloc_devices.end()) {
      // first call on this device in this context: resolve the array's
      // device address (this also makes the runtime's context current)
      void *ptr = nullptr;
      cudaError_t e = cudaGetSymbolAddress(&ptr, g_noalloc_scratch);
      if (e != cudaSuccess || !ptr) {
        (void)cudaGetLastError();
        return noalloc_fail(GBJ_ERR_CUDA, "join_agg_noalloc: cudaGetSymbolAddress failed");
      }
      NoAllocDevice nd;
      nd.scratch = static_cast<uint64_t *>(ptr);
      if (cudaDeviceGetAttribute(&nd.sm_count, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
        (void)cudaGetLastError();
        return noalloc_fail(GBJ_ERR_CUDA, "join_agg_noalloc: device query failed");
      }
      it = g_noalloc_devices.insert_or_assign({dev, current_context_id()}, nd).first;
    }
    d = it->second;
  }
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  AggSpec spec = make_spec(aggs, n_aggs);
  uint64_t slots = next_pow2(2 * (n_build ? n_build : 1));
  if (slots < 64) slots = 64;
  uint64_t *table = d.scratch;
  uint32_t *meta = reinterpret_cast<uint32_t *>(d.scratch + kNoAllocSlots);
  // the array keeps the previous call's table: clear the part this call uses
  if (cudaMemsetAsync(table, 0, slots * sizeof(uint64_t), s) != cudaSuccess ||
      cudaMemsetAsync(meta, 0, sizeof(uint32_t), s) != cudaSuccess) {
    (void)cudaGetLastError();
    return noalloc_fail(GBJ_ERR_CUDA, "join_agg_noalloc: cudaMemsetAsync failed");
  }
  k_noalloc_init_out<<<1, 32, 0, s>>>(spec, d_out);
  if (n_build)
    k_join_build<<<grid_for_sms(d.sm_count, n_build, kThreads), kThreads, 0, s>>>(d_build_keys, n_build, table,
                                                                                   slots - 1, meta);
  if (n_probe)
    launch_probe(d.sm_count, d_probe_keys, d_probe_payload, n_probe, table, slots - 1,
                 d_build_payload, meta, spec, d_out, s);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return noalloc_fail(GBJ_ERR_CUDA, cudaGetErrorString(e));
  return GBJ_OK;
}

}  // extern "C"
