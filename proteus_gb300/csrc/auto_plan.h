// The plans that calls without explicit sizing take, and the ones around them
// that the autotuner tries (host code only).
#pragma once
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <vector>

namespace gbj {

constexpr int kMaxPartBits = 15;

// ------------------------------------------------------------ radix join
// The two join kernel shapes: 1024 threads with build chunks of 9216 tuples
// (one block per SM), or 512 threads with chunks of 4608 (two blocks per
// SM; partitions then need one more radix bit).
struct JoinShape {
  int threads, rmax;
};
constexpr JoinShape kJoinWide{1024, 9216};
constexpr JoinShape kJoinPair{512, 4608};
constexpr int kPairRoom = 3900;  // a fuller 512-thread table loses more than a bit costs

// The fewest radix bits whose largest expected build partition (mean + 5 sd)
// has at most `room` tuples.
inline int radix_fit_bits(uint64_t n_build, int room) {
  int b = 1;
  while (b < kMaxPartBits) {
    const double mean = (double)n_build / (double)(1u << b);
    if (mean + 5.0 * std::sqrt(mean) <= (double)room) break;
    ++b;
  }
  return b;
}

// 256 to 1024 partitions of about 2^14 tuples of both sides: fewer leave
// SMs without work (2^16 and 2^20 rows: 4 bits 219 us, 8 bits 69), more
// cost a table set-up of 4 us each (12 bits at 2^20 and 2^24 rows 260 us, 10
// bits 200, 8 bits 316).
inline int radix_even_bits(uint64_t n_build, uint64_t n_probe) {
  int b = 0;
  while (b < 10 && (1ull << b) < ((n_build + n_probe) >> 14)) ++b;
  return std::max(8, b);
}

// Bits for a kernel shape, by its threads.
inline int radix_auto_bits(uint64_t n_build, uint64_t n_probe, int threads) {
  return std::max(radix_even_bits(n_build, n_probe),
                  radix_fit_bits(n_build, threads == kJoinPair.threads ? kPairRoom : kJoinWide.rmax));
}

// Two 512-thread blocks per SM while their partitions are small enough at 10
// bits, else 1024 threads, which take twice the tuples and so one radix bit
// less (us; 4 M and 128 M rows: 512 threads at 10 bits 1144, at 11 bits
// 1076, 1024 threads at 10 bits 1080; 16 M and 64 M: 512 at 12 bits 799,
// 1024 at 11 bits 752; 30 M and 128 M: 512 at 13 bits, two passes, 1758,
// 1024 at 12 bits 1478; 2^27 and 2^29: 15 bits 7631, 14 bits 7162).
inline int radix_auto_threads(uint64_t n_build, uint64_t n_probe) {
  return radix_auto_bits(n_build, n_probe, kJoinPair.threads) <= 10 ? kJoinPair.threads : kJoinWide.threads;
}

// What the autotuner tries with a shape: the bits around the untuned plan's and
// around the fewest whose mean partition fits.
inline std::vector<int32_t> radix_candidates(uint64_t n_build, uint64_t n_probe, int threads) {
  const JoinShape shape = threads == kJoinWide.threads ? kJoinWide : kJoinPair;
  int fit = 1;
  while (fit < kMaxPartBits && (double)n_build / (double)(1u << fit) > (double)shape.rmax) ++fit;
  const int own = radix_auto_bits(n_build, n_probe, threads);
  std::vector<int32_t> c;
  for (int b = 1; b <= kMaxPartBits; ++b)
    if (std::abs(b - fit) <= 2 || std::abs(b - own) <= 1) c.push_back(b);
  return c;
}

// ------------------------------------------------------------- group-by
// Partitions so that each holds about a quarter of the on-chip table's 4096
// slots in groups.
inline int groupby_fit_bits(uint64_t groups) {
  int b = 1;
  while (b < kMaxPartBits && (groups >> b) > 1024) ++b;
  return b;
}

// Bits of the radix-partitioned strategy: without adding a partitioning pass,
// until a partition has 16,384 rows (4 M rows, 5000 groups: 8 bits 121 us, 6
// bits 147) and is usually one work item, which is emitted directly.  One pass
// over 9 to 11 bits costs less than over 12, so there the items are longer
// instead (2^28 rows, 2^20 groups: 11 bits 2840 us, 12 bits 3032).  `least`:
// partitions of 65,536 rows, whose tables of offsets are fewer words.
inline int groupby_auto_bits(uint64_t n, uint64_t groups, bool least) {
  int bits = groupby_fit_bits(groups);
  const bool long_items = bits <= 11 && !least;
  const int free_bits = bits <= 8 ? 8 : long_items ? 11 : kMaxPartBits;
  const uint64_t rows = long_items ? 16384 : 65536;
  while (bits < free_bits && (n >> bits) > rows) ++bits;
  return bits;
}

// What the autotuner tries: as for the join.
inline std::vector<int32_t> groupby_candidates(uint64_t n, uint64_t groups) {
  const int fit = groupby_fit_bits(groups), own = groupby_auto_bits(n, groups, false);
  std::vector<int32_t> c;
  for (int b = 1; b <= kMaxPartBits; ++b)
    if ((b >= fit - 1 && b <= fit + 2) || std::abs(b - own) <= 1) c.push_back(b);
  return c;
}

}  // namespace gbj
