// What the autotuner tries has the untuned call's plan among it, at every size.
#include <cstdio>

#include "auto_plan.h"

using namespace gbj;

static bool has(const std::vector<int32_t> &c, int bits) {
  for (int b : c)
    if (b == bits) return true;
  return false;
}

int main() {
  for (int i = 0; i <= 31; ++i)
    for (int j = 0; j <= 31; ++j)
      for (uint64_t odd : {0, 1, 2}) {
        const uint64_t a = (1ull << i) + odd * ((1ull << i) / 3), b = (1ull << j) + odd * ((1ull << j) / 5);
        for (int threads : {512, 1024})
          if (!has(radix_candidates(a, b, threads), radix_auto_bits(a, b, threads))) {
            printf("join %llu x %llu, %d threads\n", (unsigned long long)a, (unsigned long long)b, threads);
            return 1;
          }
        const uint64_t groups = std::max<uint64_t>(1024, std::min(a, b));
        if (!has(groupby_candidates(b, groups), groupby_auto_bits(b, groups, false))) {
          printf("group-by %llu rows, %llu groups\n", (unsigned long long)b, (unsigned long long)groups);
          return 1;
        }
      }
  printf("ok\n");
  return 0;
}
