// The device pool's bookkeeping: best fit over one block of device memory,
// with ranges that were given back but may still be in use (host code only).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <map>
#include <unordered_map>

struct Pool {
  char *base = nullptr;
  uint64_t capacity = 0, in_use = 0, peak = 0;
  uint64_t limit = 0;  // gbj_ctx_set_pool_limit: most bytes handed out (0 = capacity)
  std::map<uint64_t, uint64_t> free_by_off;  // offset -> size, nobody's
  std::unordered_map<uint64_t, uint64_t> used;  // offset -> size
  // Given back behind work on a stream: that stream may use it again at once
  // (stream order), everyone once the event has completed.
  struct Deferred {
    uint64_t size;
    cudaStream_t stream;
    cudaEvent_t ev;
    bool captured;  // the event is part of a graph and cannot be asked
  };
  std::map<uint64_t, Deferred> deferred;  // offset -> range
};

namespace gbj {

// Takes `size` bytes for work on s: from free ranges and those that s itself
// gave back, adjacent ones together.  What is left of a range of s stays
// behind its event.  Waits for other streams' ranges when nothing else fits;
// false when that is not enough.
bool pool_take(Pool &p, uint64_t size, cudaStream_t s, uint64_t *off);
// Gives [off, off + size) back behind the work enqueued on s so far.
void pool_give(Pool &p, uint64_t off, uint64_t size, cudaStream_t s);

}  // namespace gbj
