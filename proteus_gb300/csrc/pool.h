// The device pool's bookkeeping: best fit over one block of device memory,
// with ranges that were given back but may still be in use (host code only).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <map>
#include <unordered_map>
#include <utility>
#include <vector>

// The streams that have used a block, each with an event behind its last use.
using BlockUses = std::vector<std::pair<cudaStream_t, cudaEvent_t>>;

struct Pool {
  char *base = nullptr;
  uint64_t capacity = 0, in_use = 0, peak = 0;
  uint64_t limit = 0;  // gbj_ctx_set_pool_limit: most bytes handed out (0 = capacity)
  std::map<uint64_t, uint64_t> free_by_off;  // offset -> size, nobody's
  std::unordered_map<uint64_t, uint64_t> used;  // offset -> size
  // Given back behind work on streams: everyone may use it once that has
  // ended, and the stream, when it is only one, at once (stream order).
  struct Deferred {
    uint64_t size;
    BlockUses uses;  // at least one
    bool captured;   // its event is part of a graph and cannot be asked
    bool of(cudaStream_t s) const { return uses.size() == 1 && uses[0].first == s; }
  };
  std::map<uint64_t, Deferred> deferred;  // offset -> range
};

namespace gbj {

// Takes `size` bytes for work on s: from free ranges and those that s itself
// gave back, adjacent ones together (s null: for any stream, free ranges only).
// What is left of a range of s stays behind its event.  Waits for other streams' ranges when nothing else fits;
// false when that is not enough.
bool pool_take(Pool &p, uint64_t size, cudaStream_t s, uint64_t *off);
// Gives [off, off + size) back behind the work enqueued on s so far.
void pool_give(Pool &p, uint64_t off, uint64_t size, cudaStream_t s);
// Gives it back behind the events of `uses`, which it takes over.
void pool_give(Pool &p, uint64_t off, uint64_t size, BlockUses uses);

// Notes that the work enqueued on s so far uses a block.  Work that is being
// captured is not followed: whoever replays a graph keeps what it reads.
void pool_note_use(BlockUses &uses, cudaStream_t s);

}  // namespace gbj
