// The device pool's ranges; see pool.h.  No kernels.
#include "pool.h"

#include <algorithm>
#include <iterator>
#include <utility>

namespace gbj {
namespace {

void insert_free(Pool &p, uint64_t off, uint64_t size) {
  auto it = p.free_by_off.lower_bound(off);
  if (it != p.free_by_off.end() && off + size == it->first) {
    size += it->second;
    it = p.free_by_off.erase(it);
  }
  if (it != p.free_by_off.begin()) {
    auto prev = std::prev(it);
    if (prev->first + prev->second == off) {
      prev->second += size;
      return;
    }
  }
  p.free_by_off.emplace(off, size);
}

bool completed(cudaEvent_t ev, bool wait) {
  const cudaError_t q = wait ? cudaEventSynchronize(ev) : cudaEventQuery(ev);
  if (q != cudaSuccess && q != cudaErrorNotReady) (void)cudaGetLastError();
  return q == cudaSuccess;
}

bool capturing(cudaStream_t s) {
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(s, &cap) != cudaSuccess) (void)cudaGetLastError();
  return cap != cudaStreamCaptureStatusNone;
}

// Drops the uses that have ended; true: all of them.
bool ended(BlockUses &uses, bool wait) {
  for (auto it = uses.begin(); it != uses.end();) {
    if (completed(it->second, wait)) {
      cudaEventDestroy(it->second);
      it = uses.erase(it);
    } else {
      ++it;
    }
  }
  return uses.empty();
}
void drop(BlockUses &uses) {
  for (auto &u : uses) cudaEventDestroy(u.second);
}

// Frees the other streams' ranges whose work is done; `wait` waits for it.  A
// captured event never completes: its range is everyone's again with the next
// request on its stream.
void reclaim(Pool &p, cudaStream_t s, bool wait) {
  for (auto it = p.deferred.begin(); it != p.deferred.end();) {
    Pool::Deferred &d = it->second;
    if (d.of(s) ? d.captured : ended(d.uses, wait)) {
      drop(d.uses);
      insert_free(p, it->first, d.size);
      it = p.deferred.erase(it);
    } else {
      ++it;
    }
  }
}

// Best fit among the runs of free ranges and ranges of s.
bool fit(const Pool &p, uint64_t size, cudaStream_t s, uint64_t *off) {
  auto f = p.free_by_off.begin();
  auto d = p.deferred.begin();
  uint64_t run = 0, end = 0, best = UINT64_MAX;  // the run is [run, end)
  auto close = [&] {
    if (end - run >= size && end - run < best) {
      best = end - run;
      *off = run;
    }
  };
  for (;;) {
    while (d != p.deferred.end() && !d->second.of(s)) ++d;
    const bool has_f = f != p.free_by_off.end(), has_d = d != p.deferred.end();
    if (!has_f && !has_d) break;
    uint64_t o, n;
    if (has_f && (!has_d || f->first < d->first)) {
      o = f->first, n = f->second;
      ++f;
    } else {
      o = d->first, n = d->second.size;
      ++d;
    }
    if (o != end) {
      close();
      run = o;
    }
    end = o + n;
  }
  close();
  return best != UINT64_MAX;
}

// Takes [off, off + size) out of the run that starts there.
void carve(Pool &p, uint64_t off, uint64_t size, cudaStream_t s) {
  const uint64_t end = off + size;
  for (auto it = p.free_by_off.lower_bound(off); it != p.free_by_off.end() && it->first < end;) {
    const uint64_t e = it->first + it->second;
    it = p.free_by_off.erase(it);
    if (e > end) p.free_by_off.emplace(end, e - end);
  }
  for (auto it = p.deferred.lower_bound(off); it != p.deferred.end() && it->first < end;) {
    Pool::Deferred d = std::move(it->second);
    const uint64_t e = it->first + d.size;
    it = p.deferred.erase(it);
    if (e > end) {
      d.size = e - end;
      p.deferred.emplace(end, std::move(d));
    } else {
      drop(d.uses);
    }
  }
}

}  // namespace

bool pool_take(Pool &p, uint64_t size, cudaStream_t s, uint64_t *off) {
  reclaim(p, s, false);
  if (!fit(p, size, s, off)) {
    reclaim(p, s, true);
    if (!fit(p, size, s, off)) return false;
  }
  carve(p, *off, size, s);
  return true;
}

static void defer(Pool &p, uint64_t off, Pool::Deferred d) {
  // ranges of the same stream beside it: free when their work is done, else
  // one range with it, behind the later event
  auto merges = [&](const Pool::Deferred &o) {
    return d.uses.size() == 1 && o.of(d.uses[0].first) && !o.captured && !d.captured;
  };
  auto it = p.deferred.lower_bound(off);
  if (it != p.deferred.end() && it->first == off + d.size && merges(it->second)) {
    if (completed(it->second.uses[0].second, false)) insert_free(p, it->first, it->second.size);
    else d.size += it->second.size;
    drop(it->second.uses);
    it = p.deferred.erase(it);
  }
  if (it != p.deferred.begin()) {
    auto prev = std::prev(it);
    if (prev->first + prev->second.size == off && merges(prev->second)) {
      if (completed(prev->second.uses[0].second, false)) {
        insert_free(p, prev->first, prev->second.size);
      } else {
        off = prev->first;
        d.size += prev->second.size;
      }
      drop(prev->second.uses);
      p.deferred.erase(prev);
    }
  }
  p.deferred.emplace(off, std::move(d));
}

void pool_give(Pool &p, uint64_t off, uint64_t size, cudaStream_t s) {
  const bool cap = capturing(s);
  cudaEvent_t ev = nullptr;
  if (cudaEventCreateWithFlags(&ev, cudaEventDisableTiming) != cudaSuccess || cudaEventRecord(ev, s) != cudaSuccess) {
    // an event that cannot be recorded: fall back to a full sync
    (void)cudaGetLastError();
    if (ev) cudaEventDestroy(ev);
    cudaStreamSynchronize(s);
    (void)cudaGetLastError();
    insert_free(p, off, size);
    return;
  }
  defer(p, off, {size, {{s, ev}}, cap});
}

void pool_give(Pool &p, uint64_t off, uint64_t size, BlockUses uses) {
  if (ended(uses, false)) insert_free(p, off, size);
  else defer(p, off, {size, std::move(uses), false});
}

void pool_note_use(BlockUses &uses, cudaStream_t s) {
  if (capturing(s)) return;
  cudaEvent_t ev = nullptr;
  for (auto &u : uses)
    if (u.first == s) ev = u.second;
  if (!ev) {
    if (cudaEventCreateWithFlags(&ev, cudaEventDisableTiming) == cudaSuccess) uses.push_back({s, ev});
    else ev = nullptr;
  }
  if (!ev || cudaEventRecord(ev, s) != cudaSuccess) {  // nothing left in flight instead
    (void)cudaGetLastError();
    cudaStreamSynchronize(s);
    (void)cudaGetLastError();
  }
}

}  // namespace gbj
