// The device pool against a model of streams: its CUDA calls are the fakes
// below, every stream is a queue of work that completes when the test says so.
// A range handed out must not be in use by unfinished work of another stream.
#include <cstdio>
#include <cstdlib>
#include <initializer_list>
#include <random>
#include <utility>
#include <vector>

#include "pool.h"

namespace {
struct Event {
  cudaStream_t s = nullptr;
  uint64_t at = 0;
};
uint64_t issued[4], done[4];  // by stream: work enqueued, work completed
int live_events = 0, waits = 0;
cudaStream_t stream(int i) { return reinterpret_cast<cudaStream_t>(static_cast<uintptr_t>(i + 1)); }
int index_of(cudaStream_t s) { return (int)reinterpret_cast<uintptr_t>(s) - 1; }
}  // namespace

extern "C" {
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) {
  ++live_events;
  *e = reinterpret_cast<cudaEvent_t>(new Event);
  return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
  *reinterpret_cast<Event *>(e) = {s, issued[index_of(s)]};
  return cudaSuccess;
}
cudaError_t cudaEventQuery(cudaEvent_t e) {
  const Event &v = *reinterpret_cast<Event *>(e);
  return done[index_of(v.s)] >= v.at ? cudaSuccess : cudaErrorNotReady;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
  const Event &v = *reinterpret_cast<Event *>(e);
  uint64_t &d = done[index_of(v.s)];
  if (d < v.at) d = v.at, ++waits;
  return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) {
  --live_events;
  delete reinterpret_cast<Event *>(e);
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
  done[index_of(s)] = issued[index_of(s)];
  return cudaSuccess;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus *st) {
  *st = cudaStreamCaptureStatusNone;
  return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
}

namespace {
constexpr uint64_t kUnit = 256, kUnits = 64;

struct Model {
  Pool p;
  // of each unit: the last work that used it, by stream
  uint64_t last[kUnits][4] = {};
  struct Block {
    uint64_t off, size;
  };
  std::vector<Block> held;
  Model() { p.free_by_off.emplace(0, kUnit * kUnits); }

  bool take(uint64_t units, int s) {
    uint64_t off;
    if (!gbj::pool_take(p, units * kUnit, stream(s), &off)) return false;
    for (uint64_t u = off / kUnit; u < off / kUnit + units; ++u)
      for (int o = 0; o < 4; ++o)
        if (o != s && done[o] < last[u][o]) {
          printf("unit %llu given to stream %d while stream %d uses it\n", (unsigned long long)u, s, o);
          exit(1);
        }
    for (const Block &b : held)
      if (off < b.off + b.size && b.off < off + units * kUnit) {
        printf("overlap\n");
        exit(1);
      }
    held.push_back({off, units * kUnit});
    return true;
  }
  // work on s that uses block i
  void use(size_t i, int s) {
    ++issued[s];
    for (uint64_t u = held[i].off / kUnit; u < (held[i].off + held[i].size) / kUnit; ++u) last[u][s] = issued[s];
  }
  void give(size_t i, int s) {
    const Block b = held[i];
    held.erase(held.begin() + (long)i);
    gbj::pool_give(p, b.off, b.size, stream(s));
  }
  // given back behind all that streams a, b, .. were last made to do with it
  void give_used(size_t i, std::initializer_list<int> streams) {
    BlockUses uses;
    for (int s : streams) use(i, s), gbj::pool_note_use(uses, stream(s));
    const Block b = held[i];
    held.erase(held.begin() + (long)i);
    gbj::pool_give(p, b.off, b.size, std::move(uses));
  }
  // every byte is in exactly one place
  void check() {
    uint64_t sum = 0;
    for (auto &f : p.free_by_off) sum += f.second;
    int events = 0;
    for (auto &d : p.deferred) sum += d.second.size, events += (int)d.second.uses.size();
    for (const Block &b : held) sum += b.size;
    if (sum != kUnit * kUnits || live_events != events) {
      printf("bytes or events lost\n");
      exit(1);
    }
  }
};

void require(bool ok, const char *what) {
  if (!ok) {
    printf("%s\n", what);
    exit(1);
  }
}
}  // namespace

int main() {
  {  // what a request of the same stream leaves of a range stays behind its work
    Model m;
    m.take(kUnits, 0), m.use(0, 0), m.give(0, 0);
    m.take(4, 0);
    require(waits == 0, "the same stream waited");
    m.take(kUnits - 4, 1);
    require(waits == 1, "another stream did not wait");
    m.check();
  }
  {  // neighbours given back by one stream serve it as one range
    Model m;
    for (int i = 0; i < 8; ++i) m.take(kUnits / 8, 0), m.use((size_t)i, 0);
    for (int i = 0; i < 8; ++i) m.give(m.held.size() / 2, 0), m.check();
    const int w = waits;
    require(m.take(kUnits, 0) && waits == w, "adjacent ranges were not used together");
    m.check();
  }
  {  // a block that two streams use: the one whose work has ended does not free it
    Model m;
    m.take(kUnits, 0), m.use(0, 0);
    m.give_used(0, {0, 1, 0});
    done[1] = issued[1];
    const int w = waits;
    require(m.take(4, 0) && waits == w, "the one stream left waited");
    require(m.take(4, 2) && waits == w + 1, "a third stream did not wait");
    m.check();
  }
  {  // a block for any stream is nobody's
    Model m;
    m.take(kUnits / 2, 0), m.use(0, 0), m.give(0, 0);
    const int w = waits;
    uint64_t off;
    require(gbj::pool_take(m.p, kUnit * kUnits / 2, nullptr, &off) && off == kUnit * kUnits / 2 && waits == w,
            "a range in use was given to any stream");
    require(gbj::pool_take(m.p, kUnit, nullptr, &off) && waits == w + 1, "a range in use was not waited for");
    m.held = {{0, kUnit}, {kUnit * kUnits / 2, kUnit * kUnits / 2}};
    m.check();
  }
  for (unsigned seed = 0; seed < 300; ++seed) {
    Model m;
    std::mt19937 rng(seed);
    for (int step = 0; step < 400; ++step) {
      const int s = (int)(rng() % 3);
      switch (rng() % 5) {
        case 0:
        case 1:
          if (m.take(1 + rng() % (seed % 2 ? 40 : 8), s)) m.use(m.held.size() - 1, s), m.give(m.held.size() - 1, s);
          break;
        case 2:
          if (m.held.size() < 6) m.take(1 + rng() % 8, s);
          break;
        case 3:  // a block that several streams have used for a while
          if (!m.held.empty()) {
            const size_t i = rng() % m.held.size();
            const int o = (int)(rng() % 3);
            m.give_used(i, {0, 1, 2, s, o, s});
          }
          break;
        case 4:
          if (done[s] < issued[s]) done[s] += 1 + rng() % (issued[s] - done[s]);
          break;
      }
      m.check();
    }
    for (int o = 0; o < 4; ++o) done[o] = issued[o];
    while (!m.held.empty()) m.give(0, 0);
    require(m.take(kUnits, 3), "not everything came back");
    m.give(0, 3);
    for (auto &d : m.p.deferred)
      for (auto &u : d.second.uses) cudaEventDestroy(u.second);
    m.p.deferred.clear();
  }
  printf("ok\n");
  return 0;
}
