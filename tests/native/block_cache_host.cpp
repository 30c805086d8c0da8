// Host harness of the kept device blocks (test infrastructure).
//
// Compiles rohditor_gb300/csrc/block_cache.cuh for the CPU over a pool of its own
// that counts bytes, knows which streams live and which are being captured, and
// refuses what a device would refuse. Every call on a dead or capturing stream by
// anyone but the capture itself is a fault.
//
//   block_cache_host NAME   runs one scenario; exit code 0 when it holds
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <thread>
#include <vector>

#include "../../rohditor_gb300/csrc/block_cache.cuh"

namespace {

struct FakeStream {
  bool alive = true, capturing = false;
};

struct Pool {
  std::mutex mutex;
  std::map<void*, size_t> used;
  size_t in_use = 0, capacity = ~size_t(0), next = 0x1000;
  int faults = 0, refuse_frees = 0, finishes = 0;
};
Pool g_pool;

struct FakeGpu {
  using Stream = FakeStream*;
  static int malloc_async(void** out, size_t bytes, Stream s) {
    std::lock_guard<std::mutex> lk(g_pool.mutex);
    if (!s->alive || s->capturing) ++g_pool.faults;
    if (bytes > g_pool.capacity || g_pool.in_use > g_pool.capacity - bytes) return 2;
    *out = reinterpret_cast<void*>(g_pool.next);
    g_pool.next += bytes;
    g_pool.used[*out] = bytes;
    g_pool.in_use += bytes;
    return 0;
  }
  static bool free_async(void* ptr, Stream s) {
    std::lock_guard<std::mutex> lk(g_pool.mutex);
    if (!s->alive || s->capturing) ++g_pool.faults;
    if (g_pool.refuse_frees > 0) {
      --g_pool.refuse_frees;
      return false;
    }
    const auto it = g_pool.used.find(ptr);
    if (it == g_pool.used.end()) {
      ++g_pool.faults;
      return true;
    }
    g_pool.in_use -= it->second;
    g_pool.used.erase(it);
    return true;
  }
  static void follow(Stream waiter, Stream s) {
    std::lock_guard<std::mutex> lk(g_pool.mutex);
    if (!s->alive || s->capturing || !waiter->alive || waiter->capturing) ++g_pool.faults;
  }
  static void finish(Stream s) {
    std::lock_guard<std::mutex> lk(g_pool.mutex);
    if (!s->alive || s->capturing) ++g_pool.faults;
    ++g_pool.finishes;
  }
};
using Cache = rd::BlockCache<FakeGpu>;
constexpr size_t ROOM = ~size_t(0);

void set(FakeStream& s, bool alive, bool capturing) {
  std::lock_guard<std::mutex> lk(g_pool.mutex);
  s.alive = alive;
  s.capturing = capturing;
}

int g_failed = 0;
void expect(bool ok, const char* what) {
  if (ok) return;
  std::fprintf(stderr, "failed: %s\n", what);
  ++g_failed;
}

// An allocation that finds no room takes what the other contexts keep.
void reclaim() {
  g_pool.capacity = 100;
  FakeStream sa, sb, sc;
  Cache a, b, other_device;
  a.attach(0, &sa);
  b.attach(0, &sb);
  other_device.attach(1, &sc);
  void *p = nullptr, *q = nullptr, *r = nullptr;
  expect(b.alloc(60, ROOM, &p) == 0 && other_device.alloc(20, ROOM, &r) == 0, "room at first");
  b.free(p, ROOM);
  other_device.free(r, ROOM);
  expect(b.kept_bytes() == 60 && other_device.kept_bytes() == 20, "both keep their blocks");
  expect(a.alloc(70, ROOM, &q) == 0, "the kept blocks make room");
  expect(b.kept_bytes() == 0 && other_device.kept_bytes() == 20, "of this device only");
  void* none = nullptr;
  expect(a.alloc(1000, ROOM, &none) != 0, "more than there is stays refused");
  a.free(q, ROOM);
  void* same = nullptr;
  expect(a.alloc(70, ROOM, &same) == 0 && same == q, "a kept block serves its size");
  a.free(same, ROOM);
  a.detach();
  b.detach();
  other_device.detach();
  expect(g_pool.in_use == 0, "everything is given back");
}

// A context that is being captured keeps its blocks and is not touched.
void captured() {
  g_pool.capacity = 100;
  FakeStream sa, sb;
  Cache a, b;
  a.attach(0, &sa);
  b.attach(0, &sb);
  void* p = nullptr;
  expect(b.alloc(60, ROOM, &p) == 0, "room");
  b.free(p, ROOM);
  b.close();
  set(sb, true, true);
  void* q = nullptr;
  expect(a.alloc(70, ROOM, &q) != 0 && b.kept_bytes() == 60, "its blocks stay");
  b.shrink(0);
  expect(b.kept_bytes() == 60, "and nobody frees into the capture");
  set(sb, true, false);
  b.open();
  expect(a.alloc(70, ROOM, &q) == 0 && b.kept_bytes() == 0, "after it they go");
  a.free(q, ROOM);
  a.detach();
  b.detach();
  expect(g_pool.in_use == 0, "everything is given back");
}

// A block whose return the pool refuses is not lost.
void refused() {
  FakeStream s;
  Cache c;
  c.attach(0, &s);
  void* p[2] = {};
  for (void*& q : p) expect(c.alloc(10, ROOM, &q) == 0, "room");
  for (void* q : p) c.free(q, ROOM);
  g_pool.refuse_frees = 1;
  c.shrink(0);
  expect(c.kept_bytes() == 20, "refused blocks stay kept");
  c.shrink(0);
  expect(c.kept_bytes() == 0, "and go the next time");
  c.detach();
  expect(g_pool.in_use == 0, "everything is given back");
}

// What is kept stays within the room that a call names, the oldest going first.
void room() {
  FakeStream s;
  Cache c;
  c.attach(0, &s);
  void *p[4] = {}, *q = nullptr;
  for (int k = 0; k < 4; ++k) expect(c.alloc(10 + k, ROOM, &p[k]) == 0, "room");
  c.free(p[0], 46 - 36);
  expect(c.kept_bytes() == 10, "what fits is kept");
  c.free(p[1], 46 - 25);
  expect(c.kept_bytes() == 21, "both fit");
  expect(c.alloc(20, 46 - 45, &q) == 0 && c.kept_bytes() == 0, "kept blocks make way for a new one");
  c.free(q, 10);
  expect(c.kept_bytes() == 0, "a block larger than the room is not kept");
  c.free(p[2], ROOM);
  c.free(p[3], ROOM);
  c.shrink(13);
  expect(c.kept_bytes() == 13, "the oldest goes first");
  c.detach();
  expect(g_pool.in_use == 0, "everything is given back");
}

// A block that many frees have passed by goes back.
void passed_by() {
  FakeStream s;
  Cache c;
  c.attach(0, &s);
  void* p = nullptr;
  expect(c.alloc(7, ROOM, &p) == 0, "room");
  c.free(p, ROOM);
  for (uint64_t k = 0; k <= rd::BLOCK_CACHE_FREES; ++k) {
    expect(c.kept_bytes() == (k == 0 ? 7u : 12u), "kept until then");
    expect(c.alloc(5, ROOM, &p) == 0, "room");
    c.free(p, ROOM);
  }
  expect(c.kept_bytes() == 5, "then it goes");
  c.detach();
  expect(g_pool.in_use == 0, "everything is given back");
}

// Owners that allocate, are captured, replace their streams and come and go,
// beside each other and threads whose allocations fail.
void threads() {
  g_pool.capacity = 4000;
  std::atomic<bool> stop{false};
  std::vector<std::thread> all;
  for (unsigned seed = 1; seed <= 4; ++seed)
    all.emplace_back([seed] {
      std::vector<FakeStream*> streams;
      for (int life = 0; life < 40; ++life) {
        streams.push_back(new FakeStream);
        FakeStream* s = streams.back();
        Cache c;
        c.attach(0, s);
        unsigned h = seed * 7919u + (unsigned)life;
        for (int k = 0; k < 60; ++k) {
          h = h * 1664525u + 1013904223u;
          void* p = nullptr;
          if (c.alloc(10 + (h >> 24) % 8, ROOM, &p) == 0) c.free(p, ROOM);
          if (k % 16 == 5) {
            c.close();
            set(*s, true, true);
            std::this_thread::yield();
            set(*s, true, false);
            c.open();
          }
          if (k % 16 == 11) {
            FakeStream* old = s;
            streams.push_back(new FakeStream);
            s = streams.back();
            c.replace_stream([&] {
              set(*old, false, false);
              return s;
            });
          }
        }
        c.detach();
        set(*s, false, false);
      }
      for (FakeStream* s : streams) delete s;
    });
  all.emplace_back([&stop] {
    FakeStream s;
    Cache c;
    c.attach(0, &s);
    while (!stop) {
      void* p = nullptr;
      if (c.alloc(1 << 20, ROOM, &p) == 0) std::abort();
      std::this_thread::yield();
    }
    c.detach();
  });
  for (size_t k = 0; k + 1 < all.size(); ++k) all[k].join();
  stop = true;
  all.back().join();
  expect(g_pool.in_use == 0, "everything is given back");
  expect(g_pool.finishes > 0, "the failing thread reclaimed");
}

}  // namespace

int main(int argc, char** argv) {
  const std::map<std::string, void (*)()> scenarios = {
      {"reclaim", reclaim}, {"captured", captured},   {"refused", refused},
      {"room", room},       {"passed_by", passed_by}, {"threads", threads}};
  const auto it = argc == 2 ? scenarios.find(argv[1]) : scenarios.end();
  if (it == scenarios.end()) return 2;
  it->second();
  expect(g_pool.faults == 0, "no call on a dead or captured stream, no block freed twice");
  return g_failed ? 1 : 0;
}
