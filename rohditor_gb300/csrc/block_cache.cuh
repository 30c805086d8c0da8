// Device blocks that a context has freed and keeps for its next allocations of
// the same size, and the way they are given back when the device runs out of
// memory.
//
// What is kept is bounded: by the room that the owner names with each call (its
// budget less what it has in use), by BLOCK_CACHE_BYTES, and by use, since a block
// that the next BLOCK_CACHE_FREES frees have passed by goes back (a session that
// opens frames of other sizes does not hold the old sizes' blocks for good).
//
// A cache belongs to one context and one thread at a time, its owner, who
// allocates and frees through it. Any thread whose allocation fails may take the
// kept blocks of every cache of the device (reclaim). What both touch (the kept
// blocks, the stream that they are ordered by, whether that stream is being
// captured) is guarded by the cache's mutex: the owner closes the cache before
// its stream joins a capture and opens it after the capture has ended, and
// replaces its stream under the lock. The list of caches has a mutex of its own,
// taken before a cache's; nobody waits for the device while holding either.
//
// Plain C++: `Gpu` supplies the calls (api.cu has CUDA's, a host test its own).
//   Stream                                    a copyable handle
//   int malloc_async(void**, size_t, Stream)  0, or the error
//   bool free_async(void*, Stream)            false: refused, the block is still there
//   void follow(Stream waiter, Stream s)      waiter's next work waits for what s has been given
//   void finish(Stream)                       waits for the stream
#pragma once

#include <stddef.h>
#include <stdint.h>

#include <mutex>
#include <unordered_map>
#include <vector>

namespace rd {

constexpr size_t BLOCK_CACHE_BYTES = size_t(8) << 30;
constexpr size_t BLOCK_CACHE_BLOCKS = 64;
constexpr uint64_t BLOCK_CACHE_FREES = 256;  // a dozen develops

template <class Gpu>
class BlockCache {
 public:
  using Stream = typename Gpu::Stream;
  BlockCache() = default;
  BlockCache(const BlockCache&) = delete;
  BlockCache& operator=(const BlockCache&) = delete;

  // Owner: from now on blocks are ordered by `stream`, until detach, which gives
  // every kept one back.
  void attach(int device, Stream stream) {
    device_ = device;
    stream_ = stream;
    try {
      kept_.reserve(BLOCK_CACHE_BLOCKS + 1);
    } catch (...) {  // nothing is kept then
    }
    std::lock_guard<std::mutex> all(registry().mutex);
    next_ = registry().first;
    if (next_) next_->before_ = this;
    registry().first = this;
    attached_ = true;
  }
  void detach() {
    if (!attached_) return;
    {
      std::lock_guard<std::mutex> all(registry().mutex);
      if (next_) next_->before_ = before_;
      (before_ ? before_->next_ : registry().first) = next_;
      attached_ = false;
    }
    shrink(0);
  }

  // Owner: a block of `bytes`, kept or new; no more than `room` bytes stay kept
  // beside it. When the pool has none, every cache's kept blocks are given back and
  // it is asked again. 0, or the pool's error.
  int alloc(size_t bytes, size_t room, void** out) {
    {
      std::lock_guard<std::mutex> lk(mutex_);
      for (size_t k = kept_.size(); k-- > 0;)
        if (kept_[k].bytes == bytes) {
          *out = kept_[k].ptr;
          kept_.erase(kept_.begin() + (ptrdiff_t)k);
          bytes_ -= bytes;
          hand_out(*out, bytes);
          give_back(room, BLOCK_CACHE_BLOCKS);
          return 0;
        }
      give_back(room, BLOCK_CACHE_BLOCKS);
    }
    int e = Gpu::malloc_async(out, bytes, stream_);
    if (e) {
      reclaim(device_, stream_);
      e = Gpu::malloc_async(out, bytes, stream_);
    }
    if (!e) {
      std::lock_guard<std::mutex> lk(mutex_);
      hand_out(*out, bytes);
    }
    return e;
  }

  // Owner: a block that alloc gave, to be kept where `room` bytes hold it; one that
  // it did not give, or any while the cache is closed, goes back to the pool.
  void free(void* ptr, size_t room) {
    std::lock_guard<std::mutex> lk(mutex_);
    const auto it = live_.find(ptr);
    const size_t bytes = it == live_.end() ? 0 : it->second;
    if (bytes) live_.erase(it);
    if (bytes == 0 || closed_ || bytes > room || bytes > BLOCK_CACHE_BYTES || kept_.size() == kept_.capacity()) {
      Gpu::free_async(ptr, stream_);
      return;
    }
    kept_.push_back(Kept{ptr, bytes, ++frees_});
    bytes_ += bytes;
    give_back(room < BLOCK_CACHE_BYTES ? room : BLOCK_CACHE_BYTES, BLOCK_CACHE_BLOCKS);
  }

  // Owner: before the stream joins a capture, and after the capture has ended.
  void close() {
    std::lock_guard<std::mutex> lk(mutex_);
    closed_ = true;
  }
  void open() {
    std::lock_guard<std::mutex> lk(mutex_);
    closed_ = false;
  }
  // Owner: the blocks are ordered by the stream that `replace` returns; the old
  // one, which is idle, may be destroyed in it.
  template <class Replace>
  void replace_stream(Replace&& replace) {
    std::lock_guard<std::mutex> lk(mutex_);
    stream_ = replace();
  }

  // Gives the oldest blocks back until no more than `bytes` are kept.
  void shrink(size_t bytes) {
    std::lock_guard<std::mutex> lk(mutex_);
    if (!closed_) give_back(bytes, BLOCK_CACHE_BLOCKS);
  }
  size_t kept_bytes() const {
    std::lock_guard<std::mutex> lk(mutex_);
    return bytes_;
  }

  // Any thread: the kept blocks of the device's caches back to the pool, and
  // `waiter` finished behind them.
  static void reclaim(int device, Stream waiter) {
    {
      std::lock_guard<std::mutex> all(registry().mutex);
      for (BlockCache* c = registry().first; c; c = c->next_) {
        if (c->device_ != device) continue;
        std::lock_guard<std::mutex> lk(c->mutex_);
        if (c->closed_ || c->kept_.empty()) continue;
        c->give_back(0, 0);
        Gpu::follow(waiter, c->stream_);
      }
    }
    Gpu::finish(waiter);
  }

 private:
  struct Kept {
    void* ptr;
    size_t bytes;
    uint64_t at;  // the free that brought it
  };
  struct Registry {
    std::mutex mutex;
    BlockCache* first = nullptr;
  };
  static Registry& registry() {
    static Registry r;
    return r;
  }

  // Under the lock. A block whose size cannot be noted is not kept later.
  void hand_out(void* ptr, size_t bytes) {
    try {
      live_[ptr] = bytes;
    } catch (...) {
    }
  }
  // Under the lock: the oldest first, down to so many bytes and blocks, and those
  // that were passed by. A block that the pool refuses stays.
  void give_back(size_t bytes, size_t blocks) {
    while (!kept_.empty() &&
           (bytes_ > bytes || kept_.size() > blocks || kept_.front().at + BLOCK_CACHE_FREES < frees_)) {
      if (!Gpu::free_async(kept_.front().ptr, stream_)) return;
      bytes_ -= kept_.front().bytes;
      kept_.erase(kept_.begin());
    }
  }

  mutable std::mutex mutex_;
  std::vector<Kept> kept_;                     // oldest first
  std::unordered_map<void*, size_t> live_;     // blocks handed out
  size_t bytes_ = 0;                           // of the kept blocks
  uint64_t frees_ = 0;                         // blocks kept so far
  bool closed_ = false;
  Stream stream_{};                            // changed by the owner only, under the lock
  int device_ = 0;
  bool attached_ = false;
  BlockCache* next_ = nullptr;                 // under the registry's lock
  BlockCache* before_ = nullptr;
};

}  // namespace rd
