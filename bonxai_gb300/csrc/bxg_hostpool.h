// Host buffers of a server's requests, cut from a few page-locked blocks.
#pragma once

#include <algorithm>
#include <cstdint>
#include <cstdlib>
#include <map>
#include <mutex>
#include <vector>

namespace bxg {

// Buffers that are kept between requests: the client's copy into one touches no new pages,
// and the worker's copy to the GPU reads it in place. The first block is made with the
// server (16 MB: 0.5 ms); a request that finds no room takes plain memory, because
// page-locking is a call into the driver that may not be made during a stream capture, and the
// worker then makes another block, until kMost bytes are held. Any room is good for any
// size: freed neighbours are joined. The blocks are freed with the pool.
class HostPool {
 public:
  static constexpr size_t kFirst = size_t(16) << 20;
  static constexpr size_t kBlock = size_t(32) << 20;
  static constexpr size_t kMost = size_t(256) << 20;
  using Alloc = void* (*)(size_t);  // nullptr: none
  using Free = void (*)(void*);

  HostPool(Alloc alloc, Free free) : alloc_(alloc), free_(free) {}
  HostPool(const HostPool&) = delete;
  HostPool& operator=(const HostPool&) = delete;
  ~HostPool() {
    for (Block& b : blocks_) free_(b.base);
  }

  // The first block.
  void start() { add(kFirst); }

  // *room: the bytes taken of the pool, 0 for plain memory. nullptr: no memory.
  void* take(size_t bytes, size_t* room) {
    *room = 0;
    if (bytes <= kMost) {
      const size_t want = (std::max<size_t>(bytes, 1) + kUnit - 1) / kUnit * kUnit;
      std::lock_guard<std::mutex> lk(mu_);
      for (Block& b : blocks_)
        for (auto f = b.free.begin(); f != b.free.end(); ++f) {
          if (f->second < want) continue;
          const size_t at = f->first, left = f->second - want;
          b.free.erase(f);
          if (left) b.free[at + want] = left;
          *room = want;
          return b.base + at;
        }
      missed_ = std::max(missed_, want);
    }
    return std::malloc(bytes ? bytes : 1);
  }

  void give(void* p, size_t room) {
    if (!room) {
      std::free(p);
      return;
    }
    std::lock_guard<std::mutex> lk(mu_);
    uint8_t* const q = static_cast<uint8_t*>(p);
    for (Block& b : blocks_) {
      if (q < b.base || q >= b.base + b.size) continue;
      auto f = b.free.emplace(size_t(q - b.base), room).first;
      const auto next = std::next(f);
      if (next != b.free.end() && f->first + f->second == next->first) {
        f->second += next->second;
        b.free.erase(next);
      }
      if (f != b.free.begin()) {
        const auto before = std::prev(f);
        if (before->first + before->second == f->first) {
          before->second += f->second;
          b.free.erase(f);
        }
      }
      return;
    }
  }

  // (worker) Another block after a request found no room.
  void refill() {
    size_t want = 0;
    {
      std::lock_guard<std::mutex> lk(mu_);
      std::swap(want, missed_);
    }
    if (want) add(std::max(want, kBlock));
  }

  size_t held() const {
    std::lock_guard<std::mutex> lk(mu_);
    return held_;
  }

 private:
  static constexpr size_t kUnit = 4096;
  struct Block {
    uint8_t* base;
    size_t size;
    std::map<size_t, size_t> free;  // place -> bytes
  };
  void add(size_t size) {
    {
      std::lock_guard<std::mutex> lk(mu_);
      if (held_ + size > kMost) return;
    }
    void* p = alloc_(size);
    if (!p) return;
    std::lock_guard<std::mutex> lk(mu_);
    held_ += size;
    blocks_.push_back(Block{static_cast<uint8_t*>(p), size, {{0, size}}});
  }
  Alloc alloc_;
  Free free_;
  mutable std::mutex mu_;
  std::vector<Block> blocks_;
  size_t held_ = 0, missed_ = 0;
};

}  // namespace bxg
