// HostPool on ordinary memory: prints "ok", or what was wrong.
#include <cstdio>
#include <cstring>
#include <random>
#include <set>
#include <vector>

#include "bxg_hostpool.h"

using bxg::HostPool;

static size_t g_live = 0;
static bool g_fail = false;
static void* get(size_t n) {
  if (g_fail) return nullptr;
  g_live++;
  return std::malloc(n);
}
static void put(void* p) {
  g_live--;
  std::free(p);
}

#define CHECK(c)                                   \
  do {                                             \
    if (!(c)) {                                    \
      std::printf("line %d: %s\n", __LINE__, #c);  \
      return 1;                                    \
    }                                              \
  } while (0)

int main() {
  constexpr size_t MB = 1 << 20;
  struct Held {
    uint8_t* p;
    size_t bytes, room;
    uint8_t fill;
  };
  {
    HostPool pool(get, put);
    pool.start();
    size_t room = 0;
    // the first request is served from the pool
    void* a = pool.take(100000, &room);
    CHECK(a && room >= 100000);
    pool.give(a, room);
    // many small requests at once, beyond all blocks, and then large ones
    std::vector<Held> held;
    for (int round = 0; round < 3; ++round) {
      for (int i = 0; i < 6000; ++i) {
        Held h{nullptr, 64 << 10, 0, uint8_t(i)};
        h.p = static_cast<uint8_t*>(pool.take(h.bytes, &h.room));
        CHECK(h.p);
        held.push_back(h);
        if (i % 100 == 0) pool.refill();
        CHECK(pool.held() <= HostPool::kMost);
      }
      for (Held& h : held) pool.give(h.p, h.room);
      held.clear();
    }
    void* b = pool.take(HostPool::kBlock, &room);
    CHECK(b && room == HostPool::kBlock);
    pool.give(b, room);
    // random sizes: no two buffers overlap, and everything is joined again
    std::mt19937 rng(1);
    for (int i = 0; i < 20000; ++i) {
      if (held.size() < 40 || rng() % 2) {
        Held h{nullptr, rng() % (3 * MB), 0, uint8_t(rng())};
        h.p = static_cast<uint8_t*>(pool.take(h.bytes, &h.room));
        CHECK(h.p && (!h.room || h.room >= h.bytes));
        std::memset(h.p, h.fill, std::min<size_t>(h.bytes, 512));
        if (h.bytes > 512) std::memset(h.p + h.bytes - 512, h.fill, 512);
        held.push_back(h);
      } else {
        std::swap(held[rng() % held.size()], held.back());
        Held h = held.back();
        held.pop_back();
        for (size_t k = 0; k < std::min<size_t>(h.bytes, 512); ++k) CHECK(h.p[k] == h.fill);
        for (size_t k = 1; k <= 512 && h.bytes > 512; ++k) CHECK(h.p[h.bytes - k] == h.fill);
        pool.give(h.p, h.room);
      }
    }
    for (Held& h : held) pool.give(h.p, h.room);
    b = pool.take(HostPool::kBlock, &room);
    CHECK(b && room == HostPool::kBlock);
    pool.give(b, room);
    // larger than the pool may become
    b = pool.take(HostPool::kMost + 1, &room);
    CHECK(b && room == 0);
    pool.give(b, room);
  }
  CHECK(g_live == 0);
  {  // no page-locked memory: plain memory, and nothing counted as held
    g_fail = true;
    HostPool pool(get, put);
    pool.start();
    size_t room = 1;
    void* a = pool.take(1000, &room);
    CHECK(a && room == 0);
    pool.refill();
    pool.give(a, room);
    CHECK(pool.held() == 0);
    g_fail = false;
    a = pool.take(1000, &room);
    pool.refill();
    pool.give(a, room);
    CHECK(pool.held() == HostPool::kBlock);
    a = pool.take(1000, &room);
    CHECK(room);
    pool.give(a, room);
  }
  CHECK(g_live == 0);
  std::printf("ok\n");
}
