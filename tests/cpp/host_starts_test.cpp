// The pool of words in which bucket starts reach the host (host_starts.h), on
// the host with a counting allocator: short-lived threads allocate once, threads
// alive together have slots of their own, the bound holds, slots stay with their
// context, and a refused allocation leaves nothing behind.  Prints "ok".
#include <algorithm>
#include <condition_variable>
#include <cstdio>
#include <mutex>
#include <set>
#include <thread>
#include <vector>

#include "host_starts.h"

static int g_allocs = 0;
static bool g_refuse = false;

static uint32_t* alloc(size_t words) {  // called under the pool's lock
  if (g_refuse) return nullptr;
  ++g_allocs;
  return new uint32_t[words];
}

#define CHECK(c) ((c) ? 0 : (std::printf("line %d: %s\n", __LINE__, #c), 1))

// The slots that `count` threads alive together get.
static std::vector<uint32_t*> together(gms::StartsPool& pool, int count, uint64_t context) {
  std::mutex m;
  std::condition_variable all;
  std::vector<uint32_t*> got;
  std::vector<std::thread> threads;
  for (int i = 0; i < count; ++i)
    threads.emplace_back([&] {
      gms::ThreadStarts mine(pool);
      uint32_t* p = mine.get(context);
      if (p != nullptr) std::fill(p, p + gms::kStartsWords, 1u);
      std::unique_lock<std::mutex> lock(m);
      got.push_back(p);
      all.notify_all();
      all.wait(lock, [&] { return int(got.size()) == count; });
    });
  for (auto& t : threads) t.join();
  return got;
}

int main() {
  int bad = 0;
  {  // one thread after another
    gms::StartsPool& pool = *new gms::StartsPool(alloc);
    for (int i = 0; i < 500; ++i) {
      std::thread([&] {
        gms::ThreadStarts mine(pool);
        uint32_t* p = mine.get(7);
        bad += CHECK(p != nullptr);
        bad += CHECK(mine.get(7) == p);
      }).join();
    }
    bad += CHECK(g_allocs == 1);
    // threads together: distinct slots, a slab for every 64
    const auto got = together(pool, 100, 7);
    bad += CHECK(std::set<uint32_t*>(got.begin(), got.end()).size() == 100);
    bad += CHECK(g_allocs == 2);
    // another context has slots of its own, and coming back allocates nothing
    gms::ThreadStarts mine(pool);
    uint32_t* a = mine.get(7);
    uint32_t* b = mine.get(8);
    bad += CHECK(b != nullptr && std::find(got.begin(), got.end(), b) == got.end() && b != a);
    bad += CHECK(g_allocs == 3);
    bad += CHECK(mine.get(7) == a);
    bad += CHECK(mine.get(0) == nullptr);
    bad += CHECK(g_allocs == 3);
  }
  {  // the bound, and slots handed on once they are free again
    g_allocs = 0;
    gms::StartsPool& pool = *new gms::StartsPool(alloc);
    std::vector<uint32_t*> held;
    for (size_t i = 0; i < gms::kStartsMaxSlots; ++i) held.push_back(pool.take(1));
    bad += CHECK(std::set<uint32_t*>(held.begin(), held.end()).size() == gms::kStartsMaxSlots);
    bad += CHECK(std::find(held.begin(), held.end(), nullptr) == held.end());
    bad += CHECK(pool.take(1) == nullptr);
    pool.give(1, held.back());
    bad += CHECK(pool.take(1) == held.back());
    bad += CHECK(g_allocs == int(gms::kStartsMaxSlots / gms::kStartsSlabSlots));
  }
  {  // no memory now, memory later
    gms::StartsPool& pool = *new gms::StartsPool(alloc);
    gms::ThreadStarts mine(pool);
    g_refuse = true;
    bad += CHECK(mine.get(1) == nullptr);
    g_refuse = false;
    bad += CHECK(mine.get(1) != nullptr);
  }
  if (bad == 0) std::printf("ok\n");
  return bad != 0;
}
