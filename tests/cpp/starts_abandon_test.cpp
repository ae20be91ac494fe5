// Words of a call whose wait failed (host_starts.h): its kernel may still write
// them, so neither the same thread's next call nor another thread's gets them
// again, and they count towards the bound.  Prints "ok".
#include <cstdio>
#include <thread>
#include <vector>

#include "host_starts.h"

static uint32_t* alloc(size_t words) { return new uint32_t[words]; }

#define CHECK(c) ((c) ? 0 : (std::printf("line %d: %s\n", __LINE__, #c), 1))

int main() {
  int bad = 0;
  gms::StartsPool& pool = *new gms::StartsPool(alloc);
  uint32_t* lost = nullptr;
  std::thread([&] {
    gms::ThreadStarts mine(pool);
    lost = mine.get(7);
    mine.abandon();
    uint32_t* next = mine.get(7);
    bad += CHECK(lost != nullptr && next != nullptr && next != lost);
    bad += CHECK(mine.get(7) == next);
    mine.abandon();  // ends with none in hand
  }).join();
  size_t taken = 2;
  for (uint32_t* p = pool.take(7); p != nullptr; p = pool.take(7), ++taken) bad += CHECK(p != lost);
  bad += CHECK(taken == gms::kStartsMaxSlots);
  std::printf(bad ? "bad\n" : "ok\n");
  return bad;
}
