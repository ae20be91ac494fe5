// Pinned host words in which a call's last kernel leaves the bucket starts for
// the host (capi.cu).  A call that returns starts waits for its stream before
// it returns, so a thread's words serve one call at a time; where the wait fails
// (another thread captures a stream in the global mode) its kernel may still run,
// and the words are given up.
//
// Words belong to the CUDA context in which they were allocated and vanish with
// it (cudaDeviceReset), so slots are kept per context.  Threads hand their slot
// back when they end; nothing is freed: with words allocated and freed by each
// thread, a call of 10 k pairs in a thread of its own took 196 us on an idle
// device instead of 182, and the free waits for all work on a busy one.
#pragma once

#include <cstddef>
#include <cstdint>
#include <mutex>
#include <new>
#include <vector>

namespace gms {

constexpr size_t kStartsWords = 256;       // one slot: the starts of 256 buckets
constexpr size_t kStartsSlabSlots = 64;    // slots allocated together (64 KB)
constexpr size_t kStartsMaxSlots = 1024;   // per context: threads beyond it get none

class StartsPool {
 public:
  // Allocates pinned words in the current context, or returns null.
  using Alloc = uint32_t* (*)(size_t words);

  explicit StartsPool(Alloc alloc) : alloc_(alloc) {}

  // A free slot of the context (the current one), or null.
  uint32_t* take(uint64_t context) noexcept {
    try {
      std::lock_guard<std::mutex> lock(mutex_);
      Slots& s = slots_of(context);
      if (s.free.empty()) {
        if (s.total + kStartsSlabSlots > kStartsMaxSlots) return nullptr;
        s.free.reserve(s.total + kStartsSlabSlots);  // give() never allocates
        uint32_t* slab = alloc_(kStartsSlabSlots * kStartsWords);
        if (slab == nullptr) return nullptr;
        s.total += kStartsSlabSlots;
        for (size_t i = kStartsSlabSlots; i-- > 0;) s.free.push_back(slab + i * kStartsWords);
      }
      uint32_t* slot = s.free.back();
      s.free.pop_back();
      return slot;
    } catch (const std::bad_alloc&) {
      return nullptr;
    }
  }

  void give(uint64_t context, uint32_t* slot) noexcept {
    std::lock_guard<std::mutex> lock(mutex_);
    for (Slots& s : contexts_)
      if (s.context == context) s.free.push_back(slot);
  }

 private:
  struct Slots {
    uint64_t context;
    size_t total;
    std::vector<uint32_t*> free;
  };

  Slots& slots_of(uint64_t context) {
    for (Slots& s : contexts_)
      if (s.context == context) return s;
    contexts_.push_back(Slots{context, 0, {}});
    return contexts_.back();
  }

  Alloc alloc_;
  std::mutex mutex_;
  std::vector<Slots> contexts_;
};

// A thread's slot, taken on the first call that asks for starts.
class ThreadStarts {
 public:
  explicit ThreadStarts(StartsPool& pool) : pool_(pool) {}
  ThreadStarts(const ThreadStarts&) = delete;
  ThreadStarts& operator=(const ThreadStarts&) = delete;
  ~ThreadStarts() { release(); }

  // The slot in the context (0: unknown), or null when there is none.
  uint32_t* get(uint64_t context) noexcept {
    if (slot_ != nullptr && context == context_) return slot_;
    release();
    if (context == 0) return nullptr;
    slot_ = pool_.take(context);
    context_ = context;
    return slot_;
  }

  // Drops the slot for good: a kernel that nobody waited for may still write it.
  void abandon() noexcept { slot_ = nullptr; }

 private:
  void release() noexcept {
    if (slot_ != nullptr) pool_.give(context_, slot_);
    slot_ = nullptr;
  }

  StartsPool& pool_;
  uint32_t* slot_ = nullptr;
  uint64_t context_ = 0;
};

}  // namespace gms
