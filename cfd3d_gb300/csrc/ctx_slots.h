// ctx_slots.h -- one value per CUDA context, each with a lock of its own.
//
// The map's lock is held for a lookup alone; who uses a slot's value holds that slot's lock, so
// users of different contexts (other devices, other threads' contexts) do not wait for one
// another.  Slots are never moved or removed: context ids are not reused within a process.
#pragma once
#include <list>
#include <mutex>

namespace cfd {

template <class T>
class CtxSlots {
 public:
  struct Slot {
    unsigned long long ctx;
    T value;
    std::mutex mu;
  };
  // the slot of context ctx, or null
  Slot* find(unsigned long long ctx) {
    std::lock_guard<std::mutex> lock(mu_);
    return at(ctx);
  }
  // the slot of context ctx, made with `value` if it is new (another thread may have made it)
  Slot* put(unsigned long long ctx, T value) {
    std::lock_guard<std::mutex> lock(mu_);
    if (Slot* s = at(ctx)) return s;
    slots_.emplace_back();
    slots_.back().ctx = ctx;
    slots_.back().value = value;
    return &slots_.back();
  }

 private:
  Slot* at(unsigned long long ctx) {
    for (Slot& s : slots_)
      if (s.ctx == ctx) return &s;
    return nullptr;
  }
  std::mutex mu_;
  std::list<Slot> slots_;
};

}  // namespace cfd
