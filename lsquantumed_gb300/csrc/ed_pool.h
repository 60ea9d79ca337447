// Scratch that contexts keep from call to call, and how it is given back: to the
// context's own trim, to any allocation of the library that finds the device
// full, and when the context ends.  Mem is the allocator (static int get(void**,
// size_t), static bool full(int status), static void put(void*); get returns 0 on
// success).  One lock serves all slots: calls hold it for the bookkeeping and for
// an allocation of the slot, not while they use it.
#pragma once
#include <algorithm>
#include <cstddef>
#include <mutex>
#include <vector>

// One per context.  idle: nobody uses ptr.
struct ed_scratch_slot {
  void* ptr = nullptr;
  size_t cap = 0;
  bool busy = false;
  int device = 0;
};

template <typename Mem>
class ed_scratch_pool {
 public:
  void add(ed_scratch_slot* s) {
    std::lock_guard<std::mutex> lk(mu_);
    slots_.push_back(s);
  }
  void remove(ed_scratch_slot* s) {
    std::lock_guard<std::mutex> lk(mu_);
    slots_.erase(std::remove(slots_.begin(), slots_.end(), s), slots_.end());
    drop(s);
  }
  // Gives back one slot's memory if it is idle.
  void trim(ed_scratch_slot* s) {
    std::lock_guard<std::mutex> lk(mu_);
    if (!s->busy) drop(s);
  }
  // An allocation of the library: where it does not fit, all idle slots of the
  // device are given back and it is tried once more.
  int alloc(void** p, size_t bytes, int device) {
    const int rc = Mem::get(p, bytes);
    if (rc == 0 || !Mem::full(rc)) return rc;
    std::lock_guard<std::mutex> lk(mu_);
    return again(p, bytes, device, rc);
  }
  // Memory for one call: the slot's where it is idle and bytes <= keep (grown if
  // need be), else the call's own.  null where it does not fit.
  void* take(ed_scratch_slot* s, size_t bytes, size_t keep, bool* own) {
    std::lock_guard<std::mutex> lk(mu_);
    *own = s->busy || bytes > keep;
    void* p = nullptr;
    if (*own || bytes > s->cap) {
      if (!*own) drop(s);
      int rc = Mem::get(&p, bytes);
      if (rc != 0 && Mem::full(rc)) rc = again(&p, bytes, s->device, rc);
      if (rc != 0) return nullptr;
      if (*own) return p;
      s->ptr = p;
      s->cap = bytes;
    }
    s->busy = true;
    return s->ptr;
  }
  void give(ed_scratch_slot* s, void* p, bool own) {
    if (!p) return;
    if (own) {
      Mem::put(p);
      return;
    }
    std::lock_guard<std::mutex> lk(mu_);
    s->busy = false;
  }

 private:
  static void drop(ed_scratch_slot* s) {
    if (s->ptr) Mem::put(s->ptr);
    s->ptr = nullptr;
    s->cap = 0;
  }
  int again(void** p, size_t bytes, int device, int rc) {
    bool any = false;
    for (ed_scratch_slot* s : slots_)
      if (s->device == device && !s->busy && s->ptr) {
        drop(s);
        any = true;
      }
    return any ? Mem::get(p, bytes) : rc;
  }
  std::mutex mu_;
  std::vector<ed_scratch_slot*> slots_;
};
