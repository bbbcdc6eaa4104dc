// Growth policy of a context's device scratch: one allocation that grows on demand.  The memory calls
// go through ArenaMem, so that the policy runs on the host against an allocator that refuses
// (tests/test_arena_cpu.py).
#pragma once
#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <vector>

namespace dpkem {

struct ArenaMem {
  virtual void *alloc(size_t bytes) = 0;  // nullptr: refused
  virtual void release(void *p) = 0;
  virtual void drain() = 0;  // waits for every launch that uses the arena
 protected:
  ~ArenaMem() = default;
};

class Arena {
 public:
  uint8_t *base = nullptr;
  size_t bytes = 0;

  // The arena holds at least n bytes, or false.  Growth is geometric (at least 1.5x, within the budget), or to
  // n exactly where the device has no more.  The old memory goes first: a call that needs n cannot run in it.
  bool need(size_t n, size_t budget, ArenaMem &m) {
    if (n <= bytes) return true;
    if (n > budget) return false;
    const size_t size = grown(n, budget);
    drop(m);
    return set(size, m) || (size > n && set(n, m));
  }

  // The same for memory that only makes a call faster: false leaves the arena as it is, or at least as large.
  // A size that was refused is not asked for again, and a fixed arena does not grow.  The old memory is kept
  // until the new one is there, where the budget has room for both.
  bool want(size_t n, size_t budget, ArenaMem &m) {
    if (n <= bytes) return true;
    budget -= std::min(budget, kept_bytes_);
    if (fixed_ || n > budget || n >= refused_) return false;
    const size_t size = grown(n, budget), before = bytes;
    if (before + n > budget) {  // one at a time
      if (captured_) return false;
      drop(m);
      if (set(size, m) || (size > n && set(n, m))) return true;
      refused_ = n;
      set(before, m);
      return false;
    }
    Arena next;
    if (!(before + size <= budget && next.set(size, m)) && !next.set(n, m)) {
      refused_ = n;
      return false;
    }
    drop(m);
    base = next.base;
    bytes = next.bytes;
    return true;
  }

  // A stream capture has recorded addresses of this memory: it stays allocated when the arena grows.
  void captured() { captured_ = true; }
  // The caller has sized the arena: want() takes what there is.
  void fix() {
    fixed_ = true;
    refused_ = SIZE_MAX;
  }
  void free_all(ArenaMem &m) {
    if (base) m.release(base);
    for (void *p : kept_) m.release(p);
    *this = Arena();
  }

 private:
  size_t grown(size_t n, size_t budget) const { return std::min(budget, std::max(n, bytes + bytes / 2)); }
  bool set(size_t n, ArenaMem &m) {
    base = static_cast<uint8_t *>(n ? m.alloc(n) : nullptr);
    bytes = base ? n : 0;
    return base != nullptr;
  }
  void drop(ArenaMem &m) {
    if (!base) return;
    if (captured_) {
      kept_.push_back(base);
      kept_bytes_ += bytes;
    } else {
      m.drain();
      m.release(base);
    }
    captured_ = false;
    base = nullptr;
    bytes = 0;
  }

  size_t refused_ = SIZE_MAX;  // smallest optional size that the device refused
  bool fixed_ = false, captured_ = false;
  std::vector<void *> kept_;
  size_t kept_bytes_ = 0;
};

}  // namespace dpkem
