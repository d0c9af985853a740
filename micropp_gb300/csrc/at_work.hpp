// at_work.hpp -- how many handles and standalone solves of the process are at work, for the one-launch solves' choice of
// form and share of the SMs.
#pragma once

#include <atomic>

namespace mgb {

// Held for the length of a call that solves.  The count decides how many blocks a solve takes, never its result.
class AtWork {
 public:
  AtWork() { count_.fetch_add(1, std::memory_order_relaxed); }
  ~AtWork() { count_.fetch_sub(1, std::memory_order_relaxed); }
  AtWork(const AtWork &) = delete;
  AtWork &operator=(const AtWork &) = delete;
  static int count() { return count_.load(std::memory_order_relaxed); }
  // Parts into which the handles share the SMs.  Fewer than handles, since a handle also has phases without a solve.  Two
  // solves with half of the SMs each are not much slower than one with all of them: barriers and chains of dependent
  // products bound an iteration of a small grid.
  static int parts() {
    const int n = count();
    return n < 2 ? 1 : n < 8 ? 2 : 4;
  }

 private:
  static inline std::atomic<int> count_{0};
};

}  // namespace mgb
