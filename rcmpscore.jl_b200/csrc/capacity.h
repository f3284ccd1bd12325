// A device's capacity for a kernel, asked for once (internal).
#pragma once
#include <atomic>

namespace rcmps {

// ask(): the capacity, or -1 when the query failed, which counts as 0 for this call and is asked again
// by the next. known: 0, or the capacity plus one.
template <class F>
int capacity_once(std::atomic<int>& known, F ask) {
  int n = known.load();
  if (n) return n - 1;
  n = ask();
  if (n < 0) return 0;
  known.store(n + 1);
  return n;
}

}  // namespace rcmps
