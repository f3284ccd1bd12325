// A device's capacity for a kernel, asked for once, and the admission of launches that must be
// resident as a whole (internal; host code only).
#pragma once
#include <atomic>
#include <condition_variable>
#include <mutex>

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

// Admits launches to a device while everything admitted fits: those of one kind together up to their
// kind's capacity, another kind when the device is empty. First come, first served.
class Admission {
 public:
  void enter(int kind, int count, int capacity) {
    std::unique_lock<std::mutex> lock(m_);
    const unsigned long long ticket = tickets_++;
    changed_.wait(lock, [&] {
      return ticket == turn_ && (count_ == 0 || (kind_ == kind && count_ + count <= capacity));
    });
    ++turn_;
    kind_ = kind;
    count_ += count;
    changed_.notify_all();
  }
  void leave(int count) {
    {
      std::lock_guard<std::mutex> lock(m_);
      count_ -= count;
    }
    changed_.notify_all();
  }

 private:
  std::mutex m_;
  std::condition_variable changed_;
  int kind_ = 0, count_ = 0;
  unsigned long long tickets_ = 0, turn_ = 0;
};

}  // namespace rcmps
