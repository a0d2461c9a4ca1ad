// bf_once.h -- a value asked for once a process.
#pragma once

#include <atomic>
#include <mutex>

namespace bf {

// What `query` gives the first time it succeeds.  A query that fails (a status other
// than zero, the caller's to report) is asked again the next time: kept as an answer, a
// passing failure would choose another kernel for the life of the process.
template <class T>
class AskedOnce {
 public:
  template <class Query>  // Status query(T *)
  auto get(T *out, Query query) -> decltype(query(out)) {
    using Status = decltype(query(out));
    if (!known_.load(std::memory_order_acquire)) {
      std::lock_guard<std::mutex> lk(mu_);
      if (!known_.load(std::memory_order_relaxed)) {
        T v{};
        const Status st = query(&v);
        if (st != Status{}) return st;
        value_ = v;
        known_.store(true, std::memory_order_release);
      }
    }
    *out = value_;
    return Status{};
  }

 private:
  std::atomic<bool> known_{false};
  std::mutex mu_;
  T value_{};
};

}  // namespace bf
