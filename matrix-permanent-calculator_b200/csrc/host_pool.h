// host_pool.h -- independent host tasks shared out over a few threads.
#pragma once
#include <atomic>
#include <cstddef>
#include <exception>
#include <mutex>
#include <thread>
#include <vector>

namespace perm {

// Calls fn(0) .. fn(count - 1) on this thread and up to `extra` more (fewer
// where the system gives no more).  When a call throws, those not yet begun are
// left out, and the first exception is thrown here once every thread has ended:
// none leaves a thread, which would end the process.
template <class Fn>
void for_each_shared(size_t count, size_t extra, Fn fn) {
  std::atomic<size_t> next{0};
  std::exception_ptr error;
  std::mutex mu;
  auto work = [&] {
    try {
      for (size_t i; (i = next.fetch_add(1)) < count;) fn(i);
    } catch (...) {
      next.store(count);
      std::lock_guard<std::mutex> lock(mu);
      if (!error) error = std::current_exception();
    }
  };
  std::vector<std::thread> threads;
  try {
    threads.reserve(extra);
    while (threads.size() < extra) threads.emplace_back(work);
  } catch (const std::exception&) {  // no more threads: the ones there do the work
  }
  work();
  for (std::thread& t : threads) t.join();
  if (error) std::rethrow_exception(error);
}

}  // namespace perm
