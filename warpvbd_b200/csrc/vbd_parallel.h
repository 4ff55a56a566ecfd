// Host threads for the setup.  Plain C++.
#pragma once
#include <algorithm>
#include <atomic>
#include <exception>
#include <mutex>
#include <thread>
#include <vector>

namespace vbd {

// f(0) ... f(n - 1) on up to 16 host threads; an exception of f is rethrown here, once every
// thread is done.  When a thread cannot be started (no more of them, no memory for its
// state), those there are do the work.
template <class Thread = std::thread, class F>
void for_each_parallel(int n, F f) {
  std::atomic<int> next{0};
  std::mutex mu;
  std::exception_ptr error;
  auto work = [&]() {
    for (int k; (k = next.fetch_add(1)) < n;) {
      try {
        f(k);
      } catch (...) {
        std::lock_guard<std::mutex> lock(mu);
        if (!error) error = std::current_exception();
        next = n;
      }
    }
  };
  const int nthreads =
      std::min<int>(n, std::max(1u, std::min(16u, std::thread::hardware_concurrency())));
  std::vector<Thread> pool;
  pool.reserve(std::max(0, nthreads));
  try {
    for (int i = 1; i < nthreads; ++i) pool.emplace_back(work);
  } catch (...) {
  }
  work();
  for (auto& t : pool) t.join();
  if (error) std::rethrow_exception(error);
}

}  // namespace vbd
