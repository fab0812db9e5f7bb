// srs_parallel.h — loops of the set-up and of reset over several host threads.
#pragma once
#include <algorithm>
#include <atomic>
#include <exception>
#include <mutex>
#include <thread>
#include <vector>

namespace srs {

// Threads for a loop that one thread takes `us` microseconds for: a thread more costs
// its maker about 25 us, the fifth to the eighth about 60 each (the bank order of a
// mesh, 216 ns an element: 1,260 us by one, 720 by two, 430 by four, 480 by eight;
// 2,200 us: 700 by four, 590 by eight; 5,600 channels' residuals: 110, 98, 135, 340).
inline int host_threads(double us) { return us < 200 ? 1 : us < 2000 ? 4 : 8; }

// f(0) .. f(n - 1), taken in turn by at most `most` host threads (the caller
// among them).  Threads that cannot be created are done without; an exception of
// f ends the loop and is thrown again in the caller.
template <class F>
void host_parallel(int n, int most, F&& f) {
  const int nt = std::max(1, std::min({n, most, (int)std::thread::hardware_concurrency()}));
  std::atomic<int> next{0};
  std::exception_ptr error;
  std::mutex mtx;
  auto work = [&]() noexcept {
    try {
      for (int i; (i = next.fetch_add(1)) < n;) f(i);
    } catch (...) {
      next.store(n);
      std::lock_guard<std::mutex> lock(mtx);
      if (!error) error = std::current_exception();
    }
  };
  std::vector<std::thread> pool;
  try {
    pool.reserve(nt - 1);
    while ((int)pool.size() < nt - 1) pool.emplace_back(work);
  } catch (...) {  // the threads that there are do the rest
  }
  work();
  for (auto& th : pool) th.join();
  if (error) std::rethrow_exception(error);
}

}  // namespace srs
