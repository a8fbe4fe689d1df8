// host_threads.h -- a few host threads that share one piece of work.
#pragma once

#include <new>
#include <system_error>
#include <thread>
#include <vector>

namespace knnsj {

// Runs work(0) on the calling thread and work(1) ... work(count - 1) on threads
// of their own, and returns when all have ended.  Where threads or memory are
// short fewer of them run, work(0) always: the workers take items from a shared
// counter until none is left.  (The list of threads grows before any is started:
// a growth that failed with threads running would end the process.)
template <typename F>
void run_on_threads(int count, F&& work) {
  struct Pool {
    std::vector<std::thread> t;
    ~Pool() {
      for (std::thread& x : t) x.join();
    }
  } pool;
  try {
    pool.t.reserve(count > 1 ? (size_t)count - 1 : 0);
    for (int i = 1; i < count; i++) pool.t.emplace_back([&work, i] { work(i); });
  } catch (const std::system_error&) {
  } catch (const std::bad_alloc&) {
  }
  work(0);
}

}  // namespace knnsj
