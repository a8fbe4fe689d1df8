// Shares of work on host threads (csrc/host_threads.h) when the n-th allocation,
// or the n-th thread, is refused: every item is done once, and nothing ends the
// process.
#include <dlfcn.h>
#include <errno.h>
#include <pthread.h>

#include <atomic>
#include <climits>
#include <cstdio>
#include <cstdlib>

#include "host_threads.h"

static std::atomic<int> allocs_left{INT_MAX}, threads_left{INT_MAX};

void* operator new(size_t n) {
  if (allocs_left.fetch_sub(1) <= 0) throw std::bad_alloc();
  void* p = std::malloc(n);
  if (!p) throw std::bad_alloc();
  return p;
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, size_t) noexcept { std::free(p); }

extern "C" int pthread_create(pthread_t* t, const pthread_attr_t* a, void* (*f)(void*), void* arg) {
  if (threads_left.fetch_sub(1) <= 0) return EAGAIN;
  using Fn = int (*)(pthread_t*, const pthread_attr_t*, void* (*)(void*), void*);
  static Fn next = (Fn)dlsym(RTLD_NEXT, "pthread_create");
  return next(t, a, f, arg);
}

int main() {
  constexpr int ITEMS = 500;
  static std::atomic<int> done[ITEMS];
  int bad = 0, cases = 0;
  for (int count : {1, 2, 8})
    for (int kind = 0; kind < 2; kind++)
      for (int limit = 0; limit < 24; limit++) {
        for (auto& d : done) d = 0;
        std::atomic<int> next{0}, callers{0};
        allocs_left = kind == 0 ? limit : INT_MAX;
        threads_left = kind == 1 ? limit : INT_MAX;
        knnsj::run_on_threads(count, [&](int) {
          callers++;
          for (int i; (i = next.fetch_add(1)) < ITEMS;) done[i]++;
        });
        allocs_left = threads_left = INT_MAX;
        for (auto& d : done) bad += d != 1;
        bad += callers < 1 || callers > count;
        if (kind == 1) bad += callers != (limit + 1 < count ? limit + 1 : count);
        cases++;
      }
  std::printf("cases=%d bad=%d\n", cases, bad);
  return bad != 0;
}
