// Work spread over host threads of one call, from which nothing but a status
// comes out: an exception that left a thread would end the process, and one
// that left a C entry point would as well.
#pragma once
#include <exception>
#include <new>
#include <thread>
#include <vector>

namespace gla {

constexpr int kStatusNoMemory = -1000 - 2;   // cudaErrorMemoryAllocation's status
constexpr int kStatusUnknown = -1000 - 999;  // cudaErrorUnknown's

// f's status; that of an allocation that failed, or an unknown error, when it throws.
template <class F>
int guarded(const F& f) noexcept {
  try {
    return f();
  } catch (const std::bad_alloc&) {
    return kStatusNoMemory;
  } catch (...) {
    return kStatusUnknown;
  }
}

// work(t) for t < n, each on a thread of its own, work(0) on this one, and all
// of them waited for. A thread that cannot be started is left out, with its
// share of the work to the others: at least work(0) runs. work must not throw.
template <class W>
void on_threads(int n, const W& work) {
  std::vector<std::thread> threads;
  for (int t = 1; t < n; t++) {
    try {
      threads.emplace_back([&work, t] { work(t); });
    } catch (...) {
      break;
    }
  }
  work(0);
  for (std::thread& t : threads) t.join();
}

}  // namespace gla
