// Host loops of setup over a few threads.
#pragma once

#include <algorithm>
#include <exception>
#include <thread>
#include <vector>

namespace kifmm {

// body(t, nthr) for t = 0 .. nthr - 1, each on a thread of its own (the
// caller's for t = 0); an exception of any of them is rethrown here once all
// have ended, and where no thread can be started the caller runs its part.
template <class Body>
void host_parallel(int nthr, Body&& body) {
  std::vector<std::exception_ptr> err(std::max(nthr, 1));
  auto guarded = [&](int t) {
    try {
      body(t, nthr);
    } catch (...) {
      err[t] = std::current_exception();
    }
  };
  std::vector<std::thread> ths;
  int t = 1;
  try {
    ths.reserve(std::max(nthr, 1));
    for (; t < nthr; t++) ths.emplace_back(guarded, t);
  } catch (...) {
  }
  guarded(0);
  for (; t < nthr; t++) guarded(t);
  for (auto& th : ths) th.join();
  for (auto& e : err)
    if (e) std::rethrow_exception(e);
}

inline int host_parallel_threads(int most) {
  return std::max(1, std::min(std::min(most, 16), (int)std::thread::hardware_concurrency()));
}

}  // namespace kifmm
