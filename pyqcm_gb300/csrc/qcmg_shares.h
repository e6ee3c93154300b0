// Independent shares of a call's host work on threads of their own.
#pragma once

#include <exception>
#include <system_error>
#include <thread>
#include <utility>
#include <vector>

namespace qcmg {

struct SpawnThread {
  template <class F>
  std::thread operator()(F&& f) const {
    return std::thread(std::forward<F>(f));
  }
};

// f(0) .. f(n - 1), each on its own thread; what is left when the system gives
// no more threads is done by the caller, one after the other (the shares do
// not wait on one another).  Returns when all are done; the first exception
// of a share is thrown then.
template <class F, class Spawn = SpawnThread>
void run_shares(int n, F&& f, Spawn&& spawn = Spawn()) {
  std::vector<std::exception_ptr> err(n);
  std::vector<std::thread> threads;
  threads.reserve(n);
  auto share = [&](int t) {
    try {
      f(t);
    } catch (...) {
      err[t] = std::current_exception();
    }
  };
  int t = 0;
  try {
    for (; t < n; ++t) threads.push_back(spawn([&share, t] { share(t); }));
  } catch (const std::system_error&) {
  }
  for (; t < n; ++t) share(t);
  for (auto& th : threads) th.join();
  for (auto& e : err)
    if (e) std::rethrow_exception(e);
}

}  // namespace qcmg
