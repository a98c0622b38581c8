// rs_units.h -- the parts of one piece of work side by side in threads (host).
#pragma once
#include <exception>
#include <string>
#include <thread>
#include <utility>
#include <vector>

namespace rs {

// work(0) .. work(n - 1), the first in the caller's thread and each other one in its own.  A part
// whose thread cannot be started runs in the caller's; what a part throws becomes its entry of
// *errors (empty: it returned).  All threads have ended on return, whatever happens: a started
// thread left joinable, or an exception that leaves one, would end the process.
template <class Work, class Start>
void run_units(int n, Work work, std::vector<std::string>* errors, Start start) {
  std::vector<int> here;
  here.reserve(n);
  errors->assign(n, std::string());
  auto one = [&](int u) noexcept {
    try {
      work(u);
    } catch (const std::exception& e) {
      try {
        (*errors)[u] = e.what();
      } catch (...) {
      }
      if ((*errors)[u].empty()) (*errors)[u] = "exception";  // short: not allocated
    } catch (...) {
      (*errors)[u] = "exception";
    }
  };
  struct Threads {
    std::vector<std::thread> t;
    ~Threads() {
      for (auto& x : t) x.join();
    }
  } threads;  // declared last: joined before what the threads use goes
  threads.t.reserve(n);
  here.push_back(0);
  for (int u = 1; u < n; ++u) {
    try {
      threads.t.push_back(start([&one, u] { one(u); }));
    } catch (...) {
      here.push_back(u);
    }
  }
  for (int u : here) one(u);
}
template <class Work>
void run_units(int n, Work work, std::vector<std::string>* errors) {
  run_units(n, std::move(work), errors, [](auto f) { return std::thread(std::move(f)); });
}

}  // namespace rs
