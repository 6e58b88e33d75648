// Work in pieces through a ring of buffers, its two halves on two threads (host code only).
#pragma once

#include <atomic>
#include <exception>
#include <system_error>
#include <thread>

namespace autan_b200 {

struct StartThread {
  template <class F>
  std::thread operator()(F&& f) const {
    return std::thread(f);
  }
};

// put(p) then take(p) for every piece p in [0, pieces): put on this thread, take on a second one, in
// order each, at most `ring` pieces between them. Where no thread is to be had both run on this one,
// piece by piece. The first exception of either half ends both and is thrown here.
template <class Put, class Take, class Start = StartThread>
void run_pieces(long long pieces, int ring, Put&& put, Take&& take, Start&& start = Start{}) {
  std::atomic<long long> done_put{0}, done_take{0};
  std::atomic<bool> stop{false};
  std::exception_ptr failed;
  auto taker = [&] {
    try {
      for (long long p = 0; p < pieces; ++p) {
        while (done_put.load(std::memory_order_acquire) <= p) {
          if (stop.load()) return;
          std::this_thread::yield();
        }
        take(p);
        done_take.store(p + 1, std::memory_order_release);
      }
    } catch (...) {
      failed = std::current_exception();
      stop.store(true);
    }
  };
  std::thread second;
  try {
    second = start(taker);
  } catch (const std::system_error&) {
    for (long long p = 0; p < pieces; ++p) {
      put(p);
      take(p);
    }
    return;
  }
  try {
    for (long long p = 0; p < pieces; ++p) {
      while (p - done_take.load(std::memory_order_acquire) >= ring && !stop.load()) std::this_thread::yield();
      if (stop.load()) break;
      put(p);
      done_put.store(p + 1, std::memory_order_release);
    }
  } catch (...) {
    stop.store(true);
    second.join();
    throw;
  }
  second.join();
  if (failed) std::rethrow_exception(failed);
}

}  // namespace autan_b200
