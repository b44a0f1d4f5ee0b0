// fz_wait.h -- pause between two polls of a bounded host wait for device work.
#pragma once
#include <algorithm>
#include <chrono>
#include <thread>

namespace fz {

// Polls back to back for the first 2 ms (a short run's latency is the call's latency), then sleeps for
// 1/64 of the time waited so far, 31 to 500 us: the wait ends within about 2 % of the work's own time
// at any length. (Sleeps doubling from 20 us to 2 ms, the rule before, added up to half of a 2 ms run:
// 64 steps of 26 x 22 x 18 cells, 1.1 ms on the device, took 2.1 ms with their read-back, and then 1.65.)
inline void poll_pause(std::chrono::steady_clock::time_point start) {
  const auto us =
      std::chrono::duration_cast<std::chrono::microseconds>(std::chrono::steady_clock::now() - start).count();
  if (us < 2000)
    std::this_thread::yield();
  else
    std::this_thread::sleep_for(std::chrono::microseconds(std::min<long long>(us / 64, 500)));
}

}  // namespace fz
