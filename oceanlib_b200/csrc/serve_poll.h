// oceanlib-b200: how the serving loop's dispatcher watches the batch in flight.
// Host logic only.
#pragma once

#include <algorithm>
#include <atomic>
#include <chrono>
#include <thread>

namespace ocean_b200 {

// A batch's first millisecond is watched without a pause: most batches are over
// by then (0.2 ms for 32 sessions), and a thread that slept would find out late.
// A longer one is asked about every 1/32 of the time it has taken, a millisecond
// at most, and leaves the core and the driver's lock to others meanwhile.
constexpr std::chrono::microseconds kWatchClosely{1000};

inline std::chrono::microseconds watch_pause(std::chrono::microseconds taken)
{
    if (taken < kWatchClosely) return std::chrono::microseconds(0);
    return std::min(taken / 32, std::chrono::microseconds(1000));
}

// With `lk` held: watches, without it, for `over()` to become true or for
// `poked` to be set (and `cv` notified) by whoever brings new work, and returns
// whether it was over. It asks at least once each time, so that new work that
// keeps coming does not hold back the end of the batch. (What came before is
// looked at already: the flag is cleared under the lock.) The batch has been
// the one to watch since `since`.
template <class Lock, class Cv, class Over>
bool watch_batch(Lock& lk, Cv& cv, std::atomic<bool>& poked, std::chrono::steady_clock::time_point since, Over&& over)
{
    const auto new_work = [&] { return poked.load(std::memory_order_acquire); };
    poked.store(false, std::memory_order_relaxed);
    lk.unlock();
    bool done = over();
    while (!done && !new_work()) {
        const auto pause = watch_pause(
            std::chrono::duration_cast<std::chrono::microseconds>(std::chrono::steady_clock::now() - since));
        if (pause.count() == 0) {
            std::this_thread::yield();
        } else {
            lk.lock();
            cv.wait_for(lk, pause, new_work);
            lk.unlock();
        }
        done = over();
    }
    lk.lock();
    return done;
}

}  // namespace ocean_b200
