// oceanlib-b200: how the serving loop's dispatcher watches the batch in flight.
// Host logic only.
#pragma once

#include <atomic>
#include <thread>

namespace ocean_b200 {

// With `lk` held: watches, without it, for `over()` to become true or for
// `poked` to be set by whoever brings new work, and returns whether it was
// over. It asks at least once each time, so that new work that keeps coming
// does not hold back the end of the batch. (What came before is looked at
// already: the flag is cleared under the lock.)
template <class Lock, class Over>
bool watch_batch(Lock& lk, std::atomic<bool>& poked, Over&& over)
{
    poked.store(false, std::memory_order_relaxed);
    lk.unlock();
    bool done = over();
    while (!done && !poked.load(std::memory_order_acquire)) {
        std::this_thread::yield();
        done = over();
    }
    lk.lock();
    return done;
}

}  // namespace ocean_b200
