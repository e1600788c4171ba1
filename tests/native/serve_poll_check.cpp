// watch_batch (csrc/serve_poll.h): the end of a batch is seen however often new
// work arrives, new work ends the watch, and a long batch is asked about with
// pauses in between, which new work ends too.
#include "serve_poll.h"

#include <condition_variable>
#include <cstdio>
#include <mutex>

namespace {

std::atomic<bool> poked{false};

// New work that arrives as soon as the lock is free, every time.
struct BusyLock {
    bool held = true;
    void unlock()
    {
        held = false;
        poked = true;
    }
    void lock() { held = true; }
};

struct QuietLock : BusyLock {
    void unlock() { held = false; }
};

int failures = 0;

void expect(bool ok, const char* what)
{
    if (ok) return;
    std::printf("failed: %s\n", what);
    ++failures;
}

using Clock = std::chrono::steady_clock;

// For the short watches, which never wait.
struct NoCv {
    template <class... A>
    bool wait_for(A&&...)
    {
        expect(false, "a pause in a batch's first millisecond");
        return true;
    }
} no_cv;

}  // namespace

int main()
{
    const auto now = [] { return Clock::now(); };
    const auto young = now() + std::chrono::hours(1);  // a batch whose first millisecond this program never leaves
    BusyLock busy;
    int asked = 0;
    for (int turn = 1; turn <= 3; ++turn) {
        const bool over = ocean_b200::watch_batch(busy, no_cv, poked, young, [&] {
            expect(!busy.held, "asked without the lock");
            return ++asked == 3;
        });
        expect(asked == turn, "asked once a turn");
        expect(over == (turn == 3), "over at the third turn");
        expect(busy.held, "the lock is held again");
    }

    QuietLock quiet;
    poked = true;  // of work that has been looked at
    asked = 0;
    expect(ocean_b200::watch_batch(quiet, no_cv, poked, young, [&] { return ++asked == 5; }) && asked == 5, "watches to the end");
    asked = 0;
    expect(!ocean_b200::watch_batch(quiet, no_cv, poked, young,
                                    [&] {
                                        if (++asked == 4) poked = true;
                                        return false;
                                    }) &&
               asked == 4,
           "new work ends the watch");

    // A batch of 40 ms: after its first millisecond it is asked about at most
    // every 1/32 of its age, 32 ln 40 times, and a few for the rounding.
    std::mutex mu;
    std::condition_variable cv;
    std::unique_lock<std::mutex> lk(mu);
    const auto t0 = now();
    int late = 0;
    expect(ocean_b200::watch_batch(lk, cv, poked, t0,
                                   [&] {
                                       const auto age = now() - t0;
                                       late += age > std::chrono::milliseconds(1);
                                       return age > std::chrono::milliseconds(40);
                                   }),
           "a long batch is over");
    expect(lk.owns_lock(), "the lock is held after a pause");
    expect(late >= 1 && late <= 140, "pauses in a long batch");

    // New work ends a watch that pauses (a batch that never ends by itself).
    std::thread worker([&] {
        std::this_thread::sleep_for(std::chrono::milliseconds(200));
        poked = true;
        cv.notify_all();
    });
    expect(!ocean_b200::watch_batch(lk, cv, poked, t0, [&] { return now() - t0 > std::chrono::seconds(20); }),
           "new work ends a pausing watch");
    worker.join();
    using std::chrono::microseconds;
    expect(ocean_b200::watch_pause(microseconds(999)).count() == 0 &&
               ocean_b200::watch_pause(microseconds(1000)).count() == 31 &&
               ocean_b200::watch_pause(microseconds(1000000)).count() == 1000,
           "pauses by age");
    std::printf("%s\n", failures == 0 ? "ok" : "FAILED");
    return failures == 0 ? 0 : 1;
}
