// watch_batch (csrc/serve_poll.h): the end of a batch is seen however often new
// work arrives, and new work ends the watch.
#include "serve_poll.h"

#include <cstdio>

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

}  // namespace

int main()
{
    BusyLock busy;
    int asked = 0;
    for (int turn = 1; turn <= 3; ++turn) {
        const bool over = ocean_b200::watch_batch(busy, poked, [&] {
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
    expect(ocean_b200::watch_batch(quiet, poked, [&] { return ++asked == 5; }) && asked == 5, "watches to the end");
    asked = 0;
    expect(!ocean_b200::watch_batch(quiet, poked,
                                    [&] {
                                        if (++asked == 4) poked = true;
                                        return false;
                                    }) &&
               asked == 4,
           "new work ends the watch");
    std::printf("%s\n", failures == 0 ? "ok" : "FAILED");
    return failures == 0 ? 0 : 1;
}
