// PoolBlock (csrc/serve_block.h) over a pool that runs out: what a block says
// it holds is memory that it has, whatever growth failed before.
#include "serve_block.h"

#include <cstdio>
#include <map>

namespace {

struct FakePool {
    size_t left;
    std::map<void*, size_t> live;
    char memory[1 << 16];
    size_t next = 0;

    void* alloc(size_t bytes)
    {
        if (bytes > left) return nullptr;
        left -= bytes;
        void* p = memory + next++;
        live[p] = bytes;
        return p;
    }
    void free(void* p)
    {
        left += live.at(p);  // throws for a pointer freed twice
        live.erase(p);
    }
};

int failures = 0;

void expect(bool ok, const char* what)
{
    if (ok) return;
    std::printf("failed: %s\n", what);
    ++failures;
}

// The block's memory is live in the pool and as large as it says.
void expect_sound(const ocean_b200::PoolBlock<FakePool>& b, const FakePool& pool, const char* what)
{
    const auto it = pool.live.find(b.get());
    expect(b.get() == nullptr ? b.bytes() == 0 && pool.live.empty()
                              : it != pool.live.end() && it->second == b.bytes() && pool.live.size() == 1,
           what);
}

}  // namespace

int main()
{
    FakePool pool{100, {}, {}};
    ocean_b200::PoolBlock<FakePool> b;
    expect_sound(b, pool, "empty at first");
    expect(b.reserve(pool, 0, 0) && b.get() == nullptr, "nothing asked for");
    expect(b.reserve(pool, 40, 60) && b.bytes() == 60, "grows to more than asked");
    expect_sound(b, pool, "after a growth");
    void* const p = b.get();
    expect(b.reserve(pool, 50, 100) && b.get() == p, "what it holds already");
    expect(b.reserve(pool, 80, 120) && b.bytes() == 80, "grows to what there is");
    expect_sound(b, pool, "after a smaller growth");
    expect(!b.reserve(pool, 101, 200), "more than there is");
    expect_sound(b, pool, "after a growth that failed");
    expect(b.bytes() == 0 && b.get() == nullptr, "empty after a growth that failed");
    expect(b.reserve(pool, 70, 140) && b.get() != nullptr && b.bytes() == 70, "a size it once held is fetched again");
    expect_sound(b, pool, "after the failure");
    b.release(pool);
    b.release(pool);
    expect(pool.left == 100, "all given back");
    expect_sound(b, pool, "released");
    std::printf("%s\n", failures == 0 ? "ok" : "FAILED");
    return failures == 0 ? 0 : 1;
}
