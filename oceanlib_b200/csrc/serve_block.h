// oceanlib-b200: a device block of the serving loop that grows with what its
// batches need (a batch's staging, a size's larger ring). Host logic only: the
// pool it allocates from is a parameter.
#pragma once

#include <cstddef>

namespace ocean_b200 {

// Pool: void* alloc(size_t bytes), null when it cannot; void free(void*).
// After a growth that failed the block is empty and says so, so that whoever
// asks next does not take its former size for memory it still has.
template <class Pool>
class PoolBlock {
public:
    void* get() const { return p_; }
    size_t bytes() const { return bytes_; }

    // Whether the block holds `want` bytes now. It grows to `grown` if the pool
    // has that much, else to `want`; a growth does not keep the contents.
    bool reserve(Pool& pool, size_t want, size_t grown)
    {
        if (want <= bytes_) return true;
        release(pool);
        if (grown > want) {
            p_ = pool.alloc(grown);
            if (p_ != nullptr) bytes_ = grown;
        }
        if (p_ == nullptr) {
            p_ = pool.alloc(want);
            if (p_ != nullptr) bytes_ = want;
        }
        return p_ != nullptr;
    }
    void release(Pool& pool)
    {
        void* const p = p_;
        p_ = nullptr;
        bytes_ = 0;
        if (p != nullptr) pool.free(p);
    }

private:
    void* p_ = nullptr;
    size_t bytes_ = 0;
};

}  // namespace ocean_b200
