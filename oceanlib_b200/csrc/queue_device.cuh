// oceanlib-b200: what the persistent launches' work queues share - counter
// adds and bounded waits between CTAs, and the clearing of the next launch's
// words.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace ocean_b200 {

__device__ __forceinline__ uint32_t smem_addr(const void* p)
{
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// Release add at GPU scope: every write that happens before it (the CTA's,
// through the preceding barrier) is visible to an acquirer that sees the sum.
__device__ __forceinline__ void red_release_add(unsigned* p, unsigned v)
{
    asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

__device__ __forceinline__ unsigned ld_acquire(const unsigned* p)
{
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ unsigned long long global_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Spin until *counter >= target or the error word is set or limit_ns passes.
// Returns false on timeout / abort.
__device__ inline bool wait_at_least(const unsigned* counter, unsigned target, unsigned* error,
                              unsigned long long limit_ns)
{
    if (ld_acquire(counter) >= target) return true;
    const unsigned long long t0 = global_ns();
    while (true) {
        __nanosleep(64);
        if (ld_acquire(counter) >= target) return true;
        if (ld_acquire(error) != 0u) return false;
        if (global_ns() - t0 > limit_ns) {
            atomicCAS(error, 0u, 1u);
            return false;
        }
    }
}

// Zeroes the next launch's queue words, each CTA its share (QueueArgs).
__device__ __forceinline__ void clear_words(unsigned* words, uint32_t count, int tid, int nt)
{
    for (uint32_t i = blockIdx.x * nt + tid; i < count; i += gridDim.x * nt) words[i] = 0u;
}

}  // namespace ocean_b200
