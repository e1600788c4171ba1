// oceanlib-b200: host-side error types and RAII device/pinned buffers.
#pragma once

#include "../../include/ocean_b200.h"

#include <cuda_runtime.h>

#include <cstring>
#include <stdexcept>
#include <utility>

namespace ocean_b200 {

// A CUDA call failed.
struct DeviceError : std::runtime_error {
    cudaError_t code;
    DeviceError(cudaError_t c, const char* what) : std::runtime_error(what), code(c) {}
};

// A bounded device wait gave up (a persistent kernel's error word was set).
struct TimeoutError : std::runtime_error {
    TimeoutError() : std::runtime_error("device wait timed out") {}
};

inline void check(cudaError_t e, const char* what)
{
    if (e != cudaSuccess) {
        // Reset the runtime's last-error slot, so a later launch's
        // cudaGetLastError reports that launch and not this failure (sticky
        // errors that poison the context stay set regardless).
        cudaGetLastError();
        throw DeviceError(e, what);
    }
}

inline ocean_status status_of(const DeviceError& e)
{
    return e.code == cudaErrorMemoryAllocation ? OCEAN_ERROR_OUT_OF_MEMORY : OCEAN_ERROR_DEVICE;
}

// Maps the exceptions of a host call to ocean_status (no exception may cross
// the C boundary).
template <typename Fn>
ocean_status guarded(Fn&& fn)
{
    try {
        fn();
        return OCEAN_OK;
    } catch (const std::invalid_argument&) {
        return OCEAN_ERROR_INVALID_ARG;
    } catch (const TimeoutError&) {
        return OCEAN_ERROR_TIMEOUT;
    } catch (const DeviceError& e) {
        return status_of(e);
    } catch (const std::bad_alloc&) {
        return OCEAN_ERROR_OUT_OF_MEMORY;
    } catch (...) {
        return OCEAN_ERROR_UNKNOWN;
    }
}

template <typename T>
struct DevBuf {
    T* p = nullptr;
    size_t n = 0;
    DevBuf() = default;
    explicit DevBuf(size_t count) : n(count)
    {
        if (count) check(cudaMalloc(&p, count * sizeof(T)), "cudaMalloc");
    }
    DevBuf(const DevBuf&) = delete;
    DevBuf& operator=(const DevBuf&) = delete;
    DevBuf(DevBuf&& o) noexcept : p(o.p), n(o.n) { o.p = nullptr; o.n = 0; }
    DevBuf& operator=(DevBuf&& o) noexcept
    {
        std::swap(p, o.p);
        std::swap(n, o.n);
        return *this;
    }
    ~DevBuf() { if (p) cudaFree(p); }
};

template <typename T>
struct HostBuf {
    T* p = nullptr;
    size_t n = 0;
    HostBuf() = default;
    explicit HostBuf(size_t count, bool zero = true) : n(count)
    {
        if (count) check(cudaMallocHost(&p, count * sizeof(T)), "cudaMallocHost");
        if (p && zero) std::memset(p, 0, count * sizeof(T));
    }
    HostBuf(const HostBuf&) = delete;
    HostBuf& operator=(const HostBuf&) = delete;
    HostBuf(HostBuf&& o) noexcept : p(o.p), n(o.n) { o.p = nullptr; o.n = 0; }
    HostBuf& operator=(HostBuf&& o) noexcept
    {
        std::swap(p, o.p);
        std::swap(n, o.n);
        return *this;
    }
    ~HostBuf() { if (p) cudaFreeHost(p); }
};

// The queue words (a ticket, then rows_done[count] and cols_done[count]) of a
// batch's persistent launches. Two sets take turns: a launch works on one and
// zeroes the other for the launch after it, so that no memset stands in front
// of a frame. It would pay to clear a launch's own words at its end, but its
// last CTA must then know that all others are done, a fence and an atomic
// round trip in each (3 x 256^2 cascade levels: 0.7 us a frame). While a
// stream is captured the launch gets a third set, zeroed by a memset in the
// same graph: a graph may be launched any number of times in a row, so its
// launches cannot take turns.
class FrameQueue {
public:
    struct Set {
        unsigned* ticket;
        unsigned* counters;  // rows_done, then cols_done
        unsigned* clear;     // the next launch's words, or null
        uint32_t words;      // of the next launch
        bool turn;           // call launched() once the launch is queued
    };

    FrameQueue() = default;
    // Zeroed on `st`: later launches come after that.
    FrameQueue(size_t count, cudaStream_t st) : words_(1 + 2 * count), w_(3 * words_)
    {
        check(cudaMemsetAsync(w_.p, 0, w_.n * sizeof(unsigned), st), "queue");
    }
    Set take(cudaStream_t st) const
    {
        cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
        check(cudaStreamIsCapturing(st, &cap), "capture status");
        if (cap != cudaStreamCaptureStatusNone) {
            unsigned* own = w_.p + 2 * words_;
            check(cudaMemsetAsync(own, 0, words_ * sizeof(unsigned), st), "queue reset");
            return {own, own + 1, nullptr, 0u, false};
        }
        unsigned* own = w_.p + turn_ * words_;
        return {own, own + 1, w_.p + (turn_ ^ 1) * words_, static_cast<uint32_t>(words_), true};
    }
    void launched(const Set& s)
    {
        if (s.turn) turn_ ^= 1;
    }

private:
    size_t words_ = 0;
    DevBuf<unsigned> w_;
    int turn_ = 0;
};

}  // namespace ocean_b200
