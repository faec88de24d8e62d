// The host's wait for a number that the last kernel of a step writes to pinned
// memory.
#pragma once
#include <cuda_runtime.h>
#include <atomic>
#include <chrono>
#include <thread>

namespace fin {

// Polls at first: a stream synchronisation adds 3 to 4 us to a step (27 us at 96 x
// 80, 420 at 1023 x 1025).  From TIGHT_US on the polls give the core away in
// between, so that more solver threads than cores do not sit out one another's
// time slices (done from the start it cost 0.5 us a step).  From SPIN_US on, and
// always under a schedule flag that asks for yielding or blocking
// (cudaDeviceScheduleYield, cudaDeviceScheduleBlockingSync), the wait is
// cudaStreamSynchronize's.
// *there: the number has come; without it and without an error the stream ended
// without a result.
inline cudaError_t wait_number(const volatile unsigned long long* got, unsigned long long seq, cudaStream_t stream,
                               bool* there)
{
    constexpr int TIGHT_US = 60, SPIN_US = 2000, POLLS = 64;
    unsigned flags = 0;
    cudaError_t e = cudaGetDeviceFlags(&flags);
    if (e != cudaSuccess) return e;
    const unsigned sched = flags & cudaDeviceScheduleMask;
    if (sched != cudaDeviceScheduleYield && sched != cudaDeviceScheduleBlockingSync) {
        const auto t0 = std::chrono::steady_clock::now();
        for (;;) {
            for (int k = 0; k < POLLS; k++) {
                if (*got == seq) {
                    std::atomic_thread_fence(std::memory_order_acquire);
                    *there = true;
                    return cudaSuccess;
                }
#if defined(__x86_64__)
                __builtin_ia32_pause();
#endif
            }
            const auto us = std::chrono::duration_cast<std::chrono::microseconds>(std::chrono::steady_clock::now() - t0);
            if (us.count() >= SPIN_US) break;
            if (us.count() >= TIGHT_US) std::this_thread::yield();
        }
    }
    e = cudaStreamSynchronize(stream);
    std::atomic_thread_fence(std::memory_order_acquire);
    *there = *got == seq;
    return e;
}

}  // namespace fin
