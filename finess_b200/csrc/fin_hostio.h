// Device results into fresh host arrays in pageable memory (numpy, dTensor)
// through a small pinned ring: the CPU moves one chunk while the copy engine
// brings the next ones, and what arrives is laid out or folded while it is read
// out of the ring, so that no second host array is needed.
#pragma once
#include <cuda_runtime.h>

namespace fin {

// Bound by the CPU's copy and the page faults of the fresh array (3.2 MB: 190 us
// of the 260 that a copy through the ring takes).  Plain stores: the page that a
// fault has just cleared is in the cache, and streaming stores throw it out (345 ->
// 520 us).  An array whose pages are there already is better left to the runtime's
// own copy (217 against 250 us), as are copies to the device.  Chunks of 128 KB
// (64 KB: 450 us); helper threads fault against one another (4: 800 us).
struct HostRing {
    static constexpr size_t CHUNK = size_t(128) << 10;
    static constexpr int N = 4;
    char* buf;   // null, like the events, at first: the owner is zeroed
    cudaEvent_t ev[N];

    // Half a megabyte of pinned memory took 2 us to get, a megabyte 2.5 ms (B200,
    // driver 580): measured, and nothing but the time rests on it.
    cudaError_t ensure()
    {
        if (buf) return cudaSuccess;
        for (int k = 0; k < N; k++)
            if (!ev[k]) {
                const cudaError_t e = cudaEventCreateWithFlags(&ev[k], cudaEventDisableTiming);
                if (e != cudaSuccess) return e;
            }
        return cudaMallocHost(reinterpret_cast<void**>(&buf), N * CHUNK);
    }
    void destroy()
    {
        if (buf) cudaFreeHost(buf);
        for (int k = 0; k < N; k++)
            if (ev[k]) cudaEventDestroy(ev[k]);
    }
    // take(offset, chunk, n) in doubles, in order; all of src has been read on return.
    template <class F>
    cudaError_t down(const double* src, size_t len, cudaStream_t st, F&& take)
    {
        cudaError_t e = ensure();
        if (e != cudaSuccess) return e;
        constexpr size_t C = CHUNK / sizeof(double);
        const size_t chunks = (len + C - 1) / C;
        auto issue = [&](size_t k) {
            const size_t n = len - k * C < C ? len - k * C : C;
            cudaError_t r = cudaMemcpyAsync(buf + (k % N) * CHUNK, src + k * C, n * sizeof(double),
                                            cudaMemcpyDeviceToHost, st);
            return r != cudaSuccess ? r : cudaEventRecord(ev[k % N], st);
        };
        for (size_t k = 0; k < chunks && k < N; k++)
            if ((e = issue(k)) != cudaSuccess) return e;
        for (size_t k = 0; k < chunks; k++) {
            if ((e = cudaEventSynchronize(ev[k % N])) != cudaSuccess) return e;
            take(k * C, reinterpret_cast<const double*>(buf + (k % N) * CHUNK), len - k * C < C ? len - k * C : C);
            if (k + N < chunks && (e = issue(k + N)) != cudaSuccess) return e;
        }
        return cudaSuccess;
    }
};

}  // namespace fin
