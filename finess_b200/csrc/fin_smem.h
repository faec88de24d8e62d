// Dynamic shared memory above 48 KB is granted to a kernel by an attribute that
// belongs to the device's copy of the kernel and goes with its context.  A solver
// sets it at the first launch of each kernel it uses: not once per process, which
// would leave a second device's kernels, or those of a context made after
// cudaDeviceReset, without it.
#pragma once
#include <cuda_runtime.h>

namespace fin {

struct SmemGrants {
    static constexpr int MAX = 8;   // kernels a solver uses (beyond: granted at each launch)
    const void* kern[MAX];          // the owner is zeroed
    int n;

    template <class K>
    cudaError_t allow(K* k, size_t bytes)
    {
        const void* f = reinterpret_cast<const void*>(k);
        for (int i = 0; i < n; i++)
            if (kern[i] == f) return cudaSuccess;
        const cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, int(bytes));
        if (e == cudaSuccess && n < MAX) kern[n++] = f;
        return e;
    }
};

}  // namespace fin
