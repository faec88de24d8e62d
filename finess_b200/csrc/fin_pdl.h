// Launches on a stream that let the kernel start before the kernel ahead of it
// has ended (programmatic dependent launch).  The kernel runs
// griddepcontrol.wait before it reads anything an earlier kernel wrote, and
// griddepcontrol.launch_dependents so that its own successor may be placed; the
// wait returns when the kernel ahead has completed and its writes are visible.
// Such a kernel reads what earlier kernels wrote by plain loads, ld_dep
// (fin_device.cuh), cp.async or TMA, never through the non-coherent path.
#pragma once
#include <cuda_runtime.h>

namespace fin {

template <class... P, class... A>
inline cudaError_t launch_pdl(void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A&&... args)
{
    cudaLaunchConfig_t c = {};
    c.gridDim = grid;
    c.blockDim = block;
    c.dynamicSmemBytes = smem;
    c.stream = stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    c.attrs = at;
    c.numAttrs = 1;
    return cudaLaunchKernelEx(&c, kern, P(args)...);
}

}  // namespace fin
