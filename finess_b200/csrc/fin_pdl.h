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

// Blocks for tiles of ti x tj cells: columns of tiles in x, rows in y and, as y
// takes 65,535, the rest in z (tile_row).  The last few rows of tiles may then lie
// past the grid, like the cells of a partial tile.
inline dim3 tile_grid(long long mx, long long my, int ti, int tj)
{
    const long long rows = (mx + ti - 1) / ti, cols = (my + tj - 1) / tj, z = (rows + 65534) / 65535;
    return dim3(unsigned(cols), unsigned((rows + z - 1) / z), unsigned(z));
}
#ifdef __CUDACC__
__device__ __forceinline__ int tile_row() { return int(blockIdx.z * gridDim.y + blockIdx.y); }
#endif

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
