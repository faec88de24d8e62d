// Launch of a Runge-Kutta stage of a spatial order other than 5 (fin_hi.cu).
#pragma once
#include <cuda_runtime.h>

namespace fin {
struct StageArgs;
namespace hi {

// One stage of space_order 1, 7, 9 or 11 with the given WENO version (power2:
// power_param is 2); cudaErrorInvalidValue for a pair that is not built.
cudaError_t launch(int order, int weno_version, bool power2, const StageArgs& a, cudaStream_t stream);

}  // namespace hi
}  // namespace fin
