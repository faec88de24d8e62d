// Launch of a Runge-Kutta stage of a spatial order other than 5 (fin_hi.cu).
#pragma once
#include <cuda_runtime.h>
#include "fin_smem.h"

namespace fin {
struct StageArgs;
namespace hi {

inline bool built(int order) { return order == 1 || order == 7 || order == 9 || order == 11; }

// One stage of a space_order that is built, with the given WENO version (power2:
// power_param is 2).
cudaError_t launch(int order, int weno_version, bool power2, const StageArgs& a, SmemGrants& smem, cudaStream_t stream);

}  // namespace hi
}  // namespace fin
