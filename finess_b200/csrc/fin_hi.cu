// The stage kernel of the spatial orders other than 5 (space_order 1, 7, 9,
// 11; ConstructL.cpp:31-33, 62-358), FP64: k_stage with a halo of r =
// (space_order + 1) / 2 cells and the reconstructions of fin_weno_hi.cuh.  A
// translation unit of its own (26 instantiations).
//
// What bounds it: the FP64 pipe, and shared-memory reads of the longer stencils
// beside it (65 and 76 % busy for WENO7-JS).  Two SSP-RK3 steps at 1024^2, ms,
// first as one thread per face of the whole grid (stencil gathered from global
// memory, fluxes and projections of its points in 688 to 1008 bytes of local
// arrays, face fluxes through HBM, a second kernel for the update), then as this
// fused tile with the indicators on differences: LLF 0.84 -> 0.56, JS7 2.93 ->
// 1.53, Z7 3.30 -> 1.58, FD7 2.11 -> 1.30, JS9 3.58 -> 2.03, Z9 3.98 -> 2.01.
#include "fin_hi.h"
#include "fin_pdl.h"
#include "fin_stage.cuh"

namespace fin {
namespace hi {

template <int ORDER, int VER, bool P2, bool LONG = false>
cudaError_t launch_t(const StageArgs& a, cudaStream_t stream)
{
    using Cfg = TileCfg<15, 16, 256, (ORDER + 1) / 2>;
    if (!LONG && (a.mx + Cfg::TI - 1) / Cfg::TI > 65535) return launch_t<ORDER, VER, P2, true>(a, stream);
    auto kern = k_stage<double, VER, P2, Cfg, false, ORDER, LONG>;
    const size_t smem = Cfg::template smem_bytes<double>();
    static bool configured = false;   // per instantiation; the attribute is per device function
    if (!configured) {
        const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
        if (e != cudaSuccess) return e;
        configured = true;
    }
    return launch_pdl(kern, tile_grid(a.mx, a.my, Cfg::TI, Cfg::TJ), dim3(Cfg::NT), smem, stream, a);
}

template <int ORDER>
cudaError_t launch_o(int v, bool p2, const StageArgs& a, cudaStream_t s)
{
    if (v == FIN_WENO_FD) return launch_t<ORDER, FIN_WENO_FD, true>(a, s);
    if (v == FIN_WENO_Z) return p2 ? launch_t<ORDER, FIN_WENO_Z, true>(a, s) : launch_t<ORDER, FIN_WENO_Z, false>(a, s);
    return p2 ? launch_t<ORDER, FIN_WENO_JS, true>(a, s) : launch_t<ORDER, FIN_WENO_JS, false>(a, s);
}

cudaError_t launch(int order, int v, bool p2, const StageArgs& a, cudaStream_t s)
{
    switch (order) {
    case 1: return launch_t<1, FIN_WENO_JS, true>(a, s);
    case 7: return launch_o<7>(v, p2, a, s);
    case 9: return launch_o<9>(v, p2, a, s);
    case 11: return p2 ? launch_t<11, FIN_WENO_JS, true>(a, s) : launch_t<11, FIN_WENO_JS, false>(a, s);
    }
    return cudaErrorInvalidValue;
}

}  // namespace hi
}  // namespace fin
