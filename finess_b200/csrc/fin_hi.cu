// The stage kernel of the spatial orders other than 5 (space_order 1, 7, 9,
// 11; ConstructL.cpp:31-33, 62-358), FP64: k_stage with a halo of r =
// (space_order + 1) / 2 cells and the reconstructions of fin_weno_hi.cuh.  A
// translation unit of its own (30 instantiations).
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

// Powers other than 2 take the kernel over: three to six calls of pow a
// reconstruction, each a long chain of dependent operations.  On few tiles, and in
// order 11, whose 15 x 16 tile leaves one CTA per SM, tiles of 7 x 16 with a thread
// for every face spread them; there, and in the Z form, whose divisions the
// compiler schedules badly among inlined powers, pow is one function.  One step
// with power 1.5, us, as one thread per face of the whole grid / fused with 15 x
// 16 tiles and inlined powers / now:
//   JS7 64 x 70 136 / 182 / 102, 200 x 210 218 / 222 / 201, 1024^2 3022 / 2840 / 2840;
//   Z7  144 / 213 / 104, 218 / 239 / 203, 3038 / 3110 / 2960;
//   JS9 158 / 237 / 120, 259 / 279 / 241, 3960 / 3672 / 3672;
//   Z9  159 / 262 / 126, 264 / 301 / 252, 4008 / 4008 / 3801;
//   JS11 173 / 296 / 154, 348 / 551 / 314, 5321 / 8260 / 5180.
// The smaller tile serves up to 200 tiles of 15 x 16 (the FP64 stage's line; at
// 256^2, 288 tiles, JS7 takes 222 with the larger and 238 with the smaller) and,
// up to three waves (two CTAs on each of 148 SMs), grids whose last wave of the
// larger tile is at most a third full: JS9 at 270^2 (306 tiles) 369 with one
// thread per face, 462 with the larger tile, 361 with the smaller, at 300^2 (380)
// 437 / 466 / 415, at 315^2 (420) 480 / 467 / 482, at 400^2 (675) 692 / 703 / 668.
// Where a second wave of the smaller tile has just begun (185^2, 324 tiles) it
// takes 203 in JS7 (186 with one thread per face) and 306 in JS11 (259); three
// CTAs per SM (80 registers) take 187 and 386 there, and 3 to 60 % more beyond.
constexpr long long SMALL_TILES = 200, WAVE = 2 * 148;
inline bool small_tile(long long tiles)
{
    const long long last = tiles % WAVE;
    return tiles <= SMALL_TILES || (tiles > WAVE && tiles < 3 * WAVE && last > 0 && last <= WAVE / 3);
}

template <int ORDER, int VER, bool P2, bool SMALL, bool LONG = false>
cudaError_t launch_tile(const StageArgs& a, SmemGrants& g, cudaStream_t stream)
{
    using Cfg = TileCfg<(SMALL ? 7 : 15), 16, 256, (ORDER + 1) / 2>;
    if constexpr (!LONG && (!SMALL || ORDER == 11)) {
        if ((a.mx + Cfg::TI - 1) / Cfg::TI > 65535) return launch_tile<ORDER, VER, P2, SMALL, true>(a, g, stream);
    }
    auto kern = k_stage<double, VER, P2, Cfg, false, ORDER, LONG>;
    const size_t smem = Cfg::template smem_bytes<double>();
    const cudaError_t e = g.allow(kern, smem);
    if (e != cudaSuccess) return e;
    return launch_pdl(kern, tile_grid(a.mx, a.my, Cfg::TI, Cfg::TJ), dim3(Cfg::NT), smem, stream, a);
}

template <int ORDER, int VER, bool P2>
cudaError_t launch_t(const StageArgs& a, SmemGrants& g, cudaStream_t stream)
{
    if constexpr (P2) {
        return launch_tile<ORDER, VER, P2, false>(a, g, stream);
    } else if constexpr (ORDER == 11) {
        return launch_tile<ORDER, VER, P2, true>(a, g, stream);
    } else {
        const long long tiles = (long long)((a.mx + 14) / 15) * ((a.my + 15) / 16);
        return small_tile(tiles) ? launch_tile<ORDER, VER, P2, true>(a, g, stream)
                                 : launch_tile<ORDER, VER, P2, false>(a, g, stream);
    }
}

template <int ORDER>
cudaError_t launch_o(int v, bool p2, const StageArgs& a, SmemGrants& g, cudaStream_t s)
{
    if (v == FIN_WENO_FD) return launch_t<ORDER, FIN_WENO_FD, true>(a, g, s);
    if (v == FIN_WENO_Z) return p2 ? launch_t<ORDER, FIN_WENO_Z, true>(a, g, s) : launch_t<ORDER, FIN_WENO_Z, false>(a, g, s);
    return p2 ? launch_t<ORDER, FIN_WENO_JS, true>(a, g, s) : launch_t<ORDER, FIN_WENO_JS, false>(a, g, s);
}

cudaError_t launch(int order, int v, bool p2, const StageArgs& a, SmemGrants& g, cudaStream_t s)
{
    switch (order) {
    case 1: return launch_t<1, FIN_WENO_JS, true>(a, g, s);
    case 7: return launch_o<7>(v, p2, a, g, s);
    case 9: return launch_o<9>(v, p2, a, g, s);
    case 11: return p2 ? launch_t<11, FIN_WENO_JS, true>(a, g, s) : launch_t<11, FIN_WENO_JS, false>(a, g, s);
    }
    return cudaErrorInvalidValue;
}

}  // namespace hi
}  // namespace fin
