// The fused stage kernel: one launch computes, for a TI x TJ tile of cells,
//   L(q_in)   (ConstructL, lib/2d/ConstructL.cpp:62-401)
//   q_out = a1*A + a2*B + (beta*dt)*L     (UpdateSoln, lib/2d/UpdateSoln.cpp:29-35)
// and, in its epilogue, the two maxima the next stage and the CFL need:
//   * the wave-speed maxima alpha1/alpha2 of q_out over interior cells
//     (GlobalWaveSpd, lib/2d/GlobalWaveSpd.cpp:52-78), which the *next*
//     stage uses as its global alpha, so no stage needs a separate pass over
//     its own input;
//   * the maxima of the face speeds over the faces GetCFL reads
//     (lib/2d/GetCFL.cpp:54-59 reads smax(i,j,.) for i<=mx, j<=my).
// Maxima are exact, so computing them in a different order or place than the
// reference changes no bit of the result.
//
// Data layout in HBM: one plane per component, plane m holds mx*my values
// with j (y) fastest -- the reference's own axis order (x slowest,
// lib/tensors.h:267-273) without its ghost frame.  Ghost values are produced
// on load by the boundary remap (no ghost writes, no BC pass).
//
// Per block, shared memory holds (R = double or float):
//   prim [4][TI+6][TJ+6]  u, v, p, c of the cells
//   qs  [M][TI+6][TJ+6]   stage input with a 3-cell halo (corners unused)
//   fs  [M][TI+6][TJ]     x flux f at the x-stencil cells
//   gs  [M][TI][TJ+6]     y flux g at the y-stencil cells
//   Fh  [M][TI+1][TJ]     x-face numerical fluxes
//   Gh  [M][TI][TJ+1]     y-face numerical fluxes
//   opnd [M][TI][TJ]      the stage operand that is not q_in (FP64)
// Phases: load (coalesced along j) and flux per cell (FluxFunc once per cell,
// not six times per face as the reference does) -> one thread per face, x
// faces then y faces (projection, LLF split, two WENO5, back projection, all
// in registers) -> per cell flux difference + RK update + next-stage wave
// speed -> block max -> one atomicMax per block.
//
// What bounds it: the FP64 form is bound by the FP64 pipe and by the latency
// of dependent FP64 operations at 16 warps per SM (128 registers), so what
// counts is instructions per face and registers.  Measured, SSP-RK3 step at
// 4096^2 (three launches, ms): 10.54 with candidates and smoothness
// indicators on point values, projection rows written out and one face body
// for both directions; 8.75 with the difference form (weno5_diff), the shared
// projection sums (Euler::Face) and the upwind part of the flux parked in its
// slot; 7.58 with one body per direction (constant stencil offsets: integer
// multiply-adds and moves fell from 17 to 4 % of the instructions, spills
// from 180 to 70 bytes), load and flux phases in one, the stage operand
// copied behind the face phase (q_in's own values taken from shared memory)
// and the warp maxima by two reduce instructions each (FP64 pipe 61 % busy,
// 52 % before); 7.33 with the upwind part projected with the rest and
// everything that only the end of a face needs waiting in its flux slots
// (no spills; the batch form of the kernel, which had spilled 246 bytes, took
// 134 instead of 153 ms for a batch of 48).  The same body changes took the
// FP32 form's step from 1.69 to 1.48 ms (two steps of 4001 x 515).
#pragma once
#include "fin_device.cuh"
#include "fin_pdl.h"
#include "fin_tc.cuh"
#include "fin_weno_face.cuh"
#include "fin_weno_hi.cuh"
#include <type_traits>

namespace fin {

struct StageArgs {
    const double* qin;     // stage input planes
    const double* A;       // a1 term (may alias qin); nullptr = term absent
    const double* B;       // a2 term; nullptr = term absent
    double* qout;          // output planes (never aliases qin)
    double a1, a2, bdt;    // bdt = beta*dt
    int mx, my;
    size_t plane;          // elements per component plane (>= mx*my)
    double rdx, rdy;       // 1/dx, 1/dy
    double gamma, eps, pw, alpha_scaling;
    float gamma_f, eps_f, pw_f, alpha_scaling_f;   // the same in FP32 (set by the launcher)
    const double* alpha_in;   // [2] global alpha of q_in (x, y); nullptr = local LLF
    double* alpha_out;        // [2] max cell speed of q_out; nullptr = skip
    double* smax_out;         // [2] max face speed over GetCFL's faces; nullptr = skip
    double* face_alpha_x;     // optional per-face alpha, (mx+1)*my, face-major i then j
    double* face_alpha_y;     // optional per-face alpha, mx*(my+1)
    unsigned int* status;     // bit 0: non-finite speed, bit 1: negative p or rho, bit 3: TMA wait ran out,
                              // bit 4: misaligned TMA destination (remap path taken)
    int bc[4];                // xlow, xhigh, ylow, yhigh
    // Lax-Wendroff / multiderivative stages (ConstructLxWL): the split fluxes
    // are the time-integrated F, G (ghosted (mx+6) x (my+6) planes) instead of
    // FluxFunc of q_in (lib/2d/ConstructLxWL.cpp:150-155).
    const double* Fg;
    const double* Gg;
    size_t gplane;
    // Lax-Wendroff with the MPP limiter (FinSolveLxW.cpp:126-151): the stage
    // writes its face fluxes (flux_x [m][mx+1][my], flux_y [m][mx][my+1],
    // ConstructLxWL's Fhat / Ghat) and no update (flux_only), and leaves the
    // first face of each direction out of the face-speed maximum, whose smax
    // entry ConstructLFL.cpp:62-65 overwrites with the global wave speed.
    double* flux_x;
    double* flux_y;
    int flux_only;
    // Hybrid form: troubled-face flags of the step as bit masks (layout of
    // flag_wx / flag_wy below, written by the indicator).  A face takes full
    // WENO when any flag in the 3 x 3 window of same-direction faces around
    // it is set, else the linear FD5 weights (lib/WenoReconstruct.cpp:580-616).
    const unsigned* flags;
    // Hybrid form on grids whose row pitch suits TMA (my even): tensor maps
    // of q_in (box (TJ+8) x (TI+6) x 5, the tile with its halo) and of the
    // stage operand that is not q_in (box TJ x TI x 5); tiles clear of the
    // domain boundary stage both with one TMA transaction each.
    int tma;
    CUtensorMap tm_in;
    CUtensorMap tm_A;
    // The same two maps held in global memory (batches, whose stage
    // arguments live in global memory): used instead of tm_in / tm_A when
    // set, after a tensormap-proxy acquire fence.
    const CUtensorMap* gtm_in;
    const CUtensorMap* gtm_A;
};

// Troubled-face flags, one bit per face: x faces (rows 0 .. mx) take
// flag_wx words per row, bit b of word k being column 32 k + b; the y faces
// (rows 0 .. mx-1, columns 0 .. my) follow with flag_wy words per row.
__host__ __device__ __forceinline__ int flag_wx(int my) { return (my + 31) >> 5; }
__host__ __device__ __forceinline__ int flag_wy(int my) { return (my + 32) >> 5; }
__host__ __device__ __forceinline__ size_t flag_words(int mx, int my)
{
    return size_t(mx + 1) * flag_wx(my) + size_t(mx) * flag_wy(my);
}
// Bits of columns b0 .. b0+31 of one mask row from the words holding them
// (k = b0 >> 5 and k + 1; columns outside the row read as 0).
__device__ __forceinline__ unsigned row_bits(unsigned lo, unsigned hi, int b0)
{
    return unsigned(((unsigned long long)hi << 32 | lo) >> (b0 & 31));
}

// A tile of TI x TJ cells, NT threads, stencils reaching H cells out.
template <int TI_, int TJ_, int NT_, int H_ = 3>
struct TileCfg {
    static constexpr int TI = TI_, TJ = TJ_, NT = NT_, H = H_;
    static constexpr int RI = TI + 2 * H, RJ = TJ + 2 * H;
    static constexpr int NFX = (TI + 1) * TJ, NFY = TI * (TJ + 1);
    static constexpr bool ONE_ROUND = NFX + NFY <= NT;   // a thread per face of the tile
    static constexpr int NPRIM = 4;   // per-cell u, v, p, c of the cross region
    // FP32 faces of a 15 x 16 tile go to threads so that the two half-warps
    // of a warp take face rows 8 apart (XROW8): 8 rows of RJ = 22 words are
    // 176 words, 16 modulo 32, so the two rows' words fall in opposite
    // halves of the banks; the x-direction flux rows get a pitch of 18 for
    // the same reason (8 x 18 = 144).  FP64 (a half-warp reads one row of
    // 8-byte words) keeps the row-by-row order.
    template <class R>
    __host__ __device__ static constexpr bool XROW8() { return sizeof(R) == 4 && TI == 15 && TJ == 16; }
    template <class R>
    __host__ __device__ static constexpr int FSJ() { return XROW8<R>() ? TJ + 2 : TJ; }
    // byte offsets of the staged stage operand (FP64) and of the reduction
    // scratch (after the arrays, 16-B aligned)
    template <class R>
    __host__ __device__ static constexpr size_t red_offset()
    {
        return opnd_offset<R>() + (sizeof(R) == 8 ? size_t(MEQN) * TI * TJ * 8 : 0);
    }
    template <class R>
    __host__ __device__ static constexpr size_t opnd_offset()
    {
        return (sizeof(R) * (size_t(MEQN) * (size_t(RI) * RJ + size_t(RI) * FSJ<R>() + size_t(TI) * RJ +
                                             size_t(TI + 1) * TJ + size_t(TI) * (TJ + 1)) +
                             size_t(NPRIM) * RI * RJ) + 15) / 16 * 16;
    }
    template <class R>
    __host__ __device__ static constexpr size_t smem_bytes() { return red_offset<R>() + 4 * (NT / 32) * sizeof(double); }
    // Hybrid form (k_stage_hyb): the flag windows of the 3 x 3 dilation as
    // one bit mask per face row (x faces: rows i0-1 .. i0+TI+1, bit c =
    // column j0-1+c, c < TJ+2; y faces: rows i0-1 .. i0+TI, c < TJ+3).
    static constexpr int FXR = TI + 3, FXC = TJ + 2, FYR = TI + 2, FYC = TJ + 3;
    static constexpr bool MASKS_FIT = FYC <= 32;   // flag row masks are 32-bit words
    // The FP64 staging tile of q_in (rows i0-3 .. i0+TI+2, columns j0-4 ..
    // j0+TJ+3, so the TMA box starts on a 16-byte boundary); a TMA destination
    // starts on a 128-byte boundary, so offsets are padded to multiples of 128.
    static constexpr int SJ = TJ + 8;
    static constexpr size_t STG_BYTES = size_t(MEQN) * RI * SJ * 8;
    __host__ __device__ static constexpr size_t pad128(size_t b) { return (b + 127) / 128 * 128; }
};

// Staging of q_in's tile + 3-cell halo (the cross region: rows i0-3 ..
// i0+TI+2 at columns j0 .. j0+TJ-1, columns j0-3 .. j0+TJ+2 at rows i0 ..
// i0+TI-1) as FP64 in stg [M][RI][SJ], column jj of the tile frame at jj+1.
// A tile whose box (rows i0-3 .. i0+TI+2, columns j0-4 .. j0+TJ+3) lies in
// the domain is staged by one TMA copy; any other by loads through the
// boundary remap.
template <class Cfg>
__device__ __forceinline__ bool tma_interior(int i0, int j0, int mx, int my)
{
    return i0 >= Cfg::H && i0 + Cfg::TI + Cfg::H <= mx && j0 >= 4 && j0 + Cfg::TJ + 4 <= my;
}

template <class Cfg>
__device__ __forceinline__ void stage_remap(double* stg, const double* q, size_t plane, int i0, int j0, int mx, int my,
                                            const int* bc, int tid)
{
    constexpr int H = Cfg::H, TI = Cfg::TI, TJ = Cfg::TJ, RI = Cfg::RI, RJ = Cfg::RJ;
    for (int e = tid; e < RI * RJ; e += Cfg::NT) {
        const int ii = e / RJ, jj = e - ii * RJ;
        const bool xin = ii >= H && ii < H + TI, yin = jj >= H && jj < H + TJ;
        if (!xin && !yin) continue;
        const int gi = bc_remap(i0 + ii - H, mx, bc[0], bc[1]);
        const int gj = bc_remap(j0 + jj - H, my, bc[2], bc[3]);
        const size_t g = size_t(gi) * my + gj;
#pragma unroll
        for (int m = 0; m < MEQN; m++) stg[(m * RI + ii) * Cfg::SJ + jj + 1] = ld_dep(q + m * plane + g);
    }
}

template <class Cfg, class R>
__device__ __forceinline__ void stage_convert(const double* stg, R* qs, int tid)
{
    constexpr int H = Cfg::H, TI = Cfg::TI, TJ = Cfg::TJ, RI = Cfg::RI, RJ = Cfg::RJ;
    for (int e = tid; e < RI * RJ; e += Cfg::NT) {
        const int ii = e / RJ, jj = e - ii * RJ;
        const bool xin = ii >= H && ii < H + TI, yin = jj >= H && jj < H + TJ;
        if (!xin && !yin) continue;
#pragma unroll
        for (int m = 0; m < MEQN; m++) qs[m * RI * RJ + e] = R(stg[(m * RI + ii) * Cfg::SJ + jj + 1]);
    }
}

// 6-point flux of a face that takes the linear FD5 weights: with v+- =
// 0.5 f +- l q, the reference's characteristic form R FD5(L v+) + R FD5'(L v-)
// (ConstructL.cpp:179-250 with WenoReconstruct_FD5, WenoReconstruct.cpp:
// 580-616) equals FD5(v+) + FD5'(v-) component by component, because the
// reconstruction is linear and R L = I.  FD5 has the weights (2, -13, 47, 27,
// -3)/60 on points 0..4 and FD5' the same on points 5..1, so the face flux is
//   (1/30) [ (f0+f5) - 8 (f1+f4) + 37 (f2+f3)                      (0.5 f terms)
//          + l ((q0-q5) - 5 (q1-q4) + 10 (q2-q3)) ]                  (l = lah)
// with f the half fluxes held in shared memory: 12 operations per component
// instead of a projection, two reconstructions and a back projection.
template <class R>
__device__ __forceinline__ R linear_face(const R* f, int fstr, const R* q, int qstr, R lah)
{
    const R sf = fma(R(37), f[-1 * fstr] + f[0], fma(R(-8), f[-2 * fstr] + f[fstr], f[-3 * fstr] + f[2 * fstr]));
    const R sq = fma(R(10), q[-1 * qstr] - q[0], fma(R(-5), q[-2 * qstr] - q[qstr], q[-3 * qstr] - q[2 * qstr]));
    return fma(lah, sq, sf) * R(1.0 / 30.0);
}

// Resident blocks per SM the register budget is sized for.  Measured on B200 at
// 4096^2, WENO5-Z, ms a stage: FP64 one block (164 registers) 3.33, two (122, no
// spills) 2.39; FP32 two blocks (100 registers) 1.61, three (80, no spills) 1.281,
// four (64, 20 bytes spilled) 1.285.
#ifndef FIN_MINB_F64
#define FIN_MINB_F64 2
#endif
#ifndef FIN_MINB_F32
#define FIN_MINB_F32 3
#endif
template <class R> struct MinBlocks { static constexpr int value = FIN_MINB_F64; };
template <> struct MinBlocks<float> { static constexpr int value = FIN_MINB_F32; };

// Scalar parameters read from kernel-parameter space where they are used
// (keeps them out of the register budget of the face loop).
template <class R> struct Par;
template <> struct Par<double> {
    __device__ static double gamma(const StageArgs& a) { return a.gamma; }
    __device__ static double eps(const StageArgs& a) { return a.eps; }
    __device__ static double pw(const StageArgs& a) { return a.pw; }
    __device__ static double ascale(const StageArgs& a) { return a.alpha_scaling; }
};
template <> struct Par<float> {
    __device__ static float gamma(const StageArgs& a) { return a.gamma_f; }
    __device__ static float eps(const StageArgs& a) { return a.eps_f; }
    __device__ static float pw(const StageArgs& a) { return a.pw_f; }
    __device__ static float ascale(const StageArgs& a) { return a.alpha_scaling_f; }
};

// Scheduling fences: an empty volatile asm that reads and writes x.  Volatile
// asm statements keep their order, so fencing the inputs and result of each
// pair of WENO reconstructions stops the scheduler from evaluating all ten of
// a face at once (which wants ~230 registers in FP64).
__device__ __forceinline__ void fence(double& x) { asm volatile("" : "+d"(x)); }
__device__ __forceinline__ void fence(float& x) { asm volatile("" : "+f"(x)); }
template <class R>
__device__ __forceinline__ void fence4(R* u)
{
#pragma unroll
    for (int k = 0; k < 4; k++) fence(u[k]);
}

// Corrections (weno5_diff) of gp and gm of one characteristic field from the
// differences of their stencils, fenced as a unit.
template <class R, int VER, bool P2>
__device__ __forceinline__ R weno_pair(R* dp, R* dm, R eps4, R pw)
{
    fence4(dp);
    fence4(dm);
    R g = weno5_diff<R, VER, P2>(dp[0], dp[1], dp[2], dp[3], eps4, pw) +
          weno5_diff<R, VER, P2>(dm[0], dm[1], dm[2], dm[3], eps4, pw);
    fence(g);
    return g;
}

// A correction of another order, fenced.
template <int ORDER, int VER, bool P2, bool CALL>
__device__ __forceinline__ double hi_fenced(double* d, double eps, double pw)
{
#pragma unroll
    for (int k = 0; k < ORDER - 1; k++) fence(d[k]);
    double c = hi::correction<ORDER, VER, P2, CALL>(d, eps, pw);
    fence(c);
    return c;
}

// Max over a warp of non-negative doubles, as the maximum of their high words
// and then of the low words that go with it (two warp-reduce instructions
// instead of five rounds of two shuffles, a compare and two selects).
__device__ __forceinline__ double warp_max_nonneg(double v)
{
    const unsigned hi = unsigned(__double2hiint(v));
    const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
    const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? unsigned(__double2loint(v)) : 0u);
    return __hiloint2double(int(mh), int(ml));
}

__device__ __forceinline__ float warp_max_nonneg(float v)
{
    return __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(v)));
}

// Shared-memory arrays of a stage tile.
template <class R, class Cfg>
struct StageSmem {
    static constexpr int PQ = Cfg::RI * Cfg::RJ, FS = Cfg::template FSJ<R>();
    R* prim;   // [4][RI][RJ]   u, v, p, c
    R* qs;     // [M][RI][RJ]
    R* fs;     // [M][RI][FS]   0.5 * f
    R* gs;     // [M][TI][RJ]   0.5 * g
    R* Fh;     // [M][TI+1][TJ]
    R* Gh;     // [M][TI][TJ+1]
    double* opnd;   // [M][TI*TJ] the stage operand that is not q_in (FP64)
    double* red;
    __device__ __forceinline__ explicit StageSmem(unsigned char* raw)
    {
        prim = reinterpret_cast<R*>(raw);
        qs = prim + Cfg::NPRIM * PQ;
        fs = qs + MEQN * PQ;
        gs = fs + MEQN * Cfg::RI * FS;
        Fh = gs + MEQN * Cfg::TI * Cfg::RJ;
        Gh = Fh + MEQN * (Cfg::TI + 1) * Cfg::TJ;
        opnd = reinterpret_cast<double*>(raw + Cfg::template opnd_offset<R>());
        red = reinterpret_cast<double*>(raw + Cfg::template red_offset<R>());
    }
};

// The start of a kernel launched by launch_pdl (fin_pdl.h): its successor may
// be placed, and it waits for its predecessor.
__device__ __forceinline__ void grid_dependency()
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// Flux of face k of direction x (ISX: between rows fi-1 and fi of the tile)
// or y (between columns fj-1 and fj), in registers; the direction is a
// template parameter, so every stencil address is a constant offset.  Returns
// the face's LLF speed and whether it enters GetCFL's maximum in *in_cfl.
template <class R, int VER, bool P2, class Cfg, bool FG, bool ISX, int ORDER>
__device__ __forceinline__ R stage_face(const StageArgs& a, const StageSmem<R, Cfg>& S, int w, int i0, int j0, R ag,
                                        bool& neg, bool& in_cfl)
{
    constexpr int TI = Cfg::TI, TJ = Cfg::TJ, H = Cfg::H, RI = Cfg::RI, RJ = Cfg::RJ;
    constexpr int PQ = RI * RJ, FS = Cfg::template FSJ<R>();
    constexpr int CN = ISX ? 1 : 2, CT = ISX ? 2 : 1;   // normal / tangential momentum
    constexpr int QSTR = ISX ? RJ : 1, FSTR = ISX ? FS : 1, FP = ISX ? RI * FS : TI * RJ;
    constexpr int OP = ISX ? (TI + 1) * TJ : TI * (TJ + 1);
#define gamma (Par<R>::gamma(a))
#define eps (Par<R>::eps(a))
#define pw (Par<R>::pw(a))
    int fi, fj;
    if (ISX) {
        if constexpr (Cfg::template XROW8<R>()) {
            fi = (w >> 5) + ((w >> 1) & 8); fj = w & 15;   // half-warps on rows r and r + 8
        } else {
            fi = w / TJ; fj = w - fi * TJ;
        }
    } else {
        // taken by rows of TJ, then the last column, so a half-warp reads one
        // row of the staged tile (FP32: half-warps on rows r and r + 8; the
        // last warp takes row 7 and the last column)
        if constexpr (Cfg::template XROW8<R>()) {
            const int wv = w >> 5, ln = w & 31;
            if (wv < 7) { fi = wv + (ln & 16 ? 8 : 0); fj = ln & 15; }
            else if (ln < 16) { fi = 7; fj = ln; }
            else { fi = ln - 16; fj = TJ; }
        } else {
            fi = w < TI * TJ ? w / TJ : w - TI * TJ;
            fj = w < TI * TJ ? w - fi * TJ : TJ;
        }
    }
    const R* const qb = S.qs + (H + fi) * RJ + (H + fj);
    const R* const pb = S.prim + (H + fi) * RJ + (H + fj);
    const R* const fb = ISX ? S.fs + (H + fi) * FS + fj : S.gs + fi * RJ + (H + fj);
    R* const out = ISX ? S.Fh + fi * TJ + fj : S.Gh + fi * (TJ + 1) + fj;
    // Face average (ConstructL.cpp:72-77) in the normal frame.
    R Qa[MEQN];
    Qa[0] = R(0.5) * (qb[0] + qb[-QSTR]);
    Qa[1] = R(0.5) * (qb[CN * PQ] + qb[CN * PQ - QSTR]);
    Qa[2] = R(0.5) * (qb[CT * PQ] + qb[CT * PQ - QSTR]);
    Qa[3] = R(0.5) * (qb[3 * PQ] + qb[3 * PQ - QSTR]);
    Qa[4] = R(0.5) * (qb[4 * PQ] + qb[4 * PQ - QSTR]);
    const Euler::Face<R> ev = Euler::face(gamma, Qa);
    // SetWaveSpd.cpp:39-68 from the two cells' u_n, p, c (nmag = 1) and
    // the LLF alpha of ConstructL.cpp:172-174.
    R alpha;
    {
        constexpr int UN = ISX ? 0 : 1;
        const R unl = pb[UN * PQ - QSTR], unr = pb[UN * PQ];
        const R pl = pb[2 * PQ - QSTR], pr = pb[2 * PQ];
        const R cl = pb[3 * PQ - QSTR], cr = pb[3 * PQ];
        const R ua = R(0.5) * (unl + unr);
        const R pa = R(0.5) * (pl + pr);
        const R ca = sqrt_fast(fabs(gamma * pa * ev.ir));
        if (pa < R(0) || Qa[0] < R(0)) neg = true;
        const R s1 = MinN(unl - cl, ua - ca);
        const R s2 = MaxN(unr + cr, ua + ca);
        alpha = MaxN(ag, MaxN(R(fabs(s1)), R(fabs(s2))));
    }
    // GetCFL's Max skips NaN entries (Max(NaN, c) = c), so only finite face
    // speeds enter the CFL maximum.
    const int gi = i0 + fi, gj = j0 + fj;
    in_cfl = gi < a.mx && gj < a.my && !(FG && a.flux_only && gi == 0 && gj == 0);
    {
        double* const fa = ISX ? a.face_alpha_x : a.face_alpha_y;
        if (fa && gi < a.mx + (ISX ? 1 : 0) && gj < a.my + (ISX ? 0 : 1))
            fa[size_t(gi) * (a.my + (ISX ? 0 : 1)) + gj] = double(alpha);
    }
    // gp = 0.5 (L f + l_alpha L q) = L (0.5 f + 0.5 l_alpha q), points
    // 0..4; gm the same with -l_alpha, points 5..1 (ConstructL.cpp:179-185).
    const R lah = R(0.5) * Par<R>::ascale(a) * alpha;
    R fh[MEQN];
    if constexpr (sizeof(R) == 4) {
        auto pt = [&](int s, f2* v) {
            const int oq = (s - 3) * QSTR, of = (s - 3) * FSTR;
            v[0] = f2_make(fb[of], qb[oq]);
            v[1] = f2_make(fb[CN * FP + of], qb[CN * PQ + oq]);
            v[2] = f2_make(fb[CT * FP + of], qb[CT * PQ + oq]);
            v[3] = f2_make(fb[3 * FP + of], qb[3 * PQ + oq]);
            v[4] = f2_make(fb[4 * FP + of], qb[4 * PQ + oq]);
        };
        auto slot = [&](int m) -> R& { return out[(m == 1 ? CN : m == 2 ? CT : m) * OP]; };
        weno_char_flux<VER, P2>(ev, lah, eps, pw, pt, [&](int m, R x) { slot(m) = x; }, [&](int m) { return slot(m); }, fh);
    } else if constexpr (ORDER != 5) {
        // The other orders (FP64): split by split -- gp from v+ at the points
        // 0 .. ORDER-1, gm from v- at the points ORDER .. 1 -- fields 0, 1 and
        // 4, then 2 and 3; the fields' sums wait in the face's flux slots.
        constexpr int NW = ORDER, C = (ORDER - 1) / 2;   // points, the upwind one
        constexpr bool CALL = Cfg::ONE_ROUND || VER == FIN_WENO_Z;
        auto half = [&](auto minus) {
            constexpr bool M = decltype(minus)::value;
            const R l = M ? -lah : lah;
            auto put = [&](int k, R x) {
                if (M) out[k * OP] += x;
                else out[k * OP] = x;
            };
            {
                R d0[NW], d1[NW], d4[NW], c0, c1, c4;
#pragma unroll
                for (int t = 0; t < NW; t++) {
                    asm volatile("" ::: "memory");
                    const int s = M ? NW - t : t, oq = (s - H) * QSTR, of = (s - H) * FSTR;
                    const R v[MEQN] = {fb[of] + l * qb[oq], fb[CN * FP + of] + l * qb[CN * PQ + oq],
                                       fb[CT * FP + of] + l * qb[CT * PQ + oq], fb[3 * FP + of] + l * qb[3 * PQ + oq],
                                       fb[4 * FP + of] + l * qb[4 * PQ + oq]};
                    R w0, w1, w4;
                    Euler::left014(ev, v, w0, w1, w4);
                    if (t > 0) { d0[t - 1] = w0 - c0; d1[t - 1] = w1 - c1; d4[t - 1] = w4 - c4; }
                    if (t == C) { put(0, w0); put(1, w1); put(4, w4); }
                    c0 = w0; c1 = w1; c4 = w4;
                }
                out[0] += hi_fenced<ORDER, VER, P2, CALL>(d0, eps, pw);
                out[4 * OP] += hi_fenced<ORDER, VER, P2, CALL>(d4, eps, pw);
                out[OP] += hi_fenced<ORDER, VER, P2, CALL>(d1, eps, pw);
            }
            {
                R d2[NW], d3[NW], c2, c3;
#pragma unroll
                for (int t = 0; t < NW; t++) {
                    asm volatile("" ::: "memory");
                    const int s = M ? NW - t : t, oq = (s - H) * QSTR, of = (s - H) * FSTR;
                    const R v0 = fb[of] + l * qb[oq];
                    const R w2 = (fb[CT * FP + of] + l * qb[CT * PQ + oq]) - ev.u2 * v0;
                    const R w3 = (fb[3 * FP + of] + l * qb[3 * PQ + oq]) - ev.u3 * v0;
                    if (t > 0) { d2[t - 1] = w2 - c2; d3[t - 1] = w3 - c3; }
                    if (t == C) { put(2, w2); put(3, w3); }
                    c2 = w2; c3 = w3;
                }
                out[2 * OP] += hi_fenced<ORDER, VER, P2, CALL>(d2, eps, pw);
                out[3 * OP] += hi_fenced<ORDER, VER, P2, CALL>(d3, eps, pw);
            }
        };
        half(std::false_type{});
        half(std::true_type{});
        const R g[MEQN] = {out[0], out[OP], out[2 * OP], out[3 * OP], out[4 * OP]};
        Euler::right(ev, g, fh);
    } else {
        // Characteristic values as their upwind points (v+ of the left cell
        // plus v- of the right cell) plus corrections / 6 from differences of
        // the projected points (weno5_diff).  Fields 0, 4 and 1 in one sweep
        // of the stencil, then 2 and 3 (all five at once want more registers
        // than two CTAs per SM leave); what only the end of the face needs
        // waits in its flux slots.
        R g[MEQN];
        const R eps4 = R(4) * eps, s6 = R(1) / R(6);
        {
            out[3 * OP] = ev.c;
            out[4 * OP] = ev.h;
            R p0[4], p4[4], m0[4], m4[4], p1[4], m1[4];
            R cp0, cp1, cp4, cm0, cm1, cm4;   // the previous point's values
#pragma unroll
            for (int s = 0; s < 6; s++) {
                // keep the compiler from hoisting every stencil point's loads
                // ahead of the arithmetic
                asm volatile("" ::: "memory");
                const int oq = (s - 3) * QSTR, of = (s - 3) * FSTR;
                const R q0 = qb[oq], qn = qb[CN * PQ + oq], qt = qb[CT * PQ + oq], qw = qb[3 * PQ + oq],
                        qe = qb[4 * PQ + oq];
                const R f0 = fb[of], fn = fb[CN * FP + of], ft = fb[CT * FP + of], fw = fb[3 * FP + of],
                        fe = fb[4 * FP + of];
                R w0, w1, w4;
                if (s < 5) {
                    const R v[MEQN] = {f0 + lah * q0, fn + lah * qn, ft + lah * qt, fw + lah * qw, fe + lah * qe};
                    Euler::left014(ev, v, w0, w1, w4);
                    if (s > 0) { p0[s - 1] = w0 - cp0; p1[s - 1] = w1 - cp1; p4[s - 1] = w4 - cp4; }
                    if (s == 2) { out[0] = w0; out[OP] = w1; out[2 * OP] = w4; }
                    cp0 = w0; cp1 = w1; cp4 = w4;
                }
                if (s > 0) {
                    const R v[MEQN] = {f0 - lah * q0, fn - lah * qn, ft - lah * qt, fw - lah * qw, fe - lah * qe};
                    Euler::left014(ev, v, w0, w1, w4);
                    if (s > 1) { m0[5 - s] = cm0 - w0; m1[5 - s] = cm1 - w1; m4[5 - s] = cm4 - w4; }
                    if (s == 3) { out[0] += w0; out[OP] += w1; out[2 * OP] += w4; }
                    cm0 = w0; cm1 = w1; cm4 = w4;
                }
            }
            g[0] = s6 * weno_pair<R, VER, P2>(p0, m0, eps4, pw) + out[0];
            g[4] = s6 * weno_pair<R, VER, P2>(p4, m4, eps4, pw) + out[2 * OP];
            g[1] = s6 * weno_pair<R, VER, P2>(p1, m1, eps4, pw) + out[OP];
        }
        {
            // fields 2 and 3 (rows v_t - u2 v0 and v_w - u3 v0)
            R p2[4], p3[4], m2[4], m3[4];
            R cp2, cp3, cm2, cm3;
#pragma unroll
            for (int s = 0; s < 6; s++) {
                asm volatile("" ::: "memory");
                const int oq = (s - 3) * QSTR, of = (s - 3) * FSTR;
                const R q0 = qb[oq], qt = qb[CT * PQ + oq], qw = qb[3 * PQ + oq];
                const R f0 = fb[of], ft = fb[CT * FP + of], fw = fb[3 * FP + of];
                if (s < 5) {
                    const R v0 = f0 + lah * q0;
                    const R w2 = (ft + lah * qt) - ev.u2 * v0, w3 = (fw + lah * qw) - ev.u3 * v0;
                    if (s > 0) { p2[s - 1] = w2 - cp2; p3[s - 1] = w3 - cp3; }
                    if (s == 2) { out[0] = w2; out[OP] = w3; }
                    cp2 = w2; cp3 = w3;
                }
                if (s > 0) {
                    const R v0 = f0 - lah * q0;
                    const R w2 = (ft - lah * qt) - ev.u2 * v0, w3 = (fw - lah * qw) - ev.u3 * v0;
                    if (s > 1) { m2[5 - s] = cm2 - w2; m3[5 - s] = cm3 - w3; }
                    if (s == 3) { out[0] += w2; out[OP] += w3; }
                    cm2 = w2; cm3 = w3;
                }
            }
            g[2] = s6 * weno_pair<R, VER, P2>(p2, m2, eps4, pw) + out[0];
            g[3] = s6 * weno_pair<R, VER, P2>(p3, m3, eps4, pw) + out[OP];
        }
        Euler::Face<R> er = ev;
        er.c = out[3 * OP];
        er.h = out[4 * OP];
        Euler::right(er, g, fh);
    }
    // Back to (rho, rho u, rho v, rho w, E) and store.
    const R o[MEQN] = {fh[0], fh[CN], fh[CT], fh[3], fh[4]};
#pragma unroll
    for (int m = 0; m < MEQN; m++) out[m * OP] = o[m];
    if (FG) {
        double* const fo = ISX ? a.flux_x : a.flux_y;
        const int ni = a.mx + (ISX ? 1 : 0), nj = a.my + (ISX ? 0 : 1);
        if (fo && gi < ni && gj < nj) {
#pragma unroll
            for (int m = 0; m < MEQN; m++) fo[(size_t(m) * ni + gi) * nj + gj] = double(o[m]);
        }
    }
#undef gamma
#undef eps
#undef pw
    return alpha;
}

// One tile (rows i0 .., columns j0 ..) of a stage; the whole CTA takes part.
template <class R, int VER, bool P2, class Cfg, bool FG = false, int ORDER = 5>
__device__ __forceinline__ void stage_tile(const StageArgs& a, const int i0, const int j0)
{
    constexpr int TI = Cfg::TI, TJ = Cfg::TJ, NT = Cfg::NT, H = Cfg::H;
    constexpr int RI = Cfg::RI, RJ = Cfg::RJ;
    constexpr int PQ = RI * RJ;                    // plane size of qs and prim
    constexpr int FS = Cfg::template FSJ<R>();
    extern __shared__ __align__(128) unsigned char smem_raw[];
    const StageSmem<R, Cfg> S(smem_raw);

    const int tid = threadIdx.x;
    const int mx = a.mx, my = a.my;
    // The stage operand other than q_in (FP64: copied to shared memory behind
    // the face phase; q_in's own interior values are already there).
    const double* const ext = (a.A && a.A != a.qin) ? a.A : ((a.B && a.B != a.qin) ? a.B : nullptr);
    constexpr bool OPND = sizeof(R) == 8;
    if (OPND && ext && !(FG && a.flux_only)) {
        for (int c = tid; c < TI * TJ; c += NT) {
            const int ci = c / TJ, gi = i0 + ci, gj = j0 + (c - ci * TJ);
            if (gi < mx && gj < my) {
                const double* src = ext + size_t(gi) * my + gj;
                const unsigned dst = unsigned(__cvta_generic_to_shared(S.opnd + c));
#pragma unroll
                for (int m = 0; m < MEQN; m++)
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst + m * TI * TJ * 8), "l"(src + m * a.plane));
            }
        }
    }

    // ---- phase 1: load the tile + halo, boundary conditions by remap, and per
    // cell of the cross region FluxFunc (FluxFunc.cpp:19-42, once per cell
    // instead of once per stencil point of every face), halved for the LLF
    // split, and the cell's u, v, p, c for SetWaveSpd.cpp:24-50 ----
    // FP64: all of a thread's loads are issued before its arithmetic (one
    // memory round trip per tile, not one per pass over the region).  FP32
    // (3 CTAs per SM, whose register budget it tightens) keeps one pass at a
    // time.
    {
        constexpr int NIT = (PQ + NT - 1) / NT;
        constexpr int NV = sizeof(R) == 8 ? NIT : 1;
        auto in_cross = [&](int e, int& ii, int& jj) {
            ii = e / RJ;
            jj = e - ii * RJ;
            return e < PQ && ((ii >= H && ii < H + TI) || (jj >= H && jj < H + TJ));
        };
        auto load = [&](int e, R* v) {
            int ii, jj;
            if (!in_cross(e, ii, jj)) return;
            const int gi = bc_remap(i0 + ii - H, mx, a.bc[0], a.bc[1]);
            const int gj = bc_remap(j0 + jj - H, my, a.bc[2], a.bc[3]);
            const size_t g = size_t(gi) * my + gj;
#pragma unroll
            for (int m = 0; m < MEQN; m++) v[m] = R(ld_dep(a.qin + m * a.plane + g));
        };
        auto cell = [&](int e, const R* v) {
            int ii, jj;
            if (!in_cross(e, ii, jj)) return;
            const bool xin = ii >= H && ii < H + TI, yin = jj >= H && jj < H + TJ;
            const R gam = Par<R>::gamma(a);
#pragma unroll
            for (int m = 0; m < MEQN; m++) S.qs[m * PQ + e] = v[m];
            const R rho = v[0], m1 = v[1], m2 = v[2], m3 = v[3], en = v[4];
            const R ir = rcp(rho);
            const R u1 = m1 * ir, u2 = m2 * ir, u3 = m3 * ir;
            const R press = (gam - R(1)) * (en - R(0.5) * rho * (u1 * u1 + u2 * u2 + u3 * u3));
            S.prim[e] = u1;
            S.prim[PQ + e] = u2;
            S.prim[2 * PQ + e] = press;
            S.prim[3 * PQ + e] = sqrt_fast(fabs(gam * press * ir));
            if (FG) {
                // 0.5 * F, 0.5 * G of the integrated-flux kernel, unremapped: it
                // covers the 3-cell ghost frame; cells of a partial tile beyond it
                // only feed discarded faces, so their index is clamped.
                int ci = i0 + ii - H, cj = j0 + jj - H;
                ci = ci < -3 ? -3 : (ci > mx + 2 ? mx + 2 : ci);
                cj = cj < -3 ? -3 : (cj > my + 2 ? my + 2 : cj);
                const size_t o = size_t(ci + 3) * (my + 6) + (cj + 3);
                if (yin) {
                    const int d = ii * FS + (jj - H);
#pragma unroll
                    for (int m = 0; m < MEQN; m++) S.fs[m * RI * FS + d] = R(0.5 * ld_dep(a.Fg + m * a.gplane + o));
                }
                if (xin) {
                    const int d = (ii - H) * RJ + jj;
#pragma unroll
                    for (int m = 0; m < MEQN; m++) S.gs[m * TI * RJ + d] = R(0.5 * ld_dep(a.Gg + m * a.gplane + o));
                }
                return;
            }
            const R hr = R(0.5) * rho, hep = R(0.5) * (en + press);
            if (yin) {
                const int o = ii * FS + (jj - H);
                S.fs[o] = hr * u1;
                S.fs[RI * FS + o] = hr * u1 * u1 + R(0.5) * press;
                S.fs[2 * RI * FS + o] = hr * u1 * u2;
                S.fs[3 * RI * FS + o] = hr * u1 * u3;
                S.fs[4 * RI * FS + o] = u1 * hep;
            }
            if (xin) {
                const int o = (ii - H) * RJ + jj;
                S.gs[o] = hr * u2;
                S.gs[TI * RJ + o] = hr * u2 * u1;
                S.gs[2 * TI * RJ + o] = hr * u2 * u2 + R(0.5) * press;
                S.gs[3 * TI * RJ + o] = hr * u2 * u3;
                S.gs[4 * TI * RJ + o] = u2 * hep;
            }
        };
        R v[NV][MEQN];
        if constexpr (NV > 1) {
#pragma unroll
            for (int it = 0; it < NIT; it++) load(tid + it * NT, v[it]);
#pragma unroll
            for (int it = 0; it < NIT; it++) cell(tid + it * NT, v[it]);
        } else {
            for (int e = tid; e < PQ; e += NT) {
                load(e, v[0]);
                cell(e, v[0]);
            }
        }
    }
    __syncthreads();

    // ---- phase 2: one thread per face, x faces then y faces ----
    R smax_x = R(0), smax_y = R(0);
    bool neg = false, nonfinite = false;
    {
        const R ag1 = a.alpha_in ? R(a.alpha_in[0]) : R(0);
        const R ag2 = a.alpha_in ? R(a.alpha_in[1]) : R(0);
        auto face_x = [&](int k) {
            bool in_cfl;
            const R al = stage_face<R, VER, P2, Cfg, FG, true, ORDER>(a, S, k, i0, j0, ag1, neg, in_cfl);
            if (!(al <= R(1e30))) nonfinite = true;
            else if (in_cfl) smax_x = MaxN(smax_x, al);
        };
        auto face_y = [&](int k) {
            bool in_cfl;
            const R al = stage_face<R, VER, P2, Cfg, FG, false, ORDER>(a, S, k, i0, j0, ag2, neg, in_cfl);
            if (!(al <= R(1e30))) nonfinite = true;
            else if (in_cfl) smax_y = MaxN(smax_y, al);
        };
        if constexpr (Cfg::ONE_ROUND) {
            // a thread for every face of the tile, both directions at once
            static_assert(Cfg::NFX % 32 == 0, "a warp's faces share their direction");
            if (tid < Cfg::NFX) face_x(tid);
            else if (tid < Cfg::NFX + Cfg::NFY) face_y(tid - Cfg::NFX);
        } else {
#pragma unroll 1
            for (int k = tid; k < Cfg::NFX; k += NT) face_x(k);
#pragma unroll 1
            for (int k = tid; k < Cfg::NFY; k += NT) face_y(k);
        }
    }
    if (OPND) asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();

    // ---- phase 3: flux difference, stage update, next-stage wave speed ----
    R cs_x = R(0), cs_y = R(0);
    const double gam = a.gamma;
    for (int c = tid; c < ((FG && a.flux_only) ? 0 : TI * TJ); c += NT) {
        const int ci = c / TJ, cj = c - ci * TJ;
        const int gi = i0 + ci, gj = j0 + cj;
        if (gi >= mx || gj >= my) continue;
        const size_t g = size_t(gi) * my + gj;
        // every operand load ahead of the first store: qout may alias A or
        // B as far as the compiler knows, so loads interleaved with the
        // stores would wait one memory round trip per component
        double va[MEQN], vb[MEQN];
        if constexpr (OPND) {
            const R* const qc = S.qs + (H + ci) * RJ + (H + cj);
#pragma unroll
            for (int m = 0; m < MEQN; m++) {
                const double own = qc[m * PQ], oth = ext ? S.opnd[m * TI * TJ + c] : 0.0;
                va[m] = a.A == a.qin ? own : oth;
                // A and B apart from each other and from q_in: B is not staged
                vb[m] = a.B == a.qin ? own : (a.B == ext ? oth : (a.B ? a.B[m * a.plane + g] : 0.0));
            }
        } else {
#pragma unroll
            for (int m = 0; m < MEQN; m++) {
                va[m] = a.A ? a.A[m * a.plane + g] : 0.0;
                vb[m] = a.B ? a.B[m * a.plane + g] : 0.0;
            }
        }
        double qn[MEQN];
#pragma unroll
        for (int m = 0; m < MEQN; m++) {
            // ConstructL.cpp:396-398
            // (the FP32 forms difference their FP32 fluxes in FP32 and widen
            // the result once)
            const R f1 = S.Fh[m * (TI + 1) * TJ + (ci + 1) * TJ + cj], f0 = S.Fh[m * (TI + 1) * TJ + ci * TJ + cj];
            const R g1 = S.Gh[m * TI * (TJ + 1) + ci * (TJ + 1) + cj + 1], g0 = S.Gh[m * TI * (TJ + 1) + ci * (TJ + 1) + cj];
            R Lr = -(f1 - f0) * R(a.rdx);
            Lr = Lr - (g1 - g0) * R(a.rdy);
            const double L = double(Lr);
            double v = 0.0;
            {
                if (a.A) v = a.a1 * va[m];
                if (a.B) v = v + a.a2 * vb[m];
            }
            v = v + a.bdt * L;
            qn[m] = v;
            a.qout[m * a.plane + g] = v;
        }
        if (a.alpha_out) {
            // GlobalWaveSpd.cpp:71-76 on the new state, both directions:
            // max(|u_n - c|, |u_n + c|) = |u_n| + c.  The FP32 forms use it
            // only as the FP32 LLF speed of the next stage, so they evaluate
            // it in FP32.
            const R qx[MEQN] = {R(qn[0]), R(qn[1]), R(qn[2]), R(qn[3]), R(qn[4])};
            const typename Euler::Cell<R> w = Euler::cell(R(gam), qx);
            const R sx = fabs(w.un) + w.c, sy = fabs(qx[2] * rcp(qx[0])) + w.c;
            const R big = sizeof(R) == 8 ? R(1e300) : R(3e38f);
            if (!(sx <= big) || !(sy <= big)) nonfinite = true;
            if (sx <= big) cs_x = MaxN(cs_x, sx);
            if (sy <= big) cs_y = MaxN(cs_y, sy);
        }
    }

    // ---- block reductions of the four maxima, one atomic each ----
    // Non-finite speeds were flagged per value above (a NaN does not survive
    // Max(NaN, b) = b), so the reduction only sees finite ones.
    const R v4[4] = {smax_x, smax_y, cs_x, cs_y};
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const double v = double(warp_max_nonneg(v4[k]));
        if ((tid & 31) == 0) S.red[(tid >> 5) * 4 + k] = v;
    }
    if (neg) atomicOr(a.status, 2u);
    if (nonfinite) atomicOr(a.status, 1u);
    __syncthreads();
    if (tid < 4) {
        double v = 0.0;
        for (int wv = 0; wv < NT / 32; wv++) v = Max(v, S.red[wv * 4 + tid]);
        double* dst = tid < 2 ? a.smax_out : a.alpha_out;
        if (dst) atomic_max_nonneg(dst + (tid & 1), v);
    }
}

// LONG: rows of tiles in blockIdx.y and .z (tile_grid), for grids of more than
// 65,535 rows of tiles; a kernel of its own, as the row's index costs a register
// that the orders above 5 have not got (WENO7-JS 1.477 -> 1.543 ms, two steps
// at 1024^2).
template <class R, int VER, bool P2, class Cfg, bool FG = false, int ORDER = 5, bool LONG = false>
__global__ void __launch_bounds__(Cfg::NT, MinBlocks<R>::value * 256 / Cfg::NT) k_stage(const __grid_constant__ StageArgs a)
{
    grid_dependency();
    static_assert(ORDER == 5 ? Cfg::H == 3 : Cfg::H == (ORDER + 1) / 2 && sizeof(R) == 8 && !FG, "halo of the stencil");
    stage_tile<R, VER, P2, Cfg, FG, ORDER>(a, (LONG ? tile_row() : int(blockIdx.y)) * Cfg::TI, blockIdx.x * Cfg::TJ);
}

// GlobalWaveSpd (lib/2d/GlobalWaveSpd.cpp:52-78) on a state already in HBM:
// grid-stride over interior cells, block max, one atomicMax per block.
__global__ void k_wave_spd_max(const double* q, int mx, int my, size_t plane, double gamma,
                               double* alpha_out, unsigned int* status);

// Reference ghosted AoS (i, j, m) <-> device planes.
__global__ void k_aos_to_planes(const double* aos, double* planes, int mx, int my, int mbc, size_t plane);
__global__ void k_planes_to_aos(const double* planes, double* aos, int mx, int my, int mbc, size_t plane,
                                int bc0, int bc1, int bc2, int bc3);

}  // namespace fin
