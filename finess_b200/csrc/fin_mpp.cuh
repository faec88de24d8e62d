// The maximum-principle-preserving (positivity) limiter of the Lax-Wendroff
// step, FinSolveLxW.cpp:126-158: the high-order face fluxes fhat, ghat of
// ConstructLxWL (written by the stage kernel in its flux-only mode), the
// Lax-Friedrichs fluxes of ConstructLFL.cpp:92-108, ApplyMPPLimiter2D
// (apps/2d/euler/lib/ApplyMPPLimiter2D.cpp:27-285) and the conservative
// update of FinSolveLxW.cpp:143-151.
//
// Two kernels, one thread per cell of a 16 x 16 tile whose states and fluxes
// sit in shared memory (each cell's three divisions once, not once per face
// and component: the update kernel 0.130 -> 0.071 ms at 1023 x 1025; both are
// now bound by the latency of their flux loads); launched while their predecessor
// ends, which takes two steps at 64 x 80 from 92 to 85 us, 1023 x 1025 836 -> 826:
//   k_mpp_limit   the cell's four limiting factors amin[k] (k = left, right,
//                 bottom, top face): the density step (:57-92) and the
//                 pressure step over the 16 on/off combinations of the faces
//                 with its 9-step bisection (:97-217);
//   k_mpp_update  the face factors theta = min of the two cells' (one-sided
//                 at the domain boundary, :222-243), the limited fluxes
//                 theta (fhat - fLF) + fLF (:248-270), the update, and the
//                 new state's global wave speeds (GlobalWaveSpd.cpp:71-76).
// The Lax-Friedrichs fluxes are recomputed where needed (cheap) instead of
// stored.  Every operation that enters a result follows the reference's order with correctly
// rounded IEEE operations (no contraction), so equal inputs give equal
// results.
#pragma once
#include "fin_stage.cuh"

namespace fin {
namespace mpp {

__device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double sub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double dvd(double a, double b) { return __ddiv_rn(a, b); }
// dog_math.h:18-22
__device__ __forceinline__ double Mn(double a, double b) { return a < b ? a : b; }

struct MppArgs {
    const double* q;      // q^n planes
    double* qout;         // q^{n+1} planes
    size_t plane;
    int mx, my;
    int bc[4];
    const double* fhat;   // [m][mx+1][my]  high-order x-face fluxes (face i between cells i-1, i)
    const double* ghat;   // [m][mx][my+1]  high-order y-face fluxes
    double* amin;         // [4][mx][my]
    const double* alpha;  // [2] global wave speeds of q^n (GlobalWaveSpd, ConstructLFL.cpp:62-65)
    double dt, dx, dy, gamma;
    double* alpha_out;    // [2] GlobalWaveSpd of q^{n+1}
    unsigned int* status; // bit 0: non-finite wave speed of q^{n+1}
};

// A block's TI x TJ cells with one cell around them: states and fluxes
// (FluxFunc.cpp:19-42) of the cross region, each evaluated once.  The f and g
// arrays hold the rows (columns) that the tile's x (y) faces read.
constexpr int TI = 16, TJ = 16, NT = TI * TJ, CI = TI + 2, CJ = TJ + 2;
struct Tile {
    double q[MEQN][CI][CJ];
    double f[MEQN][CI][TJ];
    double g[MEQN][TI][CJ];
};

__device__ __forceinline__ void load_tile(const MppArgs& a, Tile& T, int i0, int j0)
{
    for (int e = threadIdx.x; e < CI * CJ; e += NT) {
        const int ii = e / CJ, jj = e - ii * CJ;
        const bool xin = ii >= 1 && ii <= TI, yin = jj >= 1 && jj <= TJ;
        if (!xin && !yin) continue;
        const size_t o = size_t(bc_remap(i0 + ii - 1, a.mx, a.bc[0], a.bc[1])) * a.my +
                         bc_remap(j0 + jj - 1, a.my, a.bc[2], a.bc[3]);
        double Q[MEQN];
#pragma unroll
        for (int m = 0; m < MEQN; m++) {
            Q[m] = a.q[m * a.plane + o];
            T.q[m][ii][jj] = Q[m];
        }
        const double rho = Q[0];
        const double u1 = dvd(Q[1], rho), u2 = dvd(Q[2], rho), u3 = dvd(Q[3], rho);
        const double energy = Q[4];
        const double ke = add(add(mul(u1, u1), mul(u2, u2)), mul(u3, u3));
        const double press = mul(sub(a.gamma, 1.0e0), sub(energy, mul(mul(0.5e0, rho), ke)));
        if (yin) {
            const int c = jj - 1;
            T.f[0][ii][c] = mul(rho, u1);
            T.f[1][ii][c] = add(mul(mul(rho, u1), u1), press);
            T.f[2][ii][c] = mul(mul(rho, u1), u2);
            T.f[3][ii][c] = mul(mul(rho, u1), u3);
            T.f[4][ii][c] = mul(u1, add(energy, press));
        }
        if (xin) {
            const int r = ii - 1;
            T.g[0][r][jj] = mul(rho, u2);
            T.g[1][r][jj] = mul(mul(rho, u2), u1);
            T.g[2][r][jj] = add(mul(mul(rho, u2), u2), press);
            T.g[3][r][jj] = mul(mul(rho, u2), u3);
            T.g[4][r][jj] = mul(u2, add(energy, press));
        }
    }
}

// Lax-Friedrichs flux of the face between cells L and R, one component
// (ConstructLFL.cpp:92-108): 0.5 (f(L) + f(R)) + 0.5 alpha (q_L - q_R).
__device__ __forceinline__ double lf(double fL, double fR, double qL, double qR, double alpha)
{
    return add(mul(0.5, add(fL, fR)), mul(mul(0.5, alpha), sub(qL, qR)));
}

// The four faces of tile cell (ci, cj), component m: high-order and
// Lax-Friedrichs fluxes (k = 0: x face i, 1: x face i+1, 2: y face j, 3: y
// face j+1).
__device__ __forceinline__ void cell_faces(const MppArgs& a, const Tile& T, int i, int j, int ci, int cj, int m,
                                           double ax, double ay, double (&fh)[4], double (&fl)[4])
{
    const double qc = T.q[m][ci + 1][cj + 1];
    fl[0] = lf(T.f[m][ci][cj], T.f[m][ci + 1][cj], T.q[m][ci][cj + 1], qc, ax);
    fl[1] = lf(T.f[m][ci + 1][cj], T.f[m][ci + 2][cj], qc, T.q[m][ci + 2][cj + 1], ax);
    fl[2] = lf(T.g[m][ci][cj], T.g[m][ci][cj + 1], T.q[m][ci + 1][cj], qc, ay);
    fl[3] = lf(T.g[m][ci][cj + 1], T.g[m][ci][cj + 2], qc, T.q[m][ci + 1][cj + 2], ay);
    const int mx = a.mx, my = a.my;
    fh[0] = a.fhat[(size_t(m) * (mx + 1) + i) * my + j];
    fh[1] = a.fhat[(size_t(m) * (mx + 1) + i + 1) * my + j];
    fh[2] = a.ghat[(size_t(m) * mx + i) * (my + 1) + j];
    fh[3] = a.ghat[(size_t(m) * mx + i) * (my + 1) + j + 1];
}

// Pressure of a state, ApplyMPPLimiter2D.cpp:108-113.
__device__ __forceinline__ double pressure(const double* Q, double gm1)
{
    const double rho = Q[0];
    const double u1 = dvd(Q[1], rho), u2 = dvd(Q[2], rho), u3 = dvd(Q[3], rho);
    const double ke = add(add(mul(u1, u1), mul(u2, u2)), mul(u3, u3));
    return mul(gm1, sub(Q[4], mul(mul(0.5, rho), ke)));
}

// The pressure step's rescaling factors, ApplyMPPLimiter2D.cpp:97-217: for
// each of the 16 on/off combinations of the faces the state with those faces'
// (density-limited) high-order fluxes, bisected against the Lax-Friedrichs
// state when its pressure is negative.  Run by the cells whose states
// k_mpp_limit could not show to be positive.
__device__ __noinline__ void pressure_step(const MppArgs& a, const Tile& T, int i, int j, int ci, int cj, double dtx,
                                           double dty, const double* amin, double* rescale2)
{
    const double ax = a.alpha[0], ay = a.alpha[1], gm1 = sub(a.gamma, 1.0);
    double fh[4 * MEQN], fl[4 * MEQN], qc[MEQN], qlf[MEQN];
#pragma unroll
    for (int m = 0; m < MEQN; m++) {
        double h[4], l[4];
        cell_faces(a, T, i, j, ci, cj, m, ax, ay, h, l);
#pragma unroll
        for (int k = 0; k < 4; k++) {
            fh[k * MEQN + m] = h[k];
            fl[k * MEQN + m] = l[k];
        }
        qc[m] = T.q[m][ci + 1][cj + 1];
        qlf[m] = add(add(qc[m], mul(dtx, sub(l[0], l[1]))), mul(dty, sub(l[2], l[3])));
    }
    if (pressure(qlf, gm1) < 0.0) atomicOr(a.status, 2u);   // "Negative solution in Lax-Friedrich's flux"
#pragma unroll 1
    for (int combo = 0; combo < 16; combo++) {
        // combo bits (i1 i2 i3 i4) with i1 the most significant, as the
        // reference's nested loops enumerate them
        const int on[4] = {(combo >> 3) & 1, (combo >> 2) & 1, (combo >> 1) & 1, combo & 1};
        double aa[4], qh[MEQN];
#pragma unroll
        for (int k = 0; k < 4; k++) aa[k] = mul(double(on[k]), amin[k]);
#pragma unroll
        for (int m = 0; m < MEQN; m++) {
            double f4[4];
#pragma unroll
            for (int k = 0; k < 4; k++) f4[k] = add(mul(aa[k], fh[k * MEQN + m]), mul(sub(1.0, aa[k]), fl[k * MEQN + m]));
            qh[m] = add(add(qc[m], mul(dtx, sub(f4[0], f4[1]))), mul(dty, sub(f4[2], f4[3])));
        }
        double phigh = pressure(qh, gm1);
        if (phigh < 0.0) {
            double root1 = 0.0, root2 = 1.0, rate = 0.0;
#pragma unroll 1
            for (int nn = 1; nn < 10; nn++) {
                rate = mul(add(root1, root2), 0.5);
                double q2[MEQN];
#pragma unroll
                for (int m = 0; m < MEQN; m++) q2[m] = add(mul(rate, qh[m]), mul(sub(1.0, rate), qlf[m]));
                phigh = pressure(q2, gm1);
                if (phigh < 0.0) root2 = rate;
                else root1 = rate;
            }
            const double r = phigh > 0.0 ? rate : root1;
            // :220-227: each face's factor is the least over the combinations it is on in
#pragma unroll
            for (int k = 0; k < 4; k++)
                if (on[k]) rescale2[k] = Mn(rescale2[k], r);
        }
    }
}

// The cell's four factors.  Bound by memory (fluxes and states once); the
// pressure step's 16 candidate states a cell, each with three correctly
// rounded divisions, took 0.33 ms at 1023 x 1025 when every cell ran them,
// against 0.078 ms with the test below that all sixteen are positive.
//
// Every candidate is q_LF plus a subset of the faces' contributions d_k =
// +-amin_k dt/dx (fhat_k - fLF_k), so its components lie within mid +- rad,
// mid = q_LF + sum d_k / 2, rad = sum |d_k| / 2.  With rad widened by 1e-13 of
// the sum of the magnitudes that enter (a thousand roundings), rho_min > 0
// and 2 rho_min E_min > (1 + 1e-11) max |m|^2 mean that the pressure the
// reference's formula computes for each candidate is not negative, so every
// rescaling factor is 1 and no candidate need be formed: the same factors bit
// for bit.  Cells that fail the test (near-vacuum ones) take pressure_step.
__global__ void __launch_bounds__(NT, 4) k_mpp_limit(const MppArgs a)
{
    grid_dependency();
    __shared__ Tile T;
    const int mx = a.mx, my = a.my;
    const int i0 = int(blockIdx.y) * TI, j0 = int(blockIdx.x) * TJ;
    load_tile(a, T, i0, j0);
    __syncthreads();
    const int ci = threadIdx.x / TJ, cj = threadIdx.x - ci * TJ;
    const int i = i0 + ci, j = j0 + cj;
    if (i >= mx || j >= my) return;
    const double ax = a.alpha[0], ay = a.alpha[1];
    const double eps = 1.0e-12, rho_min = eps;
    const double dtx = dvd(a.dt, a.dx), dty = dvd(a.dt, a.dy);
    // component m's bounds over the candidates, from its faces' fluxes
    double amin[4];
    auto bounds = [&](int m, const double (&fh)[4], const double (&fl)[4], double& mid, double& rad) {
        const double qc = T.q[m][ci + 1][cj + 1];
        const double d0 = amin[0] * dtx * (fh[0] - fl[0]), d1 = amin[1] * dtx * (fl[1] - fh[1]);
        const double d2 = amin[2] * dty * (fh[2] - fl[2]), d3 = amin[3] * dty * (fl[3] - fh[3]);
        mid = qc + dtx * (fl[0] - fl[1]) + dty * (fl[2] - fl[3]) + 0.5 * ((d0 + d1) + (d2 + d3));
        const double mag = fabs(qc) + dtx * ((fabs(fl[0]) + fabs(fl[1])) + (fabs(fh[0]) + fabs(fh[1]))) +
                           dty * ((fabs(fl[2]) + fabs(fl[3])) + (fabs(fh[2]) + fabs(fh[3])));
        rad = 0.5 * ((fabs(d0) + fabs(d1)) + (fabs(d2) + fabs(d3))) + 1e-13 * mag;
    };
    double rmin, ratio;
    {
        double fh[4], fl[4];
        cell_faces(a, T, i, j, ci, cj, 0, ax, ay, fh, fl);
        // ---- step 1: density (:57-92) ----
        const double gmin = sub(rho_min, add(add(T.q[0][ci + 1][cj + 1], mul(dtx, sub(fl[0], fl[1]))),
                                             mul(dty, sub(fl[2], fl[3]))));
        double ff[4];
        ff[0] = mul(dtx, sub(fh[0], fl[0]));
        ff[1] = mul(-dtx, sub(fh[1], fl[1]));
        ff[2] = mul(dty, sub(fh[2], fl[2]));
        ff[3] = mul(-dty, sub(fh[3], fl[3]));
        int isgn[4];
#pragma unroll
        for (int k = 0; k < 4; k++) isgn[k] = ff[k] < 0.0 ? 1 : 0;
        double ffsum = mul(double(isgn[0]), ff[0]);
#pragma unroll
        for (int k = 1; k < 4; k++) ffsum = add(ffsum, mul(double(isgn[k]), ff[k]));
        // gmin / (ffsum - eps) with a negative denominator: at least 1, and so
        // cut to 1, exactly when gmin does not exceed it
        const double den = sub(ffsum, eps);
        ratio = gmin <= den && den < 0.0 ? 1.0 : Mn(dvd(gmin, den), 1.e0);
#pragma unroll
        for (int k = 0; k < 4; k++) amin[k] = isgn[k] == 1 ? ratio : 1.e0;
        double mid, rad;
        bounds(0, fh, fl, mid, rad);
        rmin = mid - rad;
    }
    // ---- step 2: pressure (:97-217) ----
    double m2 = 0.0, emin = 0.0;
#pragma unroll 1
    for (int m = 1; m < MEQN; m++) {
        double fh[4], fl[4], mid, rad;
        cell_faces(a, T, i, j, ci, cj, m, ax, ay, fh, fl);
        bounds(m, fh, fl, mid, rad);
        const double w = fabs(mid) + rad;
        if (m < 4) m2 += w * w;
        else emin = mid - rad;
    }
    const bool positive = rmin > 0.0 && 2.0 * rmin * emin > (1.0 + 1e-11) * m2 && ratio >= 0.0;
    double rescale2[4] = {1.0, 1.0, 1.0, 1.0};
    if (!positive) pressure_step(a, T, i, j, ci, cj, dtx, dty, amin, rescale2);
    const size_t nc = size_t(mx) * my, c = size_t(i) * my + j;
#pragma unroll
    for (int k = 0; k < 4; k++) a.amin[k * nc + c] = mul(rescale2[k], amin[k]);
}

__global__ void __launch_bounds__(NT) k_mpp_update(const MppArgs a)
{
    grid_dependency();
    __shared__ Tile T;
    __shared__ double red[2][NT / 32];
    const int mx = a.mx, my = a.my;
    const int i0 = int(blockIdx.y) * TI, j0 = int(blockIdx.x) * TJ;
    load_tile(a, T, i0, j0);
    __syncthreads();
    const int ci = threadIdx.x / TJ, cj = threadIdx.x - ci * TJ;
    const int i = i0 + ci, j = j0 + cj;
    double sx = 0.0, sy = 0.0;
    bool nonfinite = false;
    if (i < mx && j < my) {
        const size_t nc = size_t(mx) * my, c = size_t(i) * my + j;
        // face factors (:222-243): min of the two cells' entries, the
        // cell's own at the domain boundary
        const double* am = a.amin;
        double th[4];
        th[0] = i > 0 ? Mn(am[0 * nc + c], am[1 * nc + (c - my)]) : am[0 * nc + c];
        th[1] = i < mx - 1 ? Mn(am[0 * nc + (c + my)], am[1 * nc + c]) : am[1 * nc + c];
        th[2] = j > 0 ? Mn(am[2 * nc + c], am[3 * nc + (c - 1)]) : am[2 * nc + c];
        th[3] = j < my - 1 ? Mn(am[2 * nc + (c + 1)], am[3 * nc + c]) : am[3 * nc + c];
        const double dtdx = dvd(a.dt, a.dx), dtdy = dvd(a.dt, a.dy);
        const double ax = a.alpha[0], ay = a.alpha[1];
        double qn[MEQN];
#pragma unroll
        for (int m = 0; m < MEQN; m++) {
            double fh[4], fl[4], f[4];
            cell_faces(a, T, i, j, ci, cj, m, ax, ay, fh, fl);
#pragma unroll
            for (int k = 0; k < 4; k++) f[k] = add(mul(th[k], sub(fh[k], fl[k])), fl[k]);
            // FinSolveLxW.cpp:145-148
            double v = sub(T.q[m][ci + 1][cj + 1], mul(dtdx, sub(f[1], f[0])));
            v = sub(v, mul(dtdy, sub(f[3], f[2])));
            qn[m] = v;
            a.qout[m * a.plane + c] = v;
        }
        // GlobalWaveSpd.cpp:71-76 on the new state
        const double rho = qn[0];
        const double u1 = dvd(qn[1], rho), u2 = dvd(qn[2], rho), u3 = dvd(qn[3], rho);
        const double ke = add(add(mul(u1, u1), mul(u2, u2)), mul(u3, u3));
        const double press = mul(sub(a.gamma, 1.0), sub(qn[4], mul(mul(0.5, rho), ke)));
        const double cs = sqrt(fabs(dvd(mul(a.gamma, press), rho)));
        sx = add(fabs(u1), cs);
        sy = add(fabs(u2), cs);
        if (!(sx <= 1e300) || !(sy <= 1e300)) nonfinite = true;
        if (!(sx <= 1e300)) sx = 0.0;
        if (!(sy <= 1e300)) sy = 0.0;
    }
    for (int o = 16; o > 0; o >>= 1) {
        sx = Max(sx, __shfl_xor_sync(0xffffffffu, sx, o));
        sy = Max(sy, __shfl_xor_sync(0xffffffffu, sy, o));
    }
    if ((threadIdx.x & 31) == 0) {
        red[0][threadIdx.x >> 5] = sx;
        red[1][threadIdx.x >> 5] = sy;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < NT / 32; w++) {
            sx = Max(sx, red[0][w]);
            sy = Max(sy, red[1][w]);
        }
        if (a.alpha_out) {
            atomic_max_nonneg(a.alpha_out, sx);
            atomic_max_nonneg(a.alpha_out + 1, sy);
        }
    }
    if (nonfinite) atomicOr(a.status, 1u);
}

}  // namespace mpp
}  // namespace fin
