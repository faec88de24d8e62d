// WENO reconstructions of the orders other than 5 that ConstructL accepts
// (space_order 1, 7, 9, 11; lib/WenoReconstruct.cpp:151-375, 440-575, 618-695),
// on the first differences of the stencil.
//
// The method is defined by its numbers: candidate-stencil weights, linear
// weights and the smoothness-indicator polynomials of Balsara & Shu (J. Comput.
// Phys. 160, 2000).  The indicators are quadratic forms that vanish on
// constants, so each equals a form in the r - 1 differences of its candidate's
// points with integer coefficients again, and each candidate is u_i plus a
// combination of differences; both are written so here (exactly: the same
// rational numbers).  That takes 9, 14, 20 operations an indicator (orders 7,
// 9, 11) instead of 16, 25, 36, and removes the cancellation of coefficients
// up to 4e8 between nearly equal point values.
#pragma once
#include "fin_device.cuh"

namespace fin {
namespace hi {

// forms: x_k = eps + beta_k; values: candidate k minus u_i; weight: the linear
// weights up to a factor; d[t] = u_(t+1) - u_t of the 2r - 1 points.
template <int ORDER> struct Scheme;
template <> struct Scheme<7> {
    __device__ __forceinline__ static void forms(const double* d, double eps, double* x)
    {
        x[0] = fma(d[0], fma(1854., d[2], fma(-2788., d[1], 547. * d[0])), fma(d[1],
            fma(-5188., d[2], 3708. * d[1]), fma(d[2], 2107. * d[2], eps)));
        x[1] = fma(d[1], fma(494., d[3], fma(-1108., d[2], 267. * d[1])), fma(d[2],
            fma(-1428., d[3], 1468. * d[2]), fma(d[3], 547. * d[3], eps)));
        x[2] = fma(d[2], fma(494., d[4], fma(-1428., d[3], 547. * d[2])), fma(d[3],
            fma(-1108., d[4], 1468. * d[3]), fma(d[4], 267. * d[4], eps)));
        x[3] = fma(d[3], fma(1854., d[5], fma(-5188., d[4], 2107. * d[3])), fma(d[4],
            fma(-2788., d[5], 3708. * d[4]), fma(d[5], 547. * d[5], eps)));
    }
    __device__ __forceinline__ static void values(const double* d, double* c)
    {
        c[0] = fma(13. / 12., d[2], fma(-5. / 6., d[1], (1. / 4.) * d[0]));
        c[1] = fma(1. / 4., d[3], fma(1. / 3., d[2], (-1. / 12.) * d[1]));
        c[2] = fma(-1. / 12., d[4], fma(1. / 2., d[3], (1. / 12.) * d[2]));
        c[3] = fma(1. / 12., d[5], fma(-1. / 3., d[4], (3. / 4.) * d[3]));
    }
    __device__ __forceinline__ static double weight(int k)
    {
        constexpr double g[4] = {1., 12., 18., 4.};
        return g[k];
    }
    __device__ __forceinline__ static double tau(const double* x) { return fabs(x[0] + 3. * (x[1] - x[2]) - x[3]); }
};
template <> struct Scheme<9> {
    __device__ __forceinline__ static void forms(const double* d, double eps, double* x)
    {
        x[0] = fma(d[0], fma(-86329., d[3], fma(201678., d[2], fma(-163185., d[1], 22658. * d[0]))), fma(d[1],
            fma(325158., d[3], fma(-745293., d[2], 297120. * d[1])), fma(d[2],
            fma(-433665., d[3], 478980. * d[2]), fma(d[3], 107918. * d[3], eps))));
        x[1] = fma(d[1], fma(-18079., d[4], fma(52158., d[3], fma(-47055., d[2], 6908. * d[1]))), fma(d[2],
            fma(70218., d[4], fma(-196563., d[3], 84600. * d[2])), fma(d[3],
            fma(-94935., d[4], 125130. * d[3]), fma(d[4], 22658. * d[4], eps))));
        x[2] = fma(d[2], fma(-8209., d[5], fma(30738., d[4], fma(-37185., d[3], 6908. * d[2]))), fma(d[3],
            fma(30738., d[5], fma(-109413., d[4], 60870. * d[3])), fma(d[4], fma(-37185., d[5], 60870. * d[4]),
            fma(d[5], 6908. * d[5], eps))));
        x[3] = fma(d[3], fma(-18079., d[6], fma(70218., d[5], fma(-94935., d[4], 22658. * d[3]))), fma(d[4],
            fma(52158., d[6], fma(-196563., d[5], 125130. * d[4])), fma(d[5],
            fma(-47055., d[6], 84600. * d[5]), fma(d[6], 6908. * d[6], eps))));
        x[4] = fma(d[4], fma(-86329., d[7], fma(325158., d[6], fma(-433665., d[5], 107918. * d[4]))), fma(d[5],
            fma(201678., d[7], fma(-745293., d[6], 478980. * d[5])), fma(d[6],
            fma(-163185., d[7], 297120. * d[6]), fma(d[7], 22658. * d[7], eps))));
    }
    __device__ __forceinline__ static void values(const double* d, double* c)
    {
        c[0] = fma(77. / 60., d[3], fma(-43. / 30., d[2], fma(17. / 20., d[1], (-1. / 5.) * d[0])));
        c[1] = fma(1. / 5., d[4], fma(29. / 60., d[3], fma(-7. / 30., d[2], (1. / 20.) * d[1])));
        c[2] = fma(-1. / 20., d[5], fma(2. / 5., d[4], fma(11. / 60., d[3], (-1. / 30.) * d[2])));
        c[3] = fma(1. / 30., d[6], fma(-11. / 60., d[5], fma(3. / 5., d[4], (1. / 20.) * d[3])));
        c[4] = fma(-1. / 20., d[7], fma(7. / 30., d[6], fma(-29. / 60., d[5], (4. / 5.) * d[4])));
    }
    __device__ __forceinline__ static double weight(int k)
    {
        constexpr double g[5] = {1., 20., 60., 40., 5.};
        return g[k];
    }
    __device__ __forceinline__ static double tau(const double* x) { return fabs(x[4] - x[0]); }
};
template <> struct Scheme<11> {
    __device__ __forceinline__ static void forms(const double* d, double eps, double* x)
    {
        x[0] = fma(d[0], fma(4712740., d[4], fma(-15121610., d[3], fma(18797194., d[2],
            fma(-10645062., d[1], 1152561. * d[0])))), fma(d[1], fma(-22347430., d[4], fma(71025008., d[3],
            fma(-87652660., d[2], 24683064. * d[1]))), fma(d[2], fma(41046694., d[4],
            fma(-128482540., d[3], 78421848. * d[2])), fma(d[3], fma(-35160042., d[4], 53540984. * d[3]),
            fma(d[4], 6150211. * d[4], eps)))));
        x[1] = fma(d[1], fma(880548., d[5], fma(-3186470., d[4], fma(4222438., d[3],
            fma(-2472170., d[2], 271779. * d[1])))), fma(d[2], fma(-4254026., d[5], fma(15189424., d[4],
            fma(-19806700., d[3], 5706008. * d[2]))), fma(d[3], fma(7929610., d[5],
            fma(-27680692., d[4], 17580984. * d[3])), fma(d[4], fma(-6812870., d[5], 11400536. * d[4]),
            fma(d[5], 1152561. * d[5], eps)))));
        x[2] = fma(d[2], fma(245620., d[6], fma(-1079386., d[5], fma(1713274., d[4],
            fma(-1150710., d[3], 139633. * d[2])))), fma(d[3], fma(-1213142., d[6], fma(5189840., d[5],
            fma(-7947412., d[4], 2534504. * d[3]))), fma(d[4], fma(2249110., d[6],
            fma(-9252940., d[5], 6713736. * d[4])), fma(d[5], fma(-1837242., d[6], 3544296. * d[5]),
            fma(d[6], 271779. * d[6], eps)))));
        x[3] = fma(d[3], fma(245620., d[7], fma(-1213142., d[6], fma(2249110., d[5],
            fma(-1837242., d[4], 271779. * d[3])))), fma(d[4], fma(-1079386., d[7], fma(5189840., d[6],
            fma(-9252940., d[5], 3544296. * d[4]))), fma(d[5], fma(1713274., d[7],
            fma(-7947412., d[6], 6713736. * d[5])), fma(d[6], fma(-1150710., d[7], 2534504. * d[6]),
            fma(d[7], 139633. * d[7], eps)))));
        x[4] = fma(d[4], fma(880548., d[8], fma(-4254026., d[7], fma(7929610., d[6],
            fma(-6812870., d[5], 1152561. * d[4])))), fma(d[5], fma(-3186470., d[8], fma(15189424., d[7],
            fma(-27680692., d[6], 11400536. * d[5]))), fma(d[6], fma(4222438., d[8],
            fma(-19806700., d[7], 17580984. * d[6])), fma(d[7], fma(-2472170., d[8], 5706008. * d[7]),
            fma(d[8], 271779. * d[8], eps)))));
        x[5] = fma(d[5], fma(4712740., d[9], fma(-22347430., d[8], fma(41046694., d[7],
            fma(-35160042., d[6], 6150211. * d[5])))), fma(d[6], fma(-15121610., d[9], fma(71025008., d[8],
            fma(-128482540., d[7], 53540984. * d[6]))), fma(d[7], fma(18797194., d[9],
            fma(-87652660., d[8], 78421848. * d[7])), fma(d[8], fma(-10645062., d[9], 24683064. * d[8]),
            fma(d[9], 1152561. * d[9], eps)))));
    }
    __device__ __forceinline__ static void values(const double* d, double* c)
    {
        c[0] = fma(29. / 20., d[4], fma(-21. / 10., d[3], fma(37. / 20., d[2],
            fma(-13. / 15., d[1], (1. / 6.) * d[0]))));
        c[1] = fma(1. / 6., d[5], fma(37. / 60., d[4], fma(-13. / 30., d[3],
            fma(11. / 60., d[2], (-1. / 30.) * d[1]))));
        c[2] = fma(-1. / 30., d[6], fma(1. / 3., d[5], fma(17. / 60., d[4],
            fma(-1. / 10., d[3], (1. / 60.) * d[2]))));
        c[3] = fma(1. / 60., d[7], fma(-7. / 60., d[6], fma(1. / 2., d[5],
            fma(7. / 60., d[4], (-1. / 60.) * d[3]))));
        c[4] = fma(-1. / 60., d[8], fma(1. / 10., d[7], fma(-17. / 60., d[6],
            fma(2. / 3., d[5], (1. / 30.) * d[4]))));
        c[5] = fma(1. / 30., d[9], fma(-11. / 60., d[8], fma(13. / 30., d[7],
            fma(-37. / 60., d[6], (5. / 6.) * d[5]))));
    }
    __device__ __forceinline__ static double weight(int k)
    {
        constexpr double g[6] = {1., 30., 150., 200., 75., 6.};
        return g[k];
    }
    __device__ __forceinline__ static double tau(const double* x) { return 0.; }   // no Z weights of this order
};

// Powers other than 2 (CALL: one copy of pow instead of one a weight; which
// is better where is measured at fin_hi.cu's launch_t).
static __device__ __noinline__ double pow_call(double x, double p) { return pow(x, p); }
template <bool CALL>
__device__ __forceinline__ double power(double x, double p)
{
    return CALL ? pow_call(x, p) : pow(x, p);
}

// The reconstruction of order ORDER minus its upwind point u_i.
template <int ORDER, int VER, bool P2, bool CALL>
__device__ __forceinline__ double correction(const double* d, double eps, double pw)
{
    static_assert(ORDER == 1 || ORDER == 7 || ORDER == 9 || ORDER == 11, "orders 1, 7, 9, 11");
    if constexpr (ORDER == 1) {
        return 0.0;   // WenoReconstructLLF, :686-695
    } else {
        constexpr int R = (ORDER + 1) / 2;
        using S = Scheme<ORDER>;
        double c[R], num = 0.0, den = 0.0;
        S::values(d, c);
        if constexpr (VER == FIN_WENO_FD) {
#pragma unroll
            for (int k = 0; k < R; k++) {
                num = fma(S::weight(k), c[k], num);
                den += S::weight(k);
            }
            return num * (1.0 / den);
        } else {
            double x[R];
            S::forms(d, eps, x);
            const double tau = VER == FIN_WENO_Z ? S::tau(x) : 0.0;
#pragma unroll
            for (int k = 0; k < R; k++) {
                double w;   // (eps + beta)^-p, or 1 + (tau / (eps + beta))^p
                if (P2) {
                    const double r = VER == FIN_WENO_Z ? tau * rcp(x[k]) : rcp(x[k]);
                    w = VER == FIN_WENO_Z ? fma(r, r, 1.0) : r * r;
                } else {
                    w = VER == FIN_WENO_Z ? 1.0 + power<CALL>(tau / x[k], pw) : power<CALL>(x[k], -pw);
                }
                w *= S::weight(k);
                num = fma(w, c[k], num);
                den += w;
            }
            return num * rcp(den);
        }
    }
}

}  // namespace hi
}  // namespace fin
