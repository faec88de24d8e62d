// Full characteristic WENO flux of one face (ConstructL.cpp:62-208 for x
// faces, 214-358 for y faces) from its 6-point stencil in FP32, with the
// stencil access abstracted.  With gp_s = L (f_s + l q_s), s = 0..4, gm_s =
// L (f_{5-s} - l q_{5-s}) (ConstructL.cpp:179-185, f the half fluxes, l = 0.5
// alpha_scaling alpha) and R L = I, the face flux is
//   (f_2 + l q_2) + (f_3 - l q_3) + R c / 6,
// c the corrections weno5_diff of both splits in the five characteristic
// fields, from the first differences of the stencil only.
#pragma once
#include "fin_device.cuh"

namespace fin {

// Scheduling fence: an empty volatile asm that reads and writes x (volatile
// asm statements keep their order), so that a face's reconstructions are
// not all evaluated at once.
__device__ __forceinline__ void wfence(double& x) { asm volatile("" : "+d"(x)); }
__device__ __forceinline__ void wfence(float& x) { asm volatile("" : "+f"(x)); }

// pt(s, v): the normal-frame pairs v[0..4] = (f, q) of stencil point s = 0..5
// (cells i-3 .. i+2 of the face between i-1 and i); park(m, x) / parked(m): a
// store for the five upwind parts while the fields are reconstructed (the
// face's flux slot).
//
// f32x2 throughout: a pair's lanes are the flux and the state, so the pairs
// come from memory as they lie, difference and projection serve both terms
// of the split at once, and the two scalar operations that form f + l q and
// f - l q write the (gp, gm) pairs of the reconstruction in their registers'
// places (gm's stencil runs backwards, so its differences change place).
// About 415 operations a face against 560 and as many packing moves as pairs
// when the splits were projected point by point.  Fields 0, 4 and 1 in one
// sweep, 2 and 3 in another: all five hold more registers than three or four
// CTAs per SM leave.  Measured (B200): the FP32 stage, two steps of 4001 x
// 515, 1.48 -> 1.16 ms; the hybrid form, eight steps at 4096^2 with 40 %
// of the faces troubled, 40.0 -> 35.1 ms.
template <int VER, bool P2, class Pt, class Park, class Parked>
__device__ __forceinline__ void weno_char_flux(const Euler::Face<float>& ev, float lah, float eps, float pw, const Pt& pt,
                                               const Park& park, const Parked& parked, float* fh)
{
    constexpr bool X2 = P2 || VER == FIN_WENO_FD;
    float g[MEQN];
    const float eps4 = 4.0f * eps;
    // (gp, gm) differences of one field: dp[k], dm[k] in reconstruction order
    auto recon = [&](const float* dp, const float* dm) -> float {
        if constexpr (X2) {
            return weno5_diff_x2<VER>(f2_make(dp[0], dm[0]), f2_make(dp[1], dm[1]), f2_make(dp[2], dm[2]),
                                      f2_make(dp[3], dm[3]), eps4);
        } else {
            return weno5_diff<float, VER, P2>(dp[0], dp[1], dp[2], dp[3], eps4, pw) +
                   weno5_diff<float, VER, P2>(dm[0], dm[1], dm[2], dm[3], eps4, pw);
        }
    };
    // the split of a projected difference D_s (point s minus point s-1)
    auto split = [&](int s, f2 w, float* dp, float* dm) {
        if (s < 5) dp[s - 1] = fmaf(lah, f2_hi(w), f2_lo(w));
        if (s > 1) dm[5 - s] = fmaf(lah, f2_hi(w), -f2_lo(w));
    };
    {
        float p0[4], m0[4], p1[4], m1[4], p4[4], m4[4];
        const f2 nu1 = f2_splat(-ev.u1), nu2 = f2_splat(-ev.u2), nu3 = f2_splat(-ev.u3), hu2 = f2_splat(ev.hu2);
        const f2 kk = f2_splat(ev.k), hc = f2_splat(ev.hc), nhc = f2_splat(-ev.hc);
        f2 prev[MEQN];
        pt(0, prev);
#pragma unroll
        for (int s = 1; s < 6; s++) {
            // keep the compiler from hoisting every stencil point's loads
            // ahead of the arithmetic
            asm volatile("" ::: "memory");
            f2 v[MEQN], d[MEQN];
            pt(s, v);
#pragma unroll
            for (int m = 0; m < MEQN; m++) {
                d[m] = f2_sub(v[m], prev[m]);
                if (s == 3) park(m, fmaf(-lah, f2_hi(d[m]), f2_lo(prev[m]) + f2_lo(v[m])));
                prev[m] = v[m];
            }
            const f2 ks = f2_mul(kk, f2_fma(hu2, d[0], f2_fma(nu3, d[3], f2_fma(nu2, d[2], f2_fma(nu1, d[1], d[4])))));
            const f2 mm = f2_fma(nu1, d[0], d[1]);
            split(s, f2_fma(nhc, mm, ks), p0, m0);
            split(s, f2_fma(hc, mm, ks), p4, m4);
            split(s, f2_fma(f2_splat(-2.0f), ks, d[0]), p1, m1);
        }
        g[0] = recon(p0, m0);
        wfence(g[0]);
        g[4] = recon(p4, m4);
        wfence(g[4]);
        g[1] = recon(p1, m1);
        wfence(g[1]);
    }
    {
        // fields 2 and 3 (v_t - u2 v0, v_w - u3 v0)
        float p2[4], m2[4], p3[4], m3[4];
        const f2 nu2 = f2_splat(-ev.u2), nu3 = f2_splat(-ev.u3);
        f2 c2, c3;
#pragma unroll
        for (int s = 0; s < 6; s++) {
            asm volatile("" ::: "memory");
            f2 v[MEQN];
            pt(s, v);
            const f2 w2 = f2_fma(nu2, v[0], v[2]), w3 = f2_fma(nu3, v[0], v[3]);
            if (s > 0) {
                split(s, f2_sub(w2, c2), p2, m2);
                split(s, f2_sub(w3, c3), p3, m3);
            }
            c2 = w2;
            c3 = w3;
        }
        g[2] = recon(p2, m2);
        wfence(g[2]);
        g[3] = recon(p3, m3);
    }
    Euler::right(ev, g, fh);
#pragma unroll
    for (int m = 0; m < MEQN; m++) fh[m] = fmaf(1.0f / 6.0f, fh[m], parked(m));
}

}  // namespace fin
