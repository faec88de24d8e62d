// Ideal MHD stage kernel: one launch per SSP-RK3 stage of the reference's
// MHD application (apps/2d/mhd/lib/FinSolveRK.cpp:176-219) computes, for a
// TI x TJ tile of cells,
//   L(q_in)     ConstructL (lib/2d/ConstructL.cpp:62-401) with the MHD
//               callbacks: FluxFunc.cpp:19-54, SetWaveSpd.cpp:11-90 and the
//               8 x 8 eigenvector projections of ProjectLeftEig.cpp /
//               ProjectRightEig.cpp;
//   Laux(q_in)  ConstructHJ_L_Order1 (ConstructHJ_L.cpp:29-113): WENO
//               Hamilton-Jacobi right-hand side of the potential A3;
//   q_out, A3_out = a1*A + a2*B + (beta*dt)*(L, Laux)   (UpdateSoln.cpp:21-58);
//   B1, B2 of q_out rebuilt from A3_out (AfterStep.cpp:31-56, constrained
//               transport), which needs A3_out two cells beyond the tile: the
//               kernel updates A3 on the tile plus a 2-cell cross halo (the
//               halo values are recomputed by the neighbouring tiles with the
//               same arithmetic, so they agree bit for bit);
// and, in its epilogue, the maxima the next stage needs: the GlobalWaveSpd
// maxima of q_out (lib/2d/GlobalWaveSpd.cpp:52-78), the HJ speeds max|u1|,
// max|u2| of q_out (ConstructHJ_L.cpp:472-497), and the face-speed maxima
// over the faces GetCFL reads (apps/2d/mhd/lib/GetCFL.cpp:54-59).
//
// State in HBM: 9 planes of mx*my FP64 values (j fastest): rho, rho u1,
// rho u2, rho u3, E, B1, B2, B3 and A3.  Boundaries are doubly periodic
// (apps/2d/mhd/orszag_tang/SetBndValues.cpp), applied as an index remap on
// load.
//
// The projections are not the reference's dense 8 x 8 products: with
//   z = (v0, (v_n - u_n v0)/rho, (v_t - u_t v0)/rho, (v_w - u_w v0)/rho,
//        (gamma-1) P, v_bn, v_bt, v_bw),
//   P = |u|^2/2 v0 - u.v_m + v_E - B.v_B,
// the reference's Lmat v (ProjectLeftEig.cpp:179-206) equals ru z, ru being
// its primitive eigenvector rows, and ru has 35 nonzeros in pairs that share
// terms (fast -/+, slow -/+, Alfven -/+), so each row costs a few operations;
// the right projection (ProjectRightEig.cpp:176-203) is the transposed form.
// The per-face scalars are those of ProjectLeftEig.cpp:34-86, in FP64
// evaluated with the reference's own rounding (see mhd_eig_scalars).
#pragma once
#include "fin_device.cuh"
#include "fin_stage.cuh"   // flag masks (flag_wx, row_bits) and linear_face
#include <type_traits>

namespace fin {

constexpr int MHD_NQ = 8;   // rho, rho u1, rho u2, rho u3, E, B1, B2, B3
constexpr int MHD_NP = 9;   // + A3

struct MhdArgs {
    const double* qin;     // stage input (9 planes)
    const double* A;       // a1 operand (9 planes); nullptr = term absent
    const double* B;       // a2 operand; nullptr = term absent
    double* qout;          // output (9 planes; never aliases qin)
    double a1, a2, bdt;    // bdt = beta*dt
    int mx, my;
    size_t plane;
    double rdx, rdy;       // 1/dx, 1/dy
    double ct_y, ct_x;     // 1.0/(12.0*dy), -1.0/(12.0*dx)  (AfterStep.cpp:39-48)
    int ct;                // constrained transport on
    double gamma, eps, pw, alpha_scaling;
    float gamma_f, eps_f, pw_f, alpha_scaling_f;
    double r_sqrt2;        // 1.0/sqrt(2.0)
    double alf_deg, als_deg;   // sin(atan(1.0)/2.0), cos(atan(1.0)/2.0) (ProjectLeftEig.cpp:78-79)
    const double* alpha_in;    // [2] global alpha of q_in (x, y); nullptr = local LLF
    const double* hj_in;       // [2] max |u1|, |u2| of q_in
    double* alpha_out;         // [2] max cell speed of q_out; nullptr = skip
    double* hj_out;            // [2] max |u1|, |u2| of q_out; nullptr = skip
    double* smax_out;          // [2] max face speed over GetCFL's faces
    double* face_alpha_x;      // optional per-face alpha, (mx+1) x my, i-major
    double* face_alpha_y;      // optional per-face alpha, mx x (my+1)
    unsigned int* status;      // bit 0: non-finite speed, bit 1: negative p or rho, bit 2: a tensor-core
                               // wait ran out (indicator)
    const unsigned* flags;     // hybrid form: troubled-face bit masks (flag_wx / flag_wy layout of fin_stage.cuh)
};

// Periodic index wrap: one add or subtract for the indices a tile reaches
// (at most one period outside), the general remap otherwise (grids smaller
// than a tile and its halo).
__device__ __forceinline__ int pwrap(int k, int n)
{
    if (k < 0) k += n;
    else if (k >= n) k -= n;
    if (unsigned(k) >= unsigned(n)) k = bc_remap(k, n, FIN_BC_PERIODIC, FIN_BC_PERIODIC);
    return k;
}

template <class R> struct MPar;
template <> struct MPar<double> {
    __device__ static double gamma(const MhdArgs& a) { return a.gamma; }
    __device__ static double eps(const MhdArgs& a) { return a.eps; }
    __device__ static double pw(const MhdArgs& a) { return a.pw; }
    __device__ static double ascale(const MhdArgs& a) { return a.alpha_scaling; }
};
template <> struct MPar<float> {
    __device__ static float gamma(const MhdArgs& a) { return a.gamma_f; }
    __device__ static float eps(const MhdArgs& a) { return a.eps_f; }
    __device__ static float pw(const MhdArgs& a) { return a.pw_f; }
    __device__ static float ascale(const MhdArgs& a) { return a.alpha_scaling_f; }
};

// Products and sums with the reference's rounding (no contraction), for the
// branch conditions of ProjectLeftEig.cpp:58-86.
__device__ __forceinline__ double xmul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double xadd(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double xsub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double xdiv(double a, double b) { return __ddiv_rn(a, b); }
__device__ __forceinline__ float xmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float xadd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float xsub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float xdiv(float a, float b) { return __fdiv_rn(a, b); }

// The scalars of ProjectLeftEig.cpp:34-86 at a face-average state Q (normal
// frame).  Near degenerate states the reference's alpha_f, alpha_s and c_s are
// differences of nearly equal numbers (where B_perp -> 0 its alpha_s is
// sqrt(c_f^2 - a^2) of a rounding-level difference); the eigenvectors, and
// through the nonlinear WENO weights the fluxes, follow those rounding bits.
// The FP64 form therefore evaluates such faces' chain in the reference's order
// with IEEE operations and no contraction (EXACT), so that it takes the same
// values; where c_f^2 - a^2, a^2 - c_s^2 and c_s^2 are each above 1e-4 of
// c_f^2 - c_s^2 (resp. d) and that above 0.05 d the scalars are conditioned
// well enough (rounding reaches them amplified by about 1e2, 1e-14, and the
// fluxes only through the nonlinear weights) that the short chain serves: six
// divisions and six square roots in sequence, about 250 dependent FP64
// operations, were a seventh of the face's work and its longest latency.  The
// line lies at 1e-4 because the departure from the reference in L, for states
// whose transverse field falls to 1e-9, is then that of the exact chain at every
// face (5e-15; 1.4e-14 with the line at 1e-6), for 0.3 % of the step (2.489
// against 2.481 ms, two steps at 1024^2; 1e-3: 2.503).
// In FP32 the chain breaks down near the umbilic point (B_perp -> 0,
// a^2 -> B_n^2/rho): c_f^2 - c_s^2 = sqrt(disc) is resolved to ~3e-4 of d
// only, alpha_f and alpha_s become 0/0, and left times right eigenvectors
// departs from the identity (measured: NaN or 2e-4 in FP32, 1e-16 in FP64).
// The FP32 form recomputes such faces' scalars in FP64.
template <class R>
struct MhdEigScalars { R u1, u2, u3, um2, press, a2, cf, cs, af, as, b2, b3; };

template <class T, bool EXACT>
__device__ __forceinline__ void mhd_eig_core(T gamma, const T* Q, MhdEigScalars<T>& e, T& d, bool& umb)
{
    const T rho = Q[0], B1 = Q[5], B2 = Q[6], B3 = Q[7];
    const T bp2 = xadd(xmul(B2, B2), xmul(B3, B3));
    umb = false;
    if (EXACT) {
        e.u1 = xdiv(Q[1], rho); e.u2 = xdiv(Q[2], rho); e.u3 = xdiv(Q[3], rho);
        e.um2 = xmul(T(0.5), xadd(xadd(xmul(e.u1, e.u1), xmul(e.u2, e.u2)), xmul(e.u3, e.u3)));
        const T Bs = xadd(xadd(xmul(B1, B1), xmul(B2, B2)), xmul(B3, B3));
        e.press = xmul(xsub(gamma, T(1)), xsub(xsub(Q[4], xmul(rho, e.um2)), xmul(T(0.5), Bs)));
        e.a2 = xdiv(xmul(gamma, e.press), rho);
        d = xadd(e.a2, xdiv(Bs, rho));
        const T sq = sqrt(xsub(xmul(d, d), xdiv(xmul(xmul(xmul(T(4), e.a2), B1), B1), rho)));
        e.cf = sqrt(xmul(T(0.5), xadd(d, sq)));
        e.cs = sqrt(xmul(T(0.5), xsub(d, sq)));
        if (bp2 <= T(1.0e-12)) umb = fabs(xsub(e.a2, xdiv(xmul(B1, B1), rho))) <= T(1.0e-12);
        const T cf2 = xmul(e.cf, e.cf), cs2 = xmul(e.cs, e.cs);
        const T den = sqrt(fabs(xsub(cf2, cs2)));
        e.af = xdiv(sqrt(fabs(xsub(e.a2, cs2))), den);
        e.as = xdiv(sqrt(fabs(xsub(cf2, e.a2))), den);
    } else {
        const T ir = rcp(rho);
        e.u1 = Q[1] * ir; e.u2 = Q[2] * ir; e.u3 = Q[3] * ir;
        e.um2 = T(0.5) * (e.u1 * e.u1 + e.u2 * e.u2 + e.u3 * e.u3);
        const T Bs = B1 * B1 + B2 * B2 + B3 * B3;
        e.press = (gamma - T(1)) * (Q[4] - rho * e.um2 - T(0.5) * Bs);
        e.a2 = gamma * e.press * ir;
        d = e.a2 + Bs * ir;
        // clamped: an approximate square root may exceed d for d^2 minus a
        // tiny term (B_n -> 0)
        const T sq = sqrt_fast(Max(d * d - T(4) * e.a2 * (B1 * B1) * ir, T(0)));
        e.cf = sqrt_fast(T(0.5) * (d + sq));
        e.cs = sqrt_fast(Max(T(0.5) * (d - sq), T(0)));
        if (bp2 <= T(1.0e-12)) umb = fabs(e.a2 - B1 * B1 * ir) <= T(1.0e-12);
        const T cf2 = e.cf * e.cf, cs2 = e.cs * e.cs;
        const T iden = sizeof(T) == 8 ? rsqrt_fast(fabs(cf2 - cs2)) : rcp(fsqrt(fabs(cf2 - cs2)));
        e.af = sqrt_fast(fabs(e.a2 - cs2)) * iden;
        e.as = sqrt_fast(fabs(cf2 - e.a2)) * iden;
    }
}

// The rare chains as calls of their own: inlined, their live values and
// instructions weigh on every face's registers.
__device__ __noinline__ void mhd_eig_exact(double gamma, const double* Q, MhdEigScalars<double>* e, bool* umb)
{
    double d;
    mhd_eig_core<double, true>(gamma, Q, *e, d, *umb);
}
__device__ __noinline__ void mhd_eig_fp64(double gamma, const float* Q, MhdEigScalars<float>* e, bool* umb)
{
    double Qd[MHD_NQ], d;
#pragma unroll
    for (int m = 0; m < MHD_NQ; m++) Qd[m] = double(Q[m]);
    MhdEigScalars<double> ed;
    mhd_eig_core<double, false>(gamma, Qd, ed, d, *umb);
    e->u1 = float(ed.u1); e->u2 = float(ed.u2); e->u3 = float(ed.u3); e->um2 = float(ed.um2);
    e->press = float(ed.press); e->a2 = float(ed.a2); e->cf = float(ed.cf); e->cs = float(ed.cs);
    e->af = float(ed.af); e->as = float(ed.as);
}

template <class R>
__device__ __forceinline__ MhdEigScalars<R> mhd_eig_scalars(const MhdArgs& a, R gamma, const R* Q)
{
    MhdEigScalars<R> e;
    R d;
    bool umb;
    mhd_eig_core<R, false>(gamma, Q, e, d, umb);
    if constexpr (sizeof(R) == 8) {
        const R cf2 = e.cf * e.cf, cs2 = e.cs * e.cs, lim = R(1.0e-4) * (cf2 - cs2);
        if (!(cf2 - e.a2 > lim && e.a2 - cs2 > lim && cs2 > R(1.0e-4) * d && cf2 - cs2 > R(0.05) * d)) {
            R q[MHD_NQ];
            MhdEigScalars<R> x;
            bool u;
#pragma unroll
            for (int m = 0; m < MHD_NQ; m++) q[m] = Q[m];
            mhd_eig_exact(gamma, q, &x, &u);
            e = x;
            umb = u;
        }
    } else if (!(e.cf * e.cf - e.cs * e.cs > R(1.0e-2) * d)) {
        // near the umbilic point: the same scalars in FP64
        R q[MHD_NQ];
        MhdEigScalars<R> x;
        bool u;
#pragma unroll
        for (int m = 0; m < MHD_NQ; m++) q[m] = Q[m];
        mhd_eig_fp64(a.gamma, q, &x, &u);
        e = x;
        umb = u;
    }
    const R B2 = Q[6], B3 = Q[7];
    const R rs2 = R(a.r_sqrt2);
    if (xadd(xmul(B2, B2), xmul(B3, B3)) <= R(1.0e-12)) {
        e.b2 = rs2;
        e.b3 = rs2;
    } else {
        const R ib = sizeof(R) == 8 ? rsqrt_fast(B2 * B2 + B3 * B3) : rcp(fsqrt(B2 * B2 + B3 * B3));
        e.b2 = B2 * ib;
        e.b3 = B3 * ib;
    }
    if (umb) {
        e.af = R(a.alf_deg);
        e.as = R(a.als_deg);
    }
    return e;
}

// Per-face coefficients of the left projection passes (normal frame; the
// density and (gamma-1) factors of z folded in).
template <class R>
struct MhdFace {
    R u1, u2, u3, um2, B1, B2, B3, b2, b3;
    R kfn, ksu, kfp, ksb;   // fast rows 0 / 7: dn, S_u, P, S_b
    R ksn, kfu, ksp, kfb;   // slow rows 2 / 5
    R ra, rb;               // Alfven rows 1 / 6: T_u, T_b
    R ie;                   // entropy row 3: v0 - ie P
};
// The right projection's coefficients, parked in shared memory while the
// left passes run.
enum { MR_RHO, MR_AF, MR_AS, MR_CF, MR_CS, MR_BETA1, MR_GP, MR_ASR, MR_SR2, MR_N };

template <class R>
__device__ __forceinline__ void mhd_face_setup(const MhdArgs& a, R gamma, const R* Q, MhdFace<R>& f, R* rec,
                                               int rstride, bool& neg)
{
    const R gm1 = gamma - R(1);
    const R rho = Q[0];
    const MhdEigScalars<R> e = mhd_eig_scalars<R>(a, gamma, Q);
    f.u1 = e.u1; f.u2 = e.u2; f.u3 = e.u3; f.um2 = e.um2;
    f.B1 = Q[5]; f.B2 = Q[6]; f.B3 = Q[7];
    f.b2 = e.b2; f.b3 = e.b3;
    if (e.press < R(0) || rho < R(0)) neg = true;
    const R ir = rcp(rho);
    const R asnd = sizeof(R) == 8 ? e.a2 * rsqrt_fast(e.a2) : fsqrt(e.a2);   // the reference's sqrt: NaN when a2 < 0
    const R beta1 = f.B1 < R(0) ? R(-1) : R(1);
    const R af = e.af, as = e.as, cf = e.cf, cs = e.cs;
    const R rs2 = R(a.r_sqrt2);
    const R rsq = sqrt_fast(rho);
    const R ia2 = rcp(e.a2);
    const R h = R(0.5) * ia2 * ir;             // 1/(2 a^2 rho)
    const R hb = R(0.5) * rcp(rsq * asnd);     // 1/(2 sqrt(rho) a)
    f.kfn = af * cf * h;
    f.ksu = as * cs * beta1 * h;
    f.kfp = af * h * gm1;
    f.ksb = as * hb;
    f.ksn = as * cs * h;
    f.kfu = af * cf * beta1 * h;
    f.ksp = as * h * gm1;
    f.kfb = af * hb;
    f.ra = rs2 * ir;
    f.rb = rs2 * rcp(rsq);
    f.ie = gm1 * ia2;
    if (!rec) return;
    rec[MR_RHO * rstride] = rho;
    rec[MR_AF * rstride] = af;
    rec[MR_AS * rstride] = as;
    rec[MR_CF * rstride] = cf;
    rec[MR_CS * rstride] = cs;
    rec[MR_BETA1 * rstride] = beta1;
    rec[MR_GP * rstride] = gamma * e.press;
    rec[MR_ASR * rstride] = asnd * rsq;
    rec[MR_SR2 * rstride] = rsq * rs2;
}

// The left projection of one normal-frame vector v, whose entries are scalars
// or f2 pairs (two vectors at once).
template <class R> __device__ __forceinline__ R vmul(R c, R x) { return c * x; }
template <class R> __device__ __forceinline__ R vma(R c, R x, R a) { return c * x + a; }
template <class R> __device__ __forceinline__ R vadd(R x, R y) { return x + y; }
template <class R> __device__ __forceinline__ R vsub(R x, R y) { return x - y; }
__device__ __forceinline__ f2 vmul(float c, f2 x) { return f2_mul(f2_splat(c), x); }
__device__ __forceinline__ f2 vma(float c, f2 x, f2 a) { return f2_fma(f2_splat(c), x, a); }
__device__ __forceinline__ f2 vadd(f2 x, f2 y) { return f2_add(x, y); }
__device__ __forceinline__ f2 vsub(f2 x, f2 y) { return f2_sub(x, y); }

template <class R, class V>
__device__ __forceinline__ V mhd_P(const MhdFace<R>& f, const V* v)
{
    V t = vma(f.um2, v[0], v[4]);
    t = vma(-f.u1, v[1], t);
    t = vma(-f.u2, v[2], t);
    t = vma(-f.u3, v[3], t);
    t = vma(-f.B1, v[5], t);
    t = vma(-f.B2, v[6], t);
    return vma(-f.B3, v[7], t);
}
// fast and slow pairs (rows 0 / 7 and 2 / 5), sharing dn, S_u, P, S_b
template <class R, class V>
__device__ __forceinline__ void mhd_left_fs4(const MhdFace<R>& f, const V* v, V& w0, V& w7, V& w2, V& w5)
{
    const V dn = vma(-f.u1, v[0], v[1]);
    const V dt = vma(-f.u2, v[0], v[2]);
    const V dw = vma(-f.u3, v[0], v[3]);
    const V P = mhd_P(f, v);
    const V Su = vma(f.b2, dt, vmul(f.b3, dw));
    const V Sb = vma(f.b2, v[6], vmul(f.b3, v[7]));
    V s = vma(f.kfp, P, vmul(f.ksb, Sb)), t = vma(f.ksu, Su, vmul(-f.kfn, dn));
    w0 = vadd(s, t);
    w7 = vsub(s, t);
    s = vma(f.ksp, P, vmul(-f.kfb, Sb));
    t = vma(f.ksn, dn, vmul(f.kfu, Su));
    w2 = vsub(s, t);
    w5 = vadd(s, t);
}
// Alfven pair (rows 1 / 6)
template <class R, class V>
__device__ __forceinline__ void mhd_left_alf(const MhdFace<R>& f, const V* v, V& wm, V& wp)
{
    const V dt = vma(-f.u2, v[0], v[2]);
    const V dw = vma(-f.u3, v[0], v[3]);
    const V Tu = vmul(f.ra, vma(f.b2, dw, vmul(-f.b3, dt)));
    const V Tb = vmul(f.rb, vma(f.b2, v[7], vmul(-f.b3, v[6])));
    wm = vadd(Tu, Tb);
    wp = vsub(Tu, Tb);
}
// entropy and divergence rows (3 / 4)
template <class R, class V>
__device__ __forceinline__ void mhd_left_ent(const MhdFace<R>& f, const V* v, V& w3, V& w4)
{
    w3 = vma(-f.ie, mhd_P(f, v), v[0]);
    w4 = v[5];
}

template <int TI_, int TJ_, int NT_, int MINB_ = 1>
struct MhdCfg {
    static constexpr int TI = TI_, TJ = TJ_, NT = NT_;
    static constexpr int MINB = MINB_;   // resident blocks per SM the registers are sized for
    static constexpr int H = 3;              // q halo of the WENO stencils
    static constexpr int HA = 5;             // A3 halo (HJ stencils of the 2-cell CT halo)
    static constexpr int HN = 2;             // CT halo of the updated A3
    static constexpr int RI = TI + 2 * H, RJ = TJ + 2 * H;
    static constexpr int PI = TI + 2, PJ = TJ + 2;      // per-cell speed data (halo 1)
    static constexpr int AI = TI + 2 * HA, AJ = TJ + 2 * HA;
    static constexpr int NI = TI + 2 * HN, NJ = TJ + 2 * HN;
    static constexpr int NFX = (TI + 1) * TJ, NFY = TI * (TJ + 1);
    // R arrays: qs [8][RI*RJ], fs [8][RI*TJ], gs [8][TI*RJ], pc [4][PI*PJ],
    // Fh [8][NFX], Gh [8][NFY]; then rec [MR_N][NT] over as [AI*AJ] (FP64);
    // then FP64: an [NI*NJ], red [6][NT/32].
    // FP32 faces of a 15 x 16 tile go to threads so that the two half-warps
    // of a warp take face rows 8 apart (ROW8): 8 rows of RJ = 22 (PJ = 18)
    // words are 176 (144) words, 16 modulo 32, so the two rows' words fall
    // in opposite halves of the banks; the x-direction flux rows get a pitch
    // of FSJ = 18 for the same reason.  FP64 keeps the row-by-row order.
    template <class R>
    __host__ __device__ static constexpr bool ROW8() { return sizeof(R) == 4 && TI == 15 && TJ == 16; }
    template <class R>
    __host__ __device__ static constexpr int FSJ() { return ROW8<R>() ? TJ + 2 : TJ; }
    template <class R>
    __host__ __device__ static constexpr size_t NR()
    {
        return size_t(MHD_NQ) * (RI * RJ + RI * FSJ<R>() + TI * RJ + NFX + NFY) + 4 * PI * PJ;
    }
    // rec (while the faces run) and as (before) share their space
    template <class R>
    __host__ __device__ static constexpr size_t rec_offset() { return (NR<R>() * sizeof(R) + 15) / 16 * 16; }
    template <class R>
    __host__ __device__ static constexpr size_t dbl_offset()
    {
        const size_t rec = size_t(MR_N) * NT * sizeof(R), as = sizeof(double) * size_t(AI) * AJ;
        return (rec_offset<R>() + (rec > as ? rec : as) + 15) / 16 * 16;
    }
    template <class R>
    __host__ __device__ static constexpr size_t smem_bytes()
    {
        return dbl_offset<R>() + sizeof(double) * (size_t(NI) * NJ + 6 * (NT / 32));
    }
    // Hybrid form, after the above: the two troubled-face lists [NF]
    // (short), their counts, and the flag windows of the
    // 3 x 3 dilation as row masks (x faces: rows i0-1 .. i0+TI+1, bit c =
    // column j0-1+c, c < TJ+2; y faces: rows i0-1 .. i0+TI, c < TJ+3).
    static constexpr int NF = NFX + NFY;
    static constexpr int FXR = TI + 3, FXC = TJ + 2, FYR = TI + 2, FYC = TJ + 3;
    static_assert(FYC <= 32 && FXR <= 32 && FYR <= 32, "flag row masks are 32-bit words read by one warp each");
    template <class R>
    __host__ __device__ static constexpr size_t hyb_ntrb_offset() { return (NF * 2 + 15) / 16 * 16; }
    template <class R>
    __host__ __device__ static constexpr size_t hyb_mask_offset() { return hyb_ntrb_offset<R>() + 16; }
    template <class R>
    __host__ __device__ static constexpr size_t smem_bytes_hyb()
    {
        return smem_bytes<R>() + hyb_mask_offset<R>() + 4 * (FXR + FYR);
    }
};

// Bits of columns c0 .. c0+nb-1 (nb <= 32) of one flag-mask row of nw words,
// columns taken modulo the period (periodic boundaries; the flag arrays hold
// columns 0 .. period-1, y faces also column period, equal to column 0).
__device__ __forceinline__ unsigned mask_row_wrapped(const unsigned* row, int nw, int c0, int nb, int period)
{
    if (c0 >= 0 && c0 + nb <= period) {
        const int k = c0 >> 5;
        const unsigned lo = ld_dep(row + k), hi = k + 1 < nw ? ld_dep(row + k + 1) : 0u;
        return row_bits(lo, hi, c0) & (nb >= 32 ? 0xffffffffu : ((1u << nb) - 1u));
    }
    unsigned m = 0;
    for (int b = 0; b < nb; b++) {
        int c = c0 + b;
        if (c < 0) c += period;
        else if (c >= period) c -= period;
        m |= ((ld_dep(row + (c >> 5)) >> (c & 31)) & 1u) << b;
    }
    return m;
}

// Shared-memory arrays of a stage tile that the faces read and write.
template <class R, class Cfg>
struct MhdSmem {
    static constexpr int PQ = Cfg::RI * Cfg::RJ, PP = Cfg::PI * Cfg::PJ, FS = Cfg::template FSJ<R>();
    R* qs;    // [8][RI][RJ]
    R* fs;    // [8][RI][FS]  0.5 f
    R* gs;    // [8][TI][RJ]  0.5 g
    R* pc;    // [4][PI][PJ]  u1, u2, p, cf
    R* Fh;    // [8][TI+1][TJ]
    R* Gh;    // [8][TI][TJ+1]
    R* rec;   // [MR_N][NT]
    __device__ __forceinline__ explicit MhdSmem(unsigned char* raw)
    {
        qs = reinterpret_cast<R*>(raw);
        fs = qs + MHD_NQ * PQ;
        gs = fs + MHD_NQ * Cfg::RI * FS;
        pc = gs + MHD_NQ * Cfg::TI * Cfg::RJ;
        Fh = pc + 4 * PP;
        Gh = Fh + MHD_NQ * Cfg::NFX;
        rec = reinterpret_cast<R*>(raw + Cfg::template rec_offset<R>());
    }
};

// An FP32 correction with a power other than 2, as a call: inlined, the two
// directions' bodies hold 96 powers (spills of 280 bytes; 112 registers and none
// now).  One step at 1024^2 with power 1.5, ms, one body for both directions / a
// body each / now: JS 2.02 / 2.27 / 1.90, Z 2.66 / 2.44 / 2.25.
template <int VER>
__device__ __noinline__ float mhd_weno5_pow(float d1, float d2, float d3, float d4, float eps4, float pw)
{
    return weno5_diff<float, VER, false>(d1, d2, d3, d4, eps4, pw);
}

// The faces of direction x (ISX: face (fi, fj) between tile rows fi-1 and fi)
// or y (between columns fj-1 and fj); the direction is a template parameter,
// so stencil addresses and the normal frame (rho, m_n, m_t, m_w, E, B_n, B_t,
// B_w) are constant offsets.
template <class R, int VER, bool P2, class Cfg, bool ISX>
struct MhdDir {
    using S_ = MhdSmem<R, Cfg>;
    static constexpr int TI = Cfg::TI, TJ = Cfg::TJ, RI = Cfg::RI, RJ = Cfg::RJ, H = Cfg::H, NT = Cfg::NT;
    static constexpr int PQ = S_::PQ, PP = S_::PP, PJ = Cfg::PJ, FS = S_::FS;
    static constexpr int NF = ISX ? Cfg::NFX : Cfg::NFY;
    static constexpr int QSTR = ISX ? RJ : 1, FSTR = ISX ? FS : 1, FP = ISX ? RI * FS : TI * RJ, PSTR = ISX ? PJ : 1;
    static constexpr int NJ = ISX ? TJ : TJ + 1;
    static constexpr bool DIRECT = sizeof(R) == 4;
    __device__ __forceinline__ static constexpr int perm(int c)
    {
        return ISX ? c : (c == 1 ? 2 : c == 2 ? 1 : c == 5 ? 6 : c == 6 ? 5 : c);
    }
    // Face of work index w: by rows of TJ, then (y faces) the last column, so
    // that a half-warp reads one row of the staged tile; FP32: half-warps on
    // rows r and r + 8 (the last warp of y faces on row 7 and the last column).
    __device__ __forceinline__ static void locate(int w, int& fi, int& fj)
    {
        if constexpr (Cfg::template ROW8<R>()) {
            const int wv = w >> 5, ln = w & 31;
            if (ISX || wv < 7) { fi = wv + (ln & 16 ? 8 : 0); fj = ln & 15; }
            else if (ln < 16) { fi = 7; fj = ln; }
            else { fi = ln - 16; fj = TJ; }
        } else {
            fi = ISX || w < TI * TJ ? w / TJ : w - TI * TJ;
            fj = ISX || w < TI * TJ ? w - fi * TJ : TJ;
        }
    }
    __device__ __forceinline__ static const R* qbase(const S_& S, int fi, int fj) { return S.qs + (H + fi) * RJ + (H + fj); }
    __device__ __forceinline__ static const R* fbase(const S_& S, int fi, int fj)
    {
        return ISX ? S.fs + (H + fi) * FS + fj : S.gs + fi * RJ + (H + fj);
    }
    __device__ __forceinline__ static R* slot(const S_& S, int fi, int fj)
    {
        return ISX ? S.Fh + fi * TJ + fj : S.Gh + fi * (TJ + 1) + fj;
    }
    // SetWaveSpd.cpp:39-88 (nmag = 1; the fast speeds use B1, the x
    // component, for either normal) and the LLF alpha of ConstructL.cpp:172-174.
    __device__ __forceinline__ static R speed(const S_& S, R gamma, int fi, int fj, R ag)
    {
        const R* const q = qbase(S, fi, fj);
        const R* const p = S.pc + (fi + 1) * PJ + (fj + 1);
        constexpr int un = ISX ? 0 : 1;
        const R unl = p[un * PP - PSTR], unr = p[un * PP];
        const R pa = R(0.5) * (p[2 * PP - PSTR] + p[2 * PP]);
        const R rho = R(0.5) * (q[0] + q[-QSTR]);
        const R b5 = R(0.5) * (q[5 * PQ] + q[5 * PQ - QSTR]);
        const R b6 = R(0.5) * (q[6 * PQ] + q[6 * PQ - QSTR]);
        const R b7 = R(0.5) * (q[7 * PQ] + q[7 * PQ - QSTR]);
        const R Bm2 = b5 * b5 + b6 * b6 + b7 * b7;
        const R ir = rcp(rho);
        const R a2 = fabs(gamma * pa * ir);
        const R t = a2 + Bm2 * ir;
        const R cf = sqrt_fast(R(0.5) * (t + sqrt_fast(fabs(t * t - R(4) * a2 * (b5 * b5) * ir))));
        const R ua = R(0.5) * (unl + unr);
        const R s1 = MinN(unl - p[3 * PP - PSTR], ua - cf);
        const R s2 = MaxN(unr + p[3 * PP], ua + cf);
        return MaxN(ag, MaxN(R(fabs(s1)), R(fabs(s2))));
    }
    // One sweep over the stencil: the (gp, gm) differences of K characteristic
    // fields in reconstruction order, dp[k] from v+ = 0.5 f + lah q at points
    // 0..4 and dm[k] from v- = 0.5 f - lah q at points 5..1 (ConstructL.cpp:
    // 179-185), and in FP64 the sum up[k] of the splits' upwind points.  FP64
    // projects both splits; FP32 projects (f, q) pairs, and the split forms
    // both from one projection.
    template <int K, class Left>
    __device__ __forceinline__ static void sweep(const R* qb, const R* fb, R lah, const Left& left, R (&dp)[K][4],
                                                 R (&dm)[K][4], R* up)
    {
        if constexpr (sizeof(R) == 4) {
            f2 c[K];
#pragma unroll
            for (int s = 0; s < 6; s++) {
                // keep the compiler from hoisting every point's loads ahead of the arithmetic
                asm volatile("" ::: "memory");
                f2 v[MHD_NQ], w[K];
#pragma unroll
                for (int m = 0; m < MHD_NQ; m++)
                    v[m] = f2_make(fb[perm(m) * FP + (s - 3) * FSTR], qb[perm(m) * PQ + (s - 3) * QSTR]);
                left(v, w);
#pragma unroll
                for (int k = 0; k < K; k++) {
                    if (s > 0) {
                        const f2 d = f2_sub(w[k], c[k]);
                        if (s < 5) dp[k][s - 1] = fmaf(lah, f2_hi(d), f2_lo(d));
                        if (s > 1) dm[k][5 - s] = fmaf(lah, f2_hi(d), -f2_lo(d));
                    }
                    c[k] = w[k];
                }
            }
        } else {
            R cp[K], cm[K];
#pragma unroll
            for (int s = 0; s < 6; s++) {
                asm volatile("" ::: "memory");
                R q[MHD_NQ], f[MHD_NQ], v[MHD_NQ], w[K];
#pragma unroll
                for (int m = 0; m < MHD_NQ; m++) {
                    q[m] = qb[perm(m) * PQ + (s - 3) * QSTR];
                    f[m] = fb[perm(m) * FP + (s - 3) * FSTR];
                }
                if (s < 5) {
#pragma unroll
                    for (int m = 0; m < MHD_NQ; m++) v[m] = f[m] + lah * q[m];
                    left(v, w);
#pragma unroll
                    for (int k = 0; k < K; k++) {
                        if (s > 0) dp[k][s - 1] = w[k] - cp[k];
                        if (s == 2) up[k] = w[k];
                        cp[k] = w[k];
                    }
                }
                if (s > 0) {
#pragma unroll
                    for (int m = 0; m < MHD_NQ; m++) v[m] = f[m] - lah * q[m];
                    left(v, w);
#pragma unroll
                    for (int k = 0; k < K; k++) {
                        if (s > 1) dm[k][5 - s] = cm[k] - w[k];
                        if (s == 3) up[k] = up[k] + w[k];
                        cm[k] = w[k];
                    }
                }
            }
        }
    }
    // Corrections (weno5_diff) of K fields, one field between scheduling fences.
    template <int K>
    __device__ __forceinline__ static void fields(R (&dp)[K][4], R (&dm)[K][4], R eps4, R pw, R* g)
    {
#pragma unroll
        for (int k = 0; k < K; k++) {
#pragma unroll
            for (int t = 0; t < 4; t++) { wfence(dp[k][t]); wfence(dm[k][t]); }
            if constexpr (sizeof(R) == 4 && (P2 || VER == FIN_WENO_FD))
                g[k] = weno5_diff_x2<VER>(f2_make(dp[k][0], dm[k][0]), f2_make(dp[k][1], dm[k][1]),
                                          f2_make(dp[k][2], dm[k][2]), f2_make(dp[k][3], dm[k][3]), eps4);
            else if constexpr (sizeof(R) == 4)
                g[k] = mhd_weno5_pow<VER>(dp[k][0], dp[k][1], dp[k][2], dp[k][3], eps4, pw) +
                       mhd_weno5_pow<VER>(dm[k][0], dm[k][1], dm[k][2], dm[k][3], eps4, pw);
            else
                g[k] = weno5_diff<R, VER, P2>(dp[k][0], dp[k][1], dp[k][2], dp[k][3], eps4, pw) +
                       weno5_diff<R, VER, P2>(dm[k][0], dm[k][1], dm[k][2], dm[k][3], eps4, pw);
            wfence(g[k]);
        }
    }
    // The full characteristic WENO flux of one face (ConstructL.cpp:72-206 /
    // 224-356 with the MHD projections) into its slot, from differences of the
    // projected stencil.  FP64 (DIRECT off) projects the upwind points of the
    // splits too: close to the umbilic point the reference's alpha_f, alpha_s
    // make left times right eigenvectors depart from the identity (1e-5 of L
    // was seen), and its result is the contract.  FP32 adds the upwind points
    // in conserved variables (parked in the slot meanwhile), which takes that
    // departure out of them.
    //
    // Bound by the latency of dependent FP64 operations (8 warps per SM at 255
    // registers, FP64 pipe 47 % busy) and in FP32 by issue.  The rows go in
    // two sweeps of four fields (dn, S_u, P and S_b shared by the fast and slow
    // pairs); a sweep per pair loads the stencil twice as often and measured
    // slower (stage at 2048^2, first version: 2.98 against 2.36 ms FP64, 1.78
    // against 1.26 FP32).  Two steps at 1024^2, ms: FP64 3.27 with
    // reconstructions on point values, one body for both directions and the
    // IEEE eigen chain at every face, 3.05 with the difference form alone,
    // 2.52 now; FP32 1.68 -> 1.42; hybrid (four steps) 2.74 -> 2.65.  512 or
    // 384 FP64 threads (128, 168 registers) spill 2.4 and 1.5 KB: 3.9, 3.3 ms;
    // three FP32 CTAs per SM (80 registers) 2.0 ms.
    __device__ __forceinline__ static void flux(const MhdArgs& a, const S_& S, R gamma, R eps, R pw, int fi, int fj,
                                                R alpha, bool& neg)
    {
        const R* const qb = qbase(S, fi, fj);
        const R* const fb = fbase(S, fi, fj);
        R* const out = slot(S, fi, fj);
        R* const rc = S.rec + threadIdx.x;
        const R lah = R(0.5) * MPar<R>::ascale(a) * alpha;
        MhdFace<R> f;
        {
            R Qa[MHD_NQ];
#pragma unroll
            for (int m = 0; m < MHD_NQ; m++) {
                const R ql = qb[perm(m) * PQ - QSTR], qr = qb[perm(m) * PQ];
                Qa[m] = R(0.5) * (qr + ql);
                if (DIRECT) out[perm(m) * NF] = (fb[perm(m) * FP - FSTR] + fb[perm(m) * FP]) + lah * (ql - qr);
            }
            mhd_face_setup<R>(a, gamma, Qa, f, rc, NT, neg);
        }
        R ghat[MHD_NQ], up[4];
        const R eps4 = R(4) * eps, s6 = R(1) / R(6);
        auto put = [&](R* gg) {
#pragma unroll
            for (int k = 0; k < 4; k++)
                if (!DIRECT) gg[k] = s6 * gg[k] + up[k];
        };
        {
            // fast and slow pairs (rows 0, 7, 2, 5) in one sweep
            R dp[4][4], dm[4][4], gg[4];
            sweep<4>(qb, fb, lah, [&](const auto* v, auto* w) { mhd_left_fs4(f, v, w[0], w[1], w[2], w[3]); }, dp, dm, up);
            fields<4>(dp, dm, eps4, pw, gg);
            put(gg);
            ghat[0] = gg[0]; ghat[7] = gg[1]; ghat[2] = gg[2]; ghat[5] = gg[3];
        }
        {
            // Alfven, entropy and divergence rows (1, 6, 3, 4) in one sweep
            R dp[4][4], dm[4][4], gg[4];
            sweep<4>(qb, fb, lah, [&](const auto* v, auto* w) {
                mhd_left_alf(f, v, w[0], w[1]);
                mhd_left_ent(f, v, w[2], w[3]);
            }, dp, dm, up);
            fields<4>(dp, dm, eps4, pw, gg);
            put(gg);
            ghat[1] = gg[0]; ghat[6] = gg[1]; ghat[3] = gg[2]; ghat[4] = gg[3];
        }
        // Right projection (ProjectRightEig.cpp:89-203) in the normal frame.
        const R rho = rc[MR_RHO * NT], af = rc[MR_AF * NT], as_ = rc[MR_AS * NT];
        const R cf = rc[MR_CF * NT], cs = rc[MR_CS * NT], beta1 = rc[MR_BETA1 * NT];
        const R gp = rc[MR_GP * NT], asr = rc[MR_ASR * NT], sr2 = rc[MR_SR2 * NT];
        const R rs2 = R(a.r_sqrt2);
        const R Gp = ghat[0] + ghat[7], Gm = ghat[7] - ghat[0];
        const R Hp = ghat[2] + ghat[5], Hm = ghat[5] - ghat[2];
        const R Kp = ghat[1] + ghat[6], Km = ghat[6] - ghat[1];
        const R fsum = af * Gp + as_ * Hp;
        const R drho = rho * fsum + ghat[3];
        const R dun = af * cf * Gm + as_ * cs * Hm;
        const R X = beta1 * (af * cf * Hm - as_ * cs * Gm);
        const R dut = f.b2 * X - f.b3 * rs2 * Kp;
        const R duw = f.b3 * X + f.b2 * rs2 * Kp;
        const R dp_ = gp * fsum;
        const R dbn = ghat[4];
        const R Y = asr * (as_ * Gp - af * Hp);
        const R dbt = f.b2 * Y + f.b3 * sr2 * Km;
        const R dbw = f.b3 * Y - f.b2 * sr2 * Km;
        auto store = [&](int m, R x) { out[m * NF] = DIRECT ? s6 * x + out[m * NF] : x; };
        store(0, drho);
        store(perm(1), rho * dun + f.u1 * drho);
        store(perm(2), rho * dut + f.u2 * drho);
        store(3, rho * duw + f.u3 * drho);
        store(4, f.um2 * drho + rho * (f.u1 * dun + f.u2 * dut + f.u3 * duw) + dp_ * rcp(gamma - R(1)) + f.B1 * dbn +
                     f.B2 * dbt + f.B3 * dbw);
        store(perm(5), dbn);
        store(perm(6), dbt);
        store(7, dbw);
    }
    // The linear FD5 flux of a smooth face, component by component (linear_face).
    __device__ __forceinline__ static void linear(const MhdArgs& a, const S_& S, int fi, int fj, R alpha)
    {
        const R lah = R(0.5) * MPar<R>::ascale(a) * alpha;
        R* const out = slot(S, fi, fj);
#pragma unroll
        for (int m = 0; m < MHD_NQ; m++)
            out[m * NF] = linear_face<R>(fbase(S, fi, fj) + m * FP, FSTR, qbase(S, fi, fj) + m * PQ, QSTR, lah);
    }
};

template <class R, int VER, bool P2, class Cfg, bool HYB = false>
__global__ void __launch_bounds__(Cfg::NT, Cfg::MINB) k_mhd_stage(const __grid_constant__ MhdArgs a)
{
    grid_dependency();
    constexpr int TI = Cfg::TI, TJ = Cfg::TJ, NT = Cfg::NT, H = Cfg::H;
    constexpr int RI = Cfg::RI, RJ = Cfg::RJ, PQ = RI * RJ;
    constexpr int PI = Cfg::PI, PJ = Cfg::PJ, PP = PI * PJ;
    constexpr int AJ = Cfg::AJ, NJ = Cfg::NJ;
    constexpr int HA = Cfg::HA, HN = Cfg::HN;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    constexpr int FS = Cfg::template FSJ<R>();
    const MhdSmem<R, Cfg> S(smem_raw);
    R* const qs = S.qs;
    R* const fs = S.fs;
    R* const gs = S.gs;
    R* const pc = S.pc;
    R* const Fh = S.Fh;
    R* const Gh = S.Gh;
    double* as = reinterpret_cast<double*>(smem_raw + Cfg::template rec_offset<R>());   // [AI][AJ]
    double* an = reinterpret_cast<double*>(smem_raw + Cfg::template dbl_offset<R>());   // [NI][NJ]
    double* red = an + Cfg::NI * NJ;                 // [NT/32][6]
    unsigned char* hyb_base = smem_raw + Cfg::template smem_bytes<R>();
    unsigned* fxm = reinterpret_cast<unsigned*>(hyb_base + Cfg::template hyb_mask_offset<R>());
    unsigned* fym = fxm + Cfg::FXR;

    const int tid = threadIdx.x;
    const int mx = a.mx, my = a.my;
    const int i0 = blockIdx.y * TI, j0 = blockIdx.x * TJ;
    const R gamma = MPar<R>::gamma(a);
    bool neg = false, nonfinite = false;

    // ---- phase 0: q_in on the tile + 3-cell cross halo, A3 on the tile +
    // 5-cell frame (periodic remap) ----
    // All of a thread's loads (the state, A3 of q_in, and A3 of the other
    // stage operands for the update of phase 1b) are issued before its
    // stores: one memory round trip per tile, not one per pass over a region.
    // The operands' part of the A3 update, a1 A + a2 B (UpdateSoln.cpp:42-47),
    // is kept in an[] for phase 1b to add bdt L to.
    {
        constexpr int NQI = (PQ + NT - 1) / NT, NAI = (Cfg::AI * AJ + NT - 1) / NT;
        constexpr int NHI = (Cfg::NI * NJ + NT - 1) / NT;
        double vq[NQI][MHD_NQ], va[NAI], vab[NHI];
#pragma unroll
        for (int it = 0; it < NQI; it++) {
            const int e = tid + it * NT;
            const int ii = e / RJ, jj = e - ii * RJ;
            const bool xin = ii >= H && ii < H + TI, yin = jj >= H && jj < H + TJ;
            if (e < PQ && (xin || yin)) {
                const int gi = pwrap(i0 + ii - H, mx);
                const int gj = pwrap(j0 + jj - H, my);
                const size_t g = size_t(gi) * my + gj;
#pragma unroll
                for (int m = 0; m < MHD_NQ; m++) vq[it][m] = ld_dep(a.qin + m * a.plane + g);
            }
        }
#pragma unroll
        for (int it = 0; it < NAI; it++) {
            const int e = tid + it * NT;
            if (e < Cfg::AI * AJ) {
                const int ii = e / AJ, jj = e - ii * AJ;
                const int gi = pwrap(i0 + ii - HA, mx);
                const int gj = pwrap(j0 + jj - HA, my);
                va[it] = ld_dep(a.qin + 8 * a.plane + size_t(gi) * my + gj);
            }
        }
#pragma unroll
        for (int it = 0; it < NHI; it++) {
            const int e = tid + it * NT;
            const int ni = e / NJ, nj = e - ni * NJ;
            const int ci = ni - HN, cj = nj - HN;   // tile frame
            const bool xin = ci >= 0 && ci < TI, yin = cj >= 0 && cj < TJ;
            if (e < Cfg::NI * NJ && (xin || yin)) {
                const size_t g = 8 * a.plane + size_t(pwrap(i0 + ci, mx)) * my + pwrap(j0 + cj, my);
                double v = 0.0;
                if (a.A) v = a.a1 * ld_dep(a.A + g);
                if (a.B) v = v + a.a2 * ld_dep(a.B + g);
                vab[it] = v;
            }
        }
#pragma unroll
        for (int it = 0; it < NQI; it++) {
            const int e = tid + it * NT;
            const int ii = e / RJ, jj = e - ii * RJ;
            const bool xin = ii >= H && ii < H + TI, yin = jj >= H && jj < H + TJ;
            if (e < PQ && (xin || yin)) {
#pragma unroll
                for (int m = 0; m < MHD_NQ; m++) qs[m * PQ + e] = R(vq[it][m]);
            }
        }
#pragma unroll
        for (int it = 0; it < NHI; it++) {
            const int e = tid + it * NT;
            const int ni = e / NJ, nj = e - ni * NJ;
            const int ci = ni - HN, cj = nj - HN;
            const bool xin = ci >= 0 && ci < TI, yin = cj >= 0 && cj < TJ;
            if (e < Cfg::NI * NJ && (xin || yin)) an[e] = vab[it];
        }
#pragma unroll
        for (int it = 0; it < NAI; it++) {
            const int e = tid + it * NT;
            if (e < Cfg::AI * AJ) as[e] = va[it];
        }
    }
    if (HYB) {
        // the flag windows, rows and columns wrapped (doubly periodic), each
        // row dilated over 3 columns
        const int wx = flag_wx(my), wy = flag_wy(my);
        if (tid < Cfg::FXR) {
            int r = i0 - 1 + tid;   // x-face row (faces 0 .. mx, face mx = face 0)
            if (r < 0) r += mx;
            else if (r > mx) r -= mx;
            const unsigned m = mask_row_wrapped(a.flags + size_t(r) * wx, wx, j0 - 1, Cfg::FXC, my);
            fxm[tid] = m | (m >> 1) | (m >> 2);
        } else if (tid >= 32 && tid < 32 + Cfg::FYR) {
            int r = i0 - 1 + (tid - 32);   // y-face row (cell rows 0 .. mx-1)
            if (r < 0) r += mx;
            else if (r >= mx) r -= mx;
            const unsigned m =
                mask_row_wrapped(a.flags + size_t(mx + 1) * wx + size_t(r) * wy, wy, j0 - 1, Cfg::FYC, my);
            fym[tid - 32] = m | (m >> 1) | (m >> 2);
        }
        if (tid < 2) reinterpret_cast<int*>(hyb_base + Cfg::template hyb_ntrb_offset<R>())[tid] = 0;
    }
    __syncthreads();

    // ---- phase 1a: per cell of the cross region, FluxFunc (FluxFunc.cpp:
    // 19-54) halved for the LLF split, and for the cells next to the tile's
    // faces the per-cell terms of SetWaveSpd.cpp:24-72 ----
    for (int e = tid; e < PQ; e += NT) {
        const int ii = e / RJ, jj = e - ii * RJ;
        const bool xin = ii >= H && ii < H + TI, yin = jj >= H && jj < H + TJ;
        if (!xin && !yin) continue;
        const R rho = qs[e], m1 = qs[PQ + e], m2 = qs[2 * PQ + e], m3 = qs[3 * PQ + e], en = qs[4 * PQ + e];
        const R B1 = qs[5 * PQ + e], B2 = qs[6 * PQ + e], B3 = qs[7 * PQ + e];
        const R ir = rcp(rho);
        const R u1 = m1 * ir, u2 = m2 * ir, u3 = m3 * ir;
        const R Bsq = B1 * B1 + B2 * B2 + B3 * B3;
        const R press = (gamma - R(1)) * (en - R(0.5) * rho * (u1 * u1 + u2 * u2 + u3 * u3) - R(0.5) * Bsq);
        const R Bm = R(0.5) * Bsq;
        const R Bu = u1 * B1 + u2 * B2 + u3 * B3;
        const R eb = en + press + Bm;
        if (yin) {
            const int o = ii * FS + (jj - H);
            constexpr int SF = RI * FS;
            fs[o] = R(0.5) * (rho * u1);
            fs[SF + o] = R(0.5) * (rho * u1 * u1 + press + Bm - B1 * B1);
            fs[2 * SF + o] = R(0.5) * (rho * u1 * u2 - B1 * B2);
            fs[3 * SF + o] = R(0.5) * (rho * u1 * u3 - B1 * B3);
            fs[4 * SF + o] = R(0.5) * (u1 * eb - B1 * Bu);
            fs[5 * SF + o] = R(0);
            fs[6 * SF + o] = R(0.5) * (u1 * B2 - u2 * B1);
            fs[7 * SF + o] = R(0.5) * (u1 * B3 - u3 * B1);
        }
        if (xin) {
            const int o = (ii - H) * RJ + jj;
            constexpr int SG = TI * RJ;
            gs[o] = R(0.5) * (rho * u2);
            gs[SG + o] = R(0.5) * (rho * u1 * u2 - B2 * B1);
            gs[2 * SG + o] = R(0.5) * (rho * u2 * u2 + press + Bm - B2 * B2);
            gs[3 * SG + o] = R(0.5) * (rho * u2 * u3 - B2 * B3);
            gs[4 * SG + o] = R(0.5) * (u2 * eb - B2 * Bu);
            gs[5 * SG + o] = R(0.5) * (u2 * B1 - u1 * B2);
            gs[6 * SG + o] = R(0);
            gs[7 * SG + o] = R(0.5) * (u2 * B3 - u3 * B2);
        }
        if (ii >= H - 1 && ii <= H + TI && jj >= H - 1 && jj <= H + TJ) {
            const R a2c = fabs(gamma * press * ir);
            const R t = a2c + Bsq * ir;
            const R cfc = fsqrt(R(0.5) * (t + fsqrt(fabs(t * t - R(4) * a2c * (B1 * B1) * ir))));
            const int o = (ii - H + 1) * PJ + (jj - H + 1);
            pc[o] = u1;
            pc[PP + o] = u2;
            pc[2 * PP + o] = press;
            pc[3 * PP + o] = cfc;
        }
    }

    // ---- phase 1b: A3 on the tile + 2-cell cross halo: ConstructHJ_L_Order1
    // (ConstructHJ_L.cpp:62-111) and the update of UpdateSoln.cpp:42-47 ----
    {
        const double msx = Max(1e-15, a.hj_in[0]), msy = Max(1e-15, a.hj_in[1]);
        const R eps = MPar<R>::eps(a), pw = MPar<R>::pw(a);
        const double rdx = a.rdx, rdy = a.rdy;
        constexpr int NI = Cfg::NI;
        for (int e = tid; e < NI * NJ; e += NT) {
            const int ni = e / NJ, nj = e - ni * NJ;
            const int ci = ni - HN, cj = nj - HN;   // tile frame
            const bool xin = ci >= 0 && ci < TI, yin = cj >= 0 && cj < TJ;
            if (!xin && !yin) continue;
            const double* A = as + (ci + HA) * AJ + (cj + HA);
            R xs, xd, ys, yd;   // A3xp + A3xm, A3xp - A3xm; the same in y
            if constexpr (sizeof(R) == 4 && (P2 || VER == FIN_WENO_FD)) {
                // the two one-sided values of a direction as one f32x2 pair
                // (their differences run through the same six, backwards)
                auto hj = [&](int st, double rd, R& sum, R& dif) {
                    R d[6];
#pragma unroll
                    for (int k = 0; k < 6; k++) d[k] = R((A[(k - 2) * st] - A[(k - 3) * st]) * rd);
                    f2 e[4];
#pragma unroll
                    for (int k = 0; k < 4; k++) e[k] = f2_make(d[k + 1] - d[k], d[4 - k] - d[5 - k]);
                    const f2 c = weno5_pair_x2<VER>(e[0], e[1], e[2], e[3], R(4) * eps);
                    const R m = fmaf(R(1) / R(6), f2_lo(c), d[2]), p = fmaf(R(1) / R(6), f2_hi(c), d[3]);
                    sum = m + p;
                    dif = p - m;
                };
                hj(AJ, rdx, xs, xd);
                hj(1, rdy, ys, yd);
            } else {
            R in[5];
#pragma unroll
            for (int k = 0; k < 5; k++) in[k] = R((A[(k - 2) * AJ] - A[(k - 3) * AJ]) * rdx);
            const R xm = weno5<R, VER, P2>(in, eps, pw);
#pragma unroll
            for (int k = 0; k < 5; k++) in[k] = R((A[(3 - k) * AJ] - A[(2 - k) * AJ]) * rdx);
            const R xp = weno5<R, VER, P2>(in, eps, pw);
#pragma unroll
            for (int k = 0; k < 5; k++) in[k] = R((A[k - 2] - A[k - 3]) * rdy);
            const R ym = weno5<R, VER, P2>(in, eps, pw);
#pragma unroll
            for (int k = 0; k < 5; k++) in[k] = R((A[3 - k] - A[2 - k]) * rdy);
            const R yp = weno5<R, VER, P2>(in, eps, pw);
            xs = xm + xp; xd = xp - xm; ys = ym + yp; yd = yp - ym;
            }
            const int qe = (ci + H) * RJ + (cj + H);
            const R ir = rcp(qs[qe]);
            const R u1 = qs[PQ + qe] * ir, u2 = qs[2 * PQ + qe] * ir;
            const double La = double(-u1 * R(0.5) * xs - u2 * R(0.5) * ys) + (msx * 0.5 * double(xd) + msy * 0.5 * double(yd));
            an[e] = an[e] + a.bdt * La;   // a1 A + a2 B from phase 0
        }
    }
    __syncthreads();

    // ---- phase 2: the faces (x faces then y faces).  Plain form: one thread
    // per face, the full characteristic WENO flux.  Hybrid form: pass A gives
    // every face its speed and the smooth faces (no troubled flag in the 3 x 3
    // window of same-direction faces) the linear FD5 flux, component by
    // component (linear_face, fin_stage.cuh); the troubled faces go to a list
    // that pass B works through with the full flux ----
    const R ag1 = a.alpha_in ? R(a.alpha_in[0]) : R(0);
    const R ag2 = a.alpha_in ? R(a.alpha_in[1]) : R(0);
    const R eps = MPar<R>::eps(a), pw = MPar<R>::pw(a);
    R smax_x = R(0), smax_y = R(0);
    using DX = MhdDir<R, VER, P2, Cfg, true>;
    using DY = MhdDir<R, VER, P2, Cfg, false>;
    // the face-speed maxima GetCFL reads, and the optional per-face speeds
    auto book = [&](auto dir, int fi, int fj, R alpha) {
        constexpr bool isx = decltype(dir)::value;
        if (!(alpha <= R(1e30))) nonfinite = true;
        const int gi = i0 + fi, gj = j0 + fj;
        if (gi < mx && gj < my && alpha <= R(1e30)) {
            if (isx) smax_x = MaxN(smax_x, alpha);
            else smax_y = MaxN(smax_y, alpha);
        }
        double* const fa = isx ? a.face_alpha_x : a.face_alpha_y;
        if (fa && gi < mx + (isx ? 1 : 0) && gj < my + (isx ? 0 : 1)) fa[size_t(gi) * (my + (isx ? 0 : 1)) + gj] = double(alpha);
    };
    if (HYB) {
        // x and y faces go to lists of their own (face fi NJ + fj); pass A
        // leaves a listed face's speed in its flux slot
        short* tlist = reinterpret_cast<short*>(hyb_base);   // [NFX + NFY]
        int* ntrb = reinterpret_cast<int*>(hyb_base + Cfg::template hyb_ntrb_offset<R>());   // [2]
        auto pass_a = [&](auto dir, R ag, const unsigned* fm, int* count, short* list) {
            constexpr bool isx = decltype(dir)::value;
            using D = typename std::conditional<isx, DX, DY>::type;
#pragma unroll 1
            for (int wb = 0; wb < D::NF; wb += NT) {
                const int w = wb + tid;
                bool push = false;
                int fi = 0, fj = 0;
                if (w < D::NF) {
                    D::locate(w, fi, fj);
                    const R alpha = D::speed(S, gamma, fi, fj, ag);
                    book(dir, fi, fj, alpha);
                    push = (((fm[fi] | fm[fi + 1] | fm[fi + 2]) >> fj) & 1u) != 0;
                    if (push) *D::slot(S, fi, fj) = alpha;
                    else D::linear(a, S, fi, fj, alpha);
                }
                const unsigned bal = __ballot_sync(0xffffffffu, push);
                if (bal) {
                    int base = 0;
                    const int lead = __ffs(bal) - 1;
                    if ((tid & 31) == lead) base = atomicAdd(count, __popc(bal));
                    base = __shfl_sync(0xffffffffu, base, lead);
                    if (push) list[base + __popc(bal & ((1u << (tid & 31)) - 1u))] = short(fi * D::NJ + fj);
                }
            }
        };
        pass_a(std::true_type{}, ag1, fxm, ntrb, tlist);
        pass_a(std::false_type{}, ag2, fym, ntrb + 1, tlist + Cfg::NFX);
        __syncthreads();
        // pass B: x faces, then y faces from the next whole warp on
        const int nx = ntrb[0], ny = ntrb[1], y0 = (nx + 31) & ~31;
#pragma unroll 1
        for (int k = tid; k < y0 + ny; k += NT) {
            if (k < y0) {
                if (k < nx) {
                    const int w = tlist[k], fi = w / DX::NJ, fj = w - fi * DX::NJ;
                    DX::flux(a, S, gamma, eps, pw, fi, fj, *DX::slot(S, fi, fj), neg);
                }
            } else {
                const int w = tlist[Cfg::NFX + k - y0], fi = w / DY::NJ, fj = w - fi * DY::NJ;
                DY::flux(a, S, gamma, eps, pw, fi, fj, *DY::slot(S, fi, fj), neg);
            }
        }
    } else {
        auto face_x = [&](int w) {
            int fi, fj;
            DX::locate(w, fi, fj);
            const R alpha = DX::speed(S, gamma, fi, fj, ag1);
            book(std::true_type{}, fi, fj, alpha);
            DX::flux(a, S, gamma, eps, pw, fi, fj, alpha, neg);
        };
        auto face_y = [&](int w) {
            int fi, fj;
            DY::locate(w, fi, fj);
            const R alpha = DY::speed(S, gamma, fi, fj, ag2);
            book(std::false_type{}, fi, fj, alpha);
            DY::flux(a, S, gamma, eps, pw, fi, fj, alpha, neg);
        };
        // one loop over both directions in FP32, a loop each in FP64 (fewer
        // spills): steps at 1024^2, the other way round, 0.78 against 0.73 ms
        // in FP32 and 1.35 against 1.32 ms in FP64
        static_assert(DX::NF % 32 == 0, "a warp's faces share their direction");
        if constexpr (sizeof(R) == 4) {
#pragma unroll 1
            for (int k = tid; k < DX::NF + DY::NF; k += NT) {
                if (k < DX::NF) face_x(k);
                else face_y(k - DX::NF);
            }
        } else {
#pragma unroll 1
            for (int k = tid; k < DX::NF; k += NT) face_x(k);
#pragma unroll 1
            for (int k = tid; k < DY::NF; k += NT) face_y(k);
        }
    }
    __syncthreads();

    // ---- phase 3: flux difference (ConstructL.cpp:390-401), stage update,
    // constrained transport, next-stage maxima ----
    double cs_x = 0.0, cs_y = 0.0, hx = 0.0, hy = 0.0;
    const double gam = a.gamma;
    for (int c = tid; c < TI * TJ; c += NT) {
        const int ci = c / TJ, cj = c - ci * TJ;
        const int gi = i0 + ci, gj = j0 + cj;
        if (gi >= mx || gj >= my) continue;
        const size_t g = size_t(gi) * my + gj;
        // operand loads ahead of the first use; FP64 takes q_in's own values
        // from shared memory
        double va[MHD_NQ], vb[MHD_NQ], qn[MHD_NQ];
#pragma unroll
        for (int m = 0; m < MHD_NQ; m++) {
            if (a.ct && (m == 5 || m == 6)) continue;
            const double own = sizeof(R) == 8 ? double(qs[m * PQ + (H + ci) * RJ + H + cj]) : 0.0;
            va[m] = !a.A ? 0.0 : sizeof(R) == 8 && a.A == a.qin ? own : a.A[m * a.plane + g];
            vb[m] = !a.B ? 0.0 : sizeof(R) == 8 && a.B == a.qin ? own : a.B[m * a.plane + g];
        }
#pragma unroll
        for (int m = 0; m < MHD_NQ; m++) {
            if (a.ct && (m == 5 || m == 6)) continue;
            const R f1 = Fh[m * Cfg::NFX + (ci + 1) * TJ + cj], f0 = Fh[m * Cfg::NFX + ci * TJ + cj];
            const R g1 = Gh[m * Cfg::NFY + ci * (TJ + 1) + cj + 1], g0 = Gh[m * Cfg::NFY + ci * (TJ + 1) + cj];
            R Lr = -(f1 - f0) * R(a.rdx);
            Lr = Lr - (g1 - g0) * R(a.rdy);
            double v = 0.0;
            if (a.A) v = a.a1 * va[m];
            if (a.B) v = v + a.a2 * vb[m];
            qn[m] = v + a.bdt * double(Lr);
        }
        const double* N = an + (ci + HN) * NJ + (cj + HN);
        if (a.ct) {
            // AfterStep.cpp:39-48 on the updated potential
            qn[5] = a.ct_y * (N[-2] - 8 * N[-1] + 8 * N[1] - N[2]);
            qn[6] = a.ct_x * (N[-2 * NJ] - 8 * N[-NJ] + 8 * N[NJ] - N[2 * NJ]);
        }
#pragma unroll
        for (int m = 0; m < MHD_NQ; m++) a.qout[m * a.plane + g] = qn[m];
        a.qout[8 * a.plane + g] = N[0];
        // next stage's maxima: GlobalWaveSpd.cpp:71-76 with Ql = Qr (each
        // direction's speed is |u_n| + the cell's fast speed) and the HJ speeds
        const double ir = rcp(qn[0]);
        const double u1 = qn[1] * ir, u2 = qn[2] * ir, u3 = qn[3] * ir;
        if (a.alpha_out) {
            const R Bsq = R(qn[5] * qn[5] + qn[6] * qn[6] + qn[7] * qn[7]);
            const R press =
                R((gam - 1.0) * (qn[4] - 0.5 * qn[0] * (u1 * u1 + u2 * u2 + u3 * u3) - 0.5 * double(Bsq)));
            const R rir = R(ir);
            const R a2c = fabs(gamma * press * rir);
            const R t = a2c + Bsq * rir;
            const R B1 = R(qn[5]);
            const double cfc = double(fsqrt(R(0.5) * (t + fsqrt(fabs(t * t - R(4) * a2c * (B1 * B1) * rir)))));
            const double sx = Max(fabs(u1 - cfc), fabs(u1 + cfc));
            const double sy = Max(fabs(u2 - cfc), fabs(u2 + cfc));
            if (!(sx <= 1e300) || !(sy <= 1e300)) nonfinite = true;
            if (sx <= 1e300) cs_x = Max(cs_x, sx);
            if (sy <= 1e300) cs_y = Max(cs_y, sy);
        }
        if (a.hj_out) {
            // the HJ speeds of q_out, only where a stage produces a state (a
            // right-hand-side evaluation writes L there, whose density
            // entry may be exactly 0)
            const double ax = fabs(u1), ay = fabs(u2);
            if (ax <= 1e300) hx = Max(hx, ax); else nonfinite = true;
            if (ay <= 1e300) hy = Max(hy, ay); else nonfinite = true;
        }
    }

    // ---- block reductions, one atomic per maximum ----
    const double v6[6] = {double(smax_x), double(smax_y), cs_x, cs_y, hx, hy};
#pragma unroll
    for (int k = 0; k < 6; k++) {
        const double v = warp_max_nonneg(v6[k]);
        if ((tid & 31) == 0) red[(tid >> 5) * 6 + k] = v;
    }
    if (neg) atomicOr(a.status, 2u);
    if (nonfinite) atomicOr(a.status, 1u);
    __syncthreads();
    if (tid < 6) {
        double v = 0.0;
        for (int wv = 0; wv < NT / 32; wv++) v = Max(v, red[wv * 6 + tid]);
        double* dst = tid < 2 ? a.smax_out : (tid < 4 ? a.alpha_out : a.hj_out);
        if (dst) atomic_max_nonneg(dst + (tid & 1), v);
    }
}

// The maxima of a state already in HBM (GlobalWaveSpd and the HJ speeds),
// for a state that no stage epilogue produced (after a host upload).
__global__ void k_mhd_state_max(const double* q, int mx, int my, size_t plane, double gamma, double* alpha_out,
                                double* hj_out, unsigned int* status);
// B1 = dA3/dy, B2 = -dA3/dx by AfterStep.cpp:39-48 (in place on a state).
__global__ void k_mhd_after_step(double* q, int mx, int my, size_t plane, double ct_y, double ct_x);
// max |D_x B1 + D_y B2| over the interior with D the 4th-order central
// difference of the constrained transport.
__global__ void k_mhd_div_b(const double* q, int mx, int my, size_t plane, double rdx, double rdy, double* out);

}  // namespace fin
