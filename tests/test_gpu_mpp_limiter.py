"""The positivity limiter's kernels against a numpy restatement of
ApplyMPPLimiter2D (apps/2d/euler/lib/ApplyMPPLimiter2D.cpp:27-285) with
ConstructLFL's fluxes (lib/2d/ConstructLFL.cpp:92-108), on the device's own
high-order fluxes, so that only the limiter is compared: grids around the
tile of 16 x 16, a smooth flow (no cell limited), a near-vacuum flow and a mild
one between (cells on both sides of the test that skips the pressure step).

Tolerance 1e-13 relative L-infinity: the update is some twenty correctly rounded
operations on values of the size of the state (numpy rounds each as the device
does; only the wave speeds' maxima may differ by an ulp)."""
import ctypes as C

import numpy as np
import pytest

from conftest import interior, rel_linf
from finess_b200 import problems as P
from finess_b200._abi import FIN_TS_LXW, FIN_WENO_Z

pytestmark = pytest.mark.gpu


def _prim(Q, g):
    u = [Q[..., k] / Q[..., 0] for k in (1, 2, 3)]
    return u, (g - 1.0) * (Q[..., 4] - 0.5 * Q[..., 0] * (u[0] * u[0] + u[1] * u[1] + u[2] * u[2]))


def _flux(Q, n, g):
    u, p = _prim(Q, g)
    rho, un = Q[..., 0], u[n - 1]
    F = [rho * un, rho * un * u[0], rho * un * u[1], rho * un * u[2], un * (Q[..., 4] + p)]
    F[n] = F[n] + p
    return np.stack(F, -1)


def _limited(q, Fx, Fy, p, dt, mb):
    """q: ghosted; Fx (mx+1, my, 5), Fy (mx, my+1, 5): (limited update, smallest factor)."""
    g = p.gamma
    mx, my = p.mx, p.my
    dtx, dty = dt / ((p.xhigh - p.xlow) / mx), dt / ((p.yhigh - p.ylow) / my)
    Q = q[mb:mb + mx, mb:mb + my]
    u, pr = _prim(Q, g)
    c = np.sqrt(np.abs(g * pr / Q[..., 0]))
    ax, ay = np.max(np.abs(u[0]) + c), np.max(np.abs(u[1]) + c)
    Qx, Qy = q[mb - 1:mb + mx + 1, mb:mb + my], q[mb:mb + mx, mb - 1:mb + my + 1]
    fx, fy = _flux(Qx, 1, g), _flux(Qy, 2, g)
    Lx = 0.5 * (fx[:-1] + fx[1:]) + (0.5 * ax) * (Qx[:-1] - Qx[1:])
    Ly = 0.5 * (fy[:, :-1] + fy[:, 1:]) + (0.5 * ay) * (Qy[:, :-1] - Qy[:, 1:])
    fh, fl = [Fx[:-1], Fx[1:], Fy[:, :-1], Fy[:, 1:]], [Lx[:-1], Lx[1:], Ly[:, :-1], Ly[:, 1:]]

    def upd(f):
        return (Q + dtx * (f[0] - f[1])) + dty * (f[2] - f[3])

    eps = 1e-12
    qlf = upd(fl)
    sgn = [dtx, -dtx, dty, -dty]
    ff = [sgn[k] * (fh[k][..., 0] - fl[k][..., 0]) for k in range(4)]
    tot = sum(np.where(x < 0, x, 0.0) for x in ff)
    amin = [np.where(x < 0, np.minimum((eps - qlf[..., 0]) / (tot - eps), 1.0), 1.0) for x in ff]
    scale = [np.ones((mx, my)) for _ in range(4)]
    for combo in range(16):
        on = [(combo >> (3 - k)) & 1 for k in range(4)]
        aa = [on[k] * amin[k][..., None] for k in range(4)]
        qh = upd([aa[k] * fh[k] + (1.0 - aa[k]) * fl[k] for k in range(4)])
        ph = _prim(qh, g)[1]
        bad = ph < 0
        lo, hi, rate = np.zeros_like(ph), np.ones_like(ph), np.zeros_like(ph)
        for _ in range(9):
            rate = (lo + hi) / 2.0
            ph = _prim(rate[..., None] * qh + (1.0 - rate)[..., None] * qlf, g)[1]
            hi, lo = np.where(ph < 0, rate, hi), np.where(ph < 0, lo, rate)
        res = np.where(bad, np.where(ph > 0, rate, lo), 1.0)
        for k in range(4):
            if on[k]:
                scale[k] = np.minimum(scale[k], res)
    am = [scale[k] * amin[k] for k in range(4)]
    tx, ty = np.ones((mx + 1, my)), np.ones((mx, my + 1))
    tx[:-1], ty[:, :-1] = am[0], am[2]
    tx[1:-1], ty[:, 1:-1] = np.minimum(tx[1:-1], am[1][:-1]), np.minimum(ty[:, 1:-1], am[3][:, :-1])
    tx[-1], ty[:, -1] = am[1][-1], am[3][:, -1]
    Hx, Hy = tx[..., None] * (Fx - Lx) + Lx, ty[..., None] * (Fy - Ly) + Ly
    return (Q - dtx * (Hx[1:] - Hx[:-1])) - dty * (Hy[:, 1:] - Hy[:, :-1]), min(a.min() for a in am)


@pytest.mark.parametrize("flow", ["smooth", "mild", "vacuum"])
@pytest.mark.parametrize("mx,my", [(1, 16), (15, 17), (16, 33), (48, 31)])
def test_limiter(oracle, mx, my, flow):
    from finess_b200.solver import Solver
    rng = np.random.default_rng(7 * mx + my)
    p = P.riemann_params(n=mx, weno=FIN_WENO_Z, mbc=5, time_stepping_method=FIN_TS_LXW, time_order=3, mpp_limiter=1)
    p.my, p.yhigh = my, my / mx
    if flow == "smooth":
        q = P.random_smooth_state(p, rng)
    elif flow == "mild":
        q = P.random_riemann_state(p, rng)
    else:
        q = P.double_rarefaction_init(p, speed=2.6, rho=1.0, pr=0.2)
    q = oracle.set_bnd(p, q)
    with Solver(p) as s:
        a1, a2 = s.GlobalWaveSpd(q)
        dt = 0.2 * min((p.xhigh - p.xlow) / mx, (p.yhigh - p.ylow) / my) / max(a1, a2)
        F, G = s.ConstructIntegratedR(dt, q)
        Fh = np.zeros((mx + 1 + 2 * p.mbc, my + 2 * p.mbc, 5))
        Gh = np.zeros((mx + 2 * p.mbc, my + 1 + 2 * p.mbc, 5))
        L, _ = s.ConstructL(q)
        f = s.lib.fin_construct_lxwl
        vp = C.c_void_p
        f.argtypes = [vp] * 8
        assert f(s.h, *[x.ctypes.data_as(vp) for x in (q, F, G, L)], None, *[x.ctypes.data_as(vp) for x in (Fh, Gh)]) == 0
        s.set_state(q)
        s.step_fixed(dt)
        q1, _ = s.get_state()
    b = p.mbc
    ref, least = _limited(q, Fh[b:b + mx + 1, b:b + my], Gh[b:b + mx, b:b + my + 1], p, dt, b)
    assert rel_linf(interior(p, q1), ref) <= 1e-13
    assert flow != "smooth" or least == 1.0
