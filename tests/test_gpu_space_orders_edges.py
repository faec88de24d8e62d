"""The fused stage of the spatial orders 1, 7, 9, 11 at the edges of its tiles,
against a numpy restatement with the scheme built from first principles
(candidate values, linear weights and smoothness forms of the interpolating
polynomials in exact fractions, with the factors the reference's forms carry):
one cell, a cell less and more than a tile, several tiles, both boundary kinds,
powers other than 2.

Tolerance 1e-11 relative L-infinity of L: the forms are evaluated on differences
on both sides, so their relative rounding is some hundred ulps (1e-14) however
large the coefficients; a weight passes that on to the flux times the spread
of the candidate values, which over dx is of the size of L; three orders are left
for the projections and the division by dx (as in the FP64 form's frames)."""
import math
from fractions import Fraction as Fr

import numpy as np
import pytest

from conftest import interior, rel_linf
from finess_b200 import problems as P
from finess_b200._abi import FIN_WENO_FD, FIN_WENO_JS, FIN_WENO_Z

pytestmark = pytest.mark.gpu
SCALE = {7: 240, 9: 5040, 11: 120960}


def _scheme(order):
    r = (order + 1) // 2

    def poly(points):
        n = len(points)
        M = [[(Fr(2 * c + 1, 2) ** (k + 1) - Fr(2 * c - 1, 2) ** (k + 1)) / (k + 1) for k in range(n)]
             + [Fr(int(i == j)) for j in range(n)] for i, c in enumerate(points)]
        for i in range(n):
            M[i] = [v / M[i][i] for v in M[i]] if M[i][i] else M[i]
            if not M[i][i]:
                k = next(k for k in range(i, n) if M[k][i])
                M[i], M[k] = M[k], M[i]
                M[i] = [v / M[i][i] for v in M[i]]
            for k in range(n):
                if k != i and M[k][i]:
                    M[k] = [a - M[k][i] * b for a, b in zip(M[k], M[i])]
        return [[M[k][n + j] for k in range(n)] for j in range(n)]

    def half(P_):
        return [sum(c * Fr(1, 2) ** k for k, c in enumerate(row)) for row in P_]

    def integral(a, b):
        return sum(u * v * 2 * Fr(1, 2) ** (i + j + 1) / (i + j + 1) for i, u in enumerate(a) for j, v in enumerate(b)
                   if (i + j) % 2 == 0)

    cand, forms = [], []
    for k in range(r):
        D = poly(list(range(k - r + 1, k + 1)))
        cand.append(half(D))
        form = [[Fr(0)] * r for _ in range(r)]
        for _ in range(1, r):
            D = [[q * v for q, v in enumerate(c)][1:] for c in D]
            form = [[form[i][j] + integral(D[i], D[j]) for j in range(r)] for i in range(r)]
        forms.append([[float(v * SCALE[order]) for v in row] for row in form])
    full, lin = half(poly(list(range(1 - r, r)))), []
    for k in range(r):
        d = full[k] / cand[k][0]
        lin.append(float(d))
        for j in range(r):
            full[k + j] -= d * cand[k][j]
    return [[float(v) for v in c] for c in cand], lin, forms


def _recon(u, order, ver, eps, pw):
    if order == 1:
        return u[0]
    cand, lin, forms = _scheme(order)
    r = len(lin)
    val, x = [], []
    for k in range(r):
        s = u[k:k + r]
        val.append(u[r - 1] + sum(c * (a - u[r - 1]) for c, a in zip(cand[k], s)))
        # by pairs of differences of neighbours
        e = [s[t + 1] - s[t] for t in range(r - 1)]
        G = [[sum(forms[k][i][j] for i in range(a + 1, r) for j in range(b + 1, r)) for b in range(r - 1)] for a in range(r - 1)]
        x.append(eps + sum(G[a][b] * e[a] * e[b] for a in range(r - 1) for b in range(r - 1)))
    if ver == FIN_WENO_FD:
        w = lin
    elif ver == FIN_WENO_JS:
        w = [g * b ** (-pw) for g, b in zip(lin, x)]
    else:
        tau = np.abs(x[0] + 3 * (x[1] - x[2]) - x[3]) if order == 7 else np.abs(x[4] - x[0])
        w = [g * (1.0 + (tau / b) ** pw) for g, b in zip(lin, x)]
    return sum(a * v for a, v in zip(w, val)) / sum(w)


def _construct_l(p, q):
    from generic_oracle import EulerCallbacks, Max, global_wave_spd
    phys = EulerCallbacks(p.gamma)
    r, nw = (p.space_order + 1) // 2, p.space_order
    mb, mx, my = p.mbc, p.mx, p.my
    ag = global_wave_spd(phys, p, q) if p.global_alpha else (0.0, 0.0)
    F, smax = [], []
    for ixy in (1, 2):
        ni, nj = (mx + 1, my) if ixy == 1 else (mx, my + 1)
        pts = []
        for s in range(2 * r):
            a, b = (mb - r + s, mb) if ixy == 1 else (mb, mb - r + s)
            Q = q[a:a + ni, b:b + nj]
            pts.append((Q, phys.flux(0, 0, Q)[ixy - 1]))
        Ql, Qr = pts[r - 1][0], pts[r][0]
        s1, s2 = phys.wave_speed(*((1.0, 0.0) if ixy == 1 else (0.0, 1.0)), 0, 0, Ql, Qr)
        alpha = Max(ag[ixy - 1], Max(np.abs(s1), np.abs(s2)))
        la = (p.alpha_scaling * alpha)[..., None]
        E = phys.face(ixy, 0.5 * (Qr + Ql))
        gp = [0.5 * (phys.left(E, f) + la * phys.left(E, Q)) for Q, f in pts]
        gm = [0.5 * (phys.left(E, f) - la * phys.left(E, Q)) for Q, f in pts]
        a = (p.space_order, p.weno_version, p.epsilon, p.power_param)
        F.append(phys.right(E, _recon(gp[:nw], *a) + _recon(gm[:0:-1][:nw], *a)))
        smax.append(alpha)
    dx, dy = (p.xhigh - p.xlow) / mx, (p.yhigh - p.ylow) / my
    return -(F[0][1:] - F[0][:-1]) / dx - (F[1][:, 1:] - F[1][:, :-1]) / dy, smax


@pytest.mark.parametrize("order,weno,power", [(1, FIN_WENO_JS, 2.0), (7, FIN_WENO_JS, 2.0), (7, FIN_WENO_Z, 2.0),
                                              (7, FIN_WENO_FD, 2.0), (7, FIN_WENO_JS, 1.5), (9, FIN_WENO_JS, 2.0),
                                              (9, FIN_WENO_Z, 2.0), (9, FIN_WENO_Z, 1.5), (9, FIN_WENO_FD, 2.0),
                                              (11, FIN_WENO_JS, 2.0), (11, FIN_WENO_JS, 1.5)])
@pytest.mark.parametrize("mx,my,periodic", [(1, 1, False), (14, 17, True), (15, 16, False), (33, 50, True)])
def test_construct_l_at_tile_edges(oracle, mx, my, periodic, order, weno, power):
    from finess_b200.solver import Solver
    rng = np.random.default_rng(order * mx + my)
    p = (P.vortex_params if periodic else P.riemann_params)(n=mx, weno=weno, space_order=order, power_param=power, mbc=6)
    p.my, p.xlow, p.ylow, p.xhigh, p.yhigh = my, 0.0, 0.0, 1.0, my / mx
    q = oracle.set_bnd(p, P.random_smooth_state(p, rng))
    with Solver(p) as s:
        L, smax = s.ConstructL(q)
    L0, sm = _construct_l(p, q)
    b = p.mbc
    assert rel_linf(interior(p, L), L0) <= 1e-11
    assert math.isclose(smax[b:b + mx + 1, b:b + my, 0].max(), sm[0].max(), rel_tol=1e-13)
    assert math.isclose(smax[b:b + mx, b:b + my + 1, 1].max(), sm[1].max(), rel_tol=1e-13)
