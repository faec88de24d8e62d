"""ConstructIntegratedR at the edges of its 8 x 16 tiles (the frame of three
ghost cells belongs to them): the 1-state form with and without f_tt against
the oracle at the plain method's bar, the 2-state forms against the sum of
1-state fluxes and of their first time derivatives."""
import ctypes as C

import numpy as np
import pytest

from conftest import rel_linf
from finess_b200 import problems as P
from finess_b200._abi import FIN_BC_PERIODIC, FIN_TS_LXW, FIN_WENO_Z

pytestmark = pytest.mark.gpu


# mx + 6, my + 6: exactly one tile, one cell more, one less, and several tiles
# (periodic directions shorter than the halo are refused)
@pytest.mark.parametrize("mx,my,periodic", [(2, 10, False), (3, 11, False), (1, 9, False), (9, 27, False),
                                            (42, 58, False), (9, 27, True), (42, 58, True)])
def test_integrated_fluxes_at_tile_edges(oracle, mx, my, periodic):
    from finess_b200.solver import Solver
    rng = np.random.default_rng(100 * mx + my)
    p = P.riemann_params(n=mx, weno=FIN_WENO_Z)
    p.my, p.mbc = my, 5
    p.time_stepping_method = FIN_TS_LXW
    if periodic:
        p.bc_xlow = p.bc_xhigh = p.bc_ylow = p.bc_yhigh = FIN_BC_PERIODIC
    qs = [oracle.set_bnd(p, P.random_riemann_state(p, rng)) for _ in range(2)]
    mb, dt = p.mbc, 0.01
    E = (slice(mb - 3, mb + mx + 3), slice(mb - 3, mb + my + 3))
    f, ft = [], []
    for order in (2, 3):
        p.time_order = order
        with Solver(p) as s:
            for q in qs:
                R = s.ConstructIntegratedR(dt, q)
                for a, b in zip(R, oracle.construct_integrated_r(p, dt, q)):
                    assert rel_linf(a[E], b[E]) <= 1e-12
                if order == 2:   # F(dt) = f - dt/2 f_t
                    R0, R2 = s.ConstructIntegratedR(0.0, q), s.ConstructIntegratedR(2.0, q)
                    f.append(np.stack(R0))
                    ft.append(np.stack(R2) - np.stack(R0))
            a1, b1, a2, b2 = 0.7, 0.3, -0.4, 0.9
            want = a1 * f[0] + dt * b1 * ft[0] + a2 * f[1] + dt * b2 * ft[1]
            F, G = np.zeros_like(qs[0]), np.zeros_like(qs[0])
            dp = lambda x: x.ctypes.data_as(C.POINTER(C.c_double))
            d = C.c_double
            assert s.lib.fin_construct_integrated_r2(s.h, d(dt), d(a1), d(b1), dp(qs[0]), d(a2), d(b2), dp(qs[1]),
                                                     dp(F), dp(G)) == 0
            two = np.stack([F, G])
            assert s.lib.fin_construct_integrated_r3(s.h, d(dt), d(a1), d(b1), d(0.0), dp(qs[0]), d(a2), d(b2), d(0.0),
                                                     dp(qs[1]), dp(F), dp(G)) == 0
            three = np.stack([F, G])
            for got in (two, three):   # f_t from a difference of 1-state fluxes: a few roundings of |f| + 2 |f_t|
                scale = max(np.abs(x).max() for x in f) + dt * max(np.abs(x).max() for x in ft)
                assert np.abs(got[:, E[0], E[1]] - want[:, E[0], E[1]]).max() <= 1e-12 * scale
