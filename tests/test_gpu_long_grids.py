"""Grids with more rows of tiles than a launch takes blocks in y (65,535): the
spatial orders other than 5 (tiles of 15 rows) and the time-integrated fluxes
(blocks of 8).  The state repeats with a short period along x, so the result
has to repeat the short periodic grid's; tolerance 1e-13 relative L-infinity
(the same operations on the same values, maybe contracted differently by the
two grids' tile shapes)."""
import numpy as np
import pytest

from conftest import rel_linf
from finess_b200 import problems as P
from finess_b200._abi import FIN_BC_PERIODIC, FIN_TS_LXW, FIN_TS_MD, FIN_TS_RK, FIN_WENO_Z

pytestmark = pytest.mark.gpu
PERIOD = 20


def _step(p, q, dt):
    from finess_b200.solver import Solver
    with Solver(p) as s:
        s.set_state(q)
        cfl = s.step_fixed(dt)
        q1, _ = s.get_state()
    return q1[p.mbc:-p.mbc, p.mbc:-p.mbc], cfl


@pytest.mark.parametrize("copies,order,method,time_order,mpp", [
    (50000, 7, FIN_TS_RK, 1, 0), (50000, 1, FIN_TS_RK, 1, 0), (27000, 5, FIN_TS_MD, 4, 0), (27000, 5, FIN_TS_LXW, 3, 0),
    (27000, 5, FIN_TS_LXW, 2, 1)])
def test_a_million_rows(copies, order, method, time_order, mpp):
    my, dx = 2, 0.03125
    kw = dict(weno=FIN_WENO_Z, mbc=5, space_order=order, time_stepping_method=method, time_order=time_order,
              mpp_limiter=mpp)
    ps, pl = P.riemann_params(n=PERIOD, **kw), P.riemann_params(n=PERIOD * copies, **kw)
    for p in (ps, pl):
        p.my, p.xlow, p.xhigh, p.ylow, p.yhigh = my, 0.0, p.mx * dx, 0.0, my * dx
        p.bc_xlow = p.bc_xhigh = FIN_BC_PERIODIC
    b = ps.mbc
    q = P.random_riemann_state(ps, np.random.default_rng(order))
    ql = np.ones((pl.mx + 2 * b, my + 2 * b, 5))
    ql[b:-b, b:-b] = np.tile(q[b:-b, b:-b], (copies, 1, 1))
    want, cs = _step(ps, q, 0.05 * dx)
    got, cl = _step(pl, ql, 0.05 * dx)
    assert abs(cl - cs) <= 1e-13 * cs
    got = got.reshape(copies, PERIOD, my, 5)
    assert rel_linf(got[0], want) <= 1e-13
    assert np.array_equal(got, np.broadcast_to(got[0], got.shape)) or rel_linf(got, want[None]) <= 1e-13
