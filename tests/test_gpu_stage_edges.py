"""The stage kernels at the edges of their tiles: grids of one cell, one less
and one more than a tile, several tiles and a remainder, in every
reconstruction form and with both kinds of boundaries, against the oracle.

Tolerance: the plain form's 1e-12 relative L-infinity.  A right-hand side
divides flux differences by dx, so a relative rounding error u = 1.1e-16 of the
fluxes (some tens of operations deep, fluxes of order 3 here) reaches L as
about 50 u |F| / (dx |L|); on the small grids |L| >= 1 and 1/dx <= 64, hence
below 1.1e-12 in the worst case and far below it in practice (rounding errors
do not align), which leaves room for the finer grids of the tile rule.
"""
import numpy as np
import pytest

from conftest import interior, rel_linf
from finess_b200 import problems as P
from finess_b200._abi import FIN_PREC_FP32, FIN_TS_LXW, FIN_TS_MD, FIN_WENO_FD, FIN_WENO_JS, FIN_WENO_Z

pytestmark = pytest.mark.gpu

TOL = 1e-12


def _problem(mx, my, periodic, weno, power, local, rng):
    p = (P.vortex_params if periodic else P.riemann_params)(n=mx, weno=weno)
    p.my = my
    p.power_param = power
    p.global_alpha = 0 if local else 1
    p.xlow = p.ylow = 0.0
    p.xhigh, p.yhigh = 1.0, my / mx
    q = P.random_smooth_state(p, rng) if periodic else P.random_riemann_state(p, rng)
    return p, q


@pytest.mark.parametrize("weno,power", [(FIN_WENO_JS, 2.0), (FIN_WENO_Z, 2.0), (FIN_WENO_FD, 2.0), (FIN_WENO_JS, 1.5),
                                        (FIN_WENO_Z, 1.5)])
@pytest.mark.parametrize("mx,my,periodic", [(1, 1, False), (1, 40, False), (14, 15, False), (15, 16, True), (16, 17, True),
                                            (3, 64, True), (31, 33, False), (61, 50, True)])
def test_construct_l_and_step_at_tile_edges(oracle, mx, my, periodic, weno, power):
    _check(oracle, mx, my, periodic, weno, power)


# The count of 15 x 16 tiles at which FP64 stages turn from 7 x 16 to 15 x 16
# tiles is 200: grids of 240, 272, 224 (15 x 16 tiles) and of 200, 195 tiles.
@pytest.mark.parametrize("weno,power", [(FIN_WENO_JS, 2.0), (FIN_WENO_Z, 2.0), (FIN_WENO_FD, 2.0), (FIN_WENO_Z, 1.5)])
@pytest.mark.parametrize("mx,my,periodic", [(240, 240, True), (241, 257, False), (209, 255, True), (150, 320, False),
                                            (195, 240, True)])
def test_either_side_of_the_tile_rule(oracle, mx, my, periodic, weno, power):
    _check(oracle, mx, my, periodic, weno, power)


# FP32 stages turn at 74 tiles of 15 x 16: grids of 74, 75, 72 and 1.  A step of
# dt = 0.05 h adds twelve face fluxes of weight 0.05, each within some twenty
# roundings (1.2e-6) of its scale, which is below ten times the state's: 1e-5.
@pytest.mark.parametrize("weno,power", [(FIN_WENO_JS, 2.0), (FIN_WENO_Z, 2.0), (FIN_WENO_FD, 2.0), (FIN_WENO_Z, 1.5)])
@pytest.mark.parametrize("mx,my,periodic", [(30, 592, True), (45, 391, False), (128, 128, True), (7, 16, True)])
def test_either_side_of_the_fp32_tile_rule(oracle, mx, my, periodic, weno, power):
    from finess_b200.solver import Solver
    rng = np.random.default_rng(100 * mx + my)
    p, q = _problem(mx, my, periodic, weno, power, mx % 2 == 0, rng)
    q = oracle.set_bnd(p, q)
    dt = 0.05 * min((p.xhigh - p.xlow) / mx, (p.yhigh - p.ylow) / my)
    qo, cflo = oracle.step_fixed(p, q, dt)
    p.precision = FIN_PREC_FP32
    with Solver(p) as s:
        s.set_state(q)
        cfl = s.step_fixed(dt)
        q1, _ = s.get_state()
    assert rel_linf(interior(p, q1), interior(p, qo)) <= 1e-5
    assert abs(cfl - cflo) <= 1e-5 * cflo


@pytest.mark.parametrize("method,time_order", [(FIN_TS_MD, 4), (FIN_TS_LXW, 3)])
@pytest.mark.parametrize("mx,my", [(241, 225), (64, 49)])
def test_integrated_flux_steps_on_either_tile(oracle, mx, my, method, time_order):
    """Two steps of the multiderivative and Lax-Wendroff methods (1e-11: the
    bar of whole frames)."""
    from finess_b200.solver import Solver
    rng = np.random.default_rng(mx)
    p = P.riemann_params(n=mx, weno=FIN_WENO_Z, mbc=5, time_stepping_method=method, time_order=time_order)
    p.my, p.yhigh = my, my / mx
    q = oracle.set_bnd(p, P.random_smooth_state(p, rng))
    dt = p.max_dt = 0.05 / mx
    with Solver(p) as s:
        s.set_state(q)
        s.FinSolveRK(2 * dt, [0.0, dt, dt])
        q1, _ = s.get_state()
    qo = oracle.finsolve(p, q, 0.0, 2 * dt, dt)[1]
    assert rel_linf(interior(p, q1), interior(p, qo)) <= 1e-11


def _check(oracle, mx, my, periodic, weno, power):
    from finess_b200.solver import Solver
    rng = np.random.default_rng(100 * mx + my)
    p, q = _problem(mx, my, periodic, weno, power, mx % 2 == 0, rng)
    q = oracle.set_bnd(p, q)
    dt = 0.05 * min((p.xhigh - p.xlow) / mx, (p.yhigh - p.ylow) / my)
    with Solver(p) as s:
        L, smax = s.ConstructL(q)
        s.set_state(q)
        cfl = s.step_fixed(dt)
        q1, _ = s.get_state()
    Lo, smo = oracle.construct_l(p, q)
    qo, cflo = oracle.step_fixed(p, q, dt)
    assert rel_linf(interior(p, L), interior(p, Lo)) <= TOL
    assert rel_linf(smax, smo) <= 1e-14
    assert rel_linf(interior(p, q1), interior(p, qo)) <= TOL
    assert abs(cfl - cflo) <= 1e-14 * cflo
