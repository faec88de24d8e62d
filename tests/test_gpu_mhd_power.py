"""MHD steps with a power other than 2 (FP32 takes the weights as a call, FP64
inlines them), around the 15 x 16 tile, against the oracle.  Tolerances: FP64
the plain form's 1e-12 relative L-infinity; FP32 1e-5, the bar of the FP32
Euler steps (a step adds dt / dx = 0.05 of fluxes rounded to some ten units of
6e-8)."""
import numpy as np
import pytest

from conftest import interior, rel_linf
from finess_b200 import problems as P
from finess_b200._abi import FIN_PREC_FP32, FIN_PREC_FP64, FIN_WENO_JS, FIN_WENO_Z

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,tol", [(FIN_PREC_FP64, 1e-12), (FIN_PREC_FP32, 1e-5)])
@pytest.mark.parametrize("weno", [FIN_WENO_JS, FIN_WENO_Z])
@pytest.mark.parametrize("power", [1.5, 3.0])
@pytest.mark.parametrize("mx,my", [(15, 16), (16, 17), (44, 31)])
def test_step_with_power(oracle, mx, my, power, weno, prec, tol):
    from finess_b200.mhd import MhdSolver
    p = P.orszag_tang_params(n=mx, weno=weno, power_param=power)
    p.my = my
    q, aux = oracle.mhd_set_bnd(p, *P.mhd_random_state(p, np.random.default_rng(mx)))
    dt = 0.05 * min((p.xhigh - p.xlow) / mx, (p.yhigh - p.ylow) / my)
    q0, a0, _ = oracle.mhd_step_fixed(p, q, aux, dt)
    p.precision = prec
    with MhdSolver(p) as s:
        s.set_state(q, aux)
        s.step_fixed(dt)
        q1, a1, _ = s.get_state()
    assert rel_linf(interior(p, q1), interior(p, q0)) <= tol
    assert rel_linf(interior(p, a1), interior(p, a0)) <= tol
