"""Many steps on grids so small that several kernels of a step are resident at
once and their buffers (integrated fluxes, stage registers, slots) are written
again a kernel or two later: repeated runs give the same bits, and the oracle's
states within 1e-11 relative L-infinity (the bar of whole frames)."""
import numpy as np
import pytest

from conftest import interior, rel_linf
from finess_b200 import problems as P
from finess_b200._abi import FIN_TS_LXW, FIN_TS_MD, FIN_TS_RK, FIN_WENO_Z

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("method,time_order,mpp", [(FIN_TS_MD, 4, 0), (FIN_TS_LXW, 3, 0), (FIN_TS_LXW, 3, 1),
                                                   (FIN_TS_RK, 3, 0)])
@pytest.mark.parametrize("mx,my", [(7, 16), (31, 50)])
def test_many_small_steps(oracle, mx, my, method, time_order, mpp):
    from finess_b200.solver import Solver
    p = P.riemann_params(n=mx, weno=FIN_WENO_Z, mbc=5, time_stepping_method=method, time_order=time_order,
                         mpp_limiter=mpp)
    p.my, p.yhigh = my, my / mx
    q = oracle.set_bnd(p, P.random_smooth_state(p, np.random.default_rng(mx)))
    n = 40
    dt = p.max_dt = 0.05 / mx
    got = []
    with Solver(p) as s:
        for _ in range(5):
            s.set_state(q)
            s.FinSolveRK(n * dt, [0.0, dt, dt])
            got.append(s.get_state()[0])
    p.mpp_limiter = 0   # nothing to limit in a smooth flow
    qo = oracle.finsolve(p, q, 0.0, n * dt, dt)[1]
    assert all(np.array_equal(got[0], g) for g in got[1:])
    assert rel_linf(interior(p, got[0]), interior(p, qo)) <= 1e-11


def test_published_maxima_repeat():
    """The maxima that a step's last kernel hands to the host belong to that step:
    the CFL numbers of many short steps repeat bit for bit."""
    from finess_b200.mhd import MhdSolver
    from finess_b200.solver import Solver
    p, pm = P.vortex_params(n=24), P.orszag_tang_params(n=24)
    q = P.random_smooth_state(p, np.random.default_rng(3))
    m = P.mhd_random_state(pm, np.random.default_rng(3))
    with Solver(p) as s, MhdSolver(pm) as h:
        runs = []
        for _ in range(4):
            s.set_state(q)
            h.set_state(*m)
            runs.append([(s.step_fixed(1e-3), h.step_fixed(1e-3)) for _ in range(400)])
    assert len(set(a for a, _ in runs[0])) > 300      # every step has maxima of its own
    assert all(r == runs[0] for r in runs[1:])
