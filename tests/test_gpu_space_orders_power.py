"""Orders 7, 9 and 11 with a power other than 2, which take tiles of 7 x 16 on
few tiles or a nearly empty last wave (order 11 on all) and of 15 x 16 beyond: at
the smaller tile's edges and on either side of the lines between them (200, 210,
320 and 400 tiles of 15 x 16), against the
numpy restatement and at the tolerance of test_gpu_space_orders_edges.py (the
arithmetic is the same; derived there)."""
import numpy as np
import pytest

from conftest import interior, rel_linf
from finess_b200 import problems as P
from finess_b200._abi import FIN_WENO_JS, FIN_WENO_Z
from test_gpu_space_orders_edges import _construct_l

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order,weno", [(7, FIN_WENO_JS), (7, FIN_WENO_Z), (9, FIN_WENO_JS), (9, FIN_WENO_Z),
                                        (11, FIN_WENO_JS)])
@pytest.mark.parametrize("mx,my,periodic", [(7, 16, True), (6, 17, False), (8, 15, False), (300, 160, True),
                                            (301, 160, False), (300, 241, True), (300, 305, False)])
def test_powers_on_either_tile(oracle, mx, my, periodic, order, weno):
    from finess_b200.solver import Solver
    rng = np.random.default_rng(order * mx + my)
    p = (P.vortex_params if periodic else P.riemann_params)(n=mx, weno=weno, space_order=order, power_param=1.5, mbc=6)
    p.my, p.xlow, p.ylow, p.xhigh, p.yhigh = my, 0.0, 0.0, 1.0, my / mx
    q = oracle.set_bnd(p, P.random_smooth_state(p, rng))
    with Solver(p) as s:
        L, _ = s.ConstructL(q)
    L0, _ = _construct_l(p, q)
    assert rel_linf(interior(p, L), L0) <= 1e-11
