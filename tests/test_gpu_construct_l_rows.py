"""ConstructL's results on their way to the host: L and smax come in chunks of
16,384 doubles that end anywhere in a row, so the grids here put a chunk's end
on a row's end, inside rows of either parity, and several chunks in one row.
L against the oracle at the plain method's bar; smax is max-accumulated into
what the caller gives, exactly."""
import numpy as np
import pytest

from conftest import interior, rel_linf
from finess_b200 import problems as P
from finess_b200._abi import FIN_WENO_JS, FIN_WENO_Z

pytestmark = pytest.mark.gpu


# smax rows hold 2 (my + 1) doubles, L rows 5 my: 64 x 511 ends chunks of smax
# with its rows; the rows of 2 x 70001 take 21 (L) and 8 (smax) chunks each.
@pytest.mark.parametrize("mx,my", [(64, 511), (131, 257), (301, 263), (2, 70001), (70001, 2)])
@pytest.mark.parametrize("weno,ga", [(FIN_WENO_JS, 1), (FIN_WENO_Z, 0)])
def test_construct_l_rows(oracle, mx, my, weno, ga):
    from finess_b200.solver import Solver
    rng = np.random.default_rng(mx + my)
    p = P.riemann_params(n=mx, weno=weno, global_alpha=ga)
    p.my = my
    q = oracle.set_bnd(p, P.random_riemann_state(p, rng))
    Lo, so = oracle.construct_l(p, q)
    with Solver(p) as s:
        L, f = s.ConstructL(q)
        given = rng.uniform(-2.0, 2.0, f.shape) * f.max()
        given[rng.random(f.shape) < 0.05] = np.nan
        keep = given.copy()
        L2, sm = s.ConstructL(q, given)
    assert rel_linf(interior(p, L), interior(p, Lo)) <= 1e-12
    frame = np.ones(L.shape, bool)
    frame[p.mbc:-p.mbc, p.mbc:-p.mbc] = False
    assert np.all(L[frame] == 0.0)              # ghosts stay as the caller made them
    assert rel_linf(f, so) <= 1e-14
    assert np.array_equal(L, L2) and np.array_equal(given, keep, equal_nan=True)
    face = np.zeros(f.shape, bool)
    face[p.mbc:p.mbc + mx + 1, p.mbc:p.mbc + my, 0] = True
    face[p.mbc:p.mbc + mx, p.mbc:p.mbc + my + 1, 1] = True
    assert np.all(f[~face] == 0.0) and np.all(f[face] > 0.0)
    want = np.where(face & ~(given > f), f, given)   # Max(a, b) = a > b ? a : b
    assert np.array_equal(sm, want, equal_nan=True)
