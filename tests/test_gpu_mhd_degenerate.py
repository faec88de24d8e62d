"""MHD faces on both sides of the rule that picks the short or the reference's
own eigenvalue chain: states whose transverse field, normal field or sound
speed approach the degenerate limits in steps of ten, strip by strip, against
the oracle.

Tolerance 5e-12 relative L-infinity: where the short chain serves, rounding
reaches the eigenvector scalars amplified by at most 1e3 (1e-13), the WENO
weights by about ten times that, and the flux by that times the spread of
the candidate values, whose difference over dx is of the size of L; where the
scalars are worse conditioned the reference's own chain runs."""
import numpy as np
import pytest

from conftest import interior, rel_linf
from finess_b200 import problems as P
from finess_b200._abi import FIN_WENO_JS, FIN_WENO_Z

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("weno", [FIN_WENO_JS, FIN_WENO_Z])
@pytest.mark.parametrize("kind", ["transverse", "normal_x", "normal_y", "umbilic"])
def test_construct_l_near_degenerate_states(oracle, weno, kind):
    from finess_b200.mhd import MhdSolver
    p = P.orszag_tang_params(n=96, weno=weno, global_alpha=1)
    p.my = 40
    q, aux = P.mhd_random_state(p, np.random.default_rng(3))
    i = np.arange(q.shape[0])[:, None]
    scale = 10.0 ** -((i // 8) % 10)          # strips of eight cells, 1 .. 1e-9
    g = p.gamma
    pr = (g - 1) * (q[..., 4] - 0.5 * (q[..., 1:4] ** 2).sum(-1) / q[..., 0] - 0.5 * (q[..., 5:8] ** 2).sum(-1))
    if kind == "transverse":
        q[..., 6] *= scale
        q[..., 7] *= scale
    elif kind == "normal_x":
        q[..., 5] *= scale
    elif kind == "normal_y":
        q[..., 6] *= scale
        q[..., 7] = 0.3 + 0.1 * scale
    else:   # a^2 close to B1^2 / rho with a small transverse field
        q[..., 5] = np.sqrt(g * pr) * (1.0 + 0.3 * scale)
        q[..., 6] *= 0.1 * scale
        q[..., 7] *= 0.1 * scale
    q[..., 4] = pr / (g - 1) + 0.5 * (q[..., 1:4] ** 2).sum(-1) / q[..., 0] + 0.5 * (q[..., 5:8] ** 2).sum(-1)
    q, aux = oracle.mhd_set_bnd(p, q, aux)
    L0, s0 = oracle.mhd_construct_l(p, q)
    with MhdSolver(p) as s:
        L, sm = s.ConstructL(q, aux)
    assert rel_linf(sm, s0) <= 1e-13
    assert rel_linf(interior(p, L), interior(p, L0)) <= 5e-12
