"""FP64 MHD right-hand sides of states whose transverse field falls to 1e-9 in
strips: the scalars of the eigenvectors may not lose digits against the
reference's own chain of operations.

Tolerance 1e-14 relative L-infinity, ninety roundings (2^-53): a face's flux is
of the size of L dx and comes from some forty roundings of its own, whatever
the chain; the rest is for scalars off by a hundred roundings on the faces
beside the rule's line, which reach the flux through the nonlinear weights
only."""
import numpy as np
import pytest

from conftest import interior, rel_linf
from finess_b200 import problems as P
from finess_b200._abi import FIN_WENO_JS, FIN_WENO_Z

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("weno", [FIN_WENO_JS, FIN_WENO_Z])
@pytest.mark.parametrize("seed", range(3, 9))
def test_small_transverse_field(oracle, weno, seed):
    from finess_b200.mhd import MhdSolver
    p = P.orszag_tang_params(n=96, weno=weno, global_alpha=1)
    p.my = 40
    q, aux = P.mhd_random_state(p, np.random.default_rng(seed))
    kin, mag = 0.5 * (q[..., 1:4] ** 2).sum(-1) / q[..., 0], 0.5 * (q[..., 5:8] ** 2).sum(-1)
    pr = (p.gamma - 1) * (q[..., 4] - kin - mag)
    q[..., 6:8] *= (10.0 ** -((np.arange(q.shape[0]) // 8) % 10))[:, None, None]
    q[..., 4] = pr / (p.gamma - 1) + kin + 0.5 * (q[..., 5:8] ** 2).sum(-1)
    q, aux = oracle.mhd_set_bnd(p, q, aux)
    L0, _ = oracle.mhd_construct_l(p, q)
    with MhdSolver(p) as s:
        L, _ = s.ConstructL(q, aux)
    assert rel_linf(interior(p, L), interior(p, L0)) <= 1e-14
